"""The rules on sizes of emerge_gb300/csrc/emg_rules.cuh, compiled on the host."""
import os
import subprocess

from conftest import ROOT


def _run(tmp_path, body):
    src, exe = tmp_path / "rules.cpp", tmp_path / "rules"
    src.write_text('#include <cstdio>\n#include <algorithm>\n#include "emg_rules.cuh"\nusing namespace emg::rules;\n'
                   "int main() {\n" + body + "\nreturn 0; }\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "emerge_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_dot_chains(tmp_path):
    """FP32 sums of a thread are no longer than those over blocks of 1024 rows were (32 rows a lane up to 31
    columns, 1024 a thread from there), for any size; every row is in one block; FP64 has two blocks an SM."""
    _run(tmp_path, r"""
for (long long n : {1ll, 63ll, 64ll, 65ll, 2282ll, 20000ll, 98304ll, 265000ll, 620000ll, 5000000ll, 200000000ll})
    for (long long Bc = 1; Bc <= 700; ++Bc) {
        const long long rows = dot_rows(n, Bc, true), groups = dot_groups(Bc), chain = (std::min(rows, n) + groups - 1) / groups;
        if (chain > (Bc < 32 ? 32 : 1024)) { std::printf("n %lld columns %lld: chain %lld\n", n, Bc, chain); return 1; }
        for (bool f : {false, true})
            if (dot_rows(n, Bc, f) < 1 || dot_rows(n, Bc, f) * dot_blocks(n, Bc, f) < n ||
                dot_rows(n, Bc, f) * (dot_blocks(n, Bc, f) - 1) >= n) { std::printf("blocks %lld %lld\n", n, Bc); return 1; }
        if (dot_blocks(n, Bc, true) < dot_blocks(n, Bc, false)) { std::printf("work space %lld %lld\n", n, Bc); return 1; }
        if (dot_blocks(n, Bc, false) > 304) { std::printf("FP64 blocks %lld %lld\n", n, Bc); return 1; }
        if (dot_groups(Bc) < 1 || dot_tile(Bc) > 128) { std::printf("tile %lld\n", Bc); return 1; }
    }
""")


def test_waits_for_chunks(tmp_path):
    """The waits of the two-buffer pipelines against a model of the barriers: a wait of a parity returns when the
    barrier's current phase has the other one.  The waits after the loop, also when it ends early, cover every
    chunk that is committed and may still run, and none of them outlasts its chunk."""
    _run(tmp_path, r"""
for (int committed = 0; committed <= 40; ++committed)
    for (int done = std::max(0, committed - 2); done <= committed; ++done) {   // chunks 0 .. done - 1 have arrived
        int arrivals[2] = {0, 0};
        for (int c = 0; c < done; ++c) ++arrivals[chunk_buffer(c)];
        auto returns = [&](int c) { return (unsigned)(arrivals[chunk_buffer(c)] & 1) != chunk_parity(c); };
        if (pending_from(committed) < 0 || (committed >= 2 && pending_from(committed) > committed - 2)) return 1;
        for (int c = pending_from(committed); c < committed; ++c)
            if (returns(c) != (c < done)) { std::printf("committed %d done %d chunk %d\n", committed, done, c); return 1; }
    }
for (int ch = 2; ch < 40; ++ch)                    // the wait before a buffer is written again
    for (int done = ch - 2; done <= ch; ++done) {
        int arrivals[2] = {0, 0};
        for (int c = 0; c < done; ++c) ++arrivals[chunk_buffer(c)];
        if (chunk_buffer(ch - 2) != chunk_buffer(ch)) return 1;
        if (((unsigned)(arrivals[chunk_buffer(ch)] & 1) != chunk_parity(ch - 2)) != (done >= ch - 1)) return 1;
    }
""")


def test_pipelines_follow_the_rules():
    """Both two-buffer kernels name their barriers and parities by these rules only."""
    import re
    for name in ("emg_tc.cu", "emg_fp64.cu"):
        text = open(os.path.join(ROOT, "emerge_gb300", "csrc", name)).read()
        waits = re.findall(r"mbar_wait\(smem_u32\(&mbar\[(.*?)\]\), (.*?)\)\)?[; ]", text)
        assert len(waits) == 2 and all("rules::chunk_parity(" in p for _, p in waits), waits
        assert "for (int c = rules::pending_from(committed); c < committed; ++c)" in text

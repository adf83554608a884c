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


def test_narrow_tiles(tmp_path):
    """The choice between 128 x 16 tiles and row blocks or split tiles against measured times (width, groups, columns,
    us of the latter, us of the tiles, whose launch takes 4 more): within 4 % of the faster one."""
    _run(tmp_path, r"""
const struct { int w, G, c; double other, tiles; } t[] = {
{700, 1, 8, 8.5, 32.2}, {700, 1, 16, 8.6, 32.7}, {700, 2, 8, 10.2, 32.3}, {700, 2, 16, 12.8, 32.6}, {700, 3,
8, 10.3, 32.5}, {700, 3, 16, 13.0, 33.0}, {700, 4, 8, 14.4, 32.7}, {700, 4, 16, 18.1, 33.0}, {1000, 1, 8,
11.0, 32.4}, {1000, 1, 16, 11.5, 32.7}, {1000, 2, 8, 13.6, 32.8}, {1000, 2, 16, 17.4, 33.1}, {1000, 3, 8,
19.4, 32.7}, {1000, 3, 16, 24.9, 33.3}, {1000, 4, 8, 23.4, 33.0}, {1000, 4, 16, 24.7, 33.3}, {1250, 1, 8,
15.5, 29.8}, {1250, 1, 16, 20.6, 30.6}, {1250, 2, 8, 23.0, 30.3}, {1250, 2, 16, 29.0, 30.6}, {1250, 3, 8,
29.2, 30.6}, {1250, 3, 16, 29.2, 30.9}, {1250, 4, 8, 51.3, 49.9}, {1250, 4, 16, 52.1, 50.2}, {1500, 1, 8,
18.6, 31.2}, {1500, 1, 16, 20.1, 31.8}, {1500, 2, 8, 26.9, 31.6}, {1500, 2, 16, 33.5, 31.9}, {1500, 3, 8,
33.4, 51.3}, {1500, 3, 16, 33.6, 52.2}, {1500, 4, 8, 59.9, 51.9}, {1500, 4, 16, 60.9, 51.8}, {1750, 1, 8,
21.7, 32.7}, {1750, 1, 16, 22.4, 33.0}, {1750, 2, 8, 31.2, 53.2}, {1750, 2, 16, 38.2, 53.5}, {1750, 3, 8,
70.0, 53.2}, {1750, 3, 16, 70.3, 54.0}, {1750, 4, 8, 72.2, 74.9}, {1750, 4, 16, 73.2, 75.1}, {2000, 1, 8,
30.7, 31.2}, {2000, 1, 16, 47.0, 31.5}, {2000, 2, 8, 44.0, 49.9}, {2000, 2, 16, 44.7, 50.6}, {2000, 3, 8,
87.5, 69.6}, {2000, 3, 16, 88.7, 70.1}, {2000, 4, 8, 88.6, 92.0}, {2000, 4, 16, 90.1, 91.8}, {2250, 1, 8,
35.4, 29.0}, {2250, 1, 16, 51.3, 29.7}, {2250, 2, 8, 46.6, 48.7}, {2250, 2, 16, 47.7, 48.9}, {2250, 3, 8,
91.3, 87.7}, {2250, 3, 16, 92.7, 88.3}, {2250, 4, 8, 92.7, 104.5}, {2250, 4, 16, 93.8, 105.2}, {2500, 1, 8,
50.8, 51.2}, {2500, 1, 16, 51.5, 51.1}, {2500, 2, 8, 98.6, 73.4}, {2500, 2, 16, 98.8, 73.4}, {2500, 3, 8,
99.4, 99.8}, {2500, 3, 16, 101.3, 100.5}, {2500, 4, 8, 192.6, 133.5}, {2500, 4, 16, 194.7, 133.0}};
auto ld = [](long long w) { return (w + 3) / 4 * 4 + 2 + (16 - (w + 3) / 4 * 4 % 16) % 16; };
for (const auto& m : t) {
    const long long rounds = ((m.w + 7) / 8 * m.G + 151) / 152;            // rows8_wins
    const bool rows8 = 64 * ld(m.w) <= 200 * 1024 && (rounds == 1 || rounds * m.w * ((m.c + 7) / 8 * 8) <= 45000);
    const double got = narrow_tiles_win(m.w, m.G, m.c, 8, rows8) ? m.tiles + 4 : m.other;
    if (got > 1.04 * std::min(m.tiles + 4, m.other)) { std::printf("%d %d %d: %g\\n", m.w, m.G, m.c, got); return 1; }
}
if (narrow_tiles_win(2000, 1, 17, 8, false)) return 1;
""")

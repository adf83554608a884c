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

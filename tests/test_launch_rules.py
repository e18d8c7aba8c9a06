"""Rules that choose a launch's shape, checked on the CPU: a small C++ program
built with g++ against the library's headers calls them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "x3div_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    if not shutil.which("g++") or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")

    def build_and_run(name, source):
        d = tmp_path_factory.mktemp(name)
        src, exe = d / "main.cpp", d / "main"
        src.write_text(source)
        subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", CUDA_INC, str(src), "-o", str(exe)],
                       check=True, capture_output=True, text=True)
        return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")

    return build_and_run


X_TILES = r"""
#include <cstdio>
#include "linesolve_chunk.h"
using namespace x3d;
int main()
{
    for (int widest : {16, 32})
        for (int es : {4, 8})
            for (int C = 1; C <= 16; ++C)
                for (long lines : {1L, 600L, 4096L, 8000L, 16384L, 20800L, 40000L, 90000L, 4000000L})
                    std::printf("%d %d %d %ld %d\n", widest, es, C, lines, x_tile_lines(widest, C, lines, 148, es));
    return 0;
}
"""


def test_x_tiles_are_narrow_only_for_short_lines(run):
    got = {}
    for ln in run("x_tiles", X_TILES):
        if ln:
            w, es, c, lines, pick = map(int, ln.split())
            got[w, es, c, lines] = pick
    assert len(got) == 2 * 2 * 16 * 9
    for (w, es, c, lines), pick in got.items():
        assert pick in (8, 16, 32) and pick <= w
        # tiles of three warps or more, and launches that fill the SMs, keep their width
        if c * w > 64 or lines >= 90000:
            assert pick == w, (w, es, c, lines)
    assert [got[32, 4, 1, n] for n in (600, 16384, 40000, 90000)] == [8, 8, 16, 32]
    assert [got[32, 4, 2, n] for n in (600, 4096, 8000)] == [8, 8, 32]
    assert [got[16, 8, 2, n] for n in (600, 16384, 20800)] == [8, 8, 16]


PICKS = r"""
#include <cstdio>
#include "linesolve_chunk.h"
using namespace x3d;
int main()
{
    // a rule that names its arguments, asked for many more keys than slots, in
    // runs and interleaved, each twice
    CfgPicks<64> picks;
    long asked = 0, weighed = 0, wrong = 0;
    auto ask = [&](int dir, int nx, int ny, int nz, int nops, int acc) {
        const CfgKey k{{8, dir, nx, ny, nz, 1, nops, acc, 0, 148}};
        const int want = ((dir * 7 + nx) * 1009 + ny * 13 + nz) * 12 + nops * 2 + acc;
        for (int r = 0; r < 2; ++r) {
            const DefaultCfgs d = picks.get(k, [&] { ++weighed; return DefaultCfgs{1, {want}}; });
            ++asked;
            wrong += d.count != 1 || d.cfg[0] != want;
        }
    };
    for (int pass = 0; pass < 3; ++pass)
        for (int nx = 8; nx < 40; ++nx)
            for (int dir = 0; dir < 3; ++dir)
                for (int nops = 1; nops <= 6; ++nops) ask(dir, nx, 48 - nx, 10 + pass, nops, nops & 1);
    std::printf("%ld %ld %ld\n", asked, weighed, wrong);
    return 0;
}
"""


def test_kept_picks_are_the_rule(run):
    asked, weighed, wrong = map(int, run("picks", PICKS)[0].split())
    assert wrong == 0 and weighed == asked // 2  # new keys throughout: the second of each pair is kept

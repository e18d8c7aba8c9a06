"""The host side of the pressure solve's tables (poisson_tables.h), checked on
the CPU through a small C++ program: a context gets every table its lengths
call for in one block, and none at all where the allocation or the upload
fails, so that a later solve cannot find some of them missing; and the roots
of unity of the cosine transforms are as accurate as doubles can be."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "x3div_b200", "csrc")

HARNESS = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "poisson_tables.h"
using namespace x3d;
static WaveTables wave(int n, double s)
{
    WaveTables w;
    for (int i = 0; i < n; ++i) w.k2.push_back(s + i), w.t.push_back(-s - i);
    return w;
}
// Memory whose allocations and uploads fail on request.
struct Fake {
    bool full, broken;
    int live = 0;
    void *alloc(size_t b) { if (full) return nullptr; ++live; return std::malloc(b); }
    bool upload(void *d, const void *s, size_t b) { if (broken) return false; std::memcpy(d, s, b); return true; }
    void release(void *p) { --live; std::free(p); }
};
int main()
{
    const int sizes[][3] = {{16, 9, 12}, {30, 12, 24}, {1536, 8, 40}, {18, 12, 10}, {17, 8, 8}, {2048, 10, 1024}};
    for (auto &n : sizes) {
        const PoissonTables p = poisson_host_tables(wave(n[0], 100), wave(n[1], 200), wave(n[2], 300));
        const double *b = p.block.data();
        bool ok = p.k2x == 0;
        for (int i = 0; i < n[0]; ++i) ok = ok && b[p.k2x + i] == 100 + i && b[p.tx + i] == -100 - i;
        for (int i = 0; i < n[1]; ++i) ok = ok && b[p.k2y + i] == 200 + i && b[p.ty + i] == -200 - i;
        for (int i = 0; i < n[2]; ++i) ok = ok && b[p.k2z + i] == 300 + i && b[p.tz + i] == -300 - i;
        size_t end = 2 * (size_t)(n[0] + n[1] + n[2]);
        if (zft_supported(n[2])) {
            ok = ok && p.ztw == end && b[p.ztw] == 1.0;
            for (int k = 0; k < n[2]; ++k)
                ok = ok && b[p.ztw + 2 * (n[2] + k)] == -300 - k && b[p.ztw + 2 * (n[2] + k) + 1] == 300 + k;
            end += 4 * (size_t)n[2];
        } else ok = ok && p.ztw == 0;
        if (n[0] % 2 == 0 && zft_supported(n[0] / 2)) {
            ok = ok && p.xtw == end && b[p.xtw] == 1.0 && b[p.xtw + n[0]] == 1.0;
            end += 2 * (size_t)(n[0] + 1);
        } else ok = ok && p.xtw == 0;
        ok = ok && p.block.size() == end && p.ztw % 2 == 0 && p.xtw % 2 == 0;
        std::printf("layout %d %d %d %d\n", n[0], n[1], n[2], ok ? 1 : 0);
    }
    // the largest distance of a table entry from its root of unity, in 2^-54
    auto worst = [](const double *e, int count, long n) {
        const long double turn = 2 * std::acos(-1.0L);
        long double w = 0;
        for (int t = 0; t < count; ++t) {
            w = std::max(w, std::fabs(e[2 * t] - std::cos(turn * t / n)));
            w = std::max(w, std::fabs(e[2 * t + 1] + std::sin(turn * t / n)));
        }
        return (double)std::ldexp(w, 54);
    };
    for (int n = 8; n <= 1024; ++n) {
        if (!zft_supported(n)) continue;
        const std::vector<double> y = cosine_tables(n);
        std::printf("roots %d %.4f\n", n, std::max(worst(&y[0], n, n), worst(&y[2 * n], n, 4L * n)));
    }
    const std::vector<double> block = {1, 2, 3};
    double *out = nullptr;
    auto place = [&](const char *name, bool full, bool broken, Placed want) {
        Fake m{full, broken};
        const bool as = place_block(m, block, &out) == want;
        std::printf("%s %d %d %d\n", name, as, out ? (int)out[2] : 0, m.live);
    };
    place("no_memory", true, false, Placed::no_memory);
    place("no_upload", false, true, Placed::no_upload);
    place("ok", false, false, Placed::ok);
    return 0;
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("tables")
    src, exe = d / "tables.cpp", d / "tables"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")


def test_every_table_in_its_place(lines):
    got = [ln for ln in lines if ln.startswith("layout")]
    assert len(got) == 6 and all(ln.endswith(" 1") for ln in got), got


def test_roots_of_unity_are_rounded_once(lines):
    """Values below 1 rounded to nearest are within 2^-54; the reference here
    adds its own long-double rounding, under 2^-60."""
    got = [float(ln.split()[2]) for ln in lines if ln.startswith("roots")]
    assert len(got) == 15 and max(got) < 1.02, got


def test_a_failure_leaves_no_table(lines):
    # the status, the pointer's third entry (0: not set), blocks still allocated
    assert "no_memory 1 0 0" in lines
    assert "no_upload 1 0 0" in lines
    assert "ok 1 3 1" in lines

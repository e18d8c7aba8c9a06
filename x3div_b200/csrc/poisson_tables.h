// Host side of the pressure solve's tables (poisson.cu): which lengths have own
// transforms, and every table of a context in one block, so that a context has
// either all of them or, after a failed allocation or upload, none.
#pragma once

#include <cmath>
#include <cstddef>
#include <vector>

namespace x3d {

// The lengths with own transforms: 2^p 3^q.
#define X3D_ZFT_SIZES(X) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(384) X(512) X(768) X(1024)

inline bool zft_supported(int n)
{
#define X3D_ZFT_CASE(N) \
    if (n == N) return true;
    X3D_ZFT_SIZES(X3D_ZFT_CASE)
#undef X3D_ZFT_CASE
    return false;
}

// e^{-2 pi i t / n} to within half a unit in the last place: the angle, at most
// an eighth of a turn, and its sine and cosine in long double.
inline void unit_root(long t, long n, double *re, double *im)
{
    t %= n;
    const long q = 4 * t / n, r = 4 * t - q * n;  // quarter turns, and r / n of the next
    const long double half_pi = std::acos(-1.0L) / 2;
    const bool far = 2 * r > n;
    const long double a = half_pi * (far ? n - r : r) / n;
    const double c = (double)(far ? std::sin(a) : std::cos(a)), s = (double)(far ? std::cos(a) : std::sin(a));
    switch (q) {  // (c, -s) turned q quarters clockwise
    case 0: *re = c, *im = -s; break;
    case 1: *re = -s, *im = -c; break;
    case 2: *re = -c, *im = s; break;
    default: *re = s, *im = c; break;
    }
}

// The tables of the cosine transforms of n points (k_dct_y): e^{-2 pi i t / n},
// then e^{-i pi k / 2n}, t, k < n.
inline std::vector<double> cosine_tables(int n)
{
    std::vector<double> tw(4 * (size_t)n);
    for (int t = 0; t < n; ++t) {
        unit_root(t, n, &tw[2 * t], &tw[2 * t + 1]);
        unit_root(t, 4L * n, &tw[2 * ((size_t)n + t)], &tw[2 * ((size_t)n + t) + 1]);
    }
    return tw;
}

// (k2, t) of each mode along one direction.
struct WaveTables {
    std::vector<double> k2, t;
};

// The block, and where each table starts in it (in doubles; complex ones at
// even offsets).  ztw: e^{-2 pi i t / nz}, t < nz, then (t, k2) of each z mode,
// where nz has an own transform; xtw: e^{-2 pi i t / (nx/2)}, t < nx/2, then
// e^{-2 pi i k / nx}, k <= nx/2, where nx / 2 has one; 0 where not.
struct PoissonTables {
    std::vector<double> block;
    size_t k2x = 0, tx = 0, k2y = 0, ty = 0, k2z = 0, tz = 0, ztw = 0, xtw = 0;
};

inline PoissonTables poisson_host_tables(const WaveTables &x, const WaveTables &y, const WaveTables &z)
{
    PoissonTables p;
    auto put = [&](const std::vector<double> &v) {
        const size_t at = p.block.size();
        p.block.insert(p.block.end(), v.begin(), v.end());
        return at;
    };
    p.k2x = put(x.k2), p.tx = put(x.t);
    p.k2y = put(y.k2), p.ty = put(y.t);
    p.k2z = put(z.k2), p.tz = put(z.t);
    const double twopi = 2.0 * std::acos(-1.0);
    const int nx = (int)x.k2.size(), nz = (int)z.k2.size(), m = nx / 2;
    if (zft_supported(nz)) {
        p.ztw = p.block.size();
        for (int t = 0; t < nz; ++t) put({std::cos(twopi * t / nz), -std::sin(twopi * t / nz)});
        for (int k = 0; k < nz; ++k) put({z.t[k], z.k2[k]});
    }
    if (nx % 2 == 0 && zft_supported(m)) {
        p.xtw = p.block.size();
        for (int t = 0; t < m; ++t) put({std::cos(twopi * t / m), -std::sin(twopi * t / m)});
        for (int k = 0; k <= m; ++k) put({std::cos(twopi * k / nx), -std::sin(twopi * k / nx)});
    }
    return p;
}

// A block of doubles on the device: *out is set only when the upload is done
// too.  Mem: alloc(bytes) (null on failure), upload(dst, src, bytes), release(p).
enum class Placed { ok, no_memory, no_upload };
template <typename Mem>
Placed place_block(Mem &mem, const std::vector<double> &block, double **out)
{
    const size_t bytes = block.size() * sizeof(double);
    double *d = static_cast<double *>(mem.alloc(bytes));
    if (!d) return Placed::no_memory;
    if (!mem.upload(d, block.data(), bytes)) {
        mem.release(d);
        return Placed::no_upload;
    }
    *out = d;
    return Placed::ok;
}

}  // namespace x3d

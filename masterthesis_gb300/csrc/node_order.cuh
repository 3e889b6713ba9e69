// Numbers of the inner and the border nodes of a grid and back, by
// multiplications instead of divisions, and column tiles that fit a grid: how
// the kernels without a TMA ring deal a grid out.
#pragma once

#include <stdint.h>

#include "dadd_int.cuh"  // SCAFES_HD

namespace scafes {

// n / d for n < 2^31 by multiplication (round-up method: m = floor(2^32
// (2^s - d) / d) + 1, s = ceil(log2 d)).
struct FastDiv {
    uint32_t d = 1, m = 1, s = 0;
};
inline FastDiv make_fastdiv(uint32_t d) {
    FastDiv f;
    f.d = d;
    while ((1ull << f.s) < d) ++f.s;
    f.m = (uint32_t)((((1ull << f.s) - d) << 32) / d + 1);
    return f;
}
SCAFES_HD uint32_t fastdiv(uint32_t n, const FastDiv& f) {
#if defined(__CUDA_ARCH__)
    return (__umulhi(n, f.m) + n) >> f.s;
#else
    return (uint32_t)((((uint64_t)n * f.m) >> 32) + n) >> f.s;
#endif
}

// Numbering of the inner and of the border nodes of a grid with nl border
// layers, both in Fortran order (x fastest).
struct NodeOrder {
    uint32_t n_inner, n_border;
    uint32_t nx, ny, nz, nl;
    uint32_t zfull, mid;      // nodes of a border plane; border nodes of another plane
    FastDiv ix, ixy;          // inner extents: x, x * y
    FastDiv x, xy, pm, pair;  // nx, nx * ny, mid, 2 * nl
};
inline NodeOrder make_node_order(int nx, int ny, int nz, int nl) {
    NodeOrder o;
    o.nx = (uint32_t)nx, o.ny = (uint32_t)ny, o.nz = (uint32_t)nz, o.nl = (uint32_t)nl;
    const uint32_t ix = o.nx - 2 * o.nl, iy = o.ny - 2 * o.nl, iz = o.nz - 2 * o.nl;  // nl <= min(n) / 2
    o.n_inner = ix * iy * iz;
    o.n_border = o.nx * o.ny * o.nz - o.n_inner;
    o.zfull = o.nx * o.ny;
    o.mid = 2 * o.nl * o.nx + iy * 2 * o.nl;
    o.ix = make_fastdiv(ix ? ix : 1);
    o.ixy = make_fastdiv(ix * iy ? ix * iy : 1);
    o.x = make_fastdiv(o.nx);
    o.xy = make_fastdiv(o.zfull);
    o.pm = make_fastdiv(o.mid);
    o.pair = make_fastdiv(2 * o.nl);
    return o;
}
SCAFES_HD void inner_node(const NodeOrder& o, uint32_t m, int& x, int& y, int& z) {
    const uint32_t k = fastdiv(m, o.ixy), r = m - k * o.ixy.d, j = fastdiv(r, o.ix);
    x = (int)(r - j * o.ix.d + o.nl);
    y = (int)(j + o.nl);
    z = (int)(k + o.nl);
}
SCAFES_HD void border_node(const NodeOrder& o, uint32_t m, int& x, int& y, int& z) {
    const uint32_t low = o.nl * o.zfull, middle = (o.nz - 2 * o.nl) * o.mid;
    uint32_t r;
    if (m < low || m >= low + middle) {  // a plane within nl of a z face
        const uint32_t q = m < low ? m : m - low - middle;
        const uint32_t k = fastdiv(q, o.xy);
        r = q - k * o.zfull;
        z = (int)(m < low ? k : o.nz - o.nl + k);
        const uint32_t j = fastdiv(r, o.x);
        y = (int)j;
        x = (int)(r - j * o.nx);
        return;
    }
    const uint32_t k = fastdiv(m - low, o.pm);
    r = m - low - k * o.mid;
    z = (int)(k + o.nl);
    const uint32_t rows = o.nl * o.nx, sides = (o.ny - 2 * o.nl) * 2 * o.nl;
    if (r < rows || r >= rows + sides) {  // a row within nl of a y face
        const uint32_t q = r < rows ? r : r - rows - sides;
        const uint32_t j = fastdiv(q, o.x);
        y = (int)(r < rows ? j : o.ny - o.nl + j);
        x = (int)(q - j * o.nx);
        return;
    }
    r -= rows;
    const uint32_t j = fastdiv(r, o.pair), i = r - j * 2 * o.nl;
    y = (int)(j + o.nl);
    x = (int)(i < o.nl ? i : o.nx - 2 * o.nl + i);
}

constexpr int MARCH_THREADS = 256;

// The columns of a CTA: w x h threads (h R rows), w h <= MARCH_THREADS.
// FP64 pays for every warp whatever its active lanes, and 32 columns at a
// time leave up to a quarter of them idle (98 inner columns: 98 of 128), so
// the width follows the grid: the (w, h) with the fewest idle threads, w
// at most 64, no more tiles than ceil(columns / 16) (so w is at least 9 where
// the grid has them; 31 x 14 x 21 FP64 Lame takes 5 % longer with tiles of 29
// columns than of 15), h at most 16 (sectors; rows that share their y
// neighbours in L1; the halos that callers keep in shared memory).  Launches
// call it, so the search is over the widths, whatever the grid's.
struct ColumnTile {
    FastDiv w;
    int h, nx, ny;  // rows of threads; tiles along x and y
};
inline ColumnTile make_column_tile(int ix, int iy, int rows) {
    ColumnTile t;
    t.h = t.nx = t.ny = 0;
    if (ix <= 0 || iy <= 0) return t;
    long long best = 0;
    const int ty = (iy + rows - 1) / rows;  // rows of threads
    int last = 0;
    for (int k = ix < 64 ? ix : 64; k > 0; --k) {
        const int n = (ix + k - 1) / k, w = (ix + n - 1) / n;
        if (n > (ix + 15) / 16) break;
        if (n == last) continue;
        last = n;
        const int h = MARCH_THREADS / w < 16 ? MARCH_THREADS / w : 16, m = (ty + h - 1) / h;
        const long long threads = (long long)n * m * MARCH_THREADS;
        if (t.h == 0 || threads < best || (threads == best && h > t.h)) {
            best = threads;
            t.w = make_fastdiv((uint32_t)w);
            t.h = h;
            t.nx = n;
            t.ny = m;
        }
    }
    return t;
}

}  // namespace scafes

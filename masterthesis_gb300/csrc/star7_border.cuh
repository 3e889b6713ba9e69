// The new value of one border node, for the kernels that deal with the border
// nodes apart from the inner ones (star7_loop.cuh, star7_march.cuh), in full
// warps.  Same operations in the same order as the tile engine's border paths,
// inline: a call would pass the job through local memory, which each step of
// a loop finds flushed from L1.
#pragma once

#include "star7_tile.cuh"

namespace scafes {

// `at(dx, dy, dz)` gives the old iterate at the node (0, 0, 0) and at its
// neighbours; it is called for nodes of the grid only.
template <class P, int SRC, int BORDER, class At>
__device__ __forceinline__ typename P::T border_value_at(const TileJob<typename P::T>& J, int x, int y, int z,
                                                         const At& at) {
    using T = typename P::T;
    const Layout& L = J.L;
    const long long o = L.idx(x, y, z);
    if constexpr (BORDER == SCAFES_BORDER_DIRICHLET) {
        const T v = J.ga ? J.ga[o] : J.gval;
        return J.gb ? P::src(v, J.gb[o], J.time_new, true) : v;
    } else {
        // A neighbour outside the grid reads 0, as from the TMA halo.
        const T u = at(0, 0, 0);
        const T w = x > 0 ? at(-1, 0, 0) : P::zero(), e = x < L.nx - 1 ? at(1, 0, 0) : P::zero();
        const T s = y > 0 ? at(0, -1, 0) : P::zero(), n = y < L.ny - 1 ? at(0, 1, 0) : P::zero();
        const T b = z > 0 ? at(0, 0, -1) : P::zero(), t = z < L.nz - 1 ? at(0, 0, 1) : P::zero();
        if constexpr (BORDER == SCAFES_BORDER_NODES) {
            return node_rule_value<P>(J, x, y, z, u, w, e, s, n, b, t);
        } else if constexpr (BORDER == SCAFES_BORDER_TABLE) {
            const int mask = (x == 0) | ((x == L.nx - 1) << 1) | ((y == 0) << 2) | ((y == L.ny - 1) << 3) |
                             ((z == 0) << 4) | ((z == L.nz - 1) << 5);
            return table_rule_value<P, SRC != SRC_NONE, SRC == SRC_AB>(J, mask, o, u, w, e, s, n, b, t);
        } else {
            // Mirror border: the last face (in direction order x-, x+, y-,
            // y+, z-, z+) the node lies on decides.
            T opp;
            bool minus;
            if (z == L.nz - 1)      { opp = b; minus = true; }
            else if (z == 0)        { opp = t; minus = false; }
            else if (y == L.ny - 1) { opp = s; minus = true; }
            else if (y == 0)        { opp = n; minus = false; }
            else if (x == L.nx - 1) { opp = w; minus = true; }
            else                    { opp = e; minus = false; }
            return P::mirror(u, opp, minus ? negated(J.corr) : J.corr);
        }
    }
}

// The same from the old iterate in global memory.
template <class P, int SRC, int BORDER>
__device__ __forceinline__ typename P::T border_value(const TileJob<typename P::T>& J, const typename P::T* uo, int x,
                                                      int y, int z) {
    const Layout& L = J.L;
    const long long o = L.idx(x, y, z);
    return border_value_at<P, SRC, BORDER>(J, x, y, z, [&](int dx, int dy, int dz) {
        return uo[o + dx + dy * (long long)L.pitch + dz * L.plane];
    });
}

}  // namespace scafes

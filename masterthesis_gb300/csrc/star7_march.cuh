// One time step by plain loads: a thread owns R rows of a column and marches
// z, with below, current and above in registers and the x and y neighbours
// through L1 (which holds them from their own "above" loads a plane
// earlier).  The border nodes are left to CTAs of their own at the front of
// the grid, in full warps (star7_border.cuh); the marching threads compute
// inner nodes only, so every border kind, source and layer count is one
// kernel and no warp at a face runs a rule for one or two lanes.
//
// The FP64 sweep is bound by the FP64 pipe (16 to 19 clocks of an SM per warp
// instruction) and the integer ALU, which takes the neighbour sums and half
// or all of the centre's products (star7_policies.cuh).  The tile engine
// (star7_tile.cuh) spends as many instructions again on its ring -- barrier
// waits, block barriers, addresses -- as on the node: 268 issued per 32
// nodes, where this loop took 175 with the same arithmetic, and the memory
// path does not need the ring, since FP64 asks it for 2 TB/s.  us per step at
// 512^3 / 256^3: tile 1178 / 175; this loop 1093 / 150, with the adder of
// dadd_int.cuh as it is now 1077 / 145, with overlapped launches 1072 / 141, with
// every second plane's products on the integer pipe 1015 / 135 (132 GLUP/s).
// Six CTAs of 256 threads (40 registers, nothing spilled): 4, 5 and 8 CTAs
// measured 2 % to 0.2 % slower.
// FP32 and pairs are bound by the memory path, where the tile engine's ring
// keeps more bytes in flight (f32 400^3 89 against 123 us); they come here
// with rule tables, pairs with a source affine in time, and some grids with
// several border layers (star7_default_tile).
#pragma once

#include <algorithm>

#include "node_order.cuh"
#include "star7_border.cuh"
#include "step_launch.cuh"

namespace scafes {

template <class T>
struct MarchArgs {
    const T* uo;
    T* un;
    const T* fa;
    const T* fb;
    const T* ga;
    const T* gb;
    T gval;
    const T* c0;
    const T* ca;
    Layout L;
    NodeOrder o;
    Star7Coeffs c;
    const BorderTable* table;
    const scafes_border_node_rule* nodes;
    StepTimes t;
    uint32_t border_ctas;
    ColumnTile ct;
    FastDiv tx, txy;  // tiles along x, tiles of a layer
    int zchunk;
    const int* status;
};

// The R rows from row y of column x, planes [z0, z1), all of them inner
// planes and (row y, column x) an inner one.
template <class P, int SRC, bool VC, int R>
__device__ __forceinline__ void march_rows_of(const Layout& L, const Star7Coeffs& c, const typename P::T* __restrict__ uo,
                                              typename P::T* __restrict__ un, const typename P::T* __restrict__ fa,
                                              const typename P::T* __restrict__ fb,
                                              const typename P::T* __restrict__ c0f,
                                              const typename P::T* __restrict__ caf, const Split& t_old, int x, int y,
                                              int z0, int z1) {
    using T = typename P::T;
    constexpr bool HAS_F = SRC != SRC_NONE;
    constexpr bool has_fb = SRC == SRC_AB;
    const long long py = L.pitch, pz = L.plane;
    long long o = L.idx(x, y, z0);
    after_wait(o);
    // Rows that are border rows are computed but not stored; a row beyond the
    // grid reads the last one.
    unsigned skip = 0u;
    long long ro[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        ro[i] = (min(y + i, L.ny - 1) - y) * py;
        if (y + i >= L.ny - L.nl) skip |= 1u << i;
    }
    const long long rn = (min(y + R, L.ny - 1) - y) * py;
    // With a source or node coefficients, what streams from memory (they and
    // the plane above) is loaded a plane before it is used: FP64 ensemble 311
    // -> 303 us, 256^3 with a source 160 -> 156; without, it costs 141 -> 145.
    constexpr bool AHEAD = R == 1 && (HAS_F || VC);
    T below[R], cur[R], above[R], f[R], c0[R], ca[R];
    auto fetch = [&](long long m, T (&fo)[R], T (&c0o)[R], T (&cao)[R]) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            fo[i] = P::zero();
            if (HAS_F) fo[i] = P::src(fa[m + ro[i]], has_fb ? fb[m + ro[i]] : P::zero(), t_old, has_fb);
            if constexpr (VC) {
                c0o[i] = c0f[m + ro[i]];
                cao[i] = caf[m + ro[i]];
            }
        }
    };
#pragma unroll
    for (int i = 0; i < R; ++i) {
        below[i] = uo[o + ro[i] - pz];
        cur[i] = uo[o + ro[i]];
        if (AHEAD) above[i] = uo[o + ro[i] + pz];
    }
    if (AHEAD) fetch(o, f, c0, ca);
    // Without a source the FP64 update is short of either pipe by turns:
    // bound by the integer ALU (76 % busy, FP64 61 %) with every c0 u there, by
    // FP64 (82 %, ALU 55 %) with none, 141 us at 256^3 both ways.  Every second
    // plane's goes to the FP64 pipe: 135 us, at 512^3 1072 -> 1015.
    constexpr bool HALF = std::is_same<P, PolF64>::value && !HAS_F && !VC;
    auto plane = [&](int z, auto int_mul) {
        T w[R], e[R], v[R], next[R], fn[R], c0n[R], can[R];
        const long long on = z + 1 < z1 ? o + pz : o;  // the last plane loads its own again
        const T ym = uo[o - py], yp = uo[o + rn];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (AHEAD) next[i] = uo[on + ro[i] + pz];
            else above[i] = uo[o + ro[i] + pz];
            w[i] = uo[o + ro[i] - 1];
            e[i] = uo[o + ro[i] + 1];
        }
        if (AHEAD) fetch(on, fn, c0n, can);
        else fetch(o, f, c0, ca);
        if constexpr (VC)
            P::template star_vc_rows<HAS_F, R>(c, below, cur, above, ym, yp, w, e, f, c0, ca, 1, v, skip);
        else
            P::template star_rows<HAS_F, R, decltype(int_mul)::value>(c, below, cur, above, ym, yp, w, e, f, v, skip);
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (R == 1 || !((skip >> i) & 1u)) un[o + i * py] = v[i];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            below[i] = cur[i];
            cur[i] = above[i];
            if (AHEAD) {
                above[i] = next[i];
                f[i] = fn[i];
                c0[i] = c0n[i];
                ca[i] = can[i];
            }
        }
        o += pz;
    };
    int z = z0;
#pragma unroll 1
    for (; z + 1 < z1; z += 2) {
        plane(z, std::true_type{});
        plane(z + 1, std::integral_constant<bool, !HALF>{});
    }
    if (z < z1) plane(z, std::true_type{});
}

template <class P, int SRC, int BORDER, bool VC, int R, int MINB>
__global__ void __launch_bounds__(MARCH_THREADS, MINB)
star7_march(const __grid_constant__ MarchArgs<typename P::T> A) {
    using T = typename P::T;
    const Layout& L = A.L;
    step_wait();
    if (*(const volatile int*)A.status != 0) return;  // an earlier sweep gave up
    if (blockIdx.x < A.border_ctas) {
        const uint32_t m = blockIdx.x * (MARCH_THREADS) + threadIdx.x;
        if (m >= A.o.n_border) return;
        TileJob<T> J{nullptr, nullptr, nullptr, A.fa, A.fb, A.ga, A.gb, A.gval, L, A.t.t_old, A.t.t_new, A.t.corr};
        J.table = A.table;
        J.nodes = A.nodes;
        int x, y, z;
        border_node(A.o, m, x, y, z);
        const T* uo = A.uo;
        after_wait(uo);
        A.un[L.idx(x, y, z)] = border_value<P, SRC, BORDER>(J, uo, x, y, z);
        return;
    }
    const uint32_t q = blockIdx.x - A.border_ctas;
    const uint32_t k = fastdiv(q, A.txy), r = q - k * A.txy.d, j = fastdiv(r, A.tx);
    const uint32_t row = fastdiv(threadIdx.x, A.ct.w), col = threadIdx.x - row * A.ct.w.d;
    const int x = (int)((r - j * A.tx.d) * A.ct.w.d + col) + L.nl;
    const int y = ((int)j * A.ct.h + (int)row) * R + L.nl;
    if ((int)row >= A.ct.h || x >= L.nx - L.nl || y >= L.ny - L.nl) return;
    const int z0 = (int)k * A.zchunk + L.nl, z1 = min(z0 + A.zchunk, L.nz - L.nl);
    march_rows_of<P, SRC, VC, R>(L, A.c, A.uo, A.un, A.fa, A.fb, A.c0, A.ca, A.t.t_old, x, y, z0, z1);
    step_next();
}

// ---- host side ---------------------------------------------------------------

// Rows per thread and resident CTAs: pairs work on two rows at once (the
// paired FP32 instructions), the others on one.
template <class P>
constexpr int march_rows() {
    return std::is_same<P, PolF32x2>::value ? 2 : 1;
}
template <class P, int SRC, bool VC>
constexpr int march_ctas() {
    if (std::is_same<P, PolF32x2>::value) return 4;
    return std::is_same<P, PolF64>::value && (SRC != SRC_NONE || VC) ? 5 : 6;
}

template <class P, int SRC, int BORDER, bool VC>
static cudaError_t launch_march_typed(const Star7Launch& a, cudaStream_t stream) {
    using T = typename P::T;
    constexpr int R = march_rows<P>();
    if ((long long)a.L.nx * a.L.ny * a.L.nz >= (1LL << 31)) return cudaErrorInvalidValue;  // 32-bit node numbers
    MarchArgs<T> A;
    A.uo = (const T*)a.uo;
    A.un = (T*)a.un;
    A.fa = (const T*)a.fa;
    A.fb = (const T*)a.fb;
    A.ga = (const T*)a.ga;
    A.gb = (const T*)a.gb;
    A.gval = elem_of<T>(a.gconst);
    A.c0 = (const T*)a.c0;
    A.ca = (const T*)a.ca;
    A.L = a.L;
    A.o = make_node_order(a.L.nx, a.L.ny, a.L.nz, a.L.nl);
    A.c = a.c;
    A.table = a.table;
    A.nodes = a.nodes;
    A.t = StepTimes{make_split(a.time_old), make_split(a.time_new), make_split(a.mirror_corr)};
    A.status = a.status;
    const int nl = a.L.nl, iy = a.L.ny - 2 * nl, iz = a.L.nz - 2 * nl;
    A.border_ctas = (A.o.n_border + MARCH_THREADS - 1) / (MARCH_THREADS);
    // 8 planes per CTA (16 for pairs), 4 while that leaves under two rounds
    // of resident CTAs: 256^3 f64 145, 150, 163 us with 8, 16, 32 planes;
    // 160^3 40.4 with 4, 41.9 with 8; pairs 300 x 280 x 260 108, 104.5, 112
    // with 8, 16, 32.
    int sms = 1, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    A.ct = make_column_tile(a.L.nx - 2 * nl, iy, R);
    const long long tx = A.ct.nx, ty = A.ct.ny;
    int zc = R == 2 ? 16 : 8;
    while (zc > 4 && tx * ty * ((iz + zc - 1) / zc) < 12LL * sms) zc >>= 1;
    const long long tz = std::max(0, (iz + zc - 1) / zc);
    A.zchunk = zc;
    A.tx = make_fastdiv((uint32_t)std::max(1LL, tx));
    A.txy = make_fastdiv((uint32_t)std::max(1LL, tx * ty));
    const long long ctas = A.border_ctas + (A.o.n_inner ? tx * ty * tz : 0);
    if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;
    return launch_step(star7_march<P, SRC, BORDER, VC, R, march_ctas<P, SRC, VC>()>, dim3((unsigned)ctas),
                       dim3(MARCH_THREADS), 0, stream, A);
}

template <class P, int BORDER>
static cudaError_t launch_march_src(const Star7Launch& a, cudaStream_t stream) {
    if (a.fa == nullptr || a.c.cf == 0.0) return launch_march_typed<P, SRC_NONE, BORDER, false>(a, stream);
    if (a.fb == nullptr) return launch_march_typed<P, SRC_A, BORDER, false>(a, stream);
    return launch_march_typed<P, SRC_AB, BORDER, false>(a, stream);
}

template <class P, int BORDER>
static cudaError_t launch_march_vc(const Star7Launch& a, cudaStream_t stream) {
    if constexpr (std::is_same<P, PolF32x2>::value) {
        return cudaErrorInvalidValue;
    } else {
        if (a.fb != nullptr) return cudaErrorInvalidValue;
        if (a.fa == nullptr || a.c.cf == 0.0) return launch_march_typed<P, SRC_NONE, BORDER, true>(a, stream);
        return launch_march_typed<P, SRC_A, BORDER, true>(a, stream);
    }
}

template <class P>
cudaError_t launch_march_prec(const Star7Launch& a, cudaStream_t stream) {
    if (a.vc) {
        switch (a.border) {
            case SCAFES_BORDER_DIRICHLET: return launch_march_vc<P, SCAFES_BORDER_DIRICHLET>(a, stream);
            case SCAFES_BORDER_TABLE: return launch_march_vc<P, SCAFES_BORDER_TABLE>(a, stream);
            case SCAFES_BORDER_NODES: return launch_march_vc<P, SCAFES_BORDER_NODES>(a, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (a.border) {
        case SCAFES_BORDER_DIRICHLET: return launch_march_src<P, SCAFES_BORDER_DIRICHLET>(a, stream);
        case SCAFES_BORDER_MIRROR_POW2: return launch_march_src<P, SCAFES_BORDER_MIRROR_POW2>(a, stream);
        case SCAFES_BORDER_TABLE: return launch_march_src<P, SCAFES_BORDER_TABLE>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace scafes

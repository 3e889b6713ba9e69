// The time loop of a small star7 problem in one cooperative launch.
//
// A sweep of a small grid by the tile engine (star7_tile.cuh) is a chain of
// latencies -- launch, barrier set-up, the first TMA planes, one plane after
// the other -- on a handful of CTAs: 8.2 us a step at 17 x 15 x 16, 17.4 us
// with rule-table borders at 40 x 31 x 27, 10.3 us at 64^3, of which the
// FP64 pipe needs 0.1, 0.5 and 1.7 us.  Here the grid is dealt out node by
// node over all SMs and stays in L2: a thread loads its node's neighbours
// (plain loads, L1 within a step), stores the new value, and one grid-wide
// barrier (a counter in global memory) ends the step.  The inner nodes and
// the border nodes are numbered separately, so a warp holds one kind and the
// border rules (a chain of FP64 operations) run in full warps instead of in
// one or two lanes of every warp at a face.  A step now takes 2.1, 2.7 and
// 4.9 us on those three; of the 2.1 us of an almost empty step, most is the
// round trips to L2 (neighbours, store and release, counter, acquire).  Two
// warps per CTA and up to one CTA per SM: 1, 2 and 4 warps measure the same
// within 2 %, 16 warps 20 % slower at 17 x 15 x 16.
//
// Every node takes the operations of the tile engine in the same order
// (PolX::star / star_vc, table_rule, node_rule, mirror): same bits.
// Co-residency, which the barrier needs, comes from the cooperative launch;
// the barrier's wait is bounded like every other wait (status word, return).
#pragma once

#include <algorithm>

#include "grid_barrier.cuh"
#include "star7_cluster.cuh"

namespace scafes {

constexpr uint32_t LOOP_MIN_WARPS = 2;

// Registers and threads of a CTA leave room for a second loop on every SM where
// that costs little: with 1024 threads of 44 to 64 registers the loops of
// handles on several streams ran one after the other, each alone with its
// barriers (12 loops at 64^3, us per step and handle: FP64 4.8, FP32 2.6,
// pairs 3.0, where tile sweeps had taken 3.5, 1.6 and 1.8).  FP32 and pairs fit
// 32 registers (at most 16 bytes spilled) and 1.6 and 1.9 us, a loop by itself
// is as fast (64^3 2.60 -> 2.56, 3.00 -> 2.94).  FP64 takes 48 registers (none
// spilled), with which CTAs of up to LOOP_TWO_FIT threads go two to an SM.
// Larger ones, below LOOP_FULL_NODES inner nodes: with a Dirichlet border and no
// or a static source 32 registers (56 bytes spilled; 12 loops at 64^3 3.4, one
// 4.81 -> 4.94), else at most LOOP_PAIR_THREADS (3.7, 5.3 -> 5.6; 32 registers
// 4.0 and 5.7).  From there on a loop by itself needs all of both (80^3 7.3, 32
// registers 7.6, 640 threads 8.0) and several gain less.  Rule tables and node
// rules keep 64 registers: their tile sweeps are slower than a loop that waits
// its turn (64^3 FP64 15.4, 5.6).
template <class P, int BORDER>
constexpr int loop_registers() {
    if (BORDER != SCAFES_BORDER_DIRICHLET && BORDER != SCAFES_BORDER_MIRROR_POW2) return 64;
    return std::is_same<P, PolF64>::value ? 48 : 32;
}
constexpr uint32_t LOOP_MAX_THREADS = 1024, LOOP_TWO_FIT = 672, LOOP_PAIR_THREADS = 640;
constexpr uint32_t LOOP_FULL_NODES = 320000;

template <class P, int SRC, int BORDER, bool VC, int REGISTERS>
__global__ void __maxnreg__(REGISTERS)
star7_loop(const __grid_constant__ LoopArgs<typename P::T> A) {
    using T = typename P::T;
    constexpr bool HAS_F = SRC != SRC_NONE;
    constexpr bool has_fb = SRC == SRC_AB;
    if (__syncthreads_or(threadIdx.x == 0 && *(volatile int*)A.status != 0)) return;
    const Layout& L = A.L;
    const long long py = L.pitch, pz = L.plane;
    // This CTA's inner and border nodes; the border nodes start at a warp.
    const uint32_t i0 = blockIdx.x * A.in_cta, i1 = min(i0 + A.in_cta, A.o.n_inner);
    const uint32_t b0 = blockIdx.x * A.bd_cta, b1 = min(b0 + A.bd_cta, A.o.n_border);
    const uint32_t ni = i1 > i0 ? i1 - i0 : 0, nb = b1 > b0 ? b1 - b0 : 0;
    const uint32_t split = (ni + 31) & ~31u;
    TileJob<T> J{nullptr, nullptr, nullptr, A.fa, A.fb, A.ga, A.gb, A.gval, L};
    J.table = A.table;
    J.nodes = A.nodes;
    for (int s = 0; s < A.n_steps; ++s) {
        const T* uo = A.u[(A.first + s) & 1];
        T* un = A.u[(A.first + s + 1) & 1];
        if (A.times) {
            J.time_old = A.times[s].t_old;
            J.time_new = A.times[s].t_new;
            J.corr = A.times[s].corr;
        }
        for (uint32_t j = threadIdx.x; j < split + nb; j += blockDim.x) {
            int x, y, z;
            if (j < split) {
                if (j >= ni) continue;
                inner_node(A.o, i0 + j, x, y, z);
                const long long o = L.idx(x, y, z);
                const T w = uo[o - 1], e = uo[o + 1], sn = uo[o - py], n = uo[o + py], b = uo[o - pz], t = uo[o + pz];
                const T u = uo[o];
                T f = P::zero();
                if (HAS_F) f = P::src(A.fa[o], has_fb ? A.fb[o] : P::zero(), J.time_old, has_fb);
                if constexpr (VC)
                    un[o] = P::template star_vc<HAS_F>(A.c, u, w, e, sn, n, b, t, f, A.c0[o], A.ca[o]);
                else
                    un[o] = P::template star<HAS_F>(A.c, u, w, e, sn, n, b, t, f);
            } else {
                border_node(A.o, b0 + (j - split), x, y, z);
                un[L.idx(x, y, z)] = border_value<P, SRC, BORDER>(J, uo, x, y, z);
            }
        }
        if (s + 1 < A.n_steps && !grid_barrier(A.arrivals, (unsigned)(s + 1) * gridDim.x, A.status)) return;
    }
}

// ---- host side ---------------------------------------------------------------

template <class P, int SRC, int BORDER, bool VC>
static cudaError_t launch_loop_typed(const Star7Loop& q, cudaStream_t stream) {
    using T = typename P::T;
    const Star7Launch& a = q.step;
    LoopArgs<T> A;
    A.u[0] = (T*)q.u[0];
    A.u[1] = (T*)q.u[1];
    A.first = q.first;
    A.n_steps = q.n_steps;
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
    A.times = q.times;
    A.arrivals = q.arrivals;
    A.status = a.status;
    {
        bool done = false;
        const cudaError_t ce = launch_cluster<P, SRC, BORDER, VC>(A, stream, &done);
        if (ce != cudaSuccess || done) return ce;
    }
    // Two warps per CTA at least: fewer CTAs make the barrier cheaper, more
    // spread the FP64 pipe's work; all SMs from 2 * 32 * SMs nodes on.
    const uint32_t wi = (A.o.n_inner + 31) / 32, wb = (A.o.n_border + 31) / 32;
    const uint32_t ctas = std::max(1u, std::min((uint32_t)q.sms, (wi + wb) / LOOP_MIN_WARPS));
    A.in_cta = (A.o.n_inner + ctas - 1) / ctas;
    A.bd_cta = (A.o.n_border + ctas - 1) / ctas;
    const uint32_t want = ((A.in_cta + 31) / 32 + (A.bd_cta + 31) / 32) * 32;
    auto threads_of = [&](uint32_t most) {
        const uint32_t rounds = (want + most - 1) / most;
        return ((want / 32 + rounds - 1) / rounds) * 32;
    };
    constexpr int REGISTERS = loop_registers<P, BORDER>();
    auto kern = star7_loop<P, SRC, BORDER, VC, REGISTERS>;
    uint32_t threads = threads_of(LOOP_MAX_THREADS);
    if constexpr (REGISTERS == 48) {
        if (threads > LOOP_TWO_FIT && A.o.n_inner < LOOP_FULL_NODES) {
            if constexpr (BORDER == SCAFES_BORDER_DIRICHLET && SRC != SRC_AB && !VC)
                kern = star7_loop<P, SRC, BORDER, VC, 32>;
            else
                threads = threads_of(LOOP_PAIR_THREADS);
        }
    }
    cudaError_t e = cudaMemsetAsync(q.arrivals, 0, sizeof(unsigned), stream);
    if (e != cudaSuccess) return e;
    void* args[] = {&A};
    e = cudaLaunchCooperativeKernel((const void*)kern, dim3(ctas), dim3(threads), args, 0, stream);
    return e != cudaSuccess ? e : cudaGetLastError();
}

template <class P, int BORDER>
static cudaError_t launch_loop_src(const Star7Loop& q, cudaStream_t stream) {
    const Star7Launch& a = q.step;
    if (a.fa == nullptr || a.c.cf == 0.0) return launch_loop_typed<P, SRC_NONE, BORDER, false>(q, stream);
    if (a.fb == nullptr) return launch_loop_typed<P, SRC_A, BORDER, false>(q, stream);
    return launch_loop_typed<P, SRC_AB, BORDER, false>(q, stream);
}

template <class P, int BORDER>
static cudaError_t launch_loop_vc(const Star7Loop& q, cudaStream_t stream) {
    if constexpr (std::is_same<P, PolF32x2>::value) {
        return cudaErrorInvalidValue;
    } else {
        const Star7Launch& a = q.step;
        if (a.fb != nullptr) return cudaErrorInvalidValue;
        if (a.fa == nullptr || a.c.cf == 0.0) return launch_loop_typed<P, SRC_NONE, BORDER, true>(q, stream);
        return launch_loop_typed<P, SRC_A, BORDER, true>(q, stream);
    }
}

template <class P>
cudaError_t launch_loop_prec(const Star7Loop& q, cudaStream_t stream) {
    const Star7Launch& a = q.step;
    if (a.vc) {
        switch (a.border) {
            case SCAFES_BORDER_DIRICHLET: return launch_loop_vc<P, SCAFES_BORDER_DIRICHLET>(q, stream);
            case SCAFES_BORDER_TABLE: return launch_loop_vc<P, SCAFES_BORDER_TABLE>(q, stream);
            case SCAFES_BORDER_NODES: return launch_loop_vc<P, SCAFES_BORDER_NODES>(q, stream);
            default: return cudaErrorInvalidValue;
        }
    }
    switch (a.border) {
        case SCAFES_BORDER_DIRICHLET: return launch_loop_src<P, SCAFES_BORDER_DIRICHLET>(q, stream);
        case SCAFES_BORDER_MIRROR_POW2: return launch_loop_src<P, SCAFES_BORDER_MIRROR_POW2>(q, stream);
        case SCAFES_BORDER_TABLE: return launch_loop_src<P, SCAFES_BORDER_TABLE>(q, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace scafes

// The time loop of a very small star7 problem inside one thread-block cluster.
//
// The one-launch loop (star7_loop.cuh) still crosses L2 four times a step --
// stores, barrier counter, its readers, the neighbours -- 2.1 us when there
// is next to nothing to compute.  Here the grid lives in the shared memory of
// up to 16 CTAs of one cluster: each CTA owns a slab of z-planes with a halo
// plane on either side, both iterates, computes it from its own shared
// memory, and writes its first and last plane into the neighbours' halos as
// well (distributed shared memory); one hardware cluster barrier ends the
// step: 1.0 us at 8^3, 1.3 at 17 x 15 x 16
// (FP64).  The known fields are read from global memory.  The iterate comes
// from and goes back to global memory once per launch.
// Nodes of a slab are numbered as in the loop: inner nodes first, border
// nodes in warps of their own; same operations per node, same bits.
#pragma once

#include "per_device.cuh"
#include "star7_loop_args.cuh"

namespace scafes {

constexpr int CLUSTER_MAX = 16;        // CTAs; above 8 needs the non-portable attribute
constexpr int CLUSTER_THREADS = 512;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The address of `p` (shared memory of this CTA) in the CTA of rank `r`.
template <class T>
__device__ __forceinline__ T* in_cta(T* p, uint32_t r) {
    uint64_t q;
    asm volatile("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(reinterpret_cast<uint64_t>(p)), "r"(r));
    return reinterpret_cast<T*>(q);
}

// Planes of CTA `r` of `n`: contiguous, sizes differing by at most one.
__host__ __device__ inline int slab_begin(int nz, int n, int r) { return (int)((long long)nz * r / n); }

// Shared memory of a CTA: two iterates of `planes` + 2 planes of nx * ny nodes.
inline size_t cluster_smem(const Layout& L, int ctas, size_t esz) {
    const int planes = (L.nz + ctas - 1) / ctas + 2;
    return 2 * (size_t)planes * L.nx * L.ny * esz;
}

template <class P, int SRC, int BORDER, bool VC>
__global__ void __launch_bounds__(CLUSTER_THREADS, 1)
star7_cluster(const __grid_constant__ LoopArgs<typename P::T> A) {
    using T = typename P::T;
    constexpr bool HAS_F = SRC != SRC_NONE;
    constexpr bool has_fb = SRC == SRC_AB;
    extern __shared__ __align__(16) unsigned char csm[];
    const Layout& L = A.L;
    const int ctas = (int)gridDim.x, rank = (int)cluster_rank();
    const int za = slab_begin(L.nz, ctas, rank), zb = slab_begin(L.nz, ctas, rank + 1);
    const int np = L.nx * L.ny, planes = (L.nz + ctas - 1) / ctas + 2;  // local plane p holds z = za - 1 + p
    T* buf[2] = {reinterpret_cast<T*>(csm), reinterpret_cast<T*>(csm) + (size_t)planes * np};
    // Every CTA sees the same status: only earlier kernels write it.
    const bool run = *(volatile int*)A.status == 0;
    // The slab's planes and the neighbours' into buffer 0.
    {
        const T* uo = A.u[A.first & 1];
        const int lo = za > 0 ? za - 1 : 0, hi = min(zb + 1, L.nz);
        for (int i = threadIdx.x; i < (hi - lo) * np; i += blockDim.x) {
            const int p = (int)fastdiv((uint32_t)i, A.o.xy), r = i - p * np, y = (int)fastdiv((uint32_t)r, A.o.x);
            buf[0][(lo + p - (za - 1)) * np + r] = uo[L.idx(r - y * L.nx, y, lo + p)];
        }
    }
    cluster_sync();
    // Inner and border nodes of the slab, both a range of the grid's numbers.
    const int nl = L.nl, ixy = (int)A.o.ixy.d;
    auto inner_below = [&](int z) { return (uint32_t)(min(max(z, nl), L.nz - nl) - nl) * (A.o.n_inner ? ixy : 0); };
    auto border_below = [&](int z) { return (uint32_t)z * np - inner_below(z); };
    const uint32_t i0 = inner_below(za), ni = inner_below(zb) - i0;
    const uint32_t b0 = border_below(za), nb = border_below(zb) - b0;
    const uint32_t split = (ni + 31) & ~31u;
    TileJob<T> J{nullptr, nullptr, nullptr, A.fa, A.fb, A.ga, A.gb, A.gval, L};
    J.table = A.table;
    J.nodes = A.nodes;
    for (int s = 0; run && s < A.n_steps; ++s) {
        const T* uo = buf[s & 1];
        T* un = buf[(s & 1) ^ 1];
        T* below = rank > 0 ? in_cta(un, rank - 1) : nullptr;
        T* above = rank + 1 < ctas ? in_cta(un, rank + 1) : nullptr;
        const int top_below = za - slab_begin(L.nz, ctas, rank - 1) + 1;  // the halo plane over the slab below
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
            } else {
                border_node(A.o, b0 + (j - split), x, y, z);
            }
            const int xy = y * L.nx + x, p = z - za + 1, m = p * np + xy;
            T v;
            if (j < split) {
                const long long o = L.idx(x, y, z);
                T f = P::zero();
                if (HAS_F) f = P::src(A.fa[o], has_fb ? A.fb[o] : P::zero(), J.time_old, has_fb);
                if constexpr (VC)
                    v = P::template star_vc<HAS_F>(A.c, uo[m], uo[m - 1], uo[m + 1], uo[m - L.nx], uo[m + L.nx],
                                                   uo[m - np], uo[m + np], f, A.c0[o], A.ca[o]);
                else
                    v = P::template star<HAS_F>(A.c, uo[m], uo[m - 1], uo[m + 1], uo[m - L.nx], uo[m + L.nx],
                                                uo[m - np], uo[m + np], f);
            } else {
                v = border_value_at<P, SRC, BORDER>(
                    J, x, y, z, [&](int dx, int dy, int dz) { return uo[m + dx + dy * L.nx + dz * np]; });
            }
            un[m] = v;
            if (z == za && below) below[top_below * np + xy] = v;
            if (z == zb - 1 && above) above[xy] = v;
        }
        cluster_sync();
    }
    if (!run) return;
    const T* last = buf[A.n_steps & 1];
    T* out = A.u[(A.first + A.n_steps) & 1];
    for (int i = threadIdx.x; i < (zb - za) * np; i += blockDim.x) {
        const int p = (int)fastdiv((uint32_t)i, A.o.xy), r = i - p * np, y = (int)fastdiv((uint32_t)r, A.o.x);
        out[L.idx(r - y * L.nx, y, za + p)] = last[(p + 1) * np + r];
    }
}

// ---- host side ---------------------------------------------------------------

// CTAs of the cluster: 16, or the largest power of two that leaves every CTA
// a plane; 0 where the loop over all SMs is faster, which has ten times the
// FP64 pipes: by the nodes of the largest slab (us per step, cluster / loop):
//   FP64: 17 x 15 x 16 (255 nodes) 1.3 / 2.1, 20^3 (800) 2.25 / 2.14; with node
//     coefficients 1.9 / 2.4 and 2.8 / 2.4;
//   rule tables (FP64 in any type): 8^3 (64) 2.3 / 3.3, 17 x 15 x 16 3.3 / 3.3;
//   pairs: 20^3 1.55 / 1.82, 24^3 (1152) 2.1 / 1.8; FP32 with node
//     coefficients the same within 0.3;
//   FP32: 24^3 1.45 / 1.72, 28^3 (1568) 1.70 / 1.76.
template <class P, int BORDER, bool VC>
int cluster_ctas(const Layout& L, int most) {
    int n = most;
    while (n > L.nz) n >>= 1;
    const long long slab = (long long)((L.nz + n - 1) / n) * L.nx * L.ny;
    const long long limit = BORDER == SCAFES_BORDER_TABLE              ? 200
                            : std::is_same<P, PolF64>::value           ? 350
                            : std::is_same<P, PolF32x2>::value || VC   ? 900
                                                                       : 1500;
    return slab <= limit && cluster_smem(L, n, sizeof(typename P::T)) <= 227 * 1024 ? n : 0;
}

// Runs the loop in one cluster; *done is false where the loop over all SMs is
// the better one or the device cannot hold such a cluster (nothing ran).
template <class P, int SRC, int BORDER, bool VC>
static cudaError_t launch_cluster(const LoopArgs<typename P::T>& A, cudaStream_t stream, bool* done) {
    using T = typename P::T;
    auto kern = star7_cluster<P, SRC, BORDER, VC>;
    *done = false;
    static PerDevice largest;  // cluster the device holds, 0 none
    int dev = 0;
    cudaGetDevice(&dev);
    const int most = largest.get(dev, [&] {
        int most = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess &&
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
            for (int n = CLUSTER_MAX; n >= 1 && most == 0; n >>= 1) {
                cudaLaunchConfig_t cfg = {};
                cudaLaunchAttribute attr = {};
                cfg.gridDim = dim3(n);
                cfg.blockDim = dim3(CLUSTER_THREADS);
                cfg.dynamicSmemBytes = 227 * 1024;
                attr.id = cudaLaunchAttributeClusterDimension;
                attr.val.clusterDim = {(unsigned)n, 1, 1};
                cfg.attrs = &attr;
                cfg.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0) most = n;
            }
        }
        cudaGetLastError();
        return most;
    });
    const int n = most > 0 ? cluster_ctas<P, BORDER, VC>(A.L, most) : 0;
    if (n == 0) return cudaSuccess;
    const uint32_t planes = (A.L.nz + n - 1) / n, np = (uint32_t)A.L.nx * A.L.ny;
    const uint32_t want = (planes * np + 31) / 32 * 32 + 32;
    const uint32_t rounds = (want + CLUSTER_THREADS - 1) / CLUSTER_THREADS;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    cfg.gridDim = dim3(n);
    cfg.blockDim = dim3(((want / 32 + rounds - 1) / rounds) * 32);
    cfg.dynamicSmemBytes = cluster_smem(A.L, n, sizeof(T));
    cfg.stream = stream;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim = {(unsigned)n, 1, 1};
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, A);
    // A cluster that the device will not place has not run: the loop over all
    // SMs takes the steps.
    if (e == cudaErrorInvalidClusterSize || e == cudaErrorInvalidConfiguration || e == cudaErrorLaunchOutOfResources) {
        cudaGetLastError();
        return cudaSuccess;
    }
    *done = true;
    return e;
}

}  // namespace scafes

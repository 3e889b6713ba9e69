// Launches of step kernels that follow one another on a stream, with the
// start of each hidden behind the end of the one before (programmatic
// dependent launch): launch_step lets a kernel's CTAs be scheduled once every
// CTA of the kernel before has called step_next (or has ended), and step_wait
// holds them until that kernel has completed and its stores are visible.  A
// step kernel calls step_wait before it touches memory, on every path; after
// any other operation on the stream (a copy, a kernel without step_next) the
// launch is an ordinary one.
//
// step_next comes at the end of a CTA's work.  Called at its start, the next
// step's CTAs settle on whatever SMs have room while this step's still run,
// and a small grid's CTAs end up two and three to an SM: us per step, ordinary
// launches / early / late: FP64 Yee 40 x 37 x 45 12.3 / 11.5 / 7.2, pair Lame
// there 8.2 / 12.7 / 6.6, FP64 adjoint forward 30 x 28 x 33 4.1 / 2.4 / 1.8;
// large grids the same within 1 %: FP64 sweep 256^3 147 / 142 / 142, FP32 320 x
// 256 x 256 38.5 / 35.0 / 34.3, pairs 201 x 181 x 163 40.5 / 37.6 / 37.4, FP64
// Yee 128 x 120 x 113 64 / 59 / 59.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace scafes {

__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void step_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Ties an address computation to its place after step_wait: a load through
// the read-only path is otherwise free to move above it.
template <class T>
__device__ __forceinline__ void after_wait(T*& p) {
    asm volatile("" : "+l"(p));
}
template <class T>
__device__ __forceinline__ void after_wait(T* __restrict__& p) {
    asm volatile("" : "+l"(p));
}
__device__ __forceinline__ void after_wait(long long& o) { asm volatile("" : "+l"(o)); }

template <class... P, class... A>
cudaError_t launch_step(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace scafes

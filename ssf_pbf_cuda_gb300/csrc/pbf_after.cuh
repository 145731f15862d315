// Kernels of one call launched one by one on a stream, each set up while the
// one before it still runs (programmatic dependent launch).
#pragma once
#include <cuda_runtime.h>

namespace pbf103 {

// First in every kernel launched by launch_after, before any access to memory:
// waits until the launch before it is complete (its writes are visible from
// here on, and so, in turn, are those of the launches before that).  The
// kernel may be running while the launch before still writes, so what launches
// of the same call write is read by plain loads, __ldca or __ldcg: __ldg and const
// __restrict__ say that nobody writes the data while the kernel runs, and such
// a load may be moved above the wait.  (The caller's own input may be read so:
// the call's first launch starts when it is complete.)
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Lets the launch after this one be set up once every block of this one has
// come here (otherwise once every block is done); its blocks wait in
// after_previous themselves.  After after_previous, but for a call's first
// kernel, which is launched as usual.  Not for grids of several waves: the
// waiting blocks take their places (a frame of 32,768 particles at 1600 x 900
// 81 us without it in the blurs and normals, 91 with, 94 by plain launches; at
// 1280 x 720 63, 70 and 79).
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches fn, whose first act is after_previous().  The next launch that is
// not a launch_after waits for all of them, as any launch does.
template <class... K, class... A>
void launch_after(void (*fn)(K...), dim3 blocks, dim3 threads, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = threads;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, fn, static_cast<K>(args)...);  // (errors: the caller's cudaGetLastError)
}

}  // namespace pbf103

// Launches that follow one another on a stream without the gap between them.
//
// A solve's step is a chain of eight or nine kernels of a few microseconds
// each, and two to three microseconds lie between two of them.
// launch_chained lets a kernel's CTAs be scheduled while the kernel before it
// on the stream still runs (programmatic stream serialisation); the kernel
// starts with chain_enter(), which lets its own successor be scheduled and
// then waits until everything before it has ended and is visible.  A kernel
// without a wait must not be launched this way; one with it can be launched
// in any way.  A kernel whose CTAs stay for many tiles releases its successor
// at its last tile: the successor's waiting CTAs hold slots that a second
// stream's kernels could use (500 particles with quadrupoles: 948 us released
// at entry, 937 unchained, and 906 against 925 unchained with the late
// release).  GMRES of 500 particles, one column: 2.64 ms unchained, 2.27 now;
// an operator on 8000 particles and three columns 276 and 265 us; a spectrum
// of a 4000-particle layer 16.3 and 15.2 ms.  (Only grids below eight CTAs
// per SM chained: that operator 316 us against 301 with all of them.)
#pragma once

#include "mpm_common.cuh"

#include <utility>

namespace mpm {

__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
    chain_release();
    chain_wait();
}

template <typename... E, typename... A>
inline void launch_chained(void (*kern)(E...), dim3 grid, dim3 block, size_t shm, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = shm;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    MPM_CUDA(cudaLaunchKernelEx(&c, kern, std::forward<A>(args)...));
    note_launch();
}

}  // namespace mpm

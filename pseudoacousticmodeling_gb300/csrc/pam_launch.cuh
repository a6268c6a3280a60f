// Launches that overlap the end of the kernel before them.
//
// The time loops are chains of short kernels (3 to 160 us), each reading what
// the one before wrote.  A plain launch starts its first block when the last
// block of the kernel before has drained and its writes are flushed; a launch
// by launch_chained() has its blocks placed while that kernel's last blocks
// still run, and they wait on the device (wait_chained()) before they touch
// memory.  Measured (GB300): 2 to 4 us a kernel in a stream (acoustic migration, 8
// shots of 601 x 2101: 114.7 -> 101.8 ms; one shot of 900 x 2100: 13.3 -> 8.7 us
// a step), 0.3 to 0.6 us in a graph (8.8 -> 8.3 us a step).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace pam {

// First statement of every kernel that launch_chained() launches, in every
// thread: blocks until the kernel before in the stream has completed and its
// writes are visible (at once after a plain launch), then lets the next kernel
// of the chain be placed.  A kernel completes only when its own wait is over, so
// the third kernel of a chain is behind the first as well.
__device__ __forceinline__ void wait_chained() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// chain false: a plain launch (into a capture of the caller's, whose graph
// then has plain edges only).
template <class... P, class... A>
inline void launch_chained(bool chain, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &attr;
    c.numAttrs = chain ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, P(std::forward<A>(args))...);   // errors: cudaGetLastError of the caller
}

}  // namespace pam

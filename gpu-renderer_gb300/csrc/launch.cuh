// Launches that overlap their start with the end of the kernel before them in the
// stream (programmatic dependent launch): the blocks are set up while that kernel's
// last blocks run, and wait in wait_for_previous() until it has finished and its
// writes are visible. Every kernel launched so calls it before it touches global
// memory, on every path, so the chain of kernels keeps the stream's order.
//
// Such a grid exists while the kernel before it still writes, so what that kernel
// writes is not read-only for the grid's lifetime, as __ldg and const __restrict__
// parameters promise, and __restrict__ tells the compiler that the wait does not touch
// the memory: such loads and stores may be moved above the wait. So these kernels take
// plain pointers, which the wait orders. Data written before the kernel before may be
// read either way: that kernel has waited for its writer before it lets this one
// start. The first kernel of a chain follows whatever the caller launched, so it reads
// the caller's data through plain pointers too.
//
// It pays where kernels take microseconds and the 1-2 us between two of them count:
// LBVH of 100,003 triangles 86.3 -> 79.7 us, of 3,001 with a trace of 2,048 rays
// 108 -> 98 us, a 160 x 120 x 1 spp preview 431 -> 421 us. Where a kernel's last blocks
// run long, the next one's blocks only take their room on the SMs early: 1 M
// triangles 836 -> 838 us, Cornell box 256 x 256 x 16 spp 1,101 -> 1,111 us, glossy
// 54.1 -> 54.3 ms. So callers ask for it by size (`overlap`). The line for builds,
// 2^18 triangles: with and without 131,072 77 / 86 us, 230,000 102 / 108, 262,144
// 108 / 111, 400,000 117 / 117, 1 M 183 / 178.
#pragma once

#include <cuda_runtime.h>

namespace gr {

template <class... P, class... A>
cudaError_t launch_after(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// Waits for the kernel before this one; then lets the kernel after it be set up as
// soon as every block of this one has come here.
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace gr

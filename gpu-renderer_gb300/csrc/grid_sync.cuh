// Bounded device-side waits shared by the builders (lbvh.cu, bvh8.cu).
#pragma once

#include "gr_internal.h"

namespace gr {

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier of a cooperative launch (every block resident): block
// arrivals are counted on `ctr`, and the k-th barrier of the launch waits for
// (k + 1) * gridDim.x arrivals, at most `limit` polls (then ERR_TIMEOUT, and false
// to every thread of the block: what the other blocks should have written may be
// missing).
// The block barrier before the release puts every thread's writes ahead of the
// arrival; the block barrier after the acquire puts the other blocks' writes
// ahead of every thread's later reads (which go to L2: __ldcg).
__device__ __forceinline__ bool grid_barrier(uint32_t* ctr, uint32_t target, uint32_t* err,
                                             uint32_t limit = kSpinLimit) {
    __syncthreads();
    int gave_up = 0;
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        uint32_t spins = 0;
        while (ld_acquire(ctr) < target) {
            if (++spins > limit) {
                atomicOr(err, ERR_TIMEOUT);
                gave_up = 1;
                break;
            }
        }
    }
    return !__syncthreads_or(gave_up);
}

// The same for a launch that may be a single block, which has nobody to wait for
// (a barrier on its own counter took it 2 us).
__device__ __forceinline__ bool grid_sync(uint32_t* ctr, uint32_t target, uint32_t* err) {
    if (gridDim.x != 1) return grid_barrier(ctr, target, err);
    __syncthreads();
    return true;
}

}  // namespace gr

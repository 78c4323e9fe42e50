// The tile queue of the two-band propagate kernels (TileQueue).
#pragma once

#include "sbe_dev.h"

namespace sbe {

// The CTA's next item, or -1 (see TileQueue).  The propagate kernels have an
// instance with the queue (QU) and one without: the loop around the tile costs
// registers (14 % of a small length-gauge solve, which needs no queue).
__device__ __forceinline__ int next_item(const TileQueue &q)
{
    __shared__ int item;
    __syncthreads();   // the item before is finished with shared memory
    if (threadIdx.x == 0) {
        item = atomicAdd(q.ctr, 1);
        if (item >= q.nitems && atomicAdd(q.ctr + 1, 1) == (int)gridDim.x - 1) {
            q.ctr[1] = 0;   // every CTA has taken its last item
            __threadfence();
            q.ctr[0] = 0;
        }
    }
    __syncthreads();
    return item < q.nitems ? item : -1;
}
// Wait until the tile's state at step s0 is in memory, for `polls` reads at most (some
// 20 s); false: gave up, and every other wait of the engine's launches gives up with it
constexpr int QUEUE_POLLS = 1 << 25;
__device__ __forceinline__ bool tile_ready(const TileQueue &q, const int *prog, int s0, bool first, int polls = QUEUE_POLLS)
{
    __shared__ int ok;
    if (first) return true;
    if (threadIdx.x == 0) {
        int v = 0, n = 0;
        do {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(prog) : "memory");
        } while (v < s0 && ++n < polls && *(volatile int *)q.err == 0);
        if (v < s0) *q.err = 1;
        ok = v >= s0;
    }
    __syncthreads();
    return ok;
}
__device__ __forceinline__ void tile_done(const TileQueue &q, int *prog, int s1)
{
    __syncthreads();   // the CTA's state stores
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(prog), "r"(s1) : "memory");
    }
}

}  // namespace sbe

// gx_gridsync.cuh -- the grid barrier and the cell scan of the cooperative
// kernels that run many ticks in one launch (gx_nltick.cu, gx_adjoint.cu).
#pragma once

#include "gx_internal.cuh"

namespace gx {

constexpr uint32_t kScanTileCells = 1024;  // cell counters per scan tile
constexpr uint32_t kScanMaxTiles = 64;     // of at most 65,536 counters

// Device words of one cooperative launch, zero between launches.
struct GridSync {
    uint32_t arrived, left;          // barrier arrivals, blocks that left
    uint32_t request[3];             // rebuild requested, by turn
    uint32_t tile[kScanMaxTiles];    // scan tile totals of a rebuild
};

__device__ __forceinline__ uint32_t load_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier: arrivals only grow during a launch, and `target` (thread 0's)
// is the count at which every block has arrived.  The wait is bounded by
// `limit` polls: a block that gives up sets kErrBarrier and leaves (false),
// and the others follow as they see that word or their waits end.  The words
// are no longer zero then, so a launch that finds kErrBarrier set when it
// starts (one queued behind, before the host has read the error) does nothing.
__device__ __forceinline__ bool grid_barrier(GridSync* s, uint32_t* err, uint32_t limit, uint32_t& target, int* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        atomicAdd(&s->arrived, 1u);
        int ok = 1;
        for (uint32_t polls = 0; ok; ++polls) {
            if (polls >= limit) {
                atomicOr(err, kErrTimeout | kErrBarrier);
                ok = 0;
            } else if ((int32_t)(load_acquire(&s->arrived) - target) >= 0) {
                break;
            } else if ((polls & 1023u) == 1023u && (load_acquire(err) & kErrBarrier)) {
                ok = 0;
            }
        }
        __threadfence();
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// The end of a launch: the last block to leave clears the words.
__device__ __forceinline__ void grid_leave(GridSync* s) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&s->left, 1u) == gridDim.x - 1) {
        s->arrived = s->left = 0u;
        s->request[0] = s->request[1] = s->request[2] = 0u;
    }
}

// Exclusive scan of tile t of the m cell counts in place, from `carry` on;
// returns what the next tile would carry.  BS threads; s_warp holds BS / 32
// words.
template <int BS>
__device__ __forceinline__ uint32_t scan_tile(uint32_t* count, uint32_t t, uint32_t m, uint32_t carry, uint32_t* s_warp) {
    constexpr int kItems = kScanTileCells / BS;
    const uint32_t base = t * kScanTileCells + threadIdx.x * kItems;
    uint32_t v[kItems], local = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        v[k] = base + k < m ? count[base + k] : 0u;
        local += v[k];
    }
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t inc = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += u;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    uint32_t run = carry + inc - local, total = carry;
    for (uint32_t k = 0; k < BS / 32; ++k) {
        if (k < w) run += s_warp[k];
        total += s_warp[k];
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if (base + k < m) count[base + k] = run;
        run += v[k];
    }
    __syncthreads();  // s_warp is reused by the next tile
    return total;
}

}  // namespace gx

// A pass's counters. Every thread of a pass has its own counts; added to the
// pass's Counters one by one they queued up at a handful of addresses in L2, about
// one a cycle: 100 us of the 112 us of a 374x192 Julia frame, and half a
// millisecond of each lane pass (116,000 threads, 11 counters). They are summed
// over the warp by shuffles and over the block in shared memory first.
#pragma once
#include <cuda_runtime.h>

namespace mbx {

constexpr int kBlockCounts = 12;
struct BlockCounts {
    unsigned long long v[kBlockCounts];
};

// all threads of the block
__device__ __forceinline__ void block_counts_init(BlockCounts& s) {
    if (threadIdx.x < kBlockCounts) s.v[threadIdx.x] = 0;
    __syncthreads();
}
// the low `lanes` lanes of each warp together
__device__ __forceinline__ void block_count(BlockCounts& s, int k, unsigned long long v, int lanes = 32) {
    const unsigned mask = lanes >= 32 ? 0xffffffffu : (1u << lanes) - 1u;
    const int lane = (int)(threadIdx.x & 31u);
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_down_sync(mask, v, o);
        if (lane + o < lanes) v += u;
    }
    if (lane == 0 && v) atomicAdd(&s.v[k], v);
}
// one thread, after a __syncthreads
__device__ __forceinline__ void counts_flush(unsigned long long* to, unsigned long long v) {
    if (v) atomicAdd(to, v);
}
__device__ __forceinline__ void counts_flush(unsigned int* to, unsigned long long v) {
    if (v) atomicAdd(to, (unsigned int)v);
}

} // namespace mbx

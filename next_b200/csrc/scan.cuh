// Device-wide exclusive prefix sums inside the kernel that makes the values:
// block scans chained by a decoupled look-back.  Tiles are numbered in the
// order blocks take tickets, so every tile a block waits on is already
// running; each wait is bounded and raises kErrSort instead of hanging.
#pragma once

#include "common.cuh"

namespace nb {

constexpr unsigned long long kScanAgg = 1ull << 62;       // status word: the tile's own sum
constexpr unsigned long long kScanInc = 2ull << 62;       // ... the sum up to and including the tile
constexpr unsigned long long kScanValue = kScanAgg - 1;
constexpr int kScanSpins = 1 << 20;

// Exclusive prefix of v over the THREADS threads of the block, and the block's sum.
template <int THREADS>
__device__ __forceinline__ unsigned long long block_exclusive(unsigned long long v, unsigned long long* total) {
    __shared__ unsigned long long sums[THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) sums[w] = inc;
    __syncthreads();
    unsigned long long before = 0, all = 0;
#pragma unroll
    for (int k = 0; k < THREADS / 32; ++k) {
        if (k < w) before += sums[k];
        all += sums[k];
    }
    __syncthreads();
    *total = all;
    return before + inc - v;
}

// Sum of the tiles before `tile`, whose own sum is `sum`; called by one whole
// warp, which reads 32 earlier tiles' statuses at a time.
__device__ __forceinline__ unsigned long long look_back(unsigned long long* status, int tile, unsigned long long sum,
                                                        int* err) {
    volatile unsigned long long* vs = status;
    const int lane = threadIdx.x & 31;
    if (lane == 0) vs[tile] = (tile == 0 ? kScanInc : kScanAgg) | sum;
    unsigned long long before = 0;
    for (int top = tile - 1; top >= 0; top -= 32) {
        const int k = top - lane;
        unsigned long long v = kScanInc;
        if (k >= 0) {
            v = vs[k];
            for (int spins = 0; (v & (kScanAgg | kScanInc)) == 0; ++spins) {
                if (spins > kScanSpins) { raise_error(err, kErrSort); v = kScanInc; break; }
                v = vs[k];
            }
        }
        const unsigned inclusive = __ballot_sync(0xffffffffu, (v & kScanInc) != 0);
        unsigned long long part = inclusive && lane > __ffs(inclusive) - 1 ? 0 : v & kScanValue;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        before += part;
        if (inclusive) break;
    }
    if (lane == 0 && tile > 0) vs[tile] = kScanInc | (before + sum);
    return before;
}

}  // namespace nb

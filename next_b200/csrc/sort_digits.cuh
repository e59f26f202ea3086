// Digits of the radix sort's passes and the counting of them, shared by the
// sort and by the kernel that makes the tree's keys.
#pragma once

#include <stdint.h>

namespace nb {

constexpr int kSortRadix = 256;

// Digit mask of pass p for keys of key_bits significant bits: bits at and
// above key_bits take no part in the ordering.
__host__ __device__ __forceinline__ uint32_t pass_mask(int key_bits, int p) {
    const int left = key_bits - 8 * p;
    return left >= 8 ? 0xffu : (1u << left) - 1u;
}

// One key's digit of every pass, counted in a block's shared counts (passes x 256).
__device__ __forceinline__ void count_digits(uint64_t key, int key_bits, uint32_t* local) {
    for (int p = 0; 8 * p < key_bits; ++p) atomicAdd(local + p * kSortRadix + ((key >> (8 * p)) & pass_mask(key_bits, p)), 1u);
}

// The block's counts added to the sort's.
template <int THREADS>
__device__ __forceinline__ void add_digit_counts(const uint32_t* local, int passes, uint32_t* hist) {
    for (int i = threadIdx.x; i < passes * kSortRadix; i += THREADS) {
        const uint32_t v = local[i];
        if (v) atomicAdd(hist + i, v);
    }
}

}  // namespace nb

// Layout of the FP64 twiddle tables (ModCtx::ffwd / finv).
//
// Entries keep the natural order of the integer tables except, from N = 256
// on, those of the three stages of the smallest spans, which act on groups of
// 8 consecutive elements with 1, 2 and 4 twiddles per group: the 7 twiddles
// of 32 neighbouring groups are stored slot by slot, so that lanes holding
// neighbouring groups read neighbouring entries.  That part starts at N/8 in
// the forward table (after the entries of the larger spans) and at 0 in the
// inverse one (before them).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace axhel_impl {

constexpr uint32_t kFpTailGroups = 32;
constexpr uint32_t kFpTailMinN = 8 * kFpTailGroups;

// Slot of twiddle x of a group in the stage of span 2^b, b = 2, 1, 0.
__host__ __device__ constexpr uint32_t fp_tail_slot(int b, uint32_t x) { return b == 2 ? 0u : (b == 1 ? 1u + x : 3u + x); }

// Position of a slot of group `g` of 8 elements.
__host__ __device__ inline uint32_t fp_tail_pos(uint32_t g, uint32_t slot)
{
    return (g / kFpTailGroups * 7 + slot) * kFpTailGroups + g % kFpTailGroups;
}

// Position of the entry with natural index i >= 1 (forward: 2^t + m of stage
// t; inverse: 1 + N - N/2^s + m of stage s).
__host__ __device__ inline uint32_t fp_table_pos(bool inv, uint32_t i, uint32_t n, uint32_t logn)
{
    if (n < kFpTailMinN) return i;
    int b;
    uint32_t m;
    if (inv) {
        const uint32_t r = n - (i - 1);  // N/2^s - m
        b = 0;
        while (r <= (n >> (b + 1))) ++b;
        m = (n >> b) - r;
    } else {
        uint32_t t = 0;
        while ((2u << t) <= i) ++t;
        b = (int)(logn - 1 - t);
        m = i - (1u << t);
    }
    if (b > 2) return i;
    const uint32_t pos = fp_tail_pos(m >> (2 - b), fp_tail_slot(b, m & ((1u << (2 - b)) - 1)));
    return inv ? pos : (n >> 3) + pos;
}

}  // namespace axhel_impl

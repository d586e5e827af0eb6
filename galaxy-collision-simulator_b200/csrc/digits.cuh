// digits.cuh - the radix sort's digit histograms, accumulated in shared memory
// by the kernels that see all keys before the sort (encode, and the
// allocation-free sort's counting pass).
#pragma once
#include "gcs_internal.h"

namespace gcs {

// Blocks that count digits are few and large: every block adds up to
// kKeyPasses * kRadix counts to the same global words at its end, and 1,184
// blocks of 256 threads spent more on that than on the keys (encode stage of
// 300,000 particles 19.5 us, of 1,048,576 23.6; 11.3 and 17.4 with two blocks of
// 1,024 an SM).
constexpr int kCountThreads = 1024;
inline int count_grid(int64_t n, int sms) {
    const int64_t want = (n + kCountThreads - 1) / kCountThreads, cap = (int64_t)sms * 2;
    return (int)(want < 1 ? 1 : want < cap ? want : cap);
}

// Adds the digits of the warp's keys (all lanes call; only valid ones count).
// Neighbouring keys mostly agree in their two top digits - particles arrive in
// the last step's order - and 32 adds to one shared word go one by one: when
// all lanes agree in both, one lane adds for all.  (Testing the digits below
// as well costs more than it saves: 46 against 40 us at 4,194,304.)
__device__ __forceinline__ void count_digits(uint32_t (*hist)[kRadix], uint64_t k, bool valid) {
    constexpr int kTop = kKeyPasses - 2;
    const uint32_t live = __ballot_sync(0xFFFFFFFFu, valid);
    if (live == 0u) return;
    const int leader = __ffs(live) - 1;
    const uint32_t top = (uint32_t)(k >> (kRadixBits * kTop));
    const uint32_t first = __shfl_sync(0xFFFFFFFFu, top, leader);
    const bool same = __all_sync(0xFFFFFFFFu, !valid || top == first);
    if (same ? (threadIdx.x & 31) == leader : valid) {
        const uint32_t add = same ? (uint32_t)__popc(live) : 1u;
#pragma unroll
        for (int d = kTop; d < kKeyPasses; ++d)
            atomicAdd(&hist[d][(uint32_t)(k >> (kRadixBits * d)) & (kRadix - 1)], add);
    }
    if (valid) {
#pragma unroll
        for (int d = 0; d < kTop; ++d)
            atomicAdd(&hist[d][(uint32_t)(k >> (kRadixBits * d)) & (kRadix - 1)], 1u);
    }
}

}  // namespace gcs

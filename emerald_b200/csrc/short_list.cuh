// Ordering of the neighbour searches' short lists.
#pragma once

#include <cstdint>

namespace emerald {

// The fast path of a search: a particle with at most this many accepted
// candidates.
constexpr int kShortList = 16;

// A place without a candidate: no distance has these bits, and no two of them
// the same upper ones.
__device__ __forceinline__ uint32_t unused_key(int q) { return 0xffffff00u + 17u * q; }

struct ShortKey {
    uint32_t dist;  // bits of a distance (not negative)
    uint64_t index;
    __device__ __forceinline__ bool operator<(ShortKey const& o) const {
        return dist != o.dist ? dist < o.dist : index < o.index;
    }
};

// The order of cnt <= kShortList candidates by (distance, index): list position
// of the k-th in bits 4k..4k+3. d[q] holds the distance of the q-th with its
// last four bits replaced by q, or unused_key(q). Batcher's odd-even merge sort
// (K. Batcher, "Sorting networks and their applications", 1968) in registers,
// the same instructions in every lane whatever the counts, where an insertion
// sort costs a warp the longest of its lanes' moves at every candidate. Where
// two keys differ in nothing but the position, the exact keys decide
// afterwards.
template <class Key>
__device__ __forceinline__ uint64_t order_short_list(uint32_t (&d)[kShortList], int cnt,
                                                     Key exact) {
    constexpr int kSpan[10] = {1, 2, 2, 4, 4, 4, 8, 8, 8, 8};
    constexpr int kStep[10] = {1, 2, 1, 4, 2, 1, 8, 4, 2, 1};
#pragma unroll
    for (int t = 0; t < 10; ++t) {
        int const span = kSpan[t], k = kStep[t];
#pragma unroll
        for (int lo = 0; lo < kShortList; ++lo) {
            int const hi = lo + k;
            bool const pair = hi < kShortList && lo >= k % span &&
                              (lo - k % span) % (2 * k) < k && lo / (2 * span) == hi / (2 * span);
            if (pair) {
                uint32_t const dl = min(d[lo], d[hi]);
                d[hi] = max(d[lo], d[hi]);
                d[lo] = dl;
            }
        }
    }
    bool tie = false;
#pragma unroll
    for (int q = 1; q < kShortList; ++q) tie = tie || (d[q] ^ d[q - 1]) < 16u;
    uint32_t half[2] = {0u, 0u};
#pragma unroll
    for (int q = 0; q < kShortList; ++q) half[q / 8] |= (d[q] & 15u) << (4 * (q % 8));
    uint64_t order = (static_cast<uint64_t>(half[1]) << 32) | half[0];
    if (tie) {
        auto key = [&](int k) { return exact(static_cast<int>(order >> (4 * k)) & 15); };
#pragma unroll 1
        for (int k = 1; k < cnt; ++k) {
#pragma unroll 1
            for (int q = k; q > 0 && key(q) < key(q - 1); --q) {
                uint64_t const diff = ((order >> (4 * q)) ^ (order >> (4 * q - 4))) & 15u;
                order ^= (diff << (4 * q)) | (diff << (4 * q - 4));
            }
        }
    }
    return order;
}

}  // namespace emerald

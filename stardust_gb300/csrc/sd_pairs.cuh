// sd_pairs.cuh -- from pairs found in any order to the ascending list of
// unique pairs, shared by the tree and the sweep.
//
// A pair goes to the box of lower id: it takes that box's next place, and its
// first kPairKeep partners are kept.  The counts scanned give every box the
// place of its pairs in the list; the kept partners are sorted in registers
// and written.  Boxes with more partners are filled by a second search of
// their finder (which returns at once when there are none) straight into the
// list, and sorted there.  A list that does not fit is not written.
//
// 16 kept: 2,000,000 boxes of two pairs each never search twice, and the write
// (16 words read, the sort in registers) takes 31 us.  Lists both ways from a
// counting and a writing search, then the upper halves counted, scanned and
// copied, took 2.6 searches' time there.
#pragma once

#include "sd_common.cuh"

namespace sd {

constexpr uint32_t kPairKeep = 16;

struct PairSink {
    uint32_t* count;   // per box: pairs of which it has the lower id (zero before)
    uint32_t* keep;    // per box: the first kPairKeep partners
    uint32_t* over;    // [0] set when a box has more (zero before)
    // the second search
    const uint32_t* off;      // per box: place of its first pair; off[n] = pairs
    uint32_t* cursor;         // per box (zero before)
    unsigned long long* out;
    uint32_t n;
    uint64_t cap;
};

__device__ __forceinline__ void sink_pair(const PairSink& s, uint32_t a, uint32_t b) {
    const uint32_t i = min(a, b), j = max(a, b);
    const uint32_t at = atomicAdd(s.count + i, 1u);
    if (at < kPairKeep) s.keep[(size_t)i * kPairKeep + at] = j;
    else if (at == kPairKeep) *s.over = 1u;
}

// Pairs found on the way, set aside in shared memory: handed over one by one,
// each would hold its whole warp up for an atomic's way to L2 and back (a
// place in the box's list), some ten times a warp; set aside they are handed
// over side by side (the sweep of 2,000,000 boxes 192 -> 166 us).  Up to CAP;
// further ones go straight to the sink.
template <int CAP>
struct PairBuffer {
    uint2 pair[CAP];
    uint32_t n;  // (zero before)
};
__device__ __forceinline__ void hand_over(const PairSink& s, uint32_t i, uint32_t j) { sink_pair(s, i, j); }

template <int CAP, class SINK>
__device__ __forceinline__ void buffer_pair(PairBuffer<CAP>& b, const SINK& s, uint32_t i, uint32_t j) {
    const uint32_t at = atomicAdd(&b.n, 1u);
    if (at < (uint32_t)CAP) b.pair[at] = make_uint2(i, j);
    else hand_over(s, i, j);
}
// By `threads` threads that have met since the last buffer_pair(), this one the
// t-th.
template <int CAP, class SINK>
__device__ __forceinline__ void flush_pairs(const PairBuffer<CAP>& b, const SINK& s, uint32_t t, uint32_t threads) {
    const uint32_t n = min(b.n, (uint32_t)CAP);
    for (uint32_t k = t; k < n; k += threads) hand_over(s, b.pair[k].x, b.pair[k].y);
}

// Whether the second search has anything to do.
__device__ __forceinline__ bool sink_refill(const PairSink& s) { return *s.over != 0u && s.off[s.n] <= s.cap; }

__device__ __forceinline__ void sink_pair_again(const PairSink& s, uint32_t a, uint32_t b) {
    const uint32_t i = min(a, b), j = max(a, b);
    if (s.count[i] <= kPairKeep) return;
    const uint32_t at = s.off[i] + atomicAdd(s.cursor + i, 1u);
    if (at < s.off[i + 1] && at < s.cap) s.out[at] = ((unsigned long long)i << 32) | j;
}

// d_count: the pairs (0 when they do not fit) and the error bits, status's among
// them; both zero before.
static __global__ void pairs_write_kernel(PairSink s, uint32_t* __restrict__ d_count,
                                          const uint32_t* __restrict__ status) {
    stream_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t total = s.off[s.n];
    const bool fits = total <= s.cap;
    if (i == 0) {
        *d_count = fits ? total : 0u;
        atomicOr(d_count + 1, *status | (fits ? 0u : kErrPairOverflow));
    }
    if (i >= s.n || !fits) return;
    const uint32_t base = s.off[i], c = s.off[i + 1] - base;
    if (c == 0) return;
    if ((uint64_t)base + c > s.cap) {  // (only where 2^32 pairs or more wrapped the total)
        atomicOr(d_count + 1, kErrPairOverflow);
        return;
    }
    if (c <= kPairKeep) {
        uint32_t v[kPairKeep];
#pragma unroll
        for (uint32_t q = 0; q < kPairKeep; ++q) v[q] = q < c ? s.keep[(size_t)i * kPairKeep + q] : 0xffffffffu;
#pragma unroll
        for (uint32_t r = 0; r < kPairKeep; ++r) {  // c rounds of odd-even transposition sort c values
            if (r >= c) break;
#pragma unroll
            for (uint32_t q = r & 1u; q + 1 < kPairKeep; q += 2)
                if (v[q] > v[q + 1]) {
                    const uint32_t t = v[q];
                    v[q] = v[q + 1];
                    v[q + 1] = t;
                }
        }
#pragma unroll
        for (uint32_t q = 0; q < kPairKeep; ++q)
            if (q < c) s.out[base + q] = ((unsigned long long)i << 32) | v[q];
        return;
    }
    for (uint32_t e = base + 1; e < base + c; ++e) {
        const unsigned long long x = s.out[e];
        uint32_t m = e;
        while (m > base && s.out[m - 1] > x) {
            s.out[m] = s.out[m - 1];
            --m;
        }
        s.out[m] = x;
    }
}

}  // namespace sd

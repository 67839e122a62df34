// sd_sort.cu -- stable onesweep LSD radix sort of (u32 key, u32 value) pairs.
//
// Replaces the reference's three-kernel, 16-CTA radix sort
// (RadixTabulateCUDA / RadixSumCUDA / RadixReorderCUDA,
// src/engine/cuda/sh_collision_detection.cu:129-283, driven by
// sortCollisionList :310-360).  Its intended semantics -- a stable LSD sort
// of 32-bit cell words carrying 32-bit sphere words -- are kept; the
// algorithm is the single-pass-per-digit "onesweep" scheme:
//
//   1. one histogram kernel reads every key once and builds the digit
//      histograms of all passes (shared atomics);
//   2. per digit pass, one kernel: each CTA takes the next tile index from an
//      atomic counter, ranks its keys per digit (stable within the warp,
//      warp-ordered across the tile), publishes its per-digit tile count,
//      stages the tile in shared memory in digit order, resolves its global
//      digit offset by decoupled look-back over the predecessors' published
//      counts and writes the tile out in coalesced runs.
//
// Ranks: the lanes of equal digit find each other in a shared word per digit
// (atomicOr of the lane's bit).  __match_any_sync, whose time grows with the
// number of distinct digits, bound both kernels (4,000,037 random 30-bit keys:
// 111 us the histograms, 56 us a pass); one ballot per digit bit was bound by
// the ballots' latency (2.9 us of a tile's 6 with one CTA per SM).
//
// The look-back has two levels.  All tiles that fit the chip start at once,
// so with one chain of tiles the last of them walks hundreds of counts, a few
// per round trip (4M keys: 608 resident tiles, 8 counts per trip of ~0.5 us:
// two thirds of the pass).  Here a tile adds its counts to its group's (32
// tiles), reads the counts of the tiles before it in the group, and then the
// groups' sums back to the nearest group whose prefix is published.
// Measured (GB300), 4,000,037 keys of 30 bits: histograms 11 us (was 111), a
// pass 28 us = 2.3 TB/s (was 56), the sort 134 us (was 345); 9,437,184 words
// of 32 bits: 278 us.  A pass is bound by the latency of a tile's phases
// (ranks 4 us, look-back 3, staging and writing 3) at 24 warps per SM.
//
// Digits are up to 9 bits wide -- a key range of `key_bits` bits takes
// ceil(key_bits / 9) passes (18-bit cell keys: 2 passes; 32-bit: 4 of 8) --
// except 19- and 20-bit keys, which take 2 passes of 10-bit digits (1024
// bins) rather than 3.
// Look-back waits are bounded (kSpinLimit) and report through the status
// word instead of hanging.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sd_common.cuh"
#include "sd_internal.h"
#include "sd_sort_device.cuh"

namespace sd {

SortPlan sort_plan(int key_bits) {
    SortPlan p{};
    if (key_bits < 1) key_bits = 1;
    if (key_bits > 32) key_bits = 32;
    p.passes = (key_bits == 19 || key_bits == 20) ? 2 : (key_bits + 8) / 9;
    int base = key_bits / p.passes, extra = key_bits % p.passes, sh = 0;
    for (int i = 0; i < p.passes; ++i) {
        p.bits[i] = base + (i < extra ? 1 : 0);
        p.shift[i] = sh;
        sh += p.bits[i];
    }
    p.stride = p.bits[0] > 9 ? 1024 : 512;
    return p;
}

template <int ITEMS>
constexpr uint32_t tile_keys() { return kSortThreads * ITEMS; }

__global__ void __launch_bounds__(kHistThreads)
sort_histogram_kernel(const uint32_t* __restrict__ keys, uint32_t n, SortPlan plan, uint32_t* __restrict__ scratch,
                      bool vec, const uint32_t* __restrict__ d_n) {
    stream_wait();
    if (d_n) n = min(n, *d_n);
    __shared__ uint32_t hist[2048];  // pass p at p * plan.stride
    block_histograms<false>(keys, nullptr, n, plan, scratch, hist, vec);
}

// The radix fallback of the incremental re-sort.  When more keys changed
// than the re-sort takes (skip[1] > skip_max) it clears the passes' tile
// status, writes the slot identity into vals and builds the digit
// histograms -- the re-sort's plan kernel has cleared the tile counters and
// histograms -- else it returns at once, so that a step whose moves the
// re-sort placed pays for neither.
__global__ void __launch_bounds__(kHistThreads)
sort_hist_fallback_kernel(const uint32_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t n,
                          SortPlan plan, uint32_t* __restrict__ scratch, const uint32_t* __restrict__ skip,
                          uint32_t skip_max, uint64_t words, bool vec) {
    stream_wait();
    if (skip[1] <= skip_max) return;
    const uint64_t gstride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gstride)
        scratch[kStatusOff + w] = 0u;
    __shared__ uint32_t hist[2048];  // pass p at p * plan.stride
    block_histograms<true>(keys, vals, n, plan, scratch, hist, vec);
}

// ------------------------------------------------------------ onesweep pass
// Three CTAs per SM: with four (64 registers) the match loop spills
// (4,000,037 keys of 30 bits: 158 us the sort against 134; five: 206).
template <int BINS, int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 3)
sort_pass_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                 uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
                 int shift, int bits, int pass, uint32_t num_tiles, uint32_t hstride, uint32_t bins,
                 uint32_t* __restrict__ scratch, const uint32_t* __restrict__ skip, uint32_t skip_max,
                 const uint32_t* __restrict__ d_n) {
    stream_wait();
    if (skip && skip[1] <= skip_max) return;  // the incremental re-sort wrote the result
    if (d_n) n = min(n, *d_n);
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ uint32_t s_tile;
    if (threadIdx.x == 0) s_tile = atomicAdd(&scratch[4 + pass], 1u);
    __syncthreads();
    constexpr uint32_t kTile = kSortThreads * ITEMS;
    const uint32_t tile = s_tile;
    if (tile < n / kTile)
        sort_tile<BINS, ITEMS, true>(smem, tile, keys_in, vals_in, keys_out, vals_out, n, shift, bits, pass, num_tiles,
                                     hstride, bins, scratch);
    else if (tile < (n + kTile - 1) / kTile)  // (d_n: fewer keys than the grid's)
        sort_tile<BINS, ITEMS>(smem, tile, keys_in, vals_in, keys_out, vals_out, n, shift, bits, pass, num_tiles, hstride,
                               bins, scratch);
}

// Smallest tile the pass kernel is instantiated with; sizes the status area.
constexpr int kSortItemsMin = 8;
static int g_sort_items = 16;  // keys per thread of the pass kernel (8 or 16)

void sort_set_items(int items) { g_sort_items = items >= 16 ? 16 : 8; }
int sort_items() { return g_sort_items; }

uint64_t sort_scratch_words(uint64_t n, int key_bits) {
    SortPlan p = sort_plan(key_bits);
    uint64_t tiles = (n + tile_keys<kSortItemsMin>() - 1) / tile_keys<kSortItemsMin>();
    if (tiles == 0) tiles = 1;
    return kStatusOff + (uint64_t)p.passes * tiles * (uint64_t)p.stride;
}

uint32_t* sort_hist_ptr(uint32_t* scratch) { return scratch + kHistOff; }

static uint32_t num_tiles(uint32_t n) {
    uint32_t t = kSortThreads * (uint32_t)g_sort_items;
    return (n + t - 1) / t;
}

cudaError_t sort_clear_async(uint32_t n, const SortPlan& plan, uint32_t* scratch, cudaStream_t st, bool checked) {
    // counters, histograms and this sort's tile status; not the status word
    size_t clear_words = kStatusOff - 4 + (size_t)plan.passes * (size_t)status_words(num_tiles(n), status_bins(plan));
    return checked ? zero_async(st, {scratch + 4, clear_words})
                   : cudaMemsetAsync(scratch + 4, 0, clear_words * sizeof(uint32_t), st);
}

// Blocks of the histogram kernels: 8 keys per thread and loop trip at small
// n, and two blocks per SM at most, since every block adds each of its bins to
// the global histograms (977 blocks of 256 threads at 4M keys: 1M atomics on
// 1,024 words).
static int hist_blocks(uint32_t n) {
    const uint32_t b = (n + kHistThreads * 8 - 1) / (kHistThreads * 8);
    return b < 1u ? 1 : (b > 152u * 2u ? 152 * 2 : (int)b);
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

static cudaError_t sort_histogram_async(const uint32_t* keys, uint32_t n, const SortPlan& plan, uint32_t* scratch,
                                        cudaStream_t st, const uint32_t* d_n) {
    launch_after(st, hist_blocks(n), kHistThreads, 0, sort_histogram_kernel, keys, n, plan, scratch,
                 aligned16(keys), d_n);
    return cudaGetLastError();
}

template <int BINS, int ITEMS>
static cudaError_t launch_pass(const uint32_t* ki, const uint32_t* vi, uint32_t* ko, uint32_t* vo,
                               uint32_t n, int shift, int bits, int pass, uint32_t tiles, uint32_t stride,
                               uint32_t bins, uint32_t* scratch, cudaStream_t st, const uint32_t* skip,
                               uint32_t skip_max, const uint32_t* d_n) {
    size_t sm = sort_tile_smem<BINS, ITEMS>();
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(sort_pass_kernel<BINS, ITEMS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    launch_after(st, tiles, kSortThreads, sm, sort_pass_kernel<BINS, ITEMS>, ki, vi, ko, vo, n, shift, bits, pass,
                 tiles, stride, bins, scratch, skip, skip_max, d_n);
    return cudaGetLastError();
}

// The digit passes alone: the histograms in scratch must be complete and the
// tile status cleared (sort_clear_async + a histogram producer).
cudaError_t sort_passes_async(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp,
                              uint32_t n, const SortPlan& plan, uint32_t* scratch, cudaStream_t st,
                              bool* in_tmp, const uint32_t* skip, uint32_t skip_max, const uint32_t* d_n) {
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    const uint32_t tiles = num_tiles(n);
    uint32_t *ki = keys, *vi = vals, *ko = keys_tmp, *vo = vals_tmp;
    for (int p = 0; p < plan.passes; ++p) {
        cudaError_t e;
        const int b = plan.bits[p], sh = plan.shift[p];
        const uint32_t sd = (uint32_t)plan.stride, ss = status_bins(plan);
        if (g_sort_items >= 16)
            e = b > 9   ? launch_pass<1024, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n)
                : b > 8 ? launch_pass<512, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n)
                        : launch_pass<256, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n);
        else
            e = b > 9   ? launch_pass<1024, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n)
                : b > 8 ? launch_pass<512, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n)
                        : launch_pass<256, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max, d_n);
        if (e != cudaSuccess) return e;
        uint32_t* t;
        t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    *in_tmp = (plan.passes & 1) != 0;
    return cudaSuccess;
}

uint64_t sort_fallback_clear_words() { return kStatusOff - 4; }

cudaError_t sort_fallback_async(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp, uint32_t n,
                                const SortPlan& plan, uint32_t* scratch, cudaStream_t st, bool* in_tmp,
                                const uint32_t* skip, uint32_t skip_max) {
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    const uint64_t words = (uint64_t)plan.passes * status_words(num_tiles(n), status_bins(plan));
    launch_after(st, hist_blocks(n), kHistThreads, 0, sort_hist_fallback_kernel, keys, vals, n, plan, scratch, skip,
                 skip_max, words, aligned16(keys));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return sort_passes_async(keys, vals, keys_tmp, vals_tmp, n, plan, scratch, st, in_tmp, skip, skip_max);
}

// Sorts (keys, vals) by bits [0, key_bits).  Returns via *in_tmp whether
// the result ended in the tmp buffers (odd pass count).  d_n (may be null): a
// device word, the number of keys when it is below n.
cudaError_t sort_pairs_async(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp,
                             uint32_t n, int key_bits, uint32_t* scratch, cudaStream_t st,
                             bool* in_tmp, const uint32_t* d_n, bool checked) {
    SortPlan plan = sort_plan(key_bits);
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    cudaError_t e = sort_clear_async(n, plan, scratch, st, checked);
    if (e != cudaSuccess) return e;
    if ((e = sort_histogram_async(keys, n, plan, scratch, st, d_n)) != cudaSuccess) return e;
    return sort_passes_async(keys, vals, keys_tmp, vals_tmp, n, plan, scratch, st, in_tmp, nullptr, 0, d_n);
}

int sort_num_passes(int key_bits) { return sort_plan(key_bits).passes; }

}  // namespace sd

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

namespace sd {

constexpr int kSortThreads = 256;
constexpr int kHistThreads = 512;
constexpr int kSortWarps = kSortThreads / kWarp;
constexpr uint32_t kGroup = 32;               // tiles per look-back group
constexpr uint32_t kTileDone = 1u << 15;      // tile status: published | count (<= 4096)
constexpr uint32_t kSumOne = 1u << 24;        // group sum: tiles added (kGroup of them: complete) | count
constexpr uint32_t kSumMask = kSumOne - 1u;
constexpr uint32_t kPrefixDone = 1u << 31;    // group prefix: published | keys up to and including the group
constexpr int kLookback = 16;                 // statuses read per look-back round trip
constexpr uint32_t kPollNs = 100;             // pause between two polls of a status

// Scratch layout (u32 words):
//   [0]                 status word (error bits; never cleared by the sort)
//   [4 .. 8)            per-pass tile counters
//   [16 .. 16+2048)     per-pass global digit histograms, pass q at
//                       q * stride (4 x 512, or 2 x 1024)
//   [kStatusOff ..)     per pass: tile status [tile][bins] of 16 bits, then,
//                       with more than one group of tiles, group sums and
//                       group prefixes [group][bins] (status_words)
constexpr uint64_t kHistOff = 16;
constexpr uint64_t kStatusOff = kHistOff + 4 * 512;

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

// Bins the passes' status rows hold: those of the widest digit (bits[0]).
static uint32_t status_bins(const SortPlan& p) { return p.bits[0] > 9 ? 1024u : (p.bits[0] > 8 ? 512u : 256u); }

// Words of one pass's status.  At most tiles * bins: half of that for the
// tiles, and two rows per 32 tiles for the groups of more than 32 tiles.
__host__ __device__ __forceinline__ uint64_t status_words(uint32_t tiles, uint32_t bins) {
    const uint32_t groups = (tiles + kGroup - 1) / kGroup;
    return ((uint64_t)tiles * bins) / 2 + (groups > 1 ? 2ull * groups * bins : 0ull);
}

template <int ITEMS>
constexpr uint32_t tile_keys() { return kSortThreads * ITEMS; }

// --------------------------------------------------------------- histogram
// Adds a key to the block's shared digit histograms.
__device__ __forceinline__ void hist_key(uint32_t* hist, const SortPlan& plan, uint32_t k) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        if (p >= plan.passes) break;
        atomicAdd(&hist[p * plan.stride + ((k >> plan.shift[p]) & ((1u << plan.bits[p]) - 1u))], 1u);
    }
}

// The block's part of the digit histograms of keys[0, n), added to the
// global ones.  vec: keys is 16-byte aligned (four keys per load).  With
// vals, the slot identity is written there.
template <bool IDENTITY>
__device__ __forceinline__ void block_histograms(const uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                 uint32_t n, const SortPlan& plan, uint32_t* __restrict__ scratch,
                                                 uint32_t* hist, bool vec) {
    for (int i = threadIdx.x; i < 2048; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, n4 = vec ? n / 4 : 0u;
    for (uint32_t i = first; i < n4; i += stride) {
        const uint4 k = __ldg(reinterpret_cast<const uint4*>(keys) + i);
        if (IDENTITY) {
            vals[4 * i] = 4 * i;
            vals[4 * i + 1] = 4 * i + 1;
            vals[4 * i + 2] = 4 * i + 2;
            vals[4 * i + 3] = 4 * i + 3;
        }
        hist_key(hist, plan, k.x);
        hist_key(hist, plan, k.y);
        hist_key(hist, plan, k.z);
        hist_key(hist, plan, k.w);
    }
    for (uint32_t i = 4 * n4 + first; i < n; i += stride) {
        if (IDENTITY) vals[i] = i;
        hist_key(hist, plan, keys[i]);
    }
    __syncthreads();
    for (int p = 0; p < plan.passes; ++p) {
        const uint32_t nb = 1u << plan.bits[p];
        for (uint32_t d = threadIdx.x; d < nb; d += blockDim.x)
            if (hist[p * plan.stride + d]) atomicAdd(&scratch[kHistOff + p * plan.stride + d], hist[p * plan.stride + d]);
    }
}

__global__ void __launch_bounds__(kHistThreads)
sort_histogram_kernel(const uint32_t* __restrict__ keys, uint32_t n, SortPlan plan, uint32_t* __restrict__ scratch,
                      bool vec) {
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
    if (skip[1] <= skip_max) return;
    const uint64_t gstride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gstride)
        scratch[kStatusOff + w] = 0u;
    __shared__ uint32_t hist[2048];  // pass p at p * plan.stride
    block_histograms<true>(keys, vals, n, plan, scratch, hist, vec);
}

// ------------------------------------------------------------ onesweep pass
// Exclusive scan over the block of one u64 per thread (two u32 counts that
// cannot carry into each other); ws holds kSortWarps words.
__device__ __forceinline__ unsigned long long block_exclusive_scan2(unsigned long long v, unsigned long long* ws) {
    const uint32_t w = threadIdx.x / kWarp;
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane_id() >= (uint32_t)o) inc += t;
    }
    if (lane_id() == kWarp - 1) ws[w] = inc;
    __syncthreads();
    unsigned long long base = 0;
#pragma unroll
    for (uint32_t k = 0; k < (uint32_t)kSortWarps; ++k)
        if (k < w) base += ws[k];
    return base + inc - v;
}

__device__ __forceinline__ void st_relaxed16(uint16_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u16 [%0], %1;" ::"l"(p), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint32_t ld_relaxed16(const uint16_t* p) {
    uint16_t v;
    asm volatile("ld.relaxed.gpu.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}

// The count of digit d in the tiles before `tile`, from the statuses of one
// pass: tile rows, group sums, group prefixes.  Statuses are loaded kLookback
// at a time; one that is not published yet is polled by itself, with a pause,
// so that waiting leaves the issue slots to the tiles waited for (with every
// poll reloading the whole batch, waiting took most of the issue slots and
// made itself longer).  Waits are on earlier tiles only (tiles are handed out
// in order), and bounded.
__device__ __forceinline__ uint32_t look_back(const uint16_t* __restrict__ rows, const uint32_t* __restrict__ sums,
                                              const uint32_t* __restrict__ prefixes, uint32_t bins, uint32_t tile,
                                              uint32_t d, uint32_t* __restrict__ errors) {
    const uint32_t g = tile / kGroup;
    uint32_t excl = 0, spins = 0;
    for (uint32_t t = g * kGroup; t < tile; t += kLookback) {  // the group's own tiles
        const uint16_t* row = rows + (uint64_t)t * bins + d;
        uint32_t v[kLookback];
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)kLookback; ++k)
            v[k] = t + k < tile ? ld_relaxed16(row + k * bins) : kTileDone;
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)kLookback; ++k) {
            while (!(v[k] & kTileDone)) {
                if (++spins > kSpinLimit) {
                    atomicOr(errors, kErrLookbackTimeout);
                    return excl;
                }
                __nanosleep(kPollNs);
                v[k] = ld_relaxed16(row + k * bins);
            }
            excl += v[k] & (kTileDone - 1u);
        }
    }
    for (uint32_t q = g; q > 0;) {  // the groups before it, nearest first
        uint32_t s[kLookback / 2], x[kLookback / 2];
        const uint32_t m = q < (uint32_t)kLookback / 2 ? q : (uint32_t)kLookback / 2;
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)kLookback / 2; ++k) {
            x[k] = k < m ? ld_relaxed(prefixes + (uint64_t)(q - 1 - k) * bins + d) : 0u;
            s[k] = k < m ? ld_relaxed(sums + (uint64_t)(q - 1 - k) * bins + d) : kGroup * kSumOne;
        }
#pragma unroll
        for (uint32_t k = 0; k < (uint32_t)kLookback / 2; ++k) {
            while (!(x[k] & kPrefixDone) && (s[k] & ~kSumMask) != kGroup * kSumOne) {
                if (++spins > kSpinLimit) {
                    atomicOr(errors, kErrLookbackTimeout);
                    return excl;
                }
                __nanosleep(kPollNs);
                s[k] = ld_relaxed(sums + (uint64_t)(q - 1 - k) * bins + d);
            }
            if (x[k] & kPrefixDone) return excl + (x[k] & ~kPrefixDone);
            excl += s[k] & kSumMask;
        }
        q -= m;
    }
    return excl;
}

// BINS: 256, 512 or 1024 digit bins (template so narrow passes do less
// per-digit work).  ITEMS: keys per thread (tile = 256 * ITEMS keys).
// hstride: the plan's histogram stride; bins: bins of a status row.  Thread t
// owns the digits [DPT * t, DPT * t + DPT).  Three CTAs per SM: with four (64
// registers) the match loop spills (4,000,037 keys of 30 bits: 158 us the
// sort against 134; five: 206).
template <int BINS, int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 3)
sort_pass_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                 uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n,
                 int shift, int bits, int pass, uint32_t num_tiles, uint32_t hstride, uint32_t bins,
                 uint32_t* __restrict__ scratch, const uint32_t* __restrict__ skip, uint32_t skip_max) {
    if (skip && skip[1] <= skip_max) return;  // the incremental re-sort wrote the result
    constexpr int TILE = kSortThreads * ITEMS;
    constexpr int DPT = BINS / kSortThreads;  // digits per thread (1, 2 or 4)
    constexpr int AREA = 2 * TILE > kSortWarps * BINS ? 2 * TILE : kSortWarps * BINS;  // words
    constexpr int U = AREA / (kSortWarps * BINS);  // items matched together (4, 2 or 1)
    static_assert(TILE < (int)kTileDone && TILE * kGroup < kSumOne, "counts fit their fields");
    extern __shared__ __align__(16) uint32_t smem[];
    uint2* s_pairs = reinterpret_cast<uint2*>(smem);  // TILE (key, value)
    uint32_t* s_whist = smem + AREA;           // kSortWarps * BINS
    uint32_t* s_gbase = s_whist + kSortWarps * BINS;  // BINS
    unsigned long long* s_ws = reinterpret_cast<unsigned long long*>(s_gbase + BINS);  // kSortWarps + tile id

    const uint32_t mask = (1u << bits) - 1u;
    const uint32_t w = threadIdx.x / kWarp;
    const uint32_t lane = lane_id();

    if (threadIdx.x == 0) reinterpret_cast<uint32_t*>(s_ws + kSortWarps)[0] = atomicAdd(&scratch[4 + pass], 1u);
    __syncthreads();
    const uint32_t tile = reinterpret_cast<uint32_t*>(s_ws + kSortWarps)[0];
    const uint32_t tile_base = tile * TILE;
    const uint32_t in_tile = n - tile_base < (uint32_t)TILE ? n - tile_base : (uint32_t)TILE;

    // all of the thread's loads first, so their latencies overlap; read once,
    // so streaming (evict-first) loads.  Item j of a warp's lane is key
    // j * 32 + lane of the warp's run.
    const uint32_t first = w * (ITEMS * kWarp) + lane;
    uint32_t key[ITEMS];
    uint32_t* wh = s_whist + w * BINS;
    uint32_t* lm = smem + w * U * BINS;
    const uint32_t lbit = 1u << lane;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
        key[j] = first + j * kWarp < in_tile ? __ldcs(keys_in + tile_base + first + j * kWarp) : 0u;
    for (int i = threadIdx.x; i < (AREA + kSortWarps * BINS) / 4; i += kSortThreads)
        reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();

    // stable ranks within the warp: the lanes of an item with equal digits
    // take consecutive ranks, and the first of them moves the warp's count of
    // the digit, one item after the other (the order of equal keys).  The
    // lanes of equal digit meet in a shared word per digit, U items at a time
    // (words in the area the tile is staged in later); those of lane 0's digit
    // are found by a ballot instead, or runs of equal digits would serialise.
    uint32_t rank2[ITEMS / 2];  // two ranks below 2^16 each
#pragma unroll
    for (int j0 = 0; j0 < ITEMS; j0 += U) {
        uint32_t same[U], peers[U], at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool valid = first + (j0 + u) * kWarp < in_tile;
            const uint32_t d = (key[j0 + u] >> shift) & mask;
            const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
            same[u] = __ballot_sync(0xffffffffu, valid && d == d0);
            if (valid && d != d0) atomicOr(&lm[u * BINS + d], lbit);
            peers[u] = d == d0 ? 0u : 1u;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t d = (key[j0 + u] >> shift) & mask;
            peers[u] = peers[u] ? lm[u * BINS + d] : same[u];
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool valid = first + (j0 + u) * kWarp < in_tile;
            const uint32_t d = (key[j0 + u] >> shift) & mask;
            at[u] = 0u;
            if (valid && (peers[u] & (lbit - 1u)) == 0u) {
                lm[u * BINS + d] = 0u;
                at[u] = atomicAdd(&wh[d], (uint32_t)__popc(peers[u]));
            }
            __syncwarp();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int leader = peers[u] ? __ffs(peers[u]) - 1 : 0;
            const uint32_t r = __shfl_sync(0xffffffffu, at[u], leader) + (uint32_t)__popc(peers[u] & (lbit - 1u));
            if ((j0 + u) & 1) rank2[(j0 + u) / 2] |= r << 16;
            else rank2[(j0 + u) / 2] = r;
        }
    }
    // the values, in flight while the tile is counted (not before the ranks,
    // which need the registers)
    uint32_t val[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
        val[j] = first + j * kWarp < in_tile ? __ldcs(vals_in + tile_base + first + j * kWarp) : 0u;
    __syncthreads();

    // per digit the tile count, published before anything else so that
    // successors can make progress; then the digit starts of the tile and of
    // the whole sort in one scan, and per warp the first position of its keys
    uint32_t cnt[DPT], gcnt[DPT];
    unsigned long long sum = 0;
    uint32_t* status = scratch + kStatusOff + (uint64_t)pass * status_words(num_tiles, bins);
    uint16_t* rows = reinterpret_cast<uint16_t*>(status);
    uint32_t* sums = status + (uint64_t)num_tiles * bins / 2;
    const uint32_t groups = (num_tiles + kGroup - 1) / kGroup, g = tile / kGroup;
    uint32_t* prefixes = sums + (uint64_t)groups * bins;
    const uint32_t* ghist = scratch + kHistOff + pass * hstride;
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        const uint32_t d = threadIdx.x * DPT + q;
        uint32_t run = 0;
#pragma unroll
        for (int ww = 0; ww < kSortWarps; ++ww) run += s_whist[ww * BINS + d];
        cnt[q] = run;
        st_relaxed16(rows + (uint64_t)tile * bins + d, kTileDone | run);
        if (g + 1 < groups) atomicAdd(sums + (uint64_t)g * bins + d, kSumOne | run);  // no one reads the last group's
    }
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        gcnt[q] = ghist[threadIdx.x * DPT + q];
        sum += ((unsigned long long)gcnt[q] << 32) | cnt[q];
    }
    const unsigned long long ex = block_exclusive_scan2(sum, s_ws);
    uint32_t t_start = (uint32_t)ex, g_start = (uint32_t)(ex >> 32);
    uint32_t gbase[DPT];
#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        const uint32_t d = threadIdx.x * DPT + q;
        uint32_t at = t_start;
#pragma unroll
        for (int ww = 0; ww < kSortWarps; ++ww) {
            const uint32_t c = s_whist[ww * BINS + d];
            s_whist[ww * BINS + d] = at;
            at += c;
        }
        gbase[q] = g_start - t_start;  // modulo 2^32: the digit's sort position less its tile position
        t_start += cnt[q];
        g_start += gcnt[q];
    }
    __syncthreads();

    // stage the tile in digit order
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (first + j * kWarp < in_tile) {
            const uint32_t at = wh[(key[j] >> shift) & mask] + ((rank2[j / 2] >> (16 * (j & 1))) & 0xffffu);
            s_pairs[at] = make_uint2(key[j], val[j]);
        }
    }

#pragma unroll
    for (int q = 0; q < DPT; ++q) {
        const uint32_t d = threadIdx.x * DPT + q;
        const uint32_t excl = look_back(rows, sums, prefixes, bins, tile, d, scratch);
        // the group's last tile knows the keys up to the end of the group
        if (tile % kGroup == kGroup - 1 && g + 1 < groups)
            st_relaxed(prefixes + (uint64_t)g * bins + d, kPrefixDone | (excl + cnt[q]));
        s_gbase[d] = gbase[q] + excl;
    }
    __syncthreads();

    // coalesced write-out: consecutive staged keys of one digit go to
    // consecutive global positions
#pragma unroll 4
    for (uint32_t s = threadIdx.x; s < in_tile; s += kSortThreads) {
        const uint2 kv = s_pairs[s];
        const uint32_t o = s_gbase[(kv.x >> shift) & mask] + s;
        // o < n whenever the histogram and look-back are consistent; the
        // check keeps a timed-out look-back from writing out of bounds
        if (o < n) {
            keys_out[o] = kv.x;
            vals_out[o] = kv.y;
        }
    }
}

template <int BINS, int ITEMS>
static size_t pass_smem_bytes() {
    constexpr size_t stage = 2 * (size_t)kSortThreads * ITEMS, hist = (size_t)kSortWarps * BINS;
    return sizeof(uint32_t) * ((stage > hist ? stage : hist) + hist + BINS) +
           sizeof(unsigned long long) * (kSortWarps + 1);
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

cudaError_t sort_clear_async(uint32_t n, const SortPlan& plan, uint32_t* scratch, cudaStream_t st) {
    // counters, histograms and this sort's tile status; not the status word
    size_t clear_words = kStatusOff - 4 + (size_t)plan.passes * (size_t)status_words(num_tiles(n), status_bins(plan));
    return cudaMemsetAsync(scratch + 4, 0, clear_words * sizeof(uint32_t), st);
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

cudaError_t sort_histogram_async(const uint32_t* keys, uint32_t n, const SortPlan& plan, uint32_t* scratch,
                                 cudaStream_t st) {
    sort_histogram_kernel<<<hist_blocks(n), kHistThreads, 0, st>>>(keys, n, plan, scratch, aligned16(keys));
    return cudaGetLastError();
}

template <int BINS, int ITEMS>
static cudaError_t launch_pass(const uint32_t* ki, const uint32_t* vi, uint32_t* ko, uint32_t* vo,
                               uint32_t n, int shift, int bits, int pass, uint32_t tiles, uint32_t stride,
                               uint32_t bins, uint32_t* scratch, cudaStream_t st, const uint32_t* skip,
                               uint32_t skip_max) {
    size_t sm = pass_smem_bytes<BINS, ITEMS>();
    if (sm > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(sort_pass_kernel<BINS, ITEMS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        if (e != cudaSuccess) return e;
    }
    sort_pass_kernel<BINS, ITEMS><<<tiles, kSortThreads, sm, st>>>(ki, vi, ko, vo, n, shift, bits,
                                                                   pass, tiles, stride, bins, scratch, skip,
                                                                   skip_max);
    return cudaGetLastError();
}

// The digit passes alone: the histograms in scratch must be complete and the
// tile status cleared (sort_clear_async + a histogram producer).
cudaError_t sort_passes_async(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp,
                              uint32_t n, const SortPlan& plan, uint32_t* scratch, cudaStream_t st,
                              bool* in_tmp, const uint32_t* skip, uint32_t skip_max) {
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    const uint32_t tiles = num_tiles(n);
    uint32_t *ki = keys, *vi = vals, *ko = keys_tmp, *vo = vals_tmp;
    for (int p = 0; p < plan.passes; ++p) {
        cudaError_t e;
        const int b = plan.bits[p], sh = plan.shift[p];
        const uint32_t sd = (uint32_t)plan.stride, ss = status_bins(plan);
        if (g_sort_items >= 16)
            e = b > 9   ? launch_pass<1024, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max)
                : b > 8 ? launch_pass<512, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max)
                        : launch_pass<256, 16>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max);
        else
            e = b > 9   ? launch_pass<1024, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max)
                : b > 8 ? launch_pass<512, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max)
                        : launch_pass<256, 8>(ki, vi, ko, vo, n, sh, b, p, tiles, sd, ss, scratch, st, skip, skip_max);
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
    sort_hist_fallback_kernel<<<hist_blocks(n), kHistThreads, 0, st>>>(keys, vals, n, plan, scratch, skip, skip_max,
                                                                       words, aligned16(keys));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return sort_passes_async(keys, vals, keys_tmp, vals_tmp, n, plan, scratch, st, in_tmp, skip, skip_max);
}

// Sorts (keys, vals) by bits [0, key_bits).  Returns via *in_tmp whether
// the result ended in the tmp buffers (odd pass count).
cudaError_t sort_pairs_async(uint32_t* keys, uint32_t* vals, uint32_t* keys_tmp, uint32_t* vals_tmp,
                             uint32_t n, int key_bits, uint32_t* scratch, cudaStream_t st,
                             bool* in_tmp) {
    SortPlan plan = sort_plan(key_bits);
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    cudaError_t e = sort_clear_async(n, plan, scratch, st);
    if (e != cudaSuccess) return e;
    if ((e = sort_histogram_async(keys, n, plan, scratch, st)) != cudaSuccess) return e;
    return sort_passes_async(keys, vals, keys_tmp, vals_tmp, n, plan, scratch, st, in_tmp);
}

int sort_num_passes(int key_bits) { return sort_plan(key_bits).passes; }

}  // namespace sd

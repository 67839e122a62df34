// sd_sort_device.cuh -- the device side of the onesweep radix sort: digit
// histograms and one tile of a digit pass, used by the sort's own kernels
// (sd_sort.cu, which describes the algorithm) and by the re-sort's radix
// fallback (sd_resort.cu).
#pragma once

#include "sd_common.cuh"

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

// Bins the passes' status rows hold: those of the widest digit (bits[0]).
inline uint32_t status_bins(const SortPlan& p) { return p.bits[0] > 9 ? 1024u : (p.bits[0] > 8 ? 512u : 256u); }

// Words of one pass's status.  At most tiles * bins: half of that for the
// tiles, and two rows per 32 tiles for the groups of more than 32 tiles.
__host__ __device__ __forceinline__ uint64_t status_words(uint32_t tiles, uint32_t bins) {
    const uint32_t groups = (tiles + kGroup - 1) / kGroup;
    return ((uint64_t)tiles * bins) / 2 + (groups > 1 ? 2ull * groups * bins : 0ull);
}

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

// One tile of a digit pass by a CTA of kSortThreads (shared memory:
// sort_tile_smem bytes, 16-byte aligned).  BINS: 256, 512 or 1024 digit bins
// (template so narrow passes do less per-digit work).  ITEMS: keys per thread
// (tile = 256 * ITEMS keys).  hstride: the plan's histogram stride; bins: bins
// of a status row.  Thread t owns the digits [DPT * t, DPT * t + DPT).  FULL:
// every key is there (all tiles but the last); instructions bound the pass, and
// the tests of each key's place are a tenth of them (4,000,000 keys 30.5 -> 28.5
// us a pass, 9,437,184 entries 51 -> 47.8).
template <int BINS, int ITEMS, bool FULL = false>
__device__ __forceinline__ void sort_tile(uint32_t* smem, uint32_t tile, const uint32_t* keys_in,
                                          const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out, uint32_t n,
                                          int shift, int bits, int pass, uint32_t num_tiles, uint32_t hstride,
                                          uint32_t bins, uint32_t* scratch) {
    constexpr int TILE = kSortThreads * ITEMS;
    constexpr int DPT = BINS / kSortThreads;  // digits per thread (1, 2 or 4)
    constexpr int AREA = 2 * TILE > kSortWarps * BINS ? 2 * TILE : kSortWarps * BINS;  // words
    constexpr int U = AREA / (kSortWarps * BINS);  // items matched together (4, 2 or 1)
    static_assert(TILE < (int)kTileDone && TILE * kGroup < kSumOne, "counts fit their fields");
    uint2* s_pairs = reinterpret_cast<uint2*>(smem);  // TILE (key, value)
    uint32_t* s_whist = smem + AREA;           // kSortWarps * BINS
    uint32_t* s_gbase = s_whist + kSortWarps * BINS;  // BINS
    unsigned long long* s_ws = reinterpret_cast<unsigned long long*>(s_gbase + BINS);  // kSortWarps

    const uint32_t mask = (1u << bits) - 1u;
    const uint32_t w = threadIdx.x / kWarp;
    const uint32_t lane = lane_id();

    const uint32_t tile_base = tile * TILE;
    const uint32_t in_tile = FULL || n - tile_base >= (uint32_t)TILE ? (uint32_t)TILE : n - tile_base;

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
        key[j] = FULL || first + j * kWarp < in_tile ? __ldcs(keys_in + tile_base + first + j * kWarp) : 0u;
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
            const bool valid = FULL || first + (j0 + u) * kWarp < in_tile;
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
            const bool valid = FULL || first + (j0 + u) * kWarp < in_tile;
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
        val[j] = FULL || first + j * kWarp < in_tile ? __ldcs(vals_in + tile_base + first + j * kWarp) : 0u;
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
        if (FULL || first + j * kWarp < in_tile) {
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
constexpr size_t sort_tile_smem() {
    constexpr size_t stage = 2 * (size_t)kSortThreads * ITEMS, hist = (size_t)kSortWarps * BINS;
    return sizeof(uint32_t) * ((stage > hist ? stage : hist) + hist + BINS) +
           sizeof(unsigned long long) * kSortWarps;
}

}  // namespace sd

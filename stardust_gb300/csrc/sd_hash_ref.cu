// sd_hash_ref.cu -- the reference's spatial-hash broad phase, bit-exact.
//
// ref_hash_build_kernel restates constructCollisionListCUDA
// (src/engine/cuda/sh_collision_detection.cu:27-127): nine (cell, sphere)
// slots per sphere, home entry first, then the phantom entries the reference
// emits, then padding.  Keys, padding words and the valid-entry count are
// reproduced exactly, including the reference's parse of its phantom test
// (:95), under which only offsets in {0,+1}^3 are ever emitted.  Unlike the
// reference's 16-CTA grid-stride launch, one thread handles one sphere on a
// grid sized to the input, and the count is warp-reduced before one atomic
// per warp.
//
// The candidate-pair kernels restate the run traversal of
// tranverseCollisionListCUDA (collision_resolution.cu:100-199): within each
// run of equal cell (key >> 1), each of the first h entries (the homes, which
// sort first because their key LSB is 0) pairs with every later entry.  The
// reference walks runs serially per thread; here every entry is independent:
// pass 1 counts each home's pairs, a decoupled-look-back scan turns counts
// into offsets, pass 2 writes the pairs at those offsets -- the same order
// the reference's traversal visits them.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sd_common.cuh"
#include "sd_internal.h"

namespace sd {

__device__ __forceinline__ uint32_t f2u_rz_sat(float q) {
    // cvt.rzi.u32.f32: truncate, saturate to [0, 2^32-1], NaN -> 0
    return __float2uint_rz(q);
}

constexpr int kBuildThreads = 256;

// The reference's 27 offsets: one of -1 along any axis never passes its test
// (a side is 0, 1 or 3, and side ^ -1 is not 0), one of +1 passes where the
// side is 1, so the emitted ones are {0, 1}^3 less the origin, in the order of
// the 27: x fastest.  A block's 9 entries per sphere are written in shared
// memory (9 words apart: no bank conflicts) and copied out in one piece; one
// thread's own 9 words, 36 bytes from its neighbour's, took 76 us for
// 1,048,576 spheres (95 MB, floor 14 us), this 28.
__global__ void __launch_bounds__(kBuildThreads)
ref_hash_build_kernel(uint32_t n, float cell_dim, uint32_t* __restrict__ cells, uint32_t* __restrict__ spheres,
                      const float* __restrict__ sizes, const float4* __restrict__ pos4,
                      uint32_t* __restrict__ d_count) {
    stream_wait();
    __shared__ uint32_t s_cells[9 * kBuildThreads], s_spheres[9 * kBuildThreads];
    const uint32_t first = blockIdx.x * kBuildThreads, i = first + threadIdx.x;
    uint32_t count = 0;
    if (i < n) {
        uint32_t* c = s_cells + 9 * threadIdx.x;
        uint32_t* s = s_spheres + 9 * threadIdx.x;
        const float4 p4 = pos4[i];
        const float pos[3] = {p4.x, p4.y, p4.z};
        const float a = sizes[i];
        uint32_t hash = 0, cell[3], side[3];
        bool in[3][2];  // the offset 0 or 1 stays in [0, 1)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float q = __fdiv_rn(pos[j], cell_dim);
            cell[j] = f2u_rz_sat(q);
            hash = (hash << 8) | cell[j];
            const float x = __fmaf_rn(-floorf(q), cell_dim, pos[j]);
            side[j] = x < a ? 3u : (__fsub_rn(cell_dim, x) < a ? 1u : 0u);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float shifted = __fadd_rn(pos[j], __fmul_rn((float)r, cell_dim));
                in[j][r] = !(shifted < 0.0f || shifted >= 1.0f) && (r == 0 || side[j] == 1u);
            }
        }
        c[0] = hash << 1;
        s[0] = (i << 1) | 1u;
        count = 1;
#pragma unroll
        for (uint32_t m = 1; m < 8; ++m) {
            const uint32_t rx = m & 1u, ry = (m >> 1) & 1u, rz = m >> 2;
            if (in[0][rx] && in[1][ry] && in[2][rz]) {
                const uint32_t h = ((((cell[0] + rx) << 8) | (cell[1] + ry)) << 8) | (cell[2] + rz);
                c[count] = (h << 1) | 1u;
                s[count] = i << 1;
                ++count;
            }
        }
        for (uint32_t m = count; m < 9; ++m) {
            c[m] = 0xffffffffu;
            s[m] = i << 2;
        }
    }
    // warp-aggregate the count, one atomic per warp
    const uint32_t v = __reduce_add_sync(0xffffffffu, count);
    if (lane_id() == 0 && v) atomicAdd(d_count, v);
    __syncthreads();
    const uint32_t words = 9 * (n - first < (uint32_t)kBuildThreads ? n - first : (uint32_t)kBuildThreads);
    for (uint32_t w = threadIdx.x; w < words; w += kBuildThreads) {
        cells[9 * (size_t)first + w] = s_cells[w];
        spheres[9 * (size_t)first + w] = s_spheres[w];
    }
}

cudaError_t ref_hash_build_async(uint32_t n, float cell_dim, uint32_t* cells, uint32_t* spheres,
                                 const float* sizes, const float4* pos, uint32_t* d_count,
                                 cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(d_count, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess || n == 0) return e;
    launch_after(st, (n + kBuildThreads - 1) / kBuildThreads, kBuildThreads, 0, ref_hash_build_kernel, n, cell_dim,
                 cells, spheres, sizes, pos, d_count);
    return cudaGetLastError();
}

// ------------------------------------------------------- candidate pairs
// Per-entry pair count: entry j at run offset o (run of length L with h
// homes) contributes L-1-o pairs when o < h, else 0; same-body partners
// are removed when body_of is given.
constexpr int kPairThreads = 256;
constexpr int kPairItems = 8;
constexpr int kPairTile = kPairThreads * kPairItems;

__device__ __forceinline__ void run_bounds(const uint32_t* cells, uint32_t count, uint32_t j,
                                           uint32_t* start, uint32_t* end) {
    uint32_t key = cells[j] >> 1;
    uint32_t s = j;
    while (s > 0 && (cells[s - 1] >> 1) == key) --s;
    uint32_t e = j + 1;
    while (e < count && (cells[e] >> 1) == key) ++e;
    *start = s;
    *end = e;
}

// Pairs contributed by entry j (0 when j is not among the run's homes).
__device__ __forceinline__ uint32_t entry_pairs(const uint32_t* cells, const uint32_t* spheres,
                                                uint32_t count, const int32_t* body_of, uint32_t j,
                                                uint32_t* rs, uint32_t* re) {
    uint32_t s, e;
    run_bounds(cells, count, j, &s, &e);
    *rs = s;
    *re = e;
    uint32_t h = 0;
    for (uint32_t k = s; k < e; ++k) h += spheres[k] & 1u;
    if (h == 0 || j - s >= h) return 0;  // run without a home, or j is a phantom slot
    if (!body_of) return e - j - 1;
    uint32_t home = spheres[j] >> 1;
    int32_t bh = body_of[home];
    uint32_t c = 0;
    for (uint32_t k = j + 1; k < e; ++k) c += body_of[spheres[k] >> 1] != bh;
    return c;
}

// Single-pass exclusive scan over 64-bit pair counts with decoupled
// look-back.  A tile's status is one 64-bit word: flag in the top two bits
// (1 aggregate, 2 inclusive), count in the low 62, so it is published and
// read atomically.
__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
constexpr unsigned long long kPairAgg = 1ull << 62, kPairInc = 2ull << 62, kPairMask = (1ull << 62) - 1;

// Tiles of kPairTile entries, taken in order; those past the last real entry
// end at once.  Entries are counted striped over the threads (coalesced, a
// warp's walks over neighbouring runs share cache lines), scanned in entry
// order through shared memory, and a tile's first pair is found by a warp that
// reads 32 predecessors at a time.  Eight consecutive entries per thread, one
// predecessor at a time and tiles over the padding took 112 us for the
// 9,437,184 entries of 1,048,576 spheres; now 50, bound by the walks to the
// ends of every run.
__global__ void __launch_bounds__(kPairThreads)
ref_pairs_kernel(const uint32_t* __restrict__ cells, const uint32_t* __restrict__ spheres,
                 const uint32_t* __restrict__ d_count, uint32_t n_entries,
                 const int32_t* __restrict__ body_of, uint32_t* __restrict__ pair_a,
                 uint32_t* __restrict__ pair_b, uint64_t cap, unsigned long long* __restrict__ d_npairs,
                 uint32_t* __restrict__ scratch) {
    stream_wait();
    __shared__ uint32_t s_np[kPairTile];              // pairs of every entry
    __shared__ unsigned long long s_off[kPairTile];   // the first of them
    __shared__ unsigned long long s_part[kPairThreads / kWarp];
    __shared__ unsigned long long s_excl;
    __shared__ uint32_t s_tile;
    const uint32_t count = min(*d_count, n_entries);
    unsigned long long* tiles = reinterpret_cast<unsigned long long*>(scratch + 16);
    if (threadIdx.x == 0) s_tile = atomicAdd(scratch + 4, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint32_t base = tile * kPairTile;
    if (base >= count) return;

    uint32_t re[kPairItems];
#pragma unroll
    for (int q = 0; q < kPairItems; ++q) {
        const uint32_t j = base + q * kPairThreads + threadIdx.x;
        uint32_t rs = 0;
        re[q] = 0;
        s_np[q * kPairThreads + threadIdx.x] =
            j < count ? entry_pairs(cells, spheres, count, body_of, j, &rs, &re[q]) : 0u;
    }
    __syncthreads();
    unsigned long long mine = 0;
#pragma unroll
    for (int q = 0; q < kPairItems; ++q) mine += s_np[threadIdx.x * kPairItems + q];
    unsigned long long inc = mine;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane_id() >= (uint32_t)o) inc += t;
    }
    const int w = threadIdx.x / kWarp;
    if (lane_id() == kWarp - 1) s_part[w] = inc;
    __syncthreads();
    unsigned long long wpre = 0, tile_total = 0;
    for (int k = 0; k < kPairThreads / kWarp; ++k) {
        if (k < w) wpre += s_part[k];
        tile_total += s_part[k];
    }
    unsigned long long run = wpre + inc - mine;
#pragma unroll
    for (int q = 0; q < kPairItems; ++q) {
        s_off[threadIdx.x * kPairItems + q] = run;
        run += s_np[threadIdx.x * kPairItems + q];
    }

    if (w == 0) {  // one warp looks back
        if (lane_id() == 0) st_relaxed64(&tiles[tile], (tile == 0 ? kPairInc : kPairAgg) | tile_total);
        unsigned long long excl = 0;
        uint32_t spins = 0;
        for (int64_t p = (int64_t)tile - 1; p >= 0;) {
            const int64_t at = p - (int64_t)lane_id();
            const unsigned long long v = at >= 0 ? ld_relaxed64(&tiles[at]) : kPairInc;
            const uint32_t missing = __ballot_sync(0xffffffffu, (v & ~kPairMask) == 0);
            const uint32_t whole = __ballot_sync(0xffffffffu, (v & kPairInc) != 0);
            // the lanes up to the nearest inclusive sum, or up to the first
            // tile that has not published
            const uint32_t stop = whole ? (uint32_t)__ffs(whole) : 32u, gap = missing ? (uint32_t)__ffs(missing) - 1u : 32u;
            const uint32_t use = min(stop, gap);
            unsigned long long add = lane_id() < use ? v & kPairMask : 0ull;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(0xffffffffu, add, o);
            excl += add;
            if (whole && stop <= gap) break;
            p -= use;
            if (use == 0) {
                if (++spins > kSpinLimit) {
                    if (lane_id() == 0) atomicOr(&scratch[0], kErrLookbackTimeout);
                    break;
                }
                __nanosleep(64);
            }
        }
        if (lane_id() == 0) {
            if (tile > 0) st_relaxed64(&tiles[tile], kPairInc | (excl + tile_total));
            s_excl = excl;
            // the tile of the last entry knows the grand total
            if (base + kPairTile >= count) {
                *d_npairs = excl + tile_total;
                if (excl + tile_total > cap) atomicOr(&scratch[0], kErrPairOverflow);
            }
        }
    }
    __syncthreads();

#pragma unroll
    for (int q = 0; q < kPairItems; ++q) {
        const uint32_t e = q * kPairThreads + threadIdx.x, j = base + e;
        if (s_np[e] == 0) continue;
        unsigned long long off = s_excl + s_off[e];
        const uint32_t home = spheres[j] >> 1;
        const int32_t bh = body_of ? body_of[home] : 0;
        for (uint32_t k = j + 1; k < re[q]; ++k) {
            const uint32_t other = spheres[k] >> 1;
            if (body_of && body_of[other] == bh) continue;
            if (off < cap) {
                pair_a[off] = home;
                pair_b[off] = other;
            }
            ++off;
        }
    }
}

uint64_t ref_pairs_scratch_words(uint64_t n_entries) {
    uint64_t tiles = (n_entries + kPairTile - 1) / kPairTile;
    if (tiles == 0) tiles = 1;
    return 16 + 2 * tiles;
}

cudaError_t ref_candidate_pairs_async(const uint32_t* cells, const uint32_t* spheres,
                                      const uint32_t* d_count, uint32_t n_entries,
                                      const int32_t* body_of, uint32_t* pair_a, uint32_t* pair_b,
                                      uint64_t cap, unsigned long long* d_npairs, uint32_t* scratch,
                                      cudaStream_t st) {
    uint64_t words = ref_pairs_scratch_words(n_entries);
    cudaError_t e = cudaMemsetAsync(scratch + 4, 0, (words - 4) * sizeof(uint32_t), st);
    if (e != cudaSuccess) return e;
    e = cudaMemsetAsync(d_npairs, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    if (n_entries == 0) return cudaSuccess;
    uint32_t tiles = (uint32_t)((n_entries + kPairTile - 1) / kPairTile);
    launch_after(st, tiles, kPairThreads, 0, ref_pairs_kernel, cells, spheres, d_count, n_entries, body_of, pair_a,
                 pair_b, cap, d_npairs, scratch);
    return cudaGetLastError();
}

}  // namespace sd

// sd_sap.cu -- sweep and prune over axis-aligned boxes.
//
// The reference's live broad phase (SAPCollision::processCollisions,
// src/engine/cuda/collisions/SAP/sap_detection.cu:668-706): per-object AABB
// from position and radius (computeAABBCUDA, :178-217), per-axis extents
// (projectAABBCUDA, :222-272), a radix sort of the lower x extents as
// uint32 float bits (sortLowestExtents, :278-290) and a windowed sweep
// (sweepAndPruneCUDA, :385-440).  Two operators here:
//
//  * sap_sweep_ref: that sweep's own rows, for drop-in use and parity: per
//    sorted position a row of up to 16 partner ids (padding 16, unused
//    entries -1), at most 9 filled, a window of 64 sorted positions, x then
//    y tested -- and, as written at :413-417, the x test of later window
//    entries compares against the home box's upper y once a y test has
//    run.  Rows are cleared to -1 first (the reference's initIdxCUDA,
//    :135-172, clears only entries [0, n + 15) because it indexes tid + i).
//  * sap_pairs: an exact broad phase -- every pair of overlapping closed
//    boxes -- by sorting the lower x extents (order-preserving float keys,
//    so negative coordinates sort correctly) and sweeping each box forward
//    while the next lower x is within its upper x.  The sweep is binned like
//    the reference's grid prototype (src/engine/testSAP.cu:341-438, objects
//    mapped to y-z cells, one x sweep per cell): a y-z grid of columns at
//    least as wide as the largest box, each box entered in the (at most 2 x 2)
//    columns it touches, entries stably sorted by column so that each column
//    keeps the x order, and each entry swept forward inside its column only.
//    A pair sharing several columns is reported in the column of its overlap's
//    lower y-z corner, so every pair is found once, by the same tests as the
//    unbinned sweep: the same pair set, listed by sd_pairs.cuh.
//    Measured, 2,000,000 boxes of one size, 2.25 entries and two pairs each:
//    425 us in all (488 in some processes); six radix passes 157, sweep 149, gather into x order 37, list
//    31, entries 22, bounds 23, scans 19.  It was 1412: four entries for every
//    box whether used or not, boxes of 48 bytes gathered through two indices,
//    and the sweep twice, once to count.
#include "sd_common.cuh"
#include "sd_engine_impl.h"
#include "sd_pairs.cuh"

namespace sd {

namespace {

constexpr int kSapThreads = 256;
constexpr int kRefWindow = 64;
constexpr int kRefPadding = 16;
constexpr int kRefMaxFill = 9;

inline uint32_t grid_for(uint64_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

// Ordered uint32 image of a float: a < b  <=>  key(a) < key(b).
__device__ __forceinline__ uint32_t float_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__global__ void aabb_kernel(uint32_t n, const float4* __restrict__ pos, const float* __restrict__ radius,
                            float4* __restrict__ lo, float4* __restrict__ hi) {
    stream_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[i];
    const float r = radius ? radius[i] : p.w;
    lo[i] = make_float4(p.x - r, p.y - r, p.z - r, 0.0f);
    hi[i] = make_float4(p.x + r, p.y + r, p.z + r, 0.0f);
}

// Keys of the lower x extents: raw float bits (the reference's cast, valid
// for non-negative x) or the order-preserving image.
__global__ void lower_x_keys_kernel(uint32_t n, const float4* __restrict__ lo, uint32_t* __restrict__ keys,
                                    uint32_t* __restrict__ vals, int ordered) {
    stream_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    keys[i] = ordered ? float_key(lo[i].x) : __float_as_uint(lo[i].x);
    vals[i] = i;
}

__global__ void sweep_ref_kernel(uint32_t n, const float* __restrict__ upperx, const float* __restrict__ lowerx_sorted,
                                 const float* __restrict__ uppery, const float* __restrict__ lowery,
                                 const uint32_t* __restrict__ idx_sorted, int32_t* __restrict__ rows) {
    stream_wait();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= n) return;
    int32_t row[kRefPadding];
#pragma unroll
    for (int k = 0; k < kRefPadding; ++k) row[k] = -1;
    int len = 0;
    const uint32_t home = idx_sorted[tid];
    float home_upper = upperx[home];
    const uint32_t end = min(tid + (uint32_t)kRefWindow, n);
    for (uint32_t i = tid + 1; i < end; ++i) {
        const float pl = lowerx_sorted[i];
        const uint32_t ph = idx_sorted[i];
        if (pl <= home_upper) {
            home_upper = uppery[home];  // as written: later x tests use the upper y
            if (lowery[ph] <= home_upper) {
                bool unique = true;
#pragma unroll
                for (int k = 0; k < kRefPadding; ++k) unique &= row[k] != (int32_t)ph;
                if (unique && len < kRefMaxFill && ph != tid) row[len++] = (int32_t)ph;
            }
        }
    }
    int4* out = reinterpret_cast<int4*>(rows + (size_t)tid * kRefPadding);
#pragma unroll
    for (int k = 0; k < kRefPadding / 4; ++k) out[k] = make_int4(row[4 * k], row[4 * k + 1], row[4 * k + 2], row[4 * k + 3]);
}

inline size_t al256(size_t x) { return (x + 255) & ~(size_t)255; }

// ---- the column grid of the binned sweep
constexpr int kMaxCols = 255;  // per axis
constexpr int kSlots = 4;      // most entries per box: 2 x 2 columns

struct SapGrid {
    float y0, z0, inv;  // column of v: floor((v - v0) * inv), clamped
    int gy, gz;
};

__device__ __forceinline__ int sap_col(float v, float v0, float inv, int g) {
    const float t = floorf((v - v0) * inv);
    return t >= 0.0f ? (t < (float)g ? (int)t : g - 1) : 0;  // NaN -> 0
}

__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Bounds of the boxes in y and z and their largest y or z extent, as
// ordered keys (minima stored complemented, so every word is a maximum; the
// words start at 0), and the sum and number of the extents.  NaN coordinates
// are skipped.  Also the sort keys of the lower x extents.
struct SapBounds {
    uint32_t w[5], count;
    double sum;
    uint32_t done;  // blocks that have added theirs
    SapGrid grid;   // made by the last of them
};

// Columns at least 1.0001 x the largest extent wide (so a box spans at most
// two columns per axis, rounding included), twice the mean extent (boxes of
// one size then take 2.25 entries each instead of 4, for as many tests), and
// at most kMaxCols per axis.  The width never changes the pairs.  (Made once:
// made by every thread of the kernels that use it, its division of doubles was
// 38 of the sweep's 230 us and 18 of the entries' 40.)
__device__ __forceinline__ SapGrid sap_grid(const SapBounds& b) {
    SapGrid r{0.0f, 0.0f, 0.0f, 1, 1};
    if (b.w[0] && b.w[1] && b.w[2] && b.w[3]) {
        const float y0 = key_float(~b.w[0]), y1 = key_float(b.w[1]), z0 = key_float(~b.w[2]), z1 = key_float(b.w[3]);
        const float ext = b.w[4] ? key_float(b.w[4]) : 0.0f;
        const float mean = b.count ? (float)(b.sum / b.count) : 0.0f;
        float c = fmaxf(fmaxf(ext * 1.0001f, (y1 - y0) / (float)kMaxCols), (z1 - z0) / (float)kMaxCols);
        if (mean > 0.0f) c = fmaxf(c, 2.0f * mean);
        if (c > 0.0f && c < INFINITY) {
            r.y0 = y0;
            r.z0 = z0;
            r.inv = 1.0f / c;
            r.gy = min(kMaxCols, max(1, (int)fminf((y1 - y0) * r.inv, 1e6f) + 1));
            r.gz = min(kMaxCols, max(1, (int)fminf((z1 - z0) * r.inv, 1e6f) + 1));
        }
    }
    return r;
}

constexpr int kBoundBlocks = 152 * 4;

__global__ void __launch_bounds__(kSapThreads)
sap_bounds_kernel(uint32_t n, const float4* __restrict__ lo, const float4* __restrict__ hi, SapBounds* __restrict__ out,
                  uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    stream_wait();
    __shared__ uint32_t s_w[5], s_count;
    __shared__ double s_sum;
    if (threadIdx.x < 5) s_w[threadIdx.x] = 0u;
    if (threadIdx.x == 0) {
        s_count = 0u;
        s_sum = 0.0;
    }
    __syncthreads();
    uint32_t m[5] = {0u, 0u, 0u, 0u, 0u}, count = 0;
    float sum = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = lo[i], b = hi[i];
        keys[i] = float_key(a.x);
        vals[i] = i;
        const float ly = fminf(a.y, b.y), hy = fmaxf(a.y, b.y), lz = fminf(a.z, b.z), hz = fmaxf(a.z, b.z);
        const float ey = hy - ly, ez = hz - lz;
        if (ly == ly) {
            m[0] = max(m[0], ~float_key(ly));
            m[1] = max(m[1], float_key(hy));
        }
        if (lz == lz) {
            m[2] = max(m[2], ~float_key(lz));
            m[3] = max(m[3], float_key(hz));
        }
        if (ey == ey) m[4] = max(m[4], float_key(ey));
        if (ez == ez) m[4] = max(m[4], float_key(ez));
        if (ey + ez < INFINITY) {
            sum += ey + ez;
            count += 2;
        }
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const uint32_t r = __reduce_max_sync(0xffffffffu, m[k]);
        if (lane_id() == 0 && r) atomicMax(&s_w[k], r);
    }
    const uint32_t c = __reduce_add_sync(0xffffffffu, count);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane_id() == 0 && c) {
        atomicAdd(&s_count, c);
        atomicAdd(&s_sum, (double)sum);
    }
    __syncthreads();
    if (threadIdx.x < 5 && s_w[threadIdx.x]) atomicMax(&out->w[threadIdx.x], s_w[threadIdx.x]);
    if (threadIdx.x == 0 && s_count) {
        atomicAdd(&out->count, s_count);
        atomicAdd(&out->sum, s_sum);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&out->done, 1u) == gridDim.x - 1) {
        __threadfence();
        SapBounds b{};
        for (int k = 0; k < 5; ++k) b.w[k] = __ldcg(&out->w[k]);
        b.count = __ldcg(&out->count);
        b.sum = __ldcg(&out->sum);
        out->grid = sap_grid(b);
    }
}

// Columns of a box, y-major.
struct SapSpan {
    int y0, y1, z0, z1;
};
__device__ __forceinline__ SapSpan sap_span(const SapGrid& g, float4 a, float4 b) {
    return SapSpan{sap_col(fminf(a.y, b.y), g.y0, g.inv, g.gy), sap_col(fmaxf(a.y, b.y), g.y0, g.inv, g.gy),
                   sap_col(fminf(a.z, b.z), g.z0, g.inv, g.gz), sap_col(fmaxf(a.z, b.z), g.z0, g.inv, g.gz)};
}

// The boxes in x order, 32 bytes each with the id in the lower corner's w
// lane and its first columns (y, z: a byte each) in the upper one's, the columns
// each touches (first y, first z, one more in y, in z: a byte
// each) and their number.
__global__ void sap_gather_kernel(uint32_t n, const uint32_t* __restrict__ svals, const float4* __restrict__ lo,
                                  const float4* __restrict__ hi, const SapBounds* __restrict__ bounds,
                                  float4* __restrict__ box, uint32_t* __restrict__ span, uint32_t* __restrict__ count,
                                  uint32_t* __restrict__ status) {
    stream_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const SapGrid g = bounds->grid;
    const uint32_t id = svals[k];
    const float4 a = lo[id], b = hi[id];
    box[2 * (size_t)k] = make_float4(a.x, a.y, a.z, __uint_as_float(id));
    const SapSpan s = sap_span(g, a, b);
    box[2 * (size_t)k + 1] = make_float4(b.x, b.y, b.z, __uint_as_float((uint32_t)s.y0 | (uint32_t)s.z0 << 8));
    if (s.y1 - s.y0 > 1 || s.z1 - s.z0 > 1) atomicOr(status, kErrBadInput);  // excluded by the column width
    const uint32_t dy = (uint32_t)min(s.y1 - s.y0, 1), dz = (uint32_t)min(s.z1 - s.z0, 1);
    span[k] = (uint32_t)s.y0 | (uint32_t)s.z0 << 8 | dy << 16 | dz << 24;
    count[k] = (dy + 1u) * (dz + 1u);
}

// (The columns and counts are used up: span and count, cleared, are the sink's.)
__global__ void sap_entries_kernel(uint32_t n, uint32_t* __restrict__ span, uint32_t* __restrict__ count,
                                   const SapBounds* __restrict__ bounds, const uint32_t* __restrict__ off,
                                   uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    stream_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const SapGrid g = bounds->grid;
    const uint32_t s = span[k], y0 = s & 255u, z0 = (s >> 8) & 255u;
    uint32_t e = off[k];
    for (uint32_t y = y0; y <= y0 + ((s >> 16) & 1u); ++y)
        for (uint32_t z = z0; z <= z0 + (s >> 24); ++z) {
            keys[e] = y * (uint32_t)g.gz + z;
            vals[e++] = k;
        }
    span[k] = 0u;
    count[k] = 0u;
}

// Forward sweep of entry p inside its column: entries m > p of the same
// column with lower x <= upper x of p's box (x order within the column, the
// first miss ends it), tested on y, z and x like the unbinned sweep; a pair
// counts in the column of its overlap's lower y-z corner only: in y and in z
// the later of the two boxes' first columns.  A block's
// kSweep entries and the kSweepAhead behind them are fetched once, into shared
// memory (an entry is tested against some nine before it; fetched anew for each
// test -- column, index, box, one load waiting for the other -- the sweep of
// 2,000,000 boxes took 215 us, now 149: 64 the fetching, 38 the tests, 47 the
// pairs); what lies further is fetched.  256 entries to a block; with 128, 512 or
// a block walking over tiles, the next one's indices loaded ahead, it takes 270,
// 165 and 162.
constexpr int kSweep = 256, kSweepAhead = 32, kSweepTile = kSweep + kSweepAhead;
constexpr uint32_t kSweepBlocks = 128;  // per SM: a block takes one tile of up to 5 million entries

template <bool REFILL>
__global__ void __launch_bounds__(kSweep)
sweep_binned_kernel(const uint32_t* __restrict__ d_entries, const uint32_t* __restrict__ ckeys,
                    const uint32_t* __restrict__ cvals, const float4* __restrict__ box,
                    const SapBounds* __restrict__ bounds, PairSink sink) {
    stream_wait();
    __shared__ float s_lx[kSweepTile], s_ly[kSweepTile], s_lz[kSweepTile], s_hx[kSweepTile], s_hy[kSweepTile],
        s_hz[kSweepTile];
    __shared__ uint32_t s_col[kSweepTile], s_id[kSweepTile], s_first[kSweepTile];
    __shared__ PairBuffer<REFILL ? 1 : 1024> s_found;
    const uint32_t n_entries = *d_entries;
    if (REFILL && !sink_refill(sink)) return;
    const uint32_t gz = (uint32_t)bounds->grid.gz, t = threadIdx.x;
    for (uint32_t p0 = blockIdx.x * kSweep; p0 < n_entries; p0 += gridDim.x * kSweep) {
        const uint32_t end = min(n_entries - p0, (uint32_t)kSweepTile);
        if (t == 0) s_found.n = 0u;
        for (uint32_t i = t; i < end; i += kSweep) {
            const size_t m = cvals[p0 + i];
            const float4 lo = box[2 * m], hi = box[2 * m + 1];
            s_col[i] = ckeys[p0 + i];
            s_lx[i] = lo.x;
            s_ly[i] = lo.y;
            s_lz[i] = lo.z;
            s_id[i] = __float_as_uint(lo.w);
            s_hx[i] = hi.x;
            s_hy[i] = hi.y;
            s_hz[i] = hi.z;
            s_first[i] = __float_as_uint(hi.w);
        }
        __syncthreads();
        if (t < end) {
            const uint32_t col = s_col[t], id = s_id[t];
            const float lx = s_lx[t], ly = s_ly[t], lz = s_lz[t], hx = s_hx[t], hy = s_hy[t], hz = s_hz[t];
            const uint32_t first = s_first[t];
            const auto found = [&](uint32_t theirs, uint32_t other) {
                const uint32_t cy = max(first & 255u, theirs & 255u), cz = max(first >> 8, theirs >> 8);
                if (cy * gz + cz != col) return;
                if (REFILL) sink_pair_again(sink, id, other);
                else buffer_pair(s_found, sink, id, other);
            };
            uint32_t i = t + 1;
            for (; i < end; ++i) {
                if (s_col[i] != col || !(s_lx[i] <= hx)) break;
                const float bly = s_ly[i], bhy = s_hy[i];
                if (!(bly <= hy && ly <= bhy)) continue;
                const float blz = s_lz[i], bhz = s_hz[i];
                if (blz <= hz && lz <= bhz && lx <= s_hx[i]) found(s_first[i], s_id[i]);
            }
            if (i == (uint32_t)kSweepTile)  // past what the block holds
                for (uint32_t q = p0 + i; q < n_entries && ckeys[q] == col; ++q) {
                    const size_t m = cvals[q];
                    const float4 lo = box[2 * m];
                    if (!(lo.x <= hx)) break;
                    const float4 hi = box[2 * m + 1];
                    if (lo.y <= hy && ly <= hi.y && lo.z <= hz && lz <= hi.z && lx <= hi.x)
                        found(__float_as_uint(hi.w), __float_as_uint(lo.w));
                }
        }
        __syncthreads();
        if (!REFILL) {
            flush_pairs(s_found, sink, t, kSweep);
            if (p0 + gridDim.x * kSweep < n_entries) __syncthreads();
        }
    }
}

__global__ void project_kernel(uint32_t n, const float4* __restrict__ lo, const float4* __restrict__ hi,
                               float* __restrict__ upperx, float* __restrict__ uppery, float* __restrict__ lowery) {
    stream_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    upperx[i] = hi[i].x;
    uppery[i] = hi[i].y;
    lowery[i] = lo[i].y;
}

}  // namespace

// The kept partners lie over what the columns' sort is done with when the sweep
// begins: the *_tmp arrays (two passes end where they began) and its scratch.
static uint64_t keep_more_bytes(uint64_t m) {
    const uint64_t over = 2 * al256(4 * kSlots * m) + al256(4 * sort_scratch_words(kSlots * m, 16));
    return 4 * kPairKeep * m > over ? al256(4 * kPairKeep * m - over) : 0;
}
uint64_t sap_scratch_bytes(uint64_t n, uint64_t pair_cap) {
    const uint64_t m = n ? n : 1;
    (void)pair_cap;
    return 4 * al256(4 * m) + al256(4 * sort_scratch_words(m, 32)) + al256(32 * m) + 4 * al256(4 * (m + 1)) +
           al256(4 * scan_scratch_words((uint32_t)m + 1)) + al256(16) + 4 * al256(4 * kSlots * m) +
           al256(4 * sort_scratch_words(kSlots * m, 16)) + keep_more_bytes(m) + al256(64);
}
// What sd_sap_process_collisions takes of it: the x sort, corners and projections.
static uint64_t process_scratch_bytes(uint64_t n) {
    const uint64_t m = n ? n : 1;
    return 4 * al256(4 * m) + al256(4 * sort_scratch_words(m, 32)) + al256(48 * m);
}

cudaError_t sap_aabb_async(uint32_t n, const float4* pos, const float* radius, float4* lo, float4* hi,
                           cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    launch_after(st, grid_for(n, kSapThreads), kSapThreads, 0, aabb_kernel, n, pos, radius, lo, hi);
    return cudaGetLastError();
}

cudaError_t sap_sort_lower_x_async(uint32_t n, const float4* lo, bool ordered, uint32_t* keys, uint32_t* vals,
                                   uint32_t* keys_tmp, uint32_t* vals_tmp, uint32_t* sort_scratch, bool* in_tmp,
                                   cudaStream_t st) {
    *in_tmp = false;
    if (n == 0) return cudaSuccess;
    launch_after(st, grid_for(n, kSapThreads), kSapThreads, 0, lower_x_keys_kernel, n, lo, keys, vals,
                 ordered ? 1 : 0);
    return sort_pairs_async(keys, vals, keys_tmp, vals_tmp, n, 32, sort_scratch, st, in_tmp);
}

cudaError_t sap_sweep_ref_async(uint32_t n, const float* upperx, const float* lowerx_sorted, const float* uppery,
                                const float* lowery, const uint32_t* idx_sorted, int32_t* rows, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    launch_after(st, grid_for(n, kSapThreads), kSapThreads, 0, sweep_ref_kernel, n, upperx, lowerx_sorted, uppery,
                 lowery, idx_sorted, rows);
    return cudaGetLastError();
}

cudaError_t sap_pairs_async(uint32_t n, const float4* lo, const float4* hi, void* scratch, uint64_t pair_cap,
                            unsigned long long* out, uint32_t* d_count2, cudaStream_t st) {
    const uint64_t m = n ? n : 1;
    char* p = static_cast<char*>(scratch);
    auto take = [&](size_t bytes) {
        char* r = p;
        p += al256(bytes);
        return r;
    };
    uint32_t* keys = (uint32_t*)take(4 * m);
    uint32_t* vals = (uint32_t*)take(4 * m);
    uint32_t* keys_tmp = (uint32_t*)take(4 * m);
    uint32_t* vals_tmp = (uint32_t*)take(4 * m);
    uint32_t* sort_scratch = (uint32_t*)take(4 * sort_scratch_words(m, 32));
    float4* box = (float4*)take(32 * m);
    uint32_t* counts = (uint32_t*)take(4 * (m + 1));
    uint32_t* eoff = (uint32_t*)take(4 * (m + 1));
    uint32_t* off = (uint32_t*)take(4 * (m + 1));
    uint32_t* cursor = (uint32_t*)take(4 * (m + 1));
    uint32_t* scan = (uint32_t*)take(4 * scan_scratch_words((uint32_t)m + 1));
    uint32_t* status = (uint32_t*)take(16);
    uint32_t* ckeys = (uint32_t*)take(4 * kSlots * m);
    uint32_t* cvals = (uint32_t*)take(4 * kSlots * m);
    uint32_t* ckeys_tmp = (uint32_t*)take(4 * kSlots * m);
    uint32_t* cvals_tmp = (uint32_t*)take(4 * kSlots * m);
    uint32_t* csort = (uint32_t*)take(4 * sort_scratch_words(kSlots * m, 16));
    take(keep_more_bytes(m));
    SapBounds* bounds = (SapBounds*)take(64);
    uint32_t* keep = ckeys_tmp;  // (free when the sweep begins)
    static_assert(sizeof(SapBounds) <= 64, "bounds fit their scratch");
    if (n == 0) return cudaMemsetAsync(d_count2, 0, 8, st);
    // (the caller's two pointers by memsets, which check them; the rest by kernels)
    cudaError_t e = cudaMemsetAsync(status, 0, 16, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_count2, 0, 8, st);
    if (e == cudaSuccess) e = zero_async(st, {bounds, sizeof(SapBounds) / 4});
    if (e != cudaSuccess) return e;
    const uint32_t grid = grid_for(n, kSapThreads);
    launch_after(st, std::min<uint32_t>(grid, kBoundBlocks), kSapThreads, 0, sap_bounds_kernel, n, lo, hi, bounds,
                 keys, vals);
    bool in_tmp = false;
    if ((e = sort_pairs_async(keys, vals, keys_tmp, vals_tmp, n, 32, sort_scratch, st, &in_tmp, nullptr, true)) !=
        cudaSuccess)
        return e;
    // each box's entries, stably sorted by column
    launch_after(st, grid, kSapThreads, 0, sap_gather_kernel, n, in_tmp ? vals_tmp : vals, lo, hi, bounds, box,
                 cursor, counts, status);
    if ((e = scan_exclusive_async(counts, eoff, n, scan, st)) != cudaSuccess) return e;
    launch_after(st, grid, kSapThreads, 0, sap_entries_kernel, n, cursor, counts, bounds, eoff, ckeys,
                 cvals);
    const uint32_t ne = kSlots * n;
    bool c_tmp = false;
    if ((e = sort_pairs_async(ckeys, cvals, ckeys_tmp, cvals_tmp, ne, 16, csort, st, &c_tmp, eoff + n, true)) !=
        cudaSuccess)
        return e;
    if (c_tmp) return cudaErrorUnknown;  // (16 bits: two passes)
    const PairSink sink{counts, keep, status + 1, off, cursor, out, n, pair_cap};
    launch_after(st, std::min(grid_for(ne, kSweep), 152u * kSweepBlocks), kSweep, 0, sweep_binned_kernel<false>,
                 eoff + n, ckeys, cvals, box, bounds, sink);
    if ((e = scan_exclusive_async(counts, off, n, scan, st)) != cudaSuccess) return e;
    launch_after(st, std::min(grid_for(ne, kSweep), 152u * 4), kSweep, 0, sweep_binned_kernel<true>, eoff + n, ckeys,
                 cvals, box, bounds, sink);
    launch_after(st, grid, kSapThreads, 0, pairs_write_kernel, sink, d_count2, status);
    return cudaGetLastError();
}

}  // namespace sd

// =================================================================== C ABI
extern "C" {

sd_status sd_sap_scratch_bytes(uint64_t n, uint64_t pair_cap, uint64_t* bytes) {
    if (!bytes) return sd_fail(nullptr, SD_ERR_INVALID_ARG, "bytes NULL");
    if (n >= (1ull << 30)) return sd_fail(nullptr, SD_ERR_CAPACITY, "n must be < 2^30");
    *bytes = sd::sap_scratch_bytes(n, pair_cap);
    return SD_OK;
}

sd_status sd_sap_pairs(uint64_t n, const float* d_lo4, const float* d_hi4, uint64_t* d_pairs, uint64_t cap,
                       uint32_t* d_count, void* d_scratch, uint64_t scratch_bytes, void* stream) {
    if (n && (!d_lo4 || !d_hi4 || !d_scratch)) return sd_fail(nullptr, SD_ERR_INVALID_ARG, "NULL pointer");
    if (!d_count) return sd_fail(nullptr, SD_ERR_INVALID_ARG, "d_count NULL");
    if (n >= (1ull << 30)) return sd_fail(nullptr, SD_ERR_CAPACITY, "n must be < 2^30");
    if (scratch_bytes < sd::sap_scratch_bytes(n, cap))
        return sd_fail(nullptr, SD_ERR_CAPACITY, "scratch smaller than sd_sap_scratch_bytes");
    if ((reinterpret_cast<uintptr_t>(d_lo4) | reinterpret_cast<uintptr_t>(d_hi4)) & 15u)
        return sd_fail(nullptr, SD_ERR_INVALID_ARG, "boxes must be 16-byte aligned");
    cudaError_t e = sd::sap_pairs_async((uint32_t)n, reinterpret_cast<const float4*>(d_lo4),
                                        reinterpret_cast<const float4*>(d_hi4), d_scratch, cap,
                                        reinterpret_cast<unsigned long long*>(d_pairs), d_count,
                                        static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return sd_cuda_fail(nullptr, e, "sd_sap_pairs");
    return SD_OK;
}

sd_status sd_sap_sweep(uint64_t n, const float* d_upperx, const float* d_lowerx_sorted, const float* d_uppery,
                       const float* d_lowery, const uint32_t* d_idx_sorted, int32_t* d_rows, void* stream) {
    if (n && (!d_upperx || !d_lowerx_sorted || !d_uppery || !d_lowery || !d_idx_sorted || !d_rows))
        return sd_fail(nullptr, SD_ERR_INVALID_ARG, "NULL pointer");
    if (n >= (1ull << 31) / 16) return sd_fail(nullptr, SD_ERR_CAPACITY, "n too large for 16-entry rows");
    if (reinterpret_cast<uintptr_t>(d_rows) & 15u) return sd_fail(nullptr, SD_ERR_INVALID_ARG, "rows must be 16-byte aligned");
    cudaError_t e = sd::sap_sweep_ref_async((uint32_t)n, d_upperx, d_lowerx_sorted, d_uppery, d_lowery, d_idx_sorted,
                                            d_rows, static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return sd_cuda_fail(nullptr, e, "sd_sap_sweep");
    return SD_OK;
}

sd_status sd_sap_process_collisions(uint64_t n, const float* d_pos4, const float* d_radius, int32_t* d_rows,
                                    void* d_scratch, uint64_t scratch_bytes, void* stream) {
    if (n && (!d_pos4 || !d_rows || !d_scratch)) return sd_fail(nullptr, SD_ERR_INVALID_ARG, "NULL pointer");
    if (n >= (1ull << 31) / 16) return sd_fail(nullptr, SD_ERR_CAPACITY, "n too large for 16-entry rows");
    if (scratch_bytes < sd::process_scratch_bytes(n))
        return sd_fail(nullptr, SD_ERR_CAPACITY, "scratch smaller than sd_sap_scratch_bytes(n, 0)");
    if ((reinterpret_cast<uintptr_t>(d_pos4) | reinterpret_cast<uintptr_t>(d_rows)) & 15u)
        return sd_fail(nullptr, SD_ERR_INVALID_ARG, "positions and rows must be 16-byte aligned");
    const uint32_t m = n ? (uint32_t)n : 1u;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* p = static_cast<char*>(d_scratch);
    auto take = [&](size_t bytes) {
        char* r = p;
        p += sd::al256(bytes);
        return r;
    };
    uint32_t* keys = (uint32_t*)take(4ull * m);
    uint32_t* vals = (uint32_t*)take(4ull * m);
    uint32_t* keys_tmp = (uint32_t*)take(4ull * m);
    uint32_t* vals_tmp = (uint32_t*)take(4ull * m);
    uint32_t* sort_scratch = (uint32_t*)take(4ull * sd::sort_scratch_words(m, 32));
    float4* lo = (float4*)take(48ull * m);  // lower and upper corners, then the projections
    float4* hi = lo + m;
    float* proj = reinterpret_cast<float*>(hi + m);
    float* upperx = proj;
    float* uppery = proj + m;
    float* lowery = proj + 2ull * m;
    if (n == 0) return SD_OK;
    bool in_tmp = false;
    cudaError_t e = sd::sap_aabb_async((uint32_t)n, reinterpret_cast<const float4*>(d_pos4), d_radius, lo, hi, st);
    if (e == cudaSuccess)
        e = sd::sap_sort_lower_x_async((uint32_t)n, lo, false, keys, vals, keys_tmp, vals_tmp, sort_scratch, &in_tmp,
                                       st);
    if (e == cudaSuccess) {
        sd::launch_after(st, sd::grid_for(n, sd::kSapThreads), sd::kSapThreads, 0, sd::project_kernel, (uint32_t)n,
                         lo, hi, upperx, uppery, lowery);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = sd::sap_sweep_ref_async((uint32_t)n, upperx, reinterpret_cast<const float*>(in_tmp ? keys_tmp : keys),
                                    uppery, lowery, in_tmp ? vals_tmp : vals, d_rows, st);
    if (e != cudaSuccess) return sd_cuda_fail(nullptr, e, "sd_sap_process_collisions");
    return SD_OK;
}

}  // extern "C"

// sd_resort.cu -- the step's cell sort as an incremental re-sort.
//
// Every step sorts the spheres' new cell keys (key, slot) stably, slot order
// being the sorted order of the previous step.  Between two steps almost
// every sphere keeps its cell (1,048,576 settling spheres: 0-100 changes per
// step), so the result is the previous order with a few entries moved, and
// it can be built without a radix sort:
//
//   1. the kernel that writes the new keys (contact or body kernel) appends
//      every slot whose new key differs from the sorted key it sits under
//      ("moved") to a list as (key << 32 | slot), one warp-aggregated atomic
//      per warp that has any (the list's order does not matter);
//   2. resort_plan_kernel, one block: publishes the count M and, in shared
//      memory, sorts the list by (key, slot) and the moved slots alone
//      (each entry placed by counting the smaller ones); moved entry r
//      (rank r in (key, slot) order) goes to r plus the unmoved slots that
//      sort before it -- the previous step's cell
//      table bounds the slots of its key, so that count is its slot clamped
//      to that range minus the moved slots below it.  Only positions between
//      a moved entry's old slot and its new position change hands, so it also
//      lists those intervals (with the prefix sums of their lengths) for the
//      reorder;
//   3. the in-place reorder (dem_fix_gather_kernel, dem_fix_place_kernel in
//      sd_dem.cu) visits the intervals' positions and reads the order from
//      these lists: position k holds a moved entry where one was placed,
//      else the unmoved slot of rank k - (moved entries placed before k).
//
// The unmoved slots are already in (key, slot) order, so this is a merge of
// two sorted sequences and the result is exactly the stable LSD sort's.
// When more than `mmax` keys change, the plan kernel clears the radix sort's
// counters and histograms and the step's fallback (histogram + passes, in
// the graph and returning at once otherwise) sorts; the reorder then reads
// their sorted arrays.
//
// resort_step_kernel does all of this in one cooperative launch, for runs of
// several steps (see there).
#include <cuda_runtime.h>
#include <stdint.h>

#include "sd_common.cuh"
#include "sd_internal.h"
#include "sd_reorder.cuh"
#include "sd_sort_device.cuh"

namespace sd {
namespace {

// one block of 1024 threads: one thread per moved entry of a full list
constexpr int kRsThreads = 1024;
// above this many moved entries the ranks are counted against sorted chunks
constexpr uint32_t kChunkedRankM = 256;
static_assert(kResortMaxCap <= (uint32_t)kRsThreads, "one thread per moved entry");

// scratch (u32): [0] moved count (appended to during the step, zero again
// when this kernel ends), [1] M of the step, [3] total length T of the
// shift intervals.  sort_clear: the radix fallback's tile counters and
// histograms, cleared when the fallback will run.
__global__ void __launch_bounds__(kRsThreads)
resort_plan_kernel(unsigned long long* __restrict__ list, uint32_t* __restrict__ pos_out,
                   uint32_t* __restrict__ q_out, uint32_t* __restrict__ iv_lo, uint32_t* __restrict__ iv_pre,
                   uint32_t mmax, uint32_t* __restrict__ scratch, const uint32_t* __restrict__ cell_start,
                   uint32_t ncells, uint32_t n, uint32_t* __restrict__ vl_flags, uint32_t* __restrict__ sort_clear,
                   uint32_t sort_clear_words) {
    __shared__ unsigned long long s_a[kResortMaxCap], s_b[kResortMaxCap];
    __shared__ uint32_t s_c[kResortMaxCap];
    __shared__ uint32_t s_M, ws[33];
    if (threadIdx.x == 0) {
        const uint32_t M = scratch[0];
        s_M = M;
        scratch[0] = 0u;
        scratch[1] = M;
        if (vl_flags) {  // the skin lists: build next step if a sphere left its skin this step
            if (vl_flags[0]) ++vl_flags[2];  // steps that built the lists
            else ++vl_flags[3];              // steps that used them
            vl_flags[0] = vl_flags[1];
            vl_flags[1] = 0u;
        }
    }
    __syncthreads();
    const uint32_t M = s_M;
    if (M > mmax) {  // the radix fallback sorts this step
        for (uint32_t i = threadIdx.x; i < sort_clear_words; i += blockDim.x) sort_clear[i] = 0u;
        return;
    }
    if (M == 0) {
        if (threadIdx.x == 0) scratch[3] = 0u;
        return;
    }
    if (M > kChunkedRankM) {
        // each entry is placed by counting the smaller ones (entries and
        // slots are distinct), chunk by chunk: every warp sorts 32 entries
        // by (key, slot) and their slots alone (bitonic network over the
        // lanes), then each entry adds up, over the chunks, the number of
        // smaller elements (binary search): M/32 chunks x 6 probes per
        // order instead of M comparisons
        const uint32_t lane = threadIdx.x & 31u, t = threadIdx.x;
        unsigned long long v = t < M ? list[t] : ~0ull;
        uint32_t sv = t < M ? (uint32_t)v : 0xffffffffu;
        const unsigned long long c = v;
        for (uint32_t k = 2; k <= 32; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, (int)j);
                const uint32_t os = __shfl_xor_sync(0xffffffffu, sv, (int)j);
                const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
                v = take_min ? (o < v ? o : v) : (o < v ? v : o);
                sv = take_min ? min(os, sv) : max(os, sv);
            }
        s_b[t] = v;  // chunks of 32, each ascending (padding last)
        s_c[t] = sv;
        __syncthreads();
        uint32_t ra = 0, rs = 0;
        if (t < M) {
            const uint32_t cs = (uint32_t)c, nch = (M + 31u) >> 5;
            for (uint32_t q = 0; q < nch; ++q) {
                const unsigned long long* A = s_b + 32u * q;
                const uint32_t* S = s_c + 32u * q;
                uint32_t pa = 0, ps = 0;  // elements of the chunk below c, below cs
#pragma unroll
                for (uint32_t step = 32; step > 0; step >>= 1) {
                    if (pa + step <= 32u && A[pa + step - 1u] < c) pa += step;
                    if (ps + step <= 32u && S[ps + step - 1u] < cs) ps += step;
                }
                ra += pa;
                rs += ps;
            }
        }
        __syncthreads();
        if (t < M) {
            s_a[ra] = c;
            s_b[rs] = c & 0xffffffffull;  // the moved slots, ascending
        }
        __syncthreads();
    } else {
        // each entry is placed by counting the smaller ones (entries and
        // slots are distinct): G threads per entry, G the largest power of two
        // up to 32 with G * M <= 1024, each counting a G-th of the list, then
        // summed across the G lanes; two barriers in all
        uint32_t G = 32;
        while (G > 1 && G * M > (uint32_t)kRsThreads) G >>= 1;
        if (threadIdx.x < M) s_b[threadIdx.x] = list[threadIdx.x];
        __syncthreads();
        const uint32_t r = threadIdx.x / G, g = threadIdx.x % G;
        const unsigned long long c = r < M ? s_b[r] : 0ull;
        uint32_t ra = 0, rs = 0;
        if (r < M) {
            for (uint32_t j = g; j < M; j += G) {
                const unsigned long long o = s_b[j];
                ra += o < c;
                rs += (o & 0xffffffffull) < (c & 0xffffffffull);
            }
        }
        for (uint32_t o = G >> 1; o > 0; o >>= 1) {
            ra += __shfl_xor_sync(0xffffffffu, ra, (int)o);
            rs += __shfl_xor_sync(0xffffffffu, rs, (int)o);
        }
        __syncthreads();
        if (r < M && g == 0) {
            s_a[ra] = c;
            s_b[rs] = c & 0xffffffffull;  // the moved slots, ascending
        }
        __syncthreads();
    }
    // one moved entry per thread (M <= kResortMaxCap = blockDim.x)
    const uint32_t r = threadIdx.x;
    uint32_t len = 0, lo = 0;
    if (r < M) {
        const unsigned long long c = s_a[r];
        const uint32_t key = (uint32_t)(c >> 32), slot = (uint32_t)c;
        // the previous order's slots of keys below `key` are [0, L), those
        // of `key` itself [L, U); the unmoved ones among [0, clamp(slot, L,
        // U)) sort before (key, slot)
        const uint32_t L = min(cell_start[min(key, ncells)], n);
        const uint32_t U = min(cell_start[min(key + 1, ncells)], n);
        const uint32_t x = min(max(slot, L), U);
        uint32_t a = 0, b = M;  // moved slots below x
        while (a < b) {
            const uint32_t mid = (a + b) >> 1;
            if (s_b[mid] < x) a = mid + 1;
            else b = mid;
        }
        const uint32_t p = r + x - a;
        list[r] = c;
        pos_out[r] = p;
        q_out[r] = (uint32_t)s_b[r] - r;
        // positions [min(slot, p), max(slot, p)] may change hands
        lo = min(slot, p);
        len = max(slot, p) - lo + 1u;
    }
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(len, ws, &total);
    if (r < M) {
        iv_lo[r] = lo;
        iv_pre[r] = ex;
    }
    if (threadIdx.x == 0) {
        iv_pre[M] = total;
        scratch[3] = total;
    }
}

// ------------------------------------------------- the one-kernel re-sort
constexpr int kStepThreads = kReorderThreads;
static_assert(kStepThreads == kSortThreads, "the fallback's tiles are sorted by whole blocks");

struct StepArgs {
    uint32_t n, ncells, mmax;
    const unsigned long long* list;  // the moved entries, in any order
    uint32_t* scratch;               // DemBuffers::rs_scratch
    uint32_t* vl_flags;              // may be null
    uint32_t* cell_start;
    FixState f;
    float* mesh_state;               // a mesh's pose, advanced here (may be null)
    // the radix fallback
    uint32_t *keys, *vals, *keys_tmp, *vals_tmp, *sort_scratch;
    SortPlan plan;
    uint32_t tiles, bins;
    uint64_t status_words;
    bool vec;
};

// Shared memory of the incremental path: the lists twice (a merge sort's
// source and destination), then what the reorder reads.
struct StepLists {
    unsigned long long e[2][kResortMaxCap];  // moved entries
    uint32_t s[2][kResortMaxCap];            // moved slots
    uint32_t pos[kResortMaxCap], q[kResortMaxCap], iv_lo[kResortMaxCap], iv_pre[kResortMaxCap];
};

// Waits until every block of the grid arrived (a cooperative launch: all of
// them are resident).  bar[0] counts arrivals, bar[1] the barriers passed.
// Bounded: a wait that gives up flags it and goes on.
__device__ __forceinline__ void grid_barrier(uint32_t* bar, uint32_t* errors) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const uint32_t gen = ld_relaxed(bar + 1);
        __threadfence();
        if (atomicAdd(bar, 1u) == gridDim.x - 1) {
            st_relaxed(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            uint32_t spins = 0;
            while (ld_relaxed(bar + 1) == gen) {
                if (++spins > kSpinLimit) {
                    atomicOr(errors, kErrLookbackTimeout);
                    break;
                }
                if (spins > 16) __nanosleep(20);
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// Sorts the M moved entries by (key, slot), and their slots alone: chunks of
// 32 by a bitonic network over a warp's lanes, then merges of neighbouring
// runs, every element placed by a binary search in the other run.  Returns
// the buffer (0 or 1) that holds both.  Loops stay rolled: the kernel starts
// with cold instruction caches, and fetching unrolled merges took longer (16
// us at 330 entries) than running them.
__device__ __forceinline__ uint32_t sort_moved(const unsigned long long* __restrict__ list, uint32_t M, StepLists& L) {
    uint32_t P = 32;
    while (P < M) P <<= 1;
    const uint32_t lane = threadIdx.x & 31u;
    if (M <= 32) {  // one warp, every element placed by counting the smaller ones
        if (threadIdx.x < 32) {
            const unsigned long long v = lane < M ? list[lane] : ~0ull;
            uint32_t a = 0, b = 0;
#pragma unroll 1
            for (uint32_t j = 0; j < M; ++j) {
                const unsigned long long o = __shfl_sync(0xffffffffu, v, (int)j);
                a += o < v;
                b += (uint32_t)o < (uint32_t)v;
            }
            if (lane < M) {
                L.e[0][a] = v;
                L.s[0][b] = (uint32_t)v;
            }
        }
        __syncthreads();
        return 0;
    }
    // two elements a thread, whose chains of shuffles and searches overlap
#pragma unroll 1
    for (uint32_t t0 = threadIdx.x; t0 < P; t0 += 2 * kStepThreads) {  // whole warps: P is a multiple of 32
        unsigned long long v[2];
        uint32_t sv[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t t = t0 + u * kStepThreads;
            v[u] = t < M ? list[t] : ~0ull;
            sv[u] = t < M ? (uint32_t)v[u] : 0xffffffffu;
        }
#pragma unroll 1
        for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll 1
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                const bool take_min = ((lane & j) == 0) == ((lane & k) == 0);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const unsigned long long o = __shfl_xor_sync(0xffffffffu, v[u], (int)j);
                    const uint32_t os = __shfl_xor_sync(0xffffffffu, sv[u], (int)j);
                    v[u] = take_min == (o < v[u]) ? o : v[u];
                    sv[u] = take_min ? min(os, sv[u]) : max(os, sv[u]);
                }
            }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t t = t0 + u * kStepThreads;
            if (t < P) {
                L.e[0][t] = v[u];
                L.s[0][t] = sv[u];
            }
        }
    }
    __syncthreads();
    uint32_t from = 0;
#pragma unroll 1
    for (uint32_t len = 32; len < P; len <<= 1) {
#pragma unroll 1
        for (uint32_t t0 = threadIdx.x; t0 < P; t0 += 2 * kStepThreads) {
            const unsigned long long* E[2];
            const uint32_t* S[2];
            unsigned long long x[2];
            uint32_t y[2], a[2] = {0u, 0u}, b[2] = {0u, 0u};
            bool second[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t t = min(t0 + u * kStepThreads, P - 1);
                second[u] = (t & len) != 0;
                E[u] = L.e[from] + (t & ~(2 * len - 1)) + (second[u] ? 0u : len);
                S[u] = L.s[from] + (t & ~(2 * len - 1)) + (second[u] ? 0u : len);
                x[u] = L.e[from][t];
                y[u] = L.s[from][t];
            }
            // elements of the other run before this one: below it, or (the
            // padding repeats) equal to it when this one is of the second run
#pragma unroll 1
            for (uint32_t step = len >> 1; step > 0; step >>= 1) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const unsigned long long v = E[u][a[u] + step - 1];
                    const uint32_t w = S[u][b[u] + step - 1];
                    a[u] += (v < x[u] || (second[u] && v == x[u])) ? step : 0u;
                    b[u] += (w < y[u] || (second[u] && w == y[u])) ? step : 0u;
                }
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t t = t0 + u * kStepThreads;
                if (t >= P) break;
                const unsigned long long v = E[u][a[u]];
                const uint32_t w = S[u][b[u]];
                const uint32_t at = (t & ~(2 * len - 1)) + (t & (len - 1));
                L.e[from ^ 1][at + a[u] + ((v < x[u] || (second[u] && v == x[u])) ? 1u : 0u)] = x[u];
                L.s[from ^ 1][at + b[u] + ((w < y[u] || (second[u] && w == y[u])) ? 1u : 0u)] = y[u];
            }
        }
        __syncthreads();
        from ^= 1;
    }
    return from;
}

// The radix fallback: the keys sorted stably by the sort's own tiles, all
// blocks of the grid taking tiles until none is left.  Returns whether the
// result is in the *_tmp buffers.
template <int BINS, int ITEMS>
__device__ __forceinline__ bool radix_sort_grid(const StepArgs& a, uint32_t* smem, uint32_t* s_tile, uint32_t* bar) {
    const uint64_t gt = (uint64_t)blockIdx.x * kStepThreads + threadIdx.x, gs = (uint64_t)gridDim.x * kStepThreads;
    for (uint64_t w = 4 + gt; w < kStatusOff + a.status_words; w += gs) a.sort_scratch[w] = 0u;
    grid_barrier(bar, a.sort_scratch);
    block_histograms<true>(a.keys, a.vals, a.n, a.plan, a.sort_scratch, smem, a.vec);
    grid_barrier(bar, a.sort_scratch);
    uint32_t *ki = a.keys, *vi = a.vals, *ko = a.keys_tmp, *vo = a.vals_tmp;
    for (int p = 0; p < a.plan.passes; ++p) {
        for (;;) {
            __syncthreads();  // the last tile's staging is read
            if (threadIdx.x == 0) *s_tile = atomicAdd(&a.sort_scratch[4 + p], 1u);
            __syncthreads();
            const uint32_t tile = *s_tile;
            if (tile >= a.tiles) break;
            sort_tile<BINS, ITEMS>(smem, tile, ki, vi, ko, vo, a.n, a.plan.shift[p], a.plan.bits[p], p, a.tiles,
                                   (uint32_t)a.plan.stride, a.bins, a.sort_scratch);
        }
        grid_barrier(bar, a.sort_scratch);
        uint32_t* t;
        t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    return (a.plan.passes & 1) != 0;
}

// What follows a step's contact stage -- the plan, the radix fallback when
// it is due, the in-place reorder, the mesh's pose -- in one cooperative
// launch.  As separate kernels (plan, histogram, passes, gather, place, pose)
// each costs 2-3 us whatever it has to do, and the radix kernels of a step
// that needs none still run: 13 us of a 17 us step at 4,096 spheres, 26 of 51
// at 1,048,576.  Here every block sorts the moved list and works the plan out
// for itself (M <= 1,024 entries; 2 us, where one block that hands its result
// to the others would need a barrier more), gathers its share of the
// positions, and after one grid barrier places them and shifts the cell
// table.  A step without moved slots ends at once.
// Measured (per step, the separate kernels before): 4,096 spheres 17.4 -> 7.5
// us the step; 1,048,576 falling spheres 26 -> 10 us after the contact stage
// (50-90 moved slots, up to 85,000 positions); 256 scenes of 1.57M spheres 44
// -> 16 us (340 moved slots); the drum 28 -> 11 us.  Bound by latency: load
// and sort 2-3 us (7.6 at 340 entries), plan 1.5, gather 2.4, barrier 2-4,
// place and cells 2.5.  Two blocks per SM (registers of the fallback's tiles).
template <int BINS, int ITEMS>
__global__ void __launch_bounds__(kStepThreads, 2) resort_step_kernel(StepArgs a) {
    stream_wait();
    extern __shared__ __align__(16) uint32_t smem[];
    __shared__ uint32_t ws[33], s_tile, s_keys[kReorderThreads + 1];
    const uint32_t M = a.scratch[0];
    uint32_t* const bar = a.scratch + 4;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (a.vl_flags) {  // the skin lists: build next step if a sphere left its skin this step
            if (a.vl_flags[0]) ++a.vl_flags[2];  // steps that built the lists
            else ++a.vl_flags[3];                // steps that used them
            a.vl_flags[0] = a.vl_flags[1];
            a.vl_flags[1] = 0u;
        }
        a.scratch[1] = M;
        if (a.mesh_state) mesh_pose(a.mesh_state, true);
    }
    if (M == 0) return;
    if (M > a.mmax) {
        const bool tmp = radix_sort_grid<BINS, ITEMS>(a, smem, &s_tile, bar);
        const uint32_t *keys = tmp ? a.keys_tmp : a.keys, *vals = tmp ? a.vals_tmp : a.vals;
        fix_gather_all(a.n, vals, a.f);
        grid_barrier(bar, a.sort_scratch);
        if (blockIdx.x == 0 && threadIdx.x == 0) a.scratch[0] = 0u;
        fix_place_all(a.n, a.ncells, keys, vals, a.f, a.cell_start, s_keys);
        return;
    }
    StepLists& L = *reinterpret_cast<StepLists*>(smem);
    const uint32_t in = sort_moved(a.list, M, L);
    const unsigned long long* E = L.e[in];
    const uint32_t* S = L.s[in];
    // per moved entry its position and the interval its move shifts (see the
    // plan kernel), and its old key, before any block places a key
    uint32_t* old = L.s[in ^ 1];
    uint32_t T = 0;
#pragma unroll 1
    for (uint32_t r0 = 0; r0 < M; r0 += kStepThreads) {
        const uint32_t r = r0 + threadIdx.x;
        uint32_t len = 0;
        if (r < M) {
            const uint32_t key = (uint32_t)(E[r] >> 32), slot = (uint32_t)E[r];
            old[r] = min(slot < a.n ? a.f.keys_prev[slot] : key, a.ncells);
            const uint32_t lo = min(a.cell_start[min(key, a.ncells)], a.n);
            const uint32_t hi = min(a.cell_start[min(key + 1, a.ncells)], a.n);
            const uint32_t x = min(max(slot, lo), hi);
            const uint32_t p = r + x - lower_idx(S, M, x);
            L.pos[r] = p;
            L.q[r] = S[r] - r;
            L.iv_lo[r] = min(slot, p);
            len = max(slot, p) - min(slot, p) + 1u;
        }
        uint32_t sum;
        const uint32_t ex = block_exclusive_scan(len, ws, &sum);
        if (r < M) L.iv_pre[r] = T + ex;
        T += sum;
    }
    __syncthreads();
    const MovedLists ml{M, E, L.pos, L.q, L.iv_lo, L.iv_pre};
    const bool iv = T <= a.n / 4;
    const uint32_t total = iv ? T : a.n;
    // a thread's first position crosses the barrier in registers (a few tens
    // of thousands of positions change hands in a step: all of them), others
    // through the free buffers
    const uint32_t t0 = blockIdx.x * kStepThreads + threadIdx.x, t1 = t0 + gridDim.x * kStepThreads;
    uint32_t k = a.n, src = a.n, key = 0;
    bool place = false, move = false;
    Entry e;
    if (t0 < total && (k = visit_position(t0, iv, ml)) < a.n) {
        place = sorted_entry(k, ml, &src, &key);
        if (!place && src < a.n) key = a.f.keys_new[src];
        move = src != k && src < a.n;
        place = place || src != k;
        if (move) e = take_entry(a.n, k, src, a.f);
    }
    fix_gather_moved(t1, a.n, total, iv, ml, a.f);
    grid_barrier(bar, a.sort_scratch);
    if (blockIdx.x == 0 && threadIdx.x == 0) a.scratch[0] = 0u;
    if (move) put_entry(a.n, k, e, a.f);
    if (place) a.f.keys_prev[k] = key;
    fix_place_moved(t1, a.n, total, iv, ml, a.f);
    // The cell table: a move along z shifts a few cells, one along x a whole
    // plane of columns (15,876 at 1,048,576 spheres: 27 us for one block).
    // Short ranges go one to a block, long ones over the grid.
    for (uint32_t r0 = 0; r0 < M; r0 += 32) {
        const uint32_t r = r0 + lane_id();
        const uint32_t to = r < M ? min((uint32_t)(E[r] >> 32), a.ncells) : 0u, from = r < M ? old[r] : 0u;
        const bool wide = max(from, to) - min(from, to) > 8 * kStepThreads;
        uint32_t todo = __ballot_sync(0xffffffffu, wide || (r < M && r % gridDim.x == blockIdx.x));
        const uint32_t spread = __ballot_sync(0xffffffffu, wide);
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            const bool all = (spread >> q) & 1u;
            shift_cells(__shfl_sync(0xffffffffu, from, q), __shfl_sync(0xffffffffu, to, q), a.cell_start,
                        all ? blockIdx.x : 0u, all ? gridDim.x : 1u);
        }
    }
}

template <int BINS, int ITEMS>
cudaError_t launch_step(const StepArgs& a, int per_sm, cudaStream_t st) {
    constexpr size_t tile = sort_tile_smem<BINS, ITEMS>();
    const size_t sm = tile > sizeof(StepLists) ? tile : sizeof(StepLists);
    const auto kernel = resort_step_kernel<BINS, ITEMS>;
    int dev = 0, sms = 0, fit = 0;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, kStepThreads, sm);
    if (e != cudaSuccess) return e;
    const uint32_t most = (uint32_t)(sms * (fit < per_sm ? fit : per_sm));
    const uint32_t want = (a.n + kStepThreads - 1) / kStepThreads;
    launch_chained<true>(st, want < most ? want : most, kStepThreads, sm, kernel, a);
    return cudaGetLastError();
}

}  // namespace

static uint32_t g_resort_max = 1024;

void dem_set_resort_max(uint32_t m) { g_resort_max = m; }
uint32_t dem_resort_max() { return g_resort_max; }

uint64_t resort_scratch_words(uint32_t) { return 8; }  // [4], [5]: the grid barrier

cudaError_t resort_plan_async(const DemBuffers& b, cudaStream_t st, uint32_t* vl_flags) {
    const uint32_t n = b.n, mmax = b.rs_max;
    if (n == 0 || mmax == 0) return cudaSuccess;
    if (mmax > kResortMaxCap || (mmax & (mmax - 1)) != 0) return cudaErrorInvalidValue;
    resort_plan_kernel<<<1, kRsThreads, 0, st>>>(b.rs_list, b.rs_pos, b.rs_q, b.rs_iv_lo, b.rs_iv_pre, mmax,
                                                 b.rs_scratch, b.cell_start, b.ncells, n, vl_flags,
                                                 b.sort_scratch + 4, (uint32_t)sort_fallback_clear_words());
    return cudaGetLastError();
}

cudaError_t resort_step_async(const DemBuffers& b, const SortPlan& plan, int per_sm, uint32_t* vl_flags,
                              const ListView& lv, bool slot_all, cudaStream_t st) {
    StepArgs a{};
    a.n = b.n;
    a.ncells = b.ncells;
    a.mmax = b.rs_max;
    a.list = b.rs_list;
    a.scratch = b.rs_scratch;
    a.vl_flags = vl_flags;
    a.cell_start = b.cell_start;
    a.f = FixState{b.pos_n, b.vel_n, b.omg_n, b.pos, b.vel, b.omg, b.keys_prev, b.keys, b.slot_of, slot_all, lv};
    a.mesh_state = b.mesh.ntri ? b.mesh.state : nullptr;
    a.keys = b.keys;
    a.vals = b.vals;
    a.keys_tmp = b.keys_tmp;
    a.vals_tmp = b.vals_tmp;
    a.sort_scratch = b.sort_scratch;
    a.plan = plan;
    const int items = sort_items();
    a.tiles = (b.n + kSortThreads * items - 1) / (kSortThreads * items);
    a.bins = status_bins(plan);
    a.status_words = (uint64_t)plan.passes * status_words(a.tiles, a.bins);
    a.vec = (reinterpret_cast<uintptr_t>(b.keys) & 15u) == 0;
    if (items >= 16)
        return a.bins == 1024 ? launch_step<1024, 16>(a, per_sm, st)
               : a.bins == 512 ? launch_step<512, 16>(a, per_sm, st)
                               : launch_step<256, 16>(a, per_sm, st);
    return a.bins == 1024 ? launch_step<1024, 8>(a, per_sm, st)
           : a.bins == 512 ? launch_step<512, 8>(a, per_sm, st)
                           : launch_step<256, 8>(a, per_sm, st);
}

}  // namespace sd

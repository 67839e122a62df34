// sd_reorder.cuh -- the in-place reorder of a step: the sorted order from the
// incremental re-sort's lists, the entries that change hands gathered and
// placed, the cell table.  Used by the reorder's kernels (sd_dem.cu) and by
// the one-kernel re-sort (sd_resort.cu).
#pragma once

#include "sd_common.cuh"

namespace sd {

constexpr uint32_t kIdMask = 0x7fffffffu;
constexpr int kReorderThreads = 256;

// Writes cell_start for the cells block [b0, b1) owns, (s_keys[0],
// s_keys[cnt]] (the first block starts at cell 0, the last ends at ncells),
// by binary search over the block's sorted keys s_keys[1..cnt] in shared
// memory, so that every cell's lower bound is written exactly once.  Cells
// at or before the block's first key take b0 and cells after its last key
// (only the last block has them: the tail up to ncells) take b1 without a
// search -- an empty region past the last sphere can be tens of thousands
// of cells, all in that one block.
__device__ __forceinline__ void block_cell_starts(const uint32_t* s_keys, uint32_t b0, uint32_t b1, uint32_t n,
                                                  uint32_t ncells, uint32_t* __restrict__ cell_start) {
    const int64_t lo = b0 == 0 ? -1 : (int64_t)s_keys[0];
    const int64_t hi = b1 == n ? (int64_t)ncells : min((int64_t)s_keys[b1 - b0], (int64_t)ncells);
    const uint32_t cnt = b1 - b0;
    const int64_t kfirst = cnt ? (int64_t)s_keys[1] : hi, klast = cnt ? (int64_t)s_keys[cnt] : lo;
    for (int64_t c = lo + 1 + threadIdx.x; c <= hi; c += blockDim.x) {
        if (c <= kfirst || c > klast) {
            cell_start[c] = c <= kfirst ? b0 : b1;
            continue;
        }
        uint32_t a = 0, z = cnt;  // first index in [0, cnt) with key >= c, else cnt
        while (a < z) {
            uint32_t m = (a + z) >> 1;
            if ((int64_t)s_keys[m + 1] < c) a = m + 1;
            else z = m;
        }
        cell_start[c] = b0 + a;
    }
}

// First index in [0, m) of ascending a with a[i] >= x (m if none).
__device__ __forceinline__ uint32_t lower_idx(const uint32_t* a, uint32_t m, uint32_t x) {
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// First index in [0, m) of ascending a with a[i] > x (m if none).
__device__ __forceinline__ uint32_t upper_idx(const uint32_t* a, uint32_t m, uint32_t x) {
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The sorted order the incremental re-sort found: the M moved entries in (key,
// slot) order with their sorted positions, per moved slot in ascending order
// slot - rank, and the intervals of positions their moves shift (first
// positions, and exclusive prefix sums of the lengths: M + 1 entries).
struct MovedLists {
    uint32_t M;
    const unsigned long long* list;
    const uint32_t *pos, *q, *iv_lo, *iv_pre;
};

// Source slot of sorted position k: a moved entry where one was placed
// (returns true, *key its key), else the unmoved slot of rank u = k - (moved
// entries placed before k), which is u + #{moved slots s_j with s_j - j <= u}.
// An unmoved slot's new key is its previous one.
__device__ __forceinline__ bool sorted_entry(uint32_t k, const MovedLists& ml, uint32_t* src, uint32_t* key) {
    const uint32_t lo = lower_idx(ml.pos, ml.M, k);
    if (lo < ml.M && ml.pos[lo] == k) {
        const unsigned long long c = ml.list[lo];
        *src = (uint32_t)c;
        *key = (uint32_t)(c >> 32);
        return true;
    }
    const uint32_t u = k - lo;
    *src = u + upper_idx(ml.q, ml.M, u);
    return false;
}

// The state a step sorts in place (S: the next state, in the previous slot
// order) and the free buffers (T) its moving entries pass through.
struct FixState {
    float4 *s_pos, *s_vel, *s_omg;
    float4 *t_pos, *t_vel, *t_omg;
    uint32_t* keys_prev;        // per position: the key it is sorted under
    const uint32_t* keys_new;   // per slot: the new key
    uint32_t* slot_of;          // per id: its slot (null: not kept)
    bool slot_all;              // for every sphere, else for clump spheres
    ListView lv;
};

// The in-place reorder of a step whose next state stays where the contact
// kernel wrote it (S, the *_n buffers, in the previous slot order).  Sorted
// position k needs the entry of slot src(k); where src(k) == k -- every
// slot but those shifted by the moved keys -- nothing moves.  Only
// positions between a moved entry's old slot and its new position can
// change hands, so with the re-sort's order the kernels visit those
// intervals (T positions in all; a position in several is visited by each,
// writing the same values) rather than all n, unless T is above n / 4.
// Phase 1 gathers the positions that change hands into the free buffer T
// (the step's input state, no longer read) and, with the re-sort's order,
// shifts the cell table: cell_start[c] counts the entries with key < c, so
// an entry moving from key a to key b takes one from the cells (a, b] when
// b > a and adds one to (b, a] when b < a (atomic adds: several entries may
// share cells).  Phase 2 copies the gathered entries back and records
// their keys; for the radix passes' order (more moves than the re-sort
// takes) every position is visited and the cell table is rebuilt as the
// plain reorder does.  Both kernels run on a fixed grid (grid-stride).

// Position visited by work item t: in interval mode the position of item t
// among the intervals' concatenation, else t itself.
__device__ __forceinline__ uint32_t visit_position(uint32_t t, bool iv, const MovedLists& ml) {
    if (!iv) return t;
    const uint32_t r = upper_idx(ml.iv_pre, ml.M, t) - 1u;  // iv_pre[0] = 0 <= t
    return ml.iv_lo[r] + (t - ml.iv_pre[r]);
}

// An entry on its way from one slot to another; its list's ids go through
// lv.nbr_t, four at a time.
struct Entry {
    float4 pos, vel, omg, ref;
    uint32_t cnt;
};

__device__ __forceinline__ void copy_ids(uint32_t n, uint32_t c, const uint32_t* from, uint32_t src, uint32_t* to,
                                         uint32_t dst) {
    c = min(c, kVlCap);
    for (uint32_t q = 0; q < c; q += 4) {
        uint32_t id[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (q + u < c) id[u] = from[(size_t)(q + u) * n + src];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (q + u < c) to[(size_t)(q + u) * n + dst] = id[u];
    }
}

// Slot i's entry of the state (pos, vel, omg) and the lists (cnt, ref): all
// loads before anything is stored, so that they are in flight together.
__device__ __forceinline__ Entry load_entry(const float4* pos, const float4* vel, const float4* omg,
                                            const uint32_t* cnt, const float4* ref, uint32_t i) {
    Entry e;
    e.pos = pos[i];
    e.vel = vel[i];
    e.omg = omg[i];
    e.cnt = cnt ? cnt[i] : 0u;
    e.ref = cnt ? ref[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    return e;
}

// The entry of slot src, for position k, off to the free buffers.
__device__ __forceinline__ Entry take_entry(uint32_t n, uint32_t k, uint32_t src, const FixState& f) {
    const Entry e = load_entry(f.s_pos, f.s_vel, f.s_omg, f.lv.cnt, f.lv.ref, src);
    if (f.lv.cnt) copy_ids(n, e.cnt, f.lv.nbr, src, f.lv.nbr_t, k);
    return e;
}

// Puts an entry (its ids in lv.nbr_t) at position k.
__device__ __forceinline__ void put_entry(uint32_t n, uint32_t k, const Entry& e, const FixState& f) {
    f.s_pos[k] = e.pos;
    f.s_vel[k] = e.vel;
    f.s_omg[k] = e.omg;
    const uint32_t idb = __float_as_uint(e.omg.w);
    if (f.slot_of && (f.slot_all || (idb & kClumpFlag)) && (idb & kIdMask) < n) f.slot_of[idb & kIdMask] = k;
    if (f.lv.cnt) {
        f.lv.cnt[k] = e.cnt;
        f.lv.ref[k] = e.ref;
        copy_ids(n, e.cnt, f.lv.nbr_t, k, f.lv.nbr, k);
    }
}

// Phase 1 for position k whose entry comes from slot src.
__device__ __forceinline__ void fix_gather(uint32_t n, uint32_t k, uint32_t src, const FixState& f) {
    if (src == k || src >= n) return;
    const Entry e = take_entry(n, k, src, f);
    f.t_pos[k] = e.pos;
    f.t_vel[k] = e.vel;
    f.t_omg[k] = e.omg;
    if (f.lv.cnt) {
        f.lv.cnt_t[k] = e.cnt;
        f.lv.ref_t[k] = e.ref;
    }
}

// Phase 2 for position k, which takes slot src's entry and the key.
__device__ __forceinline__ void fix_place(uint32_t n, uint32_t k, uint32_t src, uint32_t key, const FixState& f) {
    if (src != k && src < n) put_entry(n, k, load_entry(f.t_pos, f.t_vel, f.t_omg, f.lv.cnt_t, f.lv.ref_t, k), f);
    f.keys_prev[k] = key;
}

// The re-sort's order, work items t, t + grid, ... (phase 1 and 2).  A
// position that keeps its unmoved entry keeps its key too: nothing to write.
__device__ __forceinline__ void fix_gather_moved(uint32_t t, uint32_t n, uint32_t total, bool iv,
                                                 const MovedLists& ml, const FixState& f) {
    for (; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t k = visit_position(t, iv, ml);
        if (k >= n) continue;
        uint32_t src, key;
        sorted_entry(k, ml, &src, &key);
        fix_gather(n, k, src, f);
    }
}
__device__ __forceinline__ void fix_place_moved(uint32_t t, uint32_t n, uint32_t total, bool iv,
                                                const MovedLists& ml, const FixState& f) {
    for (; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t k = visit_position(t, iv, ml);
        if (k >= n) continue;
        uint32_t src, key = 0;
        const bool moved = sorted_entry(k, ml, &src, &key);
        if (src == k && !moved) continue;
        fix_place(n, k, src, moved ? key : (src < n ? f.keys_new[src] : 0u), f);
    }
}

// The radix passes' order (vals: source slot, keys: key of every position).
// Phase 2 takes chunks of kReorderThreads consecutive positions per block (a
// block of that many threads), so that each chunk rebuilds its part of the
// cell table; s_keys: kReorderThreads + 1 words.
__device__ __forceinline__ void fix_gather_all(uint32_t n, const uint32_t* vals, const FixState& f) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        fix_gather(n, k, __ldcg(vals + k), f);
}
__device__ __forceinline__ void fix_place_all(uint32_t n, uint32_t ncells, const uint32_t* keys, const uint32_t* vals,
                                              const FixState& f, uint32_t* cell_start, uint32_t* s_keys) {
    for (uint32_t b0 = blockIdx.x * kReorderThreads; b0 < n; b0 += gridDim.x * kReorderThreads) {
        const uint32_t b1 = min(b0 + kReorderThreads, n), k = b0 + threadIdx.x;
        if (k < n) {
            const uint32_t key = __ldcg(keys + k);
            fix_place(n, k, __ldcg(vals + k), key, f);
            s_keys[threadIdx.x + 1] = key;
        }
        if (threadIdx.x == 0) s_keys[0] = b0 == 0 ? 0u : __ldcg(keys + b0 - 1);
        __syncthreads();
        block_cell_starts(s_keys, b0, b1, n, ncells, cell_start);
        __syncthreads();
    }
}

// An add whose result nobody waits for (atomicAdd through a generic pointer
// was compiled to one that is waited for: 0.43 us per 256 cells).
__device__ __forceinline__ void red_add(uint32_t* p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}

// A moved entry's shift of the cell table (its key goes from a to b): cells
// (a, b] lose one when b > a, (b, a] gain one when b < a.  By block `part` of
// `parts` that share the range.
__device__ __forceinline__ void shift_cells(uint32_t a, uint32_t b, uint32_t* cell_start, uint32_t part = 0,
                                            uint32_t parts = 1) {
    const uint32_t lo = min(a, b) + 1, hi = max(a, b);  // cells [lo, hi]
    const uint32_t d = b > a ? 0xffffffffu : 1u;        // -1 or +1
    for (uint32_t cc = lo + part * blockDim.x + threadIdx.x; cc <= hi; cc += parts * blockDim.x)
        red_add(cell_start + cc, d);
}

// Rotation matrix (row-major) of a unit quaternion (s, x, y, z).
__device__ __forceinline__ void quat_rot(float qs, float qx, float qy, float qz, float* R) {
    R[0] = 1.0f - 2.0f * (qy * qy + qz * qz);
    R[1] = 2.0f * (qx * qy - qs * qz);
    R[2] = 2.0f * (qx * qz + qs * qy);
    R[3] = 2.0f * (qx * qy + qs * qz);
    R[4] = 1.0f - 2.0f * (qx * qx + qz * qz);
    R[5] = 2.0f * (qy * qz - qs * qx);
    R[6] = 2.0f * (qx * qz - qs * qy);
    R[7] = 2.0f * (qy * qz + qs * qx);
    R[8] = 1.0f - 2.0f * (qx * qx + qy * qy);
}

// The mesh pose of the next step, by one thread: q <- normalize(dq (x) q)
// (Hamilton product) when advance, then the rotation matrix of q (the
// expression of the rigid bodies).
__device__ __forceinline__ void mesh_pose(float* S, bool advance) {
    float qs = S[16], qx = S[17], qy = S[18], qz = S[19];
    if (advance) {
        const float ds = S[20], dx = S[21], dy = S[22], dz = S[23];
        const float ns = ds * qs - ((dx * qx + dy * qy) + dz * qz);
        const float nx = (ds * qx + qs * dx) + (dy * qz - dz * qy);
        const float ny = (ds * qy + qs * dy) + (dz * qx - dx * qz);
        const float nz = (ds * qz + qs * dz) + (dx * qy - dy * qx);
        const float nrm = sqrtf((ns * ns + nx * nx) + (ny * ny + nz * nz));
        qs = ns / nrm;
        qx = nx / nrm;
        qy = ny / nrm;
        qz = nz / nrm;
        S[16] = qs;
        S[17] = qx;
        S[18] = qy;
        S[19] = qz;
    }
    quat_rot(qs, qx, qy, qz, S);
}

}  // namespace sd

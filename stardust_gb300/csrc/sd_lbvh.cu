// sd_lbvh.cu -- linear BVH broad phase over axis-aligned boxes.
//
// Replaces the LBVH prototype of sandbox/testLBVH.cu (:42-907), which
// builds its tree from Thrust/CUB calls, a depth probe with a device-to-host
// copy (:1148-1149) and depth+1 refit launches.  Here:
//   1. bounds: a two-level min/max reduction of the boxes (the global
//      domain, constructGlobalDomain, testLBVH.cu:82-89);
//   2. Morton codes exactly as computeSpaceFillingCurveCUDA (:113-151):
//      30 bits, centroid relative to the domain centre in units of
//      domain/1024, clamped to [-512, 511];
//   3. this library's onesweep radix sort of (code, index), 30-bit keys;
//   4. Karras (2012) binary radix tree, one thread per internal node, ties
//      between equal codes broken by the leaf index;
//   5. refit: subtrees of up to 128 leaves joined bottom-up in shared memory,
//      their boxes raised through the nodes above by atomic maxima;
//   6. stack traversal, a few lanes to a leaf: they take as many nodes off the
//      leaf's stack at a time.  Partner lists (both ways, per body, a count
//      pass and a write pass) or the unique pairs (each found once, from the
//      leaf that comes first along the curve; sd_pairs.cuh).
// The pair set is the exact set of overlapping closed boxes, independent of
// the tree's shape.
#include "sd_common.cuh"
#include "sd_pairs.cuh"

#include <algorithm>
#include <utility>

namespace sd {

namespace {

constexpr int kLbvhThreads = 256;
constexpr uint32_t kLeaf = 0x80000000u;
constexpr int kTreelet = 128;  // leaves of a subtree that a block's shared memory joins
constexpr int kStack = 64;  // one lane's stack: at most an entry a level (tree_levels) and one more
static_assert(kLbvhUnique >= (int)kPairKeep, "the sink keeps its partners in Lbvh::first");

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;
constexpr uint32_t kScanDirect = 2048;  // tiles

// Internal nodes on the longest path of a tree of n leaves, at most: the common
// prefix grows with every one of them, through the 30 code bits and, between
// equal codes, the bits in which two indices below n can differ (60 at 2^30).
inline int tree_levels(uint32_t n) {
    int bits = 0;
    while (bits < 32 && ((uint64_t)1 << bits) < n) ++bits;
    return 30 + bits;
}

// The number of top nodes, behind the global box.
__host__ __device__ inline uint32_t* top_count(float* bounds) { return reinterpret_cast<uint32_t*>(bounds + 6); }

__device__ __forceinline__ bool box_overlap(float4 alo, float4 ahi, float4 blo, float4 bhi) {
    return blo.x <= ahi.x && alo.x <= bhi.x && blo.y <= ahi.y && alo.y <= bhi.y && blo.z <= ahi.z &&
           alo.z <= bhi.z;
}

// ---------------------------------------------------------------- scan

__global__ void scan_reduce_kernel(const uint32_t* __restrict__ in, uint32_t n, uint32_t* __restrict__ part) {
    stream_wait();
    __shared__ uint32_t ws[33];
    const uint32_t base = blockIdx.x * kScanTile;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t i = base + k * kScanThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    uint32_t total;
    block_exclusive_scan(s, ws, &total);
    if (threadIdx.x == 0) part[blockIdx.x] = total;
}

// One block: exclusive scan of the tile sums; part[nt] = grand total.
__global__ void scan_partials_kernel(uint32_t* __restrict__ part, uint32_t nt, uint32_t* __restrict__ total_out) {
    stream_wait();
    __shared__ uint32_t ws[33];
    uint32_t carry = 0;
    for (uint32_t b = 0; b < nt; b += blockDim.x) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < nt ? part[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan(v, ws, &tot);
        if (i < nt) part[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) *total_out = carry;
}

// SUMS: part holds the tiles' sums as they are; each block adds up those
// before its own (and the first all of them, for the total).
template <bool SUMS>
__global__ void __launch_bounds__(kScanThreads)
scan_apply_kernel(const uint32_t* __restrict__ in, uint32_t n, const uint32_t* __restrict__ part,
                  uint32_t* __restrict__ out) {
    stream_wait();
    __shared__ uint32_t ws[33];
    uint32_t before = 0;
    if constexpr (SUMS) {
        __shared__ uint32_t s_sum;
        const uint32_t nt = gridDim.x, upto = blockIdx.x == 0 ? nt : blockIdx.x;
        if (threadIdx.x == 0) s_sum = 0u;
        uint32_t x = 0;
        for (uint32_t k = threadIdx.x; k < upto; k += kScanThreads) x += part[k];
        __syncthreads();
        x = __reduce_add_sync(0xffffffffu, x);
        if (lane_id() == 0 && x) atomicAdd(&s_sum, x);
        __syncthreads();
        if (blockIdx.x == 0) {
            if (threadIdx.x == 0) out[n] = s_sum;
        } else {
            before = s_sum;
        }
    } else {
        before = part[blockIdx.x];
    }
    const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    const bool vec = base + kScanItems <= n &&
                     ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    uint32_t v[kScanItems];
    uint32_t s = 0;
    if (vec) {
#pragma unroll
        for (int k = 0; k < kScanItems; k += 4) {
            const uint4 x = *reinterpret_cast<const uint4*>(in + base + k);
            v[k] = x.x;
            v[k + 1] = x.y;
            v[k + 2] = x.z;
            v[k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    uint32_t tot;
    uint32_t run = before + block_exclusive_scan(s, ws, &tot);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t x = v[k];
        v[k] = run;
        run += x;
    }
    if (vec) {
#pragma unroll
        for (int k = 0; k < kScanItems; k += 4)
            *reinterpret_cast<uint4*>(out + base + k) = make_uint4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < n) out[base + k] = v[k];
    }
}

// Up to kScanOne words (16-byte aligned): one block, each warp a stretch of
// 128 x kScanRows of them, in one pass over memory.
constexpr int kScanRows = 8;
constexpr uint32_t kScanOne = 32 * 128 * kScanRows;

__global__ void __launch_bounds__(1024) scan_one_kernel(const uint32_t* __restrict__ in, uint32_t n,
                                                        uint32_t* __restrict__ out) {
    stream_wait();
    __shared__ uint32_t ws[33];
    const uint32_t base = (threadIdx.x >> 5) * (128 * kScanRows) + 4 * lane_id();
    uint4 v[kScanRows];
    uint32_t at[kScanRows], sum = 0;
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
        const uint32_t i = base + 128 * r;
        if (i + 4 <= n) {
            v[r] = *reinterpret_cast<const uint4*>(in + i);
        } else {
            v[r].x = i < n ? in[i] : 0u;
            v[r].y = i + 1 < n ? in[i + 1] : 0u;
            v[r].z = i + 2 < n ? in[i + 2] : 0u;
            v[r].w = 0u;
        }
    }
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
        const uint32_t s = v[r].x + v[r].y + v[r].z + v[r].w, inc = warp_inclusive_scan(s);
        at[r] = sum + inc - s;
        sum += __shfl_sync(0xffffffffu, inc, 31);
    }
    uint32_t total;
    uint32_t before = block_exclusive_scan(lane_id() == 0 ? sum : 0u, ws, &total);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (threadIdx.x == 0) out[n] = total;
#pragma unroll
    for (int r = 0; r < kScanRows; ++r) {
        const uint32_t i = base + 128 * r, a = before + at[r], b = a + v[r].x, c = b + v[r].y, d = c + v[r].z;
        if (i + 4 <= n) {
            *reinterpret_cast<uint4*>(out + i) = make_uint4(a, b, c, d);
        } else {
            if (i < n) out[i] = a;
            if (i + 1 < n) out[i + 1] = b;
            if (i + 2 < n) out[i + 2] = c;
        }
    }
}

// ------------------------------------------------------------ bounds

__global__ void bounds_partial_kernel(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n,
                                      float* __restrict__ part) {
    stream_wait();
    __shared__ float s[6][kLbvhThreads];
    float m[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 a = lo[i], b = hi[i];
        m[0] = fminf(m[0], a.x); m[1] = fminf(m[1], a.y); m[2] = fminf(m[2], a.z);
        m[3] = fmaxf(m[3], b.x); m[4] = fmaxf(m[4], b.y); m[5] = fmaxf(m[5], b.z);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) s[k][threadIdx.x] = m[k];
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                s[k][threadIdx.x] = fminf(s[k][threadIdx.x], s[k][threadIdx.x + o]);
                s[k + 3][threadIdx.x] = fmaxf(s[k + 3][threadIdx.x], s[k + 3][threadIdx.x + o]);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x < 6) part[6 * blockIdx.x + threadIdx.x] = s[threadIdx.x][0];
}

// One warp per bound (a thread per bound that reads the partials one after
// the other took 20 us).
__global__ void bounds_final_kernel(const float* __restrict__ part, uint32_t nb, float* __restrict__ bounds) {
    stream_wait();
    const uint32_t k = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    float m = k < 3 ? INFINITY : -INFINITY;
    for (uint32_t b = lane; b < nb; b += 32) m = k < 3 ? fminf(m, part[6 * b + k]) : fmaxf(m, part[6 * b + k]);
    for (int o = 16; o > 0; o >>= 1) {
        const float x = __shfl_xor_sync(0xffffffffu, m, o);
        m = k < 3 ? fminf(m, x) : fmaxf(m, x);
    }
    if (lane == 0) bounds[k] = m;
    if (threadIdx.x == 0) *top_count(bounds) = 0u;
}

// --------------------------------------------------------------- Morton

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
    x &= 0x3ffu;
    x = (x ^ (x << 16)) & 0xff0000ffu;
    x = (x ^ (x << 8)) & 0x0300f00fu;
    x = (x ^ (x << 4)) & 0x030c30c3u;
    x = (x ^ (x << 2)) & 0x09249249u;
    return x;
}

__global__ void morton_kernel(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n,
                              const float* __restrict__ bounds, uint32_t* __restrict__ keys,
                              uint32_t* __restrict__ vals) {
    stream_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = lo[i], b = hi[i];
    const float c[3] = {(a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f};
    uint32_t q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float cen = (bounds[k] + bounds[3 + k]) * 0.5f;
        const float cell = (bounds[3 + k] - bounds[k]) / 1024.0f;
        const float p = cell > 0.0f ? (c[k] - cen) / cell : 0.0f;  // all centroids equal: code 512
        int32_t d = p >= 0.0f ? (int32_t)p : (int32_t)floorf(p);
        d = d < -512 ? -512 : (d > 511 ? 511 : d);
        q[k] = (uint32_t)(d + 512);
    }
    keys[i] = spread10(q[0]) | (spread10(q[1]) << 1) | (spread10(q[2]) << 2);
    vals[i] = i;
}

// ------------------------------------------------------------ radix tree

__device__ __forceinline__ int delta(const uint32_t* __restrict__ k, int n, int i, int j) {
    if (j < 0 || j >= n) return -1;
    const uint32_t a = k[i], b = k[j];
    if (a == b) return 32 + __clz((uint32_t)(i ^ j));
    return __clz(a ^ b);
}

// Karras, "Maximizing Parallelism in the Construction of BVHs, Octrees, and
// k-d Trees" (HPG 2012), Figure 4.  parent[] holds internal nodes at
// [0, n-1) and leaves at [n-1, 2n-1).
__global__ void build_kernel(const uint32_t* __restrict__ keys, int n, int2* __restrict__ children,
                             int32_t* __restrict__ parent, int32_t* __restrict__ other, float4* __restrict__ node_lo,
                             float4* __restrict__ node_hi, uint32_t* __restrict__ top, uint32_t* __restrict__ n_top) {
    stream_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    const int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    const int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int l = 0;
    for (int t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    const int j = i + l * d;
    const int dnode = delta(keys, n, i, j);
    int s = 0, t = l;
    do {
        t = (t + 1) >> 1;
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    const int g = i + s * d + min(d, 0);
    const int lo = min(i, j), hi = max(i, j);
    const int left = lo == g ? (int)(g | kLeaf) : g;
    const int right = hi == g + 1 ? (int)((g + 1) | kLeaf) : g + 1;
    children[i] = make_int2(left, right);
    other[i] = j;
    if (l >= kTreelet) {
        top[atomicAdd(n_top, 1u)] = (uint32_t)i;
        node_lo[i] = node_hi[i] = make_float4(0.f, 0.f, 0.f, 0.f);  // (no key yet)
    }
    if (i == 0) parent[0] = -1;  // the root
    parent[lo == g ? (n - 1) + g : g] = i;
    parent[hi == g + 1 ? (n - 1) + g + 1 : g + 1] = i;
}

__device__ __forceinline__ void red_max(uint32_t* p, uint32_t v) {
    asm volatile("red.relaxed.gpu.global.max.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// A child reference is a leaf below n or an internal node below n - 1.
__device__ __forceinline__ bool child_ok(int c, int n) {
    return (c & kLeaf) ? (c & ~kLeaf) < n : (c >= 0 && c < n - 1);
}

// Bottom-up boxes.  Every node gets a record -- both children's boxes, each
// lower corner's w lane holding the child reference and each upper corner's
// the last leaf below that child -- which the traversal reads in one 64-byte
// piece instead of the children's indices and then their boxes.
//
// Treelets, the largest subtrees of at most kTreelet leaves, are joined in
// shared memory: a block takes those whose first leaf is one of its
// kRefitSpan, so kRefitSpan + kTreelet leaves hold them, and a node, whose
// index is one end of its range, lies there too.  (A treelet across two blocks'
// leaves is joined by both, to the same bits; the one with its first leaf goes
// on with it.)  Its box then rises through the top nodes as atomic maxima,
// which wait for nothing, and stops where it widens nothing: the box that
// holds it there rises itself.  top_kernel writes the top nodes' records.
//
// The chain of dependent loads bounds it: some 9 levels in shared memory, 13
// above at one load each.  With every level through global memory (a fence, an
// atomic that returns, the sibling's box: 1.7 to 2.7 us each) the refit was 41.5
// us at 32,768 leaves and 64 at 300,001; now 13.5 + 7 and 36.6 + 16.8 with cold
// caches, and the pairs of 300,001 boxes 281 us in all against 355.  Treelets
// of 32 and 64 leaves and spans of 192 to 448 are 0 to 5% behind; a block
// joining only what lies within its own 512 leaves gains nothing, as the paths
// along the blocks' edges stay as deep.
constexpr int kRefitSpan = 512;
constexpr int kRefitWindow = kRefitSpan + kTreelet;

struct Corners {
    float v[6];  // lower x, y, z, upper x, y, z
};

__device__ __forceinline__ Corners corners(float4 a, float4 b) { return Corners{{a.x, a.y, a.z, b.x, b.y, b.z}}; }

// Ordered keys that grow as the box does (NaN: 0, no bound).
__device__ __forceinline__ uint32_t bound_key(float x, bool lower) {
    if (x != x) return 0u;
    const uint32_t b = __float_as_uint(x), k = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    return lower ? ~k : k;
}
__device__ __forceinline__ float key_bound(uint32_t k, bool lower) {
    if (lower) k = ~k;
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ void write_record(float4* __restrict__ rec, int p, int2 c, const Corners& a, const Corners& b,
                                             int last) {
    // a left child's last leaf is the index in its own reference (the split)
    rec[4 * (size_t)p + 0] = make_float4(a.v[0], a.v[1], a.v[2], __int_as_float(c.x));
    rec[4 * (size_t)p + 1] = make_float4(a.v[3], a.v[4], a.v[5], __int_as_float(c.x & ~kLeaf));
    rec[4 * (size_t)p + 2] = make_float4(b.v[0], b.v[1], b.v[2], __int_as_float(c.y));
    rec[4 * (size_t)p + 3] = make_float4(b.v[3], b.v[4], b.v[5], __int_as_float(last));
}

__global__ void __launch_bounds__(kRefitWindow)
refit_kernel(int n, const uint32_t* __restrict__ vals, const float4* __restrict__ lo, const float4* __restrict__ hi,
             float4* __restrict__ leaf_lo, float4* __restrict__ leaf_hi, float4* __restrict__ node_lo,
             float4* __restrict__ node_hi, const int2* __restrict__ children, const int32_t* __restrict__ parent,
             const int32_t* __restrict__ other, float4* __restrict__ rec, uint32_t* __restrict__ counts,
             uint32_t* __restrict__ status) {
    stream_wait();
    __shared__ float s_box[2][6][kRefitWindow];  // leaves, nodes
    __shared__ int2 s_children[kRefitWindow];
    __shared__ int s_parent[kRefitWindow], s_other[kRefitWindow];
    __shared__ uint32_t s_visit[kRefitWindow];
    const int t = (int)threadIdx.x, b0 = (int)blockIdx.x * kRefitSpan, k = b0 + t;
    Corners box{};
    int p = -1;
    s_visit[t] = 0u;
    if (k < n) {
        const uint32_t id = vals[k];
        if (n > 1) p = parent[(n - 1) + k];
        if (k < n - 1) {
            s_children[t] = children[k];
            s_parent[t] = parent[k];
            s_other[t] = other[k];
        }
        const float4 a = lo[id], b = hi[id];
        if (t < kRefitSpan) {
            counts[k] = 0u;  // (for the search that follows)
            leaf_lo[k] = a;
            leaf_hi[k] = b;
        }
        box = corners(a, b);
#pragma unroll
        for (int c = 0; c < 6; ++c) s_box[0][c][t] = box.v[c];
    }
    __syncthreads();
    if (k >= n) return;
    int cur = -1, first = k;  // (no node yet: the leaf itself)
    for (int level = 0;; ++level) {
        if (p < 0) return;  // no top: the whole tree is a treelet
        if (level > 2 * kStack || p >= n - 1) {  // a malformed tree: report, never loop or stray
            atomicOr(status, kErrBadInput);
            return;
        }
        const int q = p - b0, e = q >= 0 && q < kRefitWindow ? s_other[q] : other[p];
        const int f = min(p, e), l = max(p, e);
        if (l - f >= kTreelet) break;                       // what this thread holds is a treelet
        if (f < b0 || l >= b0 + kRefitWindow) return;       // a neighbour's
        __threadfence_block();
        if (atomicAdd(&s_visit[q], 1u) == 0u) return;       // the sibling subtree is not done yet
        __threadfence_block();
        const int2 c = s_children[q];
        const int a = (c.x & ~kLeaf) - b0, b = (c.y & ~kLeaf) - b0;
        if (a < 0 || a >= kRefitWindow || b < 0 || b >= kRefitWindow) {
            atomicOr(status, kErrBadInput);
            return;
        }
        Corners x, y;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            x.v[m] = s_box[(c.x & kLeaf) ? 0 : 1][m][a];
            y.v[m] = s_box[(c.y & kLeaf) ? 0 : 1][m][b];
            box.v[m] = m < 3 ? fminf(x.v[m], y.v[m]) : fmaxf(x.v[m], y.v[m]);
            s_box[1][m][q] = box.v[m];
        }
        write_record(rec, p, c, x, y, l);
        cur = p;
        first = f;
        p = s_parent[q];
    }
    if (first < b0 || first >= b0 + kRefitSpan) return;  // a neighbour goes on with it
    if (cur >= 0) {
        node_lo[cur] = make_float4(box.v[0], box.v[1], box.v[2], 0.f);
        node_hi[cur] = make_float4(box.v[3], box.v[4], box.v[5], 0.f);
    }
    uint32_t key[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) key[m] = bound_key(box.v[m], m < 3);
    for (int level = 0; p >= 0; ++level) {
        if (level > 2 * kStack || p >= n - 1) {
            atomicOr(status, kErrBadInput);
            return;
        }
        uint32_t* const wl = reinterpret_cast<uint32_t*>(node_lo + p);
        uint32_t* const wh = reinterpret_cast<uint32_t*>(node_hi + p);
        const uint4 l4 = __ldcg(reinterpret_cast<const uint4*>(wl)), h4 = __ldcg(reinterpret_cast<const uint4*>(wh));
        const int up = parent[p];
        const uint32_t have[6] = {l4.x, l4.y, l4.z, h4.x, h4.y, h4.z};
        bool wider = false;
#pragma unroll
        for (int m = 0; m < 6; ++m)
            if (key[m] > have[m]) {
                red_max((m < 3 ? wl : wh - 3) + m, key[m]);
                wider = true;
            }
        if (!wider) return;
        p = up;
    }
}

__global__ void top_kernel(int n, const uint32_t* __restrict__ top, const uint32_t* __restrict__ n_top,
                           const float4* __restrict__ leaf_lo, const float4* __restrict__ leaf_hi, float4* node_lo,
                           float4* node_hi, const int2* __restrict__ children, const int32_t* __restrict__ other,
                           float4* __restrict__ rec, uint32_t* __restrict__ status) {
    stream_wait();
    const uint32_t m = min(*n_top, (uint32_t)n);
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        const int p = (int)top[i];
        const int2 c = children[p];
        const int e = other[p], first = min(p, e), last = max(p, e);
        if (!child_ok(c.x, n) || !child_ok(c.y, n)) {
            atomicOr(status, kErrBadInput);
            continue;
        }
        Corners box[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int x = h ? c.y : c.x, j = x & ~kLeaf;
            if (x & kLeaf) {
                box[h] = corners(leaf_lo[j], leaf_hi[j]);
                continue;
            }
            const float4 a = node_lo[j], b = node_hi[j];
            box[h] = corners(a, b);
            if ((h ? last - j : j - first) >= kTreelet) {  // a top node itself: keys, cleared for the next refit
#pragma unroll
                for (int w = 0; w < 6; ++w) box[h].v[w] = key_bound(__float_as_uint(box[h].v[w]), w < 3);
                node_lo[j] = node_hi[j] = none;
            }
        }
        if (p == 0) node_lo[0] = node_hi[0] = none;
        write_record(rec, p, c, box[0], box[1], last);
    }
}

// What a traversal does with the pairs it finds.
enum QueryMode {
    kCount,    // each pair once: counts of both boxes (zero before), and their first kLbvhFirst partners
    kWrite,    // partners of body id at [off[id], off[id + 1]), ascending, and self[] of each entry
    kPairs,    // each pair once, into the sink
    kRefill    // each pair once, for the sink's boxes that have more than it kept
};

constexpr int kQueryThreads = 128;

struct QueryOut {
    uint32_t* count;  // per box id, as first: kLbvhFirst words a box
    const uint32_t* off;
    uint32_t* partners;
    uint32_t* self;
    uint64_t cap;
    uint32_t* first;
};

// A pair for the lists of both its boxes.
struct BothWays {
    uint32_t *count, *first;
};
__device__ __forceinline__ void hand_over(const BothWays& s, uint32_t a, uint32_t b) {
    const uint32_t i = atomicAdd(s.count + a, 1u), j = atomicAdd(s.count + b, 1u);
    if (i < (uint32_t)kLbvhFirst) s.first[(size_t)a * kLbvhFirst + i] = b;
    if (j < (uint32_t)kLbvhFirst) s.first[(size_t)b * kLbvhFirst + j] = a;
}

// G lanes walk the tree for one leaf: each takes a node off the leaf's stack,
// reads its record and tests both children's boxes; the lanes' finds are
// pushed or listed together, in lane order.  A walk is some 60 visits, each a
// load that depends on the one before when a thread makes it alone; down the
// tree only one or two nodes are open, near the leaves many.
// Latency bounds it: 300,001 boxes' pairs 99 us with two lanes, 106 with each
// pair handed over as it is found (one lane and both directions of every pair,
// twice: 2 x 100 us).  One warp walking for 32
// neighbouring leaves under their common box took seven times as long: where
// the curve jumps, that box covers much of the domain.
//
// A walk never runs out of stack.  G nodes are taken at a time only from a
// stack of up to `batch` entries, which then has batch + G at most; one node at
// a time adds at most an entry for every level below the node it starts from,
// tree_levels - 1 in all: batch + G + tree_levels - 1 <= kDepth.  (A box over
// small boxes graded toward a corner fills whatever `batch` allows and then
// goes down 40 levels; walks among boxes of like sizes stay below it.)
template <int G>
constexpr int query_depth() { return kStack + 2 * G; }

template <int MODE, int G>
__global__ void __launch_bounds__(kQueryThreads)
query_kernel(int n, int batch, const uint32_t* __restrict__ vals, const float4* __restrict__ leaf_lo,
             const float4* __restrict__ leaf_hi, const float4* __restrict__ rec, QueryOut q, PairSink sink,
             uint32_t* __restrict__ status) {
    stream_wait();
    constexpr bool kUnique = MODE != kWrite;  // each pair once, from the leaf that comes first
    constexpr bool kBuffer = MODE == kPairs || MODE == kCount;
    constexpr int kLeaves = kQueryThreads / G, kDepth = query_depth<G>();
    __shared__ int s_stack[kDepth][kLeaves];
    __shared__ PairBuffer<kBuffer ? 128 : 1> s_found[kQueryThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, sub = threadIdx.x % G, group = lane & ~(uint32_t)(G - 1);
    const uint32_t below = (1u << sub) - 1u;
    const int at = threadIdx.x / G, k = (int)blockIdx.x * kLeaves + at;
    if (MODE == kRefill && !sink_refill(sink)) return;
    PairBuffer<kBuffer ? 128 : 1>& found = s_found[threadIdx.x >> 5];
    if (lane == 0) found.n = 0u;
    if (MODE == kPairs && sub == 0 && k < n) sink.cursor[k] = 0u;
    bool walk = k < n;
    const uint32_t id = walk ? vals[k] : 0u;
    uint32_t c = 0;
    const uint32_t base = MODE == kWrite && walk ? q.off[id] : 0u, lim = MODE == kWrite && walk ? q.off[id + 1] : 0u;
    if constexpr (MODE == kWrite) {
        if (walk && (uint64_t)lim > q.cap) {
            atomicOr(status, kErrPairOverflow);
            walk = false;
        } else if (walk && lim - base <= (uint32_t)kLbvhFirst) {
            // the partners the counting pass kept, each lane placing its share
            // by counting the smaller ones (ids are distinct)
            const uint32_t m = lim - base;
            const uint32_t* list = q.first + (size_t)id * kLbvhFirst;
            for (uint32_t i = sub; i < m; i += G) {
                const uint32_t v = list[i];
                uint32_t r = 0;
                for (uint32_t j = 0; j < m; ++j) r += list[j] < v;
                q.partners[base + r] = v;
                q.self[base + i] = id;
            }
            walk = false;
        }
    }
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 qlo = walk ? leaf_lo[k] : zero, qhi = walk ? leaf_hi[k] : zero;
    int sp = walk && n > 1 ? 1 : 0;
    if (sp && sub == 0) s_stack[0][at] = 0;
    __syncwarp();
    for (int trips = 0; __any_sync(0xffffffffu, sp > 0); ++trips) {
        if (trips > 2 * n + 64) {  // more visits than a tree has nodes: malformed, never loop
            if (lane == 0) atomicOr(status, kErrBadInput);
            break;
        }
        const int m = sp <= batch ? min(sp, G) : 1;
        const bool mine = (int)sub < m;
        const int node = mine ? s_stack[sp - 1 - (int)sub][at] : 0;
        sp -= m;
        __syncwarp();
        float4 r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) r[u] = mine ? __ldg(&rec[4 * (size_t)node + u]) : zero;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float4 blo = r[2 * h], bhi = r[2 * h + 1];
            const int x = __float_as_int(blo.w), j = x & ~kLeaf;
            bool go = mine;
            if (go && !child_ok(x, n)) {
                atomicOr(status, kErrBadInput);
                go = false;
            }
            // (pairs once: only leaves behind this one)
            go = go && box_overlap(qlo, qhi, blo, bhi) && (!kUnique || __float_as_int(bhi.w) > k);
            const bool leaf = go && (x & kLeaf) && j != k, inner = go && !(x & kLeaf);
            const uint32_t mi = (__ballot_sync(0xffffffffu, inner) >> group) & ((1u << G) - 1u);
            if (inner) {
                const int to = sp + __popc(mi & below);
                if (to < kDepth) s_stack[to][at] = x;
                else atomicOr(status, kErrBadInput);  // (no tree of n leaves: see above)
            }
            sp = min(sp + __popc(mi), kDepth);
            if constexpr (kUnique) {
                if (leaf) {
                    if (MODE == kPairs) buffer_pair(found, sink, id, vals[j]);
                    else if (MODE == kCount) buffer_pair(found, BothWays{q.count, q.first}, id, vals[j]);
                    else sink_pair_again(sink, id, vals[j]);
                }
            } else {
                const uint32_t ml = (__ballot_sync(0xffffffffu, leaf) >> group) & ((1u << G) - 1u);
                if (leaf) {
                    const uint32_t to = c + (uint32_t)__popc(ml & below);
                    if (base + to < lim) q.partners[base + to] = vals[j];
                }
                c += (uint32_t)__popc(ml);
            }
        }
        __syncwarp();
    }
    if constexpr (MODE == kPairs) flush_pairs(found, sink, lane, 32u);  // (the warp met at the end of its last trip)
    if constexpr (MODE == kCount) flush_pairs(found, BothWays{q.count, q.first}, lane, 32u);
    if constexpr (MODE == kWrite) {
        __syncwarp();  // (the group's lanes wrote the list)
        if (!walk || sub != 0) return;
        // sort the body's partner list ascending (insertion sort: lists are short)
        for (uint32_t e = base + 1; e < lim; ++e) {
            const uint32_t x = q.partners[e];
            uint32_t m = e;
            while (m > base && q.partners[m - 1] > x) {
                q.partners[m] = q.partners[m - 1];
                --m;
            }
            q.partners[m] = x;
        }
        for (uint32_t e = base; e < lim; ++e) q.self[e] = id;
    }
}

inline uint32_t grid_for(uint64_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

inline uint32_t bounds_blocks(uint32_t n) {
    uint32_t b = grid_for(n, kLbvhThreads);
    return b < 1 ? 1 : (b > 304 ? 304 : b);
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

uint64_t scan_scratch_words(uint32_t n) { return grid_for(n, kScanTile) + 1; }

cudaError_t scan_exclusive_async(const uint32_t* in, uint32_t* out, uint32_t n, uint32_t* scratch,
                                 cudaStream_t st) {
    const uint32_t nt = grid_for(n, kScanTile);
    if (n == 0) return cudaMemsetAsync(out, 0, 4, st);
    // One block up to 32,768 words (5.6 us; three launches of 3 to 4 us and the
    // gaps between them before); up to kScanDirect tiles each block of the second
    // kernel adds up the tiles' sums before it, a launch less; beyond, that
    // would be more reads than the words themselves.
    const bool aligned = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    if (n <= kScanOne && aligned) {
        launch_after(st, 1, 1024, 0, scan_one_kernel, in, n, out);
        return cudaGetLastError();
    }
    launch_after(st, nt, kScanThreads, 0, scan_reduce_kernel, in, n, scratch);
    if (nt <= kScanDirect) {
        launch_after(st, nt, kScanThreads, 0, scan_apply_kernel<true>, in, n, scratch, out);
        return cudaGetLastError();
    }
    launch_after(st, 1, 1024, 0, scan_partials_kernel, scratch, nt, out + n);
    launch_after(st, nt, kScanThreads, 0, scan_apply_kernel<false>, in, n, scratch, out);
    return cudaGetLastError();
}

uint64_t lbvh_scratch_bytes(uint32_t n, int first) {
    const uint64_t m = n ? n : 1;
    size_t b = 0;
    b += 4 * align256(4 * m);                                      // keys, vals, keys_tmp, vals_tmp
    b += align256(4 * sort_scratch_words(m, 30));                  // sort
    b += align256(4 * 8) + align256(4 * 6 * 304);                  // bounds + partials
    b += align256(8 * m) + align256(4 * (2 * m)) + 2 * align256(4 * m);  // children, parent, other, top
    b += 4 * align256(16 * m);                                     // node lo/hi, leaf lo/hi
    b += align256(4 * (m + 1)) + align256(4 * scan_scratch_words((uint32_t)m + 1));
    b += align256(4 * (uint64_t)first * m);                        // first partners per box
    b += align256(64 * m);                                         // node records
    b += align256(4 * 4);                                          // status
    return b;
}

void lbvh_carve(void* scratch, uint32_t n, Lbvh* t, int first) {
    const uint64_t m = n ? n : 1;
    char* p = static_cast<char*>(scratch);
    auto take = [&](size_t bytes) {
        char* r = p;
        p += align256(bytes);
        return r;
    };
    t->n = n;
    t->keys = (uint32_t*)take(4 * m);
    t->vals = (uint32_t*)take(4 * m);
    t->keys_tmp = (uint32_t*)take(4 * m);
    t->vals_tmp = (uint32_t*)take(4 * m);
    t->sort_scratch = (uint32_t*)take(4 * sort_scratch_words(m, 30));
    t->bounds = (float*)take(4 * 8);
    t->bound_part = (float*)take(4 * 6 * 304);
    t->children = (int2*)take(8 * m);
    t->parent = (int32_t*)take(4 * 2 * m);
    t->other = (int32_t*)take(4 * m);
    t->top = (uint32_t*)take(4 * m);
    t->node_lo = (float4*)take(16 * m);
    t->node_hi = (float4*)take(16 * m);
    t->leaf_lo = (float4*)take(16 * m);
    t->leaf_hi = (float4*)take(16 * m);
    t->counts = (uint32_t*)take(4 * (m + 1));
    t->scan_scratch = (uint32_t*)take(4 * scan_scratch_words((uint32_t)m + 1));
    t->first = (uint32_t*)take(4 * (uint64_t)first * m);
    t->rec = (float4*)take(64 * m);
    t->status = (uint32_t*)take(16);
    t->skeys = t->keys;
    t->svals = t->vals;
}

cudaError_t lbvh_morton_async(Lbvh& t, const float4* lo, const float4* hi, cudaStream_t st) {
    const uint32_t n = t.n;
    if (n == 0) return cudaSuccess;
    const uint32_t nb = bounds_blocks(n);
    launch_after(st, nb, kLbvhThreads, 0, bounds_partial_kernel, lo, hi, n, t.bound_part);
    launch_after(st, 1, 6 * 32, 0, bounds_final_kernel, t.bound_part, nb, t.bounds);
    launch_after(st, grid_for(n, kLbvhThreads), kLbvhThreads, 0, morton_kernel, lo, hi, n, t.bounds, t.keys, t.vals);
    return cudaGetLastError();
}

cudaError_t lbvh_build_async(Lbvh& t, const float4* lo, const float4* hi, cudaStream_t st) {
    const uint32_t n = t.n;
    cudaError_t e;
    if (n == 0) return cudaSuccess;
    if ((e = lbvh_morton_async(t, lo, hi, st)) != cudaSuccess) return e;
    bool in_tmp = false;
    if ((e = sort_pairs_async(t.keys, t.vals, t.keys_tmp, t.vals_tmp, n, 30, t.sort_scratch, st, &in_tmp, nullptr,
                              true)) != cudaSuccess)
        return e;
    t.skeys = in_tmp ? t.keys_tmp : t.keys;
    t.svals = in_tmp ? t.vals_tmp : t.vals;
    if (n > 1)
        launch_after(st, grid_for(n - 1, kLbvhThreads), kLbvhThreads, 0, build_kernel, t.skeys, (int)n, t.children,
                     t.parent, t.other, t.node_lo, t.node_hi, t.top, top_count(t.bounds));
    return lbvh_refit_async(t, lo, hi, st);
}

cudaError_t lbvh_refit_async(Lbvh& t, const float4* lo, const float4* hi, cudaStream_t st) {
    const uint32_t n = t.n;
    if (n == 0) return cudaSuccess;
    launch_after(st, grid_for(n, kRefitSpan), kRefitWindow, 0, refit_kernel, (int)n, t.svals, lo, hi, t.leaf_lo,
                 t.leaf_hi, t.node_lo, t.node_hi, t.children, t.parent, t.other, t.rec, t.counts,
                 t.status);
    if (n > (uint32_t)kTreelet)
        launch_after(st, std::min(152u, grid_for(n, kTreelet)), 128, 0, top_kernel, (int)n, t.top,
                     top_count(t.bounds), t.leaf_lo, t.leaf_hi, t.node_lo, t.node_hi, t.children, t.other, t.rec,
                     t.status);
    return cudaGetLastError();
}

static int g_lbvh_rebuild = 16;
void lbvh_set_rebuild_every(int k) { g_lbvh_rebuild = k < 1 ? 1 : k; }
int lbvh_rebuild_every() { return g_lbvh_rebuild; }

// Below this many leaves four lanes walk for one (too few leaves to fill the
// chip with two: 20,000 boxes 186 us the pairs against 198, 32,768 hulls 3144
// us ten steps against 3278), from it two (100,000 boxes 232 against 238,
// 300,001 315 against 336, 2,000,000 1184 against 1425).  One lane is behind
// everywhere (215 us, 249, 367, 1476), and eight too (3202 us the hulls).
constexpr uint32_t kWideLeaves = 1u << 16;

template <int MODE>
static void launch_query(const Lbvh& t, const QueryOut& q, const PairSink& sink, cudaStream_t st) {
    const int n = (int)t.n;
    const auto go = [&](auto kernel, int lanes, int depth) {
        launch_after(st, grid_for(t.n, kQueryThreads / lanes), kQueryThreads, 0, kernel, n,
                     depth - lanes - tree_levels(t.n) + 1, t.svals, t.leaf_lo, t.leaf_hi, t.rec, q, sink, t.status);
    };
    if (t.n < kWideLeaves) go(query_kernel<MODE, 4>, 4, query_depth<4>());
    else go(query_kernel<MODE, 2>, 2, query_depth<2>());
}

cudaError_t lbvh_partners_async(Lbvh& t, uint32_t* off, uint32_t* partners, uint32_t* self, uint64_t cap,
                                cudaStream_t st) {
    const uint32_t n = t.n;
    if (n == 0) return cudaMemsetAsync(off, 0, 4, st);
    const QueryOut q{t.counts, off, partners, self, cap, t.first};
    launch_query<kCount>(t, q, PairSink{}, st);
    cudaError_t e = scan_exclusive_async(t.counts, off, n, t.scan_scratch, st);
    if (e != cudaSuccess) return e;
    launch_query<kWrite>(t, q, PairSink{}, st);
    return cudaGetLastError();
}

cudaError_t lbvh_unique_pairs_async(Lbvh& t, uint32_t* off, unsigned long long* out, uint64_t cap, uint32_t* d_count2,
                                    cudaStream_t st) {
    const uint32_t n = t.n;
    cudaError_t e;
    if (n == 0) return cudaSuccess;
    // t.keys: the codes are used up, the cursors take their place (cleared by the
    // first search, for the second)
    const PairSink sink{t.counts, t.first, t.status + 1, off, t.keys, out, n, cap};
    launch_query<kPairs>(t, QueryOut{}, sink, st);
    if ((e = scan_exclusive_async(t.counts, off, n, t.scan_scratch, st)) != cudaSuccess) return e;
    launch_query<kRefill>(t, QueryOut{}, sink, st);
    launch_after(st, grid_for(n, kLbvhThreads), kLbvhThreads, 0, pairs_write_kernel, sink, d_count2, t.status);
    return cudaGetLastError();
}

}  // namespace sd

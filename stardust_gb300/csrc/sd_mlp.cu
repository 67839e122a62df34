// sd_mlp.cu -- the GJK warm-start network on the 5th-generation tensor
// cores: forward (inference) and backward (training) kernels built from
// tcgen05.mma (BF16 operands in shared memory, FP32 accumulators in tensor
// memory), plus the Adam update.
//
// Network: 16 inputs (12 used, see hull_prev_seed_kernel) -> 64 -> ReLU ->
// 64 -> ReLU -> 16 outputs (3 used), added to inputs 8..10 (the pair's
// previous separating direction, zero for a new pair): a residual network
// whose output is a GJK search direction in the body frame of the pair's
// first hull.  With the last layer at zero it reproduces the previous
// direction; training learns the correction.  Weights are kept in FP32 (master copy, Adam
// moments) and re-packed after every update into BF16 operand images in the
// UMMA canonical K-major layout without swizzle, so a CTA copies them to
// shared memory as-is.
//
// Every GEMM is M = 128 rows (one row per thread of a team of 128 threads,
// which is also the TMEM lane), N in {16, 64}, K in {16, 64, 128}, issued by
// one thread as K/16 tcgen05.mma instructions of kind::f16 and completed
// through tcgen05.commit on an mbarrier.  Weight gradients are GEMMs over the
// samples (K = the 128 rows of a tile) and accumulate in tensor memory across
// the tiles a CTA processes; per-CTA partial sums are reduced in a fixed order.
//
// The weight gradients read the tile's activations where the forward and
// backward GEMMs left them: the core matrices (8 rows of 16 bytes) of a
// K-major 128 x K operand are, with rows and columns exchanged, those of an
// MN-major K x 128 one, so the descriptors alone transpose.  Rows of a product
// that nobody reads hold whatever lies behind an operand.
//
// Training sums in one order whatever runs beside it -- 148 chains of tiles, a
// tile's bias sums row by row, the chains one after the other: a last bit of a
// gradient moves roundings of the BF16 weights some steps later, and near a
// minimum the gradient by 1e-4.  (Taking 304 chains and the bias sums as
// columns of the GEMMs saves 12% more.)
//
// Measured (GB300): 100,003 rows, an Adam step 110 + 10 + 3.5 us (gradient,
// reduction, packing) -> 30 + 5 us with the same bits, the forward pass 24 ->
// 12.  The gradient was bound by 2-byte shared-memory stores and by building
// transposed copies (18 us per tile, one tile at a time); now by a tile's chain
// of five dependent GEMM steps and their epilogues, of which two teams keep two
// in flight, the inputs of the next tile loading behind them.
//
// No counterpart in the reference: the learned warm start is new.
#include "sd_common.cuh"

#include <cuda_bf16.h>

#include <cstddef>

namespace sd {

namespace {

constexpr int kRows = 128;    // tile rows = threads per CTA = TMEM lanes
constexpr int kIn = 16, kHid = 64, kOut = 16;
constexpr uint32_t kMmaSpin = 1u << 22;

// parameter offsets (floats)
constexpr int kW1 = 0, kB1 = kW1 + kHid * kIn, kW2 = kB1 + kHid, kB2 = kW2 + kHid * kHid, kW3 = kB2 + kHid,
              kB3 = kW3 + kOut * kHid, kParams = kB3 + kOut;
static_assert(kParams == 6288, "parameter layout");

// packed BF16 operand images (bytes), canonical K-major layouts
constexpr uint32_t kImgW1 = 0;                       // N 64 x K 16
constexpr uint32_t kImgW2 = kImgW1 + kHid * kIn * 2;  // N 64 x K 64
constexpr uint32_t kImgW3 = kImgW2 + kHid * kHid * 2; // N 16 x K 64
constexpr uint32_t kImgW2T = kImgW3 + kOut * kHid * 2;  // N 64 x K 64 (W2 transposed)
constexpr uint32_t kImgW3T = kImgW2T + kHid * kHid * 2; // N 64 x K 16 (W3 transposed)
constexpr uint32_t kImgBytes = kImgW3T + kHid * kOut * 2;

// Byte offset of element (r, k) of a K-major BF16 operand with K columns:
// 8x8 core matrices of 128 contiguous bytes, K-adjacent cores 128 B apart
// (leading byte offset), 8-row groups (K/8)*128 B apart (stride byte offset).
__host__ __device__ constexpr uint32_t cm_off(uint32_t r, uint32_t k, uint32_t K) {
    return ((r >> 3) * (K >> 3) + (k >> 3)) * 128u + (r & 7u) * 16u + (k & 7u) * 2u;
}

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor (tcgen05): start >> 4, LBO >> 4, SBO >> 4,
// version 1 at bit 46, no swizzle.
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

// Instruction descriptor, kind::f16: D FP32, A and B BF16, both K-major (or
// both MN-major).
__host__ __device__ constexpr uint32_t idesc(uint32_t M, uint32_t N, bool mn_major = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (mn_major ? 3u << 15 : 0u) | ((N >> 3) << 17) | ((M >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(id), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(arrivals) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n .reg .b64 s;\n mbarrier.arrive.shared::cta.b64 s, [%0];\n}" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    for (uint32_t it = 0; it < kMmaSpin; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (it > 64) __nanosleep(32);
    }
    return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(dst)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive FP32 columns of this thread's lane.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

__device__ __forceinline__ uint16_t bf16_bits(float x) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ float bf16_val(uint16_t b) { return __bfloat162float(__ushort_as_bfloat16(b)); }

// Eight values as BF16, the first in the low half of the first word.
__device__ __forceinline__ uint4 pack8(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        w[k] = (uint32_t)bf16_bits(v[2 * k]) | ((uint32_t)bf16_bits(v[2 * k + 1]) << 16);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Byte offset of columns 8c .. 8c + 7 of row r of an operand whose 8-row
// groups are `group` bytes apart: one row of a core matrix.  Core matrices of
// an operand that a CTA builds are kCore = 128 + 16 bytes apart, so that a row's
// columns lie in different banks.
constexpr uint32_t kCore = 144;

__device__ __forceinline__ uint32_t cm_row(uint32_t r, uint32_t c, uint32_t group) {
    return (r >> 3) * group + c * kCore + (r & 7u) * 16u;
}

// Sixteen columns of a row, as two stores.
__device__ __forceinline__ void st_row16(uint8_t* base, uint32_t r, uint32_t c0, uint32_t group, const float* v) {
    *reinterpret_cast<uint4*>(base + cm_row(r, c0 >> 3, group)) = pack8(v);
    *reinterpret_cast<uint4*>(base + cm_row(r, (c0 >> 3) + 1, group)) = pack8(v + 8);
}

// D (tmem columns at d) = A (128 x K, K-major, 8-row groups group_a bytes
// apart) * B (N x K, K-major, packed)^T.
__device__ __forceinline__ void gemm_issue(uint32_t d, const uint8_t* A, uint32_t group_a, const uint8_t* B, uint32_t N,
                                           uint32_t K) {
    const uint32_t id = idesc(kRows, N), group_b = (K >> 3) * 128u;
    for (uint32_t s = 0; s < K / 16; ++s)
        mma_f16(d, sdesc(saddr(A) + s * 2u * kCore, kCore, group_a), sdesc(saddr(B) + s * 256u, 128u, group_b), id,
                s > 0 ? 1u : 0u);
}

// D (tmem columns at d) [+]= A^T B over the tile's 128 rows, A and B stored as
// above: with K the rows, MN-major operands whose 8-element blocks along M or
// N are kCore bytes apart and along K a group apart.  (For MN-major operands
// without swizzle the descriptor's leading offset is the K one.)
__device__ __forceinline__ void gemm_rows_issue(uint32_t d, const uint8_t* A, uint32_t group_a, const uint8_t* B,
                                                uint32_t group_b, uint32_t N, bool accumulate) {
    const uint32_t id = idesc(kRows, N, true);
    for (uint32_t s = 0; s < kRows / 16; ++s)
        mma_f16(d, sdesc(saddr(A) + s * 2u * group_a, group_a, kCore), sdesc(saddr(B) + s * 2u * group_b, group_b, kCore),
                id, (accumulate || s > 0) ? 1u : 0u);
}

// A team: 128 threads of a CTA, with a named barrier of their own, that take a
// tile of 128 rows through the network together (thread = row = TMEM lane).
struct Team {
    uint32_t id, tid;
};
__device__ __forceinline__ void team_sync(const Team& m) {
    asm volatile("barrier.cta.sync %0, 128;" ::"r"(m.id + 1u) : "memory");
}
__device__ __forceinline__ bool team_all(const Team& m, bool mine) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.and.pred q, %2, 128, p;\n selp.u32 %0, 1, 0, q;\n}"
        : "=r"(r)
        : "r"((uint32_t)mine), "r"(m.id + 1u)
        : "memory");
    return r != 0u;
}

// Makes every thread's shared-memory writes and tensor-memory reads visible
// to MMAs that the team's thread 0 issues next.
__device__ __forceinline__ void gemm_ready(const Team& m) {
    fence_async_smem();
    tc_fence_before();
    team_sync(m);
    tc_fence_after();
}

// Waits for thread 0's last commit to bar.  Returns false (and flags) if the
// wait gave up: one verdict for the whole team.
__device__ __forceinline__ bool gemm_wait(const Team& m, uint64_t* bar, uint32_t& phase, uint32_t* status) {
    const bool mine = mbar_wait(bar, phase);
    const bool ok = team_all(m, mine);
    if (ok) phase ^= 1u;
    else atomicOr(status, kErrWaitTimeout);
    tc_fence_after();
    return ok;
}

// One GEMM step: thread 0 issues and commits, the team does `meanwhile` (which
// may read the operands) and waits for the commit.
template <class F>
__device__ __forceinline__ bool gemm_sync(const Team& m, uint32_t d, const uint8_t* A, uint32_t group_a,
                                          const uint8_t* B, uint32_t N, uint32_t K, uint64_t* bar, uint32_t& phase,
                                          uint32_t* status, F&& meanwhile) {
    gemm_ready(m);
    if (m.tid == 0) {
        gemm_issue(d, A, group_a, B, N, K);
        mma_commit(bar);
    }
    meanwhile();
    return gemm_wait(m, bar, phase, status);
}
__device__ __forceinline__ bool gemm_sync(const Team& m, uint32_t d, const uint8_t* A, uint32_t group_a,
                                          const uint8_t* B, uint32_t N, uint32_t K, uint64_t* bar, uint32_t& phase,
                                          uint32_t* status) {
    return gemm_sync(m, d, A, group_a, B, N, K, bar, phase, status, [] {});
}

// Column c of an operand summed over the tile's rows, first to last.
__device__ __forceinline__ float column_sum(const uint8_t* base, uint32_t c, uint32_t group) {
    const uint8_t* p = base + (c >> 3) * kCore + (c & 7u) * 2u;
    float a = 0.0f;
#pragma unroll 4
    for (uint32_t r = 0; r < kRows; r += 8)
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
            a += bf16_val(*reinterpret_cast<const uint16_t*>(p + (r >> 3) * group + k * 16u));
    return a;
}

// After a wait gave up: wait once more (bounded) for the MMAs in flight
// before the caller frees tensor memory.
__device__ __forceinline__ void drain(uint64_t* bar, uint32_t phase) { (void)mbar_wait(bar, phase); }

// The CTA's shared-memory view, aligned to 1 KB (the launch adds 1 KB).
__device__ __forceinline__ uint8_t* aligned_smem(uint8_t* raw) {
    const uint32_t pad = (1024u - (saddr(raw) & 1023u)) & 1023u;
    return raw + pad;
}

// The first BYTES of the operand images, which shared memory holds in the same
// order: all of a thread's loads in flight together (a loop per image took 3 us
// of a training kernel).
template <uint32_t BYTES, uint32_t THREADS>
__device__ __forceinline__ void copy_images(uint8_t* dst, const uint8_t* src) {
    constexpr uint32_t kPieces = BYTES / 16, kEach = (kPieces + THREADS - 1) / THREADS;
    uint4 v[kEach];
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k)
        if (k * THREADS + threadIdx.x < kPieces) v[k] = reinterpret_cast<const uint4*>(src)[k * THREADS + threadIdx.x];
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k)
        if (k * THREADS + threadIdx.x < kPieces) reinterpret_cast<uint4*>(dst)[k * THREADS + threadIdx.x] = v[k];
}

// 8-row groups of the operands a CTA builds: 2 or 8 core matrices.
constexpr uint32_t kGroup16 = 2 * kCore, kGroup64 = 8 * kCore;
constexpr uint32_t kGroups = kRows / 8;

// Sixteen inputs of a row (zeros when not live); vec: feat is 16-byte aligned.
__device__ __forceinline__ void load_row16(const float* __restrict__ feat, uint64_t e, bool live, float* v,
                                           bool vec = true) {
    if (!vec) {
#pragma unroll
        for (int k = 0; k < kIn; ++k) v[k] = live ? __ldg(feat + 16 * e + k) : 0.0f;
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 f = live ? __ldg(reinterpret_cast<const float4*>(feat) + 4 * e + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * k] = f.x;
        v[4 * k + 1] = f.y;
        v[4 * k + 2] = f.z;
        v[4 * k + 3] = f.w;
    }
}

// relu(accumulator + bias) of this thread's row, 64 columns, as the next
// layer's operand.
__device__ __forceinline__ void relu_row64(uint32_t taddr, const float* bias, uint8_t* h, uint32_t group, uint32_t row) {
#pragma unroll
    for (int c = 0; c < kHid; c += 16) {
        float v[16];
        tmem_ld16(taddr + c, v);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = fmaxf(v[k] + bias[c + k], 0.0f);
        st_row16(h, row, c, group, v);
    }
}

// The accumulator where the activation (bf16, this thread's row) is positive,
// else 0, as an operand.
__device__ __forceinline__ void mask_row64(uint32_t taddr, const uint8_t* h, uint32_t group_h, uint8_t* dz, uint32_t row) {
#pragma unroll
    for (int c = 0; c < kHid; c += 16) {
        float v[16];
        tmem_ld16(taddr + c, v);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const uint4 a = *reinterpret_cast<const uint4*>(h + cm_row(row, (c >> 3) + q, group_h));
            const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (!(bf16_val((uint16_t)(w[k >> 1] >> (16 * (k & 1)))) > 0.0f)) v[8 * q + k] = 0.0f;
        }
        st_row16(dz, row, c, kGroup64, v);
    }
}

struct InferSmem {
    // the images W1, W2, W3, as packed
    alignas(1024) uint8_t w1[kHid * kIn * 2];
    alignas(1024) uint8_t w2[kHid * kHid * 2];
    alignas(1024) uint8_t w3[kOut * kHid * 2];
    alignas(1024) uint8_t x[kGroups * kGroup16];
    alignas(1024) uint8_t h1[kGroups * kGroup64];
    alignas(1024) uint8_t h2[kGroups * kGroup64];
    float b[kHid + kHid + kOut];
    uint64_t bar;
    uint32_t tmem;
};

// Forward pass over tiles of 128 rows of feat (16 floats per row).
// MODE 0: seeds[e] = (y0, y1, y2, 1) for rows with the previous-contact flag
//         (feat[7] == 1), else zero; rows e < *d_count.
// MODE 1: out[e] = (y0, y1, y2, 0), rows e < n.
template <int MODE>
__global__ void __launch_bounds__(kRows) mlp_forward_kernel(const uint8_t* __restrict__ img,
                                                           const float* __restrict__ params,
                                                           const float* __restrict__ feat, float4* __restrict__ out,
                                                           const uint32_t* __restrict__ d_count, uint64_t n,
                                                           uint32_t* __restrict__ status) {
    stream_wait();
    extern __shared__ __align__(16) uint8_t smem_raw[];
    InferSmem& S = *reinterpret_cast<InferSmem*>(aligned_smem(smem_raw));
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    const Team team{0u, tid};
    const uint64_t rows = MODE == 0 ? min((uint64_t)*d_count, n) : n;
    const uint64_t tiles = (rows + kRows - 1) / kRows;
    if ((uint64_t)blockIdx.x >= tiles) return;
    float x[kIn];
    load_row16(feat, (uint64_t)blockIdx.x * kRows + tid, (uint64_t)blockIdx.x * kRows + tid < rows, x);
    if (warp == 0) tmem_alloc(&S.tmem, 256);
    copy_images<kImgW2T, kRows>(S.w1, img);
    for (uint32_t i = tid; i < kHid; i += kRows) {
        S.b[i] = params[kB1 + i];
        S.b[kHid + i] = params[kB2 + i];
    }
    if (tid < kOut) S.b[2 * kHid + tid] = params[kB3 + tid];
    if (tid == 0) mbar_init(&S.bar, 1);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = S.tmem;
    const uint32_t lane_base = (warp * 32u) << 16;
    uint32_t phase = 0;
    bool ok = true;
    for (uint64_t t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const uint64_t e = t * kRows + tid, e2 = e + (uint64_t)gridDim.x * kRows;
        const bool live = e < rows;
        const float f7 = x[7], skip[3] = {x[8], x[9], x[10]};
        st_row16(S.x, tid, 0, kGroup16, x);
        load_row16(feat, e2, e2 < rows, x);  // the next tile's, in flight behind this one's
        if (!(ok = gemm_sync(team, tm + 0, S.x, kGroup16, S.w1, kHid, kIn, &S.bar, phase, status))) break;
        relu_row64(tm + lane_base, S.b, S.h1, kGroup64, tid);
        if (!(ok = gemm_sync(team, tm + 64, S.h1, kGroup64, S.w2, kHid, kHid, &S.bar, phase, status))) break;
        relu_row64(tm + lane_base + 64, S.b + kHid, S.h2, kGroup64, tid);
        if (!(ok = gemm_sync(team, tm + 128, S.h2, kGroup64, S.w3, kOut, kHid, &S.bar, phase, status))) break;
        float y[16];
        tmem_ld16(tm + lane_base + 128, y);
        if (live) {
            const float y0 = (y[0] + S.b[2 * kHid]) + skip[0], y1 = (y[1] + S.b[2 * kHid + 1]) + skip[1],
                        y2 = (y[2] + S.b[2 * kHid + 2]) + skip[2];
            if (MODE == 0)
                out[e] = f7 == 1.0f ? make_float4(y0, y1, y2, 1.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
            else
                out[e] = make_float4(y0, y1, y2, 0.f);
        }
        // the next tile's first GEMM step orders these reads before its MMAs
    }
    if (!ok) drain(&S.bar, phase);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tm, 256);
}

// What a team works on.  A weight gradient's MMAs may read up to 1.2 KB behind
// an operand (products that nobody reads).
struct TeamSmem {
    alignas(1024) uint8_t x[kGroups * kGroup16];
    alignas(1024) uint8_t h1[kGroups * kGroup64];
    alignas(1024) uint8_t h2[kGroups * kGroup64];
    alignas(1024) uint8_t dz2[kGroups * kGroup64];
    alignas(1024) uint8_t dz1[kGroups * kGroup64];
    alignas(1024) uint8_t dy[kGroups * kGroup16];
};
struct TrainSmem {
    TeamSmem team[2];
    alignas(1024) uint8_t w1[kHid * kIn * 2];
    alignas(1024) uint8_t w2[kHid * kHid * 2];
    alignas(1024) uint8_t w3[kOut * kHid * 2];
    alignas(1024) uint8_t w2t[kHid * kHid * 2];
    alignas(1024) uint8_t w3t[kHid * kOut * 2];
    float b[kHid + kHid + kOut], gb[kHid + kHid + 4];
    // per team: its GEMM steps, its weight gradients, its bias sums
    uint64_t step[2], grad[2], sums[2];
    uint32_t tmem;
};
static_assert(offsetof(InferSmem, w2) - offsetof(InferSmem, w1) == kImgW2 &&
                  offsetof(InferSmem, w3) - offsetof(InferSmem, w1) == kImgW3 &&
                  offsetof(TrainSmem, w2) - offsetof(TrainSmem, w1) == kImgW2 &&
                  offsetof(TrainSmem, w3) - offsetof(TrainSmem, w1) == kImgW3 &&
                  offsetof(TrainSmem, w2t) - offsetof(TrainSmem, w1) == kImgW2T &&
                  offsetof(TrainSmem, w3t) - offsetof(TrainSmem, w1) == kImgW3T && kImgW1 == 0,
              "shared memory holds the operand images as packed");

// Forward + backward of the cosine loss 1 - y.t/|y| (mean over valid rows)
// for the tiles of this CTA; per-CTA gradient partials to part[cta][6288]
// (none from a CTA without tiles).  tgt rows: (tx, ty, tz, valid).
//
// Two teams take the CTA's tiles in turn, a tile each at a time, so that one's
// MMAs run behind the other's epilogues.  The sums keep the order of one team:
// the weight gradients of a tile are issued once those of the tile before it
// are complete, into the same accumulators, and the bias sums are added in
// tile order.
__global__ void __launch_bounds__(2 * kRows, 1) mlp_train_kernel(const uint8_t* __restrict__ img,
                                                                const float* __restrict__ params,
                                                                const float* __restrict__ feat,
                                                                const float4* __restrict__ tgt, uint32_t n,
                                                                float inv_batch, float* __restrict__ part,
                                                                uint32_t* __restrict__ status,
                                                                const uint32_t* __restrict__ d_count, bool vec) {
    stream_wait();
    extern __shared__ __align__(16) uint8_t smem_raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(aligned_smem(smem_raw));
    const uint32_t warp = threadIdx.x >> 5, me = threadIdx.x / kRows, tid = threadIdx.x % kRows;
    const Team team{me, tid};
    TeamSmem& T = S.team[me];
    if (d_count) n = min(n, *d_count);  // rows: the step's entry count, read on the device
    const uint32_t tiles = (n + kRows - 1) / kRows;
    if (blockIdx.x >= tiles) return;
    const uint32_t turn = 2 * gridDim.x;  // tiles from one of this team's to the next
    uint32_t t = blockIdx.x + me * gridDim.x, e = t * kRows + tid;
    float x[kIn];
    load_row16(feat, e, t < tiles && e < n, x, vec);
    float4 g = t < tiles && e < n ? tgt[e] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (warp == 0) tmem_alloc(&S.tmem, 512);
    copy_images<kImgBytes, 2 * kRows>(S.w1, img);
    if (me == 0 && tid < kHid) {
        S.b[tid] = params[kB1 + tid];
        S.b[kHid + tid] = params[kB2 + tid];
        S.gb[tid] = S.gb[kHid + tid] = 0.0f;
        if (tid < kOut) S.b[2 * kHid + tid] = params[kB3 + tid];
        if (tid < 4) S.gb[2 * kHid + tid] = 0.0f;
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 2; ++k) {
            mbar_init(&S.step[k], 1);
            mbar_init(&S.grad[k], 1);
            mbar_init(&S.sums[k], kHid);
        }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = S.tmem;
    const uint32_t lane_base = ((warp & 3u) * 32u) << 16;
    // tensor-memory columns: a team's forward and activation gradients in 128
    // of its own, the weight gradients, accumulated over tiles, in [256, 352)
    const uint32_t cA = me * 128, cB = cA + 64, cG3 = 256, cG2 = 272, cG1 = 336;
    uint32_t phase = 0, own = 0, other = 0;  // parities: GEMM steps, this team's gradients, the other's
    bool ok = true;
    for (bool first = true; t < tiles; t += turn, first = false) {
        // this team's last weight gradients have read the operands
        if (!first && !(ok = gemm_wait(team, &S.grad[me], own, status))) break;
        const float skip[3] = {x[8], x[9], x[10]};
        const float4 target = g;
        st_row16(T.x, tid, 0, kGroup16, x);
        e += turn * kRows;  // the next tile's rows, in flight behind this one's
        load_row16(feat, e, t + turn < tiles && e < n, x, vec);
        g = t + turn < tiles && e < n ? tgt[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (!(ok = gemm_sync(team, tm + cA, T.x, kGroup16, S.w1, kHid, kIn, &S.step[me], phase, status))) break;
        relu_row64(tm + lane_base + cA, S.b, T.h1, kGroup64, tid);
        if (!(ok = gemm_sync(team, tm + cB, T.h1, kGroup64, S.w2, kHid, kHid, &S.step[me], phase, status))) break;
        relu_row64(tm + lane_base + cB, S.b + kHid, T.h2, kGroup64, tid);
        if (!(ok = gemm_sync(team, tm + cA, T.h2, kGroup64, S.w3, kOut, kHid, &S.step[me], phase, status))) break;
        {
            float y[16];
            tmem_ld16(tm + lane_base + cA, y);
            float d[16] = {};
            if (target.w != 0.0f) {
                const float y0 = (y[0] + S.b[2 * kHid]) + skip[0], y1 = (y[1] + S.b[2 * kHid + 1]) + skip[1],
                            y2 = (y[2] + S.b[2 * kHid + 2]) + skip[2];
                const float nn = sqrtf(((y0 * y0 + y1 * y1) + y2 * y2) + 1e-8f);
                const float c = ((y0 * target.x + y1 * target.y) + y2 * target.z) / nn;
                const float s = -inv_batch / nn;
                d[0] = s * (target.x - c * y0 / nn);
                d[1] = s * (target.y - c * y1 / nn);
                d[2] = s * (target.z - c * y2 / nn);
            }
            st_row16(T.dy, tid, 0, kGroup16, d);
        }
        // dH2 = dY W3  (B = W3^T, N 64 x K 16), then dH1 = dZ2 W2; the bias
        // gradients, sums over the rows, behind the MMAs
        float a1 = 0.0f, a2 = 0.0f, a3 = 0.0f;
        if (!(ok = gemm_sync(team, tm + cB, T.dy, kGroup16, S.w3t, kHid, kOut, &S.step[me], phase, status, [&] {
                  if (tid < 3) a3 = column_sum(T.dy, tid, kGroup16);
              })))
            break;
        mask_row64(tm + lane_base + cB, T.h2, kGroup64, T.dz2, tid);
        if (!(ok = gemm_sync(team, tm + cA, T.dz2, kGroup64, S.w2t, kHid, kHid, &S.step[me], phase, status, [&] {
                  if (tid < kHid) a2 = column_sum(T.dz2, tid, kGroup64);
              })))
            break;
        mask_row64(tm + lane_base + cA, T.h1, kGroup64, T.dz1, tid);
        // weight gradients, K = the tile's rows: dW3^T (j, o) = H2^T dY, dW2
        // (k, j) = dZ2^T H1, dW1 (j, i) = dZ1^T X, after the tile before's.
        // Nobody waits for them before this team's next tile.
        gemm_ready(team);
        const bool chained = !first || me != 0;  // (the CTA's first tile has none before it)
        if (tid == 0) {
            if (chained && !mbar_wait(&S.grad[me ^ 1u], other)) ok = false;
            tc_fence_after();
            if (ok) {
                gemm_rows_issue(tm + cG3, T.h2, kGroup64, T.dy, kGroup16, kOut, chained);
                gemm_rows_issue(tm + cG2, T.dz2, kGroup64, T.h1, kGroup64, kHid, chained);
                gemm_rows_issue(tm + cG1, T.dz1, kGroup64, T.x, kGroup16, kIn, chained);
            }
            mma_commit(&S.grad[me]);
        }
        if (tid < kHid) {
            a1 = column_sum(T.dz1, tid, kGroup64);
            if (chained && !mbar_wait(&S.sums[me ^ 1u], other)) ok = false;
            S.gb[tid] += a1;
            S.gb[kHid + tid] += a2;
            if (tid < 3) S.gb[2 * kHid + tid] += a3;
            mbar_arrive(&S.sums[me]);
        }
        if (chained) other ^= 1u;
        if (!(ok = team_all(team, ok))) {
            if (tid == 0) atomicOr(status, kErrWaitTimeout);
            break;
        }
    }
    const bool ran = blockIdx.x + me * gridDim.x < tiles;
    if (ok && ran) ok = gemm_wait(team, &S.grad[me], own, status);
    const bool mine = ok;
    tc_fence_before();
    ok = __syncthreads_and(ok) != 0;
    tc_fence_after();
    float* P = part + (size_t)blockIdx.x * kParams;
    if (ok) {
        if (threadIdx.x < kHid) {  // lanes 0..63 hold the 64 rows of every weight gradient
            const uint32_t r = tid;
            float v[16];
            tmem_ld16(tm + lane_base + cG3, v);  // dW3^T row j = r
#pragma unroll
            for (int o = 0; o < kOut; ++o) P[kW3 + o * kHid + r] = o < 3 ? v[o] : 0.0f;
#pragma unroll
            for (int c = 0; c < kHid; c += 16) {
                tmem_ld16(tm + lane_base + cG2 + c, v);
#pragma unroll
                for (int k = 0; k < 16; k += 4)
                    *reinterpret_cast<float4*>(P + kW2 + r * kHid + c + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
            }
            tmem_ld16(tm + lane_base + cG1, v);
#pragma unroll
            for (int k = 0; k < 16; k += 4)
                *reinterpret_cast<float4*>(P + kW1 + r * kIn + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
            P[kB1 + r] = S.gb[r];
            P[kB2 + r] = S.gb[kHid + r];
            if (r < kOut) P[kB3 + r] = r < 3 ? S.gb[2 * kHid + r] : 0.0f;
        }
    } else {
        for (uint32_t i = threadIdx.x; i < kParams; i += 2 * kRows) P[i] = 0.0f;
        if (!mine) {
            drain(&S.step[me], phase);
            drain(&S.grad[me], own);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tm, 512);
}

// BF16 operand images of parameter p: W1, W2, W3 and the transposes W2^T, W3^T.
__device__ __forceinline__ void pack_param(uint32_t p, float x, uint8_t* __restrict__ img) {
    const uint16_t b = bf16_bits(x);
    auto put = [&](uint32_t at) { *reinterpret_cast<uint16_t*>(img + at) = b; };
    if (p < (uint32_t)kB1) {  // W1 [n][k]
        put(kImgW1 + cm_off(p / kIn, p % kIn, kIn));
    } else if (p >= (uint32_t)kW2 && p < (uint32_t)kB2) {  // W2 [n][k] and W2^T [n = k_in][k = k_out]
        const uint32_t r = (p - kW2) / kHid, k = (p - kW2) % kHid;
        put(kImgW2 + cm_off(r, k, kHid));
        put(kImgW2T + cm_off(k, r, kHid));
    } else if (p >= (uint32_t)kW3 && p < (uint32_t)kB3) {  // W3 [o][j] and W3^T [j][o]
        const uint32_t o = (p - kW3) / kHid, j = (p - kW3) % kHid;
        put(kImgW3 + cm_off(o, j, kHid));
        put(kImgW3T + cm_off(j, o, kOut));
    }
}

// grad[p] = sum over CTAs of part[c][p] in the CTAs' order, kBatch loads in
// flight at a time (one after the other took 10 us at 148 CTAs).  Then (adam !=
// 0) an Adam step on the master parameters and their operand images (W3, b3
// rows 3..15 stay zero).  CTAs past the rows' tiles wrote no part.
constexpr int kReduceThreads = 32, kBatch = 37;
__global__ void __launch_bounds__(kReduceThreads)
mlp_reduce_kernel(const float* __restrict__ part, uint32_t nparts, uint32_t n, const uint32_t* __restrict__ d_count,
                  float* __restrict__ grad, float* __restrict__ params, float* __restrict__ m1,
                  float* __restrict__ m2, uint8_t* __restrict__ img, int adam, float lr, float c1, float c2) {
    stream_wait();
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (uint32_t)kParams) return;
    if (d_count) n = min(n, *d_count);
    nparts = min(nparts, (n + kRows - 1) / kRows);
    float g = 0.0f;
    uint32_t c = 0;
    for (; c + kBatch <= nparts; c += kBatch) {  // loads together, sums in the CTAs' order
        float v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) v[k] = part[(size_t)(c + k) * kParams + p];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) g += v[k];
    }
    for (; c < nparts; ++c) g += part[(size_t)c * kParams + p];
    const bool dead = (p >= (uint32_t)kW3 && p < (uint32_t)kB3 && (p - kW3) / kHid >= 3) || (p >= (uint32_t)kB3 + 3);
    if (dead) g = 0.0f;
    if (grad) grad[p] = g;
    if (!adam || dead) return;
    const float a = 0.9f * m1[p] + 0.1f * g;
    const float b = 0.999f * m2[p] + 0.001f * (g * g);
    m1[p] = a;
    m2[p] = b;
    const float x = params[p] - lr * (a * c1) / (sqrtf(b * c2) + 1e-8f);
    params[p] = x;
    pack_param(p, x, img);
}

__global__ void mlp_pack_kernel(const float* __restrict__ params, uint8_t* __restrict__ img) {
    stream_wait();
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < (uint32_t)kParams) pack_param(p, params[p], img);
}

inline uint32_t grid_for(uint64_t n, int threads) { return (uint32_t)((n + threads - 1) / threads); }

constexpr uint32_t kMaxTrainCtas = 148;  // partial sums, and so the gradients' bits, go by this

}  // namespace

// Device state: params | m1 | m2 | grad | image | partials | status
uint64_t mlp_state_bytes() {
    return 4ull * kParams * 4 + kImgBytes + 4ull * kParams * kMaxTrainCtas + 256;
}
uint32_t mlp_param_count() { return kParams; }

MlpState mlp_carve(void* base) {
    MlpState s;
    char* p = static_cast<char*>(base);
    s.params = reinterpret_cast<float*>(p);
    s.m1 = s.params + kParams;
    s.m2 = s.m1 + kParams;
    s.grad = s.m2 + kParams;
    s.img = reinterpret_cast<uint8_t*>(s.grad + kParams);
    s.part = reinterpret_cast<float*>(s.img + kImgBytes);
    s.status = reinterpret_cast<uint32_t*>(s.part + (size_t)kParams * kMaxTrainCtas);
    return s;
}

cudaError_t mlp_init_kernels() {
    cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(InferSmem) + 1024);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_forward_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(InferSmem) + 1024);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(TrainSmem) + 1024);
    return e;
}

cudaError_t mlp_set_params_async(MlpState& s, const float* host_params, cudaStream_t st) {
    cudaError_t e = cudaMemcpyAsync(s.params, host_params, 4ull * kParams, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(s.m1, 0, 8ull * kParams, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(s.img, 0, kImgBytes, st);
    if (e != cudaSuccess) return e;
    launch_after(st, grid_for(kParams, 256), 256, 0, mlp_pack_kernel, s.params, s.img);
    return cudaGetLastError();
}

// The dynamic shared memory base is only 16-byte aligned by default; the
// launch asks for 1 KB more and the kernel uses an aligned view.  (The
// __align__ on the extern array gives 1024-byte alignment on sm_90+.)
cudaError_t mlp_forward_async(const MlpState& s, const float* feat, float4* out, const uint32_t* d_count, uint64_t n,
                              bool seeds, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint32_t tiles = grid_for(n, kRows);
    const uint32_t grid = tiles < 304 ? tiles : 304;
    const size_t sm = sizeof(InferSmem) + 1024;
    if (seeds)
        launch_after(st, grid, kRows, sm, mlp_forward_kernel<0>, s.img, s.params, feat, out, d_count, n, s.status);
    else
        launch_after(st, grid, kRows, sm, mlp_forward_kernel<1>, s.img, s.params, feat, out, nullptr, n, s.status);
    return cudaGetLastError();
}

cudaError_t mlp_train_async(MlpState& s, const float* feat, const float4* tgt, uint32_t n, uint32_t n_valid, float lr,
                            uint32_t adam_step, bool update, cudaStream_t st, const uint32_t* d_count) {
    if (n == 0) return cudaSuccess;
    const uint32_t tiles = grid_for(n, kRows);
    const uint32_t ctas = tiles < kMaxTrainCtas ? tiles : kMaxTrainCtas;
    const float inv = n_valid ? 1.0f / (float)n_valid : 0.0f;
    launch_after(st, ctas, 2 * kRows, sizeof(TrainSmem) + 1024, mlp_train_kernel, s.img, s.params, feat, tgt, n, inv,
                 s.part, s.status, d_count, (reinterpret_cast<uintptr_t>(feat) & 15u) == 0);
    const float c1 = update ? (float)(1.0 / (1.0 - std::pow(0.9, (double)adam_step))) : 0.f;
    const float c2 = update ? (float)(1.0 / (1.0 - std::pow(0.999, (double)adam_step))) : 0.f;
    launch_after(st, grid_for(kParams, kReduceThreads), kReduceThreads, 0, mlp_reduce_kernel, s.part, ctas, n, d_count, s.grad,
                 s.params, s.m1, s.m2, s.img, update ? 1 : 0, lr, c1, c2);
    return cudaGetLastError();
}

}  // namespace sd

// sd_common.cuh -- shared device helpers for the stardust-gb300 kernels.
//
// Every kernel in this library is compiled with -fmad=false: each float
// operation rounds once, in the order written, so results are reproducible
// bit-for-bit by the plain-C restatement that the tests compare against.
// Where a fused multiply-add is part of the specification (the reference's
// in-cell offset, sh_collision_detection.cu:66) it is written explicitly
// as __fmaf_rn.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <initializer_list>
#include <utility>

#include "../../include/stardust.h"
#include "sd_internal.h"

namespace sd {

constexpr int kWarp = 32;

// Bounded spin: a wait on another CTA's flag gives up after this many polls
// (with a short back-off), records kErrLookbackTimeout and carries on, so a
// kernel never hangs the GPU.  Far above any legitimate wait (a predecessor
// CTA that is already resident publishes within microseconds).
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & (kWarp - 1); }

// Inclusive warp scan of a u32.
__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t v) {
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane_id() >= (uint32_t)o) v += t;
    }
    return v;
}

// Exclusive scan over the block of one u32 per thread (blockDim.x <= 1024,
// a multiple of 32).  `ws` is shared scratch of >= 33 words.  Returns the
// exclusive prefix; *total receives the block sum.  Contains __syncthreads.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const int nwarps = blockDim.x / kWarp;
    const int w = threadIdx.x / kWarp;
    uint32_t inc = warp_inclusive_scan(v);
    if (lane_id() == kWarp - 1) ws[w] = inc;
    __syncthreads();
    if (w == 0) {
        uint32_t x = lane_id() < (uint32_t)nwarps ? ws[lane_id()] : 0u;
        uint32_t xi = warp_inclusive_scan(x);
        if (lane_id() < (uint32_t)nwarps) ws[lane_id()] = xi - x;
        if (lane_id() == (uint32_t)nwarps - 1) ws[32] = xi;
    }
    __syncthreads();
    uint32_t r = ws[w] + inc - v;
    *total = ws[32];
    __syncthreads();
    return r;
}

// Launches that overlap their predecessor's end.  A kernel launched by
// launch_after() is set up, and its blocks started, while the kernel before it
// in the stream drains; stream_wait(), the first thing it does, returns once
// that kernel is complete and its writes are visible.  No kernel lets its
// successor start any earlier, so blocks never compete.  4.1 us from one small
// kernel to the next in a stream become 1.4 (0.2 us between a graph's nodes:
// a captured launch stays a plain one).
__device__ __forceinline__ void stream_wait() {
    // (a block of its own, so that no load that the compiler takes for
    // invariant is placed before the wait)
    uint32_t wait;
    asm volatile("mov.u32 %0, 1;" : "=r"(wait));
    if (wait) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// launch_chained(): also between the nodes of a graph (0.2 us less each), for
// graphs that the engine captures for itself; launch_after() captures a plain
// launch, as the graph is then a caller's.
template <bool COOPERATIVE = false, class... P, class... A>
inline void launch_chained(cudaStream_t st, dim3 grid, dim3 block, size_t smem, void (*kernel)(P...), A&&... args) {
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = attr;
    c.numAttrs = COOPERATIVE ? 2 : 1;
    cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);  // (an error is the next cudaGetLastError's)
}

template <class... P, class... A>
inline void launch_after(cudaStream_t st, dim3 grid, dim3 block, size_t smem, void (*kernel)(P...), A&&... args) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
        launch_chained(st, grid, block, smem, kernel, std::forward<A>(args)...);
    else
        kernel<<<grid, block, smem, st>>>(std::forward<A>(args)...);
}

// Up to four ranges of words set to zero by one launch of the chain (a memset
// between two kernels ends it: 3 us each); while capturing, memsets, as before.
struct ZeroRange {
    void* p;
    uint64_t words;
};
static __global__ void zero_kernel(ZeroRange a, ZeroRange b, ZeroRange c, ZeroRange d) {
    stream_wait();
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    const ZeroRange r[4] = {a, b, c, d};
#pragma unroll
    for (int k = 0; k < 4; ++k)
        for (uint64_t i = first; i < r[k].words; i += step) static_cast<uint32_t*>(r[k].p)[i] = 0u;
}
static inline cudaError_t zero_async(cudaStream_t st, ZeroRange a, ZeroRange b = {nullptr, 0}, ZeroRange c = {nullptr, 0},
                                     ZeroRange d = {nullptr, 0}) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        uint64_t most = 1;
        for (const ZeroRange& r : {a, b, c, d}) most = r.words > most ? r.words : most;
        const uint64_t blocks = (most + 1023) / 1024;
        launch_chained(st, (unsigned)(blocks < 608 ? blocks : 608), 256, 0, zero_kernel, a, b, c, d);
        return cudaGetLastError();
    }
    for (const ZeroRange& r : {a, b, c, d})
        if (r.words)
            if (cudaError_t e = cudaMemsetAsync(r.p, 0, 4 * r.words, st)) return e;
    return cudaSuccess;
}

}  // namespace sd

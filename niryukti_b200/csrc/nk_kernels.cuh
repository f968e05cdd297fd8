// Device primitives shared by the engine's kernels: CTA geometry, load flavours
// and a deterministic CTA reduction.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace nk {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Streaming loads for single-use matrix data (evict-first), cached loads for
// the gathered vector, which stays resident in L2.
#ifndef NK_STREAM_HINT
#define NK_STREAM_HINT 1 // 1: evict-first loads for matrix entries, 0: default caching
#endif
template <class T> __device__ __forceinline__ T stream_load(const T *p) {
#if NK_STREAM_HINT
    return __ldcs(p);
#else
    return *p;
#endif
}
template <class T> __device__ __forceinline__ T gather_load(const T *p) { return __ldg(p); }

// Exchange between the CTAs of a cooperative grid: an arrival releases the CTA's
// writes (those of its other threads too, after a CTA barrier), and a thread that
// has seen the count acquires them (for its CTA after another CTA barrier).
// Every acquire drops the SM's L1.  Polling with it is cheaper than relaxed polls
// and one fence behind them: 6.6 against 7.3 us a trial of the resident kernel on
// a 2,000 x 5,000 LP.
__device__ __forceinline__ void release_arrival(unsigned *counter) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}
__device__ __forceinline__ unsigned acquire_arrivals(const unsigned *counter) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
    return v;
}

// Deterministic CTA reduction of NV doubles (fixed tree) over a CTA of W
// warps; result in thread 0.
template <int NV, int W = kWarps>
__device__ __forceinline__ void cta_sum(double (&v)[NV], double *smem /* W*NV */) {
#pragma unroll
    for (int t = 0; t < NV; ++t)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            v[t] += __shfl_xor_sync(0xffffffffu, v[t], off);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0)
#pragma unroll
        for (int t = 0; t < NV; ++t)
            smem[w * NV + t] = v[t];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int t = 0; t < NV; ++t) {
            double s = 0;
            for (int i = 0; i < W; ++i)
                s += smem[i * NV + t];
            v[t] = s;
        }
    }
    __syncthreads();
}

} // namespace nk

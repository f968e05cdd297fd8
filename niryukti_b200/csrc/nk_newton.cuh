// BiCGSTAB for the barrier method's Newton systems (cuda_linear_solve,
// src/cuda.cu:1304-1434; caller src/barrier.cpp:280-300).  The optimizer logic
// stays with the reference's barrier.cpp; this solves K x = b on the GPU.
//
// The systems are small (tens of thousands of unknowns, a few entries a row), so
// an iteration is latency: as separate launches (two products, five dots in two
// stages, the vector updates and one-thread scalar steps: 26 of them, and one
// read of the state) it took about 75 us.  One cooperative kernel runs the
// iterations instead.  A thread owns element e of every vector, a CTA 256
// consecutive ones, and the rows of K with them, so a product and its dot need
// no exchange; what is left are five grid barriers an iteration, each with one
// or two reductions: CTA partials, which every CTA adds up for itself in one
// fixed order, and with them forms the step scalars in the reference's
// expressions and order.  Vectors that others gather (y and z) go through L2.
// A call on a saddle point of 24,000 unknowns and 184 k entries, with its uploads
// and allocations: 5.9 ms before, 1.8 ms now (one allocation, too).
//
// A row of more than 32 entries has a warp of the whole grid to itself, before the
// product's elements are formed, for a barrier more a product: left to the warp of
// its element it waits its turn among 32 rows.  Calls with and without the extra
// phase, ms, and as separate launches: 2,000 rows of 800 entries 3.6 / 6.5 / 11.5,
// 24,000 short rows with 64 long ones of 3,000 entries 2.3 / 13.9 / 6.2, 200,000
// with 32 of 25,000 9.5 / 109 / 23, 24,000 rows of 46 entries 3.1 / 3.9 / 8.2.
// From 32 entries on, because a lane then has one at most in the short rows' turns;
// 64 and 128 are no faster (10,000 rows of 100: 2.8, 2.9 and 3.2 ms).
//
// The grid is resident (cooperative launch) and its waits are bounded; a CTA
// that gives up sets NewtonState::fault.
// Included by nk_engine.cu.
#pragma once
#include "nk_common.cuh"
#include "nk_kernels.cuh"
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <vector>

namespace nk {

struct NewtonState {
    double rho, previous, alpha, omega, target;
    int stop;      // 0 running, 1 converged, 2 breakdown, 3 out of time
    int converged; // 1 once a residual met the target
    int fault;     // a wait was given up
};

constexpr int kNewtonLong = 32;          // rows of more entries have a warp each
constexpr int kNewtonChunk = 64;         // iterations of one launch
constexpr int kNewtonMaxPolls = 4 << 20; // seconds: the barrier's bound
constexpr int64_t kNewtonStage = int64_t(1) << 24; // FP64 entries held at a time for FP32 ones

template <class V> struct NewtonView {
    int64_t n;
    const int64_t *ptr, *idx;
    const V *val;
    const int64_t *long_rows; // rows of more than kNewtonLong entries
    int64_t nlong;
    int element_ctas;         // the first CTAs: those that own elements
    const double *rhs, *dinv;
    double *x, *r, *p, *v, *s, *t, *y, *z;
    double *part;   // two sums per CTA, for each of the iteration's barriers in turn
    unsigned *sync; // [0] arrivals, [1] CTAs done; zero between launches
    NewtonState *st;
    double *late;     // nonzero once the launch has run for `budget`
    long long budget; // nanoseconds
    double tolerance;
    int iterations, first; // of this launch; first: form r, rho and the target
};

__device__ __forceinline__ long long clock_ns() {
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Row `base + lane`'s product with x, for the warp's 32 rows: 8, 16 or 32 lanes a
// row (the warp's longest row decides), lane-strided, then a fixed shuffle tree.
// A row's sum is the 32-lane one whatever the width: the other lanes would add
// zeros.  Loads of four turns are in flight together.  A long row's product is 0
// here: newton_long_rows has it.
template <class V>
__device__ __forceinline__ double newton_rows(const NewtonView<V> &K, int64_t base, const double *x) {
    const int lane = threadIdx.x & 31;
    const int64_t row = base + lane, at = K.ptr[row < K.n ? row : K.n],
                  entries = row < K.n ? K.ptr[row + 1] - at : 0;
    const int len = entries > kNewtonLong ? 0 : int(entries);
    const int top = __reduce_max_sync(0xffffffffu, len);
    const int L = top <= 8 ? 8 : top <= 16 ? 16 : 32, per = 32 / L; // lanes a row, rows a turn
    constexpr int U = 4;
    double mine = 0;
    for (int it0 = 0; it0 < L; it0 += U) {
        int64_t j[U], from[U];
        double w[U], acc[U];
        int rest[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = (it0 + u) * per + lane / L, k = lane % L;
            from[u] = __shfl_sync(0xffffffffu, at, q) + k;
            rest[u] = __shfl_sync(0xffffffffu, len, q) - k;
            j[u] = rest[u] > 0 ? K.idx[from[u]] : -1;
            w[u] = rest[u] > 0 ? double(K.val[from[u]]) : 0.;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            acc[u] = j[u] >= 0 ? 0. + w[u] * __ldcg(x + j[u]) : 0.;
        for (int off = L / 2; off > 0; off >>= 1)
#pragma unroll
            for (int u = 0; u < U; ++u)
                acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const double total = __shfl_sync(0xffffffffu, acc[u], (lane % per) * L);
            if (lane / per == it0 + u)
                mine = total;
        }
    }
    return mine;
}

// The long rows' products with x into out, one warp a row over the whole grid:
// lane-strided sums, loads of eight strides in flight, and the tree of newton_rows.
template <class V>
__device__ __forceinline__ void newton_long_rows(const NewtonView<V> &K, const double *x,
                                                 double *out) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = int64_t(gridDim.x) * kWarps;
    for (int64_t q = int64_t(blockIdx.x) * kWarps + (threadIdx.x >> 5); q < K.nlong; q += stride) {
        const int64_t row = K.long_rows[q], end = K.ptr[row + 1];
        constexpr int U = 8;
        double acc = 0;
        for (int64_t k = K.ptr[row] + lane; k < end; k += 32 * U) {
            double w[U], g[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const bool in = k + 32 * u < end;
                w[u] = in ? double(K.val[k + 32 * u]) : 0.;
                g[u] = in ? __ldcg(x + K.idx[k + 32 * u]) : 0.;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (k + 32 * u < end)
                    acc += w[u] * g[u];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0)
            __stcg(out + row, acc);
    }
}

// Grid barrier; false when the wait was given up.  What the CTA wrote before it is
// released, what the others wrote acquired.
template <class V>
__device__ __forceinline__ bool newton_barrier(const NewtonView<V> &K, unsigned *barrier, int *ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        release_arrival(K.sync);
        const unsigned need = ++*barrier * gridDim.x;
        unsigned seen;
        int polls = 0;
        do
            seen = acquire_arrivals(K.sync);
        while (seen < need && ++polls < kNewtonMaxPolls);
        if (seen < need) {
            *ok = 0;
            atomicExch(&K.st->fault, 1);
        }
    }
    __syncthreads();
    return *ok != 0;
}

// Grid-wide sums of (a, b) in every thread: CTA trees, a barrier, and the CTAs'
// sums added by every CTA in one order.  `turn` picks the partials' place.  In
// turn 4, what CTA 0 left at K.late before the barrier comes along in out[2].
template <class V>
__device__ __forceinline__ bool newton_sum(const NewtonView<V> &K, int turn, unsigned *barrier,
                                           double (&ab)[2], double *red, double *out, int *ok) {
    double *part = K.part + size_t(turn) * 2 * gridDim.x;
    cta_sum<2>(ab, red);
    if (threadIdx.x == 0) {
        __stcg(part + 2 * blockIdx.x, ab[0]);
        __stcg(part + 2 * blockIdx.x + 1, ab[1]);
    }
    if (!newton_barrier(K, barrier, ok))
        return false;
    const double late = turn == 4 && threadIdx.x == 0 ? __ldcg(K.late) : 0.;
    ab[0] = ab[1] = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += kThreads) {
        ab[0] += __ldcg(part + 2 * b);
        ab[1] += __ldcg(part + 2 * b + 1);
    }
    cta_sum<2>(ab, red);
    if (threadIdx.x == 0) {
        out[0] = ab[0];
        out[1] = ab[1];
        out[2] = late;
    }
    __syncthreads();
    ab[0] = out[0];
    ab[1] = out[1];
    return true;
}

template <class V>
__global__ void __launch_bounds__(kThreads, 4) newton_kernel(NewtonView<V> K) {
    __shared__ double red[kWarps * 2], sums[3];
    __shared__ unsigned barrier; // thread 0's count
    __shared__ int ok;
    // the CTAs past element_ctas only walk long rows
    const int64_t n = blockIdx.x < K.element_ctas ? K.n : 0,
                  first = int64_t(blockIdx.x) * kThreads + threadIdx.x,
                  stride = int64_t(K.element_ctas) * kThreads;
    const int64_t tops = (n + 31) / 32 * 32; // whole warps for the row products
    // element e of K x; with long rows `out` (v or t) holds theirs
    auto product = [&](int64_t e, const double *x, const double *out) {
        const double short_row = newton_rows(K, e - (threadIdx.x & 31), x);
        return e < n && K.nlong > 0 && K.ptr[e + 1] - K.ptr[e] > kNewtonLong ? __ldcg(out + e)
                                                                           : short_row;
    };
    if (threadIdx.x == 0) {
        barrier = 0;
        ok = 1;
    }
    __syncthreads();
    const long long start = clock_ns();
    double rho, previous = 1, alpha = 1, omega = 1, target;
    int stop = 0, converged = 0, it = 0;
    auto leave = [&] {
        if (threadIdx.x != 0)
            return;
        if (blockIdx.x == 0) {
            K.st->rho = rho;
            K.st->previous = previous;
            K.st->alpha = alpha;
            K.st->omega = omega;
            K.st->target = target;
            K.st->stop = stop;
            K.st->converged = converged;
        }
        if (atomicAdd(K.sync + 1, 1u) == gridDim.x - 1) { // the last CTA out
            K.sync[0] = 0;
            K.sync[1] = 0;
        }
    };
    if (K.first) {
        double ab[2] = {0, 0};
        for (int64_t e = first; e < n; e += stride) {
            const double b = K.rhs[e];
            K.x[e] = K.p[e] = K.v[e] = 0;
            K.r[e] = b;
            ab[0] += b * b;
        }
        if (!newton_sum(K, 0, &barrier, ab, red, sums, &ok))
            return;
        const double norm = sqrt(ab[0]);
        rho = ab[0]; // the shadow residual is rhs too
        target = K.tolerance * (1 + norm);
        converged = norm <= target;
        stop = converged;
    } else {
        rho = K.st->rho;
        previous = K.st->previous;
        alpha = K.st->alpha;
        omega = K.st->omega;
        target = K.st->target;
    }
    for (; !stop && it < K.iterations; ++it) {
        if (!isfinite(rho) || fabs(rho) < 1e-300 || fabs(omega) < 1e-300) {
            stop = 2;
            break;
        }
        const double beta = (rho / previous) * (alpha / omega);
        // p = r + beta p - beta omega v, y = M^-1 p
        for (int64_t e = first; e < n; e += stride) {
            const double p = 1. * K.r[e] + beta * K.p[e] + (-beta * omega) * K.v[e];
            K.p[e] = p;
            __stcg(K.y + e, K.dinv[e] * p);
        }
        if (!newton_barrier(K, &barrier, &ok)) // y is complete
            return;
        if (K.nlong > 0) {
            newton_long_rows(K, K.y, K.v);
            if (!newton_barrier(K, &barrier, &ok))
                return;
        }
        // v = K y, <shadow, v>
        double ab[2] = {0, 0};
        for (int64_t e = first; e < tops; e += stride) {
            const double v = product(e, K.y, K.v);
            if (e < n) {
                K.v[e] = v;
                ab[0] += K.rhs[e] * v;
            }
        }
        if (!newton_sum(K, 1, &barrier, ab, red, sums, &ok))
            return;
        if (!isfinite(ab[0]) || fabs(ab[0]) < 1e-300) {
            stop = 2;
            break;
        }
        alpha = rho / ab[0];
        // s = r - alpha v, z = M^-1 s, <s, s>
        ab[0] = ab[1] = 0;
        for (int64_t e = first; e < n; e += stride) {
            const double v = K.v[e], s = 1. * K.r[e] + (-alpha) * v + 0. * v;
            K.s[e] = s;
            __stcg(K.z + e, K.dinv[e] * s);
            ab[0] += s * s;
        }
        if (!newton_sum(K, 2, &barrier, ab, red, sums, &ok))
            return;
        if (sqrt(ab[0]) <= target) { // converged on s: x = x + alpha y
            for (int64_t e = first; e < n; e += stride) {
                const double y = K.y[e];
                K.x[e] = 1. * K.x[e] + alpha * y + 0. * y;
            }
            converged = 1;
            stop = 1;
            break;
        }
        if (K.nlong > 0) {
            newton_long_rows(K, K.z, K.t);
            if (!newton_barrier(K, &barrier, &ok))
                return;
        }
        // t = K z, <t, t>, <t, s>
        ab[0] = ab[1] = 0;
        for (int64_t e = first; e < tops; e += stride) {
            const double t = product(e, K.z, K.t);
            if (e < n) {
                K.t[e] = t;
                ab[0] += t * t;
                ab[1] += t * K.s[e];
            }
        }
        if (!newton_sum(K, 3, &barrier, ab, red, sums, &ok))
            return;
        if (!isfinite(ab[0]) || ab[0] < 1e-300) {
            stop = 2;
            break;
        }
        omega = ab[1] / ab[0];
        // x = x + alpha y + omega z, r = s - omega t, <r, r> and the next <shadow, r>
        ab[0] = ab[1] = 0;
        for (int64_t e = first; e < n; e += stride) {
            const double t = K.t[e], r = 1. * K.s[e] + (-omega) * t + 0. * t;
            K.x[e] = 1. * K.x[e] + alpha * K.y[e] + omega * K.z[e];
            K.r[e] = r;
            ab[0] += r * r;
            ab[1] += K.rhs[e] * r;
        }
        // CTA 0 looks at the clock for all, since all must stop after the same iteration
        if (blockIdx.x == 0 && threadIdx.x == 0)
            __stcg(K.late, clock_ns() - start >= K.budget ? 1. : 0.);
        if (!newton_sum(K, 4, &barrier, ab, red, sums, &ok))
            return;
        converged = sqrt(ab[0]) <= target;
        stop = converged;
        if (!stop && it + 1 < K.iterations && sums[2] != 0)
            stop = 3;
        previous = rho;
        rho = ab[1];
    }
    leave();
}

// Diagonal right preconditioner of a Newton matrix, 1 / (its scale) per row:
// |K_ii| where the diagonal carries the row; where it does not (a saddle
// point's regularised zero block, |K_ii| < 1e-8 max_j |K_ij|), the diagonal of
// the row's Schur complement, sum_j K_ij^2 / |K_jj| over the other entries.
// Rows with neither keep 1.  Two passes: the diagonals and whether they carry
// their rows (diag: 0 where not), then the scales; each over rows [first, last) or
// a part of the long rows, whose entries val holds.  A thread takes a row; a long
// row (newton_long_*) a warp, which loads 32 entries at a time and adds them in
// the same order, entry by entry.
__device__ __forceinline__ double carrying(double d, double big) {
    return fabs(d) >= 1e-8 * big ? d : 0.;
}
__device__ __forceinline__ double schur_term(double a, int64_t i, int64_t j, const double *diag) {
    return j != i && diag[j] != 0 ? a * a / fabs(diag[j]) : 0.;
}
__device__ __forceinline__ double newton_scale(double d, double schur) {
    return d != 0 ? 1 / fabs(d) : schur > 0 && isfinite(schur) ? 1 / schur : 1.;
}
__global__ void newton_diagonal(int64_t first, int64_t last, const int64_t *__restrict__ ptr,
                                const int64_t *__restrict__ idx, const double *__restrict__ val,
                                double *__restrict__ diag) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = first + int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < last; i += stride) {
        const int64_t b = ptr[i], e = ptr[i + 1];
        if (e - b > kNewtonLong)
            continue;
        double d = 0, big = 0;
        for (int64_t k = b; k < e; ++k) {
            const double a = fabs(val[k]);
            big = big < a ? a : big;
            if (idx[k] == i)
                d += val[k];
        }
        diag[i] = carrying(d, big);
    }
}
__global__ void newton_long_diagonal(int64_t nlong, const int64_t *__restrict__ long_rows,
                                     const int64_t *__restrict__ ptr,
                                     const int64_t *__restrict__ idx,
                                     const double *__restrict__ val, double *__restrict__ diag) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t q = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; q < nlong; q += stride) {
        const int64_t i = long_rows[q], e = ptr[i + 1];
        double d = 0, big = 0;
        for (int64_t k0 = ptr[i]; k0 < e; k0 += 32) {
            const bool in = k0 + lane < e;
            const double v = in ? val[k0 + lane] : 0., a = fabs(v);
            big = big < a ? a : big;
            for (unsigned hits = __ballot_sync(0xffffffffu, in && idx[k0 + lane] == i); hits;
                 hits &= hits - 1)
                d += __shfl_sync(0xffffffffu, v, __ffs(int(hits)) - 1);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const double a = __shfl_xor_sync(0xffffffffu, big, off);
            big = big < a ? a : big;
        }
        if (lane == 0)
            diag[i] = carrying(d, big);
    }
}
__global__ void newton_scales(int64_t first, int64_t last, const int64_t *__restrict__ ptr,
                              const int64_t *__restrict__ idx, const double *__restrict__ val,
                              const double *__restrict__ diag, double *__restrict__ dinv) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = first + int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < last; i += stride) {
        const int64_t b = ptr[i], e = ptr[i + 1];
        double schur = 0;
        if (diag[i] == 0) {
            if (e - b > kNewtonLong)
                continue;
            for (int64_t k = b; k < e; ++k)
                schur += schur_term(val[k], i, idx[k], diag);
        }
        dinv[i] = newton_scale(diag[i], schur);
    }
}
__global__ void newton_long_scales(int64_t nlong, const int64_t *__restrict__ long_rows,
                                   const int64_t *__restrict__ ptr,
                                   const int64_t *__restrict__ idx,
                                   const double *__restrict__ val,
                                   const double *__restrict__ diag, double *__restrict__ dinv) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t q = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; q < nlong; q += stride) {
        const int64_t i = long_rows[q], e = ptr[i + 1];
        if (diag[i] != 0) // newton_scales has it
            continue;
        constexpr int U = 4;
        double schur = 0;
        for (int64_t k0 = ptr[i]; k0 < e; k0 += 32 * U) {
            double term[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int64_t k = k0 + 32 * u + lane;
                term[u] = k < e ? schur_term(val[k], i, idx[k], diag) : 0.;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int l = 0; l < 32; ++l)
                    schur += __shfl_sync(0xffffffffu, term[u], l);
        }
        if (lane == 0)
            dinv[i] = newton_scale(0., schur);
    }
}
__global__ void newton_ones(int64_t n, double *dinv) {
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        dinv[i] = 1;
}

// Solves K x = rhs (K: n x n CSR, host arrays) by BiCGSTAB, right-preconditioned
// by newton_scales when `precondition` (without it, the iteration is the
// reference's one exactly: every scaling is by 1).  The residual r stays the
// unpreconditioned one, so the stopping test is the reference's.  Returns true
// when a residual met the target ((fp32 ? 1e-6 : 1e-10) (1 + |rhs|)) before
// breakdown, the iteration cap (min(20000, 10 n + 100)) or the time limit (looked
// at before every iteration: by the host between launches of kNewtonChunk, by the
// kernel within one); x gets the last iterate either way.  The arguments are
// checked by the caller.
template <class V>
inline bool newton_solve_t(const nk_csr &K, const double *rhs, bool precondition, double time_limit,
                           double *x_out, bool *timed_out) {
    const int64_t n = K.rows, nnz = K.ptr[K.rows];
    constexpr bool fp32 = sizeof(V) == 4;
    *timed_out = false;
    cudaStream_t s = nullptr;
    cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "Newton stream");
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() {
            cudaStreamSynchronize(s);
            cudaStreamDestroy(s);
        }
    } guard_stream{s};
    const size_t nn = size_t(n), nz = size_t(std::max<int64_t>(1, nnz));
    int dev = 0, sms = 148, per = 0;
    cuda_check(cudaGetDevice(&dev), "device");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, newton_kernel<V>, kThreads, 0),
               "Newton occupancy");
    int64_t all_short = -1; // negative while every row is
    for (int64_t i = 0; i < n; ++i)
        all_short &= K.ptr[i + 1] - K.ptr[i] - (kNewtonLong + 1);
    std::vector<int64_t> long_rows;
    for (int64_t i = 0; all_short >= 0 && i < n; ++i)
        if (K.ptr[i + 1] - K.ptr[i] > kNewtonLong)
            long_rows.push_back(i);
    const int64_t nlong = int64_t(long_rows.size()), resident = int64_t(sms) * std::min(4, per);
    // the dots' grouping, and their bits, are those of the CTAs that own elements
    const int element_ctas =
        int(std::max<int64_t>(1, std::min<int64_t>((n + kThreads - 1) / kThreads, resident)));
    const int grid = int(std::max<int64_t>(
        element_ctas, std::min<int64_t>((nlong + kWarps - 1) / kWarps, resident)));
    constexpr size_t kTurns = 5;
    // the FP64 values: all of them, or for FP32 ones as many whole rows at a time as
    // hold kNewtonStage entries (one row at least), to be converted
    std::vector<int64_t> cuts{0};
    int64_t staged = 1;
    while (cuts.back() < n) {
        const int64_t r = cuts.back(), from = K.ptr[r],
                      to = fp32 ? from + std::min(nnz - from, kNewtonStage) : nnz;
        const int64_t fit = std::upper_bound(K.ptr + r, K.ptr + n + 1, to) - K.ptr - 1;
        cuts.push_back(std::max(fit, r + 1));
        staged = std::max(staged, K.ptr[cuts.back()] - from);
    }
    DevParts mem;
    const size_t optr = mem.add<int64_t>(nn + 1), oidx = mem.add<int64_t>(nz),
                 oval = mem.add<double>(size_t(staged)), oval32 = mem.add<float>(fp32 ? nz : 0),
                 olong = mem.add<int64_t>(size_t(nlong)), orhs = mem.add<double>(nn),
                 ovec = mem.add<double>(10 * nn),
                 opart = mem.add<double>(kTurns * 2 * size_t(grid) + 1),
                 ostate = mem.add<NewtonState>(1), osync = mem.add<unsigned>(2);
    mem.alloc();
    int64_t *dptr = mem.at<int64_t>(optr), *didx = mem.at<int64_t>(oidx);
    double *dval = mem.at<double>(oval), *vec = mem.at<double>(ovec);
    auto up = [&](void *d, const void *h, size_t bytes) {
        if (bytes)
            cuda_check(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s), "Newton upload");
    };
    up(dptr, K.ptr, (nn + 1) * 8);
    up(didx, K.index, size_t(nnz) * 8);
    up(mem.at<double>(orhs), rhs, nn * 8);
    int64_t *dlong = mem.at<int64_t>(olong);
    up(dlong, long_rows.data(), size_t(nlong) * 8);
    cuda_check(cudaMemsetAsync(mem.at<unsigned>(osync), 0, 8, s), "Newton counters");
    cuda_check(cudaMemsetAsync(mem.at<NewtonState>(ostate), 0, sizeof(NewtonState), s),
               "Newton state");
    NewtonView<V> v{};
    v.n = n;
    v.ptr = dptr;
    v.idx = didx;
    if constexpr (fp32)
        v.val = mem.at<float>(oval32);
    else
        v.val = dval;
    v.long_rows = dlong;
    v.nlong = nlong;
    v.element_ctas = element_ctas;
    v.rhs = mem.at<double>(orhs);
    double *dinv = vec, *diag = vec + nn;
    v.dinv = dinv;
    double **dst[] = {&v.x, &v.r, &v.p, &v.v, &v.s, &v.t, &v.y, &v.z};
    for (size_t k = 0; k < 8; ++k)
        *dst[k] = vec + (2 + k) * nn;
    v.part = mem.at<double>(opart);
    v.late = v.part + kTurns * 2 * size_t(grid);
    cuda_check(cudaMemsetAsync(v.late, 0, sizeof(double), s), "Newton state");
    v.sync = mem.at<unsigned>(osync);
    v.st = mem.at<NewtonState>(ostate);
    v.tolerance = fp32 ? 1e-6 : 1e-10;
    // Rows [cuts[q], cuts[q + 1]): their FP64 values to the device (unless they are
    // there, being all), then rows(first, last, long rows, their number, values by
    // the entries' own offsets).
    bool uploaded = false;
    auto for_values = [&](auto rows) {
        for (size_t q = 0; q + 1 < cuts.size(); ++q) {
            const int64_t r0 = cuts[q], r1 = cuts[q + 1], k0 = K.ptr[r0], count = K.ptr[r1] - k0;
            if (!uploaded)
                up(dval, K.value + k0, size_t(count) * 8);
            const auto l0 = std::lower_bound(long_rows.begin(), long_rows.end(), r0),
                       l1 = std::lower_bound(l0, long_rows.end(), r1);
            rows(r0, r1, dlong + (l0 - long_rows.begin()), int64_t(l1 - l0), dval - k0);
        }
        uploaded = cuts.size() == 2;
    };
    for_values([&](int64_t r0, int64_t r1, const int64_t *rows, int64_t count, const double *val) {
        if constexpr (fp32)
            if (const int64_t k0 = K.ptr[r0], k1 = K.ptr[r1]; k1 > k0)
                to_float<<<grid_for(k1 - k0), kThreads, 0, s>>>(k1 - k0, val + k0,
                                                               mem.at<float>(oval32) + k0);
        if (!precondition)
            return;
        newton_diagonal<<<grid_for(r1 - r0), kThreads, 0, s>>>(r0, r1, dptr, didx, val, diag);
        if (count)
            newton_long_diagonal<<<grid_for(32 * count), kThreads, 0, s>>>(count, rows, dptr, didx,
                                                                          val, diag);
    });
    if (precondition)
        for_values([&](int64_t r0, int64_t r1, const int64_t *rows, int64_t count,
                       const double *val) {
            newton_scales<<<grid_for(r1 - r0), kThreads, 0, s>>>(r0, r1, dptr, didx, val, diag,
                                                                dinv);
            if (count)
                newton_long_scales<<<grid_for(32 * count), kThreads, 0, s>>>(count, rows, dptr, didx,
                                                                            val, diag, dinv);
        });
    else
        newton_ones<<<grid_for(n), kThreads, 0, s>>>(n, dinv);
    cuda_check(cudaGetLastError(), "Newton preconditioner");
    const int64_t cap = std::min<int64_t>(20000, 10 * n + 100);
    const auto start = std::chrono::steady_clock::now();
    NewtonState h{};
    for (int64_t it = 0; !h.stop && (it < cap || it == 0); it += v.iterations) {
        // a first launch without time forms the target only, and a residual that
        // already meets it still counts
        const double left =
            time_limit -
            std::chrono::duration<double>(std::chrono::steady_clock::now() - start).count();
        const bool late = left <= 0;
        v.budget = left < 1e9 ? (long long)(1e9 * left) : INT64_MAX;
        if (late && it > 0) {
            *timed_out = true;
            break;
        }
        v.first = it == 0;
        v.iterations = late ? 0 : int(std::min<int64_t>(kNewtonChunk, cap - it));
        void *args[] = {&v};
        cuda_check(cudaLaunchCooperativeKernel((const void *)newton_kernel<V>, dim3(unsigned(grid)),
                                               dim3(kThreads), args, 0, s),
                   "Newton iterations");
        cuda_check(cudaMemcpyAsync(&h, v.st, sizeof(h), cudaMemcpyDeviceToHost, s), "Newton state");
        cuda_check(cudaStreamSynchronize(s), "Newton state");
        if (h.fault)
            throw Error(NK_ERR_CUDA, "a wait inside the Newton kernel was given up");
        if (late || h.stop == 3) {
            *timed_out = !h.stop || h.stop == 3;
            break;
        }
    }
    cuda_check(cudaMemcpyAsync(x_out, v.x, nn * 8, cudaMemcpyDeviceToHost, s), "Newton solution");
    cuda_check(cudaStreamSynchronize(s), "Newton solution");
    return h.converged != 0;
}

inline bool newton_solve(const nk_csr &K, const double *rhs, bool fp32, bool precondition,
                         double time_limit, double *x_out, bool *timed_out) {
    return fp32 ? newton_solve_t<float>(K, rhs, precondition, time_limit, x_out, timed_out)
                : newton_solve_t<double>(K, rhs, precondition, time_limit, x_out, timed_out);
}

} // namespace nk

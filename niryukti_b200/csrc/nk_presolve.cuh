// Device side of the reference's GPU presolve (--gpu-presolve):
//   compact_csr      cuda_compact_matrix (src/cuda.cu:953-1032): the CSR of the
//                    kept rows with their kept columns renumbered, entries in
//                    their original order (an exact, integer/byte operation).
//   propagate_bounds cuda_propagate_integer_bounds (src/cuda.cu:448-529,
//                    1033-1135): activity-based bound proposals with directed
//                    rounding, integer columns rounded inward.  Proposals only:
//                    the reference's host replays them with outward-rounded
//                    proofs before any is used.
// Included by nk_engine.cu.
#pragma once
#include "nk_common.cuh"
#include "nk_kernels.cuh"
#include <cub/device/device_scan.cuh>
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

namespace nk {

// One warp per output row: the number of the source row's entries whose column
// is kept (lane-strided over the row, coalesced; a fixed shuffle tree).
__global__ void compact_count(int64_t rows, const int64_t *__restrict__ kept,
                              const int64_t *__restrict__ ptr, const int64_t *__restrict__ index,
                              const int64_t *__restrict__ map, int64_t *__restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const int64_t first = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = first; r < rows; r += stride) {
        const int64_t i = kept[r], b = ptr[i], e = ptr[i + 1];
        int64_t c = 0;
        for (int64_t k = b + lane; k < e; k += 32)
            c += map[index[k]] >= 0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            c += __shfl_xor_sync(0xffffffffu, c, off);
        if (lane == 0)
            counts[r] = c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        counts[rows] = 0; // the exclusive scan over rows + 1 counts ends in the total
}

// One warp per output row: 32 entries at a time, the kept ones are written in
// order at the row's offset (ballot + prefix popcount), so reads and writes
// stay coalesced and the entry order is the source order.
__global__ void compact_scatter(int64_t rows, const int64_t *__restrict__ kept,
                                const int64_t *__restrict__ ptr,
                                const int64_t *__restrict__ index,
                                const double *__restrict__ value,
                                const int64_t *__restrict__ map,
                                const int64_t *__restrict__ out_ptr,
                                int64_t *__restrict__ out_index, double *__restrict__ out_value) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int64_t first = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t stride = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = first; r < rows; r += stride) {
        const int64_t i = kept[r], b = ptr[i], e = ptr[i + 1];
        int64_t dest = out_ptr[r];
        for (int64_t k0 = b; k0 < e; k0 += 32) { // warp-uniform bounds
            const int64_t k = k0 + lane;
            int64_t col = -1;
            double v = 0;
            if (k < e) {
                col = map[index[k]];
                v = value[k];
            }
            const unsigned keep = __ballot_sync(0xffffffffu, col >= 0);
            if (col >= 0) {
                const int64_t at = dest + __popc(keep & below);
                out_index[at] = col;
                out_value[at] = v;
            }
            dest += __popc(keep);
        }
    }
}

// Host driver: uploads the source CSR and the maps, counts, scans, scatters and
// copies the result into the caller's arrays (out_ptr: rows + 1 entries;
// out_index / out_value: `capacity` entries).  Returns the kept entries.  The
// arguments are checked by the caller.
inline int64_t compact_csr(const nk_csr &M, int64_t rows, const int64_t *kept, const int64_t *map,
                           int64_t *out_ptr, int64_t *out_index, double *out_value,
                           int64_t capacity) {
    cudaStream_t s = nullptr;
    cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "compaction stream");
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard_stream{s};
    const int64_t nnz = M.ptr[M.rows];
    size_t temp = 0;
    cuda_check(cub::DeviceScan::ExclusiveSum(nullptr, temp, static_cast<int64_t *>(nullptr),
                                             static_cast<int64_t *>(nullptr), rows + 1, s),
               "compaction scan size");
    // one allocation; the output too (at most `capacity` entries and the source's)
    // where that is 16 MB at most, else in memory of its own once its size is known
    const int64_t most = std::min(nnz, capacity);
    const bool together = most <= int64_t(1) << 20;
    const size_t reserved = together ? size_t(std::max<int64_t>(1, most)) : 0;
    DevParts mem;
    const size_t optr_ = mem.add<int64_t>(size_t(M.rows + 1)), oidx_ = mem.add<int64_t>(size_t(nnz)),
                 oval_ = mem.add<double>(size_t(nnz)), okept_ = mem.add<int64_t>(size_t(rows)),
                 omap_ = mem.add<int64_t>(size_t(M.cols)),
                 ocounts_ = mem.add<int64_t>(size_t(rows + 1)),
                 oout_ = mem.add<int64_t>(size_t(rows + 1)), owork_ = mem.add<unsigned char>(temp),
                 ooidx_ = mem.add<int64_t>(reserved), ooval_ = mem.add<double>(reserved);
    mem.alloc();
    int64_t *dptr = mem.at<int64_t>(optr_), *didx = mem.at<int64_t>(oidx_),
            *dkept = mem.at<int64_t>(okept_), *dmap = mem.at<int64_t>(omap_),
            *counts = mem.at<int64_t>(ocounts_), *optr = mem.at<int64_t>(oout_),
            *oidx = mem.at<int64_t>(ooidx_);
    double *dval = mem.at<double>(oval_), *oval = mem.at<double>(ooval_);
    auto up = [&](void *d, const void *h, size_t bytes) {
        if (bytes)
            cuda_check(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s), "compaction upload");
    };
    up(dptr, M.ptr, size_t(M.rows + 1) * 8);
    up(didx, M.index, size_t(nnz) * 8);
    up(dval, M.value, size_t(nnz) * 8);
    up(dkept, kept, size_t(rows) * 8);
    up(dmap, map, size_t(M.cols) * 8);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = int(std::max<int64_t>(1, std::min<int64_t>((rows + kWarps - 1) / kWarps,
                                                                int64_t(sms) * 8)));
    compact_count<<<grid, kThreads, 0, s>>>(rows, dkept, dptr, didx, dmap, counts);
    cuda_check(cudaGetLastError(), "compaction count");
    cuda_check(cub::DeviceScan::ExclusiveSum(mem.at<unsigned char>(owork_), temp, counts, optr,
                                             rows + 1, s),
               "compaction scan");
    cuda_check(cudaMemcpyAsync(out_ptr, optr, size_t(rows + 1) * 8, cudaMemcpyDeviceToHost, s),
               "compaction offsets");
    cuda_check(cudaStreamSynchronize(s), "compaction offsets");
    const int64_t total = out_ptr[rows];
    if (total > capacity)
        throw Error(NK_ERR_INVALID, "compaction output capacity is too small");
    if (total) {
        DevBuf<int64_t> own_idx(together ? 0 : size_t(total));
        DevBuf<double> own_val(together ? 0 : size_t(total));
        if (!together) {
            oidx = own_idx.p;
            oval = own_val.p;
        }
        compact_scatter<<<grid, kThreads, 0, s>>>(rows, dkept, dptr, didx, dval, dmap, optr, oidx,
                                                  oval);
        cuda_check(cudaGetLastError(), "compaction scatter");
        cuda_check(cudaMemcpyAsync(out_index, oidx, size_t(total) * 8, cudaMemcpyDeviceToHost, s),
                   "compaction indices");
        cuda_check(cudaMemcpyAsync(out_value, oval, size_t(total) * 8, cudaMemcpyDeviceToHost, s),
                   "compaction values");
        cuda_check(cudaStreamSynchronize(s), "compaction completion");
    }
    return total;
}

// ---------------------------------------------------------------- bound propagation
// new = max(new, v) / min(new, v) for doubles, by compare-and-swap: the result
// is the extreme proposal whatever the order the rows arrive in.
__device__ __forceinline__ void propose_lower(double *address, double value) {
    auto *bits = reinterpret_cast<unsigned long long *>(address);
    unsigned long long old = *reinterpret_cast<volatile unsigned long long *>(bits);
    while (value > __longlong_as_double((long long)old)) {
        const unsigned long long seen =
            atomicCAS(bits, old, (unsigned long long)__double_as_longlong(value));
        if (seen == old)
            break;
        old = seen;
    }
}
__device__ __forceinline__ void propose_upper(double *address, double value) {
    auto *bits = reinterpret_cast<unsigned long long *>(address);
    unsigned long long old = *reinterpret_cast<volatile unsigned long long *>(bits);
    while (value < __longlong_as_double((long long)old)) {
        const unsigned long long seen =
            atomicCAS(bits, old, (unsigned long long)__double_as_longlong(value));
        if (seen == old)
            break;
        old = seen;
    }
}

// The least and greatest of an entry's contribution to its row's activity.
__device__ __forceinline__ double term_low(double v, double lb, double ub) {
    return __dmul_rd(v, v > 0 ? lb : ub);
}
__device__ __forceinline__ double term_high(double v, double lb, double ub) {
    return __dmul_ru(v, v > 0 ? ub : lb);
}

// A row's activity range: the finite terms' directed-rounding sums in entry
// order (not split across lanes: the order is part of the result) and how many
// terms are infinite.
struct RowActivity {
    double low = 0, high = 0;
    int low_inf = 0, high_inf = 0;
    __device__ __forceinline__ void add(double lo, double hi) {
        if (isinf(lo))
            ++low_inf;
        else
            low = __dadd_rd(low, lo);
        if (isinf(hi))
            ++high_inf;
        else
            high = __dadd_ru(high, hi);
    }
    __device__ __forceinline__ bool misses(double rlo, double rhi) const {
        return (!low_inf && low > rhi) || (!high_inf && high < rlo);
    }
};

// The bounds that entry v of a row implies on its column j.
__device__ __forceinline__ void propose_entry(double v, int64_t j, const RowActivity &r, double rlo,
                                              double rhi, const int *integer, double lb, double ub,
                                              double *new_lb, double *new_ub) {
    const double end_low = v > 0 ? lb : ub, end_high = v > 0 ? ub : lb;
    const double tl = __dmul_rd(v, end_low), th = __dmul_ru(v, end_high);
    // the rest of the row: removing a term needs the opposite rounding
    const double rest_low = r.low_inf - int(isinf(tl)) ? -INFINITY
                            : isinf(tl)                ? r.low
                                        : __dsub_rd(r.low, __dmul_ru(v, end_low));
    const double rest_high = r.high_inf - int(isinf(th)) ? INFINITY
                             : isinf(th)                 ? r.high
                                         : __dsub_ru(r.high, __dmul_rd(v, end_high));
    double l = -INFINITY, u = INFINITY;
    if (isfinite(rlo) && isfinite(rest_high)) {
        const double num = __dsub_rd(rlo, rest_high);
        if (v > 0)
            l = __ddiv_rd(num, v);
        else
            u = __ddiv_ru(num, v);
    }
    if (isfinite(rhi) && isfinite(rest_low)) {
        const double num = __dsub_ru(rhi, rest_low);
        if (v > 0)
            u = __ddiv_ru(num, v);
        else
            l = __ddiv_rd(num, v);
    }
    const bool whole = integer[j] != 0;
    if (isfinite(l) && (!whole || fabs(l) < 0x1p52))
        propose_lower(new_lb + j, whole ? ceil(l) : l);
    if (isfinite(u) && (!whole || fabs(u) < 0x1p52))
        propose_upper(new_ub + j, whole ? floor(u) : u);
}

// One pass over the rows.  Reads the bounds of the previous pass (lb, ub) and
// proposes into new_lb / new_ub; flags a row whose activity range misses
// [rl, ru].  A thread per row walking its entries twice is two chains of
// dependent, uncoalesced loads; so a warp takes 32 rows together, kPropEntries
// entries at a time: the terms are formed flat, entry by entry, into shared memory,
// a lane adds up its row's in order, and when all are added the proposals are
// formed flat again.  us a pass with a thread per row / so: 20,000 rows of 16
// entries 79 / 47, of 24 entries 103 / 68, 1,000,000 of 24 2,340 / 1,600, 400,000 of
// 60 1,270 / 1,150, 2,000 of 7,250 26,000 / 23,300 (a long row's sum is one chain).
constexpr int kPropWarps = 4, kPropEntries = 640;
__global__ void __launch_bounds__(kPropWarps * 32)
    propagate_rows(int64_t rows, const int64_t *__restrict__ ptr,
                   const int64_t *__restrict__ index, const double *__restrict__ a,
                   const int *__restrict__ integer, const double *__restrict__ lb,
                   const double *__restrict__ ub, const double *__restrict__ rl,
                   const double *__restrict__ ru, double *new_lb, double *new_ub, int *failed) {
    // a term's place is its entry's plus its row's, so that lanes reading rows of
    // one length do not meet in a bank
    __shared__ double lows[kPropWarps][kPropEntries + 32], highs[kPropWarps][kPropEntries + 32];
    __shared__ unsigned char owner[kPropWarps][kPropEntries];
    __shared__ RowActivity activity[kPropWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t groups = (rows + 31) / 32, stride = int64_t(gridDim.x) * kPropWarps;
    for (int64_t g = int64_t(blockIdx.x) * kPropWarps + w; g < groups; g += stride) {
        const int64_t row = 32 * g + lane, base = ptr[32 * g];
        const int64_t b = ptr[row < rows ? row : rows], e = ptr[row < rows ? row + 1 : rows];
        const double rlo = row < rows ? rl[row] : 0., rhi = row < rows ? ru[row] : 0.;
        const int64_t end = __shfl_sync(0xffffffffu, e, 31);
        RowActivity r;
        // the lane's own entries among the n from k0 on, each marked as its row's
        int first = 0, last = 0;
        auto own = [&](int64_t k0, int n) {
            first = int(b < k0 ? 0 : b - k0 < n ? b - k0 : n);
            last = int(e < k0 ? 0 : e - k0 < n ? e - k0 : n);
            for (int k = first; k < last; ++k)
                owner[w][k] = static_cast<unsigned char>(lane);
            __syncwarp();
        };
        for (int64_t k0 = base; k0 < end; k0 += kPropEntries) {
            const int n = int(end - k0 < kPropEntries ? end - k0 : kPropEntries);
            own(k0, n);
            for (int k = lane; k < n; k += 32) {
                const double v = a[k0 + k];
                const int64_t j = index[k0 + k];
                const double l = lb[j], u = ub[j];
                const int at = k + owner[w][k];
                // a zero coefficient has no term, whatever its column's bounds
                lows[w][at] = v != 0 ? term_low(v, l, u) : 0.;
                highs[w][at] = v != 0 ? term_high(v, l, u) : 0.;
            }
            __syncwarp();
#pragma unroll 4
            for (int k = first; k < last; ++k)
                r.add(lows[w][k + lane], highs[w][k + lane]);
            __syncwarp();
        }
        if (row < rows && r.misses(rlo, rhi))
            atomicExch(failed, 1);
        activity[w][lane] = r;
        __syncwarp();
        for (int64_t k0 = base; k0 < end; k0 += kPropEntries) {
            const int n = int(end - k0 < kPropEntries ? end - k0 : kPropEntries);
            if (end - base > kPropEntries) // else the marks still stand
                own(k0, n);
            for (int q0 = 0; q0 < n; q0 += 32) { // whole warps: the bounds come by shuffle
                const int k = q0 + lane, q = k < n ? owner[w][k] : 0;
                const double lo = __shfl_sync(0xffffffffu, rlo, q),
                             hi = __shfl_sync(0xffffffffu, rhi, q);
                if (k < n && a[k0 + k] != 0) {
                    const int64_t j = index[k0 + k];
                    propose_entry(a[k0 + k], j, activity[w][q], lo, hi, integer, lb[j], ub[j],
                                  new_lb, new_ub);
                }
            }
            __syncwarp();
        }
    }
}

// `passes` propagation passes over A (host arrays in, lb / ub updated in
// place).  Returns false when some row's activity range misses its bounds or a
// column's bounds cross.  The arguments are checked by the caller.
inline bool propagate_bounds(const nk_csr &A, const int *integer, const double *rl,
                             const double *ru, double *lb, double *ub, int passes) {
    const int64_t n = A.cols, m = A.rows, nnz = A.ptr[A.rows];
    if (m == 0 || passes == 0)
        return true;
    cudaStream_t s = nullptr;
    cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "propagation stream");
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard_stream{s};
    // one allocation; the bounds of the last pass and of this one lie together
    DevParts mem;
    const size_t optr_ = mem.add<int64_t>(size_t(m + 1)), oidx_ = mem.add<int64_t>(size_t(nnz)),
                 oval_ = mem.add<double>(size_t(nnz)), orl_ = mem.add<double>(2 * size_t(m)),
                 oold_ = mem.add<double>(2 * size_t(n)), onew_ = mem.add<double>(2 * size_t(n)),
                 oint_ = mem.add<int>(size_t(n)), ofail_ = mem.add<int>(1);
    mem.alloc();
    int64_t *dptr = mem.at<int64_t>(optr_), *didx = mem.at<int64_t>(oidx_);
    double *dval = mem.at<double>(oval_), *drl = mem.at<double>(orl_), *dru = drl + m;
    double *olb = mem.at<double>(oold_), *oub = olb + n, *nlb = mem.at<double>(onew_), *nub = nlb + n;
    int *dint = mem.at<int>(oint_), *dfail = mem.at<int>(ofail_);
    auto up = [&](void *d, const void *h, size_t bytes) {
        if (bytes)
            cuda_check(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s), "propagation upload");
    };
    up(dptr, A.ptr, size_t(m + 1) * 8);
    up(didx, A.index, size_t(nnz) * 8);
    up(dval, A.value, size_t(nnz) * 8);
    up(drl, rl, size_t(m) * 8);
    up(dru, ru, size_t(m) * 8);
    up(dint, integer, size_t(n) * sizeof(int));
    up(olb, lb, size_t(n) * 8);
    up(oub, ub, size_t(n) * 8);
    cuda_check(cudaMemcpyAsync(nlb, olb, size_t(n) * 16, cudaMemcpyDeviceToDevice, s),
               "propagation bounds");
    cuda_check(cudaMemsetAsync(dfail, 0, sizeof(int), s), "propagation flag");
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = int(std::max<int64_t>(1, std::min<int64_t>(
        (m + 32 * kPropWarps - 1) / (32 * kPropWarps), int64_t(sms) * 8)));
    for (int pass = 0; pass < passes; ++pass) {
        propagate_rows<<<grid, kPropWarps * 32, 0, s>>>(m, dptr, didx, dval, dint, olb, oub, drl, dru,
                                                        nlb, nub, dfail);
        cuda_check(cudaGetLastError(), "propagation pass");
        if (pass + 1 < passes)
            cuda_check(cudaMemcpyAsync(olb, nlb, size_t(n) * 16, cudaMemcpyDeviceToDevice, s),
                       "propagation bounds");
    }
    int failed = 0;
    cuda_check(cudaMemcpyAsync(&failed, dfail, sizeof(int), cudaMemcpyDeviceToHost, s),
               "propagation flag");
    cuda_check(cudaMemcpyAsync(lb, nlb, size_t(n) * 8, cudaMemcpyDeviceToHost, s),
               "propagation lower");
    cuda_check(cudaMemcpyAsync(ub, nub, size_t(n) * 8, cudaMemcpyDeviceToHost, s),
               "propagation upper");
    cuda_check(cudaStreamSynchronize(s), "propagation completion");
    if (failed)
        return false;
    for (int64_t j = 0; j < n; ++j)
        if (lb[j] > ub[j])
            return false;
    return true;
}

} // namespace nk

// Resident trials: one cooperative launch runs a whole chunk of PDHG trials of a
// small or medium model.
//
// What bounds such a model is latency, not bandwidth.  A 2,000 x 5,000 LP spends
// 16 us a trial in the two fused kernels for 0.6 MB of matrix: a launch each, a
// handful of CTAs, and one lane per row walking its entries in dependent rounds
// of loads.  Here, 6.3 us a trial (30,011 x 60,037 with 360 k entries: 8.4 us
// against 21.6), a persistent grid keeps its rows and columns for all trials:
//   - CTA b owns a contiguous range of SELL chunks of A^T and one of A, of
//     balanced length; the state of their columns and rows stays in its shared
//     memory from trial to trial, and with it, as far as there is room, their
//     bounds and their entries (L1 and L2 hold the rest);
//   - the products of those entries are formed flat, one entry per thread, all
//     gathers in flight at once (through L2: other SMs write the vectors), and
//     land in shared memory; then a lane adds its row's products in CSR order,
//     so a row's sum is the sequential sum of the two-kernel path bit for bit;
//   - y's leading entries -- the longest rows', which the entries of A^T name over
//     and over -- are copied to shared memory once a trial: gathers of a few
//     hot lines by every SM queue up in L2 (a 40,200 x 80,000 block-angular LP
//     with 200 rows of 4,000 entries took 55 us a trial without the copy);
//   - two grid barriers replace the launches of a trial: after the primal part
//     (dx is complete) and after the dual part (y and the step rule's terms are);
//   - the last CTA holds no rows.  It adds the step rule's terms in the order of
//     the two-kernel path (per CTA list of its schedule, then the last CTA's
//     tree), takes the decision and sends it to the others, which meanwhile form
//     the products and row sums with the trial y -- the next iterate unless the
//     trial is rejected.  One reader of the terms, because 147 of them at once
//     queue up in L2: every CTA deciding for itself took 3.4 us of a 9.1 us trial
//     of a 30,011 x 60,037 LP.
// So a trajectory is the same, bit for bit, whichever path runs it -- except with
// column panels (nk_panel.cuh), whose runs of a long row are added in another order:
// those models run resident under fixed and Halpern steps only, which don't amplify
// the rounding.
//
// What is left of a trial is mostly the two barriers (1.2 to 1.4 us each), the
// decision (about 2 us, less what the gathers beside it take) and the gathers,
// one lookup per SM cycle (0.55 ns per entry of a CTA).  512 threads: with 768 or
// 1,024 the registers spill (8.9 us on the 360 k LP).
//
// The barrier is an atomic arrival counter that one thread per CTA polls, each
// arrival a release and each poll an acquire.  (Relaxed polls save up to 0.4 us a
// trial, but then nothing orders what the other CTAs wrote before the reads.)  The
// grid is launched cooperatively, so every CTA is resident; the polls are
// bounded all the same, and a CTA that gives up sets Control::fault, which the
// host turns into an error.
#pragma once
#include "nk_device.cuh"
#include <cuda_runtime.h>
#include <cstdint>

#ifndef NK_RES_THREADS
#define NK_RES_THREADS 512
#endif

namespace nk {

constexpr int kResThreads = NK_RES_THREADS;
constexpr int kResWarps = kResThreads / 32;
constexpr int kResMaxLists = 256;     // CTA lists of the two-kernel schedule
constexpr int kResWords = 5;          // of a decision message
constexpr int kResMaxPolls = 4 << 20; // seconds: the barrier's bound

struct ResidentView {
    const int *own_t, *own_a;   // CTA b owns chunks [own[b], own[b+1]); the last CTA none
    const int *slot_t, *slot_a; // chunk -> its place (list * width + position)
    const int *own_q;           // sparse Q: CTA b owns its rows [own_q[b], own_q[b+1])
    int lists_p, lists_d;       // CTA lists of the two-kernel schedule
    int width_p, width_d;       // their lengths, padded to a multiple of 32 (zero slots)
    double *sum_p;              // dx^2 per chunk, for every other trial in turn
    double *sum_d;              // dy^2 per chunk, then dy * delta per chunk; likewise
    unsigned long long *word;   // the decision message
    double *last_x, *last_y;    // Halpern: the trial points T not yet copied to xa, ya
    // shared memory: entries of the products, of A^T and of A, virtual columns
    // and rows (each the largest CTA's; columns and rows are multiples of 64)
    int products, entries_t, entries_a, cols, rows;
    int hot;   // leading entries of y that a CTA copies for its gathers (a multiple of 32)
    int stage; // what is copied to shared memory: 0 the state, 1 also the bounds, 2 also the entries
    unsigned *sync; // [0] barrier arrivals, [1] CTAs done; zero between launches
    __device__ double *sums_p(int trial) const { return sum_p + (trial & 1) * lists_p * width_p; }
    __device__ double *sums_d(int trial) const {
        return sum_d + (trial & 1) * 2 * lists_d * width_d;
    }
};

// A CTA's dynamic shared memory: the products; y's hot entries; per virtual column x twice, its
// average and (stage 1) c, lb, ub, q, per virtual row y twice, A x twice, y's
// average and (stage 1) rl, ru, and their lengths; two ints per chunk; the
// entries (stage 2).
inline size_t resident_shared_bytes(const ResidentView &R, size_t value_bytes) {
    const size_t cols = size_t(R.cols), rows = size_t(R.rows);
    return (size_t(R.products) + size_t(R.hot) + (R.stage ? 7 : 3) * cols + (R.stage ? 7 : 5) * rows) * 8 +
           (cols + rows) * 4 + (cols + rows) / 32 * 8 +
           (R.stage == 2 ? (size_t(R.entries_t) + size_t(R.entries_a)) * (value_bytes + 4) : 0);
}

// Waits until `need` arrivals have been counted, and acquires what the arrived CTAs
// wrote; false when the wait was given up.
__device__ __forceinline__ bool wait_arrivals(const unsigned *counter, unsigned need, Control *ctl,
                                              int *ok) {
    if (threadIdx.x == 0) {
        int polls = 0;
        unsigned seen;
        do
            seen = acquire_arrivals(counter);
        while (seen < need && ++polls < kResMaxPolls);
        if (seen < need) {
            *ok = 0;
            atomicExch(&ctl->fault, 1);
        }
    }
    __syncthreads();
    return *ok != 0;
}

// The arrivals counted when grid barrier k of a launch (k = 1, 2, ...: two a
// trial) is complete: those of the CTAs that hold rows at each, and the last CTA's
// once a trial from the second on, before its first barrier (see there).
__device__ __forceinline__ unsigned arrivals_at(unsigned k) {
    return k * (gridDim.x - 1) + (k - 1) / 2;
}

// Grid barrier k for a CTA that holds rows; the arrival releases the CTA's writes.
__device__ __forceinline__ bool grid_barrier(unsigned *counter, unsigned k, Control *ctl, int *ok) {
    __syncthreads();
    if (threadIdx.x == 0)
        release_arrival(counter);
    return wait_arrivals(counter, arrivals_at(k), ctl, ok);
}

// src[j], from the copy of its first `hot` entries where it lies there, else
// through L2.
__device__ __forceinline__ double gather_hot(const double *src, unsigned copy, int j, int hot) {
    double v;
    asm("{\n\t"
        ".reg .pred p;\n\t"
        "setp.lt.s32 p, %3, %4;\n\t"
        "@p ld.shared.f64 %0, [%1];\n\t"
        "@!p ld.global.cg.f64 %0, [%2];\n\t"
        "}"
        : "=d"(v)
        : "r"(copy + 8u * unsigned(j)), "l"(src + j), "r"(j), "r"(hot)
        : "memory");
    return v;
}

// prod[e] = value * src[column] of the CTA's `count` entries (column -1: padding,
// which no row reads).  ip and vp point to shared or global memory.  HOT: src's
// first `hot` entries are in shared memory at `copy`.
template <bool HOT, class V>
__device__ __forceinline__ void flat_products(const int32_t *ip, const V *vp, int count,
                                              const double *src, double *prod, const double *copy,
                                              int hot) {
    constexpr int U = 6, T = kResThreads;
    const unsigned at = HOT ? unsigned(__cvta_generic_to_shared(copy)) : 0u;
    for (int e = threadIdx.x; e < count; e += U * T) {
        int j[U]; // all columns before the first gather, all gathers before the first product
        V w[U];
        double g[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e + u * T < count) {
                j[u] = ip[e + u * T];
                w[u] = vp[e + u * T];
            } else
                j[u] = -1;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if constexpr (HOT)
                g[u] = gather_hot(src, at, j[u] >= 0 ? j[u] : 0, hot);
            else
                g[u] = j[u] >= 0 ? __ldcg(src + j[u]) : 0.;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (e + u * T < count)
                prod[e + u * T] = double(w[u]) * g[u];
    }
}

// The real row whose state virtual row `vr` keeps, -1 for none (padding, and the
// segments of a split row but its first).
template <bool SPLIT, class V>
__device__ __forceinline__ int real_row(const Sell<V, int32_t> &M, int vr) {
    if (SPLIT && vr < M.nsv)
        return M.seg[vr].x >= 0 && M.seg[vr].y == vr ? M.seg[vr].x : -1;
    return vr < M.nv ? vr - int(M.nsv) + int(M.nsr) : -1;
}

// acc + the lane's `len` products (32 apart), one by one.
__device__ __forceinline__ double add_products(const double *p, int len, double acc) {
    constexpr int U = 4;
    int k = 0;
    for (; k + U <= len; k += U) {
        double a[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            a[u] = p[(k + u) * 32];
#pragma unroll
        for (int u = 0; u < U; ++u)
            acc = acc + a[u];
    }
    double a[U - 1];
#pragma unroll
    for (int u = 0; u < U - 1; ++u)
        a[u] = k + u < len ? p[(k + u) * 32] : 0.;
#pragma unroll
    for (int u = 0; u < U - 1; ++u)
        if (k + u < len)
            acc = acc + a[u];
    return acc;
}

// The sums of lists q, q + step, ... (L of them, those below `lists`), as
// ordered_slots() adds them: lane-strided, then the shuffle tree (the zero
// padding changes nothing).  Lane 0 gets them.
template <int L>
__device__ __forceinline__ void list_sums(const double *slots, int q, int step, int lists, int width,
                                          double (&s)[L]) {
#pragma unroll
    for (int u = 0; u < L; ++u)
        s[u] = 0;
    for (int k = threadIdx.x & 31; k < width; k += 64) {
        double a[L], b[L]; // two strides in flight
#pragma unroll
        for (int u = 0; u < L; ++u) {
            const double *at = slots + (q + u * step) * width + k;
            a[u] = q + u * step < lists ? __ldcg(at) : 0.;
            b[u] = q + u * step < lists && k + 32 < width ? __ldcg(at + 32) : 0.;
        }
#pragma unroll
        for (int u = 0; u < L; ++u)
            s[u] = s[u] + a[u] + b[u];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int u = 0; u < L; ++u)
            s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
}

// The sums of all lists, by the whole CTA.
__device__ __forceinline__ void all_list_sums(const double *slots, int lists, int width,
                                              double *out) {
    constexpr int L = 4;
    for (int q = threadIdx.x >> 5; q < lists; q += kResWarps * L) {
        double s[L];
        list_sums<L>(slots, q, kResWarps, lists, width, s);
        if ((threadIdx.x & 31) == 0)
#pragma unroll
            for (int u = 0; u < L; ++u)
                if (q + u * kResWarps < lists)
                    out[q + u * kResWarps] = s[u];
    }
}

// A decision as kResWords words, each 32 bits of it beside the trial's tag, so
// that a word is its own flag: the new factor, the averaging weight, and whether
// the trial was accepted (bit 0) and a restart requested (bit 1).
__device__ __forceinline__ unsigned long long decision_word(const Control &c, int k, unsigned tag) {
    const unsigned long long f = (unsigned long long)__double_as_longlong(c.factor),
                             w = (unsigned long long)__double_as_longlong(c.weight);
    const unsigned half = k == 0   ? unsigned(f)
                          : k == 1 ? unsigned(f >> 32)
                          : k == 2 ? unsigned(w)
                          : k == 3 ? unsigned(w >> 32)
                                   : (c.accept != 0 ? 1u : 0u) | (c.restart != 0 ? 2u : 0u);
    return (unsigned long long)half << 32 | tag;
}

// The last CTA: the step rule of every trial.  Warp 0 keeps the control state in
// registers, the same in every lane: the decision is a serial chain, and each of
// its links would otherwise pass through shared memory.
template <bool HALPERN>
__device__ __forceinline__ void resident_decider(const ResidentView &R, Vecs &v, Control &c, int &ok,
                                                 int trials, unsigned tag) {
    __shared__ double list_p[kResMaxLists], list_d[2 * kResMaxLists], tree[3][kResMaxLists / 32];
    __shared__ double powers[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool adaptive = (c.flags & 1) != 0;
    const int top = R.lists_p > R.lists_d ? R.lists_p : R.lists_d;
    const int rows = (top + 31) / 32; // warps of the two-kernel path's last CTA that hold a term
    Control s = c;
    int t = 0;
    for (; t < trials && c.restart == 0; ++t) {
        if (adaptive && warp == kResWarps - 1 && lane < 2)
            powers[lane] = pow(c.accepted + 2, lane ? -.6 : -.3);
        if (!wait_arrivals(R.sync, arrivals_at(2u * unsigned(t) + 1u), v.ctl, &ok)) // dx^2
            return;
        all_list_sums(R.sums_p(t), R.lists_p, R.width_p, list_p);
        if (!wait_arrivals(R.sync, arrivals_at(2u * unsigned(t) + 2u), v.ctl, &ok)) // dy^2, dy * delta
            return;
        all_list_sums(R.sums_d(t), 2 * R.lists_d, R.width_d, list_d);
        __syncthreads();
        if (warp < rows) {
            const int b = warp * 32 + lane;
            double w[3] = {b < R.lists_p ? list_p[b] : 0., b < R.lists_d ? list_d[b] : 0.,
                           b < R.lists_d ? list_d[R.lists_d + b] : 0.};
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    w[k] += __shfl_xor_sync(0xffffffffu, w[k], off);
            if (lane < 3)
                tree[lane][warp] = lane == 0 ? w[0] : lane == 1 ? w[1] : w[2];
        }
        __syncthreads();
        if (warp == 0) {
            double sum[3] = {0, 0, 0};
            for (int w = 0; w < rows; ++w)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    sum[k] += tree[k][w];
            // lane 0: p / tau, lane 1: d / sigma, lane 2: the averaging weight
            const double num = lane == 0 ? sum[0] : lane == 1 ? sum[1] : s.factor;
            const double den = lane == 0   ? s.tau * s.factor
                               : lane == 1 ? s.sigma * s.factor
                                           : s.mass + s.factor;
            const double q = num / den;
            const double energy =
                __shfl_sync(0xffffffffu, q, 0) + __shfl_sync(0xffffffffu, q, 1);
            decide<HALPERN>(s, energy, sum[2], __shfl_sync(0xffffffffu, q, 2), powers[0], powers[1]);
            if (HALPERN && s.accept != 0)
                s.cur ^= 1; // the trial buffers hold the committed point
            if (lane < kResWords)
                asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(R.word + lane),
                             "l"(decision_word(s, lane, tag + unsigned(t)))
                             : "memory");
            if (lane == 0) {
                c.accepted = s.accepted;
                c.restart = s.restart;
            }
        }
        __syncthreads();
        // The terms of this trial are read: if another follows, its first barrier
        // waits for this arrival, and the trial after it overwrites them.  (The
        // decision words need no release: nothing that others wrote is read on
        // their account.)
        if (threadIdx.x == 0 && t + 1 < trials && c.restart == 0)
            release_arrival(R.sync);
    }
    if (threadIdx.x == 0) {
        if (t < trials) // a requested Halpern restart froze the rest
            s.accept = 0;
        s.arrive = 0;
        store_control(v.ctl, s);
    }
}

// Counts the CTA out; the last one clears the counters for the next launch.
__device__ __forceinline__ void resident_leave(const ResidentView &R) {
    if (threadIdx.x == 0 && atomicAdd(R.sync + 1, 1u) == gridDim.x - 1) {
        R.sync[0] = 0;
        R.sync[1] = 0;
    }
}

// QP: with a sparse Q, whose product with the trial x is formed in the dual part,
// beside A dx, and is the next trial's Q x unless the trial is rejected.
template <class V, bool SPLIT, bool HALPERN, bool QP>
__global__ void __launch_bounds__(kResThreads, 1)
    resident_kernel(Sell<V, int32_t> At, Sell<V, int32_t> A, QCsr<V, int32_t> Q, Vecs v,
                    ResidentView R, int trials, unsigned tag) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ double wpart[SPLIT ? kResWarps : 1][32];
    __shared__ Control c;
    __shared__ int ok;
    if (threadIdx.x == 0) {
        c = *v.ctl;
        ok = 1;
    }
    __syncthreads();
    if (c.fault) // an earlier launch gave up a wait: its counters are no longer whole
        return;
    if (blockIdx.x == gridDim.x - 1) {
        resident_decider<HALPERN>(R, v, c, ok, trials, tag);
        resident_leave(R);
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = R.own_t[blockIdx.x], nt = R.own_t[blockIdx.x + 1] - t0;
    const int a0 = R.own_a[blockIdx.x], na = R.own_a[blockIdx.x + 1] - a0;
    const int64_t tbase = At.cptr[t0], abase = A.cptr[a0];
    const int tcount = int(At.cptr[t0 + nt] - tbase), acount = int(A.cptr[a0 + na] - abase);
    double *prod = reinterpret_cast<double *>(dyn_smem);
    const int first_t = t0 * 32 - int(At.nsv) + int(At.nsr); // real column of local column 0
    const int first_a = a0 * 32 - int(A.nsv) + int(A.nsr);
    // columns: x twice (the iterate's buffer by cur), its average; rows: y twice,
    // A x twice, y's average
    double *hot = prod + R.products, *sx = hot + R.hot, *sxa = sx + 2 * R.cols, *sy = sxa + R.cols,
           *sax = sy + 2 * R.rows, *sya = sax + 2 * R.rows, *bounds = sya + R.rows;
    // the bounds by local row, or (unstaged) from the global arrays by j - first_t
    // and i - first_a, which is the local row outside the split region
    const bool staged = R.stage != 0;
    const double *bc = staged ? bounds : v.c + first_t,
                 *blb = staged ? bounds + R.cols : v.lb + first_t,
                 *bub = staged ? bounds + 2 * R.cols : v.ub + first_t,
                 *bq = staged ? bounds + 3 * R.cols : v.q ? v.q + first_t : nullptr,
                 *brl = staged ? bounds + 4 * R.cols : v.rl + first_a,
                 *bru = staged ? bounds + 4 * R.cols + R.rows : v.ru + first_a;
    int *len_t = reinterpret_cast<int *>(staged ? bounds + 4 * R.cols + 2 * R.rows : bounds),
        *len_a = len_t + R.cols;
    // per chunk: its first entry among the CTA's, and its slot
    int *at_t = len_a + R.rows, *slot_t = at_t + R.cols / 32, *at_a = slot_t + R.cols / 32,
        *slot_a = at_a + R.rows / 32;
    const int32_t *ip_t = At.idx + tbase, *ip_a = A.idx + abase;
    const V *vp_t = At.val + tbase, *vp_a = A.val + abase;
    if (R.stage == 2) {
        V *wt = reinterpret_cast<V *>(slot_a + R.rows / 32), *wa = wt + R.entries_t;
        int32_t *jt = reinterpret_cast<int32_t *>(wa + R.entries_a), *ja = jt + R.entries_t;
        for (int e = threadIdx.x; e < tcount; e += kResThreads) {
            wt[e] = vp_t[e];
            jt[e] = ip_t[e];
        }
        for (int e = threadIdx.x; e < acount; e += kResThreads) {
            wa[e] = vp_a[e];
            ja[e] = ip_a[e];
        }
        ip_t = jt;
        vp_t = wt;
        ip_a = ja;
        vp_a = wa;
    }
    __syncthreads(); // the staged entries
    const double r = v.reflection;
    // the products of A^T with y
    auto products_t = [&](const double *y) {
        if (R.hot == 0) {
            flat_products<false>(ip_t, vp_t, tcount, y, prod, nullptr, 0);
            return;
        }
        for (int k = threadIdx.x; k < R.hot; k += kResThreads)
            hot[k] = __ldcg(y + k);
        __syncthreads();
        flat_products<true>(ip_t, vp_t, tcount, y, prod, hot, R.hot);
    };
    {
        const double *x = c.cur ? v.x1 : v.x0, *y = c.cur ? v.y1 : v.y0,
                     *ax = c.cur ? v.ax1 : v.ax0;
        const int xo = c.cur ? R.cols : 0, yo = c.cur ? R.rows : 0;
        for (int k = threadIdx.x; k < nt * 32; k += kResThreads) {
            const int vr = t0 * 32 + k, j = real_row<SPLIT>(At, vr);
            len_t[k] = vr < At.nv ? At.len[vr] : 0;
            if (j >= 0) {
                sx[xo + k] = x[j];
                sxa[k] = v.xa[j];
                if (staged) {
                    bounds[k] = v.c[j];
                    bounds[R.cols + k] = v.lb[j];
                    bounds[2 * R.cols + k] = v.ub[j];
                    bounds[3 * R.cols + k] = v.q ? v.q[j] : 0.;
                }
            }
        }
        for (int k = threadIdx.x; k < na * 32; k += kResThreads) {
            const int vr = a0 * 32 + k, i = real_row<SPLIT>(A, vr);
            len_a[k] = vr < A.nv ? A.len[vr] : 0;
            if (i >= 0) {
                sy[yo + k] = y[i];
                sax[yo + k] = ax[i];
                sya[k] = v.ya[i];
                if (staged) {
                    bounds[4 * R.cols + k] = v.rl[i];
                    bounds[4 * R.cols + R.rows + k] = v.ru[i];
                }
            }
        }
        for (int k = threadIdx.x; k < nt; k += kResThreads) {
            at_t[k] = int(At.cptr[t0 + k] - tbase);
            slot_t[k] = R.slot_t[t0 + k];
        }
        for (int k = threadIdx.x; k < na; k += kResThreads) {
            at_a[k] = int(A.cptr[a0 + k] - abase);
            slot_a[k] = R.slot_a[a0 + k];
        }
        products_t(y);
    }
    // the sum of column l's products, from c_l (from 0: a split region's segment, and
    // the lanes past the last column, where an unstaged c has no entry)
    auto row_sum = [&](int k) {
        const int l = k * 32 + lane;
        const bool whole = (!SPLIT || (t0 + k) * 32 >= At.nsv) && t0 * 32 + l < At.nv;
        return add_products(prod + at_t[k] + lane, len_t[l], whole ? bc[l] : 0.);
    };
    bool unsaved = false; // Halpern: last_x / last_y hold the accepted point, the averages do not
    unsigned barrier = 0;
    int t = 0;
    __syncthreads(); // products of A^T y, the state
    double g0 = warp < nt ? row_sum(warp) : 0.; // of the warp's first chunk
    for (; t < trials && c.restart == 0; ++t) {
        const int cur = c.cur;
        const bool pending = c.pending != 0;
        const double pw = c.pending_w, lam = HALPERN ? 1 / (c.epoch + 2) : 0.; // if accepted
        // -------------------------------------------------- primal part
        {
            const double tau = c.tau * c.factor;
            const int co = cur ? R.cols : 0, to = cur ? 0 : R.cols;
            const double *qx = cur ? v.qx1 : v.qx0;
            double *gxt = cur ? v.x0 : v.x1;
            auto finish = [&](int l, int j, double g) -> double {
                const int o = staged ? l : j - first_t;
                // Halpern's vectors are in global memory: both loads go out first
                const double last = HALPERN && unsaved ? R.last_x[j] : 0.,
                             anchor = HALPERN ? v.anchor_x[j] : 0.;
                const double xj = sx[co + l], lj = blb[o], uj = bub[o], aj = sxa[l];
                const double qj = bq ? bq[o] : 0.;
                if constexpr (QP)
                    g = g + (__ldcg(qx + j) + qj * xj);
                const double den = QP ? 1. : 1 + tau * qj;
                double T = xj - tau * g;
                if (den != 1) // x / 1 is x
                    T = T / den;
                T = clampd(T, lj, uj);
                const double d = T - xj;
                __stcg(v.dx + j, d);
                if (pending)
                    sxa[l] = aj + (xj - aj) * pw;
                double xn = T;
                if (HALPERN) {
                    if (unsaved)
                        sxa[l] = last;
                    R.last_x[j] = T;
                    xn = lam * anchor + (1 - lam) * ((1 + r) * T - r * xj);
                }
                sx[to + l] = xn;
                if constexpr (QP)
                    __stcg(gxt + j, xn);
                return isfinite(T) ? d * d : INFINITY;
            };
            for (int k = warp; k < nt; k += kResWarps) {
                const int l = k * 32 + lane, j = first_t + l;
                const double sum = k == warp ? g0 : row_sum(k);
                double mine = 0;
                if (!SPLIT || (t0 + k) * 32 >= At.nsv) {
                    if (t0 * 32 + l < At.nv)
                        mine = finish(l, j, sum);
                } else {
                    const int vr = t0 * 32 + l;
                    const int4 sg = At.seg[vr];
                    const double init = sg.x >= 0 ? v.c[sg.x] : 0.;
                    double g;
                    if (split_chunk(wpart[warp], nullptr, nullptr, sg, vr, sum, init, &g))
                        mine = finish(l, sg.x, g);
                }
                mine = warp_total(mine);
                if (lane == 0)
                    __stcg(R.sums_p(t) + slot_t[k], mine);
            }
        }
        if (!grid_barrier(R.sync, ++barrier, v.ctl, &ok)) // dx is complete
            return;
        // -------------------------------------------------- dual part
        if constexpr (QP) {
            const double *xt = cur ? v.x0 : v.x1;
            double *qxt = cur ? v.qx0 : v.qx1;
            const int per = kResThreads / Q.lanes, end = R.own_q[blockIdx.x + 1];
            for (int k = R.own_q[blockIdx.x]; k < end; k += per) {
                const int row = k + int(threadIdx.x) / Q.lanes;
                const double s = q_row(Q, row, end, xt);
                if (row < end && (threadIdx.x & (Q.lanes - 1)) == 0)
                    __stcg(qxt + Q.rows[row], s);
            }
        }
        flat_products<false>(ip_a, vp_a, acount, v.dx, prod, nullptr, 0);
        double *gyt = cur ? v.y0 : v.y1;
        {
            const double sigma = c.sigma * c.factor;
            const int co = cur ? R.rows : 0, to = cur ? 0 : R.rows;
            auto finish = [&](int l, int i, double delta, double &dy2, double &cpl) {
                const int o = staged ? l : i - first_a;
                const double last = HALPERN && unsaved ? R.last_y[i] : 0.,
                             anchor = HALPERN ? v.anchor_y[i] : 0.,
                             anchor_ax = HALPERN ? v.anchor_ax[i] : 0.;
                const double yi = sy[co + l], axi = sax[co + l], rli = brl[o], rui = bru[o],
                             ai = sya[l];
                const double bar = axi + 2 * delta;
                const double z = yi + sigma * bar;
                const double T = max0(z - sigma * rui) + min0(z - sigma * rli);
                double yn = T, axn = axi + delta;
                if (pending)
                    sya[l] = ai + (yi - ai) * pw;
                if (HALPERN) {
                    if (unsaved)
                        sya[l] = last;
                    R.last_y[i] = T;
                    yn = lam * anchor + (1 - lam) * ((1 + r) * T - r * yi);
                    axn = lam * anchor_ax + (1 - lam) * ((1 + r) * axn - r * axi);
                }
                __stcg(gyt + i, yn);
                sy[to + l] = yn;
                sax[to + l] = axn;
                const double dy = T - yi;
                const bool bad = !isfinite(bar) || !isfinite(T) || !isfinite(delta);
                dy2 = bad ? INFINITY : dy * dy;
                cpl = dy * delta;
            };
            __syncthreads(); // products of A dx
            for (int k = warp; k < na; k += kResWarps) {
                const int l = k * 32 + lane, i = first_a + l;
                const double *p = prod + at_a[k] + lane;
                double dy2 = 0, cpl = 0;
                if (!SPLIT || (a0 + k) * 32 >= A.nsv) {
                    if (a0 * 32 + l < A.nv)
                        finish(l, i, add_products(p, len_a[l], 0.), dy2, cpl);
                } else {
                    const int vr = a0 * 32 + l;
                    const int4 sg = A.seg[vr];
                    const double part = add_products(p, len_a[l], 0.);
                    double delta;
                    if (split_chunk(wpart[warp], nullptr, nullptr, sg, vr, part, 0., &delta))
                        finish(l, sg.x, delta, dy2, cpl);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) {
                    dy2 += __shfl_xor_sync(0xffffffffu, dy2, off);
                    cpl += __shfl_xor_sync(0xffffffffu, cpl, off);
                }
                if (lane == 0) {
                    __stcg(R.sums_d(t) + slot_a[k], dy2);
                    __stcg(R.sums_d(t) + R.lists_d * R.width_d + slot_a[k], cpl);
                }
            }
        }
        if (!grid_barrier(R.sync, ++barrier, v.ctl, &ok)) // y and the terms are complete
            return;
        // -------------------------------------------------- decision
        const bool more = t + 1 < trials;
        if (more) { // the next trial's products and sums, should this one be accepted
            products_t(gyt);
            __syncthreads();
            g0 = warp < nt ? row_sum(warp) : 0.;
        }
        if (warp == 0) {
            unsigned long long word = 0;
            if (lane < kResWords) {
                const unsigned want = tag + unsigned(t);
                int polls = 0;
                do {
                    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                                 : "=l"(word)
                                 : "l"(R.word + lane)
                                 : "memory");
                } while (unsigned(word) != want && ++polls < kResMaxPolls);
                if (unsigned(word) != want) {
                    ok = 0;
                    atomicExch(&v.ctl->fault, 1);
                }
            }
            __syncwarp();
            const unsigned half = unsigned(word >> 32);
            unsigned h[kResWords];
#pragma unroll
            for (int k = 0; k < kResWords; ++k)
                h[k] = __shfl_sync(0xffffffffu, half, k);
            if (lane == 0) {
                const bool accept = h[4] & 1;
                c.factor = __hiloint2double(int(h[1]), int(h[0]));
                c.accept = accept ? 1 : 0;
                c.pending = accept && !HALPERN;
                c.pending_w = __hiloint2double(int(h[3]), int(h[2]));
                c.restart = h[4] & 2 ? 1 : 0;
                if (accept) {
                    c.cur ^= 1;
                    c.epoch += 1; // (Halpern's count; read by nothing else)
                }
            }
        }
        __syncthreads();
        if (ok == 0)
            return;
        unsaved = HALPERN && c.accept != 0;
        if (more && c.accept == 0) { // rejected: the products with the unchanged y
            products_t(cur ? v.y1 : v.y0);
            __syncthreads();
            g0 = warp < nt ? row_sum(warp) : 0.;
        }
    }
    // ------------------------------------------------------ close
    {
        double *x = c.cur ? v.x1 : v.x0, *y = c.cur ? v.y1 : v.y0, *ax = c.cur ? v.ax1 : v.ax0;
        const int xo = c.cur ? R.cols : 0, yo = c.cur ? R.rows : 0;
        for (int k = threadIdx.x; k < nt * 32; k += kResThreads) {
            const int j = real_row<SPLIT>(At, t0 * 32 + k);
            if (j >= 0) {
                x[j] = sx[xo + k];
                v.xa[j] = unsaved ? R.last_x[j] : sxa[k];
            }
        }
        for (int k = threadIdx.x; k < na * 32; k += kResThreads) {
            const int i = real_row<SPLIT>(A, a0 * 32 + k);
            if (i >= 0) {
                y[i] = sy[yo + k];
                ax[i] = sax[yo + k];
                v.ya[i] = unsaved ? R.last_y[i] : sya[k];
            }
        }
    }
    resident_leave(R);
}

} // namespace nk

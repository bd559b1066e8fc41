// The restarted solve's iterations of a mid-size LP in one cooperative launch per window
// (flow.cuh). Included by pdlp.cu, whose element rules it shares.
//
// An adaptive iteration is three steps of the grid: the dual candidate to the columns, the
// primal candidate to the rows, and the sums |dx|^2, |dy|^2 and dy.(A dx) to every CTA,
// which takes the accept / step decision for itself. Eight consecutive chunks go to eight
// warps of one CTA, which stand for one block of the launches: chunk sums by xor tree, the
// eight in order, then the blocks as ProbeEpi's last block combines them. So the steps have
// the launches' bits. A decision needs every CTA's sums, so nothing of an iteration is
// overwritten before the whole grid has read it; the sums themselves are kept twice, in
// turn, since a CTA that has read them says so only with its next ones.
//
// Measured on a B200 at 1,965 MHz, us per iteration with the window-end evaluations,
// launches -> this: adaptive FP64 5,000 x 11,000 (66,000 nonzeros) 14.4 -> 9.2, 15,000 x
// 30,000 (240,000) 16.0 -> 10.4, 30,000 x 60,000 (540,000) 18.9 -> 13.6, 50,000 x 100,000
// (1M) 25.1 -> 23.6; FP32 there 23.8 -> 21.1; Halpern FP64 8.6 -> 4.9, 10.2 -> 6.0, 12.5 ->
// 8.5 and 18.8 -> 15.1.
#pragma once

#include "flow.cuh"

namespace b200 {
namespace {

constexpr int kFlowThreads = 512;
constexpr int kFlowWarps = kFlowThreads / 32;
constexpr int kFlowGroups = kFlowWarps / 8;    // blocks of the launches a CTA stands for at a time
constexpr int kFlowBlocks = 1184;              // at most 8 blocks on each of 148 SMs
constexpr int kFlowRounds = 8;                 // groups of chunks a warp takes in a step, at most

template <class T, class V>
struct AdaptiveFlowArgs {
    TileCsrT<V> A, AT;
    T *x, *x_cand, *x_sum, *y, *y_cand, *y_sum, *ax, *ax_prev, *ax_cand;
    const T *c, *cl, *cu, *rl, *ru;
    const double* y_center;        // centered loop, else null
    PdlpState* st;
    double* fail;
    flow::Tagged<T>*xt, *yt;
    flow::Tagged<double>* sums;    // [2][3 kFlowBlocks]
    unsigned* count;               // CTAs that have published their sums, over all launches
    unsigned arrived;              // its value at the start
    unsigned first;                // number of the first iteration
    int iterations, polls;         // polls of a thread's waits in one iteration
};

// The chunk of this warp in round q of a step.
__device__ __forceinline__ int flow_chunk(int q) {
    const int warp = threadIdx.x >> 5;
    return 8 * ((q * kFlowGroups + (warp >> 3)) * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x)) + (warp & 7);
}

// Sum of the block values all[0 .. nb), in ProbeEpi's order (one warp): value k + 256 j of
// thread k in order, then the tree over 256 threads.
__device__ __forceinline__ double combine_blocks(const double* all, int nb) {
    const int lane = threadIdx.x & 31;
    double v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = 0.0;
        for (int g = lane + 32 * i; g < nb; g += 256) v[i] += all[g];
    }
    return warp_sum(((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7])));
}

template <class T, class V>
__global__ void __launch_bounds__(kFlowThreads, 1) k_adaptive_flow(const __grid_constant__ AdaptiveFlowArgs<T, V> a) {
    using namespace flow;
    extern __shared__ __align__(16) char smem[];
    T* prod = reinterpret_cast<T*>(smem);
    double* all = reinterpret_cast<double*>(smem + kFlowWarps * kChunkNnz * sizeof(T));   // [3 kFlowBlocks]
    __shared__ double part[3][kFlowRounds][kFlowWarps], total[3], growth[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    T* sp = prod + warp * kChunkNnz;
    const int nbc = (a.AT.ntiles + 7) / 8, nbr = (a.A.ntiles + 7) / 8;
    const double omega = a.st->omega, eta_lo = a.st->eta_min, eta_hi = a.st->eta_max;
    double eta = a.st->eta, updates = a.st->updates, accepts = a.st->accept_count;
    double dx2 = 0.0, dy2 = 0.0, cross = 0.0, limit = a.st->eta_bar;
    bool keep = false, ok = true;
    // The accepted candidate becomes the iterate (k_commit_dual's first half). All loads
    // first: behind a store that may alias, each would cost a latency of its own.
    struct RowState { T y, ax, ax_prev; };
    auto commit_row = [&](int i) {
        const T yc = a.y_cand[i], sum = a.y_sum[i], ax = a.ax[i], axc = a.ax_cand[i];
        a.y[i] = yc;
        a.y_sum[i] = sum + yc;
        a.ax_prev[i] = ax;
        a.ax[i] = axc;
        return RowState{yc, axc, ax};
    };
    auto commit_column = [&](int j) {
        const T xc = a.x_cand[j], sum = a.x_sum[j];
        a.x[j] = xc;
        a.x_sum[j] = sum + xc;
        return xc;
    };
    unsigned arrived = a.arrived;
    for (int it = 0; it < a.iterations && ok; ++it) {
        const typename TagOf<T>::type tag = a.first + it;
        const T sigma = static_cast<T>(eta * omega), tau = static_cast<T>(eta / omega);
        int left = a.polls;
        for (int q = 0, t; (t = flow_chunk(q)) < (a.A.ntiles + 7) / 8 * 8; ++q) {
            if (t >= a.A.ntiles) continue;
            const int i = __ldg(a.A.tile + t).x + lane;
            if (i >= __ldg(a.A.tile + t + 1).x) continue;
            const T lo = __ldg(a.rl + i), hi = __ldg(a.ru + i);
            const double center = a.y_center ? __ldg(a.y_center + i) : 0.0;
            const RowState s = keep ? commit_row(i) : RowState{a.y[i], a.ax[i], a.ax_prev[i]};
            const T yc = a.y_center ? dual_candidate_centered(s.y, s.ax, s.ax_prev, sigma, lo, hi, center)
                                    : dual_candidate(s.y, s.ax, s.ax_prev, sigma, lo, hi);
            a.y_cand[i] = yc;
            store_tagged(a.yt + i, yc, tag);
        }
        __syncwarp();
        for (int q = 0, t; (t = flow_chunk(q)) < (a.AT.ntiles + 7) / 8 * 8; ++q) {
            double d = 0.0;
            if (t < a.AT.ntiles) {
                const ChunkRows k = chunk_rows(a.AT, t);
                const int j = k.row;
                T x = T(0), c = T(0), lo = T(0), hi = T(0);
                if (k.owns) {
                    x = keep ? commit_column(j) : a.x[j];
                    c = __ldg(a.c + j);
                    lo = __ldg(a.cl + j);
                    hi = __ldg(a.cu + j);
                }
                const T aty = chunk_sum(a.AT, k, a.yt, tag, sp, &left);
                if (k.owns) {
                    const T xn = primal_candidate(x, aty, tau, c, lo, hi);
                    store_tagged(a.xt + j, xn, tag);
                    a.x_cand[j] = xn;
                    const double dx = static_cast<double>(xn) - static_cast<double>(x);
                    d = dx * dx;
                }
                d = warp_sum(d);
            }
            if (lane == 0) part[0][q][warp] = d;
        }
        for (int q = 0, t; (t = flow_chunk(q)) < (a.A.ntiles + 7) / 8 * 8; ++q) {
            double d = 0.0, e = 0.0;
            if (t < a.A.ntiles) {
                const ChunkRows k = chunk_rows(a.A, t);
                const int i = k.row;
                T y = T(0), yc = T(0), ax = T(0);
                if (k.owns) {
                    y = a.y[i];
                    yc = a.y_cand[i];
                    ax = a.ax[i];
                }
                const T axn = chunk_sum(a.A, k, a.xt, tag, sp, &left);
                if (k.owns) {
                    a.ax_cand[i] = axn;
                    const double dy = static_cast<double>(yc) - static_cast<double>(y);
                    d = dy * dy;
                    e = dy * (static_cast<double>(axn) - static_cast<double>(ax));
                }
                d = warp_sum(d);
                e = warp_sum(e);
            }
            if (lane == 0) {
                part[1][q][warp] = d;
                part[2][q][warp] = e;
            }
        }
        __syncthreads();
        Tagged<double>* slots = a.sums + (it & 1) * 3 * kFlowBlocks;
        const int group = threadIdx.x / 4 % kFlowGroups, round = threadIdx.x / 4 / kFlowGroups, what = threadIdx.x % 4;
        if (what < 3 && round < kFlowRounds) {   // one of the sums of one block
            const int b = (round * kFlowGroups + group) * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
            if (b < (what == 0 ? nbc : nbr)) {
                const double* p = part[what][round] + 8 * group;
                double r = p[0];
                for (int w = 1; w < 8; ++w) r = r + p[w];
                store_tagged(slots + what * kFlowBlocks + b, r, static_cast<unsigned long long>(tag));
            }
        }
        // A count of the CTAs that have come this far says when the sums are worth reading (the
        // numbers on them still decide): read at once, by the whole grid, their lines go back
        // and forth between every store.
        __syncthreads();
        arrived += gridDim.x;
        if (threadIdx.x == 0) {
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(a.count) : "memory");
            unsigned seen = 0;
            do asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.count) : "memory");
            while (static_cast<int>(seen - arrived) < 0 && --left > 0);
        }
        if (warp == kFlowWarps - 1 && lane < 2) growth[lane] = step_growth(updates + 1.0, lane == 0);
        __syncthreads();
        constexpr int kReads = sizeof(T) == 4 ? 4 : 1;   // in flight; the FP64 loop has no registers for more
        for (int b0 = threadIdx.x; b0 < nbc + 2 * nbr; b0 += kReads * kFlowThreads) {
            Tagged<double> e[kReads];
            int at[kReads];
#pragma unroll
            for (int k = 0; k < kReads; ++k) {
                const int b = b0 + k * kFlowThreads;
                at[k] = b < nbc ? b : b < nbc + nbr ? kFlowBlocks + b - nbc : 2 * kFlowBlocks + b - nbc - nbr;
                if (b < nbc + 2 * nbr) e[k] = load_tagged(slots + at[k]);
            }
#pragma unroll
            for (int k = 0; k < kReads; ++k)
                if (b0 + k * kFlowThreads < nbc + 2 * nbr)
                    all[at[k]] = e[k].tag == tag ? e[k].value
                                                 : wait_element(slots + at[k], static_cast<unsigned long long>(tag), &left);
        }
        ok = __syncthreads_and(left > 0) != 0;
        if (warp < 3) {
            const double t = combine_blocks(all + warp * kFlowBlocks, warp == 0 ? nbc : nbr);
            if (lane == 0) total[warp] = t;
        }
        __syncthreads();
        dx2 = total[0];
        dy2 = total[1];
        cross = fabs(total[2]);
        updates += 1.0;
        const StepRule rule = step_rule(eta, omega, dx2, dy2, cross, growth[0], growth[1], eta_lo, eta_hi);
        limit = rule.limit;
        eta = rule.next;
        keep = rule.keep;
        accepts += keep ? 1.0 : 0.0;
    }
    if (keep) {
        for (int q = 0, t; (t = flow_chunk(q)) < a.A.ntiles; ++q) {
            const int i = __ldg(a.A.tile + t).x + lane;
            if (i < __ldg(a.A.tile + t + 1).x) commit_row(i);
        }
        for (int q = 0, t; (t = flow_chunk(q)) < a.AT.ntiles; ++q) {
            const int j = __ldg(a.AT.tile + t).x + lane;
            if (j < __ldg(a.AT.tile + t + 1).x) commit_column(j);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        PdlpState* st = a.st;
        st->eta = eta;
        st->eta_bar = limit;
        st->dx_sq = dx2;
        st->dy_sq = dy2;
        st->interaction = cross;
        st->updates = updates;
        st->accept_count = accepts;
        st->accepted = 0.0;   // committed above
    }
    if (!ok && threadIdx.x == 0) *a.fail = 1.0;
}

template <class T, class V>
struct HalpernFlowArgs {
    TileCsrT<V> A, AT;
    T *x, *y;
    const T *x0, *y0, *c, *cl, *cu, *rl, *ru;
    const PdlpState* st;
    double* fail;
    flow::Tagged<T>*xt, *yt;
    unsigned first;        // number of the first iteration; the start has the one before
    int done, iterations;  // of the window
    int polls;             // of a thread's waits in one iteration
};

template <class T, class V>
__global__ void __launch_bounds__(kFlowThreads, 1) k_halpern_flow(const __grid_constant__ HalpernFlowArgs<T, V> a) {
    using namespace flow;
    extern __shared__ __align__(16) char smem[];
    const int warp = threadIdx.x >> 5;
    T* sp = reinterpret_cast<T*>(smem) + warp * kChunkNnz;
    const int nw = gridDim.x * kFlowWarps, mine = warp * gridDim.x + blockIdx.x;
    const T tau = static_cast<T>(a.st->eta / a.st->omega), sigma = static_cast<T>(a.st->eta * a.st->omega);
    for (int i = blockIdx.x * kFlowThreads + threadIdx.x; i < a.A.rows; i += gridDim.x * kFlowThreads)
        store_tagged(a.yt + i, a.y[i], a.first - 1);
    __syncthreads();
    for (int it = 0; it < a.iterations; ++it) {
        const typename TagOf<T>::type tag = a.first + it;
        const T lam = halpern_lambda<T>(a.st, a.done + it);
        int left = a.polls;
        for (int t = mine; t < a.AT.ntiles; t += nw) {
            const ChunkRows k = chunk_rows(a.AT, t);
            const int j = k.row;
            T x = T(0), x0 = T(0), c = T(0), lo = T(0), hi = T(0);
            if (k.owns) {
                x = a.x[j];
                x0 = __ldg(a.x0 + j);
                c = __ldg(a.c + j);
                lo = __ldg(a.cl + j);
                hi = __ldg(a.cu + j);
            }
            const T aty = chunk_sum(a.AT, k, a.yt, tag - 1, sp, &left);
            if (k.owns) {
                const T p = primal_reflected(x, aty, tau, c, lo, hi);
                store_tagged(a.xt + j, p, tag);
                a.x[j] = primal_halpern_step(lam, p, x0);
            }
        }
        for (int t = mine; t < a.A.ntiles; t += nw) {
            const ChunkRows k = chunk_rows(a.A, t);
            const int i = k.row;
            T y = T(0), y0 = T(0), lo = T(0), hi = T(0);
            if (k.owns) {
                // the first iteration takes y from its tagged copy: another thread published
                // it, and this store must not come before that thread's read
                y = it == 0 ? wait_element(a.yt + i, tag - 1, &left) : a.y[i];
                y0 = __ldg(a.y0 + i);
                lo = __ldg(a.rl + i);
                hi = __ldg(a.ru + i);
            }
            const T axb = chunk_sum(a.A, k, a.xt, tag, sp, &left);
            if (k.owns) {
                const T yn = dual_halpern_step(lam, dual_reflected(y, axb, sigma, lo, hi), y0);
                store_tagged(a.yt + i, yn, tag);
                a.y[i] = yn;
            }
        }
        if (__any_sync(0xffffffffu, left <= 0)) {
            if ((threadIdx.x & 31) == 0) *a.fail = 1.0;
            break;
        }
    }
}

}  // namespace
}  // namespace b200

// Fixed-step PDHG iterations of a small LP (or diagonal QP) on one cluster.
//
// Measured on a B200 at 1,965 MHz, us per iteration, two graph launches -> this kernel:
// 200 x 300 (900 nonzeros) 5.5 -> 1.5; 1,000 x 2,500 (12,500) 7.0 -> 2.2; 2,000 x 5,000
// (25,000) 7.7 -> 2.85; 3,000 x 7,000 (42,000) 7.7 -> 3.8. Of the 5,400 cycles of an
// iteration at 2,000 x 5,000, the two exchanges take 1,500 and 1,400 (580 each of latency,
// the rest 12.8 bytes per cycle), the rows' sums and epilogues 1,500 and the columns' 1,000:
// a serial chain of adds (12 cycles each), one divide (137) and shared-memory latencies, with
// the 16 SMs' shared-memory bandwidth next. With more than one chunk a warp (4,000 x 9,000,
// 54,000) it took 5.2 where the cooperative launch of fixed_flow.cuh takes 3.9, so it ends there.
#pragma once

#include "cluster.cuh"
#include "fixed_epi.cuh"

namespace b200 {

// The checkpoints of a solve, taken by the kernel itself: every `every` iterations (and
// after the last) the residuals of the current point, whose maxima all CTAs exchange and
// test alike (about 1.5 iterations' time), so that a solve without a time limit needs no
// launch and no host between its windows. As five launches, a copy and a wait on the host
// they took 40 us, and the next window's launch and setup 20 more: at 2,000 x 5,000, 1,000
// iterations tested every 20 (the C core's loop) 5.86 ms -> 3.50, tested every 100
// 3.35 -> 3.22. every 0: none.
struct FixedChecks {
    int every = 0;
    double tolerance = 0.0, dual_limit = 0.0;   // CUDA: the tolerance; SK: primal_tol and dual_tol (1 + anorm)
    int first = 1;          // no checkpoint of this solve before this launch
    double* x_prev = nullptr;   // CUDA: the last checkpoint's x
    double* activity = nullptr; // SK: A x of the last checkpoint
    double* out = nullptr;      // [0] iterations run, [1] verdict, [2] checkpoints, [3 ..] the last one's maxima
};
enum Verdict { kUnmet = 0, kMet = 1, kNotFinite = 2 };
// CUDA: the rows' 5 and the columns' 6 maxima, then the objective; SK: violation, step, scale, dual step.
constexpr int kCheckMaxima = 11, kObjectiveSlot = 11, kCheckTotals = 12;

// The gates on the combined maxima (sankhya_cuda_lp.cu:361-385, sk_solve.c:926-953).
template <bool SK>
__device__ __forceinline__ int gates(const double* v, const FixedChecks& k, bool first) {
    if (SK) return v[0] <= k.tolerance && v[1] <= k.tolerance * fmax(1.0, v[2]) && v[3] <= k.dual_limit ? kMet : kUnmet;
    const double objective = v[kObjectiveSlot];
    if (fmax(v[0], v[5]) > 0.0 || !isfinite(objective)) return kNotFinite;
    const double tol = k.tolerance;
    return v[1] <= tol && !first && v[6] <= tol * fmax(1.0, v[7]) && fmax(v[2], v[8]) <= tol && fmax(v[3], v[9]) <= tol &&
                   fmax(v[4], v[10]) / (1.0 + fabs(objective)) <= tol
               ? kMet : kUnmet;
}

struct FixedClusterArgs {
    TileCsr A, AT;
    const double *c, *cl, *cu, *tauv, *qdiag;  // tauv / sigv / qdiag may be null
    const double *rl, *ru, *sigv;
    double tau, sigma, theta;
    const double *x_in, *y_in;
    double *x_out, *y_out, *x_bar;  // x_bar: in and out
    double* part;                   // SK: max |y_new - y| of the last iteration, one per CTA
    int iterations, polls;          // polls of a wait
    unsigned int* fail;             // set when a wait gave up
    FixedChecks check;
};

// Shared memory of one CTA; 0 when the problem has no rows or no columns, or a CTA would
// have more chunks than warps (each stays in its warp's registers for the whole launch).
inline size_t fixed_cluster_smem(const TileCsr& A, const TileCsr& AT) {
    if (A.ntiles == 0 || AT.ntiles == 0 ||
        std::max(A.share.chunks, AT.share.chunks) > cluster::kClusterWarps)
        return 0;
    return cluster::kClusterWarps * cluster::kProducts * 8ull + cluster::slice_bytes(A) + cluster::slice_bytes(AT) + cluster::packed_bytes<double>(A) +
           cluster::packed_bytes<double>(AT) + cluster::send_bytes(A.share) + cluster::send_bytes(AT.share) +
           4 * cluster::align16(8ull * A.share.rows) + 7 * cluster::align16(8ull * AT.share.rows);
}
// What the checkpoints add: what all CTAs send of one, twice in turn, its barriers, and the
// warps' maxima.
template <bool SK>
__host__ __device__ inline int gathered_length(const TileCsr& AT) {
    return cluster::kClusterCtas * kCheckMaxima + (SK ? 0 : cluster::padded_chunks(AT.ntiles));
}
template <bool SK>
inline size_t fixed_check_smem(const TileCsr& AT) {
    return 2 * cluster::align16(8ull * gathered_length<SK>(AT)) + 16 + 8ull * cluster::kClusterWarps * kCheckMaxima;
}

template <bool SK>
__global__ void __launch_bounds__(cluster::kClusterThreads, 1) k_fixed_cluster(const __grid_constant__ FixedClusterArgs a) {
    using namespace cluster;
    extern __shared__ __align__(16) char smem[];
    __shared__ double red[kClusterWarps], own[kCheckMaxima + kClusterWarps], total[kCheckTotals];
    const unsigned rank = cta_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Arena mem{smem};
    double* sp = mem.take<double>(kClusterWarps * kProducts) + warp * kProducts;
    if (lane < 2) sp[kChunkNnz + lane] = -0.0;
    Part<double, double> rows, cols;   // of A and of A'
    SendList xs_out, ys_out;
    load_parts(a.A, a.AT, rank, mem, &rows, &cols);
    const Slice<double>&R = rows.slice, &Q = cols.slice;
    Packed<double>&xv = rows.in, &yv = cols.in;    // x_bar as R gathers it, y as Q gathers it
    double* y = mem.take<double>(a.A.share.rows);    // own elements
    double* x = mem.take<double>(a.AT.share.rows);
    double* xb = mem.take<double>(a.AT.share.rows);
    // the steps' constants too: a wait that acquires drops the SM's cached global lines
    double* rl = mem.take<double>(a.A.share.rows);
    double* ru = mem.take<double>(a.A.share.rows);
    double* sig = mem.take<double>(a.A.share.rows);
    double* c = mem.take<double>(a.AT.share.rows);
    double* cl = mem.take<double>(a.AT.share.rows);
    double* cu = mem.take<double>(a.AT.share.rows);
    double* tau = mem.take<double>(a.AT.share.rows);
    double* gathered[2] = {nullptr, nullptr};   // per CTA its maxima, then all column chunks' objectives
    unsigned long long* gathered_bar = nullptr;
    double* maxima = nullptr;
    if (a.check.every) {
        gathered[0] = mem.take<double>(gathered_length<SK>(a.AT));
        gathered[1] = mem.take<double>(gathered_length<SK>(a.AT));
        gathered_bar = mem.take<unsigned long long>(2);
        maxima = mem.take<double>(kClusterWarps * kCheckMaxima);
        if (threadIdx.x < 2) init_barrier(gathered_bar + threadIdx.x);
        for (int k = threadIdx.x; !SK && k < gathered_length<SK>(a.AT); k += blockDim.x) gathered[0][k] = gathered[1][k] = 0.0;
    }
    fill_packed(a.A, xv, a.x_bar);
    for (int r = threadIdx.x; r < R.rows; r += blockDim.x) {
        const int i = R.row0 + r;
        y[r] = a.y_in[i];
        rl[r] = a.rl[i];
        ru[r] = a.ru[i];
        sig[r] = a.sigv ? a.sigv[i] : a.sigma;
    }
    for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) {
        const int j = Q.row0 + r;
        x[r] = a.x_in[j];
        c[r] = a.c[j];
        cl[r] = a.cl[j];
        cu[r] = a.cu[j];
        tau[r] = a.tauv ? a.tauv[j] : a.tau;
    }
    cluster_sync();
    make_sends(Q.row0, Q.rows, xv, a.AT.share, mem, &xs_out);
    make_sends(R.row0, R.rows, yv, a.A.share, mem, &ys_out);
    cluster_sync();
    Chunk<double, double> rc, qc;
    if (warp < R.chunks) rc.load(R, warp, xv.v);
    if (warp < Q.chunks) qc.load(Q, warp, yv.v);
    double change = 0.0;
    Waits waits{xs_out, ys_out, a.polls};
    int it = 0, verdict = kUnmet, checks = 0;
    for (; it < a.iterations && verdict == kUnmet; ++it) {
        const bool last = it + 1 == a.iterations;
        const bool check = a.check.every && (last || (it + 1) % a.check.every == 0);
        if (warp < R.chunks) {
            const double act = rc.sum(R, xv.v, sp);
            if (rc.owns) {
                const int r = rc.r;
                const double old = y[r];
                const double yn = SK ? dual_step_sk(old, act, sig[r], rl[r], ru[r])
                                     : dual_step_cuda(old, act, sig[r], rl[r], ru[r]);
                y[r] = yn;
                if (SK && (last || check)) change = fabs(dsub(yn, old));
            }
        }
        exchange(waits, ys_out, y, yv);
        if (warp < Q.chunks) {
            const double g = qc.sum(Q, yv.v, sp);
            if (qc.owns) {
                const int r = qc.r;
                const double old = x[r], qd = a.qdiag ? __ldg(a.qdiag + Q.row0 + r) : 0.0;
                const double xn =
                    SK ? primal_step_sk(old, g, c[r], tau[r], cl[r], cu[r], a.qdiag != nullptr, qd, 0.0)
                       : primal_step_cuda(old, g, c[r], tau[r], cl[r], cu[r], a.qdiag != nullptr, qd, 0.0);
                x[r] = xn;
                xb[r] = SK ? dsub(dmul(2.0, xn), old) : dadd(xn, dmul(a.theta, dsub(xn, old)));
            }
        }
        exchange(waits, xs_out, check ? x : xb, xv);
        if (!check) continue;
        // the point's residuals: x at all CTAs for A x, y still there for A'y
        constexpr int kSlots = SK ? 4 : kCheckMaxima;
        double v[kCheckMaxima], objective = 0.0;
#pragma unroll
        for (int k = 0; k < kSlots; ++k) v[k] = 0.0;
        if (warp < R.chunks) {
            const double act = rc.sum(R, xv.v, sp);
            if (rc.owns) {
                const int r = rc.r;
                if (SK) {
                    a.check.activity[R.row0 + r] = act;
                    if (!sk_neg_inf(rl[r])) v[0] = fmax(v[0], rl[r] - act);
                    if (!sk_inf(ru[r])) v[0] = fmax(v[0], act - ru[r]);
                    v[3] = change;
                } else {
                    CheckRowsCudaEpi::Acc acc;
                    acc.init();
                    CheckRowsCudaEpi{y, rl, ru, nullptr}.row(r, act, acc);
#pragma unroll
                    for (int k = 0; k < 5; ++k) v[k] = acc.v[k];
                }
            }
        }
        if (warp < Q.chunks) {
            const double g = SK ? 0.0 : qc.sum(Q, yv.v, sp);
            if (qc.owns) {
                const int r = qc.r;
                if (SK) {
                    v[1] = fabs(xb[r] - x[r]);
                    v[2] = fabs(x[r]);
                } else {
                    CheckColsCudaEpi::Acc acc;
                    acc.init();
                    CheckColsCudaEpi{x, a.check.x_prev + Q.row0, c, a.qdiag ? a.qdiag + Q.row0 : nullptr, nullptr, cl, cu,
                                     nullptr}.row(r, g, acc);
                    v[5] = acc.v[0];
                    objective = acc.v[1];
#pragma unroll
                    for (int k = 2; k < 7; ++k) v[4 + k] = acc.v[k];
                }
            }
            if (!SK) {
                objective = warp_sum(objective);
                if (lane == 0) own[kSlots + warp] = objective;
            }
        }
#pragma unroll
        for (int k = 0; k < kSlots; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] = fmax(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
            if (lane == 0) maxima[warp * kCheckMaxima + k] = v[k];
        }
        __syncthreads();
        if (threadIdx.x < kSlots) {
            double t = maxima[threadIdx.x];
            for (int w = 1; w < kClusterWarps; ++w) t = fmax(t, maxima[w * kCheckMaxima + threadIdx.x]);
            own[threadIdx.x] = t;
        }
        __syncthreads();
        double* all = checks & 1 ? gathered[1] : gathered[0];
        double* sums = all + kClusterCtas * kCheckMaxima;
        unsigned long long* bar = gathered_bar + (checks & 1);
        if (waits.arms()) expect_bytes(bar, 8u * (kClusterCtas * kSlots + (SK ? 0 : a.AT.ntiles)));
        if (!waits.gave_up && lane < kSlots + (SK ? 0 : Q.chunks))   // warp w sends to CTA w
            send_one(remote(lane < kSlots ? all + static_cast<int>(rank) * kCheckMaxima + lane
                                          : sums + static_cast<int>(rank) * a.AT.share.chunks + lane - kSlots, warp),
                     own[lane], remote(bar, warp));
        waits.wait(bar, static_cast<unsigned>(checks >> 1) & 1u);
        if (threadIdx.x < kSlots) {
            double t = all[threadIdx.x];
            for (int w = 1; w < kClusterCtas; ++w) t = fmax(t, all[w * kCheckMaxima + threadIdx.x]);
            total[threadIdx.x] = t;
        }
        if (!SK && warp == 1) {
            const double t = tree_of_blocks(sums, padded_chunks(a.AT.ntiles));
            if (lane == 0) total[kObjectiveSlot] = t;
        }
        __syncthreads();
        verdict = gates<SK>(total, a.check, a.check.first && checks == 0);
        ++checks;
        if (verdict == kUnmet && !last) exchange(waits, xs_out, xb, xv);   // on: x_bar after all
    }
    if (waits.gave_up) *a.fail = 1u;
    cluster_sync();
    for (int j = threadIdx.x; j < Q.rows; j += blockDim.x) {
        a.x_out[Q.row0 + j] = x[j];
        a.x_bar[Q.row0 + j] = xb[j];
    }
    for (int i = threadIdx.x; i < R.rows; i += blockDim.x) a.y_out[R.row0 + i] = y[i];
    if (a.check.every) {
        if (rank == 0 && threadIdx.x < (SK ? 4 : kCheckTotals)) a.check.out[3 + threadIdx.x] = total[threadIdx.x];
        if (rank == 0 && threadIdx.x == 0) {
            a.check.out[0] = it;
            a.check.out[1] = verdict;
            a.check.out[2] = checks;
        }
    } else if (SK) {
        for (int o = 16; o > 0; o >>= 1) change = fmax(change, __shfl_xor_sync(0xffffffffu, change, o));
        if (lane == 0) red[warp] = change;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < kClusterWarps; ++k) change = fmax(change, red[k]);
            a.part[rank] = change;
        }
    }
}

}  // namespace b200

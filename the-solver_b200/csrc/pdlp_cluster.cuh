// The restarted solve's iterations of a small LP on one cluster (cluster.cuh). Included by
// pdlp.cu, whose element rules (dual_candidate, primal_candidate, the Halpern steps,
// step_rule) it shares.
//
// An adaptive iteration is three exchanges: the dual candidate to the columns' owners, the
// primal candidate to the rows' owners, and every chunk's sums (|dx|^2, |dy|^2, dy.(A dx))
// to every CTA, which then takes the same accept / step decision for itself. The sums keep
// the shape they have over the launches, where each warp of a block has one chunk: xor tree
// over a chunk's lanes, the eight chunks of a block in order, then the tree over 256 blocks
// that ProbeEpi's last block runs. So the steps, and with them the iterates, have the same
// bits (the adaptive loop would turn one different last bit into another trajectory).
//
// Measured on a B200 at 1,965 MHz, us per iteration with the window-end evaluations, three
// (Halpern: two) graph launches -> one cluster launch per window of 64: 300 x 700 adaptive
// 11.9 -> 4.3, Halpern 7.4 -> 2.8; 2,000 x 5,000 (25,000 nonzeros) adaptive FP64 13.4 -> 5.9,
// FP32 13.6 -> 5.3, Halpern 8.2 -> 4.2. An adaptive iteration at 2,000 x 5,000 takes 8,000 cycles: the two vector
// exchanges 1,500 each, the columns' and rows' sums 1,600 and 2,000 (a serial chain of adds
// and the chunk trees), the candidate 650, the sums' exchange 600, the decision 1,000.
#pragma once

#include "cluster.cuh"

namespace b200 {
namespace {

// All CTAs' chunk sums: two buffers taken in turn, since a CTA that has read the sums of an
// iteration says so only by its sums of the next one.
struct ChunkSums {
    double *all0, *all1;           // [column chunks' |dx|^2 | row chunks' |dy|^2 | row chunks' dy.(A dx)]
    unsigned long long *bar0, *bar1;
    double* own;                   // this CTA's, [columns | rows | rows]
    int cols, rows;                // padded to whole blocks
    unsigned bytes;                // of one exchange
};

template <class T, class V>
struct AdaptiveClusterArgs {
    TileCsrT<V> A, AT;
    T *x, *x_sum, *y, *y_sum, *ax, *ax_prev;
    const T *c, *cl, *cu, *rl, *ru;
    const double* y_center;        // centered loop, else null
    PdlpState* st;
    double* fail;
    int iterations, polls;         // polls of a wait
};

// Shared memory of one CTA; 0 when there are no rows or columns. (A CTA has at most a chunk
// per warp, so there are at most 32 blocks of eight.)
template <class T, class V>
inline size_t adaptive_cluster_smem(const TileCsrT<V>& A, const TileCsrT<V>& AT) {
    using namespace cluster;
    if (A.ntiles == 0 || AT.ntiles == 0) return 0;
    const size_t sums = 8ull * (padded_chunks(AT.ntiles) + 2 * padded_chunks(A.ntiles));
    return align16(kClusterWarps * kProducts * sizeof(T)) + slice_bytes(A) + slice_bytes(AT) + packed_bytes<T>(A) +
           packed_bytes<T>(AT) + send_bytes(A.share) + send_bytes(AT.share) + 2 * align16(sums) +
           align16(8ull * (AT.share.chunks + 2 * A.share.chunks)) + 32 + 8 * align16(sizeof(T) * A.share.rows) +
           align16(8ull * A.share.rows) + 6 * align16(sizeof(T) * AT.share.rows);
}

template <class T, class V>
__global__ void __launch_bounds__(cluster::kClusterThreads, 1)
    k_adaptive_cluster(const __grid_constant__ AdaptiveClusterArgs<T, V> a) {
    using namespace cluster;
    extern __shared__ __align__(16) char smem[];
    __shared__ double total[3], growth[2];
    const unsigned rank = cta_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Arena mem{smem};
    T* sp = mem.take<T>(kClusterWarps * kProducts) + warp * kProducts;
    if (lane < 2) sp[kChunkNnz + lane] = T(-0.0);
    Part<T, V> rows, cols;   // of A and of A'
    SendList xs_out, ys_out;
    load_parts(a.A, a.AT, rank, mem, &rows, &cols);
    const Slice<V>&R = rows.slice, &Q = cols.slice;
    Packed<T>&xv = rows.in, &yv = cols.in;
    ChunkSums sums;
    sums.cols = (a.AT.ntiles + 7) / 8 * 8;
    sums.rows = (a.A.ntiles + 7) / 8 * 8;
    sums.bytes = 8u * (a.AT.ntiles + 2 * a.A.ntiles);
    sums.own = mem.take<double>(a.AT.share.chunks + 2 * a.A.share.chunks);
    sums.all0 = mem.take<double>(sums.cols + 2 * sums.rows);
    sums.all1 = mem.take<double>(sums.cols + 2 * sums.rows);
    sums.bar0 = mem.take<unsigned long long>(1);
    sums.bar1 = mem.take<unsigned long long>(1);
    for (int t = threadIdx.x; t < sums.cols + 2 * sums.rows; t += blockDim.x) sums.all0[t] = sums.all1[t] = 0.0;
    if (threadIdx.x == 0) {
        init_barrier(sums.bar0);
        init_barrier(sums.bar1);
    }
    const int mr = a.A.share.rows, nr = a.AT.share.rows;
    T *y = mem.take<T>(mr), *yc = mem.take<T>(mr), *ysum = mem.take<T>(mr), *ax = mem.take<T>(mr);
    T *axp = mem.take<T>(mr), *axc = mem.take<T>(mr), *rl = mem.take<T>(mr), *ru = mem.take<T>(mr);
    double* center = mem.take<double>(mr);
    T *x = mem.take<T>(nr), *xc = mem.take<T>(nr), *xsum = mem.take<T>(nr);
    T *c = mem.take<T>(nr), *cl = mem.take<T>(nr), *cu = mem.take<T>(nr);
    for (int r = threadIdx.x; r < R.rows; r += blockDim.x) {
        const int i = R.row0 + r;
        y[r] = a.y[i];
        ysum[r] = a.y_sum[i];
        ax[r] = a.ax[i];
        axp[r] = a.ax_prev[i];
        rl[r] = a.rl[i];
        ru[r] = a.ru[i];
        if (a.y_center) center[r] = a.y_center[i];
    }
    for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) {
        const int j = Q.row0 + r;
        x[r] = a.x[j];
        xsum[r] = a.x_sum[j];
        c[r] = a.c[j];
        cl[r] = a.cl[j];
        cu[r] = a.cu[j];
    }
    cluster_sync();
    make_sends(Q.row0, Q.rows, xv, a.AT.share, mem, &xs_out);
    make_sends(R.row0, R.rows, yv, a.A.share, mem, &ys_out);
    cluster_sync();
    Chunk<T, V> rc, qc;
    if (warp < R.chunks) rc.load(R, warp, xv.v);
    if (warp < Q.chunks) qc.load(Q, warp, yv.v);
    const double omega = a.st->omega, eta_lo = a.st->eta_min, eta_hi = a.st->eta_max;
    double eta = a.st->eta, updates = a.st->updates, accepts = a.st->accept_count;
    double dx2 = 0.0, dy2 = 0.0, cross = 0.0, limit = a.st->eta_bar;
    bool keep = false;
    Waits waits{xs_out, ys_out, a.polls};
    // the accepted candidate becomes the iterate (k_commit_dual's first half)
    auto commit = [&](int r) {
        y[r] = yc[r];
        ysum[r] += yc[r];
        axp[r] = ax[r];
        ax[r] = axc[r];
    };
    auto commit_columns = [&]() {
        for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) {
            x[r] = xc[r];
            xsum[r] += xc[r];
        }
    };
    for (int it = 0; it < a.iterations; ++it) {
        const T sigma = static_cast<T>(eta * omega), tau = static_cast<T>(eta / omega);
        for (int r = threadIdx.x; r < R.rows; r += blockDim.x) {
            if (keep) commit(r);
            yc[r] = a.y_center ? dual_candidate_centered(y[r], ax[r], axp[r], sigma, rl[r], ru[r], center[r])
                               : dual_candidate(y[r], ax[r], axp[r], sigma, rl[r], ru[r]);
        }
        if (keep) commit_columns();
        exchange(waits, ys_out, yc, yv);
        if (warp < Q.chunks) {
            const T aty = qc.sum(Q, yv.v, sp);
            double d = 0.0;
            if (qc.owns) {
                const int r = qc.r;
                const T xn = primal_candidate(x[r], aty, tau, c[r], cl[r], cu[r]);
                xc[r] = xn;
                const double dx = static_cast<double>(xn) - static_cast<double>(x[r]);
                d = dx * dx;
            }
            d = warp_sum(d);
            if (lane == 0) sums.own[warp] = d;
        }
        exchange(waits, xs_out, xc, xv, [&] {
            if (warp != kClusterWarps - 1 || lane >= 2) return;   // the warp with the fewest chunks
            growth[lane] = step_growth(updates + 1.0, lane == 0);
        });
        if (warp < R.chunks) {
            const T axn = rc.sum(R, xv.v, sp);
            double d = 0.0, e = 0.0;
            if (rc.owns) {
                const int r = rc.r;
                axc[r] = axn;
                const double dy = static_cast<double>(yc[r]) - static_cast<double>(y[r]);
                d = dy * dy;
                e = dy * (static_cast<double>(axn) - static_cast<double>(ax[r]));
            }
            d = warp_sum(d);
            e = warp_sum(e);
            if (lane == 0) {
                sums.own[Q.chunks + warp] = d;
                sums.own[Q.chunks + R.chunks + warp] = e;
            }
        }
        __syncthreads();
        double* all = it & 1 ? sums.all1 : sums.all0;
        unsigned long long* bar = it & 1 ? sums.bar1 : sums.bar0;
        if (waits.arms()) expect_bytes(bar, sums.bytes);
        const unsigned to = remote(bar, warp);   // warp w sends to CTA w
        for (int k = lane; k < Q.chunks + 2 * R.chunks && !waits.gave_up; k += 32) {
            const int at = k < Q.chunks ? static_cast<int>(rank) * a.AT.share.chunks + k
                           : k < Q.chunks + R.chunks
                               ? sums.cols + static_cast<int>(rank) * a.A.share.chunks + k - Q.chunks
                               : sums.cols + sums.rows + static_cast<int>(rank) * a.A.share.chunks + k - Q.chunks - R.chunks;
            send_one(remote(all + at, warp), sums.own[k], to);
        }
        waits.wait(bar, static_cast<unsigned>(it >> 1) & 1u);
        if (warp < 3) {
            const double t = warp == 0 ? tree_of_blocks(all, sums.cols)
                                       : tree_of_blocks(all + sums.cols + (warp - 1) * sums.rows, sums.rows);
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
        for (int r = threadIdx.x; r < R.rows; r += blockDim.x) commit(r);
        commit_columns();
    }
    __syncthreads();
    for (int r = threadIdx.x; r < R.rows; r += blockDim.x) {
        const int i = R.row0 + r;
        a.y[i] = y[r];
        a.y_sum[i] = ysum[r];
        a.ax[i] = ax[r];
        a.ax_prev[i] = axp[r];
    }
    for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) {
        const int j = Q.row0 + r;
        a.x[j] = x[r];
        a.x_sum[j] = xsum[r];
    }
    cluster_sync();   // every CTA has read the state, and none has sends in flight to another
    if (rank == 0 && threadIdx.x == 0) {
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
    if (waits.gave_up) *a.fail = 1.0;
}

template <class T, class V>
struct HalpernClusterArgs {
    TileCsrT<V> A, AT;
    T *x, *y;
    const T *x0, *y0, *c, *cl, *cu, *rl, *ru;
    const PdlpState* st;
    double* fail;
    int first, iterations;   // of the window
    int polls;               // of a wait
};

template <class T, class V>
inline size_t halpern_cluster_smem(const TileCsrT<V>& A, const TileCsrT<V>& AT) {
    using namespace cluster;
    if (A.ntiles == 0 || AT.ntiles == 0) return 0;
    return align16(kClusterWarps * kProducts * sizeof(T)) + slice_bytes(A) + slice_bytes(AT) + packed_bytes<T>(A) +
           packed_bytes<T>(AT) + send_bytes(A.share) + send_bytes(AT.share) + 4 * align16(sizeof(T) * A.share.rows) +
           6 * align16(sizeof(T) * AT.share.rows);
}

template <class T, class V>
__global__ void __launch_bounds__(cluster::kClusterThreads, 1)
    k_halpern_cluster(const __grid_constant__ HalpernClusterArgs<T, V> a) {
    using namespace cluster;
    extern __shared__ __align__(16) char smem[];
    const unsigned rank = cta_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Arena mem{smem};
    T* sp = mem.take<T>(kClusterWarps * kProducts) + warp * kProducts;
    if (lane < 2) sp[kChunkNnz + lane] = T(-0.0);
    Part<T, V> rows, cols;   // of A and of A'
    SendList xs_out, ys_out;
    load_parts(a.A, a.AT, rank, mem, &rows, &cols);
    const Slice<V>&R = rows.slice, &Q = cols.slice;
    Packed<T>&xv = rows.in, &yv = cols.in;   // the reflected point as R gathers it, y as Q gathers it
    const int mr = a.A.share.rows, nr = a.AT.share.rows;
    T *y = mem.take<T>(mr), *y0 = mem.take<T>(mr), *rl = mem.take<T>(mr), *ru = mem.take<T>(mr);
    T *x = mem.take<T>(nr), *x0 = mem.take<T>(nr), *xr = mem.take<T>(nr);
    T *c = mem.take<T>(nr), *cl = mem.take<T>(nr), *cu = mem.take<T>(nr);
    for (int r = threadIdx.x; r < R.rows; r += blockDim.x) {
        const int i = R.row0 + r;
        y[r] = a.y[i];
        y0[r] = a.y0[i];
        rl[r] = a.rl[i];
        ru[r] = a.ru[i];
    }
    for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) {
        const int j = Q.row0 + r;
        x[r] = a.x[j];
        x0[r] = a.x0[j];
        c[r] = a.c[j];
        cl[r] = a.cl[j];
        cu[r] = a.cu[j];
    }
    fill_packed(a.AT, yv, static_cast<const T*>(a.y));
    cluster_sync();
    make_sends(Q.row0, Q.rows, xv, a.AT.share, mem, &xs_out);
    make_sends(R.row0, R.rows, yv, a.A.share, mem, &ys_out);
    cluster_sync();
    Chunk<T, V> rc, qc;
    if (warp < R.chunks) rc.load(R, warp, xv.v);
    if (warp < Q.chunks) qc.load(Q, warp, yv.v);
    const T tau = static_cast<T>(a.st->eta / a.st->omega), sigma = static_cast<T>(a.st->eta * a.st->omega);
    Waits waits{xs_out, ys_out, a.polls};
    for (int it = 0; it < a.iterations; ++it) {
        const T lam = halpern_lambda<T>(a.st, a.first + it);
        if (warp < Q.chunks) {
            const T aty = qc.sum(Q, yv.v, sp);
            if (qc.owns) {
                const int r = qc.r;
                const T p = primal_reflected(x[r], aty, tau, c[r], cl[r], cu[r]);
                xr[r] = p;
                x[r] = primal_halpern_step(lam, p, x0[r]);
            }
        }
        exchange(waits, xs_out, xr, xv);
        if (warp < R.chunks) {
            const T axb = rc.sum(R, xv.v, sp);
            if (rc.owns) {
                const int r = rc.r;
                y[r] = dual_halpern_step(lam, dual_reflected(y[r], axb, sigma, rl[r], ru[r]), y0[r]);
            }
        }
        exchange(waits, ys_out, y, yv);
    }
    for (int r = threadIdx.x; r < R.rows; r += blockDim.x) a.y[R.row0 + r] = y[r];
    for (int r = threadIdx.x; r < Q.rows; r += blockDim.x) a.x[Q.row0 + r] = x[r];
    if (waits.gave_up) *a.fail = 1.0;
    cluster_sync();
}

}  // namespace
}  // namespace b200

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

struct FixedClusterArgs {
    TileCsr A, AT;
    const double *c, *cl, *cu, *tauv, *qdiag;  // tauv / sigv / qdiag may be null
    const double *rl, *ru, *sigv;
    double tau, sigma, theta;
    const double *x_in, *y_in;
    double *x_out, *y_out, *x_bar;  // x_bar: in and out
    double* part;                   // SK: max |y_new - y| of the last iteration, one per CTA
    int iterations;
    unsigned int* fail;             // set when a wait gave up
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

template <bool SK>
__global__ void __launch_bounds__(cluster::kClusterThreads, 1) k_fixed_cluster(const __grid_constant__ FixedClusterArgs a) {
    using namespace cluster;
    extern __shared__ __align__(16) char smem[];
    __shared__ double red[kClusterWarps];
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
    bool ok = true;
    for (int it = 0; it < a.iterations && ok; ++it) {
        const bool last = it + 1 == a.iterations;
        if (warp < R.chunks) {
            const double act = rc.sum(R, xv.v, sp);
            if (rc.owns) {
                const int r = rc.r;
                const double old = y[r];
                const double yn = SK ? dual_step_sk(old, act, sig[r], rl[r], ru[r])
                                     : dual_step_cuda(old, act, sig[r], rl[r], ru[r]);
                y[r] = yn;
                if (SK && last) change = fmax(change, fabs(dsub(yn, old)));
            }
        }
        ok = exchange(ys_out, y, yv);
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
        ok = exchange(xs_out, xb, xv) && ok;
    }
    if (!ok && threadIdx.x == 0) *a.fail = 1u;
    cluster_sync();
    for (int j = threadIdx.x; j < Q.rows; j += blockDim.x) {
        a.x_out[Q.row0 + j] = x[j];
        a.x_bar[Q.row0 + j] = xb[j];
    }
    for (int i = threadIdx.x; i < R.rows; i += blockDim.x) a.y_out[R.row0 + i] = y[i];
    if (SK) {
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

// Fixed-step PDHG iterations of a mid-size LP (or diagonal QP) in one cooperative launch.
#pragma once

#include "fixed_epi.cuh"
#include "flow.cuh"

namespace b200 {

constexpr int kFlowThreads = 512;
constexpr int kFlowWarps = kFlowThreads / 32;

struct FixedFlowArgs {
    TileCsr A, AT;
    const double *c, *cl, *cu, *tauv, *qdiag;  // tauv / sigv / qdiag may be null
    const double *rl, *ru, *sigv;
    double tau, sigma, theta;
    const double *x_in, *y_in;
    double *x_out, *y_out, *x_bar;  // x_bar: in and out
    double* part;                   // SK: max |y_new - y| of the last iteration, one per CTA
    flow::Tagged<double>*xt, *yt;   // x_bar and y by iteration
    unsigned long long first;       // number of this launch's first iteration; its start has the one before
    int iterations;
    int polls;                      // of a thread's waits in one iteration
    unsigned int* fail;
};

template <bool SK>
__global__ void __launch_bounds__(kFlowThreads, 1) k_fixed_flow(const __grid_constant__ FixedFlowArgs a) {
    using namespace flow;
    __shared__ double prod[kFlowWarps][kChunkNnz];
    __shared__ double red[kFlowWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = gridDim.x * kFlowWarps;
    const int mine = warp * gridDim.x + blockIdx.x;   // few chunks: on as many SMs as there are
    double* sp = prod[warp];
    double change = 0.0;
    for (int j = blockIdx.x * kFlowThreads + threadIdx.x; j < a.AT.rows; j += gridDim.x * kFlowThreads)
        store_tagged(a.xt + j, a.x_bar[j], a.first - 1);   // the point the launch starts from
    for (int it = 0; it < a.iterations; ++it) {
        const bool last = it + 1 == a.iterations;
        const unsigned long long tag = a.first + it;   // of this iteration's y and x_bar
        int left = a.polls;
        for (int t = mine; t < a.A.ntiles; t += nw) {
            const ChunkRows c = chunk_rows(a.A, t);
            const int i = c.row;
            double lo = 0.0, hi = 0.0, s = a.sigma, y = 0.0;
            if (c.owns) {
                lo = __ldg(a.rl + i);
                hi = __ldg(a.ru + i);
                if (a.sigv) s = __ldg(a.sigv + i);
                y = it == 0 ? a.y_in[i] : a.y_out[i];
            }
            const double act = chunk_sum(a.A, c, a.xt, tag - 1, sp, &left);
            if (c.owns) {
                const double yn = SK ? dual_step_sk(y, act, s, lo, hi) : dual_step_cuda(y, act, s, lo, hi);
                store_tagged(a.yt + i, yn, tag);
                a.y_out[i] = yn;
                if (SK && last) change = fmax(change, fabs(dsub(yn, y)));
            }
        }
        for (int t = mine; t < a.AT.ntiles; t += nw) {
            const ChunkRows c = chunk_rows(a.AT, t);
            const int j = c.row;
            double cj = 0.0, lo = 0.0, hi = 0.0, s = a.tau, qd = 0.0, x = 0.0;
            if (c.owns) {
                cj = __ldg(a.c + j);
                lo = __ldg(a.cl + j);
                hi = __ldg(a.cu + j);
                if (a.tauv) s = __ldg(a.tauv + j);
                if (a.qdiag) qd = __ldg(a.qdiag + j);
                x = it == 0 ? a.x_in[j] : a.x_out[j];
            }
            const double g = chunk_sum(a.AT, c, a.yt, tag, sp, &left);
            if (c.owns) {
                const double xn = SK ? primal_step_sk(x, g, cj, s, lo, hi, a.qdiag != nullptr, qd, 0.0)
                                     : primal_step_cuda(x, g, cj, s, lo, hi, a.qdiag != nullptr, qd, 0.0);
                const double xb = SK ? dsub(dmul(2.0, xn), x) : dadd(xn, dmul(a.theta, dsub(xn, x)));
                store_tagged(a.xt + j, xb, tag);
                a.x_out[j] = xn;
                if (last) a.x_bar[j] = xb;   // its reader above is through: this column's rows have moved on
            }
        }
        if (__any_sync(0xffffffffu, left <= 0)) {
            if (lane == 0) *a.fail = 1u;
            break;
        }
    }
    if (SK) {
        for (int o = 16; o > 0; o >>= 1) change = fmax(change, __shfl_xor_sync(0xffffffffu, change, o));
        if (lane == 0) red[warp] = change;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < kFlowWarps; ++k) change = fmax(change, red[k]);
            a.part[blockIdx.x] = change;
        }
    }
}

}  // namespace b200

// Batched PDHG: many independent LPs of uneven size advanced together in the
// same fused launches, each with the first-order loop of sk_solve
// (c/src/sk_solve.c:849-954): diagonal steps tau_j = 0.9/(1 + |A_:j|_1),
// sigma_i = 0.9/(1 + |A_i:|_1), x_bar = 2 x_new - x_old, and every
// check_every iterations its own gates: row violation <= primal_tol,
// max |x_bar - x| <= primal_tol * max(1, |x|_inf), max |y_new - y| <=
// dual_tol * (1 + anorm_k) with anorm_k = sqrt(max column mass * max row mass)
// of that LP.
//
// The batch is one block-diagonal CSR: LP k owns rows [row_seg[k], row_seg[k+1])
// and columns [col_seg[k], col_seg[k+1]). One PDHG iteration of the whole batch
// is the usual two fused launches (the A-side dual step, the A'-side primal
// step); a window of iterations is one CUDA graph. The gates are evaluated on
// the device with per-LP maxima (atomic max on the bit patterns of non-negative
// doubles, so the result does not depend on the order); an LP that passes is
// frozen (its iterates are carried through unchanged) and the host reads only
// the number of LPs still running. Where it is faster (plan_batch), each LP runs
// by itself on one CTA or a cluster of them instead (batch_cluster.cuh). Per LP the arithmetic is exactly the
// single-LP loop's, so every LP's iterates equal a separate solve's bit for bit.
#include "batch_cluster.cuh"
#include "batch_common.cuh"

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <limits>
#include <map>

namespace b200 {

namespace {

using batch::atomic_max_nonneg;
using batch::k_abs_sums;
using batch::sk_inf;
using batch::sk_neg_inf;
using batch::slot_value;

// sk_solve.c:901-906 with LP freezing
struct BatchDualEpi {
    const double* __restrict__ y;
    const double* __restrict__ rl;
    const double* __restrict__ ru;
    const double* __restrict__ sig;
    const int* __restrict__ seg;
    const int* __restrict__ done;
    double* __restrict__ y_new;
    using Acc = NoAcc;
    struct Row {
        double y, lo, hi, s;
        int frozen;
    };
    __device__ __forceinline__ Row load(int i) const { return Row{y[i], rl[i], ru[i], sig[i], done[seg[i]]}; }
    __device__ __forceinline__ void store(int i, double act, const Row& r, Acc&) const {
        if (r.frozen) {
            y_new[i] = r.y;
            return;
        }
        const double trial = dadd(r.y, dmul(r.s, act));
        y_new[i] = dsub(trial, dmul(r.s, box_sk(ddiv(trial, r.s), r.lo, r.hi)));
    }
    __device__ __forceinline__ void finish(Acc&, double*) const {}
};

// sk_solve.c:918-923 (LP, no Q) with LP freezing
struct BatchPrimalEpi {
    const double* __restrict__ x;
    const double* __restrict__ c;
    const double* __restrict__ tauv;
    const double* __restrict__ cl;
    const double* __restrict__ cu;
    const int* __restrict__ seg;
    const int* __restrict__ done;
    double* __restrict__ x_new;
    double* __restrict__ x_bar;
    using Acc = NoAcc;
    struct Row {
        double x, c, t, lo, hi;
        int frozen;
    };
    __device__ __forceinline__ Row load(int j) const { return Row{x[j], c[j], tauv[j], cl[j], cu[j], done[seg[j]]}; }
    __device__ __forceinline__ void store(int j, double g, const Row& r, Acc&) const {
        if (r.frozen) {
            x_new[j] = r.x;
            return;
        }
        double xn = dsub(r.x, dmul(r.t, dadd(dadd(r.c, 0.0), g)));
        xn = box_sk(xn, r.lo, r.hi);
        x_new[j] = xn;
        x_bar[j] = dsub(dmul(2.0, xn), r.x);
    }
    __device__ __forceinline__ void finish(Acc&, double*) const {}
};

// Check over rows: A x (stored as the activity), per-LP row violation
// (sk_solve.c:82-95) and max |y - y_prev| of the last iteration.
struct BatchRowsEpi {
    const double* __restrict__ y;
    const double* __restrict__ y_prev;
    const double* __restrict__ rl;
    const double* __restrict__ ru;
    const int* __restrict__ seg;
    const int* __restrict__ done;
    double* __restrict__ act_out;
    unsigned long long* __restrict__ viol;
    unsigned long long* __restrict__ dstep;
    using Acc = NoAcc;
    __device__ __forceinline__ void row(int i, double act, Acc&) const {
        const int k = seg[i];
        if (done[k]) return;
        act_out[i] = act;
        double v = 0.0;
        if (!sk_neg_inf(rl[i]) && rl[i] - act > v) v = rl[i] - act;
        if (!sk_inf(ru[i]) && act - ru[i] > v) v = act - ru[i];
        atomic_max_nonneg(&viol[k], v);
        atomic_max_nonneg(&dstep[k], fabs(y[i] - y_prev[i]));
    }
    __device__ __forceinline__ void finish(Acc&, double*) const {}
};

// slots[k] = max(slots[k], v) of the lanes that are in: one atomic a warp where they share an
// LP, as nearly all warps do (with one per element the atomics were the kernels' whole time:
// 1.1M columns of 512 LPs, 137 us for k_steps_and_max and 162 for k_batch_cols).
__device__ __forceinline__ void segment_max(unsigned long long* slots, int k, bool in, unsigned long long v) {
    const unsigned lanes = __ballot_sync(0xffffffffu, in);
    if (!lanes) return;
    const int lead = __shfl_sync(0xffffffffu, k, __ffs(lanes) - 1);
    if (__all_sync(0xffffffffu, !in || k == lead)) {
        if (!in) v = 0;
        for (int o = 16; o > 0; o >>= 1) v = max_u64(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0 && v) atomicMax(slots + lead, v);
    } else if (in && v) {
        atomicMax(slots + k, v);
    }
}

__global__ void k_batch_cols(int n, const double* __restrict__ x, const double* __restrict__ x_bar,
                             const int* __restrict__ seg, const int* __restrict__ done,
                             unsigned long long* __restrict__ scale, unsigned long long* __restrict__ step) {
    for (int b = blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < n; b += blockDim.x * gridDim.x) {
        const int j = b + (threadIdx.x & 31);
        const int k = j < n ? seg[j] : 0;
        const bool in = j < n && !done[k];
        const double v = in ? x[j] : 0.0;
        segment_max(scale, k, in, max_bits(fabs(v)));
        segment_max(step, k, in, in ? max_bits(fabs(x_bar[j] - v)) : 0ull);
    }
}

// One thread per LP: the gates of sk_solve.c:926-953; clears the maxima.
__global__ void k_batch_gate(int batch, int iteration, int last, double ptol, double dtol,
                             unsigned long long* __restrict__ viol, unsigned long long* __restrict__ dstep,
                             unsigned long long* __restrict__ scale, unsigned long long* __restrict__ step,
                             const unsigned long long* __restrict__ cmax, const unsigned long long* __restrict__ rmax,
                             int* __restrict__ done, int* __restrict__ iters, double* __restrict__ report,
                             unsigned int* __restrict__ remaining) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < batch; k += blockDim.x * gridDim.x) {
        if (done[k]) continue;
        const double v = slot_value(viol[k]), ds = slot_value(dstep[k]);
        const double sc = fmax(1.0, slot_value(scale[k])), st = slot_value(step[k]);
        const double anorm = sqrt(slot_value(cmax[k]) * slot_value(rmax[k]));
        report[4 * k + 0] = v;
        report[4 * k + 1] = st;
        report[4 * k + 2] = ds;
        report[4 * k + 3] = anorm;
        viol[k] = dstep[k] = scale[k] = step[k] = 0ull;
        iters[k] = iteration;
        if (v <= ptol && st <= ptol * sc && ds <= dtol * (1.0 + anorm)) {
            done[k] = 1;
        } else if (!last) {
            atomicAdd(remaining, 1u);
        }
    }
}

__global__ void k_steps_and_max(int len, const double* __restrict__ mass, const int* __restrict__ seg,
                                double* __restrict__ steps, unsigned long long* __restrict__ segmax) {
    for (int b = blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < len; b += blockDim.x * gridDim.x) {
        const int j = b + (threadIdx.x & 31);
        const double v = j < len ? mass[j] : 0.0;
        if (j < len) steps[j] = 0.9 / (1.0 + v);
        segment_max(segmax, j < len ? seg[j] : 0, j < len, max_bits(v));
    }
}

// Nonzeros of each LP.
__global__ void k_segment_entries(int batch, const int* __restrict__ row_seg, const int* __restrict__ ptr,
                                  int* __restrict__ out) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < batch; k += blockDim.x * gridDim.x)
        out[k] = ptr[row_seg[k + 1]] - ptr[row_seg[k]];
}

// Block-diagonal structure: every nonzero of row i lies in the columns of i's LP.
__global__ void k_check_blocks(int rows, const int* __restrict__ ptr, const int* __restrict__ idx,
                               const int* __restrict__ rseg, const int* __restrict__ cseg,
                               unsigned int* __restrict__ bad) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += blockDim.x * gridDim.x) {
        const int k = rseg[r];
        for (int p = ptr[r]; p < ptr[r + 1]; ++p)
            if (cseg[idx[p]] != k) { atomicOr(bad, 1u); break; }
    }
}

__global__ void k_init_box(int n, const double* __restrict__ lo, const double* __restrict__ hi,
                           double* __restrict__ x, double* __restrict__ x_bar) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += blockDim.x * gridDim.x) {
        const double v = box_sk(0.0, lo[j], hi[j]);
        x[j] = v;
        x_bar[j] = v;
    }
}

using batch::now_s;

constexpr int kClusterWindow = 4096;   // iterations of one launch of k_batch_cluster

// How the batch runs: on the launches (ctas 0) or on clusters of `ctas`, the `together` first of
// `order` by whole clusters and the others by single CTAs.
struct BatchPlan {
    int ctas = 0, together = 0;
    std::vector<int> order;
};

// Rule: the shorter time of an iteration by what was measured on a B200 (us; z: an LP's
// nonzeros, or 4 per row and column if those are more, in thousands):
//   a single CTA     1.8 + 1.1 z, 3 at least (3.0 at 0.4, 2.9 at 0.6, 8.5 at 6, 29 at 24, 69 at 60)
//   2 or 4 CTAs      4.5 + 1.1 z / n  (four: 8.3 at 6, 10.9 at 24, 22.5 at 60)
//   the launches     8.2 + 0.004 z of the whole batch, or 0.9 + 0.0139 z when longer, and 22 + 0.032 z a
//                    check; 2 + 0.0155 z at least
// those of CTAs with a check every 20 iterations, which is 0.8 of an iteration to them (512 LPs
// of 5 to 34 rows: launches 9.1 checked every 20, 8.8 every 100; CTAs, which the model without the least
// of 3 took, 10.7 and 10.2; 160 of 500 to 1,000 checked every 5: 26.1 and 14.3)
// and the largest LPs, longer than 0.85 of a CTA's even share, by whole clusters: 512 LPs of 50
// to 5,000 rows 63.3 by single CTAs, 57.6 with the largest by pairs, 98.0 on the launches;
// 296 of 500 rows 16.8, on the launches 26.3. Batches of a few LPs, where single CTAs leave the
// others idle, stay on the launches, as does one with an LP too large for a CTA's shared memory
// (some 19,000 rows and columns).
BatchPlan plan_batch(const TileCsr& A, const TileCsr& AT, int batch, const int* row_seg, const int* col_seg,
                     const std::vector<int>& entries, int every) {
    BatchPlan p;
    int rows_max = 0, cols_max = 0;
    for (int k = 0; k < batch; ++k) {
        rows_max = std::max(rows_max, row_seg[k + 1] - row_seg[k]);
        cols_max = std::max(cols_max, col_seg[k + 1] - col_seg[k]);
    }
    for (const void* at : {static_cast<const void*>(A.val), static_cast<const void*>(A.idx), static_cast<const void*>(AT.val),
                           static_cast<const void*>(AT.idx)})
        if (reinterpret_cast<std::uintptr_t>(at) % 16) return p;   // the copy engine's alignment
    const int slots = batch_clusters(1);
    if (batch_cluster_smem(cols_max, rows_max) > kBatchClusterSmem || slots == 0 || A.ntiles == 0 || AT.ntiles == 0) return p;
    p.order.resize(static_cast<size_t>(batch));
    for (int k = 0; k < batch; ++k) p.order[k] = k;
    auto size = [&](int k) {
        return std::max<long long>(entries[k], 4ll * (row_seg[k + 1] - row_seg[k] + col_seg[k + 1] - col_seg[k]));
    };
    std::stable_sort(p.order.begin(), p.order.end(), [&](int a, int b) { return size(a) > size(b); });
    const double total = A.nnz / 1000.0;
    auto alone = [&](int at) { return std::max(3.0, 1.8 + 1.1e-3 * size(p.order[at])); };
    double sum = 0.0;
    for (int k = 0; k < batch; ++k) sum += alone(k);
    int large = 0;
    while (large < batch && alone(large) > 0.85 * sum / slots) ++large;
    const double check = (22.0 + 0.032 * total) / every;
    const double launches = std::max({8.2 + 0.004 * total + check, 0.9 + 0.0139 * total + check, 2.0 + 0.0155 * total});
    double best = launches / 1.1 / ((1.0 + 0.8 / every) / 1.04);   // / 1.1: a near tie stays where it was
    for (int n : {1, 2, 4}) {
        const int by_clusters = n > 1 ? large : 0;
        if (batch_clusters(n) == 0) continue;
        double work = 0.0, longest = 0.0;
        for (int k = 0; k < batch; ++k) {
            const double t = k < by_clusters ? 4.5 + (alone(k) - 1.8) / n : alone(k);
            work += k < by_clusters ? n * t : t;
            longest = std::max(longest, t);
        }
        const double t = std::max(longest, work / slots);
        if (t < best) {
            best = t;
            p.ctas = n;
            p.together = by_clusters;
        }
    }
    return p;
}

}  // namespace

}  // namespace b200

using namespace b200;

extern "C" void sankhya_b200_batch_default_settings(SankhyaB200BatchSettings* s) {
    if (!s) return;
    std::memset(s, 0, sizeof(*s));
    s->struct_version = 1;
    s->max_iterations = 100000;
    s->check_every = 20;
    s->primal_tol = 1e-7;
    s->dual_tol = 1e-7;
    s->time_limit = 0.0;
}

extern "C" int sankhya_b200_batch_pdhg(const SankhyaCudaCSR* matrix, int batch, const int* row_segments,
                                       const int* col_segments, const double* c, const double* rlow,
                                       const double* rupp, const double* clow, const double* cupp,
                                       const SankhyaB200BatchSettings* settings, double* x_out, double* y_out,
                                       SankhyaB200BatchResult* results) {
    clear_error();
    (void)cudaGetLastError();
    SankhyaB200BatchSettings s;
    sankhya_b200_batch_default_settings(&s);
    if (settings) {
        if (settings->struct_version != 1) return fail_msg("unsupported settings struct_version");
        s = *settings;
    }
    if (!matrix || batch <= 0 || !row_segments || !col_segments || !c || !rlow || !rupp || !clow || !cupp || !x_out ||
        !results)
        return fail_msg("invalid batch arguments");
    if (s.max_iterations <= 0 || s.check_every <= 0 || !(s.primal_tol > 0.0) || !(s.dual_tol > 0.0) ||
        s.time_limit < 0.0)
        return fail_msg("invalid batch settings");
    const int m = matrix->rows, n = matrix->cols;
    if (row_segments[0] != 0 || col_segments[0] != 0 || row_segments[batch] != m || col_segments[batch] != n)
        return fail_msg("segments do not cover the matrix");
    for (int k = 0; k < batch; ++k)
        if (row_segments[k] > row_segments[k + 1] || col_segments[k] > col_segments[k + 1])
            return fail_msg("segments are not ordered");
    for (int j = 0; j < n; ++j)
        if (!std::isfinite(c[j]) || std::isnan(clow[j]) || std::isnan(cupp[j]) || clow[j] > cupp[j])
            return fail_msg("invalid cost or column bound");
    for (int i = 0; i < m; ++i)
        if (std::isnan(rlow[i]) || std::isnan(rupp[i]) || rlow[i] > rupp[i]) return fail_msg("invalid row bound");
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0) return fail_msg("no CUDA device available");
    std::shared_ptr<Plan> plan;
    if (get_plan(matrix, &plan)) return -1;
    const double t0 = now_s();
    cudaStream_t stream = engine_stream();

    // segment maps
    std::vector<int> rseg(static_cast<size_t>(m)), cseg(static_cast<size_t>(n));
    for (int k = 0; k < batch; ++k) {
        for (int i = row_segments[k]; i < row_segments[k + 1]; ++i) rseg[i] = k;
        for (int j = col_segments[k]; j < col_segments[k + 1]; ++j) cseg[j] = k;
    }
    const size_t nb = (static_cast<size_t>(n) * 8 + 255) / 256 * 256, mb = (static_cast<size_t>(m) * 8 + 255) / 256 * 256;
    const size_t kb = (static_cast<size_t>(batch) * 8 + 255) / 256 * 256;
    DevBuf blob;
    // 8 n-vectors + the column segment map, 7 m-vectors + the row segment map,
    // 15 per-LP slots, counters
    if (blob.alloc_on(stream, 9 * nb + 8 * mb + 15 * kb + 4096, "cudaMalloc batch workspace")) return -1;
    char* p = blob.as<char>();
    auto take = [&](size_t b) { char* r = p; p += b; return r; };
    double *dc = reinterpret_cast<double*>(take(nb)), *dcl = reinterpret_cast<double*>(take(nb)),
           *dcu = reinterpret_cast<double*>(take(nb)), *tau = reinterpret_cast<double*>(take(nb)),
           *xb0 = reinterpret_cast<double*>(take(nb)), *xb1 = reinterpret_cast<double*>(take(nb)),
           *xbar = reinterpret_cast<double*>(take(nb)), *cmass = reinterpret_cast<double*>(take(nb));
    double *drl = reinterpret_cast<double*>(take(mb)), *dru = reinterpret_cast<double*>(take(mb)),
           *sig = reinterpret_cast<double*>(take(mb)), *yb0 = reinterpret_cast<double*>(take(mb)),
           *yb1 = reinterpret_cast<double*>(take(mb)), *act = reinterpret_cast<double*>(take(mb)),
           *rmass = reinterpret_cast<double*>(take(mb));
    int* d_rseg = reinterpret_cast<int*>(take(mb));
    int* d_cseg = reinterpret_cast<int*>(take(nb));
    unsigned long long* viol = reinterpret_cast<unsigned long long*>(take(kb));
    unsigned long long* dstep = reinterpret_cast<unsigned long long*>(take(kb));
    unsigned long long* scale = reinterpret_cast<unsigned long long*>(take(kb));
    unsigned long long* step = reinterpret_cast<unsigned long long*>(take(kb));
    unsigned long long* cmax = reinterpret_cast<unsigned long long*>(take(kb));
    unsigned long long* rmax = reinterpret_cast<unsigned long long*>(take(kb));
    int* done = reinterpret_cast<int*>(take(kb));
    int* iters = reinterpret_cast<int*>(take(kb));
    double* report = reinterpret_cast<double*>(take(4 * kb));
    int* d_row_seg = reinterpret_cast<int*>(take(kb + 256));
    int* d_col_seg = reinterpret_cast<int*>(take(kb + 256));
    int* d_order = reinterpret_cast<int*>(take(kb));
    unsigned int* counters = reinterpret_cast<unsigned int*>(take(256));
    const size_t n8 = sizeof(double) * static_cast<size_t>(n), m8 = sizeof(double) * static_cast<size_t>(m);
    if (n) {
        B200_TRY(cudaMemcpyAsync(dc, c, n8, cudaMemcpyHostToDevice, stream), "upload c");
        B200_TRY(cudaMemcpyAsync(dcl, clow, n8, cudaMemcpyHostToDevice, stream), "upload clow");
        B200_TRY(cudaMemcpyAsync(dcu, cupp, n8, cudaMemcpyHostToDevice, stream), "upload cupp");
        B200_TRY(cudaMemcpyAsync(d_cseg, cseg.data(), sizeof(int) * n, cudaMemcpyHostToDevice, stream), "upload seg");
    }
    if (m) {
        B200_TRY(cudaMemcpyAsync(drl, rlow, m8, cudaMemcpyHostToDevice, stream), "upload rlow");
        B200_TRY(cudaMemcpyAsync(dru, rupp, m8, cudaMemcpyHostToDevice, stream), "upload rupp");
        B200_TRY(cudaMemcpyAsync(d_rseg, rseg.data(), sizeof(int) * m, cudaMemcpyHostToDevice, stream), "upload seg");
        B200_TRY(cudaMemsetAsync(yb0, 0, m8, stream), "zero y");
    }
    B200_TRY(cudaMemsetAsync(viol, 0, 6 * kb, stream), "zero maxima");
    B200_TRY(cudaMemsetAsync(done, 0, 2 * kb, stream), "zero flags");
    B200_TRY(cudaMemsetAsync(counters, 0, 256, stream), "zero counters");
    const TileCsr& A = plan->a;
    const TileCsr& AT = plan->at;
    const int ge = elem_grid(std::max(m, n));
    const size_t seg_bytes = sizeof(int) * (static_cast<size_t>(batch) + 1);
    B200_TRY(cudaMemcpyAsync(d_row_seg, row_segments, seg_bytes, cudaMemcpyHostToDevice, stream), "upload segments");
    B200_TRY(cudaMemcpyAsync(d_col_seg, col_segments, seg_bytes, cudaMemcpyHostToDevice, stream), "upload segments");
    if (m) k_segment_entries<<<elem_grid(batch), kThreads, 0, stream>>>(batch, d_row_seg, A.ptr, d_order);
    else B200_TRY(cudaMemsetAsync(d_order, 0, sizeof(int) * static_cast<size_t>(batch), stream), "zero entries");
    if (m) k_check_blocks<<<elem_grid(m), kThreads, 0, stream>>>(m, A.ptr, A.idx, d_rseg, d_cseg, counters + 1);
    if (m) k_abs_sums<<<elem_grid(m), kThreads, 0, stream>>>(m, A.ptr, A.val, rmass);
    if (n) k_abs_sums<<<elem_grid(n), kThreads, 0, stream>>>(n, AT.ptr, AT.val, cmass);
    if (n) k_steps_and_max<<<elem_grid(n), kThreads, 0, stream>>>(n, cmass, d_cseg, tau, cmax);
    if (m) k_steps_and_max<<<elem_grid(m), kThreads, 0, stream>>>(m, rmass, d_rseg, sig, rmax);
    if (n) k_init_box<<<elem_grid(n), kThreads, 0, stream>>>(n, dcl, dcu, xb0, xbar);
    B200_TRY(cudaGetLastError(), "batch setup");
    unsigned int* host_counters = reinterpret_cast<unsigned int*>(pinned_slot());
    if (!host_counters) return fail_msg("cudaMallocHost counters");
    std::vector<int> entries(static_cast<size_t>(batch));
    B200_TRY(cudaMemcpyAsync(host_counters, counters, 8, cudaMemcpyDeviceToHost, stream), "read");
    B200_TRY(cudaMemcpyAsync(entries.data(), d_order, sizeof(int) * batch, cudaMemcpyDeviceToHost, stream), "read");
    B200_TRY(cudaStreamSynchronize(stream), "batch setup");
    if (host_counters[1]) return fail_msg("matrix is not block-diagonal over the given segments");

    const BatchPlan way = plan_batch(A, AT, batch, row_segments, col_segments, entries, s.check_every);
    const int ctas = way.ctas;
    if (ctas) B200_TRY(cudaMemcpyAsync(d_order, way.order.data(), sizeof(int) * way.order.size(), cudaMemcpyHostToDevice, stream),
                       "upload order");

    double* xb[2] = {xb0, xb1};
    double* yb[2] = {yb0, yb1};
    const int grid_d = tiled_grid<BatchDualEpi>(A), grid_p = tiled_grid<BatchPrimalEpi>(AT);
    const int grid_r = tiled_grid<BatchRowsEpi>(A);
    std::map<std::pair<int, int>, cudaGraphExec_t> graphs;
    struct Graphs {
        std::map<std::pair<int, int>, cudaGraphExec_t>* g;
        ~Graphs() {
            for (auto& kv : *g)
                if (kv.second) cudaGraphExecDestroy(kv.second);
        }
    } graphs_guard{&graphs};
    int cur = 0, it = 0, launches = 0;
    auto iterate = [&]() {
        const int nx = cur ^ 1;
        launch_tiled(A, xbar, BatchDualEpi{yb[cur], drl, dru, sig, d_rseg, done, yb[nx]}, stream, grid_d);
        launch_tiled(AT, yb[nx], BatchPrimalEpi{xb[cur], dc, tau, dcl, dcu, d_cseg, done, xb[nx], xbar}, stream,
                     grid_p);
        cur = nx;
    };
    bool timed_out = false;
    int checks = 0;
    batch::LoopEvents loop_events(timing().level >= 1, stream);
    // On clusters: windows of whole checks, one check's with a time limit to look at.
    BatchClusterArgs on_clusters{A, AT, dc, dcl, dcu, tau, drl, dru, sig, xb0, xbar, yb0, d_row_seg, d_col_seg, d_order,
                                 cmax, rmax, done, iters, report, counters, counters + 2, counters + 4, way.together, batch, 0, 0, 0, 0,
                                 s.max_iterations, s.check_every, wait_limit(cluster::kMaxTries), s.primal_tol, s.dual_tol};
    for (int k = 0; k < batch; ++k) {
        on_clusters.rows_max = std::max(on_clusters.rows_max, row_segments[k + 1] - row_segments[k]);
        on_clusters.cols_max = std::max(on_clusters.cols_max, col_segments[k + 1] - col_segments[k]);
    }
    const int window = s.time_limit > 0.0 ? s.check_every : std::max(1, kClusterWindow / s.check_every) * s.check_every;
    while (ctas && it < s.max_iterations) {
        on_clusters.begin = it;
        on_clusters.end = it = static_cast<int>(std::min<long long>(static_cast<long long>(it) + window, s.max_iterations));
        B200_TRY(cudaMemsetAsync(counters, 0, 20, stream), "zero counters");
        B200_TRY(launch_batch_cluster(on_clusters, ctas, batch_clusters(ctas), stream), "cluster launch");
        ++launches;
        B200_TRY(cudaMemcpyAsync(host_counters, counters, 20, cudaMemcpyDeviceToHost, stream), "read");
        B200_TRY(cudaStreamSynchronize(stream), "batch check");
        if (host_counters[4]) return fail_msg("a wait inside the iteration kernel gave up");
        if (host_counters[0] == 0) break;
        if (s.time_limit > 0.0 && now_s() - t0 >= s.time_limit) {
            timed_out = true;
            break;
        }
    }
    while (!ctas && it < s.max_iterations) {
        const int next = std::min((it / s.check_every + 1) * s.check_every, s.max_iterations);
        int k = next - it;
        while (k > 0) {
            const int chunk = std::min(k, 64);
            auto key = std::make_pair(chunk, cur);
            auto g = graphs.find(key);
            if (g == graphs.end()) {
                const int saved = cur;
                cudaGraph_t graph;
                B200_TRY(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal), "begin capture");
                for (int i = 0; i < chunk; ++i) iterate();
                B200_TRY(cudaStreamEndCapture(stream, &graph), "end capture");
                cudaGraphExec_t exec;
                cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
                cudaGraphDestroy(graph);
                if (e != cudaSuccess) return fail_cuda("graph instantiate", e);
                g = graphs.emplace(key, exec).first;
                cur = saved;
            }
            B200_TRY(cudaGraphLaunch(g->second, stream), "graph launch");
            launches += 2 * chunk;
            cur ^= (chunk & 1);
            k -= chunk;
        }
        it = next;
        const bool last = it >= s.max_iterations;
        ++checks;
        B200_TRY(cudaMemsetAsync(counters, 0, 4, stream), "zero counter");
        launch_tiled(A, xb[cur], BatchRowsEpi{yb[cur], yb[cur ^ 1], drl, dru, d_rseg, done, act, viol, dstep}, stream,
                     grid_r);
        if (n) k_batch_cols<<<elem_grid(n), kThreads, 0, stream>>>(n, xb[cur], xbar, d_cseg, done, scale, step);
        k_batch_gate<<<elem_grid(batch), kThreads, 0, stream>>>(batch, it, last ? 1 : 0, s.primal_tol, s.dual_tol, viol,
                                                                dstep, scale, step, cmax, rmax, done, iters, report,
                                                                counters);
        launches += 3;
        B200_TRY(cudaMemcpyAsync(host_counters, counters, 4, cudaMemcpyDeviceToHost, stream), "read");
        B200_TRY(cudaStreamSynchronize(stream), "batch check");
        if (host_counters[0] == 0) break;
        if (s.time_limit > 0.0 && now_s() - t0 >= s.time_limit) {
            timed_out = true;
            break;
        }
    }
    const double loop_ms = loop_events.stop(stream);
    std::vector<int> h_done(static_cast<size_t>(batch)), h_iters(static_cast<size_t>(batch));
    std::vector<double> h_report(static_cast<size_t>(batch) * 4);
    B200_TRY(cudaMemcpyAsync(x_out, xb[cur], n8, cudaMemcpyDeviceToHost, stream), "download x");
    if (y_out && m) B200_TRY(cudaMemcpyAsync(y_out, yb[cur], m8, cudaMemcpyDeviceToHost, stream), "download y");
    B200_TRY(cudaMemcpyAsync(h_done.data(), done, sizeof(int) * batch, cudaMemcpyDeviceToHost, stream), "download");
    B200_TRY(cudaMemcpyAsync(h_iters.data(), iters, sizeof(int) * batch, cudaMemcpyDeviceToHost, stream), "download");
    B200_TRY(cudaMemcpyAsync(h_report.data(), report, sizeof(double) * 4 * batch, cudaMemcpyDeviceToHost, stream),
             "download");
    B200_TRY(cudaStreamSynchronize(stream), "batch download");
    if (ctas) {
        // the last check that an LP took
        it = *std::max_element(h_iters.begin(), h_iters.end());
        checks = (it + s.check_every - 1) / s.check_every;
    }
    for (int k = 0; k < batch; ++k) {
        SankhyaB200BatchResult& r = results[k];
        r.status = h_done[k] ? 0 : (timed_out ? 2 : 1);
        r.iterations = h_done[k] ? h_iters[k] : it;
        double obj = 0.0;
        for (int j = col_segments[k]; j < col_segments[k + 1]; ++j) obj += c[j] * x_out[j];
        r.objective = obj;
        r.row_violation = h_report[4 * k + 0];
        r.step = h_report[4 * k + 1];
        r.dual_step = h_report[4 * k + 2];
        r.anorm = h_report[4 * k + 3];
    }
    TimingState& ts = timing();
    ts.last = SankhyaB200Timing{};
    ts.last.iterations = it;
    ts.last.kernel_launches = launches;
    ts.last.checkpoints = checks;
    ts.last.loop_ms = loop_ms;
    return 0;
}

// Batched PDHG with one CTA, or a cluster of them, per LP: the LP's x_bar and y stay in the
// CTAs' shared memory, where the products gather them, and the LP runs all of its iterations
// and gates before the CTA takes the next one (largest first).
//
// As launches over the whole batch an iteration gathers from L1 and L2 at one element a cycle
// and SM and reads the matrix from HBM; 512 LPs of 50 to 5,000 rows (6.6M nonzeros) 98.0 us
// with its share of the checks, here 57.6 (148 LPs of 60,000 nonzeros 161 -> 69, 296 of 6,000
// 26 -> 17). It is bound by the shared-memory wavefronts of the gathers and of the row sums,
// whose order is fixed (the L1 data pipe is 62 % busy, shared memory 54 %; 74 % with the copies by
// cp.async, whose wavefronts the copy engine saves), then by the chain of a chunk: 24 warps hide it best (640
// threads 60.1, 896 59.2; two chunks in flight a warp needs registers that 24 warps do not
// have: 16 warps 76.6).
#pragma once

#include "batch_common.cuh"
#include "cluster.cuh"

#include <mutex>

namespace b200 {
namespace {

constexpr int kLpThreads = 768, kLpWarps = kLpThreads / 32;
constexpr int kLpMaxCtas = 4;
constexpr size_t kBatchClusterSmem = cluster::kMaxSmem - 1024;   // the static arrays take more than cluster.cuh's

struct BatchClusterArgs {
    TileCsr A, AT;
    const double *c, *cl, *cu, *tau, *rl, *ru, *sig;
    double *x, *x_bar, *y;
    const int *row_seg, *col_seg, *order;   // order: the LPs, largest first
    const unsigned long long *cmax, *rmax;
    int *done, *iters;
    double* report;
    unsigned int *remaining, *taken, *failed;   // LPs still running; LPs given to clusters and to CTAs; a wait gave up
    int together;                           // the first of `order`, each by a whole cluster
    int batch, cols_max, rows_max;          // the largest LP's
    int begin, end, max_iterations, every;  // iterations begin .. end of the run
    int tries;                              // polls of a wait
    double ptol, dtol;
};


__device__ __forceinline__ unsigned cluster_ctas() {
    unsigned n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return n;
}
__device__ __forceinline__ void store_remote(unsigned at, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ void store_remote(unsigned at, unsigned long long v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(at), "l"(v) : "memory");
}
__device__ __forceinline__ void store_remote(unsigned at, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

// The bits of a maximum of non-negative values, NaN above all (batch_common.cuh).
__device__ __forceinline__ unsigned long long max_bits(double v) {
    if (v > 0.0) return static_cast<unsigned long long>(__double_as_longlong(v));
    return isnan(v) ? 0x7ff8000000000000ull : 0ull;
}
__device__ __forceinline__ unsigned long long max_u64(unsigned long long a, unsigned long long b) { return a > b ? a : b; }

__device__ __forceinline__ unsigned shared_address(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ int lds_int(unsigned at) {
    int v;
    asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
    return v;
}

// A warp's chunk in shared memory, at `at`: the values, then their products in place; a -0.0,
// which adds nothing; the mbarrier of the copy; the columns. An entry more at either end, as
// the copy's 16-byte blocks ask for.
constexpr unsigned kPadAt = 8 * (kChunkNnz + 2), kBarAt = kPadAt + 8, kColumnsAt = kBarAt + 8,
                   kStageBytes = kColumnsAt + 4 * (kChunkNnz + 4);
struct Stage {
    unsigned at, phase;
    int tries;   // polls of a wait
    bool dead;   // a wait gave up: the warp starts no copy and gathers nothing any more

    __device__ __forceinline__ void init() {
        asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(at + kBarAt) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        cluster::sts(at + kPadAt, -0.0);
    }
    __device__ __forceinline__ void bulk(unsigned to, const void* from, unsigned bytes) const {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to),
                     "l"(from), "r"(bytes), "r"(at + kBarAt) : "memory");
    }
    // Starts the copy of entries [p0, p1); the lanes have fenced what they wrote here. The blocks
    // read hold an entry each, so they lie in the arrays' memory.
    __device__ __forceinline__ void fetch(const double* val, const int* idx, int p0, int p1) const {
        if ((threadIdx.x & 31) || dead) return;
        const unsigned n = p1 - p0;
        const unsigned v = 8u * (((p0 & 1u) + n + 1u) & ~1u), x = 4u * (((p0 & 3u) + n + 3u) & ~3u);
        asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(at + kBarAt), "r"(v + x) : "memory");
        bulk(at, val + (p0 & ~1), v);
        bulk(at + kColumnsAt, idx + (p0 & ~3), x);
    }
    __device__ __forceinline__ bool poll(int most) const {
        unsigned done = 0;
        for (int k = 0; !done && k < most; ++k)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
                         "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(at + kBarAt), "r"(phase) : "memory");
        return done != 0;
    }
    // All lanes come to the same answer. A dead warp has one copy in flight at most, which lands
    // in its own stage; drain waits for it before the CTA's shared memory goes.
    __device__ __forceinline__ void wait() {
        if (dead) return;
        dead = __any_sync(0xffffffffu, !poll(tries));
        phase ^= dead ? 0u : 1u;
    }
    __device__ __forceinline__ void drain() const { (void)poll(cluster::kMaxTries); }
};

// Rows [r0, r1) and entries [p0, p1) of a chunk, cut to the LP's rows.
struct Cut {
    int r0, p0, r1, p1;
};
template <class P>
struct Head {   // a lane's row: its entries in the chunk and what the step needs of it
    int q0, q1;
    P pre;
};

struct Rows {   // the LP's rows lo .. hi of M, for this warp its chunks first, first + step, ... below end
    const TileCsr& M;
    int first, end, step, lo, hi;
    __device__ __forceinline__ Cut cut(int t) const {
        if (t >= end) return Cut{0, 0, 0, 0};
        const int2 b0 = __ldg(M.tile + t), b1 = __ldg(M.tile + t + 1);
        Cut c{b0.x, b0.y, b1.x, b1.y};
        if (c.r0 < lo) {
            c.r0 = lo;
            c.p0 = __ldg(M.ptr + lo);
        }
        if (c.r1 > hi) {
            c.r1 = hi;
            c.p1 = __ldg(M.ptr + hi);
        }
        return c;
    }
    template <class Load>
    __device__ __forceinline__ auto head(const Cut& c, Load load) const {
        Head<decltype(load(0))> h{};
        const int my = c.r0 + static_cast<int>(threadIdx.x & 31);
        if (my < c.r1) {
            h.q0 = __ldg(M.ptr + my) - c.p0;
            h.q1 = __ldg(M.ptr + my + 1) - c.p0;
            h.pre = load(my);
        }
        return h;
    }
    // Whether a chunk's entries are copied: there are some, and no longer row, which is read
    // where it is summed.
    static __device__ __forceinline__ bool copied(const Cut& c) { return c.p1 > c.p0 && c.p1 - c.p0 <= kChunkNnz; }
    // Starts on the first chunk, before the barrier that the gathered vector waits for.
    template <class Load>
    __device__ __forceinline__ auto prime(const Stage& st, const Cut& c0, Load load) const {
        if (copied(c0)) st.fetch(M.val, M.idx, c0.p0, c0.p1);
        return head(c0, load);
    }
};

// The primed rows times the vector that `gather` reads, each summed as k_tiled sums it;
// apply(row, sum, loaded) takes the sum.
template <class P, class Gather, class Load, class Apply>
__device__ __forceinline__ void sweep(const Rows& R, Stage& st, Cut cur, Head<P> h, Gather gather, Load load, Apply apply) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    const TileCsr& M = R.M;
    for (int t = R.first; t < R.end; t += R.step) {
        const Cut next = R.cut(t + R.step);
        const bool owns = cur.r0 + lane < cur.r1;
        double s = 0.0;
        if (Rows::copied(cur)) st.wait();
        // without its copy the stage's columns are no columns of this LP: no entry is taken, and
        // the call fails
        const int n = st.dead ? 0 : cur.p1 - cur.p0;
        if (n > kChunkNnz) {
            double s0 = 0.0, s1 = 0.0;
            int p = cur.p0 + lane;
            for (; p + 32 < cur.p1; p += 64) {
                s0 = fma(__ldg(M.val + p), gather(__ldg(M.idx + p)), s0);
                s1 = fma(__ldg(M.val + p + 32), gather(__ldg(M.idx + p + 32)), s1);
            }
            if (p < cur.p1) s0 = fma(__ldg(M.val + p), gather(__ldg(M.idx + p)), s0);
            s = warp_sum(s0 + s1);
        } else {
            const unsigned sp = st.at + 8 * (cur.p0 & 1), sv = sp + 8 * lane;
            const unsigned sx = st.at + kColumnsAt + 4 * (cur.p0 & 3) + 4 * lane;
#pragma unroll
            for (int g = 0; g < kPerLane; g += 4) {
                double v[4];
                int j[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) j[k] = lds_int(sx + 128u * (g + k));
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = 32 * (g + k) + lane < n ? gather(j[k]) : 0.0;
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = dmul(cluster::lds<double, double>(sv + 256u * (g + k)), v[k]);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (32 * (g + k) + lane < n) cluster::sts(sv + 256u * (g + k), v[k]);
            }
            __syncwarp();
            const int len = owns && n ? h.q1 - h.q0 : 0;
            const int own_len = len <= kShortRow ? len : 0;
            const int longest = __reduce_max_sync(full, own_len);
            const unsigned e = sp + 8 * h.q0, end = e + 8 * own_len, pad = st.at + kPadAt;
            for (unsigned at = e; at < e + 8 * longest; at += 32) {
                const double e0 = cluster::lds<double, double>(at < end ? at : pad), e1 = cluster::lds<double, double>(at + 8 < end ? at + 8 : pad),
                             e2 = cluster::lds<double, double>(at + 16 < end ? at + 16 : pad), e3 = cluster::lds<double, double>(at + 24 < end ? at + 24 : pad);
                s = dadd(dadd(dadd(dadd(s, e0), e1), e2), e3);
            }
            unsigned long_rows = __ballot_sync(full, len > kShortRow);
            while (long_rows) {
                const int l = __ffs(long_rows) - 1;
                long_rows &= long_rows - 1;
                const int lq0 = __shfl_sync(full, h.q0, l), lq1 = __shfl_sync(full, h.q1, l);
                double w = 0.0;
                for (int q = lq0 + lane; q < lq1; q += 32) w += cluster::lds<double, double>(sp + 8 * q);
                w = warp_sum(w);
                if (lane == l) s = w;
            }
        }
        // what this lane wrote, before the copy engine writes over it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (Rows::copied(next)) st.fetch(M.val, M.idx, next.p0, next.p1);
        if (owns) apply(cur.r0 + lane, s, h.pre);
        h = R.head(next, load);
        __syncwarp();
        cur = next;
    }
}

inline size_t batch_cluster_smem(int cols_max, int rows_max) {
    return cluster::align16(8ull * cols_max) + cluster::align16(8ull * rows_max) + kLpWarps * kStageBytes;
}

__global__ void __launch_bounds__(kLpThreads, 1) k_batch_cluster(const __grid_constant__ BatchClusterArgs a) {
    using namespace cluster;
    extern __shared__ __align__(16) char smem[];
    __shared__ unsigned long long maxima[kLpWarps][4], got[kLpMaxCtas][4];
    __shared__ int given, range[4];
    const int all_rank = static_cast<int>(cta_rank()), all_ctas = static_cast<int>(cluster_ctas());
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Arena mem{smem};
    double* xb = mem.take<double>(a.cols_max);
    double* y = mem.take<double>(a.rows_max);
    const unsigned xb_at = shared_address(xb), y_at = shared_address(y);
    Stage stage{shared_address(mem.take<char>(kLpWarps * kStageBytes)) + warp * kStageBytes, 0u, a.tries, false};
    if (lane == 0) stage.init();
    bool together = all_ctas > 1;   // the largest LPs by all CTAs of the cluster, then each CTA its own
    if (together) cluster_sync();   // every CTA runs before its shared memory is written
    for (;;) {
        const int ctas = together ? all_ctas : 1, rank = together ? all_rank : 0;
        auto sync = [&] {
            if (ctas == 1) __syncthreads();
            else cluster_sync();
        };
        auto put = [&](double* at, double v) {   // at every CTA
            if (ctas == 1) *at = v;
            else
                for (int p = 0; p < ctas; ++p) store_remote(remote(at, p), v);
        };
        if (rank == 0 && threadIdx.x == 0) {
            const int q = together ? static_cast<int>(atomicAdd(a.taken, 1u)) : a.together + static_cast<int>(atomicAdd(a.taken + 1, 1u));
            given = q;
            for (int p = 1; p < ctas; ++p) store_remote(remote(&given, p), q);
        }
        sync();
        const int q = given;
        if (together && q >= a.together) {
            sync();   // all have read it
            together = false;
            continue;
        }
        if (q >= a.batch) break;
        const int lp = a.order[q];
        const int r0 = a.row_seg[lp], r1 = a.row_seg[lp + 1], c0 = a.col_seg[lp], c1 = a.col_seg[lp + 1];
        if (threadIdx.x < 4) {
            // the chunks that hold the LP's rows and columns: from the last that starts at or
            // before the first row, to the first that starts at or after the end
            const TileCsr& M = threadIdx.x < 2 ? a.A : a.AT;
            const int first = threadIdx.x < 2 ? r0 : c0, end = threadIdx.x < 2 ? r1 : c1;
            const int row = threadIdx.x & 1 ? end : first + 1;
            int lo = 0, hi = M.ntiles;   // first chunk that starts at `row` or after
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (__ldg(M.tile + mid).x >= row) hi = mid;
                else lo = mid + 1;
            }
            range[threadIdx.x] = threadIdx.x & 1 ? lo : (lo > 0 ? lo - 1 : 0);
        }
        for (int j = threadIdx.x; j < c1 - c0; j += blockDim.x) xb[j] = a.x_bar[c0 + j];
        for (int i = threadIdx.x; i < r1 - r0; i += blockDim.x) y[i] = a.y[r0 + i];
        bool running = a.done[lp] == 0;
        sync();
        const int step = ctas * kLpWarps, me = rank * kLpWarps + warp;
        const Rows rows{a.A, range[0] + me, r1 > r0 ? range[1] : 0, step, r0, r1};
        const Rows columns{a.AT, range[2] + me, c1 > c0 ? range[3] : 0, step, c0, c1};
        if (!running) continue;
        struct Row { double lo, hi, s; };
        struct Col { double x, c, t, lo, hi; };
        auto row = [&](int i) { return Row{__ldg(a.rl + i), __ldg(a.ru + i), __ldg(a.sig + i)}; };
        auto col = [&](int j) { return Col{a.x[j], __ldg(a.c + j), __ldg(a.tau + j), __ldg(a.cl + j), __ldg(a.cu + j)}; };
        const Cut rows0 = rows.cut(rows.first), columns0 = columns.cut(columns.first);
        auto hr = rows.prime(stage, rows0, row);
        for (int it = a.begin + 1; it <= a.end && running; ++it) {
            const bool check = it % a.every == 0 || it == a.max_iterations;
            unsigned long long dstep = 0, stepped = 0, scale = 0, viol = 0;
            sweep(rows, stage, rows0, hr, [=](int j) { return cluster::lds<double, double>(xb_at + 8 * (j - c0)); }, row,
                  [&](int i, double act, const Row& r) {
                      const double old = y[i - r0], trial = dadd(old, dmul(r.s, act));
                      const double yn = dsub(trial, dmul(r.s, box_sk(ddiv(trial, r.s), r.lo, r.hi)));
                      put(y + (i - r0), yn);
                      if (check) dstep = max_u64(dstep, max_bits(fabs(yn - old)));
                  });
            const auto hc = columns.prime(stage, columns0, col);
            sync();
            sweep(columns, stage, columns0, hc, [=](int i) { return cluster::lds<double, double>(y_at + 8 * (i - r0)); }, col,
                  [&](int j, double g, const Col& r) {
                      const double xn = box_sk(dsub(r.x, dmul(r.t, dadd(dadd(r.c, 0.0), g))), r.lo, r.hi);
                      const double bar = dsub(dmul(2.0, xn), r.x);
                      a.x[j] = xn;
                      put(xb + (j - c0), bar);
                      if (check) {
                          scale = max_u64(scale, max_bits(fabs(xn)));
                          stepped = max_u64(stepped, max_bits(fabs(bar - xn)));
                      }
                  });
            hr = rows.prime(stage, rows0, row);
            sync();
            if (!check) continue;
            // A x with x from memory (the other CTAs' part is in L2 since the barrier)
            sweep(rows, stage, rows0, hr, [&](int j) { return __ldcg(a.x + j); }, row,
                  [&](int, double act, const Row& r) {
                      double v = 0.0;
                      if (!batch::sk_neg_inf(r.lo) && r.lo - act > v) v = r.lo - act;
                      if (!batch::sk_inf(r.hi) && act - r.hi > v) v = act - r.hi;
                      viol = max_u64(viol, max_bits(v));
                  });
            hr = rows.prime(stage, rows0, row);
            unsigned long long v[4] = {viol, stepped, dstep, scale};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                for (int o = 16; o > 0; o >>= 1) v[k] = max_u64(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
                if (lane == 0) maxima[warp][k] = v[k];
            }
            __syncthreads();
            if (threadIdx.x < 4) {
                unsigned long long m = 0;
                for (int w = 0; w < kLpWarps; ++w) m = max_u64(m, maxima[w][threadIdx.x]);
                if (ctas == 1) got[0][threadIdx.x] = m;   // rank 0 of the cluster may have left by now
                else
                    for (int p = 0; p < ctas; ++p) store_remote(remote(&got[rank][threadIdx.x], p), m);
            }
            sync();
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = got[0][k];
                for (int p = 1; p < ctas; ++p) v[k] = max_u64(v[k], got[p][k]);
            }
            // the gates of sk_solve.c:926-953
            const double violation = batch::slot_value(v[0]), moved = batch::slot_value(v[1]), ds = batch::slot_value(v[2]);
            const double anorm = sqrt(batch::slot_value(a.cmax[lp]) * batch::slot_value(a.rmax[lp]));
            const bool met = violation <= a.ptol && moved <= a.ptol * fmax(1.0, batch::slot_value(v[3])) &&
                             ds <= a.dtol * (1.0 + anorm);
            running = !met;
            if (rank == 0 && threadIdx.x == 0) {
                a.report[4 * lp + 0] = violation;
                a.report[4 * lp + 1] = moved;
                a.report[4 * lp + 2] = ds;
                a.report[4 * lp + 3] = anorm;
                a.iters[lp] = it;
                if (met) a.done[lp] = 1;
                else if (it == a.end && it < a.max_iterations) atomicAdd(a.remaining, 1u);
            }
        }
        if (Rows::copied(rows0)) stage.wait();   // the copy for an iteration that does not come
        const int t0 = rank * kLpThreads + static_cast<int>(threadIdx.x);
        for (int i = t0; i < r1 - r0; i += ctas * kLpThreads) a.y[r0 + i] = y[i];
        for (int j = t0; j < c1 - c0; j += ctas * kLpThreads) a.x_bar[c0 + j] = xb[j];
    }
    if (stage.dead) {
        stage.drain();
        *a.failed = 1u;
    }
}

// Clusters of `ctas` CTAs that run at once on the current device; 0 when none fits (asked once
// per device).
inline int batch_clusters(int ctas) {
    struct Entry { int device, ctas, clusters; };
    static std::mutex mu;
    static std::vector<Entry> cache;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    for (const Entry& e : cache)
        if (e.device == device && e.ctas == ctas) return e.clusters;
    const void* kernel = reinterpret_cast<const void*>(&k_batch_cluster);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kLpThreads);
    cfg.dynamicSmemBytes = kBatchClusterSmem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kBatchClusterSmem)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        clusters = 0;
    }
    cache.push_back({device, ctas, clusters});
    return clusters;
}

inline cudaError_t launch_batch_cluster(const BatchClusterArgs& a, int ctas, int clusters, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas * clusters);
    cfg.blockDim = dim3(kLpThreads);
    cfg.dynamicSmemBytes = batch_cluster_smem(a.cols_max, a.rows_max);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_batch_cluster, a);
}

}  // namespace
}  // namespace b200

// Internal declarations of the B200 PDHG engine (not installed).
//
// Device layout of a matrix ("plan"), shared by every solve that uses it:
//   A    : the caller's CSR (int32 offsets / int32 columns / f64 values) plus a
//          row-tile schedule tile_row[0..ntiles] (see build_tiles)
//   A^T  : a second CSR holding the transpose (rows of A^T = columns of A, the
//          row indices of A ascending inside each), with its own tile schedule
// Both products are gathers, so every sum has a fixed order and results are
// bit-reproducible run to run.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <cmath>
#include <cstdint>
#include <memory>
#include <mutex>
#include <vector>

#include "sankhya_b200.h"
#include "sankhya_cuda.h"

namespace b200 {

// ------------------------------------------------------------------ errors

int fail_msg(const char* message);                 // sets last error, returns -1
int fail_cuda(const char* operation, cudaError_t); // sets last error, returns -1
void clear_error();

#define B200_TRY(expr, label)                                  \
    do {                                                       \
        cudaError_t b200_err_ = (expr);                        \
        if (b200_err_ != cudaSuccess) return fail_cuda(label, b200_err_); \
    } while (0)

// ----------------------------------------------------------- tile schedule

constexpr int kThreads = 256;          // threads per block (8 warps)
constexpr int kWarps = kThreads / 32;
constexpr int kChunkNnz = 256;         // nonzeros per warp chunk (8 per lane)
constexpr int kChunkRows = 32;         // rows per warp chunk (one owning lane each)
constexpr int kPerLane = kChunkNnz / 32;
constexpr int kShortRow = 32;          // rows up to this length: owning lane, sequential sum

// Warp chunks: consecutive rows with at most kChunkNnz nonzeros and at most
// kChunkRows rows; a row longer than kChunkNnz is a chunk of its own. Returns
// the chunk boundaries as (row, first nonzero) pairs, ntiles + 1 of them.
std::vector<int> build_tiles(int rows, const int* row_offsets);
// Stable transpose of a device CSR (rows x cols, nnz): tptr[cols + 1], tidx and
// tval receive A^T with each of its rows in ascending source-row order. Device
// work on `stream`; returns 0 or -1 (an index outside [0, cols) is an error).
int device_transpose(int rows, int cols, int nnz, const int* ptr, const int* idx, const double* val, int* tptr,
                     int* tidx, double* tval, cudaStream_t stream);

// Largest part of a CSR any CTA holds when the chunks of its schedule are split
// evenly and in order over the CTAs of one cluster (cluster.cuh); chunks 0: unknown.
// And what the whole matrix's rows are like.
struct Share {
    int rows = 0, nnz = 0, chunks = 0;
    int longest = 0;   // entries of the longest row
    int tree = 0;      // entries in rows beyond kShortRow, which a warp sums together
    int streamed = 0;  // of these, in rows beyond kChunkNnz
};
Share largest_share(const std::vector<int>& tiles, const int* row_offsets);

// A CSR with its warp-chunk schedule; T is the value type (double, or float
// for the FP32 inner iterations of the refined PDLP).
template <class T>
struct TileCsrT {
    int rows = 0, cols = 0, nnz = 0, ntiles = 0;
    Share share;
    const int* ptr = nullptr;
    const int* idx = nullptr;
    const T* val = nullptr;
    const int2* tile = nullptr;   // chunk boundaries: (first row, first nonzero)

    template <class U>
    TileCsrT<U> with_values(const U* v) const {
        TileCsrT<U> o;
        o.rows = rows; o.cols = cols; o.nnz = nnz; o.ntiles = ntiles; o.share = share;
        o.ptr = ptr; o.idx = idx; o.val = v; o.tile = tile;
        return o;
    }
};
using TileCsr = TileCsrT<double>;

// Owns everything a solve needs for one matrix beyond the caller's CSR.
struct Plan {
    int device = 0;
    TileCsr a;          // view of the caller's CSR + owned tiles
    TileCsr at;         // owned transpose + tiles
    int* d_tile_a = nullptr;
    int* d_at_ptr = nullptr;
    int* d_at_idx = nullptr;
    double* d_at_val = nullptr;
    int* d_tile_at = nullptr;
    int* d_a_idx = nullptr;         // owned copies of A when the caller's arrays are not
    double* d_a_val = nullptr;      // 16-byte aligned (the bulk L2 prefetch of a chunk needs it)
    const void* src_idx = nullptr;  // the handle's device_column_indices / device_values at
    const void* src_val = nullptr;  // planning time: a handle pointing elsewhere is another matrix
    double row_mass_max = 0.0;   // filled lazily by users that need it
    std::mutex workspace_mutex;   // held by the solve that uses `solve_cache`
    std::shared_ptr<void> solve_cache; // workspace + captured graphs of the last fixed-step solve
    ~Plan();
};

// Builds A^T and both tile schedules from host CSR arrays (host-side counting
// sort, O(nnz)). d_ptr/d_idx/d_val are the device copies of the same CSR.
int make_plan(const SankhyaCudaCSR* m, const int* h_ptr, const int* h_idx, const double* h_val,
              std::shared_ptr<Plan>* out);

// Registered plan of a handle made by sankhya_cuda_csr_create, else a plan
// built now from the handle's device arrays (copied back to the host once).
// Fails (-1) when the plan lives on another device than the current one: its
// arrays are that device's memory.
int get_plan(const SankhyaCudaCSR* m, std::shared_ptr<Plan>* out);
// Registered plan only (never builds one, never allocates): -1 with a message
// when the handle has none, points at other arrays than the planned ones, or the
// plan lives on another device than the current one.
int find_plan(const SankhyaCudaCSR* m, std::shared_ptr<Plan>* out);
void register_plan(const void* key, std::shared_ptr<Plan> plan);
bool unregister_plan(const void* key);   // whether it was the last

// ------------------------------------------------------------- streams/timing

cudaStream_t engine_stream();   // one non-blocking stream per host thread and device
int grid_for(const void* kernel, int ntiles, int dynamic_smem = 0);

struct TimingState {
    int level = 0;
    SankhyaB200Timing last{};
};
TimingState& timing();

// Polls after which a wait inside an iteration kernel gives up: `usual`, or what
// sankhya_b200_set_wait_limit set on this thread.
int wait_limit(int usual);

// ------------------------------------------------------- device arithmetic
// Explicit round-to-nearest intrinsics: no multiply-add contraction, so the
// elementwise updates round exactly like the reference's host C code.

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float dadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float dmul(float a, float b) { return __fmul_rn(a, b); }

// cuda/src/sankhya_cuda_lp.cu:13-17: only IEEE infinities are absent bounds. The bounds
// were validated (no lower bound of +inf, no upper one of -inf), so an infinite one never
// compares true and needs no test of its own.
__device__ __forceinline__ double box_ieee(double v, double lo, double hi) {
    if (v < lo) v = lo;
    if (v > hi) v = hi;
    return v;
}
// c/src/sk_solve.c:18-24: the 1e30 sentinel (SK_INFINITY) marks absent bounds.
__device__ __forceinline__ double box_sk(double v, double lo, double hi) {
    if (!(lo <= -1.0e30) && v < lo) v = lo;
    if (!(hi >= 1.0e30) && v > hi) v = hi;
    return v;
}
__device__ __forceinline__ bool has_lower_gate(double v) { return isfinite(v) && v > -5.0e29; }
__device__ __forceinline__ bool has_upper_gate(double v) { return isfinite(v) && v < 5.0e29; }

// ------------------------------------------------------------- reductions

struct NoAcc {
    static constexpr int kSlots = 0;
    __device__ __forceinline__ void init() {}
};

// NS reduction slots; bit k of SumMask set = slot k is a sum, else a max.
template <int NS, unsigned SumMask>
struct Slots {
    static constexpr int kSlots = NS;
    double v[NS];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int k = 0; k < NS; ++k) v[k] = 0.0;
    }
    __device__ __forceinline__ void max(int k, double x) { v[k] = fmax(v[k], x); }
    __device__ __forceinline__ void add(int k, double x) { v[k] += x; }
};

template <unsigned SumMask>
__device__ __forceinline__ double slot_op(int k, double a, double b) {
    return ((SumMask >> k) & 1u) ? a + b : fmax(a, b);
}

// Fixed-shape block reduction; thread 0's result lands in partial[blockIdx.x*NS+k].
template <int NS, unsigned SumMask>
__device__ void block_store(Slots<NS, SumMask>& acc, double* __restrict__ partial, double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        double v = acc.v[k];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            v = slot_op<SumMask>(k, v, __shfl_xor_sync(0xffffffffu, v, off));
        if (lane == 0) smem[warp * NS + k] = v;
    }
    __syncthreads();
    if (threadIdx.x < NS) {
        const int k = threadIdx.x;
        double r = smem[k];
        for (int w = 1; w < kWarps; ++w) r = slot_op<SumMask>(k, r, smem[w * NS + k]);
        partial[blockIdx.x * NS + k] = r;
    }
    __syncthreads();
}

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// --------------------------------------------------- fused tiled SpMV kernel
//
// Warp-granular: every warp of a persistent grid walks warp chunks
// gw, gw + total_warps, ... independently (no block-wide barrier on the path).
// For a chunk of rows [r0, r1) and nonzeros [p0, p1):
//   0. lane 0 asks the TMA unit to pull the warp's NEXT chunk of values and
//      column indices into L2 (cp.async.bulk.prefetch.L2, no shared memory, no
//      completion to wait for), so that chunk's loads below hit L2, not HBM;
//   1. lane l owns row r0 + l and prefetches that row's epilogue data
//      (Epi::load: y, bounds, steps, ...) into registers;
//   2. lane l loads values and column indices p0 + l + 32 k (k < 8, coalesced,
//      evict-first) and issues its 8 gathers v[idx] back to back (the vectors
//      stay L2-resident);
//   3. products go to the warp's 2 KB shared-memory slice; rows of at most
//      kShortRow entries are summed by their owning lane sequentially in stored
//      order from 0.0 (the exact rounding of a serial CPU loop), longer rows by
//      the whole warp (lane-strided partials, xor tree);
//   4. Epi::store / Epi::row finishes the PDHG step for the row.
// A row longer than kChunkNnz is a chunk of its own, streamed by the warp.
// Reducing epilogues keep per-thread accumulators; Epi::finish combines them
// per block in a fixed order.

struct Empty {};

template <class E, class = void>
struct HasLoad {
    static constexpr bool value = false;
};
template <class E>
struct HasLoad<E, decltype(void(&E::load))> {
    static constexpr bool value = true;
};

template <class Epi, bool = HasLoad<Epi>::value>
struct RowPre {
    using type = Empty;
    static __device__ __forceinline__ type load(const Epi&, int) { return {}; }
    template <class T>
    static __device__ __forceinline__ void apply(const Epi& e, int r, T s, const type&, typename Epi::Acc& acc) {
        e.row(r, s, acc);
    }
};
template <class Epi>
struct RowPre<Epi, true> {
    using type = typename Epi::Row;
    static __device__ __forceinline__ type load(const Epi& e, int r) { return e.load(r); }
    template <class T>
    static __device__ __forceinline__ void apply(const Epi& e, int r, T s, const type& pre, typename Epi::Acc& acc) {
        e.store(r, s, pre, acc);
    }
};

// Bulk L2 prefetch of [first, last) elements of a 16-byte-aligned array; the
// range is shrunk to its 16-byte-aligned interior so it never leaves the array.
template <class T>
__device__ __forceinline__ void prefetch_l2(const T* base, int first, int last) {
    constexpr int per = 16 / static_cast<int>(sizeof(T));
    const int a = (first + per - 1) / per * per, b = last / per * per;
    if (b > a)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(base + a),
                     "r"(static_cast<unsigned>((b - a) * static_cast<int>(sizeof(T))))
                     : "memory");
}

// A stored matrix value as the arithmetic type T (the identity unless the values
// are kept narrower than the vectors, e.g. bf16 values with fp32 vectors).
template <class T, class V>
__device__ __forceinline__ T load_value(const V* p) {
    return static_cast<T>(__ldcs(p));
}
template <>
__device__ __forceinline__ float load_value<float, __nv_bfloat16>(const __nv_bfloat16* p) {
    return __bfloat162float(__ldcs(p));
}

// Before a product: what does not depend on the kernel before it in the stream, whose blocks may
// still be running (launch_early): the first chunk on its way to L2. After the wait that kernel is
// complete and its writes are visible to ordinary loads, so the gathered vector is read by those
// and not by the read-only path. A grid of up to kEarlyBlocks lets the next one in at once; a
// larger one only as its blocks leave, since blocks let in at once do not spread over the chip as
// those of a launch of its own. A x and A'y, us for both, at once / as the blocks leave / launched
// one after the other: 13 and 20 blocks 6.9 / 6.7 / 10.3 (a restarted QP's iteration there 16.2 /
// 17.6 / 17.6), 33 and 43 blocks 7.3 / 7.1 / 11.2, 63 10.3 / 7.9 / 12.3, 118 14.3 / 8.3 / 12.3, 157
// 24.9 / 10.3 / 13.8, 254 26.8 / 11.0 / 14.7.
constexpr int kEarlyBlocks = 24;
template <class V>
__device__ __forceinline__ void start_early(const TileCsrT<V>& A, int t) {
    if (gridDim.x <= kEarlyBlocks) asm volatile("griddepcontrol.launch_dependents;");
    if (t < A.ntiles && (threadIdx.x & 31) == 0) {
        const int2 b0 = __ldg(A.tile + t), b1 = __ldg(A.tile + t + 1);
        if (b1.y - b0.y <= kChunkNnz) {
            prefetch_l2(A.val, b0.y, b1.y);
            prefetch_l2(A.idx, b0.y, b1.y);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The chunks t, t + nw, ... of one warp, its products in sp.
template <class Epi, class T, class V>
__device__ __forceinline__ void tile_rows(const TileCsrT<V>& A, const T* v, const Epi& epi,
                                          typename Epi::Acc& acc, T* sp, int t, int nw) {
    using P = RowPre<Epi>;
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    int2 b0 = t < A.ntiles ? __ldg(A.tile + t) : make_int2(0, 0);
    int2 b1 = t < A.ntiles ? __ldg(A.tile + t + 1) : make_int2(0, 0);
    for (; t < A.ntiles; t += nw) {
        const int r0 = b0.x, r1 = b1.x, p0 = b0.y, p1 = b1.y;
        const int tn = t + nw;
        int2 n0 = b1, n1 = b1;
        if (tn < A.ntiles) {
            n0 = __ldg(A.tile + tn);
            n1 = __ldg(A.tile + tn + 1);
            if (lane == 0 && n1.y - n0.y <= kChunkNnz) {
                prefetch_l2(A.val, n0.y, n1.y);
                prefetch_l2(A.idx, n0.y, n1.y);
            }
        }
        const int my = r0 + lane;
        const bool owns = my < r1;
        typename P::type pre{};
        int q0 = 0, q1 = 0;
        if (owns) {
            pre = P::load(epi, my);
            q0 = __ldg(A.ptr + my) - p0;
            q1 = __ldg(A.ptr + my + 1) - p0;
        }
        if (p1 - p0 > kChunkNnz) {
            T s0 = T(0), s1 = T(0);
            int p = p0 + lane;
            for (; p + 32 < p1; p += 64) {
                s0 += load_value<T>(A.val + p) * v[__ldcs(A.idx + p)];
                s1 += load_value<T>(A.val + p + 32) * v[__ldcs(A.idx + p + 32)];
            }
            if (p < p1) s0 += load_value<T>(A.val + p) * v[__ldcs(A.idx + p)];
            const T s = warp_sum(s0 + s1);
            if (lane == 0) P::apply(epi, r0, s, pre, acc);
            b0 = n0;
            b1 = n1;
            continue;
        }
        int col[kPerLane];
        T a[kPerLane];
#pragma unroll
        for (int k = 0; k < kPerLane; ++k) {
            const int p = p0 + 32 * k + lane;
            col[k] = 0;
            a[k] = T(0);
            if (p < p1) {
                col[k] = __ldcs(A.idx + p);
                a[k] = load_value<T>(A.val + p);
            }
        }
#pragma unroll
        for (int k = 0; k < kPerLane; ++k)
            if (p0 + 32 * k + lane < p1) a[k] = dmul(a[k], v[col[k]]);
#pragma unroll
        for (int k = 0; k < kPerLane; ++k)
            if (p0 + 32 * k + lane < p1) sp[32 * k + lane] = a[k];
        __syncwarp();
        const int len = q1 - q0;
        if (owns && len <= kShortRow) {
            T s = T(0);
            for (int q = q0; q < q1; ++q) s = dadd(s, sp[q]);
            P::apply(epi, my, s, pre, acc);
        }
        unsigned long_rows = __ballot_sync(full, owns && len > kShortRow);
        while (long_rows) {
            const int l = __ffs(long_rows) - 1;
            long_rows &= long_rows - 1;
            const int lq0 = __shfl_sync(full, q0, l), lq1 = __shfl_sync(full, q1, l);
            T s = T(0);
            for (int q = lq0 + lane; q < lq1; q += 32) s += sp[q];
            s = warp_sum(s);
            if (lane == l) P::apply(epi, my, s, pre, acc);
        }
        __syncwarp();
        b0 = n0;
        b1 = n1;
    }
}

template <class Epi, class T, class V = T>
__global__ void __launch_bounds__(kThreads) k_tiled(TileCsrT<V> A, const T* v, Epi epi) {
    __shared__ T prod[kWarps][kChunkNnz];
    __shared__ double red[kWarps * 8];
    typename Epi::Acc acc;
    acc.init();
    const int warp = threadIdx.x >> 5;
    start_early(A, blockIdx.x * kWarps + warp);
    tile_rows(A, v, epi, acc, prod[warp], blockIdx.x * kWarps + warp, gridDim.x * kWarps);
    epi.finish(acc, red);
}

// Plain product y = A v.
template <class T = double>
struct StoreEpiT {
    T* y;
    using Acc = NoAcc;
    __device__ __forceinline__ void row(int r, T s, NoAcc&) const { y[r] = s; }
    __device__ __forceinline__ void finish(NoAcc&, double*) const {}
};
using StoreEpi = StoreEpiT<double>;

template <class Epi, class T = double, class V = T>
inline int tiled_grid(const TileCsrT<V>& A) {
    const void* k = reinterpret_cast<const void*>(&k_tiled<Epi, T, V>);
    return grid_for(k, (A.ntiles + kWarps - 1) / kWarps, 0);
}

// Launches a kernel that waits by itself for the one before it in the stream (start_early), so
// that its launch and its blocks' start overlap that one's end. A x and A'y by turns, us for both:
// 2,000 x 5,000 10.2 -> 6.9, 50,021 x 100,003 22.9 -> 16.2; an iteration with a Hessian at
// 100,000 x 200,000 39.9 -> 37.0; at 1,000,000 x 2,000,000 268 both ways.
template <class... P, class... Args>
inline int launch_early(void (*kernel)(P...), int grid, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    return 0;
}

template <class Epi, class T, class V>
inline int launch_tiled(const TileCsrT<V>& A, const T* v, const Epi& epi, cudaStream_t stream, int grid) {
    if (A.ntiles == 0) return 0;
    return launch_early(k_tiled<Epi, T, V>, grid, stream, A, v, epi);
}

// Two independent products in one launch: the warps go on to B's chunks where A's end, so that
// neither a second launch's start nor its last, part-filled wave is waited for.
template <class Epi, class EpiB>
__global__ void __launch_bounds__(kThreads) k_tiled_pair(TileCsr A, const double* v, Epi epi, TileCsr B, const double* w, EpiB epi_b) {
    __shared__ double prod[kWarps][kChunkNnz];
    __shared__ double red[kWarps * 8];
    typename Epi::Acc acc;
    acc.init();
    const int warp = threadIdx.x >> 5, t = blockIdx.x * kWarps + warp, nw = gridDim.x * kWarps;
    start_early(A, t);
    tile_rows(A, v, epi, acc, prod[warp], t, nw);
    NoAcc none;
    tile_rows(B, w, epi_b, none, prod[warp], (t + nw - A.ntiles % nw) % nw, nw);
    epi.finish(acc, red);
}
template <class Epi, class EpiB>
inline int tiled_pair_grid(const TileCsr& A, const TileCsr& B) {
    return grid_for(reinterpret_cast<const void*>(&k_tiled_pair<Epi, EpiB>), (A.ntiles + B.ntiles + kWarps - 1) / kWarps, 0);
}

// Final fixed-order combine of per-block partials: out[k] = op_g partial[g*NS+k].
template <int NS, unsigned SumMask>
__global__ void k_combine(const double* __restrict__ partial, int nblocks, double* __restrict__ out) {
    __shared__ double smem[kThreads];
    for (int k = 0; k < NS; ++k) {
        double r = 0.0;
        for (int g = threadIdx.x; g < nblocks; g += kThreads) r = slot_op<SumMask>(k, r, partial[g * NS + k]);
        smem[threadIdx.x] = r;
        __syncthreads();
        for (int s = kThreads / 2; s > 0; s >>= 1) {
            if (threadIdx.x < s) smem[threadIdx.x] = slot_op<SumMask>(k, smem[threadIdx.x], smem[threadIdx.x + s]);
            __syncthreads();
        }
        if (threadIdx.x == 0) out[k] = smem[0];
        __syncthreads();
    }
}

// ------------------------------------------------------------- small kernels

__global__ void k_fill(double* __restrict__ out, double value, int n);
__global__ void k_copy(double* __restrict__ dst, const double* __restrict__ src, int n);

inline int elem_grid(int n) {
    int g = (n + kThreads - 1) / kThreads;
    return g < 1 ? 1 : (g > 148 * 16 ? 148 * 16 : g);
}

// ---------------------------------------------------------- device buffers

// Device memory that is kept between solves, at most kPoolBytes of it idle per device: a
// pool of this library's own with stream-ordered allocation. Null where the device has none.
// What is idle goes back when an allocation here would fail otherwise, by
// sankhya_b200_release_memory, and, but for kPoolRest, with the last matrix handle (all of it would cost
// a program that makes and drops a handle per small solve 0.5 ms of 1.9 a time).
constexpr unsigned long long kPoolBytes = 1ull << 30, kPoolRest = 64ull << 20;
cudaMemPool_t solve_pool();
void trim_pools(unsigned long long keep);
cudaError_t device_malloc(void** p, size_t bytes);   // cudaMalloc, once more after trim_pools

// A pinned host slot of kPinnedSlot doubles for small results, one per thread; null when
// it cannot be had.
constexpr int kPinnedSlot = 64;
double* pinned_slot();

// Owning device array: cudaMalloc / cudaFree (alloc), for what outlives a call, or memory
// of the solve pool (alloc_on), for what one call uses on one stream. A call's cudaMalloc
// and cudaFree each wait for the whole device and took 0.05 to 0.4 ms, with stalls of tens
// to hundreds of milliseconds now and then; from the pool the same takes microseconds.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    bool pooled = false;
    cudaStream_t stream = nullptr;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (!p) return;
        if (pooled) cudaFreeAsync(p, stream);   // after the work enqueued on the stream so far
        else cudaFree(p);
        p = nullptr;
    }
    int alloc(size_t b, const char* what) {
        release();
        bytes = b;
        pooled = false;
        if (b == 0) return 0;
        cudaError_t e = device_malloc(&p, b);
        if (e != cudaSuccess) { p = nullptr; return fail_cuda(what, e); }
        return 0;
    }
    int alloc_on(cudaStream_t s, size_t b, const char* what) {
        release();
        cudaMemPool_t pool = b ? solve_pool() : nullptr;
        if (pool && cudaMallocFromPoolAsync(&p, b, pool, s) == cudaSuccess) {
            bytes = b;
            pooled = true;
            stream = s;
            return 0;
        }
        if (pool) (void)cudaGetLastError();
        p = nullptr;
        return alloc(b, what);
    }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

}  // namespace b200

// Small LPs on one thread-block cluster: many PDHG iterations in one launch.
//
// A launch of the fused product is bound by latency when the LP is small: at 2,000 x
// 5,000 with 25,000 nonzeros one iteration moves under 1 MB, all of it L2-resident,
// yet two graph launches took 7.7 us (launch, tile bounds -> offsets -> indices ->
// gather -> store, drain). Here a cluster of kClusterCtas CTAs keeps the whole problem
// on chip for a window of iterations. Each CTA owns a run of the chunks of A and one of
// A' (values, offsets and indices in shared memory) and keeps, of each gathered vector,
// just the elements its entries name, packed in index order; its indices point into that
// packed copy. After a step the owner of a range sends each CTA the elements of the range
// that CTA needs (a prepared list, contiguous at the destination) with st.async, which
// counts the bytes on the destination's mbarrier: a CTA goes on when its own copy is
// complete, and every gather is a local shared-memory read. No cluster-wide barrier is
// needed: CTA s sends x to CTA c exactly when c sends y to s (both mean that A has an
// entry in c's rows and s's columns), so s, which waits for c's y before it computes its
// next x, cannot overwrite an x that c has yet to read. What an exchange costs is packets:
// 12.8 bytes per SM and cycle for contiguous stores of any width and for bulk copies, and
// a partly filled packet costs a whole one, so the elements are packed per destination (a
// full copy of both vectors in every CTA took 4.7 us an iteration at 2,000 x 5,000).
//
// Row sums keep the order of k_tiled (rows up to kShortRow by their owner in stored
// order, longer ones by the warp's strided partials and xor tree, rows beyond
// kChunkNnz streamed with two partials), so every iterate has the same bits.
#pragma once

#include "engine.cuh"

namespace b200 {
namespace cluster {

constexpr int kClusterCtas = 16;       // non-portable size; checked with cudaOccupancyMaxActiveClusters
constexpr int kClusterThreads = 512;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kMaxSteps = 4096;       // iterations per launch: some ten milliseconds
constexpr int kMaxTries = 1 << 20;    // of a wait, each of up to some microseconds
constexpr int kMaxSmem = 226 * 1024;     // dynamic; the rest of the 227 KB holds the static arrays

__device__ __forceinline__ unsigned cta_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// All threads of all CTAs; earlier shared-memory writes (also to other CTAs) are visible after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Writes v to the shared-memory address `at` of a CTA and counts its bytes on the mbarrier
// `bar` of the same CTA.
__device__ __forceinline__ void send_one(unsigned at, double v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(at),
                 "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void send_one(unsigned at, float v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(at),
                 "r"(__float_as_uint(v)), "r"(bar) : "memory");
}

// Address of *p of the CTA `c` (p in this CTA's shared memory; every CTA has the same layout).
__device__ __forceinline__ unsigned remote(const void* p, unsigned c) {
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(at) : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(c));
    return at;
}
__device__ __forceinline__ unsigned load_remote(unsigned addr) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ unsigned load_remote16(unsigned addr) {
    unsigned short v;
    asm volatile("ld.shared::cluster.u16 %0, [%1];" : "=h"(v) : "r"(addr) : "memory");
    return v;
}

inline size_t align16(size_t b) { return (b + 15) / 16 * 16; }

// An mbarrier that one thread of the CTA arms with the bytes of an exchange.
__device__ __forceinline__ void init_barrier(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void expect_bytes(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(bar))), "r"(bytes) : "memory");
}
// False when the wait gave up after `most` polls; true at once with `skip`.
__device__ __forceinline__ bool wait_bytes(unsigned long long* bar, unsigned phase, int most, bool skip = false) {
    unsigned done = skip;
    for (int tries = 0; !done && tries < most; ++tries)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done)
                     : "r"(static_cast<unsigned>(__cvta_generic_to_shared(bar))), "r"(phase) : "memory");
    return done != 0;
}

// ------------------------------------------------------------ one CTA's part

// One CTA's chunks of a matrix, in shared memory. Rows and entries count from the slice's
// first; idx points into the packed copy of the gathered vector.
template <class V>
struct Slice {
    V* val;
    int* ptr;
    int* first;          // first row of each chunk, chunks + 1 of them
    unsigned short* idx;
    int row0, rows, chunks;
};

// The vector a matrix's products gather: this CTA's packed copy, which elements it holds
// (bit per element of the whole vector, and the count of set bits before each word), and
// the mbarrier that counts the arriving bytes of one exchange.
template <class T>
struct Packed {
    T* v;
    unsigned* bits;
    unsigned short* before;
    unsigned long long* bar;
    unsigned bytes;   // of one exchange
    unsigned phase;
};

// What this warp sends after the CTA has computed its own elements: elements
// src[0 .. count) go to consecutive addresses from `at` in CTA number `warp`.
struct SendList {
    unsigned short* src;
    int count;
    unsigned at, bar;
};

// Shared-memory sizes of the three for matrix M (rows of M own elements of one vector, its
// columns index the other). Sized by the largest share, so that every CTA's layout is the same.
template <class V>
__host__ __device__ inline size_t slice_bytes(const TileCsrT<V>& M) {
    const size_t nnz = static_cast<size_t>(M.share.nnz);
    return (nnz * sizeof(V) + 15) / 16 * 16 + ((M.share.rows + 1) * 4ull + 15) / 16 * 16 +
           ((M.share.chunks + 1) * 4ull + 15) / 16 * 16 + (nnz * 2 + 15) / 16 * 16;
}
__host__ __device__ inline int packed_length(int cols, const Share& s) { return cols < s.nnz ? cols : s.nnz; }
template <class T, class V>
__host__ __device__ inline size_t packed_bytes(const TileCsrT<V>& M) {
    const size_t words = (static_cast<size_t>(M.cols) + 31) / 32;
    return (static_cast<size_t>(packed_length(M.cols, M.share)) * sizeof(T) + 15) / 16 * 16 + (words * 4 + 15) / 16 * 16 +
           (words * 2 + 15) / 16 * 16 + 16;
}
// own elements x CTAs at most, and at most one (element, CTA) pair per entry
__host__ __device__ inline int send_length(const Share& s) {
    return s.nnz < s.rows * kClusterCtas ? s.nnz : s.rows * kClusterCtas;
}
__host__ __device__ inline size_t send_bytes(const Share& s) {
    return (send_length(s) * 2ull + 15) / 16 * 16;
}

// Inclusive sums over the lanes.
__device__ __forceinline__ int warp_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

struct Arena {
    char* at;
    template <class X>
    __device__ __forceinline__ X* take(size_t count) {
        X* r = reinterpret_cast<X*>(at);
        at += (count * sizeof(X) + 15) / 16 * 16;
        return r;
    }
};

// A CTA's part of one matrix.
template <class T, class V>
struct Part {
    Slice<V> slice;
    Packed<T> in;
    int2 first;   // row and entry at which the slice starts
    int nnz;

    __device__ __forceinline__ void place(const TileCsrT<V>& M, unsigned rank, Arena& mem) {
        const Share& s = M.share;
        const int words = (M.cols + 31) / 32;
        slice.val = mem.take<V>(s.nnz);
        slice.ptr = mem.take<int>(s.rows + 1);
        slice.first = mem.take<int>(s.chunks + 1);
        slice.idx = mem.take<unsigned short>(s.nnz);
        in.v = mem.take<T>(packed_length(M.cols, s));
        in.bits = mem.take<unsigned>(words);
        in.before = mem.take<unsigned short>(words);
        in.bar = mem.take<unsigned long long>(1);
        in.phase = 0;
        const int t0 = min(M.ntiles, static_cast<int>(rank) * s.chunks), t1 = min(M.ntiles, t0 + s.chunks);
        const int2 end = __ldg(M.tile + t1);
        first = __ldg(M.tile + t0);
        nnz = end.y - first.y;
        slice.row0 = first.x;
        slice.rows = end.x - first.x;
        slice.chunks = t1 - t0;
        for (int w = threadIdx.x; w < words; w += blockDim.x) in.bits[w] = 0u;
        if (threadIdx.x == 0) init_barrier(in.bar);
        for (int k = threadIdx.x; k <= slice.chunks; k += blockDim.x) slice.first[k] = __ldg(M.tile + t0 + k).x - first.x;
    }
    __device__ __forceinline__ void fetch(const TileCsrT<V>& M) const {
        for (int r = threadIdx.x; r <= slice.rows; r += blockDim.x) slice.ptr[r] = __ldg(M.ptr + first.x + r) - first.y;
#pragma unroll 4
        for (int p = threadIdx.x; p < nnz; p += blockDim.x) {
            const int j = __ldg(M.idx + first.y + p);
            const V v = M.val[first.y + p];
            atomicOr(in.bits + (j >> 5), 1u << (j & 31));
            slice.val[p] = v;
        }
    }
    __device__ __forceinline__ void count(int cols) const {   // one warp
        const int words = (cols + 31) / 32, lane = threadIdx.x & 31;
        int run = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int w = w0 + lane, c = w < words ? __popc(in.bits[w]) : 0;
            const int incl = warp_scan(c);
            if (w < words) in.before[w] = static_cast<unsigned short>(run + incl - c);
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __device__ __forceinline__ void remap(const TileCsrT<V>& M) {
        const int words = (M.cols + 31) / 32;
        in.bytes = words ? static_cast<unsigned>(sizeof(T)) * (in.before[words - 1] + __popc(in.bits[words - 1])) : 0u;
#pragma unroll 4
        for (int p = threadIdx.x; p < nnz; p += blockDim.x) {
            const int j = __ldg(M.idx + first.y + p), w = j >> 5;
            slice.idx[p] = static_cast<unsigned short>(in.before[w] + __popc(in.bits[w] & ((1u << (j & 31)) - 1u)));
        }
    }
};

// Copies this CTA's chunks of both matrices into shared memory and finds the elements they
// gather. Ends with a block barrier; other CTAs may read `in` after the next cluster barrier.
template <class T, class V>
__device__ __forceinline__ void load_parts(const TileCsrT<V>& A, const TileCsrT<V>& AT, unsigned rank, Arena& mem,
                                           Part<T, V>* a, Part<T, V>* at) {
    a->place(A, rank, mem);
    at->place(AT, rank, mem);
    __syncthreads();
    a->fetch(A);
    at->fetch(AT);
    __syncthreads();
    if (threadIdx.x < 32) a->count(A.cols);
    else if (threadIdx.x < 64) at->count(AT.cols);
    __syncthreads();
    a->remap(A);
    at->remap(AT);
    __syncthreads();
}

// Fills this CTA's packed copy from a whole vector in global memory.
template <class T, class V>
__device__ __forceinline__ void fill_packed(const TileCsrT<V>& M, const Packed<T>& in, const T* __restrict__ whole) {
    for (int j = threadIdx.x; j < M.cols; j += blockDim.x) {
        const unsigned b = in.bits[j >> 5], bit = 1u << (j & 31);
        if (b & bit) in.v[in.before[j >> 5] + __popc(b & (bit - 1u))] = whole[j];
    }
}

// This warp's send list of the elements [row0, row0 + rows) that the CTA owns of the vector
// that `in` describes (the destination's copy of `in` is read: a cluster barrier before).
template <class T>
__device__ __forceinline__ void make_sends(int row0, int rows, const Packed<T>& in, const Share& s, Arena& mem,
                                           SendList* out) {
    static_assert(kClusterWarps == kClusterCtas, "a warp per destination");
    __shared__ int counts[kClusterCtas];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    out->src = mem.take<unsigned short>(send_length(s));
    // the words of the destination's bits that cover [row0, row0 + rows), a lane each
    const int w0 = row0 >> 5, words = rows > 0 ? ((row0 + rows - 1) >> 5) - w0 + 1 : 0;
    const unsigned bits = remote(in.bits + w0, c);
    auto word = [&](int w) {
        if (w >= words) return 0u;
        unsigned b = load_remote(bits + 4u * w);
        const int lo = row0 - 32 * (w0 + w), hi = row0 + rows - 32 * (w0 + w);   // bits [lo, hi) are ours
        if (lo > 0) b &= ~0u << lo;
        if (hi < 32) b &= (1u << hi) - 1u;
        return b;
    };
    int count = 0;
    for (int w = lane; w - lane < words; w += 32) count += __reduce_add_sync(full, __popc(word(w)));
    if (lane == 0) counts[c] = count;
    __syncthreads();
    for (int k = 0; k < c; ++k) out->src += counts[k];
    out->count = count;
    out->bar = remote(in.bar, c);
    out->at = remote(in.v, c);
    if (count > 0) {
        out->at += static_cast<unsigned>(sizeof(T)) *
                   (load_remote16(remote(in.before + w0, c)) + __popc(load_remote(bits) & ((1u << (row0 & 31)) - 1u)));
        int run = 0;
        for (int w = lane; w - lane < words; w += 32) {
            unsigned b = word(w);
            const int incl = warp_scan(__popc(b));
            for (int k = run + incl - __popc(b); b; b &= b - 1u)
                out->src[k++] = static_cast<unsigned short>(32 * (w0 + w) + __ffs(b) - 1 - row0);
            run += __shfl_sync(full, incl, 31);
        }
    }
    __syncthreads();
}

// The waits of one thread, one of which may give up where other threads of the CTA see the same
// phase end. Such a thread waits once more (bounded) for what is on its way to the CTA, then
// sends, arms and waits no more but passes every block barrier as before: an early exit would
// leave the others there. Whoever waits for its elements gives up in turn, so the launch ends
// after a few limits, its sums garbage, its addresses as ever. (A test of all threads, by a
// barrier that reduces or a flag read behind one, took 1 to 2 % of a small solve.)
struct Waits {
    SendList &xs, &ys;
    const int& polls;   // of a wait
    bool gave_up = false;

    // Thread 0 arms: it knows by its own waits that the phase before has ended.
    __device__ __forceinline__ bool arms() const { return threadIdx.x == 0 && !gave_up; }
    __device__ __forceinline__ void wait(unsigned long long* bar, unsigned phase) {
        if (wait_bytes(bar, phase, polls, gave_up)) return;
        (void)wait_bytes(bar, phase, kMaxTries);
        gave_up = true;
        xs.count = ys.count = 0;
    }
};

// Sends the CTA's own elements to the CTAs that gather them, and waits until this CTA's
// packed copy has all of its elements. `meanwhile` runs while the elements are on their way.
template <class T, class F>
__device__ __forceinline__ void exchange(Waits& w, const SendList& s, const T* own, Packed<T>& in, F meanwhile) {
    __syncthreads();   // `own` is complete
    if (w.arms()) expect_bytes(in.bar, in.bytes);
    for (int k = threadIdx.x & 31; k < s.count; k += 32)
        send_one(s.at + static_cast<unsigned>(sizeof(T)) * k, own[s.src[k]], s.bar);
    meanwhile();
    w.wait(in.bar, in.phase);
    in.phase ^= 1u;
}

template <class T>
__device__ __forceinline__ void exchange(Waits& w, const SendList& s, const T* own, Packed<T>& in) {
    exchange(w, s, own, in, [] {});
}

// Shared-memory loads that stay where they are written: the entries of a batch are all
// requested before the first of them is used (the compiler otherwise moves each load
// behind the test of whether its entry exists, one memory latency per entry).
__device__ __forceinline__ unsigned smem_at(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ unsigned lds_u16(unsigned at) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at));
    return v;
}
template <class T, class V>
__device__ __forceinline__ T lds(unsigned at);
template <>
__device__ __forceinline__ double lds<double, double>(unsigned at) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at));
    return v;
}
template <>
__device__ __forceinline__ float lds<float, float>(unsigned at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at));
    return v;
}
template <>
__device__ __forceinline__ float lds<float, __nv_bfloat16>(unsigned at) {
    return __uint_as_float(lds_u16(at) << 16);
}
__device__ __forceinline__ void sts(unsigned at, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}
__device__ __forceinline__ void sts(unsigned at, float v) {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}
// Products of one warp's chunk, and one slot that holds -0.0: s + (-0.0) is s for every s,
// so a lane whose row has ended adds that slot and no add waits for a predicate.
constexpr int kProducts = kChunkNnz + 2;

// A chunk as one warp works on it: its entries in registers (lane l: entries l + 32 k, as
// k_tiled takes them) and the row of each lane.
template <class T, class V>
struct Chunk {
    T a[kPerLane];
    unsigned g[kPerLane];   // shared-memory addresses of the gathered elements
    int r;                  // local row of this lane
    int q0, len;            // its entries within the chunk; len 0 without a row
    bool owns;
    int n0, n1;             // the chunk's entries; more than kChunkNnz: one streamed row

    __device__ __forceinline__ void load(const Slice<V>& S, int j, const T* v) {
        const int lane = threadIdx.x & 31;
        const int r0 = S.first[j], r1 = S.first[j + 1];
        n0 = S.ptr[r0];
        n1 = S.ptr[r1];
        r = r0 + lane;
        owns = r < r1;
        q0 = owns ? S.ptr[r] - n0 : 0;
        len = owns ? S.ptr[r + 1] - n0 - q0 : 0;
#pragma unroll
        for (int k = 0; k < kPerLane; ++k) {
            const int p = n0 + 32 * k + lane;
            const bool live = p < n1;
            a[k] = live ? lds<T, V>(smem_at(S.val) + static_cast<unsigned>(sizeof(V)) * p) : T(0);
            g[k] = smem_at(v) + (live ? static_cast<unsigned>(sizeof(T)) * lds_u16(smem_at(S.idx) + 2u * p) : 0u);
        }
    }

    // The sum of this lane's row (whole warps), in k_tiled's order: rows up to kShortRow by
    // their owner in stored order, longer ones by strided partials and the xor tree. `sp`:
    // the warp's kProducts slots in shared memory, the last two -0.0.
    __device__ __forceinline__ T sum(const Slice<V>& S, const T* v, T* sp) const {
        const unsigned full = 0xffffffffu;
        const int lane = threadIdx.x & 31;
        const unsigned sz = static_cast<unsigned>(sizeof(T));
        if (n1 - n0 > kChunkNnz) {
            T s0 = T(0), s1 = T(0);
            auto value = [&](int q) { return lds<T, V>(smem_at(S.val) + static_cast<unsigned>(sizeof(V)) * q); };
            auto gather = [&](int q) { return v[S.idx[q]]; };
            int p = n0 + lane;
            for (; p + 32 < n1; p += 64) {
                s0 = fma(value(p), gather(p), s0);
                s1 = fma(value(p + 32), gather(p + 32), s1);
            }
            if (p < n1) s0 = fma(value(p), gather(p), s0);
            return warp_sum(s0 + s1);
        }
        const unsigned at = smem_at(sp);
        T e[kPerLane];
#pragma unroll
        for (int k = 0; k < kPerLane; ++k) e[k] = lds<T, T>(g[k]);
#pragma unroll
        for (int k = 0; k < kPerLane; ++k) sts(at + sz * (32 * k + lane), dmul(a[k], e[k]));
        __syncwarp();
        T s = T(0);
        const int n = len <= kShortRow ? len : 0;
        const int most = __reduce_max_sync(full, n);
        // eight entries at a time, the next eight requested before these are added
#pragma unroll
        for (int k = 0; k < 8; ++k) e[k] = lds<T, T>(at + sz * (k < n ? q0 + k : kChunkNnz));
        for (int b = 8; b < most; b += 8) {
            T f[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) f[k] = lds<T, T>(at + sz * (b + k < n ? q0 + b + k : kChunkNnz));
#pragma unroll
            for (int k = 0; k < 8; ++k) s = dadd(s, e[k]);
#pragma unroll
            for (int k = 0; k < 8; ++k) e[k] = f[k];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) s = dadd(s, e[k]);
        unsigned long_rows = __ballot_sync(full, len > kShortRow);
        while (long_rows) {
            const int l = __ffs(long_rows) - 1;
            long_rows &= long_rows - 1;
            const int a0 = __shfl_sync(full, q0, l), al = __shfl_sync(full, len, l);
            T t = T(0);
            for (int q = lane; q < al; q += 32) t = dadd(t, lds<T, T>(at + sz * (a0 + q)));
            t = warp_sum(t);
            if (lane == l) s = t;
        }
        __syncwarp();
        return s;
    }
};

// Chunks in whole blocks of eight, as the launches have them (at most 32 blocks: a CTA has at
// most a chunk per warp).
inline __host__ __device__ int padded_chunks(int ntiles) { return (ntiles + 7) / 8 * 8; }

// Sums of 8 chunks from v, at most 32 of them, by the tree over 256 blocks (one warp): its
// levels 128, 64 and 32 add zeros.
__device__ __forceinline__ double tree_of_blocks(const double* v, int padded) {
    const int lane = threadIdx.x & 31;
    auto leaf = [&](int g) {
        double e[8], r = 0.0;
        if (8 * g >= padded) return r;
#pragma unroll
        for (int w = 0; w < 8; ++w) e[w] = v[8 * g + w];
        r = e[0];
#pragma unroll
        for (int w = 1; w < 8; ++w) r = r + e[w];
        return r;
    };
    return warp_sum(leaf(lane));
}

// Whether a cluster of kClusterCtas CTAs of `kernel`, each with all of the shared
// memory, fits the current device (asked once per kernel and device, which also sets
// the kernel's attributes).
bool available(const void* kernel);

// Launches `kernel(args)` as one cluster on `stream`.
template <class Args>
inline cudaError_t launch(void (*kernel)(Args), const Args& args, size_t smem, cudaStream_t stream) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kClusterCtas);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kClusterCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args);
}

}  // namespace cluster
}  // namespace b200

// Mid-size LPs: many PDHG iterations in one cooperative launch, without barriers.
//
// Above the size that fits one cluster (cluster.cuh) and up to about a million nonzeros an
// iteration's launches are still mostly latency: 8.8 us for two at 8,000 x 16,000 with
// 128,000 nonzeros, where the gathers take 0.5 us each. Here every warp keeps its chunks
// of A and A' for a window of iterations, and an iterate's element travels as one aligned
// access (16 bytes in FP64, 8 in FP32) that holds the value and the number of its
// iteration: whoever gathers it reads until the number is the one it needs. So a step of
// the whole grid costs a store's way to L2 and a load's way back (2,300 cycles), where a
// grid barrier takes 2,400 and the gathers come on top, and the matrix stays in L1, which
// a barrier's acquire would empty. A read that comes too early makes the store's line
// travel again, so a lane first waits for its first entry alone.
//
// No element is overwritten before it has been read: a row's owner stores its next y only
// after it has gathered x from all the columns of the row, and those columns' owners have
// stored that x after they gathered this y (A and A' have the same entries). All CTAs are
// resident (cooperative launch), so every wait ends; each is bounded all the same. A warp (in
// the adaptive loop a CTA) whose wait gave up leaves as a whole, since the sums need all lanes;
// those that wait for its elements give up in turn.
//
// Row sums keep k_tiled's order, so every iterate has the same bits.
//
// Measured on a B200 at 1,965 MHz, us per fixed-step iteration, launches -> this: 8,000 x
// 16,000 with 128,000 nonzeros 8.7 -> 4.3; 15,000 x 30,000 (300,000) 10.9 -> 5.6; 30,000 x
// 60,000 (480,000) 13.1 -> 7.1; 50,000 x 100,000 (1M) 17.8 -> 13.4; 120,000 x 250,000 (2M)
// 31.9 -> 25.2; 300,000 x 600,000 (4.8M) 67.3 -> 66.7. With columns of up to 1,000 entries:
// 128,000 9.6 -> 5.1; 480,000 13.3 -> 12.9; 1.2M 22.8 -> 25.2. Below some 45,000 nonzeros the
// cluster is ahead (25,000: 2.8 against 3.8; 42,000: 3.8 against 3.9).
#pragma once

#include "engine.cuh"

#include <algorithm>

namespace b200 {
namespace flow {

constexpr int kMaxPolls = 1 << 22;    // loads of a thread's waits in one iteration, some seconds

// An element and the iteration it belongs to, read and written as one access.
template <class T>
struct Tagged;
template <>
struct alignas(16) Tagged<double> {
    double value;
    unsigned long long tag;
};
template <>
struct alignas(8) Tagged<float> {
    float value;
    unsigned tag;
};

__device__ __forceinline__ Tagged<double> load_tagged(const Tagged<double>* p) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi) : "l"(p) : "memory");
    return Tagged<double>{__longlong_as_double(static_cast<long long>(lo)), hi};
}
__device__ __forceinline__ Tagged<float> load_tagged(const Tagged<float>* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return Tagged<float>{__uint_as_float(static_cast<unsigned>(v)), static_cast<unsigned>(v >> 32)};
}
__device__ __forceinline__ void store_tagged(Tagged<double>* p, double v, unsigned long long tag) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(tag) : "memory");
}
__device__ __forceinline__ void store_tagged(Tagged<float>* p, float v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"(static_cast<unsigned long long>(__float_as_uint(v)) | static_cast<unsigned long long>(tag) << 32)
                 : "memory");
}

template <class T>
struct TagOf { using type = unsigned long long; };
template <>
struct TagOf<float> { using type = unsigned; };

// Waits for the element of iteration `want`. `left` counts down over all of a thread's
// waits of an iteration; at 0 nothing is waited for any more.
template <class T>
__device__ __forceinline__ T wait_element(const Tagged<T>* p, typename TagOf<T>::type want, int* left) {
    Tagged<T> e = load_tagged(p);
    while (e.tag != want && --*left > 0) e = load_tagged(p);
    return e.value;
}

template <class T, class V>
__device__ __forceinline__ T value_at(const V* p) { return static_cast<T>(__ldg(p)); }
template <>
__device__ __forceinline__ float value_at<float, __nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(__ldg(p)); }

// A chunk as one warp sees it: its bounds and the row of each lane.
struct ChunkRows {
    int p0, p1;        // entries
    int row, q0, len;  // this lane's row and its entries within the chunk; len 0 without one
    bool owns;
};
template <class V>
__device__ __forceinline__ ChunkRows chunk_rows(const TileCsrT<V>& A, int t) {
    const int2 b0 = __ldg(A.tile + t), b1 = __ldg(A.tile + t + 1);
    ChunkRows c;
    c.p0 = b0.y;
    c.p1 = b1.y;
    c.row = b0.x + static_cast<int>(threadIdx.x & 31);
    c.owns = c.row < b1.x;
    c.q0 = c.owns ? __ldg(A.ptr + c.row) - b0.y : 0;
    c.len = c.owns ? __ldg(A.ptr + c.row + 1) - b0.y - c.q0 : 0;
    return c;
}

// The sum of this lane's row (whole warps), in k_tiled's order, of the elements of
// iteration `want` of v. `sp`: the warp's kChunkNnz products. (The row beyond a chunk waits
// entry by entry on purpose: requesting eight at a time there costs the common path its
// registers, 5 to 40 % of an iteration.)
template <class T, class V>
__device__ __forceinline__ T chunk_sum(const TileCsrT<V>& A, const ChunkRows& c, const Tagged<T>* v,
                                       typename TagOf<T>::type want, T* sp, int* left) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    if (c.p1 - c.p0 > kChunkNnz) {   // one row longer than a chunk
        auto get = [&](int j) { return wait_element(v + j, want, left); };
        T s0 = T(0), s1 = T(0);
        int p = c.p0 + lane;
        for (; p + 32 < c.p1; p += 64) {
            s0 = fma(value_at<T>(A.val + p), get(__ldg(A.idx + p)), s0);
            s1 = fma(value_at<T>(A.val + p + 32), get(__ldg(A.idx + p + 32)), s1);
        }
        if (p < c.p1) s0 = fma(value_at<T>(A.val + p), get(__ldg(A.idx + p)), s0);
        return warp_sum(s0 + s1);
    }
    int col[kPerLane];
    T a[kPerLane], g[kPerLane];
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
        const int p = c.p0 + 32 * k + lane;
        col[k] = -1;
        a[k] = g[k] = T(0);
        if (p < c.p1) {
            col[k] = __ldg(A.idx + p);
            a[k] = value_at<T>(A.val + p);
        }
    }
    if (col[0] >= 0) g[0] = wait_element(v + col[0], want, left);
    __syncwarp();
    unsigned missing = 0;
#pragma unroll
    for (int k = 1; k < kPerLane; ++k)
        if (col[k] >= 0) missing |= 1u << k;
    while (missing && --*left > 0) {
        Tagged<T> e[kPerLane];
#pragma unroll
        for (int k = 1; k < kPerLane; ++k)
            if (missing >> k & 1u) e[k] = load_tagged(v + col[k]);
#pragma unroll
        for (int k = 1; k < kPerLane; ++k)
            if ((missing >> k & 1u) && e[k].tag == want) {
                g[k] = e[k].value;
                missing &= ~(1u << k);
            }
    }
#pragma unroll
    for (int k = 0; k < kPerLane; ++k)
        if (col[k] >= 0) sp[32 * k + lane] = dmul(a[k], g[k]);
    __syncwarp();
    T s = T(0);
    if (c.len <= kShortRow) {
        int q = c.q0;
        const int q1 = c.q0 + c.len;
        for (; q + 4 <= q1; q += 4) {
            const T e0 = sp[q], e1 = sp[q + 1], e2 = sp[q + 2], e3 = sp[q + 3];
            s = dadd(dadd(dadd(dadd(s, e0), e1), e2), e3);
        }
        for (; q < q1; ++q) s = dadd(s, sp[q]);
    }
    unsigned long_rows = __ballot_sync(full, c.len > kShortRow);
    while (long_rows) {
        const int l = __ffs(long_rows) - 1;
        long_rows &= long_rows - 1;
        const int a0 = __shfl_sync(full, c.q0, l), al = __shfl_sync(full, c.len, l);
        T t = T(0);
        for (int q = lane; q < al; q += 32) t = dadd(t, sp[a0 + q]);
        t = warp_sum(t);
        if (lane == l) s = t;
    }
    __syncwarp();
    return s;
}

// Where this beats the launches, with `warps` of them. us per iteration, launches -> this, FP64:
// fixed step, anchored, adaptive.
// - While each warp has one chunk of either matrix, at all row lengths up to kLongest: 12,000 x
//   27,000 (540,000; rows of 45) 12.7 -> 8.7, 16.4 -> 13.1, 19.7 -> 15.4. A row beyond a chunk
//   is waited for 64 entries at a time: 15,000 x 30,000 with a row of 700 9.6 -> 8.9, 13.0 -> 10.0,
//   17.8 -> 14.1, with one of 1,000 11.3 -> 11.4 (fixed step), and a row of 40,000 in 20,000 x 40,000
//   207 -> 430; 20,000 x 30,000 with a quarter of the entries in rows of 400 9.0 -> 7.3, half 8.9 -> 9.8.
// - With a vector of few elements every one has many readers, and the lines of those that come
//   early go back and forth. Nonzeros per row (or per column): 120 (800 x 24,000) 7.9 -> 5.9, 180 (2,000 x
//   90,000) 9.5 -> 10.2, 250 (1,200 x 75,000) 8.8 -> 13.4, 400 (800 x 80,000) 9.8 -> 25.7; transposed alike.
// - With more chunks a warp takes them one after the other, and 16 warps an SM do not hide the
//   sums of rows beyond kShortRow (a tree per row) as the launches' 64 do: 40,000 x 60,000 with
//   four fifths of A's entries in rows of 40 (776,000) 15.5 -> 22.2; a fifth in rows of 100, 100,000 x
//   100,000 (979,000) 17.2 -> 14.7. With more elements fewer of them: a quarter at 100,000 x 466,000
//   (2.8M) 39.2 -> 43.3, a fifteenth at 120,000 x 240,000 (2.9M) 38.4 -> 35.6.
// - Where only one matrix has more chunks than warps, they are mostly of light rows, 32 to a chunk, and while the other
//   has no long rows the sums stay hidden: columns of up to 82 with 0.63 of the entries, 50,000 x 80,000
//   (443,000) 12.0 -> 9.5, 14.1 -> 11.5, 19.6 -> 17.3; 0.58, 40,000 x 120,000 (550,000) 13.6 -> 11.5.
//   With two full rounds of chunks, 150,000 x 40,000 (355,000), 12.2 -> 14.3; with four fifths,
//   76,000 x 30,000 (376,000), 12.5 -> 13.6.
//   Long rows in that other matrix delay all: 15,000 x 90,000 (450,000), 0.38 in them, 11.6 -> 16.8, 15.9 -> 18.1,
//   19.3 -> 25.3; 0.25, 30,000 x 90,000 (303,000) 10.2 -> 12.6; 0.07, 15,000 x 120,000 (360,000) 11.0 -> 10.1.
// - Every launch writes the numbered copy anew, and its 16 bytes an element no longer stay near:
//   250,000 x 300,000 (1.2M) 19.0 -> 18.1, 223,000 x 487,000 (1M) 18.4 -> 20.2, 496,000 x 329,000 (1.3M)
//   21.9 -> 29.2.
// - The adaptive loop's sums cost it more: 48,000 x 59,000 (885,000) 0.94 of the launches, from
//   1.2M or 330,000 rows and columns on 0.96 to 1.04.
constexpr int kLongest = 768, kReaders = 150;
template <class V>
inline bool flow_pays(const TileCsrT<V>& A, const TileCsrT<V>& AT, int warps, bool adaptive = false) {
    if (A.ntiles == 0 || AT.ntiles == 0) return false;
    if (std::max(A.share.longest, AT.share.longest) > (A.nnz <= 400000 ? kLongest : kChunkNnz)) return false;
    if (std::max(A.share.streamed, AT.share.streamed) > A.nnz / 3 || A.nnz / kReaders > std::min(A.rows, A.cols)) return false;
    if (std::max(A.ntiles, AT.ntiles) <= warps) return true;
    const int elements = A.rows + A.cols, part = elements <= 300000 ? 4 : 10;
    const TileCsrT<V>&less = A.ntiles <= AT.ntiles ? A : AT, &more = A.ntiles <= AT.ntiles ? AT : A;
    if (less.ntiles <= warps && less.share.longest <= kShortRow && more.ntiles <= warps / 4 * 7 && more.share.tree <= A.nnz / 3 * 2)
        return true;
    auto few_long = [&](const TileCsrT<V>& M) { return M.share.tree <= M.nnz / (M.ntiles <= warps ? 14 : part); };
    return few_long(A) && few_long(AT) && (adaptive ? A.nnz <= 1000000 && elements <= 250000 : A.nnz <= 3000000 && elements <= 600000);
}

// A cooperative launch takes every SM, so solves of several threads take turns, where the launches
// fill the chip together. ms for eight solves of 1,000 iterations from as many threads, launches /
// this: 8,000 x 16,000 16.6 / 34.0, 30,000 x 60,000 46.6 / 56.2; from two 9.4 / 9.0 and 17.0 / 14.5,
// and with more than a chunk a warp (50,000 x 100,000) 25.2 / 27.4. So a solve that could take it is
// counted while in flight, and a window goes to the launches when two others are, or one and
// there is more than a chunk a warp. (Either way gives the same bits.)
class InFlight {
public:
    InFlight() = default;
    InFlight(const InFlight&) = delete;
    InFlight& operator=(const InFlight&) = delete;
    ~InFlight();
    void enter();   // once per object; counts a thread's nested solves as one
    template <class V>
    bool crowded(const TileCsrT<V>& A, const TileCsrT<V>& AT, int warps) const {
        return others() >= (std::max(A.ntiles, AT.ntiles) <= warps ? 2 : 1);
    }

private:
    int others() const;
    int device_ = -1;
};

// CTAs of `threads` threads the current device holds at a time with one per SM, 0 where
// the kernel cannot be launched cooperatively (asked once per kernel and device).
int resident_ctas(const void* kernel, int threads, size_t smem);

template <class Args>
inline cudaError_t launch(void (*kernel)(Args), const Args& args, int ctas, int threads, size_t smem, cudaStream_t stream) {
    void* p[] = {const_cast<Args*>(&args)};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(ctas), dim3(threads), p, smem, stream);
}

}  // namespace flow
}  // namespace b200

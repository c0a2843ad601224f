// level2.cu -- Level-2 BLAS on the GPU: gemv (y := alpha*op(A)*x + beta*y)
// and the rank-1 updates ger / geru / gerc (A := alpha*x*y^T + A), real and
// complex (src/level2.rs:11-104, src/complex2.rs:11-145).
//
// Both read or write each element of A once, so they are bound by HBM
// bandwidth: gemv moves m*n elements, a rank-1 update 2*m*n. A is handled
// through its column-major view (R x C, leading dimension ld): a row-major
// A is the column-major view of its transpose, which swaps the two gemv
// kernels and the roles of x and y in the rank-1 update.
//   * "column sweep" gemv (y_r = sum_c A[r,c] x_c): a CTA per (row tile, range
//     of columns), its warps on every eighth column; few columns, or rows
//     enough to fill the GPU: one thread per four rows, all columns in order.
//   * "column dot" gemv (y_c = sum_r A[r,c] x_r): two columns at a time per
//     CTA and row range, one per warp where columns are short and many; a
//     fixed-order reduction.
//   * the ranges (S of them, only when there are too few tiles to fill the
//     GPU) go through a workspace and a finalize pass in range order; a single
//     range applies rblas's beta pass and alpha itself, unless y shares memory
//     with x or A. Results do not depend on timing.
// Within one range the terms are added in rblas's order (fma(a, x, acc) for
// real, acc + a*x with rblas's complex multiply for complex), so a NoTrans
// column-major call of fewer than kSweepSplit columns, or of more than
// kSweepFullRows rows, reproduces rblas's gemv exactly; other shapes differ from
// rblas's order within rounding.
// The rank-1 update computes each element as rblas does (alpha*x_i rounded,
// then fma / complex multiply-add), so it matches rblas bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "../../include/rblas_b200.h"
#include "rb_internal.h"

namespace rb {

namespace {

template <typename T> struct C2 { T re, im; };

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// rblas's complex multiply (src/complex.rs:101-111):
// re = fma(a.re, b.re, 0 - a.im*b.im), im = fma(a.re, b.im, a.im*b.re)
template <typename T>
__device__ __forceinline__ C2<T> cmul(C2<T> a, C2<T> b) {
    return {fma(a.re, b.re, sub_rn(T(0), mul_rn(a.im, b.im))), fma(a.re, b.im, mul_rn(a.im, b.re))};
}
template <typename T>
__device__ __forceinline__ C2<T> cadd(C2<T> a, C2<T> b) { return {add_rn(a.re, b.re), add_rn(a.im, b.im)}; }
template <typename T>
__device__ __forceinline__ C2<T> cconj(C2<T> a) { return {a.re, sub_rn(T(0), a.im)}; }

// Element access: real arrays of T, complex arrays of interleaved {re, im}.
template <typename T, bool CX> struct El { using type = T; };
template <typename T> struct El<T, true> { using type = C2<T>; };

template <typename T>
__device__ __forceinline__ T ld_el(const T* p) { return __ldg(p); }
// two scalar loads: a complex array is only guaranteed T's alignment
template <typename T>
__device__ __forceinline__ C2<T> ld_el(const C2<T>* p) {
    const T* q = reinterpret_cast<const T*>(p);
    return {__ldg(q), __ldg(q + 1)};
}

// acc + a*x in rblas's order for its type
template <typename T>
__device__ __forceinline__ T mac(T acc, T a, T x) { return fma(a, x, acc); }
template <typename T>
__device__ __forceinline__ C2<T> mac(C2<T> acc, C2<T> a, C2<T> x) { return cadd(acc, cmul(a, x)); }
template <typename T>
__device__ __forceinline__ T add_el(T a, T b) { return add_rn(a, b); }
template <typename T>
__device__ __forceinline__ C2<T> add_el(C2<T> a, C2<T> b) { return cadd(a, b); }
template <typename T>
__device__ __forceinline__ T conj_el(T a) { return a; }
template <typename T>
__device__ __forceinline__ C2<T> conj_el(C2<T> a) { return cconj(a); }
template <typename T>
__device__ __forceinline__ T zero_el(T*) { return T(0); }
template <typename T>
__device__ __forceinline__ C2<T> zero_el(C2<T>*) { return {T(0), T(0)}; }
template <typename T>
__device__ __forceinline__ T shfl_el(T v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }
template <typename T>
__device__ __forceinline__ C2<T> shfl_el(C2<T> v, int o) {
    return {__shfl_down_sync(0xffffffffu, v.re, o), __shfl_down_sync(0xffffffffu, v.im, o)};
}

constexpr int kL2Threads = 256;

// V consecutive elements: one 16-byte load (VEC) or V element loads.
template <typename E, int V> struct Pack { E e[V]; };
template <bool VEC, int V, typename E>
__device__ __forceinline__ Pack<E, V> ld_pack(const E* p) {
    Pack<E, V> r;
    if constexpr (VEC) {
        static_assert(sizeof(Pack<E, V>) == 16, "a vector is 16 bytes");
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(p));
        memcpy(&r, &t, 16);
    } else {
#pragma unroll
        for (int i = 0; i < V; ++i) r.e[i] = ld_el(p + i);
    }
    return r;
}
template <typename E> constexpr int kVecLen = 16 / static_cast<int>(sizeof(E));

template <typename E>
__device__ __forceinline__ E warp_sum(E acc) {  // a fixed tree; lane 0 has the sum
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc = add_el(acc, shfl_el(acc, o));
    return acc;
}

// The last step on y_i given the sum (have) or an empty one (see gemv_finalize).
template <typename T>
__device__ __forceinline__ void finish_y(T* yp, T acc, T alpha, T beta) {
    T yi = *yp;
    if (beta != T(1)) yi = (beta == T(0)) ? T(0) : mul_rn(beta, yi);
    *yp = fma(alpha, acc, yi);
}
template <typename T>
__device__ __forceinline__ void finish_y(C2<T>* yp, C2<T> acc, C2<T> alpha, C2<T> beta) {
    C2<T> yi = *yp;
    const bool beta_zero = beta.re == T(0) && beta.im == T(0);
    yi = beta_zero ? C2<T>{T(0), T(0)} : cmul(beta, yi);
    *yp = cadd(yi, cmul(alpha, acc));
}

// Where a sum goes: y itself (one range) or the range's row of the workspace.
template <typename E>
struct GemvOut {
    E* y;
    long long incy;
    E alpha, beta;
    E* ws;  // null: finish y
    int len;
};
template <typename E>
__device__ __forceinline__ void put(const GemvOut<E>& o, int i, int s, E acc) {
    if (o.ws) o.ws[static_cast<size_t>(s) * o.len + i] = acc;
    else      finish_y(o.y + static_cast<long long>(i) * o.incy, acc, o.alpha, o.beta);
}

// Rows that a thread of the sweeps below and of the rank-1 updates takes, a CTA's
// threads apart, so that every warp load stays one contiguous run.
constexpr int kRowsPerThread = 4;
constexpr int kSweepRows = kL2Threads * kRowsPerThread;

// y_r in column order, a thread for four rows: few columns, or so many rows that
// they fill the GPU. Bound by memory, with few loads in flight: in a whole tile
// no test stands between them, so those of eight columns go out together, and
// CTAs of two warps leave a short last wave. f64 1.3M x 100: 157 us (256 threads,
// four columns, tests: 268; gemv_split_kernel, which is as good there and keeps
// another order, 162); 1.3M x 20: 41 (62); f32 1.3M x 100: 105 (146; split 92).
constexpr int kColThreads = 64;
constexpr int kColRows = kColThreads * kRowsPerThread;

template <typename E>
__global__ void __launch_bounds__(kColThreads)
    gemv_sweep_kernel(const E* __restrict__ A, size_t ld, int R, int C, const E* __restrict__ x, long long incx,
                      int conj, GemvOut<E> o) {
    const int rbase = blockIdx.x * kColRows + threadIdx.x;
    E acc[kRowsPerThread];
    bool live[kRowsPerThread];
#pragma unroll
    for (int q = 0; q < kRowsPerThread; ++q) {
        acc[q] = zero_el(static_cast<E*>(nullptr));
        live[q] = rbase + q * kColThreads < R;
    }
    auto columns = [&](auto whole) {
#pragma unroll 8
        for (int c = 0; c < C; ++c) {
            const E xc = ld_el(x + static_cast<long long>(c) * incx);
            const E* col = A + static_cast<size_t>(c) * ld + rbase;
#pragma unroll
            for (int q = 0; q < kRowsPerThread; ++q) {
                if (decltype(whole)::value || live[q]) {
                    E v = ld_el(col + q * kColThreads);
                    if (conj) v = conj_el(v);
                    acc[q] = mac(acc[q], v, xc);
                }
            }
        }
    };
    if (R - static_cast<int>(blockIdx.x) * kColRows >= kColRows) columns(std::true_type{});
    else                                                             columns(std::false_type{});
#pragma unroll
    for (int q = 0; q < kRowsPerThread; ++q)
        if (live[q]) put(o, rbase + q * kColThreads, 0, acc[q]);
}

// Column dot: y_c over rows [r0, r1) of range s. The CTA takes two columns at
// once, so that a value of x is read once for both and two 16-byte loads of A
// are in flight per step (one column with 8-byte loads: 4.3 TB/s at 6000 x
// 4000 f64; two: 6.2, four: 5.6). Short columns (at most kShortRows) of which
// there are enough take a warp each (256 x 16384 f32: 18.2 -> 6.3 us).
// VA / VX: 16-byte loads of A / x.
constexpr int kDotCols = 2;
constexpr int kShortRows = 1024;

// W warps (the CTA's 8, or 1) per group of COLS columns.
template <typename E, int W, int COLS, bool VA, bool VX>
__global__ void __launch_bounds__(kL2Threads)
    gemv_dot_kernel(const E* __restrict__ A, size_t ld, int R, int C, const E* __restrict__ x, long long incx,
                    int conj, unsigned rchunk, GemvOut<E> o) {
    constexpr int V = kVecLen<E>, LANES = W * 32;
    const int t = threadIdx.x % LANES, s = blockIdx.y;
    // rows are counted unsigned: an index past the last row may exceed INT_MAX
    const int c0 = (blockIdx.x * (kL2Threads / LANES) + threadIdx.x / LANES) * COLS;
    const unsigned r0 = static_cast<unsigned>(s) * rchunk;  // rchunk: a multiple of V
    const unsigned r1 = min(static_cast<unsigned>(R), r0 + rchunk);
    const E* a[COLS];
#pragma unroll
    for (int q = 0; q < COLS; ++q) a[q] = A + static_cast<size_t>(min(c0 + q, C - 1)) * ld;
    E acc[COLS][V];
#pragma unroll
    for (int q = 0; q < COLS; ++q)
#pragma unroll
        for (int i = 0; i < V; ++i) acc[q][i] = zero_el(static_cast<E*>(nullptr));
    if (c0 < C) {
#pragma unroll 2
        for (unsigned r = r0 + t * V; r + V <= r1; r += LANES * V) {
            Pack<E, V> v[COLS], xv;
#pragma unroll
            for (int q = 0; q < COLS; ++q) v[q] = ld_pack<VA, V>(a[q] + r);
            if constexpr (VX) {
                xv = ld_pack<true, V>(x + r);
            } else {
#pragma unroll
                for (int i = 0; i < V; ++i) xv.e[i] = ld_el(x + (static_cast<long long>(r) + i) * incx);
            }
#pragma unroll
            for (int q = 0; q < COLS; ++q)
#pragma unroll
                for (int i = 0; i < V; ++i)
                    acc[q][i] = mac(acc[q][i], conj ? conj_el(v[q].e[i]) : v[q].e[i], xv.e[i]);
        }
        const unsigned rl = r0 + (r1 - r0) / V * V + t;  // fewer than V rows are left
        if (t < V && rl < r1) {
            const E xv = ld_el(x + static_cast<long long>(rl) * incx);
#pragma unroll
            for (int q = 0; q < COLS; ++q) {
                const E v = ld_el(a[q] + rl);
                acc[q][0] = mac(acc[q][0], conj ? conj_el(v) : v, xv);
            }
        }
    }
    // fixed-order reduction: a thread's V sums, the warp tree, the warps in order
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ E part[COLS][kL2Threads / 32];
#pragma unroll
    for (int q = 0; q < COLS; ++q) {
#pragma unroll
        for (int w = V / 2; w > 0; w >>= 1)
#pragma unroll
            for (int i = 0; i < w; ++i) acc[q][i] = add_el(acc[q][i], acc[q][i + w]);
        const E sum = warp_sum(acc[q][0]);
        if constexpr (W == 1) {
            if (lane == 0 && c0 + q < C) put(o, c0 + q, s, sum);
        } else {
            if (lane == 0) part[q][warp] = sum;
        }
    }
    if constexpr (W > 1) {
        __syncthreads();
        if (threadIdx.x < COLS && c0 + static_cast<int>(threadIdx.x) < C) {
            E sum = part[threadIdx.x][0];
#pragma unroll
            for (int w = 1; w < kL2Threads / 32; ++w) sum = add_el(sum, part[threadIdx.x][w]);
            put(o, c0 + threadIdx.x, s, sum);
        }
    }
}

// Column sweep of at least kSweepSplit columns: y_r over columns [c0, c1) of
// range s. A CTA takes 64 rows; its eight warps take every eighth column of
// the range and their sums are added in warp order, so few ranges fill the
// GPU: with one thread per row and up to 198 ranges, the finalize pass's
// serial sum of the ranges was most of the time. Element loads: 16-byte ones
// of 64 to 256 rows were slower (6000 x 4000 f64: 33 us; 44-52 with them, 56
// before; 256 x 16384: 98 -> 15).
constexpr int kSweepPack = 2;
constexpr int kSweepSplit = 32;  // fewer columns: gemv_sweep_kernel in one range, rblas's own order
// More rows than these fill the GPU with four to a thread, and keep rblas's own
// order too.
constexpr int kSweepFullRows = 148 * 8 * kSweepRows - kSweepRows;
constexpr int kSplitRows = 32 * kSweepPack;

template <typename E>
__global__ void __launch_bounds__(kL2Threads)
    gemv_split_kernel(const E* __restrict__ A, size_t ld, int R, int C, const E* __restrict__ x, long long incx,
                      int conj, unsigned cchunk, GemvOut<E> o) {
    constexpr int WARPS = kL2Threads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, s = blockIdx.y;
    const int rb = blockIdx.x * kSplitRows + lane;
    // (columns unsigned, as the rows of gemv_dot_kernel)
    const unsigned c0 = static_cast<unsigned>(s) * cchunk, c1 = min(static_cast<unsigned>(C), c0 + cchunk);
    E acc[kSweepPack];
    bool live[kSweepPack];
#pragma unroll
    for (int q = 0; q < kSweepPack; ++q) {
        acc[q] = zero_el(static_cast<E*>(nullptr));
        live[q] = rb + q * 32 < R;
    }
#pragma unroll 4
    for (unsigned c = c0 + warp; c < c1; c += WARPS) {
        const E* col = A + static_cast<size_t>(c) * ld + rb;
        const E xc = ld_el(x + static_cast<long long>(c) * incx);
#pragma unroll
        for (int q = 0; q < kSweepPack; ++q)
            if (live[q]) {
                E v = ld_el(col + q * 32);
                if (conj) v = conj_el(v);
                acc[q] = mac(acc[q], v, xc);
            }
    }
    __shared__ E part[WARPS][kSplitRows];
#pragma unroll
    for (int q = 0; q < kSweepPack; ++q) part[warp][q * 32 + lane] = acc[q];
    __syncthreads();
    const int r = blockIdx.x * kSplitRows + threadIdx.x;
    if (threadIdx.x >= kSplitRows || r >= R) return;
    E sum = part[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) sum = add_el(sum, part[w][threadIdx.x]);
    put(o, r, s, sum);
}

// rblas's beta pass, then y += alpha * (sum of the S partials in range order).
// Real (src/level2.rs:91-104): beta == 1 leaves y, beta == 0 writes 0,
// else beta*y; then y = fma(alpha, acc, y). Complex (src/complex2.rs:31-43):
// the beta pass always runs (beta == 0 writes 0, else beta*y with the
// complex multiply); then y = y + alpha*acc. alpha == 0 stops after the
// beta pass.
// alpha_mode: 0 no alpha step; 2 add alpha * 0 (rblas still runs the step on
// an empty sum). A non-empty sum ends in finish_y.
template <typename T>
__global__ void gemv_beta_real(T* y, long long incy, int len, T alpha, T beta, int alpha_mode) {
    const int i = blockIdx.x * kL2Threads + threadIdx.x;
    if (i >= len) return;
    T* yp = y + static_cast<long long>(i) * incy;
    T yi = *yp;
    if (beta != T(1)) yi = (beta == T(0)) ? T(0) : mul_rn(beta, yi);
    if (alpha_mode != 0) yi = fma(alpha, T(0), yi);
    *yp = yi;
}

template <typename T>
__global__ void gemv_beta_cplx(C2<T>* y, long long incy, int len, C2<T> alpha, C2<T> beta, int alpha_mode) {
    const int i = blockIdx.x * kL2Threads + threadIdx.x;
    if (i >= len) return;
    C2<T>* yp = y + static_cast<long long>(i) * incy;
    C2<T> yi = *yp;
    const bool beta_zero = beta.re == T(0) && beta.im == T(0);
    yi = beta_zero ? C2<T>{T(0), T(0)} : cmul(beta, yi);
    if (alpha_mode != 0) yi = cadd(yi, cmul(alpha, C2<T>{T(0), T(0)}));
    *yp = yi;
}

// Sum of the S ranges' partials, then finish_y. A CTA takes 32 elements; its
// eight warps sum an eighth of the ranges each, in order, and the eighths are
// added in order.
template <typename E>
__global__ void __launch_bounds__(kL2Threads) gemv_finalize(GemvOut<E> o, int S) {
    constexpr int WARPS = kL2Threads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
    const int per = (S + WARPS - 1) / WARPS, s0 = warp * per, s1 = min(S, s0 + per);
    __shared__ E part[WARPS][32];
    E acc = zero_el(static_cast<E*>(nullptr));
    if (i < o.len && s0 < s1) {
        acc = o.ws[static_cast<size_t>(s0) * o.len + i];
#pragma unroll 8
        for (int s = s0 + 1; s < s1; ++s) acc = add_el(acc, o.ws[static_cast<size_t>(s) * o.len + i]);
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp != 0 || i >= o.len) return;
#pragma unroll
    for (int w = 1; w < WARPS; ++w)
        if (w * per < S) acc = add_el(acc, part[w][lane]);
    finish_y(o.y + static_cast<long long>(i) * o.incy, acc, o.alpha, o.beta);
}

// A[r, c] (column-major view) += alpha*x (.) y: the x index is the view's
// row when x_on_rows, else its column; y likewise on the other index.
// A CTA covers kSweepRows consecutive rows of a range of columns (each
// thread kRowsPerThread rows, 256 apart), the columns strided by gridDim.y.
template <typename T>
__global__ void __launch_bounds__(kL2Threads)
    ger_real_kernel(T* A, size_t ld, int R, int C, const T* __restrict__ x, long long incx, const T* __restrict__ y,
                    long long incy, T alpha, int x_on_rows) {
    const int rbase = blockIdx.x * kSweepRows + threadIdx.x;
    // the row-indexed factor (alpha*x_i, or y_j) does not depend on the
    // column: computed once per thread and row, with the same operations
    T rowv[kRowsPerThread];
#pragma unroll
    for (int q = 0; q < kRowsPerThread; ++q) {
        const int r = rbase + q * kL2Threads;
        rowv[q] = r < R ? (x_on_rows ? mul_rn(alpha, __ldg(x + static_cast<long long>(r) * incx))  // src/level2.rs:83
                                     : __ldg(y + static_cast<long long>(r) * incy))
                        : T(0);
    }
    // two columns per pass: 2 * kRowsPerThread loads of A in flight
    const int step = gridDim.y;
    for (int c = blockIdx.y; c < C; c += 2 * step) {
        const int c2 = c + step;
        const bool two = c2 < C;
        T* col = A + static_cast<size_t>(c) * ld;
        T* col2 = A + static_cast<size_t>(two ? c2 : c) * ld;
        const T colv = x_on_rows ? __ldg(y + static_cast<long long>(c) * incy)
                                 : mul_rn(alpha, __ldg(x + static_cast<long long>(c) * incx));
        const T colv2 = !two ? T(0)
                        : (x_on_rows ? __ldg(y + static_cast<long long>(c2) * incy)
                                     : mul_rn(alpha, __ldg(x + static_cast<long long>(c2) * incx)));
        T a1[kRowsPerThread], a2[kRowsPerThread];
#pragma unroll
        for (int q = 0; q < kRowsPerThread; ++q) {
            const int r = rbase + q * kL2Threads;
            a1[q] = r < R ? col[r] : T(0);
            a2[q] = (two && r < R) ? col2[r] : T(0);
        }
#pragma unroll
        for (int q = 0; q < kRowsPerThread; ++q) {
            const int r = rbase + q * kL2Threads;
            if (r < R) {
                // axi * y_j + a with axi = alpha*x_i (src/level2.rs:86)
                col[r] = x_on_rows ? fma(rowv[q], colv, a1[q]) : fma(colv, rowv[q], a1[q]);
                if (two) col2[r] = x_on_rows ? fma(rowv[q], colv2, a2[q]) : fma(colv2, rowv[q], a2[q]);
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kL2Threads)
    ger_cplx_kernel(C2<T>* A, size_t ld, int R, int C, const C2<T>* __restrict__ x, long long incx,
                    const C2<T>* __restrict__ y, long long incy, C2<T> alpha, int x_on_rows, int conj) {
    const int rbase = blockIdx.x * kSweepRows + threadIdx.x;
    for (int c = blockIdx.y; c < C; c += gridDim.y) {
        C2<T>* col = A + static_cast<size_t>(c) * ld;
#pragma unroll
        for (int q = 0; q < kRowsPerThread; ++q) {
            const int r = rbase + q * kL2Threads;
            if (r < R) {
                const int xi = x_on_rows ? r : c, yj = x_on_rows ? c : r;
                const C2<T> axi = cmul(alpha, ld_el(x + static_cast<long long>(xi) * incx));  // src/complex2.rs:135
                C2<T> yv = ld_el(y + static_cast<long long>(yj) * incy);
                if (conj) yv = cconj(yv);                                              // src/complex2.rs:137-141
                col[r] = cadd(col[r], cmul(axi, yv));                                  // src/complex2.rs:143
            }
        }
    }
}

// Whether [p, p + pn) and [q, q + qn) (elements) share memory.
template <typename E>
bool overlap(const E* p, size_t pn, const E* q, size_t qn) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
    return a < b + qn * sizeof(E) && b < a + pn * sizeof(E);
}

int blocks_for(long long n) { return static_cast<int>((n + kL2Threads - 1) / kL2Threads); }

int fail(cudaError_t e, int32_t* ce) {
    if (ce) *ce = static_cast<int32_t>(e);
    return RB_ERR_CUDA;
}

}  // namespace

template <typename T, bool CX>
int gemv_dev(int layout, int trans, size_t m, size_t n, T ar, T ai, const T* A, size_t lda, const T* x,
             long long incx, T br, T bi, T* y, long long incy, cudaStream_t st, int32_t* ce) {
    using E = typename El<T, CX>::type;
    const bool tr = trans != RB_NO_TRANS;
    const size_t leny = tr ? n : m;
    if (leny == 0) return RB_OK;
    if (m > 0x7fffffff || n > 0x7fffffff) return RB_ERR_INVALID_ARG;
    const bool alpha_zero = (ar == T(0)) && (!CX || ai == T(0));
    // column-major view R x C of A; y = view * x ("sweep") or view^T * x ("dot")
    const bool col = layout == RB_COL_MAJOR;
    const int R = static_cast<int>(col ? m : n), Cc = static_cast<int>(col ? n : m);
    const bool sweep = (col && !tr) || (!col && tr);
    const int conj = (CX && trans == RB_CONJ_TRANS) ? 1 : 0;
    const int len = static_cast<int>(leny);
    const bool have_work = !alpha_zero && R > 0 && Cc > 0;
    E ea, eb;
    if constexpr (CX) {
        ea = E{ar, ai};
        eb = E{br, bi};
    } else {
        ea = ar;
        eb = br;
    }
    E* yv = reinterpret_cast<E*>(y);
    if (!have_work) {
        // rblas runs the alpha step on an empty sum too, except for the real
        // Trans loop, which has no step when m == 0 (src/level2.rs:41-60,
        // src/complex2.rs:55-76)
        const int alpha_mode = alpha_zero ? 0 : ((!CX && tr) ? 0 : 2);
        if constexpr (CX) gemv_beta_cplx<T><<<blocks_for(len), kL2Threads, 0, st>>>(yv, incy, len, ea, eb, alpha_mode);
        else              gemv_beta_real<T><<<blocks_for(len), kL2Threads, 0, st>>>(yv, incy, len, ea, eb, alpha_mode);
        count_launch();
        const cudaError_t e0 = cudaGetLastError();
        return e0 == cudaSuccess ? RB_OK : fail(e0, ce);
    }
    const E* Av = reinterpret_cast<const E*>(A);
    const E* xv = reinterpret_cast<const E*>(x);
    constexpr int V = kVecLen<E>;
    const bool va = reinterpret_cast<uintptr_t>(A) % 16 == 0 && (lda * sizeof(E)) % 16 == 0;
    const bool vx = incx == 1 && reinterpret_cast<uintptr_t>(x) % 16 == 0;
    // ranges (S) so that the grid fills the GPU, each with enough work
    long long S = 1, chunk = 0;
    const long long rows = R, columns = Cc;
    dim3 grid;
    const bool split = sweep && Cc >= kSweepSplit && R <= kSweepFullRows;
    const bool short_cols = !sweep && R <= kShortRows && Cc >= 148 * 4 * (kL2Threads / 32);
    if (split) {
        const long long rb = (rows + kSplitRows - 1) / kSplitRows;
        S = std::max(1ll, std::min(148 * 8 / rb, columns / 32));
        chunk = (columns + S - 1) / S;
        S = (columns + chunk - 1) / chunk;
        grid = dim3(static_cast<unsigned>(rb), static_cast<unsigned>(S));
    } else if (sweep) {
        grid = dim3(static_cast<unsigned>((rows + kColRows - 1) / kColRows));
    } else {
        const long long cols = short_cols ? kL2Threads / 32 : kDotCols, cb = (columns + cols - 1) / cols;
        if (!short_cols) S = std::max(1ll, std::min((148 * 4 + cb - 1) / cb, rows / 1024));
        chunk = ((rows + S - 1) / S + V - 1) / V * V;
        S = (rows + chunk - 1) / chunk;
        grid = dim3(static_cast<unsigned>(cb), static_cast<unsigned>(S));
    }
    // A single range writes y in the kernel that reads x and A: where y shares
    // memory with either, its sums go through the workspace too.
    const size_t lenx = tr ? m : n, ny = (leny - 1) * static_cast<size_t>(incy) + 1;
    const bool through_ws = S > 1 || overlap<E>(yv, ny, xv, (lenx - 1) * static_cast<size_t>(incx) + 1) ||
                            overlap<E>(yv, ny, Av, static_cast<size_t>(Cc - 1) * lda + static_cast<size_t>(R));
    E* ws = nullptr;
    cudaError_t e;
    if (through_ws && (e = scratch_alloc(&ws, static_cast<size_t>(S) * len * sizeof(E), st)) != cudaSuccess)
        return fail(e, ce);
    const GemvOut<E> o{yv, incy, ea, eb, ws, len};
    if (split) {
        gemv_split_kernel<E><<<grid, kL2Threads, 0, st>>>(Av, lda, R, Cc, xv, incx, conj, static_cast<unsigned>(chunk), o);
    } else if (sweep) {
        gemv_sweep_kernel<E><<<grid, kColThreads, 0, st>>>(Av, lda, R, Cc, xv, incx, conj, o);
    } else {
#define RB_DOT(W, COLS, VA, VX) \
    gemv_dot_kernel<E, W, COLS, VA, VX><<<grid, kL2Threads, 0, st>>>(Av, lda, R, Cc, xv, incx, conj, static_cast<unsigned>(chunk), o)
        if (short_cols) {
            if (va && vx)      RB_DOT(1, 1, true, true);
            else if (va)       RB_DOT(1, 1, true, false);
            else               RB_DOT(1, 1, false, false);
        } else {
            if (va && vx)      RB_DOT(8, kDotCols, true, true);
            else if (va)       RB_DOT(8, kDotCols, true, false);
            else               RB_DOT(8, kDotCols, false, false);
        }
#undef RB_DOT
    }
    count_launch();
    if (through_ws) {
        gemv_finalize<E><<<static_cast<unsigned>((leny + 31) / 32), kL2Threads, 0, st>>>(o, static_cast<int>(S));
        count_launch();
    }
    e = cudaGetLastError();
    if (ws) cudaFreeAsync(ws, st);
    return e == cudaSuccess ? RB_OK : fail(e, ce);
}

template <typename T, bool CX>
int ger_dev(int layout, size_t m, size_t n, T ar, T ai, const T* x, long long incx, const T* y, long long incy, T* A,
            size_t lda, int conj, cudaStream_t st, int32_t* ce) {
    if (m == 0 || n == 0) return RB_OK;
    if ((ar == T(0)) && (!CX || ai == T(0))) return RB_OK;  // src/level2.rs:77-79, src/complex2.rs:128-130
    if (m > 0x7fffffff || n > 0x7fffffff) return RB_ERR_INVALID_ARG;
    const bool col = layout == RB_COL_MAJOR;
    const int R = static_cast<int>(col ? m : n), Cc = static_cast<int>(col ? n : m);
    // about 8 CTAs per SM over the row blocks, each walking a slice of columns
    const int rblocks = (R + kSweepRows - 1) / kSweepRows;
    const dim3 grid(rblocks, std::max(1, std::min({Cc, 65535, (148 * 8 * 4 + rblocks - 1) / rblocks})));
    if constexpr (CX)
        ger_cplx_kernel<T><<<grid, kL2Threads, 0, st>>>(reinterpret_cast<C2<T>*>(A), lda, R, Cc,
                                                        reinterpret_cast<const C2<T>*>(x), incx,
                                                        reinterpret_cast<const C2<T>*>(y), incy, C2<T>{ar, ai},
                                                        col ? 1 : 0, conj);
    else
        ger_real_kernel<T><<<grid, kL2Threads, 0, st>>>(A, lda, R, Cc, x, incx, y, incy, ar, col ? 1 : 0);
    count_launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? RB_OK : fail(e, ce);
}

#define RB_L2_INST(T, CX)                                                                                           \
    template int gemv_dev<T, CX>(int, int, size_t, size_t, T, T, const T*, size_t, const T*, long long, T, T, T*, \
                                 long long, cudaStream_t, int32_t*);                                               \
    template int ger_dev<T, CX>(int, size_t, size_t, T, T, const T*, long long, const T*, long long, T*, size_t,   \
                                int, cudaStream_t, int32_t*);
RB_L2_INST(float, false)
RB_L2_INST(double, false)
RB_L2_INST(float, true)
RB_L2_INST(double, true)
#undef RB_L2_INST

}  // namespace rb

// ---- C ABI: device pointers, enqueued on `stream` ---------------------------
using namespace rb;

namespace {

rb_status l2_check(int layout, int trans, size_t m, size_t n, size_t lda, size_t incy_zero_len, rb_error* err) {
    if (err) *err = rb_error{0, 0, 0, 0, 0};
    if ((layout != RB_ROW_MAJOR && layout != RB_COL_MAJOR) || trans < RB_NO_TRANS || trans > RB_CONJ_TRANS) {
        if (err) err->code = RB_ERR_INVALID_ARG;
        return RB_ERR_INVALID_ARG;
    }
    const size_t min_lead = (layout == RB_ROW_MAJOR) ? n : m;
    if (m > 0 && n > 0 && lda < min_lead) {
        if (err) *err = rb_error{RB_ERR_INVALID_LEADING_DIM, 'a', lda, min_lead, 0};
        return RB_ERR_INVALID_LEADING_DIM;
    }
    if (incy_zero_len > 1) {
        if (err) *err = rb_error{RB_ERR_ZERO_STRIDE, 'y', 0, 0, 0};
        return RB_ERR_ZERO_STRIDE;
    }
    return RB_OK;
}

rb_status l2_done(int rc, int32_t ce, rb_error* err) {
    if (rc != RB_OK && err) {
        err->code = rc;
        err->cuda_error = ce;
    }
    return static_cast<rb_status>(rc);
}

template <typename T, bool CX>
rb_status gemv_c(int layout, int trans, size_t m, size_t n, T ar, T ai, const T* a, size_t lda, const T* x,
                 size_t incx, T br, T bi, T* y, size_t incy, void* stream, rb_error* err) {
    const size_t leny = (trans != RB_NO_TRANS) ? n : m;
    const rb_status v = l2_check(layout, trans, m, n, lda, incy == 0 ? leny : 0, err);
    if (v != RB_OK) return v;
    int32_t ce = 0;
    return l2_done(gemv_dev<T, CX>(layout, trans, m, n, ar, ai, a, lda, x, static_cast<long long>(incx), br, bi, y,
                                   static_cast<long long>(incy), static_cast<cudaStream_t>(stream), &ce),
                   ce, err);
}

template <typename T, bool CX>
rb_status ger_c(int layout, size_t m, size_t n, T ar, T ai, const T* x, size_t incx, const T* y, size_t incy, T* a,
                size_t lda, int conj, void* stream, rb_error* err) {
    const rb_status v = l2_check(layout, RB_NO_TRANS, m, n, lda, 0, err);
    if (v != RB_OK) return v;
    int32_t ce = 0;
    return l2_done(ger_dev<T, CX>(layout, m, n, ar, ai, x, static_cast<long long>(incx), y,
                                  static_cast<long long>(incy), a, lda, conj, static_cast<cudaStream_t>(stream), &ce),
                   ce, err);
}

}  // namespace

extern "C" {

rb_status rb_sgemv_dev(rb_layout layout, rb_transpose trans, size_t m, size_t n, float alpha, const float* a,
                       size_t lda, const float* x, size_t incx, float beta, float* y, size_t incy, void* stream,
                       rb_error* err) {
    return gemv_c<float, false>(layout, trans, m, n, alpha, 0.f, a, lda, x, incx, beta, 0.f, y, incy, stream, err);
}
rb_status rb_dgemv_dev(rb_layout layout, rb_transpose trans, size_t m, size_t n, double alpha, const double* a,
                       size_t lda, const double* x, size_t incx, double beta, double* y, size_t incy, void* stream,
                       rb_error* err) {
    return gemv_c<double, false>(layout, trans, m, n, alpha, 0.0, a, lda, x, incx, beta, 0.0, y, incy, stream, err);
}
rb_status rb_cgemv_dev(rb_layout layout, rb_transpose trans, size_t m, size_t n, rb_complex32 alpha,
                       const rb_complex32* a, size_t lda, const rb_complex32* x, size_t incx, rb_complex32 beta,
                       rb_complex32* y, size_t incy, void* stream, rb_error* err) {
    return gemv_c<float, true>(layout, trans, m, n, alpha.re, alpha.im, reinterpret_cast<const float*>(a), lda,
                               reinterpret_cast<const float*>(x), incx, beta.re, beta.im, reinterpret_cast<float*>(y),
                               incy, stream, err);
}
rb_status rb_zgemv_dev(rb_layout layout, rb_transpose trans, size_t m, size_t n, rb_complex64 alpha,
                       const rb_complex64* a, size_t lda, const rb_complex64* x, size_t incx, rb_complex64 beta,
                       rb_complex64* y, size_t incy, void* stream, rb_error* err) {
    return gemv_c<double, true>(layout, trans, m, n, alpha.re, alpha.im, reinterpret_cast<const double*>(a), lda,
                                reinterpret_cast<const double*>(x), incx, beta.re, beta.im,
                                reinterpret_cast<double*>(y), incy, stream, err);
}
rb_status rb_sger_dev(rb_layout layout, size_t m, size_t n, float alpha, const float* x, size_t incx, const float* y,
                      size_t incy, float* a, size_t lda, void* stream, rb_error* err) {
    return ger_c<float, false>(layout, m, n, alpha, 0.f, x, incx, y, incy, a, lda, 0, stream, err);
}
rb_status rb_dger_dev(rb_layout layout, size_t m, size_t n, double alpha, const double* x, size_t incx,
                      const double* y, size_t incy, double* a, size_t lda, void* stream, rb_error* err) {
    return ger_c<double, false>(layout, m, n, alpha, 0.0, x, incx, y, incy, a, lda, 0, stream, err);
}
#define RB_CGER_DEV(NAME, T, CT, CONJ)                                                                              \
    rb_status NAME(rb_layout layout, size_t m, size_t n, CT alpha, const CT* x, size_t incx, const CT* y,           \
                   size_t incy, CT* a, size_t lda, void* stream, rb_error* err) {                                   \
        return ger_c<T, true>(layout, m, n, alpha.re, alpha.im, reinterpret_cast<const T*>(x), incx,                \
                              reinterpret_cast<const T*>(y), incy, reinterpret_cast<T*>(a), lda, CONJ, stream, err);  \
    }
RB_CGER_DEV(rb_cgeru_dev, float, rb_complex32, 0)
RB_CGER_DEV(rb_zgeru_dev, double, rb_complex64, 0)
RB_CGER_DEV(rb_cgerc_dev, float, rb_complex32, 1)
RB_CGER_DEV(rb_zgerc_dev, double, rb_complex64, 1)
#undef RB_CGER_DEV

}  // extern "C"

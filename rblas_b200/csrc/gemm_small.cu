// gemm_small.cu -- plain GEMM for products whose 128-wide tiles leave most of
// the GPU idle: 32 x 32 and 64 x 64 tiles.
//
// Such a call is a serial chain: a 256^3 SGEMM is four 128 x 128 tiles, each
// 33K clocks of FMA on one SM. A CTA of four warps here takes a 32 x 32 tile
// (f32: two warps of 4 x 4 outputs a lane, 16 shared-memory wavefronts and 16
// clocks of FMA per k; f64: four warps of 16 x 16 on DMMA) or, f32, a 64 x 64
// one (four warps of 8 x 4 a lane, 48 wavefronts). Every element's sum runs
// over k in the order of the 128-wide tiles (simt_tile.cuh), and in the ranges
// that the grouped kernel splits K into where it would, so its bits are
// theirs. (Splitting K over the warps reads less shared memory, 12 and 24
// wavefronts, and was no faster at 64 x 64; it changes the bits.)
// Operands come by cp.async into [k][m] and [k][n] tiles: 16-byte copies of an
// MN-major operand on 16 bytes; single elements otherwise, which transposes a
// K-major operand on the way and takes any alignment, so nothing is repacked
// first.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>

#include "rb_device.cuh"
#include "rb_internal.h"
#include "simt_tile.cuh"

namespace rb {

namespace {

constexpr int kSmThreads = 128;

// BM x BN tile, BK k per stage, ST stages. f32: TM x TN outputs of a lane, LM x
// LN lanes, MW x NW warps that compute. f64: 16 x 16 of DMMA per warp.
template <typename T, int BM_, int BN_, int TM_, int TN_, int LM_, int MW_, int BK_, int ST_>
struct SmCfg {
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, LM = LM_, LN = 32 / LM_, BK = BK_, ST = ST_;
    static constexpr int MW = MW_, NW = BN / (LN * TN), W = MW * NW;
    static constexpr int VEC = 16 / (int)sizeof(T);
    // padded rows of a stage, one 16-byte chunk (f64: two, for the fragment
    // reads) apart modulo 128 bytes
    static constexpr int PAD = 4;
    static constexpr int LDA = BM + PAD, LDB = BN + PAD;
    static constexpr int STAGE = BK * (LDA + LDB);  // elements
    static constexpr int SMEM = ST * STAGE * (int)sizeof(T);
    static_assert(MW * LM * TM == BM && W <= kSmThreads / 32, "the warps cover the tile");
};

template <typename T>
struct SmParams {
    int m, n, k;
    unsigned tiles_m;
    const T *a, *b;
    size_t lda, ldb;
    int a_vec, b_vec;  // 16-byte copies (MN-major, aligned)
    int k_range;       // k of a range whose sum is formed apart (a multiple of 16; INT_MAX: one range)
    SimtOut<T> o;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async_el(void* dst, const void* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES),
                 "r"(in ? BYTES : 0)
                 : "memory");
}

// One stage of one operand: rows x0.. (of X) by k0.. (of K) into dst[k][ROWS],
// row stride LD. KMAJ: element (x, k) at p[k + x * ld], else p[x + k * ld].
template <typename T, int ROWS, int LD, int BK, bool KMAJ>
__device__ __forceinline__ void sm_load(T* dst, const T* p, size_t ld, int x0, int X, int k0, int K, int vec) {
    constexpr int VEC = 16 / (int)sizeof(T), EL = (int)sizeof(T);
    if constexpr (KMAJ) {
        // a warp copies 8 consecutive k of 4 rows: whole sectors of the
        // source, and (rows of a stage being one 16-byte chunk apart modulo
        // 128 bytes) all banks of the destination
#pragma unroll
        for (int i = 0; i < ROWS * BK / kSmThreads; ++i) {
            const int idx = threadIdx.x + i * kSmThreads;
            const int k = idx % 8 + idx / 32 % (BK / 8) * 8, x = idx / 8 % 4 + idx / (4 * BK) * 4;
            const bool in = x0 + x < X && k0 + k < K;
            cp_async_el<EL>(dst + k * LD + x, in ? p + (k0 + k) + static_cast<size_t>(x0 + x) * ld : p, in);
        }
    } else if (vec) {
#pragma unroll
        for (int i = 0; i < ROWS * BK / VEC / kSmThreads; ++i) {
            const int idx = threadIdx.x + i * kSmThreads, x = idx % (ROWS / VEC) * VEC, k = idx / (ROWS / VEC);
            const int left = k0 + k < K ? min(VEC, X - (x0 + x)) : 0;  // elements of the vector that exist
            cp_async16(dst + k * LD + x, left > 0 ? p + (x0 + x) + static_cast<size_t>(k0 + k) * ld : p,
                       left > 0 ? left * EL : 0);
        }
    } else {
#pragma unroll
        for (int i = 0; i < ROWS * BK / kSmThreads; ++i) {
            const int idx = threadIdx.x + i * kSmThreads, x = idx % ROWS, k = idx / ROWS;
            const bool in = x0 + x < X && k0 + k < K;
            cp_async_el<EL>(dst + k * LD + x, in ? p + (x0 + x) + static_cast<size_t>(k0 + k) * ld : p, in);
        }
    }
}

template <typename T, class Cfg, bool A_K, bool B_K>
__global__ void __launch_bounds__(kSmThreads) small_gemm_kernel(const SmParams<T> p) {
    constexpr int VEC = Cfg::VEC, TM = Cfg::TM, TN = Cfg::TN, BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, ST = Cfg::ST;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(smem_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = static_cast<int>(blockIdx.x % p.tiles_m) * BM, n0 = static_cast<int>(blockIdx.x / p.tiles_m) * BN;
    if ((p.o.tri == 1 && m0 > n0 + BN - 1) || (p.o.tri == 2 && m0 + BM - 1 < n0)) return;
    const int num_kt = (p.k + BK - 1) / BK;
    auto load = [&](int kt) {
        if (kt < num_kt) {
            T* sa = smem + (kt % ST) * Cfg::STAGE;
            sm_load<T, BM, Cfg::LDA, BK, A_K>(sa, p.a, p.lda, m0, p.m, kt * BK, p.k, p.a_vec);
            sm_load<T, BN, Cfg::LDB, BK, B_K>(sa + BK * Cfg::LDA, p.b, p.ldb, n0, p.n, kt * BK, p.k, p.b_vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");  // empty past the end: the count below stays the same
    };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) load(s);
    const bool computes = warp < Cfg::W;
    const SimtOut<T>& o = p.o;

    if constexpr (sizeof(T) == 4) {
        const int wm0 = (warp % Cfg::MW) * Cfg::LM * TM, wn0 = (warp / Cfg::MW) * Cfg::LN * TN;
        const int lm = lane % Cfg::LM, ln = lane / Cfg::LM;
        f32x2 acc[TM / 2][TN];
#pragma unroll
        for (int i = 0; i < TM / 2; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0;
        f32x2 sum[TM / 2][TN];  // the ranges before the current one
        int flush = p.k_range;  // where the current range ends
        for (int kt = 0; kt < num_kt; ++kt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncthreads();  // stage kt is there for all; stage kt - 1 has been read
            load(kt + ST - 1);
            if (!computes) continue;
            if (kt * BK == flush) {  // (a range is whole f32 stages)
#pragma unroll
                for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        if (flush == p.k_range) sum[i][j] = acc[i][j];
                        else add_f32x2(sum[i][j], acc[i][j]);
                        acc[i][j] = 0;
                    }
                flush += p.k_range;
            }
            const T* sa = smem + (kt % ST) * Cfg::STAGE + wm0 + lm * VEC;
            const T* sb = smem + (kt % ST) * Cfg::STAGE + BK * Cfg::LDA + wn0 + ln * VEC;
#pragma unroll
            for (int q = 0; q < BK; ++q) {
                f32x2 a[TM / 2];
                float b[TN];
#pragma unroll
                for (int h = 0; h < TM / VEC; ++h) {
                    float v[VEC];
                    lds16<float>(reinterpret_cast<const uint8_t*>(sa + q * Cfg::LDA + h * Cfg::LM * VEC), v);
                    a[2 * h] = pack_f32x2(v[0], v[1]);
                    a[2 * h + 1] = pack_f32x2(v[2], v[3]);
                }
#pragma unroll
                for (int h = 0; h < TN / VEC; ++h) {
                    float v[VEC];
                    lds16<float>(reinterpret_cast<const uint8_t*>(sb + q * Cfg::LDB + h * Cfg::LN * VEC), v);
#pragma unroll
                    for (int e = 0; e < VEC; ++e) b[h * VEC + e] = v[e];
                }
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const f32x2 bb = pack_f32x2(b[j], b[j]);
#pragma unroll
                    for (int i = 0; i < TM / 2; ++i) fma_f32x2(acc[i][j], a[i], bb);
                }
            }
        }
        if (!computes) return;
        if (flush != p.k_range) {
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    add_f32x2(sum[i][j], acc[i][j]);
                    acc[i][j] = sum[i][j];
                }
        }
        float cv[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int r = m0 + wm0 + (i / VEC) * Cfg::LM * VEC + lm * VEC + i % VEC;
                const int c = n0 + wn0 + (j / VEC) * Cfg::LN * VEC + ln * VEC + j % VEC;
                cv[i][j] = (o.beta_mode != 0 && simt_live(o, r, c)) ? o.cin[r + static_cast<size_t>(c) * o.ldcin] : 0.f;
            }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int r = m0 + wm0 + (i / VEC) * Cfg::LM * VEC + lm * VEC + i % VEC;
                const int c = n0 + wn0 + (j / VEC) * Cfg::LN * VEC + ln * VEC + j % VEC;
                if (!simt_live(o, r, c)) continue;
                float lo, hi;
                unpack_f32x2(acc[i / 2][j], lo, hi);
                const float t = (o.beta_mode == 2) ? o.beta * cv[i][j] : cv[i][j];
                o.c[r + static_cast<size_t>(c) * o.ldc] = fmaf(o.alpha, (i & 1) ? hi : lo, t);
            }
    } else {
        // a warp's 16 x 16: two DMMA blocks. The fragment's k slots t and t + 4
        // take the k rows they take in dmma_mainloop (t, t + 4 for a K-major
        // A, else 2t, 2t + 1), so that the sums are its sums.
        const int wm0 = (warp % (BM / 16)) * 16, wn0 = (warp / (BM / 16)) * 16;
        const int g = lane >> 2, t = lane & 3;
        const int ka = A_K ? t : 2 * t, kb = A_K ? t + 4 : 2 * t + 1;
        double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}}, sum[2][4];
        int flush = p.k_range;
        auto end_range = [&]() {
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    sum[nb][q] = flush == p.k_range ? acc[nb][q] : sum[nb][q] + acc[nb][q];
                    acc[nb][q] = 0.0;
                }
        };
        for (int kt = 0; kt < num_kt; ++kt) {
            asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
            __syncthreads();
            load(kt + ST - 1);
            const double* sa = smem + (kt % ST) * Cfg::STAGE + wm0 + g;
            const double* sb = smem + (kt % ST) * Cfg::STAGE + BK * Cfg::LDA + wn0 + g;
#pragma unroll
            for (int q = 0; q < BK; q += 8) {
                if (q % 16 == 0 && kt * BK + q == flush) {
                    end_range();
                    flush += p.k_range;
                }
                const double a[4] = {sa[(q + ka) * Cfg::LDA], sa[(q + ka) * Cfg::LDA + 8], sa[(q + kb) * Cfg::LDA],
                                     sa[(q + kb) * Cfg::LDA + 8]};
#pragma unroll
                for (int nb = 0; nb < 2; ++nb) {
                    const double b[2] = {sb[(q + ka) * Cfg::LDB + 8 * nb], sb[(q + kb) * Cfg::LDB + 8 * nb]};
                    dmma_16x8x8(acc[nb], a, b);
                }
            }
        }
        if (flush != p.k_range) {
            end_range();
#pragma unroll
            for (int nb = 0; nb < 2; ++nb)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[nb][q] = sum[nb][q];
        }
        double cv[2][4];
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = m0 + wm0 + g + 8 * (q >> 1), c = n0 + wn0 + 8 * nb + 2 * t + (q & 1);
                cv[nb][q] = (o.beta_mode != 0 && simt_live(o, r, c)) ? o.cin[r + static_cast<size_t>(c) * o.ldcin] : 0.0;
            }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = m0 + wm0 + g + 8 * (q >> 1), c = n0 + wn0 + 8 * nb + 2 * t + (q & 1);
                if (!simt_live(o, r, c)) continue;
                const double tv = (o.beta_mode == 2) ? o.beta * cv[nb][q] : cv[nb][q];
                o.c[r + static_cast<size_t>(c) * o.ldc] = fma(o.alpha, acc[nb][q], tv);
            }
    }
}

template <typename T, class Cfg, bool A_K, bool B_K>
cudaError_t launch_variant(const SmParams<T>& p, cudaStream_t st) {
    auto kern = small_gemm_kernel<T, Cfg, A_K, B_K>;
    static bool attr_set = false;  // per instantiation; benign race (idempotent)
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM);
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    const size_t tiles = static_cast<size_t>(p.tiles_m) * ((p.n + Cfg::BN - 1) / Cfg::BN);
    if (tiles > 0x7fffffff) return cudaErrorInvalidValue;  // (small_gemm_cfg chooses far fewer)
    KernelTimer tm;
    kernel_timing_begin(sizeof(T) == 4 ? "simt_sgemm" : "simt_dgemm", 2.0 * p.m * p.n * p.k, st, &tm);
    kern<<<static_cast<unsigned>(tiles), kSmThreads, Cfg::SMEM, st>>>(p);
    kernel_timing_end(&tm, st);
    count_launch();
    return cudaGetLastError();
}

template <typename T, class Cfg>
cudaError_t launch_cfg(bool a_k, bool b_k, SmParams<T> p, cudaStream_t st) {
    p.tiles_m = static_cast<unsigned>((p.m + Cfg::BM - 1) / Cfg::BM);
    if (a_k) return b_k ? launch_variant<T, Cfg, true, true>(p, st) : launch_variant<T, Cfg, true, false>(p, st);
    return b_k ? launch_variant<T, Cfg, false, true>(p, st) : launch_variant<T, Cfg, false, false>(p, st);
}

}  // namespace

template <typename T>
cudaError_t launch_small_gemm(int cfg, bool a_kmajor, bool b_kmajor, int m, int n, int k, T alpha, const T* A, size_t lda,
                              const T* B, size_t ldb, T beta, T* C, size_t ldc, cudaStream_t st, int tri, int k_range) {
    SmParams<T> p;
    p.m = m; p.n = n; p.k = k;
    p.a = A; p.b = B;
    p.lda = lda; p.ldb = ldb;
    auto vec = [](const T* x, size_t ld) { return reinterpret_cast<uintptr_t>(x) % 16 == 0 && ld * sizeof(T) % 16 == 0; };
    p.a_vec = !a_kmajor && vec(A, lda);
    p.b_vec = !b_kmajor && vec(B, ldb);
    p.k_range = k_range > 0 ? k_range : INT_MAX;
    p.o = SimtOut<T>{C, ldc, C, ldc, m, n, alpha, beta, (beta == T(0)) ? 0 : (beta == T(1) ? 1 : 2), tri};
    if constexpr (sizeof(T) == 4)
        return cfg == 2 ? launch_cfg<T, SmCfg<T, 64, 64, 8, 4, 4, 2, 32, 4>>(a_kmajor, b_kmajor, p, st)
                        : launch_cfg<T, SmCfg<T, 32, 32, 4, 4, 8, 1, 32, 4>>(a_kmajor, b_kmajor, p, st);
    else
        return launch_cfg<T, SmCfg<T, 32, 32, 2, 4, 8, 2, 32, 4>>(a_kmajor, b_kmajor, p, st);
}

// Which small tile (1: 32 x 32; 2: 64 x 64, f32 only) an m x n x k product
// runs fastest on, or 0: the 128-wide tiles, given the grouped kernel's split
// factor for them (1: not split). Times in us: a launch, what a wave of tiles
// costs beside its k (C's stores above all: 3000^2 of k = 16 is four waves of
// wide tiles, 60 of small ones), and a time per k that a CTA alone on its SM
// takes (a chain of latencies) or its tiles per SM times what each costs there,
// by how each operand is stored: K-major or off 16 bytes it is copied element by
// element (the wide tiles repack what is off 16 bytes first). Fitted to 1669 calls
// of k 8 .. 2900, all transposes, leading dimensions on and off 16 bytes: the
// choice is 0.9 % (f64 0.2 %) off the best one in the mean; by k and the numbers
// of tiles alone it was 2.0 and 1.7 %.
// us, 128-wide -> small: SGEMM 256^3 32.8 -> 10.3, 512^3 54.7 -> 20.5, 768^3 75.9
// -> 36.9 (64 x 64); DGEMM 256^3 26.2 -> 10.3, 512^3 34.9 -> 20.5; left: SGEMM
// 1024^3 59.8 against 72, A^T B^T 1200^2 of k = 32 8.4 against 12, 3000^2 of k =
// 16 29 against 37; DGEMM 1024^3 96 against 108, A^T B 1700^2 of k = 16 12.4
// against 18.5.
template <typename T>
int small_gemm_cfg(size_t m, size_t n, size_t k, int splits, int sms, const SmallOperands& op) {
    auto waves = [&](size_t bm, size_t bn, int s = 1) {
        return std::ceil(static_cast<double>((m + bm - 1) / bm) * static_cast<double>((n + bn - 1) / bn) * s / sms);
    };
    const double K = static_cast<double>(k);
    const int a = op.a_k, b = op.b_k;  // (as numbers)
    const int rows = (!op.a_k && !op.a_vec) + (!op.b_k && !op.b_vec);  // MN-major operands copied by element
    const int packed = !op.a_vec + !op.b_vec;
    const double packed_mega = 1e-6 * K * ((op.a_vec ? 0.0 : static_cast<double>(m)) + (op.b_vec ? 0.0 : static_cast<double>(n)));
    if (sizeof(T) == 4) {
        const double w1 = waves(32, 32), w2 = waves(64, 64);
        const double t1 =
            std::max(8.5, 5.0 + 0.44 * w1 + K * std::max(0.0175 + 0.0018 * a + 0.0016 * b + 0.0040 * rows,
                                                         (0.0107 + 0.0008 * a + 0.0006 * b + 0.0032 * rows) * w1));
        const double t2 =
            std::max(8.5, 5.1 + 1.64 * w2 + K * std::max(0.0305 + 0.0045 * a + 0.0060 * b + 0.0084 * rows,
                                                         (0.0255 + 0.0020 * a + 0.0026 * b + 0.0068 * rows) * w2));
        double wide = 4.2 * packed + 4.6 * packed_mega;
        if (splits > 1) {
            const double w = waves(128, 128, splits);
            wide += 18.2 + 9.2 * w + (0.0587 + 0.0142 * a + 0.0144 * b) * K / splits * w;
        } else if (simt_narrow_f32(m, n)) {
            const double w = waves(128, 64);
            wide += 5.1 + 1.57 * w + (0.0437 + 0.0034 * a + 0.0084 * b) * K * w;
        } else {
            const double w = waves(128, 128);
            wide += 1.6 + 6.4 * w + (0.0728 + 0.0043 * a + 0.0120 * b) * K * w;
        }
        wide = std::max(7.8, wide);
        return std::min(t1, t2) >= wide ? 0 : t1 <= t2 ? 1 : 2;
    }
    const double w1 = waves(32, 32), w = waves(128, 64, splits);
    const double t1 =
        std::max(8.5, 4.1 + 0.55 * w1 + K * std::max(0.0226 - 0.001 * a + 0.001 * b + 0.0033 * rows,
                                                     (0.0134 + 0.0008 * a + 0.0032 * b + 0.0019 * rows) * w1));
    const double wide = 4.4 * packed + 7.3 * packed_mega +
                        (splits > 1 ? 9.3 + 6.1 * w + 0.069 * K / splits * w
                                    : 2.9 + 3.5 * w + (0.068 - 0.004 * a - 0.0014 * b) * K * w);
    return t1 < std::max(7.8, wide) ? 1 : 0;
}

template cudaError_t launch_small_gemm<float>(int, bool, bool, int, int, int, float, const float*, size_t, const float*,
                                              size_t, float, float*, size_t, cudaStream_t, int, int);
template cudaError_t launch_small_gemm<double>(int, bool, bool, int, int, int, double, const double*, size_t,
                                               const double*, size_t, double, double*, size_t, cudaStream_t, int, int);
template int small_gemm_cfg<float>(size_t, size_t, size_t, int, int, const SmallOperands&);
template int small_gemm_cfg<double>(size_t, size_t, size_t, int, int, const SmallOperands&);

}  // namespace rb

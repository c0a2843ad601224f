// gemm_umma.cu -- the split-precision GEMM forms on the 5th-generation tensor
// cores (tcgen05.mma, accumulators in TMEM):
//
//   BF16X3 (SGEMM): x = hi + lo with hi = bf16(x), lo = bf16(x - hi);
//     C = alpha * (Ah*Bh + Ah*Bl + Al*Bh) + beta * C, FP32 accumulation.
//   OZAKI (DGEMM): Ozaki-scheme INT8 slice emulation (Ozaki, Ogita, Oishi &
//     Rump, "Error-free transformations of matrix multiplication by using
//     fast routines of matrix multiplication and its applications", Numer.
//     Algorithms 59, 2012; Ootomo, Ozaki & Yokota, "DGEMM on integer matrix
//     multiplication unit", IJHPCA 2024). Each row of op(A) / column of op(B)
//     is scaled by a power of two 2^-e so |x| < 1, then cut into `s` signed
//     7-bit slices: x * 2^-e = sum_t sigma_t 2^-7(t+1). Slice products are
//     exact in INT32; the products of equal weight (t+u = d) share one TMEM
//     accumulator, and C = alpha * 2^(e_i+f_j) sum_d 2^-7(d+2) S_d + beta * C
//     is summed in FP64 from the smallest weight up. Pairs with t+u >= s are
//     dropped (the scheme's truncation).
//
// Both replace rblas's CPU blocking/packing/microkernel path
// (src/kernel/gemm.rs:185-429) for the precision forms that rblas does not
// have; the plain forms live in gemm_simt.cu.
//
// Large products run on CTA pairs (umma_pair_kernel, ozaki_pair_kernel; tall
// ones with A split inside: umma_split_fused_kernel). Single-CTA structure of
// the others (persistent, one CTA per SM, 6 warps; Ozaki's 18):
//   warp 0 lane 0  TMA producer: K-major operand tiles (128-byte rows, 128-byte
//                  swizzle) into a STAGES-deep shared-memory ring.
//   warp 1         allocates TMEM; lane 0 issues tcgen05.mma into one of two
//                  accumulators and commits each stage back to the producer.
//   warps 2..      epilogue: tcgen05.ld the accumulator (warp w reads TMEM
//                  lanes 32*(w%4)..+31 = tile rows), apply the form's
//                  scaling and alpha/beta, store C coalesced; release the
//                  accumulator so the next unit's MMAs overlap this drain.
// Operands are first rewritten by a pre-pass into K-major bf16 hi/lo planes
// or int8 slice planes (this also absorbs every transpose and layout).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>
#include <type_traits>
#include <utility>

#include "../../include/rblas_b200.h"
#include "rb_device.cuh"
#include "rb_internal.h"

namespace rb {

namespace {

constexpr int kUM = 128;
constexpr int kRowBytes = 128;                  // K bytes per tile row (one swizzle row)
constexpr int kATile = kUM * kRowBytes;         // 16 KiB
constexpr int kExpSentinel = -(1 << 30);        // row exponent of an all-zero row

enum { kModeBf16x3 = 0, kModeBf16x6 = 1 };

// Per BF16 form: tile N, operand planes per stage, ring depth, and the plane
// products issued per UMMA K step (smallest weights first).
template <int MODE> struct UCfg;
template <> struct UCfg<kModeBf16x3> {
    static constexpr int UN = 128, NA = 2, NB = 2, STAGES = 3, NPROD = 3, THREADS = 192;
    // lo*hi, hi*lo, hi*hi
    __host__ __device__ static constexpr int pa(int q) { return q == 0 ? 1 : 0; }
    __host__ __device__ static constexpr int pb(int q) { return q == 1 ? 1 : 0; }
};
template <> struct UCfg<kModeBf16x6> {
    static constexpr int UN = 128, NA = 3, NB = 3, STAGES = 2, NPROD = 6, THREADS = 192;
    // weight 2 (lo*hi, mid*mid, hi*lo), weight 1 (mid*hi, hi*mid), weight 0 (hi*hi)
    __host__ __device__ static constexpr int pa(int q) { return q == 0 ? 2 : (q == 1 || q == 3) ? 1 : 0; }
    __host__ __device__ static constexpr int pb(int q) { return q == 2 ? 2 : (q == 1 || q == 4) ? 1 : 0; }
};

template <int MODE>
constexpr int umma_smem_bytes() {
    using C = UCfg<MODE>;
    return C::STAGES * (C::NA * kATile + C::NB * C::UN * kRowBytes) + 256 + 1024;
}

struct UParams {
    int m, n, k;
    int tiles_m, tiles_n, num_tiles;
    int num_kt;        // 128-byte K tiles over the whole K
    int kt_per_chunk;  // K tiles per accumulation unit (FP32 promotion interval)
    int kchunks;
    int beta_mode;     // 0 beta == 0, 1 beta == 1, 2 general
    float alpha_f, beta_f;
    float* c;
    size_t ldc;
    const float* cin;  // C0, read for beta != 0: c itself, or a separate input with c's leading dimension
    uint32_t* err;
};

constexpr int kMaxStages = 8;  // mbarrier pairs in Bar: every kernel's ring must fit

struct Bar {
    uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
};
static_assert(sizeof(Bar) <= 256, "the kernels reserve 256 bytes of shared memory for Bar");

// One problem of a grouped BF16-split launch: its plane tensor maps (64-byte
// aligned for TMA) and parameters.
struct alignas(64) UGroupEntry {
    CUtensorMap tmA, tmB;
    UParams p;
};

struct UWork {
    const UParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    int t;  // tile of the problem
};

// The single-problem kernel's tiles, one problem.
struct USingleSrc {
    const UParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    __device__ __forceinline__ uint32_t* err() const { return p->err; }
    __device__ __forceinline__ int items() const { return p->num_tiles; }
    __device__ __forceinline__ UWork get(int item) const { return UWork{p, ta, tb, item}; }
};

// Grouped: item i is tile i - starts[j] of problem j (starts[j] <= i <
// starts[j+1]); problems ordered by K, longest first.
struct UGroupSrc {
    const UGroupEntry* tab;
    const int* starts;
    int nprob;
    uint32_t* error;
    __device__ __forceinline__ uint32_t* err() const { return error; }
    __device__ __forceinline__ int items() const { return __ldg(starts + nprob); }
    __device__ __forceinline__ UWork get(int item) const {
        int lo = 0, hi = nprob - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(starts + mid) <= item) lo = mid;
            else hi = mid - 1;
        }
        const UGroupEntry* g = tab + lo;
        return UWork{&g->p, &g->tmA, &g->tmB, item - __ldg(starts + lo)};
    }
};

// Work of one tile is a sequence of accumulation units: unit c covers K
// tiles [c*G, (c+1)*G) with all plane products, and the epilogue promotes
// each unit's FP32 partial into FP32 registers (tcgen05's accumulation
// truncates; short units keep that error small).
template <int MODE, class Src>
__device__ __forceinline__ void umma_body(const Src& src) {
    using Cfg = UCfg<MODE>;
    constexpr int UN = Cfg::UN, NA = Cfg::NA, NB = Cfg::NB, ST = Cfg::STAGES;
    static_assert(ST <= kMaxStages, "Bar holds kMaxStages stages");
    constexpr int BTILE = UN * kRowBytes;
    constexpr int STAGE_BYTES = NA * kATile + NB * BTILE;
    constexpr int KSTEPS = 4;  // UMMA K steps of 32 bytes per 128-byte tile row
    constexpr uint32_t IDESC = umma_idesc(1, 1, kUM, UN);  // f32 <- bf16
    // BF16X6 keeps hi*hi apart from the five smaller products: tcgen05's FP32
    // accumulation truncates, so each of its roundings costs up to one ulp of
    // the accumulator it adds into. In an accumulator of their own the small
    // products' roundings are ~2^-8 of hi*hi's, and hi*hi's own are one per
    // instruction instead of one per product. (At K ~ 400 the shared
    // accumulator left BF16X6 at up to 4x plain SGEMM's error.)
    constexpr bool SPLIT_ACC = (MODE == kModeBf16x6);
    constexpr uint32_t ACC_COLS = SPLIT_ACC ? 2 * UN : UN;  // per accumulator buffer
    constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;
    static_assert(TMEM_COLS <= 512, "two buffers must fit the SM's TMEM");

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    Bar* bar = reinterpret_cast<Bar*>(smem + ST * STAGE_BYTES);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&bar->full[s], 1);
            mbar_init(&bar->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar->acc_full[b], 1);
            mbar_init(&bar->acc_empty[b], 4);
        }
        mbar_init(&bar->drain, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(&bar->tmem_base, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bar->tmem_base;
    const int items = src.items();
    uint32_t* const err = src.err();
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // ------------------------------ TMA producer ------------------------------
        uint32_t it = 0;
        const CUtensorMap* fetched = nullptr;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const UWork w = src.get(item);
            const UParams& p = *w.p;
            if (w.ta != fetched) {
                prefetch_tmap(w.ta);
                prefetch_tmap(w.tb);
                fetched = w.ta;
            }
            int tm, tn;
            raster_tile(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * kUM, n0 = tn * UN;
            for (int kt = 0; kt < p.num_kt; ++kt, ++it) {
                const int s = it % ST;
                if (it >= ST && !mbar_wait(&bar->empty[s], ((it / ST) - 1) & 1, err, 0x201)) {
                    ok = false;
                    break;
                }
                uint8_t* sa = smem + s * STAGE_BYTES;
                uint8_t* sb = sa + NA * kATile;
                mbar_arrive_expect_tx(&bar->full[s], STAGE_BYTES);
                const int k0 = kt * 64;  // bf16 elements per 128-byte row
#pragma unroll
                for (int q = 0; q < NA; ++q) tma_load_3d(sa + q * kATile, w.ta, &bar->full[s], k0, m0, q);
#pragma unroll
                for (int q = 0; q < NB; ++q) tma_load_3d(sb + q * BTILE, w.tb, &bar->full[s], k0, n0, q);
            }
        }
        if (!ok) {
            const uint32_t first = it > (uint32_t)ST ? it - ST : 0;
            for (uint32_t j = first; j < it; ++j) mbar_wait_drain(&bar->full[j % ST], (j / ST) & 1);
        }
    } else if (warp == 1 && lane == 0) {
        // ------------------------------ MMA issuer ------------------------------
        uint32_t it = 0, uc = 0;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const UWork w = src.get(item);
            const UParams& p = *w.p;
            const int units = p.kchunks;
            for (int u = 0; ok && u < units; ++u, ++uc) {
                const int kt0 = u * p.kt_per_chunk, kt1 = min(p.num_kt, kt0 + p.kt_per_chunk);
                const uint32_t b = uc & 1;
                if (uc >= 2 && !mbar_wait(&bar->acc_empty[b], ((uc >> 1) - 1) & 1, err, 0x202)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + b * ACC_COLS;        // the products (all, or all but hi*hi)
                const uint32_t d_big = SPLIT_ACC ? d_tmem + UN : d_tmem;  // hi*hi
                uint32_t accumulate = 0;
                for (int kt = kt0; kt < kt1; ++kt, ++it) {
                    const int s = it % ST;
                    if (!mbar_wait(&bar->full[s], (it / ST) & 1, err, 0x203)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t sa = smem_u32(smem + s * STAGE_BYTES);
                    const uint32_t sb = sa + NA * kATile;
#pragma unroll
                    for (int kk = 0; kk < KSTEPS; ++kk) {
#pragma unroll
                        for (int q = 0; q < Cfg::NPROD; ++q) {
                            const bool big = SPLIT_ACC && q == Cfg::NPROD - 1;
                            umma_f16(big ? d_big : d_tmem, sw128_kmajor_desc(sa + Cfg::pa(q) * kATile) + 2 * kk,
                                     sw128_kmajor_desc(sb + Cfg::pb(q) * BTILE) + 2 * kk, IDESC,
                                     (q == 0 || big) ? accumulate : 1u);
                        }
                        accumulate = 1;
                    }
                    tc_commit(&bar->empty[s]);  // stage free once these MMAs complete
                }
                if (ok) tc_commit(&bar->acc_full[b]);
            }
        }
        // make sure nothing of ours is still in flight before TMEM is released
        tc_commit(&bar->drain);
        mbar_wait_drain(&bar->drain, 0);
    } else if (warp >= 2) {
        // ------------------------------ epilogue ------------------------------
        const int quarter = warp & 3;
        const int row_in_tile = quarter * 32 + lane;
        uint32_t uc = 0;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const UWork w = src.get(item);
            const UParams& p = *w.p;
            const int units = p.kchunks;
            int tm, tn;
            raster_tile(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * kUM, n0 = tn * UN;
            const int r = m0 + row_in_tile;
            const bool row_ok = r < p.m;
            float sum[UN];
#pragma unroll
            for (int j = 0; j < UN; ++j) sum[j] = 0.f;
            for (int u = 0; ok && u < units; ++u, ++uc) {
                const uint32_t b = uc & 1;
                if (!mbar_wait(&bar->acc_full[b], (uc >> 1) & 1, err, 0x204)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + b * ACC_COLS;
                // the smaller products first, then hi*hi (SPLIT_ACC)
#pragma unroll
                for (int part = 0; part < (SPLIT_ACC ? 2 : 1); ++part) {
#pragma unroll
                    for (int ch = 0; ch < UN / 32; ++ch) {
                        uint32_t v[32];
                        tmem_ld32(taddr + part * UN + ch * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) sum[ch * 32 + j] += __uint_as_float(v[j]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar->acc_empty[b]);
            }
            if (ok && row_ok) {
                // C0 read 16 values at a time, all requested before use, so
                // the loads' latencies overlap instead of adding up
#pragma unroll
                for (int g = 0; g < UN / 16; ++g) {
                    float cv[16];
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        cv[jj] = (p.beta_mode != 0 && col < p.n) ? p.cin[r + static_cast<size_t>(col) * p.ldc] : 0.f;
                    }
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        if (col < p.n) {
                            const float tb = (p.beta_mode == 2) ? p.beta_f * cv[jj] : cv[jj];
                            p.c[r + static_cast<size_t>(col) * p.ldc] = fmaf(p.alpha_f, sum[g * 16 + jj], tb);
                        }
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int MODE>
__global__ void __launch_bounds__(UCfg<MODE>::THREADS, 1)
    umma_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ UParams p) {
    umma_body<MODE>(USingleSrc{&p, &tmA, &tmB});
}

// Many f32 problems in one persistent launch (the serving loop's BF16-split
// batches): the same tiles and epilogue as umma_gemm_kernel.
template <int MODE>
__global__ void __launch_bounds__(UCfg<MODE>::THREADS, 1)
    umma_grouped_kernel(const UGroupEntry* __restrict__ tab, const int* __restrict__ starts, int nprob,
                        uint32_t* err) {
    umma_body<MODE>(UGroupSrc{tab, starts, nprob, err});
}

// ------------------------------------------------------------------------------
// The BF16-split GEMM on CTA pairs: 256 x 256 tiles, M = 256 N = 256 MMAs.
//
// 128 x 128 tiles take 83 bytes (3xBF16; BF16X6 62) of operands from L2 per SM
// and clock of MMA, twice what TMA was seen to land on all SMs at once (~40),
// so their tensor pipe waits. A pair's tile needs half of that: each CTA loads
// its 128 rows of A and its 128 of B for 256 x 256 outputs; the even CTA's
// warp 1 issues for both. (Shared memory itself is no limit: M = 128 N = 128
// MMAs kept their 64 clocks beside 112 bytes per clock of other writes.)
// 3xBF16 alternates two accumulators of 256 columns. BF16X6 keeps hi*hi apart
// (as umma_body does), which fills TMEM with one accumulator of each kind. A
// drain takes ~1200 clocks from the last MMA to the even CTA's knowing (the
// commit 300, the reads 340, the odd CTA's arrival 460), so a unit issues
// its small products first and its hi*hi ones (1024 clocks) last: the small
// accumulator drains behind hi*hi, and hi*hi's behind the next unit's small
// products. The hi planes then outlive the others of their stage and have a
// ring of their own. Within each accumulator the products keep umma_body's
// order, so the results are its bits.
// Per CTA: warp 0 TMA producer (both CTAs' loads of a stage complete on the even
// CTA's barrier); warp 1 TMEM owner and, in the even CTA, MMA issuer; warps
// 2..17 epilogue (four per TMEM lane quarter, 64 columns each).
// 8192^3, us a call (split pass included), 128 x 128 tiles -> pairs: 3xBF16
// 3316 -> 2319, BF16X6 5256 -> 4320; held by the power cap (SM clock 1.55 GHz).
// A cluster-scope release in the epilogue's arrival, which waits for the
// thread's stores, cost BF16X6 850 us; a word passed on by the odd CTA that its
// stage has landed, in place of loads that complete on the even CTA's barrier,
// 160 (without a release, which cost more still, it ordered nothing).
// ------------------------------------------------------------------------------
// KB: K bytes per stage row. Ring H holds the hi planes (HP of them per
// stage; every plane for 3xBF16), ring L the others.
template <int MODE> struct PairCfg;
template <> struct PairCfg<kModeBf16x3> { static constexpr int KB = 128, HP = 2, HS = 3, LP = 0, LS = 0; };  // 3 x 64 KiB
template <> struct PairCfg<kModeBf16x6> { static constexpr int KB = 64, HP = 1, HS = 6, LP = 2, LS = 4; };   // 6 x 16, 4 x 32 KiB
constexpr int kPairN = 256;
constexpr int kPairEpiWarps = 16;
constexpr int kPairCols = kPairN / (kPairEpiWarps / 4);  // columns per epilogue warp
constexpr int kPairThreads = 64 + 32 * kPairEpiWarps;
constexpr int kPairBarBytes = 512;
template <int MODE>
constexpr int pair_smem_bytes() {
    using P = PairCfg<MODE>;
    return 2 * 128 * P::KB * (P::HP * P::HS + P::LP * P::LS) + kPairBarBytes + 1024;
}
static_assert(pair_smem_bytes<kModeBf16x3>() <= 232448 && pair_smem_bytes<kModeBf16x6>() <= 232448,
              "the pair kernels' rings must fit one CTA's shared memory");

struct PairBar {
    uint64_t h_full[6], h_empty[6];  // (full: even CTA, a stage of both CTAs has landed)
    uint64_t l_full[4], l_empty[4];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];  // even CTA: both CTAs' epilogue warps
    uint64_t drain;
    uint32_t tmem_base;
    PairExit exit;
};
static_assert(sizeof(PairBar) <= kPairBarBytes, "shared memory reserved for the pair kernels' barriers");

using f32pair = unsigned long long;
__device__ __forceinline__ void add_f32pair(f32pair& s, uint32_t lo, uint32_t hi) {
    f32pair v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(s) : "l"(v));
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
    umma_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ UParams p) {
    using Cfg = UCfg<MODE>;
    using Pc = PairCfg<MODE>;
    constexpr int NP = Cfg::NA, KB = Pc::KB, HS = Pc::HS, LS = Pc::LS, HP = Pc::HP;
    constexpr int PL = 128 * KB;            // one plane's 128 rows
    constexpr int HSTAGE = 2 * HP * PL;     // A's planes, then B's
    constexpr int LSTAGE = 2 * Pc::LP * PL;
    constexpr bool TWO = LS > 0;            // two rings
    constexpr int SUB = kRowBytes / KB;     // stages per 64-element K tile
    constexpr int KSTEPS = KB / 32;
    constexpr uint32_t IDESC = umma_idesc(1, 1, 256, kPairN);  // f32 <- bf16
    constexpr bool SPLIT_ACC = (MODE == kModeBf16x6);
    static_assert(Cfg::NB == NP && HP + Pc::LP == NP && HS <= 6 && LS <= 4 && SPLIT_ACC == TWO, "rings");

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* lring = smem + HS * HSTAGE;
    PairBar* bar = reinterpret_cast<PairBar*>(lring + LS * LSTAGE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        for (int s = 0; s < HS; ++s) {
            mbar_init(&bar->h_full[s], 2);
            mbar_init(&bar->h_empty[s], 1);
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(&bar->l_full[s], 2);
            mbar_init(&bar->l_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar->acc_full[b], 1);
            mbar_init(&bar->acc_empty[b], 2 * kPairEpiWarps);
        }
        mbar_init(&bar->drain, 1);
        bar->exit = PairExit{};
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc_pair(&bar->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers are initialised too
    tc_fence_after();
    const uint32_t tmem_base = bar->tmem_base;
    uint32_t* const err = p.err;
    const int items = p.num_tiles, first = blockIdx.x >> 1, step = gridDim.x >> 1;
    const int stages = p.num_kt * SUB, per_unit = p.kt_per_chunk * SUB;
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // ------------------------------ TMA producer ------------------------------
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        uint32_t nh = 0, nl = 0;  // stages issued
        for (int item = first; ok && item < items; item += step) {
            int tm, tn;
            raster_tile(item, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * 256 + rank * 128, n0 = tn * kPairN + rank * 128;
            for (int kt = 0; kt < stages; ++kt) {
                const int k0 = kt * (KB / 2);
                const uint32_t hs = nh % HS;
                if (nh >= HS && !mbar_wait_cluster(&bar->h_empty[hs], ((nh / HS) - 1) & 1, err, 0x221)) {
                    ok = false;
                    break;
                }
                uint8_t* sh = smem + hs * HSTAGE;
                const uint32_t hf = cluster_addr(&bar->h_full[hs], 0);
                mbar_arrive_expect_tx_cluster(hf, HSTAGE);
#pragma unroll
                for (int q = 0; q < HP; ++q) tma_load_3d_pair(sh + q * PL, &tmA, hf, k0, m0, q);
#pragma unroll
                for (int q = 0; q < HP; ++q) tma_load_3d_pair(sh + (HP + q) * PL, &tmB, hf, k0, n0, q);
                ++nh;
                if constexpr (TWO) {
                    const uint32_t ls = nl % LS;
                    if (nl >= LS && !mbar_wait_cluster(&bar->l_empty[ls], ((nl / LS) - 1) & 1, err, 0x229)) {
                        ok = false;
                        break;
                    }
                    uint8_t* sl = lring + ls * LSTAGE;
                    const uint32_t lf = cluster_addr(&bar->l_full[ls], 0);
                    mbar_arrive_expect_tx_cluster(lf, LSTAGE);
#pragma unroll
                    for (int q = 0; q < Pc::LP; ++q) tma_load_3d_pair(sl + q * PL, &tmA, lf, k0, m0, HP + q);
#pragma unroll
                    for (int q = 0; q < Pc::LP; ++q)
                        tma_load_3d_pair(sl + (Pc::LP + q) * PL, &tmB, lf, k0, n0, HP + q);
                    ++nl;
                }
            }
        }
        st_cluster(&bar->exit.issued[0][rank], 0, nh);
        st_cluster(&bar->exit.issued[1][rank], 0, nl);
    } else if (warp == 1 && lane == 0 && rank == 0) {
        // ------------------------- even CTA: MMA issuer -------------------------
        uint32_t it = 0, uc = 0;
        auto landed = [&](uint32_t i) -> bool {  // stage i, in both CTAs
            if (!mbar_wait_cluster(&bar->h_full[i % HS], (i / HS) & 1, err, 0x223)) return false;
            if constexpr (TWO) {
                if (!mbar_wait_cluster(&bar->l_full[i % LS], (i / LS) & 1, err, 0x22b)) return false;
            }
            tc_fence_after();
            return true;
        };
        // A descriptor's low word is the address / 16 (plus a constant field)
        // and its high word constant: the issuing thread keeps low words and
        // adds constants, since the address arithmetic of a descriptor made
        // anew takes longer than the 128 clocks of an MMA.
        const uint64_t d0 = KB == 128 ? sw128_kmajor_desc(smem_u32(smem)) : sw64_kmajor_desc(smem_u32(smem));
        const uint32_t h_lo = static_cast<uint32_t>(d0), d_hi = static_cast<uint32_t>(d0 >> 32);
        const uint32_t l_lo = h_lo + HS * HSTAGE / 16;
        // the products Q0..Q1-1 of a stage (ring slots hs, ls) into d
        auto products = [&](uint32_t hs, uint32_t ls, auto q0, auto q1, uint32_t d, bool fresh) {
            const uint32_t hb = h_lo + hs * (HSTAGE / 16), lb = l_lo + ls * (LSTAGE / 16);
#pragma unroll
            for (int kk = 0; kk < KSTEPS; ++kk)
#pragma unroll
                for (int q = decltype(q0)::value; q < decltype(q1)::value; ++q) {
                    const int qa = Cfg::pa(q), qb = Cfg::pb(q);
                    const uint32_t a = (qa < HP ? hb + qa * (PL / 16) : lb + (qa - HP) * (PL / 16)) + 2 * kk;
                    const uint32_t b =
                        (qb < HP ? hb + (HP + qb) * (PL / 16) : lb + (Pc::LP + qb - HP) * (PL / 16)) + 2 * kk;
                    umma_f16_pair(d, (static_cast<uint64_t>(d_hi) << 32) | a, (static_cast<uint64_t>(d_hi) << 32) | b,
                                  IDESC, (kk == 0 && q == decltype(q0)::value) ? (fresh ? 0u : 1u) : 1u);
                }
        };
        using Q0 = std::integral_constant<int, 0>;
        using QB = std::integral_constant<int, Cfg::NPROD - 1>;
        using QN = std::integral_constant<int, Cfg::NPROD>;
        uint32_t hs = 0, ls = 0;  // ring slots of the next stage
        for (int item = first; ok && item < items; item += step) {
            for (int u = 0; ok && u < p.kchunks; ++u, ++uc) {
                const int n_st = min(per_unit, stages - u * per_unit);
                if constexpr (!SPLIT_ACC) {
                    const uint32_t b = uc & 1;
                    if (uc >= 2 && !mbar_wait_cluster(&bar->acc_empty[b], ((uc >> 1) - 1) & 1, err, 0x225)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    for (int j = 0; ok && j < n_st; ++j, ++it) {
                        ok = landed(it);
                        if (!ok) break;
                        products(hs, 0, Q0{}, QN{}, tmem_base + b * kPairN, j == 0);
                        tc_commit_pair(&bar->h_empty[hs]);
                        hs = hs + 1 == HS ? 0 : hs + 1;
                    }
                    if (ok) tc_commit_pair(&bar->acc_full[b]);
                } else {
                    if (uc >= 1 && !mbar_wait_cluster(&bar->acc_empty[0], (uc - 1) & 1, err, 0x226)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint32_t hj = hs;
                    for (int j = 0; ok && j < n_st; ++j) {
                        ok = landed(it + j);
                        if (!ok) break;
                        products(hj, ls, Q0{}, QB{}, tmem_base, j == 0);
                        tc_commit_pair(&bar->l_empty[ls]);
                        hj = hj + 1 == HS ? 0 : hj + 1;
                        ls = ls + 1 == LS ? 0 : ls + 1;
                    }
                    if (!ok) break;
                    tc_commit_pair(&bar->acc_full[0]);
                    if (uc >= 1 && !mbar_wait_cluster(&bar->acc_empty[1], (uc - 1) & 1, err, 0x227)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    for (int j = 0; j < n_st; ++j, ++it) {
                        products(hs, 0, QB{}, QN{}, tmem_base + kPairN, j == 0);
                        tc_commit_pair(&bar->h_empty[hs]);
                        hs = hs + 1 == HS ? 0 : hs + 1;
                    }
                    tc_commit_pair(&bar->acc_full[1]);
                }
            }
        }
        // nothing of ours is in flight before TMEM is released (arrives on the
        // odd CTA's copy too, which nobody waits on)
        tc_commit_pair(&bar->drain);
        mbar_wait_drain(&bar->drain, 0);
    } else if (warp >= 2) {
        // ------------------------------ epilogue ------------------------------
        const int quarter = warp & 3, cq = (warp - 2) >> 2;
        const int row_in_tile = quarter * 32 + lane;
        const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + cq * kPairCols;
        uint32_t uc = 0;
        for (int item = first; ok && item < items; item += step) {
            int tm, tn;
            raster_tile(item, p.tiles_m, p.tiles_n, tm, tn);
            const int r = tm * 256 + static_cast<int>(rank) * 128 + row_in_tile, n0 = tn * kPairN + cq * kPairCols;
            f32pair sum[kPairCols / 2];
#pragma unroll
            for (int j = 0; j < kPairCols / 2; ++j) sum[j] = 0ull;
            for (int u = 0; ok && u < p.kchunks; ++u, ++uc) {
                // the smaller products first, then hi*hi (SPLIT_ACC)
#pragma unroll 1
                for (int part = 0; part < (SPLIT_ACC ? 2 : 1); ++part) {
                    const uint32_t b = SPLIT_ACC ? part : (uc & 1);
                    const uint32_t ph = SPLIT_ACC ? (uc & 1) : ((uc >> 1) & 1);
                    const bool got = mbar_wait_cluster(&bar->acc_full[b], ph, err, 0x228);
                    if (!__all_sync(0xffffffffu, got)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int ch = 0; ch < kPairCols / 16; ++ch) {
                        uint32_t v[16];
                        tmem_ld16(tbase + b * kPairN + ch * 16, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; ++j) add_f32pair(sum[ch * 8 + j], v[2 * j], v[2 * j + 1]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_rank_relaxed(&bar->acc_empty[b], 0);
                }
            }
            if (ok && r < p.m) {
                // C0 read 16 values at a time, all requested before use
#pragma unroll
                for (int g = 0; g < kPairCols / 16; ++g) {
                    float cv[16];
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        cv[jj] = (p.beta_mode != 0 && col < p.n) ? p.cin[r + static_cast<size_t>(col) * p.ldc] : 0.f;
                    }
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        if (col < p.n) {
                            float lo, hi;
                            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(sum[g * 8 + jj / 2]));
                            const float tb = (p.beta_mode == 2) ? p.beta_f * cv[jj] : cv[jj];
                            p.c[r + static_cast<size_t>(col) * p.ldc] = fmaf(p.alpha_f, (jj & 1) ? hi : lo, tb);
                        }
                    }
                }
            }
        }
    }

    if (!ok) pair_fail(&bar->exit);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // no CTA leaves while the other may still reach its memory
    if (bar->exit.failed) {  // in both CTAs
        if (rank == 0 && threadIdx.x == 0) {
            pair_drain(bar->h_full, HS, bar->exit.issued[0]);
            if constexpr (TWO) pair_drain(bar->l_full, LS, bar->exit.issued[1]);
        }
        cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------
// The BF16-split forms with A split inside the GEMM (A rows contiguous:
// NoTrans), on CTA pairs: 256 x 128 tiles.
//
// Two passes read A, write its planes and read the planes again: about three
// times A's bytes, which is most of the time of a tall-skinny product
// (65536 x 128 x 8192: A is 2.1 GB). Here TMA brings 128 x 64 f32 tiles of A
// (128 contiguous rows per K column) into shared memory, and the epilogue
// warps split them, between their accumulator promotions, into the planes
// (hi, lo for 3xBF16; hi, mid, lo for BF16X6): for 3xBF16 into TMEM, as the
// MMA's A operand (row = lane, two K values per column), beside the
// accumulators' 256 columns; for BF16X6, whose accumulators fill TMEM, into the
// 128-byte-swizzled K-major tiles that a TMA load of planes gives (row r's
// 16-byte chunk c at r * 128 + ((c ^ (r & 7)) * 16)). The split is the split
// pass's (hi = rn(x), then each next plane rn of what is left) and the
// products, their order, the accumulators and the promotions are
// umma_gemm_kernel<MODE>'s, so the results are the two-pass form's bit for
// bit. B's planes come from the split pass (B is small), half of a tile's
// columns to each CTA.
// Rings: A's f32 tiles (released as soon as the splitters hold them in
// registers); stages of A's planes and B's planes, released together by the
// MMAs' one commit. B's loads and the splitter warps of both CTAs arrive on the
// even CTA's barriers.
// Warps: 0 producer of A's tiles; 1 TMEM owner and, in the even CTA, MMA issuer
// for both; 2 producer of B's planes; 3..18 splitter and epilogue: tile row
// quarter * 32 + lane (quarter = warp % 4, the TMEM lanes the warp may use) in
// both roles; K values 32 half .. + 31 of every second K tile to split (so that
// one tile's loads overlap the other's stores), columns 32 part .. + 31 of the
// tile to promote and write.
// Bound: A's bytes from memory. 65536 x 128 x 8192 back to back, 3xBF16: 430 us
// (A at 5.1 TB/s, its four waves 86 % full), BF16X6 765 (24 MMAs of 64 clocks a
// K tile); on single CTAs with planes in shared memory, one splitter group and
// one issuing lane, 634 and 900: the issuing lane took ~110 clocks an MMA.
// BF16X6's planes of the odd CTA are read by the even one's MMAs, so its
// splitters release them to the cluster, ~1000 clocks that two stages hide only
// in part: each half of a stage's K is handed over and freed by itself (805
// whole).
// Splitting with 16 warps a tile instead of two groups of 8: 523 and 768. Tiles
// of 112 rows, which fill the fourth wave, took longer (471): their columns
// start inside 128-byte lines.
// ------------------------------------------------------------------------------
template <int MODE> struct FzCfg;
template <> struct FzCfg<kModeBf16x3> { static constexpr int FS = 4, RS = 4; static constexpr bool A_TMEM = true; };
template <> struct FzCfg<kModeBf16x6> { static constexpr int FS = 2, RS = 2; static constexpr bool A_TMEM = false; };
constexpr int kFzEpiWarps = 16;
constexpr int kFzThreads = 96 + 32 * kFzEpiWarps;
constexpr int kFzN = 128;                 // tile columns
constexpr int kFzF32Tile = kUM * 64 * 4;  // 64 K columns of 128 f32 rows: 32 KiB
constexpr int kFzBTile = kFzN / 2 * kRowBytes;
constexpr int kFzUnit = 2;  // K tiles to a promotion (kt_per_chunk): one per splitter group
template <int MODE>
constexpr int fz_smem_bytes() {
    using F = FzCfg<MODE>;
    return F::FS * kFzF32Tile + F::RS * UCfg<MODE>::NA * (kFzBTile + (F::A_TMEM ? 0 : kATile)) + 256 + 1024;
}
static_assert(fz_smem_bytes<kModeBf16x3>() <= 232448 && fz_smem_bytes<kModeBf16x6>() <= 232448,
              "the fused kernels' rings must fit one CTA's shared memory");

struct FzBar {
    uint64_t f_full[4], f_empty[4];  // A's f32 tiles
    uint64_t a_full[4];              // plane stages (even CTA): both CTAs' splits of A are there (each half of K by itself
                                     // where the planes are in shared memory)
    uint64_t b_full[4];              // and loads of B
    uint64_t empty[4];               // the pair's MMAs have read them (of A, the first half of K: empty0)
    uint64_t empty0[2];
    uint64_t acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    uint32_t issued_f;  // f32 tiles that this CTA's producer issued
    PairExit exit;
};
static_assert(sizeof(FzBar) <= 256, "the fused kernels reserve 256 bytes of shared memory for their barriers");

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kFzThreads, 1)
    umma_split_fused_kernel(const __grid_constant__ CUtensorMap tmA32, const __grid_constant__ CUtensorMap tmB,
                            const __grid_constant__ UParams p) {
    using Cfg = UCfg<MODE>;
    constexpr int NP = Cfg::NA, FS = FzCfg<MODE>::FS, RS = FzCfg<MODE>::RS;
    constexpr bool A_TMEM = FzCfg<MODE>::A_TMEM;
    static_assert(FS <= 4 && RS <= 4 && Cfg::NB == NP, "FzBar holds the rings; A and B have the same planes");
    // a slot's tiles then are all one splitter group's, whose waits on it see
    // every phase (copies may land out of order)
    static_assert(FS % 2 == 0 && RS % 2 == 0, "even rings");
    constexpr int KSTEPS = 4;
    constexpr int KH = A_TMEM ? 1 : 2;  // parts of a stage that A's planes are handed over in
    static_assert(RS * KH <= 4 && (KH == 1 || RS <= 2), "FzBar holds the parts' barriers");
    constexpr uint32_t IDESC = umma_idesc(1, 1, 256, kFzN);  // f32 <- bf16
    // BF16X6 keeps hi*hi in an accumulator of its own, as umma_body does
    constexpr bool SPLIT_ACC = (MODE == kModeBf16x6);
    constexpr uint32_t ACC_COLS = SPLIT_ACC ? 2 * kFzN : kFzN;  // per accumulator buffer
    constexpr uint32_t A_COL = 2 * ACC_COLS;                    // TMEM columns of A's planes, 32 each
    static_assert(A_COL + (A_TMEM ? RS * NP * 32 : 0) <= 512, "accumulators and planes fit TMEM");

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* f32s = smem;                           // FS x 32 KiB, [k][row] f32
    uint8_t* bps = f32s + FS * kFzF32Tile;          // RS x NP planes, by TMA
    uint8_t* aps = bps + RS * NP * kFzBTile;        // RS x NP planes, swizzled K-major (BF16X6)
    FzBar* bar = reinterpret_cast<FzBar*>(aps + (A_TMEM ? 0 : RS * NP * kATile));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        for (int s = 0; s < FS; ++s) {
            mbar_init(&bar->f_full[s], 1);
            mbar_init(&bar->f_empty[s], kFzEpiWarps / 2);
        }
        for (int s = 0; s < RS; ++s) {
            for (int h = 0; h < KH; ++h) mbar_init(&bar->a_full[s * KH + h], 2 * (kFzEpiWarps / 2) / KH);
            mbar_init(&bar->b_full[s], 2);
            mbar_init(&bar->empty[s], 1);
            if (KH == 2) mbar_init(&bar->empty0[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bar->acc_full[b], 1);
            mbar_init(&bar->acc_empty[b], 2 * kFzEpiWarps);
        }
        mbar_init(&bar->drain, 1);
        bar->exit = PairExit{};
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc_pair(&bar->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers are initialised too
    tc_fence_after();
    const uint32_t tmem_base = bar->tmem_base;
    const int items = p.num_tiles, first = blockIdx.x >> 1, step = gridDim.x >> 1;
    uint32_t* const err = p.err;
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // ------------------------------ TMA producer ------------------------------
        prefetch_tmap(&tmA32);
        uint32_t it = 0, fs = 0, ph = 1;  // tiles issued, ring slot, the phase to wait for
        for (int item = first; ok && item < items; item += step) {
            int tm, tn;
            raster_tile(item, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * 256 + rank * 128;
            for (int kt = 0; kt < p.num_kt; ++kt, ++it) {
                if (!mbar_wait(&bar->f_empty[fs], ph, err, 0x211)) {  // (a fresh slot's wait passes)
                    ok = false;
                    break;
                }
                mbar_arrive_expect_tx(&bar->f_full[fs], kFzF32Tile);
                tma_load_2d(f32s + fs * kFzF32Tile, &tmA32, &bar->f_full[fs], m0, kt * 64);
                if (++fs == FS) {
                    fs = 0;
                    ph ^= 1;
                }
            }
        }
        bar->issued_f = it;
    } else if (warp == 2 && lane == 0) {
        prefetch_tmap(&tmB);
        uint32_t it = 0, rs = 0, ph = 1;
        for (int item = first; ok && item < items; item += step) {
            int tm, tn;
            raster_tile(item, p.tiles_m, p.tiles_n, tm, tn);
            const int n0 = tn * kFzN + rank * (kFzN / 2);
            for (int kt = 0; kt < p.num_kt; ++kt, ++it) {
                if (!mbar_wait_cluster(&bar->empty[rs], ph, err, 0x212)) {
                    ok = false;
                    break;
                }
                const uint32_t bf = cluster_addr(&bar->b_full[rs], 0);
                mbar_arrive_expect_tx_cluster(bf, NP * kFzBTile);
#pragma unroll
                for (int q = 0; q < NP; ++q) tma_load_3d_pair(bps + (rs * NP + q) * kFzBTile, &tmB, bf, kt * 64, n0, q);
                if (++rs == RS) {
                    rs = 0;
                    ph ^= 1;
                }
            }
        }
        st_cluster(&bar->exit.issued[0][rank], 0, it);
    } else if (warp == 1 && rank == 0) {
        // ------------------------- even CTA: MMA issuer -------------------------
        // (the whole warp runs the loop, one lane issues: see elect_one)
        const bool lead = elect_one();
        const uint64_t d0 = sw128_kmajor_desc(smem_u32(bps));  // (see umma_pair_kernel on descriptors)
        const uint32_t b_lo = static_cast<uint32_t>(d0), a_lo = b_lo + RS * NP * kFzBTile / 16;
        const uint64_t d_hi = d0 & 0xffffffff00000000ull;
        uint32_t uc = 0, rs = 0, ph = 0;  // ring slot and its phase
        for (int item = first; ok && item < items; item += step) {
            for (int u = 0; ok && u < p.kchunks; ++u, ++uc) {
                const int kt0 = u * kFzUnit, kt1 = min(p.num_kt, kt0 + kFzUnit);
                const uint32_t b = uc & 1;
                if (uc >= 2) ok = mbar_wait_cluster(&bar->acc_empty[b], ((uc >> 1) - 1) & 1, err, 0x213);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + b * ACC_COLS;         // the products (all, or all but hi*hi)
                const uint32_t d_big = SPLIT_ACC ? d_tmem + kFzN : d_tmem;  // hi*hi
                for (int kt = kt0; kt < kt1; ++kt) {
                    ok = mbar_wait_cluster(&bar->b_full[rs], ph, err, 0x214);
                    const uint32_t sb = b_lo + rs * (NP * kFzBTile / 16), sa = a_lo + rs * (NP * kATile / 16);
                    const uint32_t ta = tmem_base + A_COL + rs * (NP * 32);
#pragma unroll
                    for (int h = 0; h < KH; ++h) {
                        if (ok) ok = mbar_wait_cluster(&bar->a_full[rs * KH + h], ph, err, 0x215);
                        if (!__all_sync(0xffffffffu, ok)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int kk = h * (KSTEPS / KH); kk < (h + 1) * (KSTEPS / KH); ++kk)
#pragma unroll
                            for (int q = 0; q < Cfg::NPROD; ++q) {
                                const bool big = SPLIT_ACC && q == Cfg::NPROD - 1;
                                const uint32_t d = big ? d_big : d_tmem;
                                const uint32_t acc = (kk == 0 && (q == 0 || big)) ? (kt != kt0) : 1u;
                                const uint64_t db = d_hi | (sb + Cfg::pb(q) * (kFzBTile / 16) + 2 * kk);
                                if constexpr (A_TMEM) {
                                    if (lead) umma_f16_pair_ts(d, ta + Cfg::pa(q) * 32 + kk * 8, db, IDESC, acc);
                                } else {
                                    if (lead)
                                        umma_f16_pair(d, d_hi | (sa + Cfg::pa(q) * (kATile / 16) + 2 * kk), db, IDESC, acc);
                                }
                            }
                        // free, in both CTAs, once these MMAs complete
                        if (lead) tc_commit_pair(h + 1 < KH ? &bar->empty0[rs] : &bar->empty[rs]);
                    }
                    if (!ok) break;
                    if (++rs == RS) {
                        rs = 0;
                        ph ^= 1;
                    }
                }
                if (ok && lead) tc_commit_pair(&bar->acc_full[b]);
            }
        }
        // nothing of ours is in flight before TMEM is released (arrives on the
        // odd CTA's copy too, which nobody waits on)
        if (lead) tc_commit_pair(&bar->drain);
        mbar_wait_drain(&bar->drain, 0);
    } else if (warp >= 3) {
        // ------------------------- splitter and epilogue -------------------------
        constexpr int HC = kFzN / 4;  // columns per warp
        const int quarter = warp & 3, part = (warp - 3) >> 2, half = part >> 1;
        const int row = quarter * 32 + lane;  // tile row: TMEM lane and split row
        const uint32_t tlane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        uint32_t uc = 0, it = 0;  // units promoted, K tiles before this item
        for (int item = first; ok && item < items; item += step) {
            int tm, tn;
            raster_tile(item, p.tiles_m, p.tiles_n, tm, tn);
            const int n0 = tn * kFzN + part * HC;
            const int r = tm * 256 + static_cast<int>(rank) * 128 + row;
            f32pair sum[HC / 2];
#pragma unroll
            for (int j = 0; j < HC / 2; ++j) sum[j] = 0ull;
            int promoted = 0;
            // add unit `promoted`'s FP32 partial (TMEM) into sum, as umma_body does
            auto promote = [&]() -> bool {
                const uint32_t b = uc & 1;
                const bool got = mbar_wait_cluster(&bar->acc_full[b], (uc >> 1) & 1, err, 0x216);
                if (!__all_sync(0xffffffffu, got)) return false;
                tc_fence_after();
                // the smaller products first, then hi*hi (SPLIT_ACC)
#pragma unroll
                for (int ch = 0; ch < (SPLIT_ACC ? 2 : 1); ++ch) {
                    uint32_t v[HC];
                    tmem_ld32(tlane + b * ACC_COLS + ch * kFzN + part * HC, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < HC / 2; ++j) add_f32pair(sum[j], v[2 * j], v[2 * j + 1]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_rank_relaxed(&bar->acc_empty[b], 0);
                ++uc;
                ++promoted;
                return true;
            };
            // this group's K tiles: every second one over all items
            for (int kt = (it ^ part) & 1; kt < p.num_kt; kt += 2) {
                const uint32_t i = it + kt, fs = i % FS, rs = i % RS;
                bool got = mbar_wait_inline(&bar->f_full[fs], (i / FS) & 1, err, 0x218);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                // this warp's half of the row's 64 K values
                float v[32];
                {
                    // F[k * 128 + row]
                    const float* F = reinterpret_cast<const float*>(f32s + fs * kFzF32Tile) + half * 32 * kUM + row;
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = F[e * kUM];
                }
                // the f32 stage is free: every lane's reads are done
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar->f_empty[fs]);
                // (a fresh slot's wait passes)
                got = mbar_wait_cluster(half + 1 < KH ? &bar->empty0[rs] : &bar->empty[rs], (i / RS + 1) & 1, err, 0x217);
                if (!__all_sync(0xffffffffu, got)) {
                    ok = false;
                    break;
                }
                if constexpr (A_TMEM) tc_fence_after();
                uint8_t* const dst = aps + rs * NP * kATile + row * kRowBytes;
                // split 8 (16) values at a time into NP planes of packed
                // bf16 pairs: pl[q][j] holds plane q of K values 2 j (low
                // half) and 2 j + 1 (high half)
                constexpr int G = A_TMEM ? 16 : 8;
#pragma unroll
                for (int g = 0; g < 32 / G; ++g) {
                    uint32_t pl[NP][G / 2];
#pragma unroll
                    for (int j = 0; j < G / 2; ++j) {
                        float v0 = v[g * G + 2 * j], v1 = v[g * G + 2 * j + 1];
#pragma unroll
                        for (int q = 0; q < NP; ++q) {
                            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(pl[q][j]) : "f"(v1), "f"(v0));
                            if (q + 1 < NP)
                                asm("{\n\t.reg .b64 v, b, n;\n\t"
                                    "mov.b64 v, {%0, %1};\n\t"
                                    "mov.b64 b, {%2, %3};\n\t"
                                    "mov.b64 n, 0xbf800000bf800000;\n\t"  // -1, -1
                                    "fma.rn.f32x2 v, b, n, v;\n\t"
                                    "mov.b64 {%0, %1}, v;\n\t}"
                                    : "+f"(v0), "+f"(v1)
                                    : "r"(pl[q][j] << 16), "r"(pl[q][j] & 0xffff0000u));
                        }
                    }
                    if constexpr (A_TMEM) {
#pragma unroll
                        for (int q = 0; q < NP; ++q)
                            tmem_st8(tlane + A_COL + (rs * NP + q) * 32 + half * 16 + g * 8, pl[q]);
                    } else {
                        const uint32_t off = ((half * 4 + g) ^ (row & 7)) << 4;
#pragma unroll
                        for (int q = 0; q < NP; ++q)
                            *reinterpret_cast<uint4*>(dst + q * kATile + off) =
                                make_uint4(pl[q][0], pl[q][1], pl[q][2], pl[q][3]);
                    }
                }
                if constexpr (A_TMEM) {
                    tmem_st_wait();
                    tc_fence_before();
                } else {
                    fence_proxy_async_smem();  // the planes' generic stores, visible to the tensor cores
                }
                __syncwarp();
                if (lane == 0) {
                    if constexpr (A_TMEM) mbar_arrive_rank_relaxed(&bar->a_full[rs], 0);
                    else if (rank == 0)   mbar_arrive(&bar->a_full[rs * KH + half]);
                    else                  mbar_arrive_rank_release(&bar->a_full[rs * KH + half], 0);
                }
                // once this group's part of unit u is split, unit u - 1 is promoted:
                // the MMAs of unit u + 1 wait for that buffer
                if (kt >= kFzUnit && !promote()) {
                    ok = false;
                    break;
                }
            }
            it += p.num_kt;
            while (ok && promoted < p.kchunks)
                if (!promote()) ok = false;
            if (ok && r < p.m) {
                // C0 read 16 values at a time, all requested before use
#pragma unroll
                for (int g = 0; g < HC / 16; ++g) {
                    float cv[16];
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        cv[jj] = (p.beta_mode != 0 && col < p.n) ? p.cin[r + static_cast<size_t>(col) * p.ldc] : 0.f;
                    }
#pragma unroll
                    for (int jj = 0; jj < 16; ++jj) {
                        const int col = n0 + g * 16 + jj;
                        if (col < p.n) {
                            float lo, hi;
                            asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(sum[g * 8 + jj / 2]));
                            const float tb = (p.beta_mode == 2) ? p.beta_f * cv[jj] : cv[jj];
                            p.c[r + static_cast<size_t>(col) * p.ldc] = fmaf(p.alpha_f, (jj & 1) ? hi : lo, tb);
                        }
                    }
                }
            }
        }
    }

    if (!ok) pair_fail(&bar->exit);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // no CTA leaves while the other may still reach its memory
    if (bar->exit.failed) {  // in both CTAs
        if (threadIdx.x == 0)  // this CTA's own tiles of A
            for (uint32_t n = bar->issued_f, j = n > (uint32_t)FS ? n - FS : 0; j < n; ++j)
                mbar_wait_drain(&bar->f_full[j % FS], (j / FS) & 1);
        if (rank == 0 && threadIdx.x == 0) pair_drain(bar->b_full, RS, bar->exit.issued[0]);
        cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// ------------------------------------------------------------------------------
// Ozaki GEMM kernel.
//
// Slice products of equal weight (t + u = d: digit t has weight 2^-(7+8t))
// form diagonal d; S_d = sum_{t+u=d} A_t B_u^T is exact in INT32 over a K
// chunk. Diagonals are processed two at a time ("units" {d0, d1 = d0+1})
// with both accumulators in TMEM (2 x 256 columns). For each K tile the
// stages walk the A slices i = d1 .. 0, stage i holding A_i and B_{d1-i}:
// S_d1 takes A_i x B_{d1-i} from the stage, S_d0 takes A_i x B_{d0-i}, which
// is the B tile of the previous stage. So every stage brings one new A and
// one new B tile (48 KiB) for two MMAs, and a stage is released once the
// next one's MMAs have been issued. (The order of the INT32 additions does
// not change the exact sums.) The epilogue folds the unit exactly,
// S_d0 * 2^8 + S_d1 (< 2^40), scales by alpha * 2^(e_i + f_j + 2 - 14 -
// 8 d1) and accumulates into C in FP64; units run from the smallest weight
// up, the first one adding beta*C0.
// Warps: 0 TMA producer, 1 TMEM owner / MMA issuer, 2..17 epilogue (four
// warps per TMEM lane quarter, UN/4 columns each). With the 128 x 256 tile a
// unit's two accumulators fill TMEM, so the tensor cores wait while the
// epilogue drains them; the epilogue is written for that latency: 16 warps,
// a per-warp table of the tile's column scales in shared memory, and the
// first chunk's C values requested before the accumulator wait. The
// 128 x 128 tile keeps two sets of accumulators and alternates them, so its
// drain overlaps the next unit's MMAs.
// ------------------------------------------------------------------------------

constexpr int kOzEpiWarps = 16;
constexpr int kOzThreads = 64 + 32 * kOzEpiWarps;
constexpr int kOzColTab = 64 * (8 + 4);             // per epilogue warp: 2^fc (double) and fc (int), 64 columns
// Per tile width UN (256, or 128 for narrow problems): stages of
// (B_{d1-i}, A_i), their bytes, the columns each epilogue warp drains, and
// the dynamic shared memory.
template <int UN>
struct OzCfg {
    static_assert(UN == 256 || UN == 128, "Ozaki tiles are 128 x 256 or 128 x 128");
    static constexpr int ST = UN == 256 ? 4 : 6;
    static_assert(ST <= kMaxStages, "Bar holds kMaxStages stages");
    static constexpr int BTILE = UN * kRowBytes;
    static constexpr int STAGE = kATile + BTILE;  // 48 KiB / 32 KiB
    static constexpr int CW = UN / 4;             // four epilogue warps per TMEM lane quarter
    static constexpr int SMEM = ST * STAGE + 256 + kOzEpiWarps * kOzColTab + 1024;
    // accumulator sets of 2 x UN columns in TMEM's 512: the 128-wide tile
    // keeps two, so the MMAs of the next unit run while this one drains
    static constexpr int NBUF = 512 / (2 * UN);
};
// Tile rows per rasterisation group. A wave of 148 tiles walks R row panels
// of A and C column panels of B, each once per diagonal-pair unit; B panels
// (256 columns) are twice the A panels (128 rows), so R ~ 2C (16 x ~9)
// moves fewer digit-plane bytes through L2 than the 8 x ~18 of the plain
// kernels.
constexpr int kOzRaster = 16;

constexpr int kOzGroups = 3;  // groups of four diagonals, slices <= 12

struct OzParams {
    int m, n, k;
    int tiles_m, tiles_n, num_tiles;
    int num_kt;        // 128-byte K tiles
    int slices;
    int kt_per_chunk;  // exact-INT32 K chunk
    int kchunks;
    int beta_mode;
    double alpha, beta;
    double* c;
    size_t ldc;
    const double* cin;  // C0, read for beta != 0: c itself, or a separate input with c's leading dimension
    const int* row_exp;
    const int* col_exp;
    uint32_t* err;
    // Split tail: the last tail_tiles tiles (in raster order) run as one work
    // item per (tile, unit). Such an item's epilogue writes the unit's exact
    // FP64 terms to its own plane of ws (kUM * un doubles per tile and unit,
    // element (row, col) of the tile at row + col * kUM), and
    // ozaki_reduce_kernel folds the planes into C in unit order afterwards:
    // the same operations as the fused epilogue, so the same bits. Used where
    // whole tiles would leave SMs idle (a partial last wave, or fewer tiles
    // than SMs). 0: every tile fused.
    double* ws;
    int tail_tiles;
    int un;  // tile width (256 or 128): the split tail's plane size and the reduce kernel's tiling
    // Pair kernel's tail (see ozaki_pair_kernel): K parts of each group of
    // four diagonals, the groups in order of an item's cost (dearest first),
    // and the first workspace plane of each within a tile's `planes`.
    int parts[kOzGroups], order[kOzGroups], plane0[kOzGroups], planes;
};

// 2^x for x in [-1022, 1023]
__device__ __forceinline__ double pow2_normal(int x) {
    return __longlong_as_double(static_cast<long long>(x + 1023) << 52);
}

// v * 2^x: one multiply by an exactly representable power of two (the same
// single rounding as scalbn), scalbn only where 2^x is not a double.
__device__ __forceinline__ double scale_pow2(double v, int x) {
    if (x >= -1022 && x <= 1023) return v * __longlong_as_double(static_cast<long long>(x + 1023) << 52);
    if (x >= -1074 && x < -1022) return v * __longlong_as_double(1LL << (x + 1074));
    return scalbn(v, x);
}

// unit u (0-based) of a chunk covers diagonals d0 and d1 = d0 + 1 (d1 < 0
// when absent); units go from the highest diagonals down.
__host__ __device__ __forceinline__ void oz_unit(int slices, int u, int& d0, int& d1) {
    const int units = (slices + 1) / 2;
    d0 = 2 * (units - 1 - u);
    d1 = (d0 + 1 < slices) ? d0 + 1 : -1;
}

// Work item -> tile t and units [u_lo, u_hi). Items below the fused count are
// whole tiles (tt = -1). The others are single units of the tail tiles (tt:
// index among them), ranked by cost -- pair 0 of a chunk, the highest
// diagonals, has the most products -- and dealt to the CTAs in a snake, so
// a CTA that took an expensive unit in one pass takes a cheap one in the
// next. G is the grid size; any G gives a bijection, the balance assumes the
// fused count is a multiple of G.
__host__ __device__ __forceinline__ void oz_item(int num_tiles, int tail_tiles, int kchunks, int upc, int G,
                                                 int item, int& t, int& u_lo, int& u_hi, int& tt) {
    const int fused = num_tiles - tail_tiles;
    if (item < fused) {
        t = item;
        u_lo = 0;
        u_hi = kchunks * upc;
        tt = -1;
        return;
    }
    const int j = item - fused;
    const int total = tail_tiles * kchunks * upc;
    const int pass = j / G, q = j - pass * G;
    const int len = (total - pass * G < G) ? total - pass * G : G;
    const int rank = (pass & 1) ? pass * G + (len - 1 - q) : j;
    const int per_pair = tail_tiles * kchunks;
    const int pair = rank / per_pair, rest = rank - pair * per_pair;
    const int chunk = rest / tail_tiles;
    tt = rest - chunk * tail_tiles;
    t = fused + tt;
    u_lo = chunk * upc + pair;
    u_hi = u_lo + 1;
}

// One problem of a grouped Ozaki launch: its digit-plane tensor maps (TMA
// reads them from global memory: 64-byte aligned) and its parameters.
struct alignas(64) OzGroupEntry {
    CUtensorMap tmA, tmB;
    OzParams p;
};

// One work item as a CTA sees it: its problem, tile and units (oz_item).
struct OzWork {
    const OzParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    int t, u_lo, u_hi, tt;
};

// Work of the single-problem kernel: whole tiles, then the split tail's
// units (oz_item).
struct OzSingleSrc {
    const OzParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    __device__ __forceinline__ uint32_t* err() const { return p->err; }
    __device__ __forceinline__ int items() const {
        const int units = p->kchunks * ((p->slices + 1) / 2);
        return p->num_tiles + p->tail_tiles * (units - 1);
    }
    __device__ __forceinline__ OzWork get(int item) const {
        OzWork w{p, ta, tb, 0, 0, 0, -1};
        oz_item(p->num_tiles, p->tail_tiles, p->kchunks, (p->slices + 1) / 2, gridDim.x, item, w.t, w.u_lo, w.u_hi,
                w.tt);
        return w;
    }
};

// Work of the grouped kernel: item i is one whole tile (fused epilogue, every
// unit) of problem j, where starts[j] <= i < starts[j+1]. The host orders the
// problems by the cost of one tile, largest first, so the CTAs' strided walk
// over the items deals the long tiles out first.
struct OzGroupSrc {
    const OzGroupEntry* tab;
    const int* starts;
    int nprob;
    uint32_t* error;
    __device__ __forceinline__ uint32_t* err() const { return error; }
    __device__ __forceinline__ int items() const { return __ldg(starts + nprob); }
    __device__ __forceinline__ OzWork get(int item) const {
        int lo = 0, hi = nprob - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(starts + mid) <= item) lo = mid;
            else hi = mid - 1;
        }
        const OzGroupEntry* g = tab + lo;
        OzWork w{&g->p, &g->tmA, &g->tmB, item - __ldg(starts + lo), 0, 0, -1};
        w.u_hi = g->p.kchunks * ((g->p.slices + 1) / 2);
        return w;
    }
};

template <int UN, class Src>
__device__ __forceinline__ void ozaki_body(const Src& src) {
    using Cfg = OzCfg<UN>;
    constexpr int ST = Cfg::ST, CW = Cfg::CW, NCH = CW / 8;
    constexpr int TILE_ELEMS = kUM * UN;
    constexpr int KSTEPS = 4;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    Bar* bar = reinterpret_cast<Bar*>(smem + ST * Cfg::STAGE);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&bar->full[s], 1);
            mbar_init(&bar->empty[s], 1);
        }
        for (int b = 0; b < Cfg::NBUF; ++b) {
            mbar_init(&bar->acc_full[b], 1);
            mbar_init(&bar->acc_empty[b], kOzEpiWarps);
        }
        mbar_init(&bar->drain, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(&bar->tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bar->tmem_base;
    const int items = src.items();
    uint32_t* const err = src.err();
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // ------------------------------ TMA producer ------------------------------
        uint32_t it = 0;
        const CUtensorMap* fetched = nullptr;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const OzWork w = src.get(item);
            const OzParams& p = *w.p;
            if (w.ta != fetched) {
                prefetch_tmap(w.ta);
                prefetch_tmap(w.tb);
                fetched = w.ta;
            }
            const int upc = (p.slices + 1) / 2;
            int tm, tn;
            raster_tile<kOzRaster>(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * kUM, n0 = tn * UN;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u) {
                int d0, d1;
                oz_unit(p.slices, u % upc, d0, d1);
                const int kt0 = (u / upc) * p.kt_per_chunk, kt1 = min(p.num_kt, kt0 + p.kt_per_chunk);
                const int top = d1 >= 0 ? d1 : d0;
                for (int kt = kt0; ok && kt < kt1; ++kt) {
                    const int k0 = kt * 128;
                    for (int i = top; ok && i >= 0; --i, ++it) {  // stage: A_i and B_{top-i}
                        const int s = it % ST;
                        if (it >= ST && !mbar_wait(&bar->empty[s], ((it / ST) - 1) & 1, err, 0x301)) {
                            ok = false;
                            break;
                        }
                        uint8_t* sb = smem + s * Cfg::STAGE;
                        uint8_t* sa = sb + Cfg::BTILE;
                        mbar_arrive_expect_tx(&bar->full[s], Cfg::BTILE + kATile);
                        tma_load_3d(sb, w.tb, &bar->full[s], k0, n0, top - i);
                        tma_load_3d(sa, w.ta, &bar->full[s], k0, m0, i);
                    }
                }
            }
        }
        if (!ok) {
            const uint32_t first = it > (uint32_t)ST ? it - ST : 0;
            for (uint32_t j = first; j < it; ++j) mbar_wait_drain(&bar->full[j % ST], (j / ST) & 1);
        }
    } else if (warp == 1 && lane == 0) {
        // ------------------------------ MMA issuer ------------------------------
        uint32_t it = 0, uc = 0;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const OzWork w = src.get(item);
            const OzParams& p = *w.p;
            const int upc = (p.slices + 1) / 2;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u, ++uc) {
                int d0, d1;
                oz_unit(p.slices, u % upc, d0, d1);
                const int kt0 = (u / upc) * p.kt_per_chunk, kt1 = min(p.num_kt, kt0 + p.kt_per_chunk);
                const int bsel = static_cast<int>(uc % Cfg::NBUF);
                if (uc >= static_cast<uint32_t>(Cfg::NBUF) &&
                    !mbar_wait(&bar->acc_empty[bsel], ((uc / Cfg::NBUF) - 1) & 1, err, 0x302)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                // S_top (d1, or d0 alone) at acc + UN for a pair, acc otherwise;
                // S_d0 of a pair at acc (the epilogue's layout)
                const uint32_t acc = tmem_base + bsel * (2 * UN);
                const bool pair = d1 >= 0;
                const int top = pair ? d1 : d0;
                const uint32_t acc_top = pair ? acc + UN : acc;
                constexpr uint32_t idesc = umma_idesc(2, 1, kUM, UN);  // s32 <- s8 x s8
                uint32_t f_top = 0, f_low = 0;
                for (int kt = kt0; ok && kt < kt1; ++kt) {
                    int prev_s = -1;
                    for (int i = top; ok && i >= 0; --i, ++it) {
                        const int s = it % ST;
                        if (!mbar_wait(&bar->full[s], (it / ST) & 1, err, 0x303)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t sb = smem_u32(smem + s * Cfg::STAGE);
                        const uint32_t sa = sb + Cfg::BTILE;
                        const bool low = pair && prev_s >= 0;  // A_i x B_{d0-i}: the previous stage's B
                        const uint32_t pb = low ? smem_u32(smem + prev_s * Cfg::STAGE) : 0u;
#pragma unroll
                        for (int kk = 0; kk < KSTEPS; ++kk) {
                            const uint64_t ad = sw128_kmajor_desc(sa) + 2 * kk;
                            umma_i8(acc_top, ad, sw128_kmajor_desc(sb) + 2 * kk, idesc, f_top);
                            f_top = 1;
                            if (low) {
                                umma_i8(acc, ad, sw128_kmajor_desc(pb) + 2 * kk, idesc, f_low);
                                f_low = 1;
                            }
                        }
                        // the previous stage is consumed once these MMAs complete;
                        // without a pair the stage itself is
                        if (pair) {
                            if (prev_s >= 0) tc_commit(&bar->empty[prev_s]);
                            prev_s = s;
                        } else {
                            tc_commit(&bar->empty[s]);
                        }
                    }
                    if (pair && prev_s >= 0) tc_commit(&bar->empty[prev_s]);
                }
                if (ok) tc_commit(&bar->acc_full[bsel]);
            }
        }
        tc_commit(&bar->drain);
        mbar_wait_drain(&bar->drain, 0);
    } else if (warp >= 2) {
        // ------------------------------ epilogue ------------------------------
        const int quarter = warp & 3;      // TMEM lanes 32*quarter.. (the warp's rank in its warpgroup)
        const int cq = (warp - 2) >> 2;    // columns CW*cq .. CW*cq+CW-1 of the tile
        const int row_in_tile = quarter * 32 + lane;
        // this warp's column table: 2^fc where fc is in [-1022, 1023], else 0
        // (a zero or absent column, or an exponent outside the normal range),
        // and fc itself
        uint8_t* tab = smem + ST * Cfg::STAGE + 256 + (warp - 2) * kOzColTab;
        double* col_scale = reinterpret_cast<double*>(tab);
        int* col_e = reinterpret_cast<int*>(tab + 64 * sizeof(double));
        const uint32_t lanebase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
        // C between the units of a tile stays in L2 (the tiles in flight hold
        // ~38 MB of it) while the digit planes stream past; C0's read and the
        // last unit's write are the tile's final touches
        uint32_t uc = 0;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const OzWork w = src.get(item);
            const OzParams& p = *w.p;
            const int upc = (p.slices + 1) / 2;
            const int units = p.kchunks * upc;
            const bool split = w.tt >= 0;
            int tm, tn;
            raster_tile<kOzRaster>(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * kUM, n0 = tn * UN;
            const int r = m0 + row_in_tile;
            const bool row_ok = r < p.m;
            const int er = row_ok ? p.row_exp[r] : kExpSentinel;
            __syncwarp();  // the previous item's reads of the table are done
            // bit j of colmask: column j of the warp's CW has a nonzero table
            // scale (so it also lies inside C)
            uint64_t colmask = 0;
#pragma unroll
            for (int h = 0; h < CW / 32; ++h) {
                const int j = lane + 32 * h;
                const int col = n0 + cq * CW + j;
                const int fc = col < p.n ? __ldg(p.col_exp + col) : kExpSentinel;
                const bool normal = fc != kExpSentinel && fc >= -1022 && fc <= 1023;
                col_e[j] = fc;
                col_scale[j] = normal ? pow2_normal(fc) : 0.0;
                colmask |= static_cast<uint64_t>(__ballot_sync(0xffffffffu, normal)) << (32 * h);
            }
            __syncwarp();
            double* const crow = p.c + (row_ok ? r : 0);
            const double* const c0row = p.cin + (row_ok ? r : 0);
            const size_t ldc = p.ldc;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u, ++uc) {
                int d0, d1;
                oz_unit(p.slices, u % upc, d0, d1);
                const bool first_unit = (u == 0);
                const uint64_t pol_ld = first_unit ? l2_evict_first_policy() : l2_evict_last_policy();
                const uint64_t pol_st = (u == units - 1) ? l2_evict_first_policy() : l2_evict_last_policy();
                // the first unit reads C0 (beta * C0), the later ones the running sum in C
                const double* const srow = first_unit ? c0row : crow;
                // digits of both operands are scaled by 2^-(e+1): weight 2^-(14+8d) per diagonal
                const int wexp = 14 + 8 * (d1 >= 0 ? d1 : d0) - 2;
                // the row's part of the scale first: sv * 2^(er - wexp) is exact
                // (a nonzero integer below 2^40 times a power of two, landing in
                // [2^-1022, 2^1000)), so the second multiply, by 2^fc, is the only
                // rounding -- the same single rounding as scale_pow2(sv, er+fc-wexp)
                const int ra = er - wexp;
                const bool row_fast = er != kExpSentinel && ra >= -1022 && ra <= 960;
                const double rs = row_fast ? pow2_normal(ra) : 0.0;
                // C is read (beta*C0 on the first unit, the running sum after)
                // (a split item: the unit's terms go to its workspace plane, C is untouched)
                const bool read_c = !split && (!first_unit || p.beta_mode != 0);
                const bool live = row_ok && (split || !(er == kExpSentinel && !first_unit));
                // every live row of the warp takes the two-multiply scaling
                const bool warp_fast = __all_sync(0xffffffffu, row_fast || !live);
                double* wplane =
                    split ? p.ws + (static_cast<size_t>(w.tt) * units + u) * TILE_ELEMS + row_in_tile : nullptr;
                // chunk ch's C values are requested one chunk ahead (the first
                // chunk's before the accumulator wait), so a chunk's L2 round
                // trip overlaps the previous chunk's arithmetic
                double cv[8];
#pragma unroll
                for (int jj = 0; jj < 8; ++jj) {
                    const int cbase = n0 + cq * CW;
                    cv[jj] = (live && read_c && cbase + jj < p.n)
                                 ? ld_l2hint(srow + static_cast<size_t>(cbase + jj) * ldc, pol_ld) : 0.0;
                }
                const int bsel = static_cast<int>(uc % Cfg::NBUF);
                const uint32_t accbase = lanebase + bsel * (2 * UN);
                {
                    const bool got = mbar_wait(&bar->acc_full[bsel], (uc / Cfg::NBUF) & 1, err, 0x304);
                    if (!__all_sync(0xffffffffu, got)) {  // the whole warp goes on, or the whole warp stops
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                }
#pragma unroll 1
                for (int ch = 0; ch < NCH; ++ch) {
                    // 8 columns at a time
                    const int j0 = ch * 8;
                    const int col0 = cq * CW + j0;
                    const int cbase = n0 + col0;
                    double* const cp = crow + static_cast<size_t>(cbase) * ldc;
                    const double* const sp = srow + static_cast<size_t>(cbase) * ldc;
                    double cn[8];
#pragma unroll
                    for (int jj = 0; jj < 8; ++jj)
                        cn[jj] = (live && read_c && ch < NCH - 1 && cbase + 8 + jj < p.n)
                                     ? ld_l2hint(sp + static_cast<size_t>(8 + jj) * ldc, pol_ld) : 0.0;
                    uint32_t v0[8], v1[8];
                    tmem_ld8(accbase + col0, v0);
                    if (d1 >= 0) tmem_ld8(accbase + UN + col0, v1);
                    tmem_ld_wait();
                    if (live) {
                        if (warp_fast && ((colmask >> j0) & 0xffu) == 0xffu) {
                            // branch-free: eight independent chains the compiler can interleave
#pragma unroll
                            for (int jj = 0; jj < 8; ++jj) {
                                double sv = static_cast<double>(static_cast<int32_t>(v0[jj]));
                                if (d1 >= 0) sv = fma(sv, 256.0, static_cast<double>(static_cast<int32_t>(v1[jj])));
                                const double term = (sv * rs) * col_scale[j0 + jj];
                                if (wplane) {
                                    wplane[static_cast<size_t>(col0 + jj) * kUM] = term;
                                } else {
                                    double acc = cv[jj];
                                    if (first_unit && p.beta_mode == 2) acc = p.beta * acc;
                                    st_l2hint(cp + static_cast<size_t>(jj) * ldc, fma(p.alpha, term, acc), pol_st);
                                }
                            }
                        } else {
#pragma unroll
                            for (int jj = 0; jj < 8; ++jj) {
                                if (cbase + jj < p.n) {
                                    double sv = static_cast<double>(static_cast<int32_t>(v0[jj]));
                                    if (d1 >= 0)
                                        sv = fma(sv, 256.0, static_cast<double>(static_cast<int32_t>(v1[jj])));
                                    const double cs = col_scale[j0 + jj];
                                    double term;
                                    if (row_fast && cs != 0.0) {
                                        term = (sv * rs) * cs;
                                    } else {
                                        const int fc = col_e[j0 + jj];
                                        term = (er != kExpSentinel && fc != kExpSentinel)
                                                   ? scale_pow2(sv, er + fc - wexp) : 0.0;
                                    }
                                    if (wplane) {
                                        wplane[static_cast<size_t>(col0 + jj) * kUM] = term;
                                    } else {
                                        double acc = cv[jj];
                                        if (first_unit && p.beta_mode == 2) acc = p.beta * acc;
                                        st_l2hint(cp + static_cast<size_t>(jj) * ldc, fma(p.alpha, term, acc),
                                                  pol_st);
                                    }
                                }
                            }
                        }
                    }
#pragma unroll
                    for (int jj = 0; jj < 8; ++jj) cv[jj] = cn[jj];
                }
                if (!ok) break;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar->acc_empty[bsel]);
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

template <int UN>
__global__ void __launch_bounds__(kOzThreads, 1)
    ozaki_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ OzParams p) {
    ozaki_body<UN>(OzSingleSrc{&p, &tmA, &tmB});
}

// Many f64 problems in one persistent launch (the serving loop's Ozaki
// batches): the same tiles and epilogue as ozaki_gemm_kernel, whole tiles only.
template <int UN>
__global__ void __launch_bounds__(kOzThreads, 1)
    ozaki_grouped_kernel(const OzGroupEntry* __restrict__ tab, const int* __restrict__ starts, int nprob,
                         uint32_t* err) {
    ozaki_body<UN>(OzGroupSrc{tab, starts, nprob, err});
}

// ------------------------------------------------------------------------------
// Ozaki GEMM on CTA pairs: 256 x 128 tiles, four diagonals at a time.
//
// ozaki_body's tensor cores wait while a unit of two diagonals drains through
// C: 512 KiB per SM and unit through L2, on all SMs at once (11 us, 19 % of a
// CTA's time at K = 2048), and its operands take 52 bytes per SM and clock of
// MMA from L2. Here a unit is four diagonals {4g .. 4g+3}, whose accumulators
// (4 x 128 columns) fill TMEM, so a tile has half as many units; each
// epilogue thread keeps its outputs of the tile in FP64 registers from the
// first unit (beta * C0, loaded while the tensor cores run) to the last, so C
// is read and written once and a drain touches TMEM only. Stage st of a K
// tile brings A_{top-st} and B_st; A_{top-st} is multiplied by the B tiles of
// this stage and of up to three before it (diagonal top - lag), 31 operand
// bytes per SM and clock.
// The epilogue folds the pairs of diagonals exactly as ozaki_body does, in the
// same order, so the results are its bits: term = (S_d0 * 256 + S_d1) *
// 2^(e + f - w), acc = fma(alpha, term, acc). Where row and column exponents
// and alpha are moderate, alpha * 2^(e + f - w) is exact and one fma(sv,
// alpha * 2^(..), acc) has the same rounding.
// Tail: the tiles of the partial last wave run as items of one group over a
// part of K each, which write the exact sums S_d0 * 256 + S_d1 to workspace
// planes; ozaki_pair_reduce_kernel adds the parts (exactly) and folds.
// Warps per CTA: 0 TMA producer (both CTAs' loads of a stage complete on the even
// CTA's barrier), 1 TMEM owner and, in the even CTA, MMA issuer, 2.. epilogue
// (two or four per TMEM lane quarter).
// ------------------------------------------------------------------------------
constexpr int kPzN = 128;
// Epilogue warps EW: 8 (64 columns each) for one problem, 16 (32 columns) in
// the grouped kernel. At large sizes the power cap holds both, and 8 warps run
// fewer instructions (8192^3: 12.1 against 12.5 ms); the grouped sets end in few
// tiles, whose drains' latency 16 warps halve (eleven f64 requests of 32 .. 4096
// a side: 1587 -> 1421 us; seven: 875 -> 865).
constexpr int kPzEpiWarps = 8, kPzGroupEpiWarps = 16;
constexpr int pz_threads(int ew) { return 64 + 32 * ew; }
// Ring depths: a B tile is used for up to three stages after its own, so with
// three more B slots than A slots both rings' next slots are free once the
// stage kPzAS back is done, and one barrier per stage serves both.
constexpr int kPzAS = 8, kPzBS = kPzAS + 3;
constexpr int kPzBTile = 64 * kRowBytes;           // this CTA's half of a B tile
constexpr int kPzTabs = 4 * kPzN * 2 * 4;          // the epilogue warps' tables: fc << 20 and fc of their columns
constexpr int kPzTileElems = 256 * kPzN;
constexpr int kPzSmem = kPzAS * kATile + kPzBS * kPzBTile + 512 + kPzTabs + 1024;
static_assert(kPzSmem <= 232448, "the pair kernel's rings must fit one CTA's shared memory");

struct PzBar {
    uint64_t full[kPzAS];  // even CTA: a stage of both CTAs has landed
    uint64_t done[kPzAS];  // its MMAs are complete
    uint64_t acc_full, acc_empty, drain;
    uint32_t tmem_base;
    PairExit exit;
};
static_assert(sizeof(PzBar) <= 512, "shared memory reserved for the pair kernel's barriers");

// Diagonals 4g .. 4g + nd - 1 of group g.
__host__ __device__ __forceinline__ int pz_nd(int slices, int g) { return slices - 4 * g < 4 ? slices - 4 * g : 4; }

// A work item: units [u_lo, u_hi) of tile t over K tiles kt0.. of each chunk
// (unit u: group groups-1 - u % groups of chunk u / groups), or, in the tail
// (tt >= 0), one group over K tiles [kt0, kt1) into workspace planes from
// `plane` on.
struct PzWork {
    const OzParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    int t, u_lo, u_hi, tt, kt0, kt1, plane;
};

__host__ __device__ __forceinline__ int pz_items(const OzParams& p) {
    const int groups = (p.slices + 3) / 4;
    int per_tile = 0;
    for (int g = 0; g < kOzGroups; ++g) per_tile += g < groups ? p.parts[g] : 0;
    return p.num_tiles - p.tail_tiles + p.tail_tiles * per_tile;
}

// Tail items are ranked by cost and dealt to the G pairs in a snake, as in oz_item.
__host__ __device__ __forceinline__ void pz_item(const OzParams& p, int G, int item, PzWork& w) {
    const int groups = (p.slices + 3) / 4, fused = p.num_tiles - p.tail_tiles;
    w.tt = -1;
    w.plane = 0;
    w.kt0 = 0;
    w.kt1 = p.num_kt;
    if (item < fused) {
        w.t = item;
        w.u_lo = 0;
        w.u_hi = p.kchunks * groups;
        return;
    }
    const int j = item - fused, total = pz_items(p) - fused;
    const int pass = j / G, q = j - pass * G;
    const int len = (total - pass * G < G) ? total - pass * G : G;
    int rank = (pass & 1) ? pass * G + (len - 1 - q) : j;
    for (int i = 0; i < groups; ++i) {
        const int g = p.order[i], n = p.tail_tiles * p.parts[g];
        if (rank < n) {
            const int part = rank / p.tail_tiles;
            w.tt = rank - part * p.tail_tiles;
            w.t = fused + w.tt;
            w.u_lo = groups - 1 - g;
            w.u_hi = w.u_lo + 1;
            w.kt0 = static_cast<int>(static_cast<long long>(p.num_kt) * part / p.parts[g]);
            w.kt1 = static_cast<int>(static_cast<long long>(p.num_kt) * (part + 1) / p.parts[g]);
            w.plane = p.plane0[g] + part * ((pz_nd(p.slices, g) + 1) / 2);
            return;
        }
        rank -= n;
    }
}

struct PzSingleSrc {
    const OzParams* p;
    const CUtensorMap* ta;
    const CUtensorMap* tb;
    __device__ __forceinline__ uint32_t* err() const { return p->err; }
    __device__ __forceinline__ int items() const { return pz_items(*p); }
    __device__ __forceinline__ PzWork get(int item) const {
        PzWork w{p, ta, tb, 0, 0, 0, -1, 0, 0, 0};
        pz_item(*p, gridDim.x >> 1, item, w);
        return w;
    }
};

// Whole tiles of many problems, as OzGroupSrc.
struct PzGroupSrc {
    OzGroupSrc s;
    __device__ __forceinline__ uint32_t* err() const { return s.err(); }
    __device__ __forceinline__ int items() const { return s.items(); }
    __device__ __forceinline__ PzWork get(int item) const {
        const OzWork o = s.get(item);
        return PzWork{o.p, o.ta, o.tb, o.t, 0, o.p->kchunks * ((o.p->slices + 3) / 4), -1, 0, o.p->num_kt, 0};
    }
};

// K tiles of unit u of an item.
__device__ __forceinline__ void pz_kt(const PzWork& w, int u, int groups, int& kt0, int& kt1) {
    if (w.tt >= 0) {
        kt0 = w.kt0;
        kt1 = w.kt1;
    } else {
        kt0 = (u / groups) * w.p->kt_per_chunk;
        kt1 = min(w.p->num_kt, kt0 + w.p->kt_per_chunk);
    }
}

// sv * 2^(er + fc - wexp) for any exponents (0 for a zero row or column).
__device__ __noinline__ double pz_term(double sv, int er, int fc, int wexp) {
    return (er != kExpSentinel && fc != kExpSentinel) ? scale_pow2(sv, er + fc - wexp) : 0.0;
}

template <int EW, class Src>
__device__ __forceinline__ void ozaki_pair_body(const Src& src) {
    constexpr int COLS = kPzN / (EW / 4);  // columns per epilogue warp
    static_assert(COLS % 32 == 0, "a warp fills its table 32 columns at a time");
    constexpr int AS = kPzAS, BS = kPzBS;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* bring = smem + AS * kATile;
    PzBar* bar = reinterpret_cast<PzBar*>(bring + BS * kPzBTile);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    if (threadIdx.x == 0) {
        for (int i = 0; i < AS; ++i) {
            mbar_init(&bar->full[i], 2);
            mbar_init(&bar->done[i], 1);
        }
        mbar_init(&bar->acc_full, 1);
        mbar_init(&bar->acc_empty, 2 * EW);
        mbar_init(&bar->drain, 1);
        bar->exit = PairExit{};
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc_pair(&bar->tmem_base, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers are initialised too
    tc_fence_after();
    const uint32_t tmem_base = bar->tmem_base;
    const int items = src.items(), first = blockIdx.x >> 1, step = gridDim.x >> 1;
    uint32_t* const err = src.err();
    bool ok = true;

    if (warp == 0 && lane == 0) {
        // ------------------------------ TMA producer ------------------------------
        uint32_t it = 0;
        const CUtensorMap* fetched = nullptr;
        for (int item = first; ok && item < items; item += step) {
            const PzWork w = src.get(item);
            const OzParams& p = *w.p;
            if (w.ta != fetched) {
                prefetch_tmap(w.ta);
                prefetch_tmap(w.tb);
                fetched = w.ta;
            }
            const int groups = (p.slices + 3) / 4;
            int tm, tn;
            raster_tile<kOzRaster / 2>(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int m0 = tm * 256 + rank * 128, n0 = tn * kPzN + rank * 64;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u) {
                const int g = groups - 1 - u % groups, top = 4 * g + pz_nd(p.slices, g) - 1;
                int kt0, kt1;
                pz_kt(w, u, groups, kt0, kt1);
                for (int kt = kt0; ok && kt < kt1; ++kt)
                    for (int st = 0; st <= top; ++st, ++it) {
                        const uint32_t as = it % AS, bs = it % BS;
                        if (it >= AS && !mbar_wait_cluster(&bar->done[as], ((it / AS) - 1) & 1, err, 0x311)) {
                            ok = false;
                            break;
                        }
                        const uint32_t full = cluster_addr(&bar->full[as], 0);
                        mbar_arrive_expect_tx_cluster(full, kATile + kPzBTile);
                        tma_load_3d_pair(smem + as * kATile, w.ta, full, kt * 128, m0, top - st);
                        tma_load_3d_pair(bring + bs * kPzBTile, w.tb, full, kt * 128, n0, st);
                    }
            }
        }
        st_cluster(&bar->exit.issued[0][rank], 0, it);
    } else if (warp == 1 && rank == 0) {
        // ------------------------- even CTA: MMA issuer -------------------------
        // (the whole warp runs the loop, one lane issues: see elect_one)
        const bool lead = elect_one();
        const uint64_t d0 = sw128_kmajor_desc(smem_u32(smem));  // (see umma_pair_kernel on descriptors)
        const uint32_t a_lo = static_cast<uint32_t>(d0), b_lo = a_lo + AS * kATile / 16;
        const uint64_t d_hi = d0 & 0xffffffff00000000ull;
        constexpr uint32_t idesc = umma_idesc(2, 1, 256, kPzN);  // s32 <- s8 x s8
        uint32_t uc = 0, as = 0, ph = 0, bs = 0;  // ring slots, A's phase
        // one stage's MMAs: A (descriptor low word a) with the B tiles of NL
        // lags (b), lag l into accumulator nd-1-l; `fresh`: the last lag's
        // accumulator starts. Straight-line per NL: an MMA takes 64 clocks,
        // and a test around each of them took the issuing thread longer.
        auto stage = [&](auto nl, uint32_t a, const uint32_t (&b)[4], uint32_t d, bool fresh) {
            constexpr int NL = decltype(nl)::value;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int l = 0; l < NL; ++l)
                    umma_i8_pair(d - l * kPzN, d_hi | (a + 2 * kk), d_hi | (b[l] + 2 * kk), idesc,
                                 (kk == 0 && l == NL - 1) ? (fresh ? 0u : 1u) : 1u);
        };
        for (int item = first; ok && item < items; item += step) {
            const PzWork w = src.get(item);
            const int slices = w.p->slices, groups = (slices + 3) / 4;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u, ++uc) {
                const int g = groups - 1 - u % groups, nd = pz_nd(slices, g), top = 4 * g + nd - 1;
                int kt0, kt1;
                pz_kt(w, u, groups, kt0, kt1);
                const uint32_t d = tmem_base + (nd - 1) * kPzN;
                if (uc >= 1 &&
                    !__all_sync(0xffffffffu, mbar_wait_cluster(&bar->acc_empty, (uc - 1) & 1, err, 0x313))) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                for (int kt = kt0; ok && kt < kt1; ++kt)
                    for (int st = 0; st <= top; ++st) {
                        if (!__all_sync(0xffffffffu, mbar_wait_cluster(&bar->full[as], ph, err, 0x314))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t a = a_lo + as * (kATile / 16);
                        uint32_t b[4];
#pragma unroll
                        for (int l = 0; l < 4; ++l)
                            b[l] = b_lo + (bs >= (uint32_t)l ? bs - l : bs + BS - l) * (kPzBTile / 16);
                        const int nl = min(st + 1, nd);
                        const bool fresh = kt == kt0 && st == nl - 1;
                        if (lead) {
                            if (nl == 4)      stage(std::integral_constant<int, 4>{}, a, b, d, fresh);
                            else if (nl == 3) stage(std::integral_constant<int, 3>{}, a, b, d, fresh);
                            else if (nl == 2) stage(std::integral_constant<int, 2>{}, a, b, d, fresh);
                            else              stage(std::integral_constant<int, 1>{}, a, b, d, fresh);
                            tc_commit_pair(&bar->done[as]);
                        }
                        if (++as == AS) {
                            as = 0;
                            ph ^= 1;
                        }
                        if (++bs == BS) bs = 0;
                    }
                if (ok && lead) tc_commit_pair(&bar->acc_full);
            }
        }
        if (lead) {  // nothing of ours is in flight before TMEM is released
            tc_commit_pair(&bar->drain);
            mbar_wait_drain(&bar->drain, 0);
        }
    } else if (warp >= 2) {
        // ------------------------------ epilogue ------------------------------
        const int quarter = warp & 3, part = (warp - 2) >> 2;
        const int row_in_pair = static_cast<int>(rank) * 128 + quarter * 32 + lane;
        uint8_t* tab = reinterpret_cast<uint8_t*>(bar) + 512 + (warp - 2) * (kPzTabs / EW);
        int* col_hi = reinterpret_cast<int*>(tab);  // what 2^fc adds to a double's high word
        int* col_e = col_hi + COLS;
        const uint32_t tbase = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * COLS;
        uint32_t uc = 0;
        for (int item = first; ok && item < items; item += step) {
            const PzWork w = src.get(item);
            const OzParams& p = *w.p;
            const int groups = (p.slices + 3) / 4;
            int tm, tn;
            raster_tile<kOzRaster / 2>(w.t, p.tiles_m, p.tiles_n, tm, tn);
            const int r = tm * 256 + row_in_pair, cb = tn * kPzN + part * COLS;
            const bool row_ok = r < p.m, tail = w.tt >= 0;
            const int er = row_ok ? p.row_exp[r] : kExpSentinel;
            // moderate exponents: alpha * 2^(er - w) * 2^fc and every product
            // with it stay in the normal range
            const int ea = static_cast<int>((static_cast<unsigned long long>(__double_as_longlong(p.alpha)) >> 52) & 0x7FF);
            const bool alpha_fast = ea >= 1023 - 200 && ea <= 1023 + 200;
            const bool row_fast = er >= -200 && er <= 200 && alpha_fast;
            __syncwarp();  // the previous item's reads of the table are done
            bool cols_fast = true;
#pragma unroll
            for (int h = 0; h < COLS / 32; ++h) {
                const int j = lane + 32 * h, col = cb + j;
                const int fc = col < p.n ? __ldg(p.col_exp + col) : kExpSentinel;
                const bool mod = fc >= -200 && fc <= 200;
                col_e[j] = fc;
                col_hi[j] = mod ? fc * (1 << 20) : 0;
                cols_fast = cols_fast && (mod || col >= p.n);  // a column outside C: never stored
            }
            __syncwarp();
            // the whole warp takes the one-fma form, or none of it
            const bool fast = __all_sync(0xffffffffu, cols_fast && (row_fast || !row_ok));
            double acc[COLS];
            if (!tail) {
                const double* c0 = p.cin + (row_ok ? r : 0) + static_cast<size_t>(cb) * p.ldc;
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    acc[j] = (row_ok && p.beta_mode != 0 && cb + j < p.n) ? c0[static_cast<size_t>(j) * p.ldc] : 0.0;
                if (p.beta_mode == 2) {
#pragma unroll
                    for (int j = 0; j < COLS; ++j) acc[j] = p.beta * acc[j];
                }
            }
            bool first_pair = true;
            for (int u = w.u_lo; ok && u < w.u_hi; ++u, ++uc) {
                const int g = groups - 1 - u % groups, nd = pz_nd(p.slices, g), npair = (nd + 1) / 2;
                const bool got = mbar_wait_cluster(&bar->acc_full, uc & 1, err, 0x317);
                if (!__all_sync(0xffffffffu, got)) {  // the whole warp goes on, or the whole warp stops
                    ok = false;
                    break;
                }
                tc_fence_after();
#pragma unroll 1
                for (int pi = 0; pi < npair; ++pi) {
                    const int j0 = 2 * (npair - 1 - pi);  // diagonals 4g + j0 and, in a pair, 4g + j0 + 1
                    const bool pair = j0 + 1 < nd;
                    const int wexp = 14 + 8 * (4 * g + j0 + (pair ? 1 : 0)) - 2;
                    const int mul = pair ? 256 : 0;
                    const double ars = fast && row_ok ? p.alpha * pow2_normal(er - wexp) : 0.0;
                    double* wplane = tail ? p.ws + (static_cast<size_t>(w.tt) * p.planes + w.plane + pi) * kPzTileElems +
                                                row_in_pair + static_cast<size_t>(part * COLS) * 256
                                          : nullptr;
                    const bool live = row_ok && (first_pair || er != kExpSentinel);
                    // chunks of 4 columns, each requested before the one ahead
                    // of it is used (4-column ones: 64 outputs in FP64 leave
                    // registers for two chunks of 2 x 4)
                    constexpr int CH = 4, NCH = COLS / CH;
                    uint32_t v0[2][CH], v1[2][CH];
                    auto request = [&](int ch) {
                        tmem_ld4(tbase + j0 * kPzN + ch * CH, v0[ch & 1]);
                        tmem_ld4(tbase + (pair ? j0 + 1 : j0) * kPzN + ch * CH, v1[ch & 1]);
                    };
                    // T = S_d0 * 256 + S_d1 (below 2^40) as a double: exact, by the
                    // bits of 1.5 * 2^52 + 2^31 + T, where S_d1 + 2^31 is a low
                    // word (alone, S_d0: mul 0 + 1 * v1)
                    auto sum = [&](int ch, int jj) {
                        const long long biased = 0x4338000000000000LL | (v1[ch & 1][jj] ^ 0x80000000u);
                        const long long T = static_cast<long long>(static_cast<int32_t>(v0[ch & 1][jj])) * mul + biased;
                        return __longlong_as_double(T) - 6755401588539392.0;
                    };
                    // ars * 2^fc, in the normal range (fast)
                    auto scale = [&](int j) {
                        return __hiloint2double(__double2hiint(ars) + col_hi[j], __double2loint(ars));
                    };
                    // one loop per case, so that a chunk's chains interleave
                    request(0);
                    if (tail) {
#pragma unroll 2
                        for (int ch = 0; ch < NCH; ++ch) {
                            tmem_ld_wait();
                            if (ch + 1 < NCH) request(ch + 1);
#pragma unroll
                            for (int jj = 0; jj < CH; ++jj)
                                wplane[static_cast<size_t>(ch * CH + jj) * 256] = sum(ch, jj);
                        }
                    } else if (fast) {
#pragma unroll
                        for (int ch = 0; ch < NCH; ++ch) {
                            tmem_ld_wait();
                            if (ch + 1 < NCH) request(ch + 1);
#pragma unroll
                            for (int jj = 0; jj < CH; ++jj)
                                acc[ch * CH + jj] = fma(sum(ch, jj), scale(ch * CH + jj), acc[ch * CH + jj]);
                        }
                    } else {
#pragma unroll
                        for (int ch = 0; ch < NCH; ++ch) {
                            tmem_ld_wait();
                            if (ch + 1 < NCH) request(ch + 1);
                            if (live) {
#pragma unroll
                                for (int jj = 0; jj < CH; ++jj)
                                    acc[ch * CH + jj] = fma(p.alpha, pz_term(sum(ch, jj), er, col_e[ch * CH + jj], wexp),
                                                            acc[ch * CH + jj]);
                            }
                        }
                    }
                    first_pair = false;
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_rank_relaxed(&bar->acc_empty, 0);
            }
            if (ok && row_ok && !tail) {
                double* c = p.c + r + static_cast<size_t>(cb) * p.ldc;
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (cb + j < p.n) c[static_cast<size_t>(j) * p.ldc] = acc[j];
            }
        }
    }

    if (!ok) pair_fail(&bar->exit);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // no CTA leaves while the other may still reach its memory
    if (bar->exit.failed) {  // in both CTAs
        if (rank == 0 && threadIdx.x == 0) pair_drain(bar->full, AS, bar->exit.issued[0]);
        cluster_sync();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pz_threads(kPzEpiWarps), 1)
    ozaki_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ OzParams p) {
    ozaki_pair_body<kPzEpiWarps>(PzSingleSrc{&p, &tmA, &tmB});
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pz_threads(kPzGroupEpiWarps), 1)
    ozaki_pair_grouped_kernel(const OzGroupEntry* __restrict__ tab, const int* __restrict__ starts, int nprob,
                              uint32_t* err) {
    ozaki_pair_body<kPzGroupEpiWarps>(PzGroupSrc{OzGroupSrc{tab, starts, nprob, err}});
}

// The pair kernel's tail: per element, beta * C0, then for each pair of
// diagonals from the highest down the exact sum of its K parts, scaled and
// folded as in the epilogue. Two rows per thread (planes are 256 x 128, rows
// contiguous, so every plane read is 16 bytes).
__global__ void __launch_bounds__(256) ozaki_pair_reduce_kernel(const OzParams p) {
    const int fused = p.num_tiles - p.tail_tiles, groups = (p.slices + 3) / 4;
    const size_t total = static_cast<size_t>(p.tail_tiles) * (kPzTileElems / 2);
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int tt = static_cast<int>(idx / (kPzTileElems / 2));
        const int local = 2 * static_cast<int>(idx - static_cast<size_t>(tt) * (kPzTileElems / 2));
        int tm, tn;
        raster_tile<kOzRaster / 2>(fused + tt, p.tiles_m, p.tiles_n, tm, tn);
        const int r = tm * 256 + local % 256, col = tn * kPzN + local / 256;
        if (r >= p.m || col >= p.n) continue;
        const bool two = r + 1 < p.m;
        double* cp = p.c + r + static_cast<size_t>(col) * p.ldc;
        const double* c0 = p.cin + r + static_cast<size_t>(col) * p.ldc;
        double acc[2] = {p.beta_mode ? c0[0] : 0.0, p.beta_mode && two ? c0[1] : 0.0};
        if (p.beta_mode == 2) {
            acc[0] = p.beta * acc[0];
            acc[1] = p.beta * acc[1];
        }
        const int er[2] = {p.row_exp[r], two ? p.row_exp[r + 1] : kExpSentinel};
        const int fc = p.col_exp[col];
        const double* w = p.ws + static_cast<size_t>(tt) * p.planes * kPzTileElems + local;
        bool first_pair = true;
        for (int g = groups - 1; g >= 0; --g) {
            const int nd = pz_nd(p.slices, g), npair = (nd + 1) / 2;
            for (int pi = 0; pi < npair; ++pi) {
                const int j0 = 2 * (npair - 1 - pi);
                const int wexp = 14 + 8 * (4 * g + j0 + (j0 + 1 < nd ? 1 : 0)) - 2;
                double sv[2] = {0.0, 0.0};
                for (int part = 0; part < p.parts[g]; ++part) {
                    const double2 v = *reinterpret_cast<const double2*>(
                        w + static_cast<size_t>(p.plane0[g] + part * npair + pi) * kPzTileElems);
                    sv[0] += v.x;
                    sv[1] += v.y;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (first_pair || er[h] != kExpSentinel)
                        acc[h] = fma(p.alpha,
                                     (er[h] != kExpSentinel && fc != kExpSentinel) ? scale_pow2(sv[h], er[h] + fc - wexp)
                                                                                   : 0.0,
                                     acc[h]);
                first_pair = false;
            }
        }
        cp[0] = acc[0];
        if (two) cp[1] = acc[1];
    }
}

// Split tail: C of the tail tiles = the fused epilogue's sequence over the
// unit planes, element by element -- acc = beta-pass(C0) for the first unit,
// then acc = fma(alpha, term_u, acc) in unit order; rows with a zero exponent
// take only the first unit's step, as in the fused epilogue. Consecutive
// threads take consecutive rows of a tile column (coalesced C and planes).
__global__ void ozaki_reduce_kernel(const OzParams p, int units) {
    const int fused = p.num_tiles - p.tail_tiles;
    const int tile_elems = kUM * p.un;
    const size_t total = static_cast<size_t>(p.tail_tiles) * tile_elems;
    for (size_t idx = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const int tt = static_cast<int>(idx / tile_elems);
        const int local = static_cast<int>(idx - static_cast<size_t>(tt) * tile_elems);
        int tm, tn;
        raster_tile<kOzRaster>(fused + tt, p.tiles_m, p.tiles_n, tm, tn);
        const int r = tm * kUM + local % kUM, col = tn * p.un + local / kUM;
        if (r >= p.m || col >= p.n) continue;
        double* cp = p.c + r + static_cast<size_t>(col) * p.ldc;
        const double c0 = p.beta_mode ? p.cin[r + static_cast<size_t>(col) * p.ldc] : 0.0;
        double acc = 0.0;
        if (p.beta_mode == 1) acc = c0;
        else if (p.beta_mode == 2) acc = p.beta * c0;
        const double* w = p.ws + static_cast<size_t>(tt) * units * tile_elems + local;
        const int last = (p.row_exp[r] == kExpSentinel) ? 1 : units;
        for (int u = 0; u < last; ++u) acc = fma(p.alpha, w[static_cast<size_t>(u) * tile_elems], acc);
        *cp = acc;
    }
}

// ------------------------------------------------------------------------------
// Pre-pass kernels. An operand is viewed as R x K with element (r, p) at
// x[r*rs + p*ps]; outputs are K-major planes [plane][R][kp] (kp = padded K).
// ------------------------------------------------------------------------------

__device__ __forceinline__ int frexp_exp(double x) {
    // exponent e with |x| in [2^(e-1), 2^e); x != 0
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x));
    const int f = static_cast<int>((bits >> 52) & 0x7FF);
    if (f != 0) return f - 1022;
    int e;
    frexp(x, &e);
    return e;
}

__global__ void fill_int_kernel(int* p, int n, int v) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// e[r] = max over p of frexp_exp(x(r,p)) (kExpSentinel if the row is zero);
// atomicMax merges the K slabs. frexp_exp is non-decreasing in |x|, and the
// bit patterns of non-negative doubles (subnormals, inf and NaN included)
// order as their values, so the row's exponent is frexp_exp of the largest
// |x| bit pattern: one mask and one 64-bit max per element (0 for a zero row).
__device__ __forceinline__ long long abs_bits(double v) {
    return __double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFLL;
}
// K-contiguous view: one warp per row (8 rows per 256-thread block), a
// 1024-wide K slab per block row by.
__device__ __forceinline__ void row_exp_kcontig(const double* __restrict__ x, size_t rs, int R, int K,
                                                int* __restrict__ e, int bx, int by) {
    const int r = bx * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (r >= R) return;
    const int p0 = by * 1024, p1 = min(K, p0 + 1024);
    long long best = 0;
#pragma unroll 8
    for (int q = p0 + (threadIdx.x & 31); q < p1; q += 32) best = max(best, abs_bits(x[static_cast<size_t>(r) * rs + q]));
    for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best != 0) atomicMax(e + r, frexp_exp(__longlong_as_double(best)));
}
// R-contiguous view: one thread per row (coalesced across the warp), a
// 32-wide K slab per block row by so the grid covers the whole matrix.
__device__ __forceinline__ void row_exp_rcontig(const double* __restrict__ x, size_t ps, int R, int K,
                                                int* __restrict__ e, int bx, int by) {
    const int r = bx * blockDim.x + threadIdx.x;
    if (r >= R) return;
    const int p0 = by * 32, p1 = min(K, p0 + 32);
    long long best = 0;
#pragma unroll 8
    for (int q = p0; q < p1; ++q) best = max(best, abs_bits(x[r + static_cast<size_t>(q) * ps]));
    if (best != 0) atomicMax(e + r, frexp_exp(__longlong_as_double(best)));
}
// The same for the real form of a complex operand (cx: see load_tile_complex), whose
// rows 2 i and 2 i + 1 hold row i's parts and their negatives: R and K are the
// complex sizes here.
__device__ __forceinline__ void row_exp_complex(const double* __restrict__ x, size_t ld, int cx, int R, int K,
                                                int* __restrict__ e, int bx, int by) {
    long long best = 0;
    int r;
    if (cx == 1) {  // rows contiguous: a thread per row, 32 columns
        r = bx * blockDim.x + threadIdx.x;
        if (r >= R) return;
        const int p0 = by * 32, p1 = min(K, p0 + 32);
#pragma unroll 8
        for (int q = p0; q < p1; ++q) {
            const double* v = x + 2 * (r + static_cast<size_t>(q) * ld);
            best = max(best, max(abs_bits(v[0]), abs_bits(v[1])));
        }
    } else {  // K contiguous: a warp per row, 1024 columns
        r = bx * (blockDim.x / 32) + (threadIdx.x >> 5);
        if (r >= R) return;
        const double* v = x + 2 * static_cast<size_t>(r) * ld;
        const int p1 = 2 * min(K, (by + 1) * 1024);
#pragma unroll 8
        for (int q = by * 2048 + (threadIdx.x & 31); q < p1; q += 32) best = max(best, abs_bits(v[q]));
        for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        if ((threadIdx.x & 31) != 0) return;
    }
    if (best != 0) {
        const int ex = frexp_exp(__longlong_as_double(best));
        atomicMax(e + 2 * r, ex);
        atomicMax(e + 2 * r + 1, ex);
    }
}
constexpr int kTile = 64;

// Load a 64 x 64 tile of the R x K view into shared memory (coalesced along
// the view's contiguous dimension); out-of-range elements read as 0. Blocks
// of 256 threads: each thread issues its 16 loads before the first store, so
// the loads are in flight together instead of one latency each.
constexpr int kTileThreads = 256;
template <typename T>
__device__ __forceinline__ void load_tile(const T* __restrict__ x, size_t rs, size_t ps, int R, int K,
                                          int r0, int p0, T (*tile)[kTile + 1]) {
    constexpr int PER = kTile * kTile / kTileThreads;
    const bool kcontig = (ps == 1);
    T v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % kTile, b = idx / kTile;
        const int r = kcontig ? b : a;
        const int q = kcontig ? a : b;
        v[i] = (r0 + r < R && p0 + q < K) ? x[static_cast<size_t>(r0 + r) * rs + static_cast<size_t>(p0 + q) * ps]
                                          : T(0);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % kTile, b = idx / kTile;
        tile[kcontig ? b : a][kcontig ? a : b] = v[i];
    }
}

// Ozaki slicing. With e[r] the row exponent (|x| < 2^e), y = x * 2^-(e+1)
// lies in (-1/2, 1/2). For s slices let N = 7 + 8(s-1) and
//   Y = floor(y * 2^N) = floor(x * 2^(N-e-1)),
// computed exactly from x's bits (x = m * 2^q with an integer m of at most
// 53 bits: Y = m << (q+N-e-1), or an arithmetic right shift -- a floor --
// when that exponent is negative; |Y| < 2^(N-1) <= 2^94 fits an __int128).
// Its base-256 digits, the top one signed, are
//   d_0 = floor(y * 2^7) in [-64, 63],  d_t = floor(y * 2^(7+8t)) mod 256,
// which are then balanced from the least significant up: d_t >= 128 becomes
// d_t - 256 with a carry of 1 into d_{t-1} (d_0 <= 64 after the carry). The
// result: signed 8-bit digits with y = sum_t d_t 2^-(7+8t) + rem,
// 0 <= rem < 2^-N, and tail digits symmetric about zero, so the dropped cross
// products do not accumulate a bias along K. No floating-point rounding
// occurs anywhere in the extraction (slices: 2 to 12).

// floor(x * 2^n) for |x * 2^n| < 2^94 (Int = __int128) or < 2^62 (long long)
template <typename Int>
__device__ __forceinline__ Int floor_scaled(double x, int n) {
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x));
    const int ex = static_cast<int>((bits >> 52) & 0x7FF);
    long long m = static_cast<long long>(bits & ((1ull << 52) - 1));
    if (ex != 0) m |= (1ll << 52);
    if (m == 0) return 0;
    if (bits >> 63) m = -m;
    const int sh = (ex == 0 ? 1 : ex) - 1075 + n;  // x = m * 2^((ex|1) - 1075)
    if (sh >= 0) return static_cast<Int>(m) << sh;
    if (sh <= -63) return m < 0 ? -1 : 0;
    return static_cast<Int>(m >> (-sh));  // arithmetic shift: floor
}

// S slices known at compile time: up to 8 digits the integer fits 64 bits.
// One 64 x 64 tile of the R x K view per 256-thread block: K tile bx, row
// tile by.
// The slice pass's tile: rows of kSliceLD doubles (1 mod 16), and every
// 16-column group shifted by 4 more, so that the reads below (a half-warp on
// rows r and groups c, tid = 4r + c) and the loads' stores both touch
// distinct banks; with 65-double rows the four groups of a row shared theirs.
constexpr int kSliceLD = 81;
__device__ __forceinline__ int slice_col(int col) { return col + (col >> 4) * 4; }

__device__ __forceinline__ void load_tile_sliced(const double* __restrict__ x, size_t rs, size_t ps, int R, int K,
                                                 int r0, int p0, double (*tile)[kSliceLD]) {
    constexpr int PER = kTile * kTile / kTileThreads;
    const bool kcontig = (ps == 1);
    double v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % kTile, b = idx / kTile;
        const int r = kcontig ? b : a;
        const int q = kcontig ? a : b;
        v[i] = (r0 + r < R && p0 + q < K) ? x[static_cast<size_t>(r0 + r) * rs + static_cast<size_t>(p0 + q) * ps]
                                          : 0.0;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % kTile, b = idx / kTile;
        if (kcontig) tile[b][slice_col(a)] = v[i];
        else         tile[a][slice_col(b)] = v[i];
    }
}

// The tile of the real form [[Re, -Im], [Im, Re]] (by element: rows 2 i, 2 i + 1,
// columns 2 p, 2 p + 1) of op(A), A complex column-major with leading dimension
// ld: cx 1 A, 2 A^T, 3 A^H. r0, p0, R, K in the real form.
__device__ __forceinline__ void load_tile_complex(const double* __restrict__ x, size_t ld, int cx, int R, int K,
                                                  int r0, int p0, double (*tile)[kSliceLD]) {
    constexpr int CT = kTile / 2, PER = CT * CT / kTileThreads;
    double re[PER], im[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % CT, b = idx / CT;  // along the columns of A, across them
        const int r = r0 / 2 + (cx == 1 ? a : b), q = p0 / 2 + (cx == 1 ? b : a);
        const double* v = x + 2 * (cx == 1 ? r + static_cast<size_t>(q) * ld : q + static_cast<size_t>(r) * ld);
        const bool in = r < R / 2 && q < K / 2;
        re[i] = in ? v[0] : 0.0;
        im[i] = in ? v[1] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int a = idx % CT, b = idx / CT;
        const int r = 2 * (cx == 1 ? a : b), q = 2 * (cx == 1 ? b : a);
        const double v = cx == 3 ? 0.0 - im[i] : im[i];
        tile[r][slice_col(q)] = re[i];
        tile[r + 1][slice_col(q)] = v;
        tile[r][slice_col(q + 1)] = 0.0 - v;
        tile[r + 1][slice_col(q + 1)] = re[i];
    }
}

// cx != 0: x is a complex operand with leading dimension rs (load_tile_complex).
template <int S>
__device__ __forceinline__ void ozaki_slice_tile(const double* __restrict__ x, size_t rs, size_t ps, int cx, int R,
                                                 int K, const int* __restrict__ e, int8_t* __restrict__ out,
                                                 size_t kp, size_t plane, int bx, int by) {
    using Int = typename std::conditional<(S <= 8), long long, __int128>::type;
    constexpr int slices = S;
    __shared__ double tile[kTile][kSliceLD];
    const int r0 = by * kTile, p0 = bx * kTile;
    if (cx) load_tile_complex(x, rs, cx, R, K, r0, p0, tile);
    else    load_tile_sliced(x, rs, ps, R, K, r0, p0, tile);
    __syncthreads();
    const int r = threadIdx.x >> 2, c = threadIdx.x & 3;  // 64 rows x 4 chunks of 16
    if (r0 + r >= R) return;
    if (p0 + c * 16 >= static_cast<int>(kp)) return;
    const int er = e[r0 + r];
    const int n = 7 + 8 * (slices - 1) - er - 1;  // Y = floor(x * 2^n)
    uint32_t w[S][4];
    if constexpr (S <= 8) {
        // Balancing by bytes: adding 0x80 to each of the S-1 low bytes of Y
        // makes the carries of the loop below (a byte >= 128 becomes byte-256
        // and carries 1 upward); flipping those bytes back (xor 0x80) leaves
        // each balanced digit as a two's-complement byte, and byte S-1 (the
        // top digit, carry included) is already one. So digit t is byte
        // S-1-t of Z = (Y + B) ^ B, and four elements' digit t pack into one
        // word with byte permutes.
        constexpr unsigned long long B = 0x0080808080808080ull >> (8 * (8 - S));
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const long long Y = (er == kExpSentinel) ? 0LL : floor_scaled<long long>(tile[r][slice_col(c * 16 + g * 4 + q)], n);
                const unsigned long long Z = (static_cast<unsigned long long>(Y) + B) ^ B;
                lo[q] = static_cast<uint32_t>(Z);
                hi[q] = static_cast<uint32_t>(Z >> 32);
            }
#pragma unroll
            for (int t = 0; t < S; ++t) {
                const int b = S - 1 - t;  // byte of Z holding digit t
                const uint32_t* src = b < 4 ? lo : hi;
                const uint32_t sel = static_cast<uint32_t>((b & 3) | (((b & 3) + 4) << 4));
                const uint32_t x01 = __byte_perm(src[0], src[1], sel);
                const uint32_t x23 = __byte_perm(src[2], src[3], sel);
                w[t][g] = __byte_perm(x01, x23, 0x5410);
            }
        }
    } else {
#pragma unroll
    for (int t = 0; t < S; ++t) w[t][0] = w[t][1] = w[t][2] = w[t][3] = 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const Int Y = (er == kExpSentinel) ? Int(0) : floor_scaled<Int>(tile[r][slice_col(c * 16 + i)], n);
        int d[S];
#pragma unroll
        for (int t = 0; t < S; ++t) {
            const int sh = 8 * (S - 1 - t);
            d[t] = (t == 0) ? static_cast<int>(Y >> sh) : static_cast<int>((Y >> sh) & 0xFF);
        }
#pragma unroll
        for (int t = S - 1; t >= 1; --t) {
            if (d[t] >= 128) {
                d[t] -= 256;
                d[t - 1] += 1;
            }
        }
#pragma unroll
        for (int t = 0; t < S; ++t) w[t][i >> 2] |= (static_cast<uint32_t>(d[t]) & 0xFFu) << (8 * (i & 3));
    }
    }
    const size_t off = static_cast<size_t>(r0 + r) * kp + p0 + c * 16;
#pragma unroll
    for (int t = 0; t < S; ++t)
        *reinterpret_cast<uint4*>(out + t * plane + off) = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
}

// ---- pre-pass: one launch per pass over both operands, or every one of a batch ------

// One operand, viewed as R x K (element (r, p) at
// x[r*rs + p*ps]): its exponents e[R] and digit planes out[slices][R][kp].
// exp_blocks / slice_blocks: the blocks it takes in each pass (the grid's
// blocks are dealt to operands by the prefix sums exp_start / slice_start).
struct OzOperand {
    const double* x;
    size_t rs, ps;
    int cx;  // != 0: complex, leading dimension rs (load_tile_complex)
    int R, K;
    int* e;
    int8_t* out;
    size_t kp, plane;
    int exp_gx, slice_gx;  // blocks along R (exponent pass) / along K (slice pass)
    int exp_start, slice_start;
};

__device__ __forceinline__ int oz_find_operand(const OzOperand* ops, int nops, int b, bool slice) {
    int lo = 0, hi = nops - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((slice ? ops[mid].slice_start : ops[mid].exp_start) <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Block b of an operand's exponent pass (e pre-filled with the zero-row
// sentinel), of its slice pass. CX: operands may be complex (a test of o.cx cost
// the grouped passes 4 % of a call).
template <bool CX>
__device__ __forceinline__ void oz_exp_block(const OzOperand& o, int b) {
    const int bx = b % o.exp_gx, by = b / o.exp_gx;
    if (CX && o.cx)     row_exp_complex(o.x, o.rs, o.cx, o.R / 2, o.K / 2, o.e, bx, by);
    else if (o.ps == 1) row_exp_kcontig(o.x, o.rs, o.R, o.K, o.e, bx, by);
    else                row_exp_rcontig(o.x, o.ps, o.R, o.K, o.e, bx, by);
}
template <int S, bool CX>
__device__ __forceinline__ void oz_slice_block(const OzOperand& o, int b) {
    ozaki_slice_tile<S>(o.x, o.rs, o.ps, CX ? o.cx : 0, o.R, o.K, o.e, o.out, o.kp, o.plane, b % o.slice_gx, b / o.slice_gx);
}
// Sets o's blocks along R and K and the first block after those before it
// (exp, slice: blocks so far, advanced).
void oz_operand_blocks(OzOperand* o, int* exp, int* slice) {
    const int R = o->cx ? o->R / 2 : o->R, K = o->cx ? o->K / 2 : o->K;
    const bool kcontig = o->cx ? o->cx != 1 : o->ps == 1;
    o->exp_gx = kcontig ? (R + 7) / 8 : (R + 255) / 256;
    o->exp_start = *exp;
    *exp += o->exp_gx * (kcontig ? (K + 1023) / 1024 : (K + 31) / 32);
    o->slice_gx = static_cast<int>((o->kp + kTile - 1) / kTile);
    o->slice_start = *slice;
    *slice += o->slice_gx * ((o->R + kTile - 1) / kTile);
}

__global__ void __launch_bounds__(256) ozaki_exp_grouped_kernel(const OzOperand* __restrict__ ops, int nops) {
    const OzOperand& o = ops[oz_find_operand(ops, nops, blockIdx.x, false)];
    oz_exp_block<false>(o, blockIdx.x - o.exp_start);
}
template <int S>
__global__ void __launch_bounds__(256) ozaki_slice_grouped_kernel(const OzOperand* __restrict__ ops, int nops) {
    const OzOperand& o = ops[oz_find_operand(ops, nops, blockIdx.x, true)];
    oz_slice_block<S, false>(o, blockIdx.x - o.slice_start);
}

// One problem: its operands as kernel parameters, A's blocks then B's, so the
// two share a launch's tail (five launches before: 1024^3 91 -> 81 us).
struct OzPair {
    OzOperand op[2];
};
__global__ void __launch_bounds__(256) ozaki_exp_kernel(const __grid_constant__ OzPair p) {
    const int b = blockIdx.x, i = b >= p.op[1].exp_start;
    oz_exp_block<true>(p.op[i], b - p.op[i].exp_start);
}
template <int S>
__global__ void __launch_bounds__(256) ozaki_slice_kernel(const __grid_constant__ OzPair p) {
    const int b = blockIdx.x, i = b >= p.op[1].slice_start;
    oz_slice_block<S, true>(p.op[i], b - p.op[i].slice_start);
}

// Exponents (op[0].e, op[1].e adjacent) and digit planes of both operands;
// slices 2 .. 12.
void launch_ozaki_prepass(OzPair p, int slices, cudaStream_t st) {
    int exp = 0, slice = 0;
    for (OzOperand& o : p.op) oz_operand_blocks(&o, &exp, &slice);
    fill_int_kernel<<<64, 256, 0, st>>>(p.op[0].e, p.op[0].R + p.op[1].R, kExpSentinel);
    ozaki_exp_kernel<<<exp, 256, 0, st>>>(p);
    switch (slices) {
#define RB_SLICES(S) \
    case S: ozaki_slice_kernel<S><<<slice, 256, 0, st>>>(p); break;
        RB_SLICES(2) RB_SLICES(3) RB_SLICES(4) RB_SLICES(5) RB_SLICES(6) RB_SLICES(7) RB_SLICES(8)
        RB_SLICES(9) RB_SLICES(10) RB_SLICES(11) RB_SLICES(12)
#undef RB_SLICES
        default: break;
    }
    count_launch(3);
}

// BF16 split into `planes` (2 or 3) planes: out[0] = bf16(x),
// out[1] = bf16(x - out[0]), out[2] = bf16(x - out[0] - out[1]); every
// difference is exact in FP32.
// One 64 x 64 tile of the R x K view per 256-thread block (K tile bx, row tile by).
// The f32 tile loader with 16-byte loads along the view's contiguous
// dimension when its lines start on 16 bytes (4 loads per thread instead of
// 16); the element loader otherwise.
__device__ __forceinline__ void load_tile_f32(const float* __restrict__ x, size_t rs, size_t ps, int R, int K,
                                              int r0, int p0, float (*tile)[kTile + 1]) {
    const bool kcontig = (ps == 1);
    const size_t ld = kcontig ? rs : ps;         // between the contiguous lines
    const int L = kcontig ? R : K, E = kcontig ? K : R;
    const int l0 = kcontig ? r0 : p0, e0 = kcontig ? p0 : r0;
    if ((!kcontig && rs != 1) || (reinterpret_cast<uintptr_t>(x) & 15) != 0 || (ld & 3) != 0) {
        load_tile<float>(x, rs, ps, R, K, r0, p0, tile);
        return;
    }
    constexpr int PER = kTile * kTile / 4 / kTileThreads;  // float4 per thread
    float4 v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int l = l0 + idx / (kTile / 4), e = e0 + 4 * (idx % (kTile / 4));
        const float* src = x + static_cast<size_t>(l) * ld + e;
        if (l < L && e + 3 < E) {
            v[i] = __ldg(reinterpret_cast<const float4*>(src));
        } else {
            v[i].x = (l < L && e < E) ? src[0] : 0.f;
            v[i].y = (l < L && e + 1 < E) ? src[1] : 0.f;
            v[i].z = (l < L && e + 2 < E) ? src[2] : 0.f;
            v[i].w = (l < L && e + 3 < E) ? src[3] : 0.f;
        }
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int idx = threadIdx.x + i * kTileThreads;
        const int ln = idx / (kTile / 4), el = 4 * (idx % (kTile / 4));
        const float w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (kcontig) tile[ln][el + j] = w[j];  // row = line, column = k
            else         tile[el + j][ln] = w[j];  // row = contiguous index, column = line (k)
        }
    }
}

// VEC: the 16-byte loader (the single-problem pass over large operands);
// the grouped pass keeps the element loader, whose kernel stays at five CTAs
// per SM
template <bool VEC>
__device__ __forceinline__ void bf16_split_tile(const float* __restrict__ x, size_t rs, size_t ps, int R, int K,
                                                int planes, __nv_bfloat16* __restrict__ out, size_t kp, size_t plane,
                                                int bx, int by) {
    __shared__ float tile[kTile][kTile + 1];
    const int r0 = by * kTile, p0 = bx * kTile;
    if constexpr (VEC) load_tile_f32(x, rs, ps, R, K, r0, p0, tile);
    else               load_tile<float>(x, rs, ps, R, K, r0, p0, tile);
    __syncthreads();
    for (int job = threadIdx.x; job < kTile * 8; job += blockDim.x) {
        const int r = job >> 3, c = job & 7;  // 64 rows x 8 chunks of 8
        if (r0 + r >= R || p0 + c * 8 >= static_cast<int>(kp)) continue;
        __align__(16) __nv_bfloat16 h[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            // hi, then the rest rounded again (mid / lo); the single-problem
            // pass skips the third plane when the 3xBF16 form does not write
            // it (the grouped pass, branch-free, measured faster without the test)
            float v = tile[r][c * 8 + i];
            h[0][i] = __float2bfloat16_rn(v);
            v = v - __bfloat162float(h[0][i]);
            h[1][i] = __float2bfloat16_rn(v);
            if (!VEC || planes > 2) {
                v = v - __bfloat162float(h[1][i]);
                h[2][i] = __float2bfloat16_rn(v);
            }
        }
        const size_t off = static_cast<size_t>(r0 + r) * kp + p0 + c * 8;
        for (int q = 0; q < planes; ++q)
            *reinterpret_cast<uint4*>(out + q * plane + off) = *reinterpret_cast<const uint4*>(h[q]);
    }
}

__global__ void __launch_bounds__(256) bf16_split_kernel(const float* __restrict__ x, size_t rs, size_t ps,
                                                         int R, int K, int planes,
                                                         __nv_bfloat16* __restrict__ out, size_t kp,
                                                         size_t plane) {
    bf16_split_tile<true>(x, rs, ps, R, K, planes, out, kp, plane, blockIdx.x, blockIdx.y);
}

// One operand of a grouped BF16-split launch, viewed as R x K, and its
// planes out[planes][R][kp]; gx K tiles per row tile, `start` its first block.
struct BsOperand {
    const float* x;
    size_t rs, ps;
    int R, K, planes;
    __nv_bfloat16* out;
    size_t kp, plane;
    int gx, start;
};

// The split pass over every operand of a batch (grid = all their tiles).
__global__ void __launch_bounds__(256) bf16_split_grouped_kernel(const BsOperand* __restrict__ ops, int nops) {
    int lo = 0, hi = nops - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (ops[mid].start <= static_cast<int>(blockIdx.x)) lo = mid;
        else hi = mid - 1;
    }
    const BsOperand& o = ops[lo];
    const int b = blockIdx.x - o.start;
    bf16_split_tile<false>(o.x, o.rs, o.ps, o.R, o.K, o.planes, o.out, o.kp, o.plane, b % o.gx, b / o.gx);
}

CUresult make_tmap_planes(CUtensorMap* map, const void* base, CUtensorMapDataType dtype, size_t elem,
                          uint64_t k, uint64_t rows, uint64_t planes, uint64_t kp, uint32_t box_rows,
                          int row_bytes = kRowBytes) {
    return make_tmap_3d(map, base, dtype, elem, k, rows, planes, kp, kp * rows, row_bytes / elem,
                        box_rows, 1, row_bytes);
}

template <int MODE>
cudaError_t launch_umma(const CUtensorMap& ta, const CUtensorMap& tb, const UParams& p, cudaStream_t st) {
    auto kern = umma_gemm_kernel<MODE>;
    constexpr int smem = umma_smem_bytes<MODE>();
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = p.num_tiles < sms ? p.num_tiles : sms;
    const double work = 2.0 * p.m * p.n * static_cast<double>(p.k) * UCfg<MODE>::NPROD;
    const char* name = (MODE == kModeBf16x3) ? "umma_bf16x3" : "umma_bf16x6";
    KernelTimer tm;
    kernel_timing_begin(name, work, st, &tm);
    kern<<<grid, UCfg<MODE>::THREADS, smem, st>>>(ta, tb, p);
    kernel_timing_end(&tm, st);
    count_launch();
    return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_umma_pair(const CUtensorMap& ta, const CUtensorMap& tb, const UParams& p, int sms, cudaStream_t st) {
    auto kern = umma_pair_kernel<MODE>;
    constexpr int smem = pair_smem_bytes<MODE>();
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int grid = 2 * std::min(p.num_tiles, sms / 2);
    KernelTimer tm;
    kernel_timing_begin((MODE == kModeBf16x3) ? "umma_bf16x3" : "umma_bf16x6",
                        2.0 * p.m * p.n * static_cast<double>(p.k) * UCfg<MODE>::NPROD, st, &tm);
    kern<<<grid, kPairThreads, smem, st>>>(ta, tb, p);
    kernel_timing_end(&tm, st);
    count_launch();
    return cudaGetLastError();
}

inline size_t round_up(size_t x, size_t m) { return (x + m - 1) / m * m; }

// Tensor-pipe throughput probe: one CTA per SM, smem operands filled once
// with a fixed bit pattern, thread 0 issues `iters` back-to-back MMAs
// (M=128, N=256, one 32-byte K step) into a TMEM accumulator.
template <bool I8>
__global__ void __launch_bounds__(128, 1) umma_peak_kernel(int iters, uint32_t* err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* done = reinterpret_cast<uint64_t*>(smem + kATile + 256 * kRowBytes);
    uint32_t* tbase = reinterpret_cast<uint32_t*>(done + 1);
    for (int i = threadIdx.x; i < (kATile + 256 * kRowBytes) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t*>(smem)[i] = 0x3c003c00u ^ (i * 2654435761u & 0x00ff00ffu);
    fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        mbar_init(done, 1);
        fence_barrier_init();
    }
    if ((threadIdx.x >> 5) == 0) {
        tmem_alloc(tbase, 256);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tbase;
    if (threadIdx.x == 0) {
        const uint32_t sa = smem_u32(smem), sb = sa + kATile;
        constexpr uint32_t idesc = I8 ? umma_idesc(2, 1, kUM, 256) : umma_idesc(1, 1, kUM, 256);
        for (int i = 0; i < iters; ++i) {
            const uint64_t a = sw128_kmajor_desc(sa) + 2 * (i & 3), b = sw128_kmajor_desc(sb) + 2 * (i & 3);
            if (I8) umma_i8(tmem, a, b, idesc, i > 0);
            else    umma_f16(tmem, a, b, idesc, i > 0);
        }
        tc_commit(done);
        mbar_wait(done, 0, err, 0x2f0);
    }
    tc_fence_before();
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 256);
    }
}

}  // namespace

double probe_umma_peak(int i8, int iters) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int smem = kATile + 256 * kRowBytes + 64 + 1024;
    auto k0 = umma_peak_kernel<false>;
    auto k1 = umma_peak_kernel<true>;
    auto kern = i8 ? k1 : k0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1.0;
    uint32_t* err = device_error_word();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    kern<<<sms, 128, smem>>>(iters / 8 + 1, err);  // warm-up
    cudaEventRecord(e0);
    kern<<<sms, 128, smem>>>(iters, err);
    cudaEventRecord(e1);
    count_launch(2);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (cudaGetLastError() != cudaSuccess || ms <= 0.f) return -1.0;
    const double per_mma = 2.0 * kUM * 256 * (i8 ? 32 : 16);
    return per_mma * iters * sms / (ms * 1e-3) / 1e12;
}

// op(A) viewed as m x k: (i,p) at A[i + p*lda] (NoTrans) or A[p + i*lda] (Trans).
// op(B)^T viewed as n x k: (j,p) at B[p + j*ldb] (NoTrans) or B[j + p*ldb] (Trans).
static void operand_views(bool ta, bool tb, size_t lda, size_t ldb, size_t& ars, size_t& aps,
                          size_t& brs, size_t& bps) {
    if (!ta) { ars = 1; aps = lda; } else { ars = lda; aps = 1; }
    if (!tb) { brs = ldb; bps = 1; } else { brs = 1; bps = ldb; }
}

// The BF16-split forms split A inside the GEMM (umma_split_fused_kernel) when
// A's rows are contiguous (NoTrans, 16-byte aligned base and column stride)
// and C has at most two 128-wide column tiles, so the f32 tiles TMA brings
// are read about once: there the split pass's read and write of A cost more
// than the GEMM. Wider products keep the two passes (their GEMM is
// compute-bound and the deeper plane ring of the two-pass kernel feeds it
// better).
bool bf16_fused_a(bool ta, int n, const float* A, size_t lda) {
    return !ta && n <= 256 && (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (lda & 3) == 0;
}

// Whether an m x n product runs on CTA pairs (256 x 256 tiles) rather than
// 128 x 128 tiles: by the number of waves, one of pairs taking 1.7 times one of
// small tiles (BF16X6; 3xBF16 1.4) for four times the C per pair of SMs.
// Measured per wave: 8192^3 305 against 180 us (X6), 159 against 112 (3x);
// 2048^3 88 against 52, 50 against 39. One wave of either (777 x 999 x 1234,
// X6): 77 us on pairs, 56 on small tiles.
bool bf16_pair_tiles(int planes, int m, int n, int sms) {
    const long t128 = static_cast<long>((m + 127) / 128) * ((n + 127) / 128);
    const long t256 = static_cast<long>((m + 255) / 256) * ((n + 255) / 256);
    const long w128 = (t128 + sms - 1) / sms, w256 = (t256 + sms / 2 - 1) / std::max(sms / 2, 1);
    return sms >= 2 && (planes == 2 ? 14 : 17) * w256 < 10 * w128;
}

template <int MODE>
cudaError_t launch_bf16_fused(const CUtensorMap& ta32, const CUtensorMap& tb, const UParams& p, int sms,
                              cudaStream_t st) {
    auto kern = umma_split_fused_kernel<MODE>;
    constexpr int smem = fz_smem_bytes<MODE>();
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int grid = 2 * std::min(p.num_tiles, sms / 2);
    const char* name = (MODE == kModeBf16x3) ? "umma_bf16x3" : "umma_bf16x6";
    KernelTimer tm;
    kernel_timing_begin(name, 2.0 * p.m * p.n * static_cast<double>(p.k) * UCfg<MODE>::NPROD, st, &tm);
    kern<<<grid, kFzThreads, smem, st>>>(ta32, tb, p);
    kernel_timing_end(&tm, st);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_bf16_split_gemm(int planes, bool ta, bool tb, int m, int n, int k, float alpha,
                                   const float* A, size_t lda, const float* B, size_t ldb, float beta,
                                   float* C, size_t ldc, cudaStream_t st, CUresult* cu_err) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool fused = bf16_fused_a(ta, n, A, lda);
    const bool pair = !fused && bf16_pair_tiles(planes, m, n, sms);
    const int UM = pair || fused ? 256 : kUM, UN = pair ? kPairN : 128;
    const size_t kp = round_up(static_cast<size_t>(k), 8);  // 16-byte rows of bf16
    const size_t pa = fused ? 0 : static_cast<size_t>(m) * kp, pb = static_cast<size_t>(n) * kp;
    void* buf = nullptr;
    const size_t a_bytes = round_up(planes * pa * sizeof(__nv_bfloat16), 256);
    cudaError_t e = scratch_alloc(&buf, a_bytes + planes * pb * sizeof(__nv_bfloat16), st);
    if (e != cudaSuccess) return e;
    __nv_bfloat16* sa = static_cast<__nv_bfloat16*>(buf);
    __nv_bfloat16* sb = reinterpret_cast<__nv_bfloat16*>(static_cast<uint8_t*>(buf) + a_bytes);
    size_t ars, aps, brs, bps;
    operand_views(ta, tb, lda, ldb, ars, aps, brs, bps);
    const dim3 ga((k + kTile - 1) / kTile, (m + kTile - 1) / kTile);
    const dim3 gb((k + kTile - 1) / kTile, (n + kTile - 1) / kTile);
    if (!fused) {
        bf16_split_kernel<<<ga, 256, 0, st>>>(A, ars, aps, m, k, planes, sa, kp, pa);
        count_launch();
    }
    bf16_split_kernel<<<gb, 256, 0, st>>>(B, brs, bps, n, k, planes, sb, kp, pb);
    count_launch();
    // rows of the plane boxes: one stage's K (BF16X6 pairs take half a K tile)
    const int rb = (pair && planes == 3) ? PairCfg<kModeBf16x6>::KB : kRowBytes;
    CUtensorMap tma, tmb;
    // fused: A itself as an m x k f32 tensor, 128-row x 64-column boxes
    CUresult r = fused ? make_tmap_2d(&tma, A, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(float), m, k, lda, kUM, 64,
                                      false)
                       : make_tmap_planes(&tma, sa, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k, m, planes, kp, 128, rb);
    if (r == CUDA_SUCCESS)
        r = make_tmap_planes(&tmb, sb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k, n, planes, kp, fused ? kFzN / 2 : 128, rb);
    if (r != CUDA_SUCCESS) {
        if (cu_err) *cu_err = r;
        cudaFreeAsync(buf, st);
        return cudaErrorInvalidValue;
    }
    UParams p{};
    p.m = m; p.n = n; p.k = k;
    p.tiles_m = (m + UM - 1) / UM;
    p.tiles_n = (n + UN - 1) / UN;
    p.num_tiles = p.tiles_m * p.tiles_n;
    p.num_kt = static_cast<int>((k + 63) / 64);
    p.kt_per_chunk = 2;  // FP32 promotion every 128 elements of K
    p.kchunks = (p.num_kt + p.kt_per_chunk - 1) / p.kt_per_chunk;
    p.beta_mode = (beta == 0.f) ? 0 : (beta == 1.f ? 1 : 2);
    p.alpha_f = alpha; p.beta_f = beta;
    p.c = C; p.ldc = ldc;
    p.cin = C;
    p.err = device_error_word();
    if (pair)
        e = (planes == 2) ? launch_umma_pair<kModeBf16x3>(tma, tmb, p, sms, st)
                          : launch_umma_pair<kModeBf16x6>(tma, tmb, p, sms, st);
    else if (fused)
        e = (planes == 2) ? launch_bf16_fused<kModeBf16x3>(tma, tmb, p, sms, st)
                          : launch_bf16_fused<kModeBf16x6>(tma, tmb, p, sms, st);
    else
        e = (planes == 2) ? launch_umma<kModeBf16x3>(tma, tmb, p, st) : launch_umma<kModeBf16x6>(tma, tmb, p, st);
    cudaFreeAsync(buf, st);
    return e;
}

// Many f32 GEMMs in a BF16-split form (planes 2: 3xBF16, 3: BF16X6) with two
// launches for the whole batch: one split pass over every operand, then one
// persistent umma_grouped_kernel over every problem's tiles. C0 of problem i
// comes from cin[i] (leading dimension ldcin[i]) or probs[i].c. Each result
// equals that problem's own rb_sgemm_dev(..., form, ...) bit for bit.
int bf16_grouped_dev(int planes, const rb_gemm_problem* probs, size_t count, const void* const* cin,
                     const size_t* ldcin, cudaStream_t st, int32_t* ce) {
    constexpr int UN = 128;
    struct Job {
        bool ta, tb;
        int m, n, k;
        const float *a, *b;
        size_t lda, ldb;
        float* c;
        const float* c0;
        size_t ldc;
        float alpha, beta;
        size_t kp, off_a, off_b;
        int num_kt;
    };
    std::vector<Job> jobs;
    jobs.reserve(count);
    size_t elems = 0;  // bf16 plane elements, every operand 256-byte aligned
    cudaError_t e = cudaSuccess;
    for (size_t i = 0; i < count; ++i) {
        const rb_gemm_problem& q = probs[i];
        if (q.dtype != 0) return RB_ERR_UNSUPPORTED;
        const int v = validate_problem(q);
        if (v != RB_OK) return v;
        const bool col = q.layout == RB_COL_MAJOR;
        const size_t m = col ? q.m : q.n, n = col ? q.n : q.m;
        if (m == 0 || n == 0) continue;
        if (m > 0x7fffffff || n > 0x7fffffff || q.k > 0x7fffffff) return RB_ERR_INVALID_ARG;
        float* c = static_cast<float*>(q.c);
        const float* c0 = cin ? static_cast<const float*>(cin[i]) : c;
        const size_t ldc0 = cin ? ldcin[i] : q.ldc;
        const float beta = static_cast<float>(q.beta), alpha = static_cast<float>(q.alpha);
        if (beta != 0.f && c0 != c && ldc0 != q.ldc) {
            // the kernels read C0 with C's leading dimension: bring it into C first
            e = cudaMemcpy2DAsync(c, q.ldc * 4, c0, ldc0 * 4, m * 4, n, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) break;
            c0 = c;
        }
        if (q.k == 0 || alpha == 0.f) {  // C = beta * C0 only (gemm_contig's early out)
            if (beta != 0.f && c0 != c) {
                e = cudaMemcpy2DAsync(c, q.ldc * 4, c0, q.ldc * 4, m * 4, n, cudaMemcpyDeviceToDevice, st);
                if (e != cudaSuccess) break;
            }
            e = launch_scale_c<float>(static_cast<int>(m), static_cast<int>(n), beta, c, q.ldc, st);
            if (e != cudaSuccess) break;
            continue;
        }
        Job j{};
        const bool ta = q.transa != RB_NO_TRANS, tb = q.transb != RB_NO_TRANS;
        j.ta = col ? ta : tb;
        j.tb = col ? tb : ta;
        j.m = static_cast<int>(m);
        j.n = static_cast<int>(n);
        j.k = static_cast<int>(q.k);
        j.a = static_cast<const float*>(col ? q.a : q.b);
        j.b = static_cast<const float*>(col ? q.b : q.a);
        j.lda = col ? q.lda : q.ldb;
        j.ldb = col ? q.ldb : q.lda;
        j.c = c;
        j.c0 = c0;
        j.ldc = q.ldc;
        j.alpha = alpha;
        j.beta = beta;
        j.kp = round_up(q.k, 8);  // 16-byte rows of bf16
        j.num_kt = static_cast<int>((q.k + 63) / 64);
        j.off_a = elems;
        elems += round_up(planes * m * j.kp, 128);
        j.off_b = elems;
        elems += round_up(planes * n * j.kp, 128);
        jobs.push_back(j);
    }
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        return RB_ERR_CUDA;
    }
    if (jobs.empty()) return RB_OK;
    // longest tiles first: the CTAs walk the items with a stride of the grid
    std::stable_sort(jobs.begin(), jobs.end(), [](const Job& x, const Job& y) { return x.num_kt > y.num_kt; });
    const int np = static_cast<int>(jobs.size());
    // device image: [entries][starts][operands], then the planes
    const size_t ent_bytes = round_up(np * sizeof(UGroupEntry), 256);
    const size_t starts_bytes = round_up((np + 1) * sizeof(int), 256);
    const size_t ops_bytes = round_up(2 * np * sizeof(BsOperand), 256);
    const size_t img_bytes = ent_bytes + starts_bytes + ops_bytes;
    uint8_t* mem = nullptr;
    e = scratch_alloc(reinterpret_cast<void**>(&mem), img_bytes + elems * sizeof(__nv_bfloat16), st);
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? RB_ERR_ALLOC : RB_ERR_CUDA;
    }
    std::vector<uint8_t> img(img_bytes, 0);
    int* starts = reinterpret_cast<int*>(img.data() + ent_bytes);
    BsOperand* ops = reinterpret_cast<BsOperand*>(img.data() + ent_bytes + starts_bytes);
    __nv_bfloat16* dplanes = reinterpret_cast<__nv_bfloat16*>(mem + img_bytes);
    uint32_t* err_word = device_error_word();
    int tiles = 0, split_blocks = 0;
    double work = 0;
    CUresult r = CUDA_SUCCESS;
    for (int i = 0; i < np && r == CUDA_SUCCESS; ++i) {
        const Job& j = jobs[i];
        __nv_bfloat16* sa = dplanes + j.off_a;
        __nv_bfloat16* sb = dplanes + j.off_b;
        size_t ars, aps, brs, bps;
        operand_views(j.ta, j.tb, j.lda, j.ldb, ars, aps, brs, bps);
        const int gx = (j.k + kTile - 1) / kTile;
        const struct { const float* x; size_t rs, ps; int R; __nv_bfloat16* out; } od[2] = {
            {j.a, ars, aps, j.m, sa}, {j.b, brs, bps, j.n, sb}};
        for (int h = 0; h < 2; ++h) {
            BsOperand& o = ops[2 * i + h];
            o.x = od[h].x; o.rs = od[h].rs; o.ps = od[h].ps;
            o.R = od[h].R; o.K = j.k; o.planes = planes;
            o.out = od[h].out;
            o.kp = j.kp; o.plane = static_cast<size_t>(od[h].R) * j.kp;
            o.gx = gx;
            o.start = split_blocks;
            split_blocks += gx * ((o.R + kTile - 1) / kTile);
        }
        UGroupEntry g{};  // 64-byte aligned here; copied into the image below
        r = make_tmap_planes(&g.tmA, sa, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, j.k, j.m, planes, j.kp, kUM);
        if (r == CUDA_SUCCESS)
            r = make_tmap_planes(&g.tmB, sb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, j.k, j.n, planes, j.kp, UN);
        UParams& p = g.p;
        p.m = j.m; p.n = j.n; p.k = j.k;
        p.tiles_m = (j.m + kUM - 1) / kUM;
        p.tiles_n = (j.n + UN - 1) / UN;
        p.num_tiles = p.tiles_m * p.tiles_n;
        p.num_kt = j.num_kt;
        p.kt_per_chunk = 2;  // FP32 promotion every 128 elements of K
        p.kchunks = (p.num_kt + p.kt_per_chunk - 1) / p.kt_per_chunk;
        p.beta_mode = (j.beta == 0.f) ? 0 : (j.beta == 1.f ? 1 : 2);
        p.alpha_f = j.alpha; p.beta_f = j.beta;
        p.c = j.c; p.ldc = j.ldc;
        p.cin = j.c0;
        p.err = err_word;
        std::memcpy(img.data() + i * sizeof(UGroupEntry), &g, sizeof(UGroupEntry));
        starts[i] = tiles;
        tiles += p.num_tiles;
        work += 2.0 * j.m * j.n * static_cast<double>(j.k) * (planes == 2 ? 3 : 6);
    }
    starts[np] = tiles;
    if (r != CUDA_SUCCESS) {
        if (ce) *ce = static_cast<int32_t>(r);
        cudaFreeAsync(mem, st);
        return RB_ERR_CUDA;
    }
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int grid = tiles < sms ? tiles : sms;
    // a pageable source: the driver has staged the image when the call returns
    e = cudaMemcpyAsync(mem, img.data(), img_bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        bf16_split_grouped_kernel<<<split_blocks, 256, 0, st>>>(
            reinterpret_cast<const BsOperand*>(mem + ent_bytes + starts_bytes), 2 * np);
        const UGroupEntry* dtab = reinterpret_cast<const UGroupEntry*>(mem);
        const int* dstarts = reinterpret_cast<const int*>(mem + ent_bytes);
        KernelTimer tmr;
        if (planes == 2) {
            constexpr int smem = umma_smem_bytes<kModeBf16x3>();
            static bool attr3 = false;
            if (!attr3) {
                e = cudaFuncSetAttribute(umma_grouped_kernel<kModeBf16x3>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
                attr3 = e == cudaSuccess;
            }
            kernel_timing_begin("umma_bf16x3_grouped", work, st, &tmr);
            if (e == cudaSuccess)
                umma_grouped_kernel<kModeBf16x3><<<grid, UCfg<kModeBf16x3>::THREADS, smem, st>>>(dtab, dstarts, np,
                                                                                                 err_word);
        } else {
            constexpr int smem = umma_smem_bytes<kModeBf16x6>();
            static bool attr6 = false;
            if (!attr6) {
                e = cudaFuncSetAttribute(umma_grouped_kernel<kModeBf16x6>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
                attr6 = e == cudaSuccess;
            }
            kernel_timing_begin("umma_bf16x6_grouped", work, st, &tmr);
            if (e == cudaSuccess)
                umma_grouped_kernel<kModeBf16x6><<<grid, UCfg<kModeBf16x6>::THREADS, smem, st>>>(dtab, dstarts, np,
                                                                                                 err_word);
        }
        kernel_timing_end(&tmr, st);
        count_launch(2);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    cudaFreeAsync(mem, st);
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        return RB_ERR_CUDA;
    }
    return RB_OK;
}

// Dynamic shared memory of both Ozaki tile widths, set once per process.
cudaError_t ozaki_kernel_attributes() {
    static std::once_flag once;
    static cudaError_t result = cudaSuccess;
    std::call_once(once, [] {
        result = cudaFuncSetAttribute(ozaki_gemm_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      OzCfg<256>::SMEM);
        if (result == cudaSuccess)
            result = cudaFuncSetAttribute(ozaki_gemm_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          OzCfg<128>::SMEM);
        if (result == cudaSuccess)
            result = cudaFuncSetAttribute(ozaki_grouped_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          OzCfg<256>::SMEM);
        if (result == cudaSuccess)
            result = cudaFuncSetAttribute(ozaki_grouped_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          OzCfg<128>::SMEM);
        if (result == cudaSuccess)
            result = cudaFuncSetAttribute(ozaki_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPzSmem);
        if (result == cudaSuccess)
            result = cudaFuncSetAttribute(ozaki_pair_grouped_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kPzSmem);
    });
    return result;
}

// Tail tiles to run unit by unit (OzParams::tail_tiles): the tiles of the
// partial last wave (all tiles when there are fewer than SMs), when dealing
// their units as oz_item does finishes clearly before one more whole tile
// would, counting the reduce pass over their planes and C; else 0. Times are
// modelled from the products per unit (a diagonal d has d + 1) at the B200's
// INT8 rate per SM and its copy rate; only their ratio matters.
int ozaki_tail_tiles(int num_tiles, int slices, int kchunks, int k, int sms, int un) {
    const int upc = (slices + 1) / 2;
    if (kchunks != 1 || upc < 2 || sms < 1) return 0;
    const int full = num_tiles / sms;
    const int tail = num_tiles - full * sms;
    if (tail == 0) return 0;
    const int total = tail * upc;
    const int G = full > 0 ? sms : std::min(total, sms);
    std::vector<int> load(G, 0);
    for (int j = 0; j < total; ++j) {
        int t, lo, hi, tt, d0, d1;
        oz_item(num_tiles, tail, 1, upc, G, num_tiles - tail + j, t, lo, hi, tt);
        oz_unit(slices, lo % upc, d0, d1);
        load[(num_tiles - tail + j) % G] += (d0 + 1) + (d1 >= 0 ? d1 + 1 : 0);
    }
    const int max_load = *std::max_element(load.begin(), load.end());
    const double tile_elems = static_cast<double>(kUM) * un;
    const double product_s = 2.0 * tile_elems * static_cast<double>(k) / (4.4e15 / 148);
    const double whole_tile_s = product_s * slices * (slices + 1) / 2;
    const double reduce_s = 4e-6 + tail * (upc + 2.0) * tile_elems * sizeof(double) / 6.5e12;
    const bool fits = tail * upc * tile_elems * sizeof(double) <= static_cast<double>(size_t(512) << 20);
    return (fits && product_s * max_load + reduce_s < 0.9 * whole_tile_s) ? tail : 0;
}

// Time (us) of the fullest pair when the tail's items are dealt as pz_item does:
// ranks in order of cost, G to a pass, every other pass mirrored. A (group, part)
// is `tail` ranks of one cost, so a pass takes each as one run of pairs; dealing
// item by item took up to 45 us of every call.
double ozaki_pair_tail_load(const OzParams& p, const int (&cost)[kOzGroups], int pairs, double prod_us) {
    const int groups = (p.slices + 3) / 4;
    int total = 0;
    for (int g = 0; g < groups; ++g) total += p.tail_tiles * p.parts[g];
    std::vector<std::pair<long long, int>> step(pairs + 1);  // products, items: from this pair on
    int rank = 0;
    for (int i = 0; i < groups; ++i) {
        const int g = p.order[i], parts = p.parts[g];
        for (int part = 0; part < parts; ++part) {
            const long long nkt = p.num_kt, kts = nkt * (part + 1) / parts - nkt * part / parts;
            for (const int end = rank + p.tail_tiles; rank < end;) {
                const int pass = rank / pairs, len = std::min(pairs, total - pass * pairs);
                const int to = std::min(end, (pass + 1) * pairs);
                int lo = rank - pass * pairs, hi = to - pass * pairs;
                if (pass & 1) {
                    const int l = len - hi;
                    hi = len - lo;
                    lo = l;
                }
                step[lo].first += cost[g] * kts;
                step[hi].first -= cost[g] * kts;
                ++step[lo].second;
                --step[hi].second;
                rank = to;
            }
        }
    }
    double load = 0;
    long long products = 0, items = 0;
    for (int q = 0; q < pairs; ++q) {
        products += step[q].first;
        items += step[q].second;
        load = std::max(load, products * prod_us + 3.0 * items);
    }
    return load;
}

// The pair kernel's tail (OzParams::tail_tiles, parts, order, plane0, planes):
// the tiles of the partial last wave (all tiles when there are fewer than
// pairs), cut into groups of diagonals and K parts, where that finishes
// before a whole further wave would. Costs in products (36 per K tile of a
// whole tile at 8 slices) over the K tiles; a product of a 256 x 128 tile and
// one K tile takes 256 clocks, an item 3 us beside its products, the planes'
// traffic and the second launch 10 us and their bytes at 5 TB/s. Measured
// against whole tiles (us; parts of the dearer group): 300 x 300 x 4000 -121
// (4), 512^3 -12 (4), 3000 x 5000 x 2048 -34 (3), 4096 x 2048 x 4096 -33 (3);
// 1024^3 +10 and 777 x 999 x 1234 +6 (1), 1500^3 +42 (1): left whole.
void ozaki_pair_tail(OzParams& p, int pairs) {
    const int groups = (p.slices + 3) / 4;
    p.tail_tiles = 0;
    p.planes = 0;
    int cost[kOzGroups] = {};
    for (int g = 0; g < kOzGroups; ++g) {
        p.parts[g] = 0;
        p.order[g] = 0;
        p.plane0[g] = 0;
        if (g >= groups) continue;
        p.parts[g] = 1;
        for (int d = 4 * g; d < 4 * g + pz_nd(p.slices, g); ++d) cost[g] += d + 1;
    }
    const int tail = p.num_tiles % pairs;
    if (p.kchunks != 1 || tail == 0) return;
    const int all = p.slices * (p.slices + 1) / 2;
    const double prod_us = 256 / 1.7e3;                   // one product, one K tile
    double best = all * p.num_kt * prod_us + 4.0;         // a whole tile's wave
    OzParams cand = p;
    cand.tail_tiles = tail;
    // parts of the dearest group; the others in proportion to their cost
    for (int pd = 1; pd <= 16 && pd <= p.num_kt; pd = pd < 3 ? pd + 1 : pd + pd / 2) {
        int dear = 0;
        for (int g = 1; g < groups; ++g)
            if (cost[g] > cost[dear]) dear = g;
        int planes = 0, order[kOzGroups];
        for (int g = 0; g < groups; ++g) {
            cand.parts[g] = std::max(1, std::min(p.num_kt, (cost[g] * pd + cost[dear] / 2) / cost[dear]));
            cand.plane0[g] = planes;
            planes += cand.parts[g] * ((pz_nd(p.slices, g) + 1) / 2);
            order[g] = g;
        }
        std::sort(order, order + groups, [&](int x, int y) {
            return static_cast<double>(cost[x]) / cand.parts[x] > static_cast<double>(cost[y]) / cand.parts[y];
        });
        for (int g = 0; g < groups; ++g) cand.order[g] = order[g];
        cand.planes = planes;
        const size_t bytes = static_cast<size_t>(tail) * planes * kPzTileElems * sizeof(double);
        if (bytes > (size_t(512) << 20)) break;
        const double load = ozaki_pair_tail_load(cand, cost, pairs, prod_us);
        const double t = load + 10.0 + (bytes + 2.0 * tail * kPzTileElems * sizeof(double)) / 5e6;
        if (t < best) {
            best = t;
            p.tail_tiles = tail;
            p.planes = planes;
            for (int g = 0; g < kOzGroups; ++g) {
                p.parts[g] = cand.parts[g];
                p.order[g] = cand.order[g];
                p.plane0[g] = cand.plane0[g];
            }
        }
    }
}

// Whether an m x n product takes the pair kernel: unless one tile row of 128 is
// all it has, or a pair's 256 rows pad so much more than 128 that the wide
// tiles' larger cost (per 128 x 256 C of one SM 1 against 0.85 for a pair's
// 256 x 128) is the smaller one.
bool ozaki_pair_tiles(int m, int n) {
    if (m <= 128) return false;
    const double wide = static_cast<double>((m + 127) / 128) * ((n + 255) / 256);
    return n <= 128 || 0.85 * ((m + 255) / 256) * ((n + 127) / 128) <= wide;
}

cudaError_t launch_ozaki_gemm(bool ta, bool tb, int m, int n, int k, double alpha, const double* A,
                              size_t lda, const double* B, size_t ldb, double beta, double* C,
                              size_t ldc, int slices, cudaStream_t st, CUresult* cu_err, int a_cx) {
    const size_t kp = round_up(static_cast<size_t>(k), 16);
    const size_t pa = static_cast<size_t>(m) * kp, pb = static_cast<size_t>(n) * kp;
    void* buf = nullptr;
    const size_t exps = round_up((static_cast<size_t>(m) + n) * sizeof(int), 256);
    const size_t a_bytes = round_up(slices * pa, 256);
    // the partial last wave runs unit by unit when that pays (see OzParams)
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const bool pair = sms >= 2 && ozaki_pair_tiles(m, n);
    const int un = pair ? kPzN : ozaki_tile_n(m, n, k), um = pair ? 256 : kUM;
    const int upc = (slices + 1) / 2;
    OzParams p{};
    p.m = m; p.n = n; p.k = k;
    p.un = un;
    p.tiles_m = (m + um - 1) / um;
    p.tiles_n = (n + un - 1) / un;
    p.num_tiles = p.tiles_m * p.tiles_n;
    p.num_kt = static_cast<int>((k + 127) / 128);
    p.slices = slices;
    // exact INT32: a diagonal has <= slices products of |d_t d_u| <= 128*128 per K element
    p.kt_per_chunk = static_cast<int>(std::max(2147483647LL / (static_cast<long long>(slices) * 128 * 128) / 128, 1LL));
    p.kchunks = (p.num_kt + p.kt_per_chunk - 1) / p.kt_per_chunk;
    if (pair) ozaki_pair_tail(p, sms / 2);
    else      p.tail_tiles = ozaki_tail_tiles(p.num_tiles, slices, p.kchunks, k, sms, un);
    const size_t b_bytes = round_up(slices * pb, 256);
    const size_t w_bytes = static_cast<size_t>(p.tail_tiles) * (pair ? p.planes : upc) * um * un * sizeof(double);
    cudaError_t e = scratch_alloc(&buf, exps + a_bytes + b_bytes + w_bytes, st);
    if (e != cudaSuccess) return e;
    int* ea = static_cast<int*>(buf);
    int* eb = ea + m;
    int8_t* sla = reinterpret_cast<int8_t*>(static_cast<uint8_t*>(buf) + exps);
    int8_t* slb = sla + a_bytes;
    size_t ars, aps, brs, bps;
    operand_views(ta, tb, lda, ldb, ars, aps, brs, bps);
    if (a_cx) ars = lda;
    launch_ozaki_prepass(OzPair{{{A, ars, aps, a_cx, m, k, ea, sla, kp, pa, 0, 0, 0, 0},
                                 {B, brs, bps, 0, n, k, eb, slb, kp, pb, 0, 0, 0, 0}}},
                         slices, st);
    CUtensorMap tma, tmb;
    CUresult r = make_tmap_planes(&tma, sla, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, k, m, slices, kp, kUM);
    if (r == CUDA_SUCCESS)
        r = make_tmap_planes(&tmb, slb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, k, n, slices, kp, pair ? 64 : un);
    if (r != CUDA_SUCCESS) {
        if (cu_err) *cu_err = r;
        cudaFreeAsync(buf, st);
        return cudaErrorInvalidValue;
    }
    p.beta_mode = (beta == 0.0) ? 0 : (beta == 1.0 ? 1 : 2);
    p.alpha = alpha; p.beta = beta;
    p.c = C; p.ldc = ldc;
    p.cin = C;
    p.row_exp = ea; p.col_exp = eb;
    p.err = device_error_word();
    if (p.tail_tiles > 0)
        p.ws = reinterpret_cast<double*>(static_cast<uint8_t*>(buf) + exps + a_bytes + b_bytes);

    e = ozaki_kernel_attributes();
    if (e != cudaSuccess) { cudaFreeAsync(buf, st); return e; }
    KernelTimer tmr;
    kernel_timing_begin("umma_ozaki_i8", 2.0 * m * n * static_cast<double>(k) * slices * (slices + 1) / 2, st, &tmr);
    if (pair) {
        ozaki_pair_kernel<<<2 * std::min(pz_items(p), sms / 2), pz_threads(kPzEpiWarps), kPzSmem, st>>>(tma, tmb, p);
    } else {
        const int items = p.num_tiles + p.tail_tiles * (p.kchunks * upc - 1);
        const int grid = items < sms ? items : sms;
        if (un == 256) ozaki_gemm_kernel<256><<<grid, kOzThreads, OzCfg<256>::SMEM, st>>>(tma, tmb, p);
        else           ozaki_gemm_kernel<128><<<grid, kOzThreads, OzCfg<128>::SMEM, st>>>(tma, tmb, p);
    }
    kernel_timing_end(&tmr, st);
    count_launch();
    if (p.tail_tiles > 0) {
        const size_t work = static_cast<size_t>(p.tail_tiles) * um * un / (pair ? 2 : 1);
        const unsigned blocks = static_cast<unsigned>(std::min<size_t>((work + 255) / 256, static_cast<size_t>(sms) * 16));
        if (pair) ozaki_pair_reduce_kernel<<<blocks, 256, 0, st>>>(p);
        else      ozaki_reduce_kernel<<<blocks, 256, 0, st>>>(p, p.kchunks * upc);
        count_launch();
    }
    e = cudaGetLastError();
    cudaFreeAsync(buf, st);
    return e;
}

// The problems of one kind of tile (0: pairs; 1, 2: 256- and 128-wide tiles of
// one CTA) in a grouped Ozaki launch, longest K first.
struct OzGroupKind {
    std::vector<std::pair<int, int>> jobs;  // tiles, K tiles
    double per_kt, per_tile;                // us: one tile's K tile, the rest of it
    // of `workers` (pairs, CTAs), each with every workers-th tile: the first's time
    double time(int workers) const {
        double t = 0;
        long long at = 0;
        for (const auto& j : jobs) {
            const long long end = at + j.first;
            t += ((end + workers - 1) / workers - (at + workers - 1) / workers) * (j.second * per_kt + per_tile);
            at = end;
        }
        return t;
    }
    int workers_for(double us, int cap) const {  // the fewest that finish in `us` (cap + 1: none do)
        if (jobs.empty()) return 0;
        int lo = 1, hi = cap + 1;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (time(mid) <= us) hi = mid;
            else                 lo = mid + 1;
        }
        return lo;
    }
};

// Workers of each kind's launch when the kinds share the SMs and start together:
// the split that ends first, or false where one after the other does about as
// well. A persistent CTA holds its SM, so launches of the whole GPU each run one
// after the other however few tiles they have, and each ends in its longest
// chain. 40 mixed requests up to 512 a side took 155 us in two kinds of tile, 208
// with pairs as a third, 148 sharing; 24 up to 2048 a side 358, 458 and 270. Costs
// as fitted to 41 sets: a product of a pair's tile 250 clocks, of a 128 x 256 one
// 540, of a 128 x 128 one 450; a tile's drains 10, 50 and 20 us. What the split
// leaves over goes to the kind that ends last.
bool ozaki_share_sms(OzGroupKind (&kinds)[3], int slices, int sms, int (&workers)[3]) {
    const double prod_us = slices * (slices + 1) / 2 / 1.7e3;
    const double clocks[3] = {250, 540, 450}, tile_us[3] = {10, 50, 20};
    const int sm[3] = {2, 1, 1};
    int cap[3] = {sms / 2, sms, sms};
    double lo = 0, hi = 0;
    int used = 0;
    for (int q = 0; q < 3; ++q) {
        workers[q] = 0;
        if (kinds[q].jobs.empty()) continue;
        kinds[q].per_kt = clocks[q] * prod_us;
        kinds[q].per_tile = tile_us[q];
        long long tiles = 0;
        for (const auto& j : kinds[q].jobs) tiles += j.first;
        cap[q] = static_cast<int>(std::min<long long>(cap[q], tiles));
        const double t = kinds[q].time(cap[q]);
        lo = std::max(lo, t);
        hi += t;
        ++used;
    }
    hi *= 0.95;
    int left = 0;
    auto fits = [&](double us) {
        left = sms;
        bool all = true;
        for (int q = 0; q < 3; ++q) {
            workers[q] = kinds[q].workers_for(us, cap[q]);
            left -= sm[q] * workers[q];
            all = all && workers[q] <= cap[q];
        }
        return all && left >= 0;
    };
    if (used < 2 || !fits(hi)) return false;
    for (int i = 0; i < 7; ++i) {
        const double mid = 0.5 * (lo + hi);
        if (fits(mid)) hi = mid;
        else           lo = mid;
    }
    fits(hi);
    for (;;) {
        int last = -1;
        double end = 0;
        for (int q = 0; q < 3; ++q) {
            if (workers[q] >= cap[q] || left < sm[q]) continue;
            const double t = kinds[q].time(workers[q]);
            if (t > end) {
                end = t;
                last = q;
            }
        }
        if (last < 0) return true;
        const int more = std::min(cap[last] - workers[last], std::max(1, left / sm[last] / 4));
        workers[last] += more;
        left -= sm[last] * more;
    }
}

// Many f64 GEMMs in the Ozaki form: one exponent pass and one slice pass over
// every operand, then a persistent launch per kind of tile
// (ozaki_pair_grouped_kernel, ozaki_grouped_kernel of either width) over the
// problems of that kind. probs[i] is
// column-major or row-major like rb_gemm_problem; its C0 is read from
// cin[i] (leading dimension ldcin[i]; probs[i].c itself when cin is null) and
// the result goes to probs[i].c. Every tile folds its terms in the order of the
// single call, so each result equals that problem's own
// rb_dgemm_dev(..., RB_PREC_OZAKI, ...) bit for bit.
int ozaki_grouped_dev(const rb_gemm_problem* probs, size_t count, const void* const* cin, const size_t* ldcin,
                      cudaStream_t st, int32_t* ce) {
    const int slices = rb_get_ozaki_slices();
    const long long kt_chunk = std::max(2147483647LL / (static_cast<long long>(slices) * 128 * 128) / 128, 1LL);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    struct Job {
        bool ta, tb;
        int m, n, k;
        const double *a, *b;
        size_t lda, ldb;
        double* c;
        const double* c0;
        size_t ldc;
        double alpha, beta;
        size_t kp, off_exp, off_a, off_b;
        int num_kt;
        int kind;  // 0: CTA pairs; 1, 2: 256- and 128-wide tiles
    };
    std::vector<Job> jobs;
    jobs.reserve(count);
    size_t exps = 0, planes = 0;
    cudaError_t e = cudaSuccess;
    for (size_t i = 0; i < count; ++i) {
        const rb_gemm_problem& q = probs[i];
        if (q.dtype != 1) return RB_ERR_UNSUPPORTED;
        const int v = validate_problem(q);
        if (v != RB_OK) return v;
        const bool col = q.layout == RB_COL_MAJOR;
        const size_t m = col ? q.m : q.n, n = col ? q.n : q.m;
        if (m == 0 || n == 0) continue;
        if (m > 0x7fffffff || n > 0x7fffffff || q.k > 0x7fffffff) return RB_ERR_INVALID_ARG;
        double* c = static_cast<double*>(q.c);
        const double* c0 = cin ? static_cast<const double*>(cin[i]) : c;
        const size_t ldc0 = cin ? ldcin[i] : q.ldc;
        if (q.beta != 0.0 && c0 != c && ldc0 != q.ldc) {
            // the kernels read C0 with C's leading dimension: bring it into C first
            e = cudaMemcpy2DAsync(c, q.ldc * 8, c0, ldc0 * 8, m * 8, n, cudaMemcpyDeviceToDevice, st);
            if (e != cudaSuccess) break;
            c0 = c;
        }
        if (q.k == 0 || q.alpha == 0.0) {  // C = beta * C0 only (gemm_contig's early out)
            if (q.beta != 0.0 && c0 != c) {
                e = cudaMemcpy2DAsync(c, q.ldc * 8, c0, q.ldc * 8, m * 8, n, cudaMemcpyDeviceToDevice, st);
                if (e != cudaSuccess) break;
            }
            e = launch_scale_c<double>(static_cast<int>(m), static_cast<int>(n), q.beta, c, q.ldc, st);
            if (e != cudaSuccess) break;
            continue;
        }
        Job j{};
        const bool ta = q.transa != RB_NO_TRANS, tb = q.transb != RB_NO_TRANS;
        j.ta = col ? ta : tb;
        j.tb = col ? tb : ta;
        j.m = static_cast<int>(m);
        j.n = static_cast<int>(n);
        j.k = static_cast<int>(q.k);
        j.a = static_cast<const double*>(col ? q.a : q.b);
        j.b = static_cast<const double*>(col ? q.b : q.a);
        j.lda = col ? q.lda : q.ldb;
        j.ldb = col ? q.ldb : q.lda;
        j.c = c;
        j.c0 = c0;
        j.ldc = q.ldc;
        j.alpha = q.alpha;
        j.beta = q.beta;
        j.kp = round_up(q.k, 16);
        j.num_kt = static_cast<int>((q.k + 127) / 128);
        j.kind = sms >= 2 && ozaki_pair_tiles(j.m, j.n) ? 0 : ozaki_tile_n(j.m, j.n, j.k) == 256 ? 1 : 2;
        j.off_exp = exps;
        exps += m + n;
        j.off_a = planes;
        planes += round_up(slices * m * j.kp, 256);
        j.off_b = planes;
        planes += round_up(slices * n * j.kp, 256);
        jobs.push_back(j);
    }
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        return RB_ERR_CUDA;
    }
    if (jobs.empty()) return RB_OK;
    // one launch per kind of tile; inside each, longest tiles first: the CTAs
    // walk the items with a stride of the grid
    std::stable_sort(jobs.begin(), jobs.end(), [](const Job& x, const Job& y) {
        return x.kind != y.kind ? x.kind < y.kind : x.num_kt > y.num_kt;
    });
    const int np = static_cast<int>(jobs.size());
    // device image: [entries][starts][operands] then exponents, then planes
    const size_t ent_bytes = round_up(np * sizeof(OzGroupEntry), 256);
    const size_t starts_bytes = round_up((np + 3) * sizeof(int), 256);  // each kind's starts and its end
    const size_t ops_bytes = round_up(2 * np * sizeof(OzOperand), 256);
    const size_t img_bytes = ent_bytes + starts_bytes + ops_bytes;
    const size_t exp_bytes = round_up(exps * sizeof(int), 256);
    uint8_t* mem = nullptr;
    e = scratch_alloc(reinterpret_cast<void**>(&mem), img_bytes + exp_bytes + planes, st);
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();
        return e == cudaErrorMemoryAllocation ? RB_ERR_ALLOC : RB_ERR_CUDA;
    }
    std::vector<uint8_t> img(img_bytes, 0);
    int* starts = reinterpret_cast<int*>(img.data() + ent_bytes);
    OzOperand* ops = reinterpret_cast<OzOperand*>(img.data() + ent_bytes + starts_bytes);
    int* dexp = reinterpret_cast<int*>(mem + img_bytes);
    int8_t* dplanes = reinterpret_cast<int8_t*>(mem + img_bytes + exp_bytes);
    uint32_t* err_word = device_error_word();
    int exp_blocks = 0, slice_blocks = 0;
    int kind_first[3] = {}, kind_count[3] = {}, kind_tiles[3] = {};  // problems and tiles of each launch
    OzGroupKind group_kinds[3];
    for (const Job& j : jobs) ++kind_count[j.kind];
    for (int q = 1; q < 3; ++q) kind_first[q] = kind_first[q - 1] + kind_count[q - 1];
    double work = 0;
    CUresult r = CUDA_SUCCESS;
    for (int i = 0; i < np && r == CUDA_SUCCESS; ++i) {
        const Job& j = jobs[i];
        int* ea = dexp + j.off_exp;
        int* eb = ea + j.m;
        int8_t* sla = dplanes + j.off_a;
        int8_t* slb = dplanes + j.off_b;
        size_t ars, aps, brs, bps;
        operand_views(j.ta, j.tb, j.lda, j.ldb, ars, aps, brs, bps);
        ops[2 * i] = {j.a, ars, aps, 0, j.m, j.k, ea, sla, j.kp, static_cast<size_t>(j.m) * j.kp, 0, 0, 0, 0};
        ops[2 * i + 1] = {j.b, brs, bps, 0, j.n, j.k, eb, slb, j.kp, static_cast<size_t>(j.n) * j.kp, 0, 0, 0, 0};
        for (int h = 0; h < 2; ++h) oz_operand_blocks(&ops[2 * i + h], &exp_blocks, &slice_blocks);
        OzGroupEntry g{};  // 64-byte aligned here; copied into the image below
        r = make_tmap_planes(&g.tmA, sla, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, j.k, j.m, slices, j.kp, kUM);
        if (r == CUDA_SUCCESS)
            r = make_tmap_planes(&g.tmB, slb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, j.k, j.n, slices, j.kp,
                                 j.kind == 0 ? 64 : j.kind == 1 ? 256 : 128);
        OzParams& p = g.p;
        p.m = j.m; p.n = j.n; p.k = j.k;
        const int um = j.kind == 0 ? 256 : kUM;
        p.un = j.kind == 1 ? 256 : 128;
        p.tiles_m = (j.m + um - 1) / um;
        p.tiles_n = (j.n + p.un - 1) / p.un;
        p.num_tiles = p.tiles_m * p.tiles_n;
        p.num_kt = j.num_kt;
        p.slices = slices;
        p.kt_per_chunk = static_cast<int>(kt_chunk);
        p.kchunks = (p.num_kt + p.kt_per_chunk - 1) / p.kt_per_chunk;
        p.beta_mode = (j.beta == 0.0) ? 0 : (j.beta == 1.0 ? 1 : 2);
        p.alpha = j.alpha; p.beta = j.beta;
        p.c = j.c; p.ldc = j.ldc;
        p.cin = j.c0;
        p.row_exp = ea; p.col_exp = eb;
        p.err = err_word;
        std::memcpy(img.data() + i * sizeof(OzGroupEntry), &g, sizeof(OzGroupEntry));
        // kind q's starts, counting from its own first tile, and its end at
        // [kind_first[q] + q, kind_first[q] + kind_count[q] + q]
        starts[i + j.kind] = kind_tiles[j.kind];
        kind_tiles[j.kind] += p.num_tiles;
        group_kinds[j.kind].jobs.emplace_back(p.num_tiles, j.num_kt);
        work += 2.0 * j.m * j.n * static_cast<double>(j.k) * slices * (slices + 1) / 2;
    }
    for (int q = 0; q < 3; ++q) starts[kind_first[q] + kind_count[q] + q] = kind_tiles[q];
    if (r != CUDA_SUCCESS) {
        if (ce) *ce = static_cast<int32_t>(r);
        cudaFreeAsync(mem, st);
        return RB_ERR_CUDA;
    }
    e = ozaki_kernel_attributes();
    // a pageable source: the driver has staged the image when the call returns
    if (e == cudaSuccess) e = cudaMemcpyAsync(mem, img.data(), img_bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        const OzOperand* dops = reinterpret_cast<const OzOperand*>(mem + ent_bytes + starts_bytes);
        fill_int_kernel<<<static_cast<unsigned>(std::min<size_t>((exps + 255) / 256, 1024)), 256, 0, st>>>(
            dexp, static_cast<int>(exps), kExpSentinel);
        ozaki_exp_grouped_kernel<<<exp_blocks, 256, 0, st>>>(dops, 2 * np);
        switch (slices) {
#define RB_SLICES(S) \
    case S: ozaki_slice_grouped_kernel<S><<<slice_blocks, 256, 0, st>>>(dops, 2 * np); break;
            RB_SLICES(2) RB_SLICES(3) RB_SLICES(4) RB_SLICES(5) RB_SLICES(6) RB_SLICES(7) RB_SLICES(8)
            RB_SLICES(9) RB_SLICES(10) RB_SLICES(11) RB_SLICES(12)
#undef RB_SLICES
            default: break;
        }
        KernelTimer tmr;
        kernel_timing_begin("umma_ozaki_grouped_i8", work, st, &tmr);
        const OzGroupEntry* dtab = reinterpret_cast<const OzGroupEntry*>(mem);
        const int* dstarts = reinterpret_cast<const int*>(mem + ent_bytes);
        // With more than one kind, the first goes on st and the others on forked
        // streams. Where they share the SMs each has one of its own; else the
        // others have one together, and their CTAs take the SMs that the first
        // launch's leave as they finish. (Pairs first: they need both SMs of a
        // TPC.)
        const int kinds = (kind_count[0] > 0) + (kind_count[1] > 0) + (kind_count[2] > 0);
        int workers[3] = {};
        ForkedStream fk;
        const bool share = kinds > 1 && ozaki_share_sms(group_kinds, slices, sms, workers);
        const bool fork = kinds > 1 && fork_stream(st, &fk, share && kinds == 3) == cudaSuccess;
        if (!share || !fork) {
            workers[0] = sms / 2;
            workers[1] = workers[2] = sms;
        }
        int started = 0;
        for (int q = 0; q < 3; ++q) {
            if (kind_count[q] == 0) continue;
            const cudaStream_t ks = !started || !fork ? st : started == 2 && fk.s2 ? fk.s2 : fk.s;
            ++started;
            const OzGroupEntry* kt = dtab + kind_first[q];
            const int* ks0 = dstarts + kind_first[q] + q;
            const int grid = std::min(kind_tiles[q], workers[q]);
            if (q == 0)
                ozaki_pair_grouped_kernel<<<2 * grid, pz_threads(kPzGroupEpiWarps), kPzSmem, ks>>>(kt, ks0, kind_count[0],
                                                                                                   err_word);
            else if (q == 1)
                ozaki_grouped_kernel<256><<<grid, kOzThreads, OzCfg<256>::SMEM, ks>>>(kt, ks0, kind_count[1], err_word);
            else
                ozaki_grouped_kernel<128><<<grid, kOzThreads, OzCfg<128>::SMEM, ks>>>(kt, ks0, kind_count[2], err_word);
        }
        e = cudaGetLastError();
        if (fork) {
            const cudaError_t je = join_stream(st, &fk);
            if (e == cudaSuccess) e = je;
        }
        kernel_timing_end(&tmr, st);
        count_launch(3 + kinds);
        if (e == cudaSuccess) e = cudaGetLastError();
    }
    cudaFreeAsync(mem, st);
    if (e != cudaSuccess) {
        if (ce) *ce = e;
        return RB_ERR_CUDA;
    }
    return RB_OK;
}

}  // namespace rb

// ==============================================================================
// Allocation-free Ozaki DGEMM.
//
// Some callers cannot let a library call cudaMalloc: a serving process that
// has handed all of the GPU's memory to its own pool up front, or code on a
// latency-critical path where an allocation could block on the device or fail
// halfway through a run. For them, rb_dgemm_ozaki_noalloc runs the same
// Ozaki kernels as rb_dgemm_dev(..., RB_PREC_OZAKI, ...) with every scratch
// buffer (digit planes, exponents, the device status word) carved out of the
// fixed array below. The array is a file-scope __device__ object: every GPU
// that loads this library holds its 64 MiB + 64 KiB until the process exits.
// In host code `g_noalloc_scratch` is only a host-side stand-in for the
// symbol, so its device address is looked up with cudaGetSymbolAddress, once
// per device, on the first call made with that device current (and again
// if that device's context has been replaced since, e.g. after a
// cudaDeviceReset, since the old address then belongs to a dead context).
// ==============================================================================

namespace rb {
namespace {

constexpr size_t kNoAllocScratchBytes = (64u << 20) + (64u << 10);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
struct NoAllocAddr {
    void* ptr;
    unsigned long long ctx;  // the context the address was looked up in (0: unknown)
};
NoAllocAddr g_noalloc_addr[64] = {};

// Bytes of the array one problem uses: the status word, the exponents and
// both digit planes. Returns false (nothing computed) when that exceeds
// `cap`; each step is checked before it can wrap, since m, n and k may each
// be up to 2^31 - 1.
bool noalloc_bytes_needed(size_t m, size_t n, size_t kp, int slices, size_t cap, size_t* need) {
    *need = cap + 1;
    if (m > cap || n > cap || kp > cap) return false;
    const size_t per_k = static_cast<size_t>(slices) * (m + n);  // < 12 * 2^33
    if (kp != 0 && per_k > cap / kp) return false;
    *need = 256 + round_up((m + n) * sizeof(int), 256) + round_up(slices * m * kp, 256) + slices * n * kp;
    return *need <= cap;
}

}  // namespace
}  // namespace rb

extern "C" rb_status rb_dgemm_ozaki_noalloc(rb_layout layout, rb_transpose transa, rb_transpose transb,
                                            size_t m, size_t n, size_t k, double alpha, const double* a,
                                            size_t lda, const double* b, size_t ldb, double beta, double* c,
                                            size_t ldc, void* stream, rb_error* err) {
    using namespace rb;
    auto fail = [&](rb_status s, uint64_t got = 0, uint64_t need = 0, int32_t ce = 0, char which = 0) {
        if (err) {
            err->code = s;
            err->which = which;
            err->got = got;
            err->min_or_need = need;
            err->cuda_error = ce;
        }
        return s;
    };
    if (err) *err = rb_error{0, 0, 0, 0, 0};
    if ((layout != RB_ROW_MAJOR && layout != RB_COL_MAJOR) || transa < RB_NO_TRANS || transa > RB_CONJ_TRANS ||
        transb < RB_NO_TRANS || transb > RB_CONJ_TRANS)
        return fail(RB_ERR_INVALID_ARG);
    // leading dimensions, as check_matrix (src/level3.rs:107-140)
    const bool ta = transa != RB_NO_TRANS, tb = transb != RB_NO_TRANS;
    struct Chk { char w; size_t rows, cols, ld; } chk[3] = {
        {'a', ta ? k : m, ta ? m : k, lda}, {'b', tb ? n : k, tb ? k : n, ldb}, {'c', m, n, ldc}};
    for (const Chk& q : chk) {
        if (q.rows == 0 || q.cols == 0) continue;
        const size_t min_lead = (layout == RB_ROW_MAJOR) ? q.cols : q.rows;
        if (q.ld < min_lead) return fail(RB_ERR_INVALID_LEADING_DIM, q.ld, min_lead, 0, q.w);
    }
    if (m == 0 || n == 0) return RB_OK;
    // row-major -> column-major by swapping operands (src/level3.rs:52-60)
    bool cta = ta, ctb = tb;
    size_t cm = m, cn = n, clda = lda, cldb = ldb;
    const double* ca = a;
    const double* cb = b;
    if (layout == RB_ROW_MAJOR) {
        cta = tb; ctb = ta;
        cm = n; cn = m;
        ca = b; cb = a;
        clda = ldb; cldb = lda;
    }
    if ((k > 0 && (!a || !b)) || !c) return fail(RB_ERR_INVALID_ARG);
    if (cm > 0x7fffffff || cn > 0x7fffffff || k > 0x7fffffff) return fail(RB_ERR_INVALID_ARG);
    const int slices = rb_get_ozaki_slices();
    const size_t kp = round_up(k, 16);
    size_t need = 0;
    if (!noalloc_bytes_needed(cm, cn, kp, slices, kNoAllocScratchBytes, &need))
        return fail(RB_ERR_SCRATCH_LIMIT, need, kNoAllocScratchBytes);

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return fail(RB_ERR_CUDA, 0, 0, e);
    uint8_t* base;
    {
        // set-up, once per device (and context): the array's device address
        unsigned long long ctx = 0;
        const bool have_ctx = current_context_id(&ctx);
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        NoAllocAddr& s = g_noalloc_addr[dev];
        if (!s.ptr || !have_ctx || s.ctx != ctx) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) return fail(RB_ERR_CUDA, 0, 0, e);
            s.ptr = p;
            // without a context id the lookup is simply repeated on every call
            if (!have_ctx) current_context_id(&ctx);
            s.ctx = ctx;
        }
        base = static_cast<uint8_t*>(s.ptr);
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t* status = reinterpret_cast<uint32_t*>(base);
    e = cudaMemsetAsync(status, 0, sizeof(uint32_t), st);  // the previous call's word is stale
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, 0, 0, e);

    if (k == 0 || alpha == 0.0) {
        e = launch_scale_c<double>(static_cast<int>(cm), static_cast<int>(cn), beta, c, ldc, st);
    } else {
        const int M = static_cast<int>(cm), N = static_cast<int>(cn), K = static_cast<int>(k);
        const size_t exps = round_up((cm + cn) * sizeof(int), 256);
        const size_t pa = cm * kp, pb = cn * kp;
        int* ea = reinterpret_cast<int*>(base + 256);
        int* eb = ea + cm;
        int8_t* sla = reinterpret_cast<int8_t*>(base + 256 + exps);
        int8_t* slb = sla + round_up(slices * pa, 256);
        size_t ars, aps, brs, bps;
        operand_views(cta, ctb, clda, cldb, ars, aps, brs, bps);
        launch_ozaki_prepass(OzPair{{{ca, ars, aps, 0, M, K, ea, sla, kp, pa, 0, 0, 0, 0},
                                     {cb, brs, bps, 0, N, K, eb, slb, kp, pb, 0, 0, 0, 0}}},
                             slices, st);
        CUtensorMap tma, tmb;
        CUresult r = make_tmap_planes(&tma, sla, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, M, slices, kp, kUM);
        if (r == CUDA_SUCCESS) r = make_tmap_planes(&tmb, slb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, K, N, slices, kp, 256);
        if (r != CUDA_SUCCESS) return fail(RB_ERR_CUDA, 0, 0, static_cast<int32_t>(r));
        OzParams p{};
        p.m = M; p.n = N; p.k = K;
        p.un = 256;  // always the wide tile, and never the split tail: its scratch is sized for that
        p.tiles_m = (M + kUM - 1) / kUM;
        p.tiles_n = (N + 255) / 256;
        p.num_tiles = p.tiles_m * p.tiles_n;
        p.num_kt = (K + 127) / 128;
        p.slices = slices;
        const long long max_k = 2147483647LL / (static_cast<long long>(slices) * 128 * 128);
        p.kt_per_chunk = static_cast<int>(max_k / 128) > 0 ? static_cast<int>(max_k / 128) : 1;
        p.kchunks = (p.num_kt + p.kt_per_chunk - 1) / p.kt_per_chunk;
        p.beta_mode = (beta == 0.0) ? 0 : (beta == 1.0 ? 1 : 2);
        p.alpha = alpha; p.beta = beta;
        p.c = c; p.ldc = ldc;
        p.cin = c;
        p.row_exp = ea; p.col_exp = eb;
        p.err = status;
        e = ozaki_kernel_attributes();
        if (e != cudaSuccess) return fail(RB_ERR_CUDA, 0, 0, e);
        int sms = 148;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        ozaki_gemm_kernel<256><<<p.num_tiles < sms ? p.num_tiles : sms, kOzThreads, OzCfg<256>::SMEM, st>>>(
            tma, tmb, p);
        count_launch();
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, 0, 0, e);
    // The call returns once its work has finished, with the kernels' status word read back.
    uint32_t word = 0;
    e = cudaMemcpyAsync(&word, status, sizeof(word), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(RB_ERR_CUDA, 0, 0, e);
    if (word != 0) return fail((word >> 24) == (RB_DEVERR_TIMEOUT >> 24) ? RB_ERR_TIMEOUT : RB_ERR_DEVICE, word);
    return RB_OK;
}

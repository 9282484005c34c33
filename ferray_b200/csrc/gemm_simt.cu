// gemm_simt.cu -- host launchers of the plain FP64 / FP32 / complex GEMMs
// (FP64 pipe and FFMA; see simt_gemm.cuh).
#include "prep_kernels.cuh"
#include "runtime.h"
#include "simt_gemm.cuh"
#include "dmma_gemm.cuh"
#include "ffma_sgemm.cuh"
#include "ffma_tile64.cuh"
#include "tune.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace fgrt {

using namespace fg;

static BatchMap batch_map(const Gemm& g) {
    BatchMap bm{};
    bm.bdims = g.bdims;
    for (int d = 0; d < 4; ++d) {
        bm.bshape[d] = g.bshape[d];
        bm.a_bstride[d] = g.a_istride[d] * g.a_mstride;
        bm.b_bstride[d] = g.b_istride[d] * g.b_mstride;
    }
    bm.c_bstride = g.c_stride;
    return bm;
}

static int grid_for(long long total) {
    return static_cast<int>(std::min<long long>(std::max<long long>((total + 255) / 256, 1), 4096));
}

// Plain real GEMM with the tuned tile variant and split-K count.  Split-K
// writes `splits` partial products into a workspace and a combine pass
// applies alpha / beta (the partial sums are added in split order).
template <typename T, int TMM, int TNN>
static fg_status launch_simt_real(const Gemm& g, BatchMap bm, int splits_want, cudaStream_t st) {
    constexpr int BTM = 16 * TMM, BTN = 16 * TNN;
    constexpr long long KUNIT = 64;  // split granularity in K
    const long long kunits = (g.K + KUNIT - 1) / KUNIT;
    int kps = static_cast<int>(kunits);
    const int splits = plan_splits(splits_want, static_cast<int>(kunits), g.M * g.N * g.batch,
                                   sizeof(T), &kps);
    if ((long long)splits * g.batch > 65535) return set_error(FG_ERR_UNSUPPORTED, "batch above 65535");
    dim3 grid((g.N + BTN - 1) / BTN, (g.M + BTM - 1) / BTM, g.batch * splits);
    const T* A = static_cast<const T*>(g.A);
    const T* B = static_cast<const T*>(g.B);
    if (splits <= 1) {
        simt_gemm_real<T, 8, TMM, TNN><<<grid, 256, 0, st>>>((int)g.M, (int)g.N, (int)g.K, (T)g.alpha_re, A,
                                                       g.lda, B, g.ldb, (T)g.beta_re,
                                                       static_cast<T*>(g.C), g.ldc, bm, g.batch, (int)g.K);
        count_launch();
        FG_CUDA(cudaGetLastError());
        return FG_OK;
    }
    Scratch ws;
    const long long out_elems = g.M * g.N * g.batch;
    FG_TRY(ws.alloc(static_cast<size_t>(splits * out_elems) * sizeof(T), st));
    BatchMap wbm = bm;
    wbm.c_bstride = g.M * g.N;
    simt_gemm_real<T, 8, TMM, TNN><<<grid, 256, 0, st>>>((int)g.M, (int)g.N, (int)g.K, T(1), A, g.lda, B,
                                                   g.ldb, T(0), static_cast<T*>(ws.p), g.N, wbm,
                                                   g.batch, (int)(kps * KUNIT));
    splitk_reduce<T>(static_cast<const T*>(ws.p), splits, g.M, g.N, g.batch, static_cast<T*>(g.C), g.ldc,
        g.c_stride, (T)g.alpha_re, (T)g.beta_re, 0, st);
    count_launch(2);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// Plain DGEMM on the FP64 tensor path (DMMA): accumulation runs of kps * 64 along K,
// `runs` of them one after the other in a CTA and `parts` such ranges of K as CTAs of
// their own, whose sums a second pass combines.
template <class Cfg, bool VEC, bool FOLD>
static fg_status launch_dmma_as(const Gemm& g, BatchMap bm, int runs, int kps, int parts, cudaStream_t st) {
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    auto kernel = dmma_gemm_f64_kernel<Cfg, VEC, FOLD>;
    std::call_once(once, [kernel] {
        attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(Cfg::SMEM));
    });
    FG_CUDA(attr_err);
    if ((long long)parts * g.batch > 65535) return set_error(FG_ERR_UNSUPPORTED, "batch above 65535");
    const int seg = kps * 64 / Cfg::BK;
    dim3 grid((g.N + Cfg::BN - 1) / Cfg::BN, (g.M + Cfg::BM - 1) / Cfg::BM, g.batch * parts);
    const double* A = static_cast<const double*>(g.A);
    const double* B = static_cast<const double*>(g.B);
    if (parts <= 1) {
        kernel<<<grid, Cfg::THREADS, Cfg::SMEM, st>>>(
            (int)g.M, (int)g.N, (int)g.K, g.alpha_re, A, g.lda, B, g.ldb, g.beta_re,
            static_cast<double*>(g.C), g.ldc, bm, g.batch, (int)g.K, seg);
        count_launch();
        FG_CUDA(cudaGetLastError());
        return FG_OK;
    }
    Scratch ws;
    const long long out_elems = g.M * g.N * g.batch;
    FG_TRY(ws.alloc(static_cast<size_t>(parts * out_elems) * sizeof(double), st));
    BatchMap wbm = bm;
    wbm.c_bstride = g.M * g.N;
    kernel<<<grid, Cfg::THREADS, Cfg::SMEM, st>>>(
        (int)g.M, (int)g.N, (int)g.K, 1.0, A, g.lda, B, g.ldb, 0.0, static_cast<double*>(ws.p), g.N, wbm,
        g.batch, runs * kps * 64, seg);
    splitk_reduce<double>(static_cast<const double*>(ws.p), parts, g.M, g.N, g.batch, static_cast<double*>(g.C), g.ldc,
        g.c_stride, g.alpha_re, g.beta_re, 0, st);
    count_launch(2);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

template <class Cfg>
static fg_status launch_dmma_fold(const Gemm& g, BatchMap bm, int runs, int kps, int parts, cudaStream_t st) {
    // 16-byte copies where every row of A and B starts on 16 bytes
    bool vec = g.lda % 2 == 0 && g.ldb % 2 == 0 &&
               ((reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B)) & 15) == 0;
    for (int d = 0; d < 4; ++d) vec = vec && bm.a_bstride[d] % 2 == 0 && bm.b_bstride[d] % 2 == 0;
    if constexpr (Cfg::BM == 64) {
        if (runs > 1)
            return vec ? launch_dmma_as<Cfg, true, true>(g, bm, runs, kps, parts, st)
                       : launch_dmma_as<Cfg, false, true>(g, bm, runs, kps, parts, st);
    }
    return vec ? launch_dmma_as<Cfg, true, false>(g, bm, 1, kps, parts, st)
               : launch_dmma_as<Cfg, false, false>(g, bm, 1, kps, parts, st);
}

// Few rows: 32 x 256 tiles, every run a CTA of its own.
static fg_status launch_dmma_skinny(const Gemm& g, BatchMap bm, int splits_want, cudaStream_t st) {
    const long long kunits = (g.K + 63) / 64;
    int kps = static_cast<int>(kunits);
    const int splits = plan_splits(splits_want, static_cast<int>(kunits), g.M * g.N * g.batch, sizeof(double), &kps);
    return launch_dmma_fold<DmmaSkinnyCfg>(g, bm, 1, kps, splits, st);
}

// Microseconds of a DMMA launch: a unit's FMAs at 64 a cycle of its SM, over the
// share of that rate which the CTAs together on an SM reach (three of 64 x 64 0.87,
// two 0.74, one 0.53; two of 128 x 64 0.85, one 0.53), in groups of as many as fit,
// and the combine pass.  Fitted on a B200 to 12 shapes from 200^3 to 4096 x 4096 x
// 1024 with 1 to 8 parts.
static double dmma_us(int sms, const Gemm& g, bool wide, long long k_part, int parts) {
    static const double share[2][3] = {{0.53, 0.74, 0.87}, {0.53, 0.85, 0.85}};
    const int res = wide ? 2 : 3;
    const long long bm = wide ? 128 : 64;
    const long long units = (g.M + bm - 1) / bm * ((g.N + 63) / 64) * g.batch * parts, n = (units + sms - 1) / sms;
    const double unit = static_cast<double>(bm * k_part) / 1930.0;
    double us = n / res * (res * unit / share[wide][res - 1]);
    if (n % res) us += n % res * unit / share[wide][n % res - 1];
    if (parts > 1) us += 3.0 + (parts + 1.0) * g.M * g.N * g.batch / 1e6;
    return us;
}

// Tile (128 x 64 or 64 x 64) and parts by that model; the accumulation runs are the
// tuned split's, so results do not depend on the choice beyond the order in which
// the runs' sums are added.  Against 128 x 128 tiles with every run a CTA of its own
// (us): 768^3 74 -> 42, 1024^3 99 -> 90, 2048^3 670 -> 560, 4096 x 4096 x 1024 1194
// -> 1088, 300 x 700 x 2000 92 -> 49, 1201 x 333 x 999 95 -> 55.
// forced: a chosen variant of the table, 128 x 64 with `splits_want` parts.
static fg_status launch_dmma(fg_ctx* ctx, const Gemm& g, BatchMap bm, int splits_want, bool forced, cudaStream_t st) {
    const long long kunits = (g.K + 63) / 64;
    int kps = static_cast<int>(kunits);
    const int splits = plan_splits(splits_want, static_cast<int>(kunits), g.M * g.N * g.batch,
                                   sizeof(double), &kps);
    bool wide = true;
    int parts = splits;
    if (!forced) {
        double best = 1e30;
        for (int runs = splits; runs >= 1; --runs) {
            const int p = (splits + runs - 1) / runs;
            if (runs > 1 && p == (splits + runs - 2) / (runs - 1)) continue;  // fewer runs a part do as well
            const long long k_part = std::min<long long>(g.K, (long long)runs * kps * 64);
            for (int w = 0; w < 2; ++w) {
                // 128 x 64 with two sums an output would spill; 64 rows a tile have to
                // fit the grid
                if (w ? runs > 1 : (g.M + 63) / 64 > 65535) continue;
                const double us = dmma_us(ctx->sm_count, g, w != 0, k_part, p);
                if (us < best) {
                    best = us;
                    wide = w != 0;
                    parts = p;
                }
            }
        }
    }
    const int runs = (splits + parts - 1) / parts;
    return wide ? launch_dmma_fold<DmmaCfg>(g, bm, runs, kps, parts, st)
                : launch_dmma_fold<DmmaCfg64>(g, bm, runs, kps, parts, st);
}

// ---- plain SGEMM on the cp.async FFMA kernel (ffma_sgemm.cuh)
//
// Which tile and split-K count a shape takes.  The per-output order does not
// depend on the tile, so this is about time alone; it is a model of the kernel
// rather than a table by size bucket, because how full the last wave is
// changes between two buckets.  A CTA alone on an SM runs at its latency-bound
// rate, CTAs together share the SM's rate for that tile; the grid runs in
// waves of occupancy x SMs, the last one spread evenly; two-warp CTAs fill the
// four schedulers in pairs (an odd number of them takes the time of the next
// even one); splits add the combine pass.  Rates and constants are a fit to
// 1100 runs on a B200 (1.965 GHz; 7 tiles x 10 split counts over 21 shapes from
// 256^3 to 4096^3 and 8 to 64 rows of 8192 x 8192): residual 7 %, and the
// choice is within 6 % of the best of those runs for every shape, 1 % on
// average.
struct FfmaTileInfo {
    int bm, bn, occ;
    bool pairs;           // two-warp CTAs
    double alone, most;   // GFLOP/s of an SM: one CTA, many
};
using FfmaT0 = FfmaTile<128, 128, 16, 8, 2, 0>;
using FfmaT1 = FfmaTile<64, 128, 16, 8, 4, 0>;
using FfmaT2 = FfmaTile<64, 64, 8, 8, 6, 4>;
using FfmaT3 = FfmaTile<64, 64, 4, 8, 4, 4>;
using FfmaT4 = FfmaTile<32, 128, 8, 8, 5, 4>;
using FfmaT5 = FfmaTile<32, 64, 4, 8, 8, 4>;
using FfmaT6 = FfmaTile<16, 128, 4, 8, 6, 0>;
constexpr int FFMA_TILES = 7;
constexpr FfmaTileInfo kFfmaTiles[FFMA_TILES] = {
    {128, 128, 2, false, 425, 440}, {64, 128, 4, true, 230, 428}, {64, 64, 6, true, 220, 415},
    {64, 64, 4, false, 308, 360},   {32, 128, 5, true, 185, 390}, {32, 64, 8, true, 185, 349},
    {16, 128, 6, true, 185, 339},
};

// K units of 64 per accumulator when the shape is split `want` ways.
static int chain_units(const Gemm& g, int want) {
    int kps = 0;
    plan_splits(want, static_cast<int>((g.K + 63) / 64), g.M * g.N * g.batch, sizeof(float), &kps);
    return kps;
}

struct FfmaChoice {
    int tile, splits;
    double us;
};

// fixed_splits > 0: that split count; only_tile >= 0: that tile.  max_chain: the
// longest run of k that one accumulator may take (64-deep units): the size
// table's split count also bounds the rounding error, which grows with the square
// root of that run, so the model may split further than the table, never less.
// us stays 1e300 where the grid's z extent (65535) leaves no such split.
static FfmaChoice ffma_plan(int sms, long long M, long long N, long long K, long long batch, int fixed_splits,
                            int only_tile, int max_chain) {
    FfmaChoice best{std::max(only_tile, 0), std::max(fixed_splits, 1), 1e300};
    const long long ku = (K + 63) / 64;
    for (int s = fixed_splits > 0 ? fixed_splits : 1;; ++s) {
        int kps = 0;
        const int ns = plan_splits(s, static_cast<int>(ku), M * N * batch, sizeof(float), &kps);
        if (fixed_splits > 0 || (ns == s && kps <= max_chain && ns * batch <= 65535)) {
            const double kk = static_cast<double>(std::min<long long>(K, 64LL * kps));
            const double combine = ns > 1 ? 3.0 + (2.0 * ns + 1) * M * N * 4 * batch / 5.0e6 : 0.0;
            for (int t = 0; t < FFMA_TILES; ++t) {
                if (only_tile >= 0 && t != only_tile) continue;
                const FfmaTileInfo& f = kFfmaTiles[t];
                if ((M + f.bm - 1) / f.bm > 65535) continue;  // the grid's y extent
                const double work = 2.0 * f.bm * f.bn * kk / 1e3;  // us at 1 GFLOP/s
                auto dur = [&](long long c) {
                    if (f.pairs) c = (c + 1) / 2 * 2;
                    const double a = c * f.alone / f.most, a2 = a * a;
                    const double rate = f.most * a / std::sqrt(std::sqrt(1.0 + a2 * a2));
                    return c * work / rate + 0.3;
                };
                const long long units = (M + f.bm - 1) / f.bm * ((N + f.bn - 1) / f.bn) * ns * batch;
                const long long slots = (long long)sms * f.occ, rem = units % slots;
                double us = (units / slots) * dur(f.occ) + (rem ? dur((rem + sms - 1) / sms) : 0.0);
                us = std::max(us, (M * K + K * N) * 4.0 * batch / 5.8e6) + 4.9 + combine;
                if (us < best.us) best = FfmaChoice{t, ns, us};
            }
        }
        if (fixed_splits > 0 || s >= TUNE_MAX_SPLITS || s >= ku) break;
    }
    return best;
}

// The packed transpose wants a K grid below 65536 blocks of 64, the kernel a row
// grid below 65536 blocks: of 128 rows, the planner leaves out the tiles that are
// lower than M needs (2 M x 256 x 256: 4.9 ms, 7.4 register-staged; 1050000 x 160 x
// 144: 1.25 against 2.10).
static bool ffma_ok(long long M, long long K) { return K <= 32LL * 65535 && M <= 128LL * 65535; }
static bool ffma_ok(const Gemm& g) { return ffma_ok(g.M, g.K); }

// One launch: At packed, B in place, into C or (splits > 1) into partials.
template <class Cfg>
static fg_status launch_ffma_tile(const Gemm& g, const float* At, long long ldat, const BatchMap& bm, int splits,
                                  int ksplit, float alpha, float beta, float* C, long long ldc, cudaStream_t st) {
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        attr_err = cudaFuncSetAttribute(ffma_sgemm_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(Cfg::SMEM));
    });
    FG_CUDA(attr_err);
    dim3 grid(static_cast<unsigned>((g.N + Cfg::BN - 1) / Cfg::BN), static_cast<unsigned>((g.M + Cfg::BM - 1) / Cfg::BM),
              static_cast<unsigned>(g.batch * splits));
    ffma_sgemm_kernel<Cfg><<<grid, Cfg::THREADS, Cfg::SMEM, st>>>(
        (int)g.M, (int)g.N, (int)g.K, alpha, At, ldat, static_cast<const float*>(g.B), g.ldb, beta, C, ldc, bm, g.batch,
        ksplit);
    count_launch();
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

template <class T>
struct FfmaShifted;  // the same tile with B rows at any alignment
template <int BM, int BN, int TM, int TN, int MINB, int BPAD>
struct FfmaShifted<FfmaTile<BM, BN, TM, TN, MINB, BPAD, false>> {
    using type = FfmaTile<BM, BN, TM, TN, MINB, BPAD, true>;
};

// Every row of every one of these f32 matrices starts on 16 bytes.
static bool rows16(const void* X, long long ld, long long count, long long mstride) {
    return (reinterpret_cast<uintptr_t>(X) & 15) == 0 && ld % 4 == 0 && (count == 1 || mstride % 4 == 0);
}

// Deep problems that the table (tuned with the slower kernel this family replaced)
// still gives a register-staged tile: does the packed kernel pay for its transpose of
// A?  From 630 shapes of 33 to 30000 rows, 2 to 1000 columns and K from 1100 to 12000
// (us, register-staged / packed):
//  * not for up to K = 1024 (279 x 195 x 802 17 / 21);
//  * with enough outputs to fill the chip, unless they are a few columns, where the
//    copy of A is most of the work: 33 x 7000 x 1100 41 / 26, 3000 x 64 x 2000 37 /
//    28, but 7000 x 9 x 3000 81 / 101, 1000 x 64 x 2000 21 / 23;
//  * with few outputs where K is long and B comes in whole granules: 300 x 100 x
//    6000 39 / 33, 64 x 20 x 12000 47 / 37, 2 x 20 x 3000 18.5 / 16.5, but 300 x 33 x 6000
//    28 / 31;
//  * few rows of a wide B: 17 x 1000 x 3000 1.18 x;
//  * where the table's 64 x 64 tiles times its splits just pass one wave: 220 x 130
//    x 3365 29 / 25 (220 x 65 x 3365 22 / 25).
static bool packed_pays(int sms, const Gemm& g, TuneChoice table) {
    if (g.K <= 1024) return false;
    if (g.N > 32 && g.M * g.N >= 90000) return true;
    if (g.K >= (g.M <= 32 ? 3000 : 6000) && g.M <= 1000 && rows16(g.B, g.ldb, 1, 0)) return true;
    if (table.variant == 2 && g.N >= 1000) return true;
    int kps = 0;
    const int splits = plan_splits(table.splits, static_cast<int>((g.K + 63) / 64), g.M * g.N, sizeof(float), &kps);
    return table.variant == 1 && g.K > 3000 && g.N >= 100 && (g.M + 63) / 64 * ((g.N + 63) / 64) * splits > sms;
}

// A transposed into packed scratch, B in place, same split-K scheme as
// launch_simt_real.  Results are bit-identical to simt_gemm_real<float, 8, 8, 8>
// at equal split count.
// `table`: the tuned choice for the shape (its split count fixed when forced).
// no_room(): what to do without memory for A's copy or the partial products.
// family: the name it is profiled under (null: the caller's).
template <class NoRoom>
static fg_status launch_ffma(fg_ctx* ctx, const Gemm& g, TuneChoice table, int only_tile, cudaStream_t st,
                             NoRoom no_room, const char* family = "ffma_sgemm") {
    const long long M = g.M, N = g.N, K = g.K;
    const long long Mp = (M + 3) / 4 * 4;
    const FfmaChoice c = ffma_plan(ctx->sm_count, M, N, K, g.batch, tune_forced(TUNE_F32) ? table.splits : 0, only_tile,
                                   chain_units(g, table.splits));
    const int kunits = static_cast<int>((K + 63) / 64);
    int kps = kunits;
    int splits = plan_splits(c.splits, kunits, M * N * g.batch, sizeof(float), &kps);
    if ((long long)splits * g.batch > 65535) return set_error(FG_ERR_UNSUPPORTED, "batch above 65535");
    Scratch sa, ws;
    if (!sa.try_alloc(static_cast<size_t>(g.a_count * K * Mp) * sizeof(float), st)) return no_room();
    // before the next allocation, which the device then does not wait for (32 x 8192 x 8192:
    // the call 119 us, 121 after it)
    ProfScope prof(family, st);
    float* At = static_cast<float*>(sa.p);
    transpose_pack_kernel<<<dim3(static_cast<unsigned>((Mp + 63) / 64), static_cast<unsigned>((K + 63) / 64),
                                 static_cast<unsigned>(g.a_count)),
                            256, 0, st>>>(static_cast<const float*>(g.A), (int)M, (int)K, g.lda, g.a_mstride, At, Mp);
    count_launch();
    if (splits > 1 && !ws.try_alloc(static_cast<size_t>(splits * M * N * g.batch) * sizeof(float), st)) {
        // the table's own split count keeps the length of an accumulation run too
        const int fewer = plan_splits(table.splits, kunits, M * N * g.batch, sizeof(float), &kps);
        const bool room = fewer < splits &&
                          (fewer == 1 || ws.try_alloc(static_cast<size_t>(fewer * M * N * g.batch) * sizeof(float), st));
        if (!room) {
            prof.drop();
            return no_room();
        }
        splits = fewer;
    }
    BatchMap bm = batch_map(g);
    for (int d = 0; d < 4; ++d) bm.a_bstride[d] = g.a_istride[d] * K * Mp;
    float* C = static_cast<float*>(g.C);
    long long ldc = g.ldc;
    float alpha = static_cast<float>(g.alpha_re), beta = static_cast<float>(g.beta_re);
    if (splits > 1) {
        C = static_cast<float*>(ws.p);
        ldc = N;
        bm.c_bstride = M * N;
        alpha = 1.f;
        beta = 0.f;
    }
    const int ksplit = splits > 1 ? kps * 64 : static_cast<int>(K);
    const bool aligned = rows16(g.B, g.ldb, g.b_count, g.b_mstride);
    auto run = [&](auto tile) {
        using T = decltype(tile);
        if (aligned) return launch_ffma_tile<T>(g, At, Mp, bm, splits, ksplit, alpha, beta, C, ldc, st);
        return launch_ffma_tile<typename FfmaShifted<T>::type>(g, At, Mp, bm, splits, ksplit, alpha, beta, C, ldc, st);
    };
    fg_status s = FG_OK;
    switch (c.tile) {
        case 0: s = run(FfmaT0{}); break;
        case 1: s = run(FfmaT1{}); break;
        case 2: s = run(FfmaT2{}); break;
        case 3: s = run(FfmaT3{}); break;
        case 4: s = run(FfmaT4{}); break;
        case 5: s = run(FfmaT5{}); break;
        default: s = run(FfmaT6{}); break;
    }
    if (s != FG_OK || splits == 1) return s;
    splitk_reduce<float>(C, splits, M, N, g.batch, static_cast<float*>(g.C), g.ldc, g.c_stride, (float)g.alpha_re, (float)g.beta_re, 0, st);
    count_launch();
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

static fg_status ffma_oom() { return set_error(FG_ERR_OOM, "no memory for the packed copy of A or the partial products"); }

// Time of a stack by launch_tile64: a 16-deep K block takes 2.25 us with six CTAs
// on an SM, 1 us alone, less where tiles have half the rows or columns (fit to
// 512^3 x 16, 256^3 x 64, 1024 x 1024 x 256 x 4 and 300 x 700 x 2000 x 3, within 16 %).
static double tile64_us(int sms, const Gemm& g) {
    const long long tm = (g.M + 63) / 64, tn = (g.N + 63) / 64, units = tm * tn * g.batch, slots = 6LL * sms;
    const double whole = static_cast<double>((g.M + 31) / 32 * ((g.N + 31) / 32)) / (4 * tm * tn);
    const long long last = (units % slots + sms - 1) / sms;
    return 4.9 + (g.K + 15) / 16 * whole * (2.25 * (units / slots) + (last ? 0.75 + 0.25 * last : 0.0));
}

// Stacks of small problems: one CTA of 64 threads per 64 x 64 tile.  Where the
// tuned table splits K (the shape's latency, for one matrix), the kernel closes an
// accumulator at the same places, so the rounding stays that of the split.
static fg_status launch_tile64(const Gemm& g, const BatchMap& bm, TuneChoice table, cudaStream_t st) {
    const long long tn = (g.N + 63) / 64, tm = (g.M + 63) / 64;
    const Tile64Args a{(int)g.M, (int)g.N, (int)g.K, static_cast<const float*>(g.A), static_cast<const float*>(g.B),
                       static_cast<float*>(g.C), g.lda, g.ldb, g.ldc, (float)g.alpha_re, (float)g.beta_re};
    const int chain = 4 * chain_units(g, table.splits);  // 16-deep K blocks
    const bool vec = rows16(g.A, g.lda, g.a_count, g.a_mstride) && rows16(g.B, g.ldb, g.b_count, g.b_mstride);
    const bool tall = tm > tn;
    const long long longer = std::max(tm, tn), gy = std::min<long long>(longer, 65535), chunks = (longer + gy - 1) / gy;
    const long long gz = std::min(tm, tn) * chunks;
    if (gz > 65535) return set_error(FG_ERR_UNSUPPORTED, "stacked matrix of too many tiles");
    const dim3 grid(static_cast<unsigned>(g.batch), static_cast<unsigned>(gy), static_cast<unsigned>(gz));
    auto kernel = vec ? sgemm_tile64_kernel<true> : sgemm_tile64_kernel<false>;
    kernel<<<grid, 64, 0, st>>>(a, bm, tall, static_cast<int>(longer), static_cast<int>(chunks), chain);
    count_launch();
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// Matrix-vector shapes (one operand is a vector; ferray's matmul of a 1-D
// operand, products/mod.rs:362-437) go to the GEMV kernels.
template <typename T>
static fg_status launch_gemv(fg_ctx* ctx, const Gemm& g, cudaStream_t st) {
    const T* A = static_cast<const T*>(g.A);
    const T* B = static_cast<const T*>(g.B);
    T* C = static_cast<T*>(g.C);
    if (g.N == 1) {
        const long long blocks = (g.M * 32 + 255) / 256;
        gemv_rows_kernel<T><<<static_cast<unsigned>(blocks), 256, 0, st>>>(
            (int)g.M, (int)g.K, (T)g.alpha_re, A, g.lda, B, g.ldb, (T)g.beta_re, C, g.ldc);
        count_launch();
        FG_CUDA(cudaGetLastError());
        return FG_OK;
    }
    constexpr int CW = 32 * (16 / sizeof(T));
    const long long cblocks = (g.N + CW - 1) / CW;
    // split K across blocks until there are about 4 blocks per SM
    int splits = static_cast<int>(std::min<long long>(
        std::max<long long>(1, (4LL * ctx->sm_count) / cblocks), std::max<long long>(1, g.K / 256)));
    splits = std::min(splits, 64);
    const int ksplit = static_cast<int>((g.K + splits - 1) / splits);
    splits = static_cast<int>((g.K + ksplit - 1) / ksplit);
    dim3 grid(static_cast<unsigned>(cblocks), static_cast<unsigned>(splits));
    if (splits == 1) {
        gemv_cols_kernel<T><<<grid, 256, 0, st>>>((int)g.N, (int)g.K, ksplit, (T)g.alpha_re, A, 1, B,
                                                  g.ldb, (T)g.beta_re, C, 0);
        count_launch();
        FG_CUDA(cudaGetLastError());
        return FG_OK;
    }
    Scratch ws;
    FG_TRY(ws.alloc(static_cast<size_t>(splits * g.N) * sizeof(T), st));
    gemv_cols_kernel<T><<<grid, 256, 0, st>>>((int)g.N, (int)g.K, ksplit, (T)g.alpha_re, A, 1, B, g.ldb,
                                              (T)g.beta_re, static_cast<T*>(ws.p), g.N);
    splitk_reduce<T>(static_cast<const T*>(ws.p), splits, 1, g.N, 1,
                                                           C, g.ldc, 0, (T)g.alpha_re, (T)g.beta_re, 0, st);
    count_launch(2);
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

// A plain DGEMM that leaves the table's variant for the small DMMA tiles.
static bool small_dmma(int sms, const Gemm& g, const TuneChoice& c) {
    if (c.variant == 5) return g.batch > 1 && g.N < 512;
    if (c.variant == 1 && g.batch > 1 && g.K <= 24) {
        // two short K blocks: not where the last wave of 64 x 64 tiles, three an SM, is
        // mostly empty (40 x 300 x 300 x 16 16.5 us register-staged, 18.5 so; 100 x 128 x
        // 128 x 24 12.3, 10.3 so)
        const long long units = (g.M + 63) / 64 * ((g.N + 63) / 64) * g.batch, slots = 3LL * sms;
        if (5 * units < 4 * ((units + slots - 1) / slots) * slots) return false;
    }
    return c.variant < 4 && g.K > (g.batch > 1 ? 8 : 16);
}

fg_status launch_simt(fg_ctx* ctx, const Gemm& g, cudaStream_t st) {
    if (g.batch == 1 && (g.N == 1 || g.M == 1) && (g.dtype == FG_F64 || g.dtype == FG_F32)) {
        ProfScope prof(g.dtype == FG_F64 ? "gemv_f64" : "gemv_f32", st);
        return g.dtype == FG_F64 ? launch_gemv<double>(ctx, g, st) : launch_gemv<float>(ctx, g, st);
    }
    const BatchMap bm = batch_map(g);
    if (g.batch > 65535) return set_error(FG_ERR_UNSUPPORTED, "batch above 65535");
    // each launch profiled under the kernel that runs
    auto named = [st](const char* family, auto launch) {
        ProfScope prof(family, st);
        return launch();
    };
    switch (g.dtype) {
        case FG_F64: {
            const TuneChoice c = tune_lookup(TUNE_F64, g.M, g.N, g.K);
            const bool forced = tune_forced(TUNE_F64);
            // The register-staged tiles (0..3) only where they are chosen by hand: the
            // small DMMA tiles do as well or better wherever the table (tuned with the
            // 128 x 128 one) has them (100^3 15.6 -> 11.2 us, 400 x 300 x 100 17.9 ->
            // 10.0, 500 x 120 x 900 20 -> 15, stacks of 128^3 x 100 51 -> 23, 250^3 x 16
            // 59 -> 28, 33 x 65 x 129 x 500 101 -> 56).
            // Outer products of up to 16 (one K block; in stacks 8) stay: 1000 x 1000 x 8
            // 5.9 against 7.3 us, 128 x 128 x 8 x 100 8.4 against 8.9.  Stacks of few rows and less than two 32 x 256 tiles too
            // (16^3 x 1000 18.6 -> 11.8, 10 x 300 x 300 x 8 18 -> 13; but 8 x 1000 x 1000
            // x 4 24.6 against 28.6).
            if (c.variant == 4 || (!forced && small_dmma(ctx->sm_count, g, c)))
                return named("dmma_dgemm", [&] { return launch_dmma(ctx, g, bm, c.splits, forced, st); });
            if (c.variant == 5)
                return named("dmma_dgemm_skinny", [&] { return launch_dmma_skinny(g, bm, c.splits, st); });
            return named("simt_dgemm", [&] {
                switch (c.variant) {
                    case 1: return launch_simt_real<double, 4, 4>(g, bm, c.splits, st);
                    case 2: return launch_simt_real<double, 2, 8>(g, bm, c.splits, st);
                    case 3: return launch_simt_real<double, 8, 2>(g, bm, c.splits, st);
                    default: return launch_simt_real<double, 8, 8>(g, bm, c.splits, st);
                }
            });
        }
        case FG_F32: {
            const TuneChoice c = tune_lookup(TUNE_F32, g.M, g.N, g.K);
            const bool forced = tune_forced(TUNE_F32);  // else ffma_plan's splits and tile
            // Stacks: one CTA of 64 threads per tile or the packed kernel,
            // whichever its model puts first (96 x 80 x 64 x 512: 22 us against 33,
            // 47 register-staged; 300 x 700 x 2000 x 3: 135 against 70), unless there
            // are fewer tiles than SMs, or with a K of one or two blocks than twice
            // the SMs, where 256 threads a tile have the shorter latency (191 x 37 x 44 x
            // 32: 5.9 us, 8.3 with 64; 826 x 157 x 17 x 6 6.2, 8.2).
            const long long stack_tiles = (g.M + 63) / 64 * ((g.N + 63) / 64) * g.batch;
            if (!forced && g.batch > 1 && stack_tiles > (g.K <= 24 ? 2 : 1) * ctx->sm_count) {
                const double packed = 4.0 + ffma_plan(ctx->sm_count, g.M, g.N, g.K, g.batch, 0, -1, chain_units(g, c.splits)).us;
                auto tile64 = [&] { return named("sgemm_tile64", [&] { return launch_tile64(g, bm, c, st); }); };
                if (!ffma_ok(g) || tile64_us(ctx->sm_count, g) < packed) return tile64();
                return launch_ffma(ctx, g, c, -1, st, tile64);
            }
            auto staged = [&] {
                return named("simt_sgemm", [&] {
                    switch (c.variant) {
                        case 1: return launch_simt_real<float, 4, 4>(g, bm, c.splits, st);
                        case 2: case 5: return launch_simt_real<float, 2, 8>(g, bm, c.splits, st);
                        case 3: return launch_simt_real<float, 8, 2>(g, bm, c.splits, st);
                        default: return launch_simt_real<float, 8, 8>(g, bm, c.splits, st);
                    }
                });
            };
            if (!forced && c.variant < 4 && g.batch == 1 && ffma_ok(g) && packed_pays(ctx->sm_count, g, c))
                return launch_ffma(ctx, g, c, -1, st, staged);  // A's copy may not fit: those tiles need none
            if (c.variant >= 4 && ffma_ok(g)) return launch_ffma(ctx, g, c, forced && c.variant == 5 ? 4 : -1, st, ffma_oom);
            return staged();
        }
        case FG_C64: {
            ProfScope prof("simt_zgemm", st);
            // Real scalars and one output matrix: the real-embedded GEMM on
            // the DMMA kernel (same 8MNK flops, FP64 FMA per product).
            if (g.batch == 1 && g.alpha_im == 0.0 && g.beta_im == 0.0 && g.K > 0 &&
                (reinterpret_cast<uintptr_t>(g.B) & 15) == 0) {  // 16-byte complex loads of B
                Scratch bx;
                FG_TRY(bx.alloc(static_cast<size_t>(4 * g.K * g.N) * sizeof(double), st));
                zgemm_expand_b_kernel<<<grid_for(g.K * g.N), 256, 0, st>>>(
                    static_cast<const double2*>(g.B), g.K, g.N, g.ldb, static_cast<double*>(bx.p));
                count_launch();
                Gemm r = g;
                r.dtype = FG_F64;
                r.M = g.M;
                r.N = 2 * g.N;
                r.K = 2 * g.K;
                r.lda = 2 * g.lda;
                r.B = bx.p;
                r.ldb = 2 * g.N;
                r.ldc = 2 * g.ldc;
                const TuneChoice c = tune_lookup(TUNE_F64, r.M, r.N, r.K);
                return launch_dmma(ctx, r, batch_map(r), c.variant == 4 ? c.splits : 1, false, st);
            }
            dim3 grid((g.N + 63) / 64, (g.M + 63) / 64, g.batch);
            simt_gemm_cplx<double, 8><<<grid, 256, 0, st>>>(
                (int)g.M, (int)g.N, (int)g.K, g.alpha_re, g.alpha_im,
                static_cast<const Cplx<double>*>(g.A), g.lda, static_cast<const Cplx<double>*>(g.B),
                g.ldb, g.beta_re, g.beta_im, static_cast<Cplx<double>*>(g.C), g.ldc, bm);
            break;
        }
        case FG_C32: {
            ProfScope prof("simt_cgemm", st);
            // Real scalars, one output matrix and a tuned f32 choice of the
            // cp.async FFMA kernel for the embedded shape: the real-embedded
            // GEMM (M x 2K) (2K x 2N) on it (same 8MNK flops, one FMA per
            // product); otherwise the 4M kernel.
            if (g.batch == 1 && g.alpha_im == 0.0 && g.beta_im == 0.0 && g.M > 0 && g.N > 0 && g.K > 0 &&
                ffma_ok(g.M, 2 * g.K) && (reinterpret_cast<uintptr_t>(g.B) & 7) == 0) {
                const TuneChoice c = tune_lookup(TUNE_F32, g.M, 2 * g.N, 2 * g.K);
                if (c.variant == 4) {
                    Scratch bx;
                    FG_TRY(bx.alloc(static_cast<size_t>(4 * g.K * g.N) * sizeof(float), st));
                    cgemm_expand_b_kernel<<<grid_for(g.K * g.N), 256, 0, st>>>(
                        static_cast<const float2*>(g.B), g.K, g.N, g.ldb, static_cast<float*>(bx.p));
                    count_launch();
                    Gemm r = g;
                    r.dtype = FG_F32;
                    r.N = 2 * g.N;
                    r.K = 2 * g.K;
                    r.lda = 2 * g.lda;
                    r.B = bx.p;
                    r.ldb = 2 * g.N;
                    r.ldc = 2 * g.ldc;
                    return launch_ffma(ctx, r, c, -1, st, ffma_oom, nullptr);
                }
            }
            dim3 grid((g.N + 63) / 64, (g.M + 63) / 64, g.batch);
            simt_gemm_cplx<float, 8><<<grid, 256, 0, st>>>(
                (int)g.M, (int)g.N, (int)g.K, (float)g.alpha_re, (float)g.alpha_im,
                static_cast<const Cplx<float>*>(g.A), g.lda, static_cast<const Cplx<float>*>(g.B),
                g.ldb, (float)g.beta_re, (float)g.beta_im, static_cast<Cplx<float>*>(g.C), g.ldc, bm);
            break;
        }
        default:
            return set_error(FG_ERR_DTYPE, "SIMT path handles f64/f32/c64/c32 only");
    }
    count_launch();
    FG_CUDA(cudaGetLastError());
    return FG_OK;
}

}  // namespace fgrt

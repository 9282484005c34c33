// ffma_tile64.cuh -- one 64 x 64 tile of a plain SGEMM by a CTA of 64 threads,
// for many small problems at once (ragged batches, stacked matmul).
//
// Each thread accumulates 8 x 8 outputs, one FP32 fused multiply-add per
// product with k ascending (the per-output order of simt_gemm_real), issued in
// pairs of adjacent columns (ffma2, ffma_sgemm.cuh).  What bounds small
// problems is work done for padding and the latency of a short K loop:
//  * a thread's rows and columns lie in two halves 32 apart, and a tile whose
//    problem ends in its first 32 rows or columns runs a loop without the other
//    half, so padding is to 32 while whole tiles keep the 8 x 8 register tile
//    (a 4 x 4 one reaches 46 TFLOP/s of FMAs on registers, 8 x 8 60);
//  * operands pass through registers one 16-deep K block ahead, A landing
//    transposed in shared memory, in 4-byte loads that need no alignment (small
//    problems have odd leading dimensions as often as not); where all rows are
//    16-byte aligned A takes 16-byte loads and B cp.async (512 stacked 96 x 80 x
//    64 products: 22 us, against 37 with 4-byte loads);
//  * the K loop is unrolled 8 deep, not over the whole block: with 16 the four
//    loops of the kernel outgrow the instruction cache (ragged batch of 4096:
//    753 us, 504 with 8).
// Six such CTAs per SM hide each other's latency (8 deep K blocks with eight CTAs
// of 128 registers: 559 us).
#pragma once
#include "ffma_sgemm.cuh"

namespace fg {

struct Tile64Smem {
    alignas(16) float a[2][16][68];  // [k][m]; the pitch keeps 16-byte reads aligned
    alignas(16) float b[2][16][64];
};

struct Tile64Args {
    int M, N, K;
    const float* A;
    const float* B;
    float* C;
    long long lda, ldb, ldc;
    float alpha, beta;
};

// Sums of the closed accumulators of a tile, each thread its own.
struct Tile64Totals {
    float4 x[16][64];
};

// Adds the accumulators to the totals (sets them the first time) and clears
// them, or on the last call leaves the sum in them.
template <int RH, int CH>
__device__ __forceinline__ void tile64_fold(uint64_t (&acc)[8][4], Tile64Totals& tot, bool first, bool more) {
#pragma unroll
    for (int i = 0; i < RH * 4; ++i)
#pragma unroll
        for (int h = 0; h < CH; ++h) {
            float4& t = tot.x[i * 2 + h][threadIdx.x];
            const float2 u = unpack2(acc[i][2 * h]), w = unpack2(acc[i][2 * h + 1]);
            float4 v = make_float4(u.x, u.y, w.x, w.y);
            if (!first) {
                const float4 o = t;
                v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
            }
            if (more) {
                t = v;
                acc[i][2 * h] = acc[i][2 * h + 1] = 0;
            } else {
                acc[i][2 * h] = pack2(v.x, v.y);
                acc[i][2 * h + 1] = pack2(v.z, v.w);
            }
        }
}

// acc over all of K for RH row halves and CH column halves.  VEC: rows of A and
// B are 16-byte aligned; A comes in 16-byte loads, B by 16-byte cp.async.
template <int RH, int CH, bool VEC, bool FOLD, class Last>
__device__ __forceinline__ void tile64_loop(const Tile64Args& p, int m0, int n0, Tile64Smem& s,
                                            uint64_t (&acc)[8][4], Last last, Tile64Totals* tot, int chain) {
    constexpr int BK = 16, T = 64, U = 8;
    const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;
    // A, 4-byte: 8 k of 8 rows per step of 64 threads, the two k halves of the
    // block in turn (a warp's transposed stores then meet 32 different banks);
    // 16-byte: 16 k of 16 rows.  B, 4-byte: one or two k rows per step.
    constexpr int AN = RH * 8;  // floats of A a thread loads per K block
    constexpr int BW = CH * 32, BR = T / BW, BN = BK / BR;
    const int ar = VEC ? tid / 4 : tid / 8, ak = VEC ? tid % 4 * 4 : tid % 8;
    const int bk = VEC ? tid / (BW / 4) : tid / BW, bn = VEC ? tid % (BW / 4) * 4 : tid % BW;
    const float* pa = p.A + (long long)(m0 + ar) * p.lda + ak;
    const float* pb = p.B + (long long)bk * p.ldb + n0 + bn;
    const long long sa = (VEC ? 16 : 8) * p.lda, sb = BR * (VEC ? 4 : 1) * p.ldb;
    const int rows = p.M - m0 - ar;  // row ar + j exists: j < rows
    const int cols = p.N - n0 - bn;
    float ra[AN], rb[VEC ? 1 : BN];
    auto load = [&](int k0, int buf) {
        const float* q = pa + k0;
        const float* u = pb + k0 * p.ldb;
        if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < AN / 4; ++i) {
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (16 * i < rows) {
                    const int left = p.K - k0 - ak;
                    if (left >= 4) {
                        v = __ldg(reinterpret_cast<const float4*>(q));
                    } else {
                        if (left > 0) v.x = __ldg(q);
                        if (left > 1) v.y = __ldg(q + 1);
                        if (left > 2) v.z = __ldg(q + 2);
                    }
                }
                ra[4 * i] = v.x; ra[4 * i + 1] = v.y; ra[4 * i + 2] = v.z; ra[4 * i + 3] = v.w;
                q += sa;
            }
            constexpr int KS = BR * 4;  // k rows per step
#pragma unroll
            for (int i = 0; i < BK / KS; ++i) {
                const bool ok = k0 + bk + KS * i < p.K && cols > 0;
                cp_async16(static_cast<uint32_t>(__cvta_generic_to_shared(&s.b[buf][bk + KS * i][bn])), ok ? u : p.B,
                           ok ? min(cols, 4) * 4 : 0);
                u += sb;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
            const bool inner = k0 + BK <= p.K;
            if (inner && m0 + RH * 32 <= p.M) {
#pragma unroll
                for (int i = 0; i < AN / 2; ++i) {
                    ra[2 * i] = __ldg(q);
                    ra[2 * i + 1] = __ldg(q + 8);
                    q += sa;
                }
            } else {
#pragma unroll
                for (int i = 0; i < AN / 2; ++i) {
                    ra[2 * i] = (8 * i < rows && k0 + ak < p.K) ? __ldg(q) : 0.f;
                    ra[2 * i + 1] = (8 * i < rows && k0 + ak + 8 < p.K) ? __ldg(q + 8) : 0.f;
                    q += sa;
                }
            }
            if (inner && n0 + BW <= p.N) {
#pragma unroll
                for (int i = 0; i < BN; ++i) {
                    rb[i] = __ldg(u);
                    u += sb;
                }
            } else {
#pragma unroll
                for (int i = 0; i < BN; ++i) {
                    rb[i] = (cols > 0 && k0 + bk + BR * i < p.K) ? __ldg(u) : 0.f;
                    u += sb;
                }
            }
        }
    };
    auto store = [&](int buf) {
        if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < AN; ++i) s.a[buf][ak + i % 4][ar + 16 * (i / 4)] = ra[i];
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else {
#pragma unroll
            for (int i = 0; i < AN; ++i) s.a[buf][ak + 8 * (i % 2)][ar + 8 * (i / 2)] = ra[i];
#pragma unroll
            for (int i = 0; i < BN; ++i) s.b[buf][bk + BR * i][bn] = rb[i];
        }
    };
    auto step = [&](int buf, int k) {
        const float* as = &s.a[buf][k][ty * 4];
        const float* bs = &s.b[buf][k][tx * 4];
        float a[RH * 4];
        uint64_t b[CH * 2];
#pragma unroll
        for (int h = 0; h < RH; ++h) {
            const float4 v = *reinterpret_cast<const float4*>(as + 32 * h);
            a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
        }
#pragma unroll
        for (int h = 0; h < CH; ++h) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(bs + 32 * h);
            b[2 * h] = v.x;
            b[2 * h + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < RH * 4; ++i) {
            const uint64_t aa = dup2(a[i]);
#pragma unroll
            for (int j = 0; j < CH * 2; ++j) ffma2(acc[i][j], aa, b[j]);
        }
    };
    const int kblocks = (p.K + BK - 1) / BK;
    __syncthreads();  // readers of an earlier tile are done with the buffers
    load(0, 0);
    store(0);
    __syncthreads();
    for (int kb = 0; kb < kblocks; ++kb) {
        const int cur = kb & 1;
        if (kb + 1 < kblocks)
            load((kb + 1) * BK, cur ^ 1);
        else
            last();
        const int left = min(p.K - kb * BK, BK);
        int k = 0;
#pragma unroll 1
        for (; k + U <= left; k += U) {
#pragma unroll
            for (int u = 0; u < U; ++u) step(cur, k + u);
        }
#pragma unroll 1
        for (; k < left; ++k) step(cur, k);
        if (kb + 1 < kblocks) {
            store(cur ^ 1);
            __syncthreads();
        }
        if constexpr (FOLD) {
            if ((kb + 1) % chain == 0 || kb + 1 == kblocks) tile64_fold<RH, CH>(acc, *tot, kb < chain, kb + 1 < kblocks);
        }
    }
}

// C tile (m0, n0) = alpha A B + beta C.  All 64 threads of the CTA.  `last` runs
// before the last K block is computed, `done` between the K loop and the stores.
// FOLD: an accumulator is closed every `chain` K blocks.
template <bool VEC, bool FOLD, class Last, class Done>
__device__ __forceinline__ void sgemm_tile64(const Tile64Args& p, int m0, int n0, Tile64Smem& s, Last last, Done done,
                                             Tile64Totals* tot = nullptr, int chain = 0) {
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    const bool r2 = p.M - m0 > 32, c2 = p.N - n0 > 32;
    if (r2 && c2)
        tile64_loop<2, 2, VEC, FOLD>(p, m0, n0, s, acc, last, tot, chain);
    else if (r2)
        tile64_loop<2, 1, VEC, FOLD>(p, m0, n0, s, acc, last, tot, chain);
    else if (c2)
        tile64_loop<1, 2, VEC, FOLD>(p, m0, n0, s, acc, last, tot, chain);
    else
        tile64_loop<1, 1, VEC, FOLD>(p, m0, n0, s, acc, last, tot, chain);
    done();
    const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;
    const bool vec = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = m0 + (i / 4) * 32 + ty * 4 + i % 4;
        if (r >= p.M) continue;
        float* row = p.C + (long long)r * p.ldc;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int c = n0 + g * 32 + tx * 4;
            const float2 u = unpack2(acc[i][2 * g]), w = unpack2(acc[i][2 * g + 1]);
            float v[4] = {p.alpha * u.x, p.alpha * u.y, p.alpha * w.x, p.alpha * w.y};
            if (vec && c + 3 < p.N) {
                float4* d = reinterpret_cast<float4*>(row + c);
                if (p.beta != 0.f) {
                    const float4 o = *d;
                    v[0] = fmaf(p.beta, o.x, v[0]); v[1] = fmaf(p.beta, o.y, v[1]);
                    v[2] = fmaf(p.beta, o.z, v[2]); v[3] = fmaf(p.beta, o.w, v[3]);
                }
                *d = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (c + j < p.N) row[c + j] = p.beta != 0.f ? fmaf(p.beta, row[c + j], v[j]) : v[j];
            }
        }
    }
}

// Problem blockIdx.x of a stack; y and z are the tile's indices along the matrix's
// longer and shorter side (TALL: rows are the longer one).  A grid's y extent ends at
// 65535, a side may have more tiles (`longer` of them): then z counts `chunks` of y for
// every index of the shorter side.  No division where one chunk serves: these CTAs
// are short (688 x 20 x 12 x 463: 22.6 us, 24.6 with one).  CTAs that run together
// work on the same tile of different problems, so on the same one of the four loops.
template <bool VEC>
static __global__ void __launch_bounds__(64, 6)
    sgemm_tile64_kernel(Tile64Args p, BatchMap bm, bool tall, int longer, int chunks, int chain) {
    __shared__ Tile64Smem s;
    __shared__ Tile64Totals tot;
    int ty = blockIdx.y, tz = blockIdx.z;
    if (chunks > 1) {
        ty += tz % chunks * gridDim.y;
        tz /= chunks;
        if (ty >= longer) return;
    }
    const int m0 = (tall ? ty : tz) * 64, n0 = (tall ? tz : ty) * 64;
    long long oa, ob;
    batch_offsets(bm, blockIdx.x, oa, ob);
    p.A += oa;
    p.B += ob;
    p.C += blockIdx.x * bm.c_bstride;
    sgemm_tile64<VEC, true>(p, m0, n0, s, [] {}, [] {}, &tot, chain);
}

}  // namespace fg

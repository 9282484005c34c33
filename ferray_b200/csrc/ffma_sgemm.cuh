// ffma_sgemm.cuh -- plain SGEMM on the FP32 pipe with a cp.async ring.
//
// A CTA owns a BM x BN tile of C; each thread accumulates TM x TN outputs, one
// FP32 fused multiply-add per product with k ascending (the per-output order
// of simt_gemm_real, so results are bit-identical to it at equal split-K).
//
// What bounds it is the FMA pipe and how its operands reach it:
//  * the multiply-adds are issued two at a time, `fma.rn.f32x2` on pairs of
//    adjacent columns (each half an ordinary round-to-nearest FMA).  Scalar
//    FMAs spend an issue slot each and meet register-bank conflicts: an 8 x 8
//    outer product on registers alone runs at 51 TFLOP/s on a B200, the paired
//    form at 62, and with 16 x 8 outputs a thread and a column pair taken down
//    all 16 rows at 65;
//  * A is first transposed into a packed K x Mp scratch (Mp = M rounded up to
//    4, zero padded), so both operand tiles are rows of 16-byte chunks that
//    `cp.async` copies without passing through registers.  Transposing inside
//    the kernel was slower at every size above 512 (4-byte copies 48 TFLOP/s,
//    through registers 52, against 58 with the same 8 x 8 tile);
//  * a thread's copies keep one column of chunks, so their addresses advance
//    by one add each (recomputing them and their bounds: 53 against 57).
// 8192^3: 66.0 TFLOP/s (128 x 128 tiles, 16 x 8 a thread, two CTAs of 128
// threads per SM), against 52.9 for the scalar 8 x 8 kernel it replaced.
//
// Which tile and split-K count a shape takes is ffma_plan's choice
// (gemm_simt.cu).  B is read in place.  Where its rows are not 16-byte aligned (SHIFT) they are
// copied as the aligned 16-byte granules that hold them and read from shared
// memory at the row's offset, four bytes at a time.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "simt_gemm.cuh"

namespace fg {

template <int BM_, int BN_, int TM_, int TN_, int MINB_, int BPAD_, bool SHIFT_ = false>
struct FfmaTile {
    static constexpr bool SHIFT = SHIFT_;
    static constexpr int BK = 16, STAGES = 4, BPAD = BPAD_;
    static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, MINB = MINB_;
    static constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
    static constexpr int AP = BM + 4;                   // pitch of A's k rows (floats)
    static constexpr int BP = BN + (SHIFT ? 4 : BPAD);  // of B's
    static constexpr int AS = BK * AP, BS = BK * BP;    // floats per stage
    static constexpr size_t SMEM = size_t(STAGES) * (AS + BS) * sizeof(float);
    static_assert(TM % 4 == 0 && TN % 4 == 0 && THREADS % 32 == 0, "tile shape");
};

// 16 bytes global -> shared, the first `bytes` of them from memory, the rest
// zero.
__device__ __forceinline__ void cp_async16(uint32_t s, const void* gmem, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}

// d += a * b on both halves of a register pair, each rounded to nearest.
__device__ __forceinline__ void ffma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t dup2(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ uint64_t pack2(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// At[z] (K x ldat, zero beyond M) = A[z]^T for the `count` distinct A
// matrices (row-major M x K, leading dimension lda, matrix stride ms).
// Grid: x over 64-row blocks of M, y over 64-column blocks of K, z over the
// matrices; 256 threads.  16-byte loads along K where A's rows allow it,
// 16-byte stores along M (ldat is a multiple of 4).
static __global__ void __launch_bounds__(256)
    transpose_pack_kernel(const float* __restrict__ A, int M, int K, long long lda, long long ms,
                          float* __restrict__ At, long long ldat) {
    __shared__ float t[64][65];
    const int m0 = blockIdx.x * 64, k0 = blockIdx.y * 64;
    const float* a = A + blockIdx.z * ms;
    float* at = At + blockIdx.z * (long long)K * ldat;
    const bool vec = lda % 4 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = threadIdx.x + 256 * i, m = c / 16, k = c % 16 * 4;
        const float* p = a + (long long)(m0 + m) * lda + k0 + k;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m0 + m < M) {
            if (vec && k0 + k + 3 < K) {
                v = __ldg(reinterpret_cast<const float4*>(p));
            } else {
                if (k0 + k < K) v.x = __ldg(p);
                if (k0 + k + 1 < K) v.y = __ldg(p + 1);
                if (k0 + k + 2 < K) v.z = __ldg(p + 2);
                if (k0 + k + 3 < K) v.w = __ldg(p + 3);
            }
        }
        t[m][k] = v.x; t[m][k + 1] = v.y; t[m][k + 2] = v.z; t[m][k + 3] = v.w;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int c = threadIdx.x + 256 * i, k = c / 16, m = c % 16 * 4;
        if (k0 + k < K && m0 + m < ldat)
            *reinterpret_cast<float4*>(at + (long long)(k0 + k) * ldat + m0 + m) =
                make_float4(t[m][k], t[m + 1][k], t[m + 2][k], t[m + 3][k]);
    }
}

// CGEMM as a real GEMM (the ZGEMM embedding of dmma_gemm.cuh in f32):
// interleaved complex A (M x K) is the real M x 2K matrix it lies as, and
// B' (2K x 2N, pitch 2N) holds [[br, bi], [-bi, br]] for every complex b,
// so columns 2n and 2n + 1 of A B' are Re and Im of (AB)[:, n].
static __global__ void cgemm_expand_b_kernel(const float2* __restrict__ B, long long K, long long N, long long ldb,
                                             float* __restrict__ Bx) {
    const long long total = K * N;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long k = e / N, n = e - k * N;
        const float2 b = B[k * ldb + n];
        float* r0 = Bx + (2 * k) * (2 * N) + 2 * n;
        float* r1 = r0 + 2 * N;
        *reinterpret_cast<float2*>(r0) = make_float2(b.x, b.y);
        *reinterpret_cast<float2*>(r1) = make_float2(-b.y, b.x);
    }
}

// Copies one operand's tiles (BK rows of W floats, a K block after the other)
// into shared-memory rows of PITCH floats.  Rows at or past the end of K and
// columns at or past `cols` read zeros.  SHIFT: rows start at any float; each
// is copied as the W / 4 + 1 aligned 16-byte granules that hold it, so it
// begins (float address mod 4) floats into its shared row.
template <int BK, int W, int PITCH, int THREADS, bool SHIFT>
struct FfmaLoader {
    static constexpr int RSTEP = THREADS / (W / 4), CNT = BK / RSTEP;
    static_assert(THREADS % (W / 4) == 0 && BK % RSTEP == 0 && CNT > 0, "whole rows of copies");
    static_assert(!SHIFT || (BK <= THREADS && PITCH >= W + 4), "one extra granule per row");
    const float* base;
    const float* p;    // this thread's next copy
    long long step;    // RSTEP rows
    int row, left;     // its row in the block; floats of a row from its column on (may be <= 0)
    uint32_t dst;      // shared byte offset of its first copy
    const float* px;   // SHIFT: the granule past the W / 4 (row threadIdx.x)
    long long stepx;

    __device__ __forceinline__ void init(const float* X, long long ldx, int c0, int cols) {
        const int col = static_cast<int>(threadIdx.x) % (W / 4) * 4;
        row = static_cast<int>(threadIdx.x) / (W / 4);
        left = cols - c0 - col;
        base = X;
        const bool in = SHIFT || left > 0;
        step = in ? RSTEP * ldx : 0;
        p = in ? X + row * ldx + c0 + col : X;
        dst = (row * PITCH + col) * 4;
        if constexpr (SHIFT) {
            px = X + static_cast<int>(threadIdx.x) % BK * ldx + c0 + W;
            stepx = BK * ldx;
        }
    }
    // the aligned granule around q, of which `n` floats from q on belong to the row
    __device__ __forceinline__ void granule(uint32_t d, const float* q, int n, bool ok) const {
        const uintptr_t u = reinterpret_cast<uintptr_t>(q);
        const int f = ok ? min(max(n + static_cast<int>(u / 4 % 4), 0), 4) : 0;
        cp_async16(d, reinterpret_cast<const void*>((f ? u : reinterpret_cast<uintptr_t>(base)) & ~uintptr_t(15)), f * 4);
    }
    // The next block; its rows [0, rows) exist (rows >= BK for all but the last).
    __device__ __forceinline__ void load(uint32_t stage, int rows) {
        if constexpr (SHIFT) {
#pragma unroll
            for (int i = 0; i < CNT; ++i) {
                granule(stage + dst + i * RSTEP * PITCH * 4, p, left, row + i * RSTEP < rows);
                p += step;
            }
            if (threadIdx.x < BK) {
                const int n = left + static_cast<int>(threadIdx.x) % (W / 4) * 4 - W;
                granule(stage + (threadIdx.x * PITCH + W) * 4, px, n, static_cast<int>(threadIdx.x) < rows);
            }
            px += stepx;
        } else if (rows >= BK) {
            const int bytes = min(max(left, 0), 4) * 4;
#pragma unroll
            for (int i = 0; i < CNT; ++i) {
                cp_async16(stage + dst + i * RSTEP * PITCH * 4, p, bytes);
                p += step;
            }
        } else {
            const int bytes = min(max(left, 0), 4) * 4;
#pragma unroll
            for (int i = 0; i < CNT; ++i) {
                const bool ok = row + i * RSTEP < rows;
                cp_async16(stage + dst + i * RSTEP * PITCH * 4, ok ? p : base, ok ? bytes : 0);
                p += ok ? step : 0;
            }
        }
    }
};

// acc += the products of one k.  as points at this thread's first row, bs at
// its first column of the k row: groups of 4 adjacent columns TX * 4 apart
// (16-byte reads), or with SHIFT single columns TX apart.
template <class Cfg>
__device__ __forceinline__ void ffma_step(const float* as, const float* bs, uint64_t (&acc)[Cfg::TM][Cfg::TN / 2]) {
    constexpr bool SHIFT = Cfg::SHIFT;
    float a[Cfg::TM];
    uint64_t b[Cfg::TN / 2];
#pragma unroll
    for (int g = 0; g < Cfg::TM / 4; ++g) {
        const float4 v = *reinterpret_cast<const float4*>(as + g * Cfg::TY * 4);
        a[4 * g] = v.x; a[4 * g + 1] = v.y; a[4 * g + 2] = v.z; a[4 * g + 3] = v.w;
    }
    if constexpr (SHIFT) {
#pragma unroll
        for (int j = 0; j < Cfg::TN / 2; ++j) b[j] = pack2(bs[2 * j * Cfg::TX], bs[(2 * j + 1) * Cfg::TX]);
    } else {
#pragma unroll
        for (int g = 0; g < Cfg::TN / 4; ++g) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(bs + g * Cfg::TX * 4);
            b[2 * g] = v.x;
            b[2 * g + 1] = v.y;
        }
    }
    if constexpr (Cfg::TM == 16) {  // a column pair down all rows (see above)
        uint64_t aa[Cfg::TM];
#pragma unroll
        for (int i = 0; i < Cfg::TM; ++i) aa[i] = dup2(a[i]);
#pragma unroll
        for (int j = 0; j < Cfg::TN / 2; ++j)
#pragma unroll
            for (int i = 0; i < Cfg::TM; ++i) ffma2(acc[i][j], aa[i], b[j]);
    } else {
#pragma unroll
        for (int i = 0; i < Cfg::TM; ++i) {
            const uint64_t aa = dup2(a[i]);
#pragma unroll
            for (int j = 0; j < Cfg::TN / 2; ++j) ffma2(acc[i][j], aa, b[j]);
        }
    }
}

// C = alpha At^T B + beta C.  At: packed K x ldat per A matrix (batch offsets
// from bm.a_bstride in packed elements).  blockIdx.z = split * nbatch + batch
// index; split s covers K rows [s * ksplit, (s + 1) * ksplit) and writes output
// matrix blockIdx.z (a partial-sum workspace when split).
template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::MINB)
    ffma_sgemm_kernel(int M, int N, int K, float alpha, const float* __restrict__ At, long long ldat,
                      const float* __restrict__ B, long long ldb, float beta, float* __restrict__ C, long long ldc,
                      BatchMap bm, int nbatch, int ksplit) {
    constexpr bool SHIFT = Cfg::SHIFT;
    constexpr int BK = Cfg::BK, STAGES = Cfg::STAGES, TM = Cfg::TM, TN = Cfg::TN, TX = Cfg::TX, TY = Cfg::TY;
    extern __shared__ __align__(16) float ffma_sm[];
    float* As = ffma_sm;                      // [STAGES][BK][AP]
    float* Bs = ffma_sm + STAGES * Cfg::AS;   // [STAGES][BK][BP]

    const int zb = blockIdx.z % nbatch, zs = blockIdx.z / nbatch;
    long long oa, ob;
    batch_offsets(bm, zb, oa, ob);
    const int k_begin = zs * ksplit;
    At += oa + (long long)k_begin * ldat;
    B += ob + (long long)k_begin * ldb;
    C += blockIdx.z * bm.c_bstride;
    K = min(K - k_begin, ksplit);

    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int m0 = blockIdx.y * Cfg::BM, n0 = blockIdx.x * Cfg::BN;
    const int kblocks = (K + BK - 1) / BK;
    FfmaLoader<BK, Cfg::BM, Cfg::AP, Cfg::THREADS, false> la;
    FfmaLoader<BK, Cfg::BN, Cfg::BP, Cfg::THREADS, SHIFT> lb;
    la.init(At, ldat, m0, static_cast<int>(ldat));
    lb.init(B, ldb, n0, N);
    const uint32_t sa = static_cast<uint32_t>(__cvta_generic_to_shared(As));
    const uint32_t sb = static_cast<uint32_t>(__cvta_generic_to_shared(Bs));
    auto load = [&](int kb) {
        const int s = kb % STAGES;
        la.load(sa + s * Cfg::AS * 4, K - kb * BK);
        lb.load(sb + s * Cfg::BS * 4, K - kb * BK);
    };

    uint64_t acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < kblocks) load(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // SHIFT: float address mod 4 of this block's first B row, and its step per row
    int sh = static_cast<int>(reinterpret_cast<uintptr_t>(B) / 4 % 4);
    const int dsh = static_cast<int>(ldb % 4);
    for (int kb = 0; kb < kblocks; ++kb) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();  // stage kb landed for all threads; stage kb - 1 is free
        if (kb + STAGES - 1 < kblocks) load(kb + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = As + (kb % STAGES) * Cfg::AS + ty * 4;
        const float* bs = Bs + (kb % STAGES) * Cfg::BS + (SHIFT ? tx : tx * 4);
        if (K - kb * BK >= BK) {
#pragma unroll
            for (int k = 0; k < BK; ++k)
                ffma_step<Cfg>(as + k * Cfg::AP, bs + k * Cfg::BP + (SHIFT ? (sh + k * dsh) & 3 : 0), acc);
        } else {
#pragma unroll 1
            for (int k = 0; k < K - kb * BK; ++k)
                ffma_step<Cfg>(as + k * Cfg::AP, bs + k * Cfg::BP + (SHIFT ? (sh + k * dsh) & 3 : 0), acc);
        }
        if constexpr (SHIFT) sh = (sh + BK * dsh) & 3;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    const bool vec_c = !SHIFT && (ldc % 4 == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = m0 + (i / 4) * TY * 4 + ty * 4 + i % 4;
        if (r >= M) continue;
        float* row = C + (long long)r * ldc;
#pragma unroll
        for (int g = 0; g < TN / 4; ++g) {
            const float2 u = unpack2(acc[i][2 * g]), w = unpack2(acc[i][2 * g + 1]);
            float v[4] = {alpha * u.x, alpha * u.y, alpha * w.x, alpha * w.y};
            const int c = n0 + (SHIFT ? g * 4 * TX + tx : g * TX * 4 + tx * 4);
            if (vec_c && c + 3 < N) {
                float4* p = reinterpret_cast<float4*>(row + c);
                if (beta != 0.f) {
                    const float4 o = *p;
                    v[0] = fmaf(beta, o.x, v[0]); v[1] = fmaf(beta, o.y, v[1]);
                    v[2] = fmaf(beta, o.z, v[2]); v[3] = fmaf(beta, o.w, v[3]);
                }
                *p = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int cj = c + j * (SHIFT ? TX : 1);
                    if (cj < N) row[cj] = beta != 0.f ? fmaf(beta, row[cj], v[j]) : v[j];
                }
            }
        }
    }
}

}  // namespace fg

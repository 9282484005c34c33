// ozaki_kernels.cuh -- operand slicing for the INT8 Ozaki DGEMM / ZGEMM.
//
// Method (Ozaki, Ogita, Oishi error-free splitting, in the INT8 form of
// Ootomo/Ozaki/Yokota and Uchino/Ozaki/Imamura): every row i of A is scaled
// by 2^-e_i, with e_i the frexp exponent of max_k |a_ik|, so |a_ik 2^-e_i| < 1;
// the scaled value t is written as S signed base-128 digits by exact
// scale-and-truncate steps, t = sum_{s=1..S} d_s 128^-s + r, |d_s| <= 127,
// |r| < 128^-S, each digit plane stored as an int8 slice.  Before that the
// inner dimension is balanced: AB = (A D)(D^-1 B) with D = diag(2^shift_k)
// chosen from A's column maxima and B's row maxima, so a term a_ik b_kj is
// represented relative to magnitudes near its own rather than to the largest
// entry of its row (which is what keeps exponent-spread inputs accurate).  Columns of B likewise with
// their own exponents f_j.  Then
//     C_ij = 2^(e_i+f_j) sum_{s,t} 2^(-7(s+t)) (A_s B_t)_ij
// and the products A_s B_t are exact int32 GEMMs on the integer tensor cores.
// Pairs with s + t > S + 1 are dropped (each is below K * 2^-7S of
// row-max * col-max).
//
// Layouts chosen so every group d = s + t is ONE plain int8 GEMM over a
// concatenated K: A slices side by side, A_all = [A_1 | A_2 | ... | A_S]
// (M x S*Kp), and B slices stacked in reverse, B_all = [B_S; ...; B_1]
// (S*Kp x N).  Group d is then A_all[:, 0:(d-1)Kp] times the last (d-1)Kp
// rows of B_all, i.e. sum_{s=1..d-1} A_s B_{d-s}.
//
// Complex operands use the real embedding [Ar Ai] and [[Br Bi], [-Bi Br]]
// (M x 2K and 2K x 2N) while slicing.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace fg {

// |x| as ordered bits (monotone for non-negative doubles, NaN above Inf).
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7FFFFFFFFFFFFFFFull;
}

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }  // |e| <= 1000

// x 2^sh, |sh| <= 2000, with one rounding: what is beyond 1000 is multiplied first,
// which is exact unless the result is zero or infinite anyway.  No branch: ldexp in
// a loop over a row kept its loads from being in flight together (4096^2: row
// scales 48 -> 37 us, column maxima 53 -> 25).
__device__ __forceinline__ double scale_pow2(double x, int sh) {
    const int b = max(-1000, min(1000, sh));
    return (x * pow2(sh - b)) * pow2(b);
}

// 2^e with frexp(max) = m * 2^e, m in [0.5, 1); zero rows get 1, non-finite
// rows get NaN so their outputs come out NaN.
__device__ __forceinline__ double scale_from_max_bits(unsigned long long bits) {
    const double mx = __longlong_as_double(static_cast<long long>(bits));
    if (mx == 0.0) return 1.0;
    if (!isfinite(mx)) return __longlong_as_double(0x7FF8000000000000ll);
    int e;
    frexp(mx, &e);
    return ldexp(1.0, e);
}

// Block-wide max of one value per thread (blockDim.x a multiple of 32, at
// most 1024); every thread gets the result.
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v) {
    __shared__ unsigned long long red[32];
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    __syncthreads();  // red[] may still be read from the previous call
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = threadIdx.x < blockDim.x / 32 ? red[threadIdx.x] : 0ull;
    if (threadIdx.x < 32)
        for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    if (threadIdx.x == 0) red[0] = v;
    __syncthreads();
    return red[0];
}

// Row maxima of a real (cplx = 0) or complex (cplx = 1: Re and Im) matrix,
// one block per row (blocks stride over the rows), so a row's loads are
// spread over the block's warps.
// `shift` (may be null) holds the balancing exponent of each K index: the row
// maxima are those of A * diag(2^shift).
static __global__ void ozaki_row_scale_kernel(const double* __restrict__ A, long long M,
                                              long long K, long long lda, int cplx,
                                              const int* __restrict__ shift,
                                              double* __restrict__ scale) {
    const long long len = cplx ? 2 * K : K;
    for (long long row = blockIdx.x; row < M; row += gridDim.x) {
        const double* r = A + row * (cplx ? 2 * lda : lda);
        unsigned long long mx = 0;
#pragma unroll 8
        for (long long k = threadIdx.x; k < len; k += blockDim.x) {
            const int sh = shift ? shift[cplx ? (k >> 1) : k] : 0;
            mx = max(mx, abs_bits(scale_pow2(r[k], sh)));
        }
        mx = block_max_u64(mx);
        if (threadIdx.x == 0) scale[row] = scale_from_max_bits(mx);
    }
}

// Column maxima, pass 1: each thread scans `rows_per` rows of one (complex:
// embedded) column and folds the result into colmax_bits with atomicMax.
// Real B: N columns.  Complex B: the embedded B' has 2N columns, column c < N
// holds (Br, -Bi) and c >= N holds (Bi, Br) -> both have max(|Br|, |Bi|) of
// complex column c mod N, so N maxima suffice.
// The column maxima are those of diag(2^-shift) * B (shift may be null).
static __global__ void ozaki_col_max_kernel(const double* __restrict__ B, long long K, long long N,
                                            long long ldb, int cplx, long long rows_per,
                                            const int* __restrict__ shift,
                                            unsigned long long* __restrict__ colmax_bits) {
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= N) return;
    const long long k0 = blockIdx.y * rows_per, k1 = min(K, k0 + rows_per);
    unsigned long long mx = 0;
#pragma unroll 8
    for (long long k = k0; k < k1; ++k) {
        const int sh = shift ? -shift[k] : 0;
        if (cplx) {
            const double2 v = reinterpret_cast<const double2*>(B)[k * ldb + j];
            mx = max(mx, max(abs_bits(scale_pow2(v.x, sh)), abs_bits(scale_pow2(v.y, sh))));
        } else {
            mx = max(mx, abs_bits(scale_pow2(B[k * ldb + j], sh)));
        }
    }
    atomicMax(colmax_bits + j, mx);
}

// Balancing of the inner dimension: AB = (A D)(D^-1 B) for D = diag(2^shift_k).
// Pass 1: column maxima of A (over rows, atomicMax of ordered bits).
static __global__ void ozaki_a_colmax_kernel(const double* __restrict__ A, long long M, long long K,
                                             long long lda, int cplx, long long rows_per,
                                             unsigned long long* __restrict__ out) {
    const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (k >= K) return;
    const long long i0 = blockIdx.y * rows_per, i1 = min(M, i0 + rows_per);
    unsigned long long mx = 0;
#pragma unroll 8
    for (long long i = i0; i < i1; ++i) {
        if (cplx) {
            const double2 v = reinterpret_cast<const double2*>(A)[i * lda + k];
            mx = max(mx, max(abs_bits(v.x), abs_bits(v.y)));
        } else {
            mx = max(mx, abs_bits(A[i * lda + k]));
        }
    }
    atomicMax(out + k, mx);
}

// Pass 2: row maxima of B, one block per row (blocks stride over the rows).
static __global__ void ozaki_b_rowmax_kernel(const double* __restrict__ B, long long K, long long N,
                                             long long ldb, int cplx,
                                             unsigned long long* __restrict__ out) {
    const long long len = cplx ? 2 * N : N;
    for (long long row = blockIdx.x; row < K; row += gridDim.x) {
        const double* r = B + row * (cplx ? 2 * ldb : ldb);
        unsigned long long mx = 0;
#pragma unroll 8
        for (long long j = threadIdx.x; j < len; j += blockDim.x) mx = max(mx, abs_bits(r[j]));
        mx = block_max_u64(mx);
        if (threadIdx.x == 0) out[row] = mx;
    }
}

// Pass 3: shift_k = floor((eB_k - eA_k) / 2), so column k of A D and row k of
// D^-1 B peak at about the same magnitude.  Zero or non-finite maxima: 0.
static __global__ void ozaki_shift_kernel(const unsigned long long* __restrict__ a_colmax,
                                          const unsigned long long* __restrict__ b_rowmax,
                                          long long K, int* __restrict__ shift) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K;
         k += (long long)gridDim.x * blockDim.x) {
        const double ma = __longlong_as_double(static_cast<long long>(a_colmax[k]));
        const double mb = __longlong_as_double(static_cast<long long>(b_rowmax[k]));
        int sh = 0;
        if (ma > 0.0 && mb > 0.0 && isfinite(ma) && isfinite(mb)) {
            int ea, eb;
            frexp(ma, &ea);
            frexp(mb, &eb);
            const int d = eb - ea;
            sh = d >= 0 ? d / 2 : -((-d + 1) / 2);
        }
        shift[k] = sh;
    }
}

static __global__ void ozaki_col_scale_kernel(const unsigned long long* __restrict__ colmax_bits,
                                              long long N, double* __restrict__ scale) {
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < N;
         j += (long long)gridDim.x * blockDim.x)
        scale[j] = scale_from_max_bits(colmax_bits[j]);
}

// Signed base-128 digits of t = x / scale, |t| < 1, by repeated exact
// scaling and truncation: t = sum_s d_s 128^-(s+1) + r, |r| < 128^-S, all
// digits carrying the sign of x (each step is exact in FP64).
template <int S>
__device__ __forceinline__ void ozaki_digits(double x, double inv_scale, int8_t (&d)[S]) {
    double t = x * inv_scale;  // power-of-two scaling: exact
    if (!isfinite(t)) t = 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        t *= 128.0;
        const double q = trunc(t);
        t -= q;
        d[s] = static_cast<int8_t>(static_cast<int>(q));
    }
}

// A slices: A_all[i, s*Kp + k] = digit s of A[i, k] (s = 0 most significant);
// complex A is embedded as [Ar | Ai] (width 2K).  Kp >= width, padding zero.
// Chunked: this launch writes embedded columns [k0, k0 + Kp) of the plane.
template <int S>
__global__ void ozaki_slice_a_kernel(const double* __restrict__ A, long long M, long long K,
                                     long long lda, int cplx, const int* __restrict__ shift,
                                     const double* __restrict__ scale,
                                     int8_t* __restrict__ out, long long Kp, long long k0) {
    const long long W = cplx ? 2 * K : K;
    const long long total = M * Kp;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long i = e / Kp, kl = e - i * Kp, k = k0 + kl;
        double x = 0.0;
        if (k < W) {
            if (cplx) {
                const long long kk = k < K ? k : k - K;
                x = ldexp(A[2 * (i * lda + kk) + (k < K ? 0 : 1)], shift[kk]);
            } else {
                x = ldexp(A[i * lda + k], shift[k]);
            }
        }
        int8_t d[S];
        ozaki_digits<S>(x, 1.0 / scale[i], d);
        int8_t* o = out + i * (S * Kp) + kl;
#pragma unroll
        for (int s = 0; s < S; ++s) o[s * Kp] = d[s];
    }
}

// B slices stacked in reverse: B_all[(S-1-s)*Kp + k, j] = digit s of B[k, j].
// Complex B is embedded as [[Br, Bi], [-Bi, Br]] (2K x 2N); Np >= width.
// Chunked: this launch writes embedded rows [k0, k0 + Kp) of the planes.
template <int S>
__global__ void ozaki_slice_b_kernel(const double* __restrict__ B, long long K, long long N,
                                     long long ldb, int cplx, const int* __restrict__ shift,
                                     const double* __restrict__ scale,
                                     int8_t* __restrict__ out, long long Kp, long long Np,
                                     long long k0) {
    const long long H = cplx ? 2 * K : K;   // embedded rows
    const long long W = cplx ? 2 * N : N;   // embedded columns
    const long long total = Kp * Np;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const long long kl = e / Np, j = e - kl * Np, k = k0 + kl;
        double x = 0.0;
        double sc = 1.0;
        if (k < H && j < W) {
            if (cplx) {
                const bool top = k < K, left = j < N;
                const long long kk = top ? k : k - K, jj = left ? j : j - N;
                const double2 v = reinterpret_cast<const double2*>(B)[kk * ldb + jj];
                // top-left Br, top-right Bi, bottom-left -Bi, bottom-right Br
                x = ldexp(top ? (left ? v.x : v.y) : (left ? -v.y : v.x), -shift[kk]);
                sc = scale[jj];
            } else {
                x = ldexp(B[k * ldb + j], -shift[k]);
                sc = scale[j];
            }
        }
        int8_t d[S];
        ozaki_digits<S>(x, 1.0 / sc, d);
#pragma unroll
        for (int s = 0; s < S; ++s) out[((S - 1 - s) * Kp + kl) * Np + j] = d[s];
    }
}

// ---------------------------------------------------------------- scheme II
// Ozaki scheme II (Ozaki, Uchino, Imamura: integer emulation of FP64 GEMM by
// the Chinese remainder theorem).  After the same balancing and row / column
// scaling as the slices above, every entry becomes one integer
//     a'_ik = rint(2^P a_ik 2^sh_k / 2^e_i),  |a'| <= 2^P,
// exactly representable as a double (below 2^53 it is an integer, above it
// t 2^P already is one), and likewise b'_kj with 2^-sh_k / 2^f_j.  For
// pairwise coprime moduli m_1..m_n <= 256 with product Mp > 2 K 2^(2P), the
// exact C' = A'B' is fixed by its residues C' mod m_l = (A' mod m_l)
// (B' mod m_l) mod m_l: ONE int8 GEMM per modulus on symmetric residues in
// [-128, 127] (exact int32 accumulation for K < 2^17), against the S(S+1)/2
// slice products of scheme I.  C' is rebuilt from the residue bytes in
// double arithmetic (oz2_reconstruct_kernel) and scaled back by 2^(e_i +
// f_j - 2P).
struct Oz2Consts {
    int n, P;
    int m[24];
    uint32_t magic[24];             // ceil(2^32 / m_l)
    uint32_t c_lo[24], c_hi[24];    // bytes 256^b mod m_l of the two words of an integer
    uint32_t corr[24];              // (m_l / 2 - 2^60) mod m_l
    double inv_M;                   // 1 / Mp, for the CRT quotient
    uint32_t pm[10][2];             // moduli pair (2t, 2t + 1): m_(2t+1), m_2t (1, 0 for a single last)
    double pW[10][5];               // Mp / (m_2t m_(2t+1)) in base-2^33 digits, least significant first
    double Mc[5];                   // Mp in base-2^33 digits
};

// 1 / s of a power of two (or NaN).
__device__ __forceinline__ double recip_pow2(double s) {
    const int hi = __double2hiint(s);
    if (static_cast<unsigned>(hi - 0x00100000) < 0x7FD00000u) return __hiloint2double(0x7FE00000 - hi, 0);
    return 1.0 / s;
}

// rint(v) + 2^60 of |v| <= 2^59 (a non-finite entry counts as zero: its row's or
// column's NaN scale marks the outputs).
__device__ __forceinline__ uint2 oz2_biased(double v) {
    const bool finite = (__double2hiint(v) & 0x7FF00000) != 0x7FF00000;
    const unsigned long long u = static_cast<unsigned long long>(finite ? __double2ll_rn(v) : 0ll) + (1ull << 60);
    return make_uint2(static_cast<uint32_t>(u), static_cast<uint32_t>(u >> 32));
}

// Symmetric residues in [-(m/2), m - 1 - (m/2)] of eight such integers, packed.
// The integer's bytes times 256^b mod m (two dp4a) give an x < 2^20 of the same
// residue, x mod m is the high word of (x ceil(2^32 / m) mod 2^32) m (Lemire, Kaser
// and Kurz, "Faster remainder by direct computation", 2019), and m/2, added before, is
// taken off all four bytes of a word at once.
__device__ __forceinline__ uint2 oz2_pack8(const uint2 (&a)[8], const Oz2Consts& c, int l) {
    const uint32_t m = static_cast<uint32_t>(c.m[l]), magic = c.magic[l], c_lo = c.c_lo[l], c_hi = c.c_hi[l];
    const uint32_t corr = c.corr[l], h4 = (m / 2) * 0x01010101u;
    uint32_t w[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint32_t r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            r[u] = __umulhi(__dp4a(a[4 * q + u].x, c_lo, __dp4a(a[4 * q + u].y, c_hi, corr)) * magic, m);
        const uint32_t p = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
        w[q] = ((p | 0x80808080u) - (h4 & 0x7F7F7F7Fu)) ^ ((p ^ ~h4) & 0x80808080u);
    }
    return make_uint2(w[0], w[1]);
}

// A residue planes: A_all[i, l*Kp + k] = a'_ik mod m_l (complex A embedded
// as [Ar | Ai], width 2K; columns past the width are zero).  A thread takes
// eight consecutive k of one row and writes 8 bytes per plane; a block is 8 rows
// of 256 k.  Instructions per entry and modulus bound it, about six (4096^2, 16
// moduli: 127 us; 234 with three-limb residues and ldexp).
// VEC: real A whose rows start on 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(256, 4) oz2_residue_a_kernel(
    const double* __restrict__ A, long long M, long long K, long long lda, int cplx, const int* __restrict__ shift,
    const double* __restrict__ scale, int8_t* __restrict__ out, long long Kp, const __grid_constant__ Oz2Consts c) {
    const long long W = cplx ? 2 * K : K;
    const long long k0 = (blockIdx.x * 32ll + threadIdx.x) * 8;
    if (k0 >= Kp) return;
    double f[8];  // of the shifts up to 1000; `more`: some go beyond
    bool more = false;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const long long k = k0 + u;
        const int sh = k < W ? shift[k < K ? k : k - K] : 0, b = max(-1000, min(1000, sh));
        f[u] = pow2(b);
        more |= sh != b;
    }
    const double up = pow2(c.P);
    for (long long i = blockIdx.y * 8ll + threadIdx.y; i < M; i += gridDim.y * 8ll) {
        const double inv = recip_pow2(scale[i]);
        double x[8];
        if (VEC && k0 + 8 <= K) {
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
                const double2 v = *reinterpret_cast<const double2*>(A + i * lda + k0 + u);
                x[u] = v.x;
                x[u + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const long long k = k0 + u;
                x[u] = k >= W ? 0.0 : cplx ? A[2 * (i * lda + (k < K ? k : k - K)) + (k < K ? 0 : 1)] : A[i * lda + k];
            }
        }
        if (more) {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const long long k = k0 + u;
                const int sh = k < W ? shift[k < K ? k : k - K] : 0;
                x[u] *= pow2(sh - max(-1000, min(1000, sh)));
            }
        }
        uint2 a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = oz2_biased((x[u] * f[u] * inv) * up);
        int8_t* o = out + i * (c.n * Kp) + k0;
        for (int l = 0; l < c.n; ++l) *reinterpret_cast<uint2*>(o + l * Kp) = oz2_pack8(a, c, l);
    }
}

// B residue planes: B_all[l*Kp + k, j] = b'_kj mod m_l (complex B embedded
// as [[Br, Bi], [-Bi, Br]]).  A thread takes eight consecutive j, whose scales it
// keeps over its rows; bound as for A (122 us; 239 before).
template <bool VEC>
__global__ void __launch_bounds__(256, 4) oz2_residue_b_kernel(
    const double* __restrict__ B, long long K, long long N, long long ldb, int cplx, const int* __restrict__ shift,
    const double* __restrict__ scale, int8_t* __restrict__ out, long long Kp, long long Np,
    const __grid_constant__ Oz2Consts c) {
    const long long H = cplx ? 2 * K : K, Wn = cplx ? 2 * N : N;
    const long long j0 = (blockIdx.x * 32ll + threadIdx.x) * 8;
    if (j0 >= Np) return;
    const double up = pow2(c.P);
    double inv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const long long j = j0 + u;
        inv[u] = j < Wn ? recip_pow2(scale[j < N ? j : j - N]) : 1.0;
    }
    for (long long k = blockIdx.y * 8ll + threadIdx.y; k < Kp; k += gridDim.y * 8ll) {
        const bool top = k < K;
        const long long kk = top ? k : k - K;
        const int sh = k < H ? -shift[kk] : 0;
        double x[8];
        if (VEC && top && j0 + 8 <= N) {
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
                const double2 v = *reinterpret_cast<const double2*>(B + k * ldb + j0 + u);
                x[u] = v.x;
                x[u + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const long long j = j0 + u;
                const bool left = j < N;
                if (k >= H || j >= Wn) {
                    x[u] = 0.0;
                } else if (cplx) {
                    const double v = B[2 * (kk * ldb + (left ? j : j - N)) + (top == left ? 0 : 1)];
                    x[u] = !top && left ? -v : v;
                } else {
                    x[u] = B[k * ldb + j];
                }
            }
        }
        uint2 b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) b[u] = oz2_biased((scale_pow2(x[u], sh) * inv[u]) * up);
        int8_t* o = out + k * Np + j0;
        for (int l = 0; l < c.n; ++l) *reinterpret_cast<uint2*>(o + l * Kp * Np) = oz2_pack8(b, c, l);
    }
}

// C from the residue bytes R[l][i, j] = (C'_ij mod m_l) y_l mod m_l, |C'| < Mp / 4:
// C' = sum_l R_l Mp / m_l - q Mp.  Two moduli at a time, R_a Mp / m_a + R_b Mp / m_b
// = (R_a m_b + R_b m_a) Mp / (m_a m_b) with a factor below 2^17, so the sum is exact
// in base-2^33 digit sums (each below 2^53: 33 bits, and the factors of all pairs
// add up to less than 2^20); q = rint(sum / Mp) (at most n, far from a tie),
// the digits of C' follow exactly and are balanced into [-2^32, 2^32] with exact
// carries.  The digits above the two lowest are joined first, what that rounds off
// (Dekker's Fast2Sum) is added to the lowest, and the final sum is the one rounding that
// counts
// (rounding twice showed: 17 moduli 1.3e-18 of ||A|| ||B|| at 2048^3, 2e-19 so).
// Then C = alpha 2^(e_i + f_j - 2P) C' (+ beta C).
// Complex: embedded column j < N is Re of column j, j >= N Im of column j - N
// (interleaved C).  FP64 and instruction issue bound it about evenly (some 70
// FP64 operations an output at 16 moduli); a thread has four columns, so that one
// load brings four bytes (two columns: 165 us).  4096^2, 16 moduli: 133 us; 241 with
// one output a thread, one modulus at a time, base 2^40 and integer carries.
// Registers: 80 a thread (three blocks an SM) up to 18 moduli, 128 with the fifth
// digit of 19 and 20 (80: 418 us, 177 so); complex outputs two columns at a time (four
// at once spill: 4096^2 16 moduli 434 us, 271 so, 19 moduli 1382, 369 so).
template <int ND>
__device__ __forceinline__ double oz2_rebuild(double (&d)[ND], const Oz2Consts& c) {
    constexpr double B = 0x1p33, MAGIC = 0x1.8p52;
    double est = d[ND - 1];
#pragma unroll
    for (int k = ND - 2; k >= 0; --k) est = fma(est, B, d[k]);
    const double q = fma(est, c.inv_M, MAGIC) - MAGIC;
#pragma unroll
    for (int k = 0; k < ND; ++k) d[k] = fma(-q, c.Mc[k], d[k]);
#pragma unroll
    for (int k = 0; k + 1 < ND; ++k) {
        const double cy = fma(d[k], 0x1p-33, MAGIC) - MAGIC;
        d[k] = fma(-cy, B, d[k]);
        d[k + 1] += cy;
    }
    double t = d[ND - 1];  // |C'| <= K 2^(2P) < 2^135: what lies above digit 2 is an integer below 2^36, exact
#pragma unroll
    for (int k = ND - 2; k >= 3; --k) t = fma(t, B, d[k]);
    t *= B;
    const double hi = t + d[2], lost = d[2] - (hi - t);
    return fma(hi, 0x1p66, fma(lost, 0x1p66, fma(d[1], B, d[0])));
}

template <int N, bool CPLX>
__global__ void __launch_bounds__(256, N <= 18 ? 3 : 2) oz2_reconstruct_kernel(
    const uint8_t* __restrict__ R, long long M, long long cols, long long pitch, const double* __restrict__ rsc,
    const double* __restrict__ csc, double* __restrict__ C, long long ldc, double alpha, double beta,
    const __grid_constant__ Oz2Consts c) {
    constexpr int PAIRS = (N + 1) / 2, ND = N <= 18 ? 4 : 5, UNROLL = CPLX ? 2 : 4;
    // complex: even lanes take the real parts of four columns, odd lanes the imaginary
    // ones, and each stores two of the columns
    const int part = CPLX ? threadIdx.x & 1 : 0;
    const long long j0 = (CPLX ? blockIdx.x * 16ll + threadIdx.x / 2 : blockIdx.x * 32ll + threadIdx.x) * 4;
    const bool live = j0 < cols;
    const long long plane = M * pitch;
    const bool aligned = !CPLX || cols % 4 == 0;  // of the imaginary columns' bytes
    const bool vec = j0 + 4 <= cols && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (CPLX || ldc % 2 == 0);
    for (long long i = blockIdx.y * 8ll + threadIdx.y; i < M; i += gridDim.y * 8ll) {
        const uint8_t* r = R + i * pitch + part * cols + (live ? j0 : 0);
        uint32_t w[N];
        if (aligned || part == 0) {
#pragma unroll
            for (int l = 0; l < N; ++l) w[l] = *reinterpret_cast<const uint32_t*>(r + l * plane);
        } else {
#pragma unroll
            for (int l = 0; l < N; ++l) {
                w[l] = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j0 + u < cols) w[l] |= static_cast<uint32_t>(r[l * plane + u]) << (8 * u);
            }
        }
        const double rs = ldexp(rsc[i], -2 * c.P) * alpha;
        double o[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll UNROLL
        for (int u = 0; u < 4; ++u) {
            double d[ND];
#pragma unroll
            for (int k = 0; k < ND; ++k) d[k] = 0.0;
#pragma unroll
            for (int t = 0; t < PAIRS; ++t) {
                uint32_t f = ((w[2 * t] >> (8 * u)) & 0xFFu) * c.pm[t][0];
                if (2 * t + 1 < N) f += ((w[2 * t + 1 < N ? 2 * t + 1 : 0] >> (8 * u)) & 0xFFu) * c.pm[t][1];
                const double v = __hiloint2double(0x43300000, static_cast<int>(f)) - 0x1p52;
#pragma unroll
                for (int k = 0; k < ND; ++k) d[k] = fma(v, c.pW[t][k], d[k]);
            }
            const double x = oz2_rebuild<ND>(d, c) * rs * csc[j0 + u < cols ? j0 + u : 0];
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = u == q ? x : o[q];  // no run-time index into registers
        }
        if (CPLX) {
            const double a = __shfl_xor_sync(0xFFFFFFFFu, part ? o[0] : o[2], 1);
            const double b = __shfl_xor_sync(0xFFFFFFFFu, part ? o[1] : o[3], 1);
            const double re[2] = {part ? a : o[0], part ? b : o[1]}, im[2] = {part ? o[2] : a, part ? o[3] : b};
            double* dst = C + 2 * (i * ldc + j0 + 2 * part);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (j0 + 2 * part + u >= cols) break;
                double x = re[u], y = im[u];
                if (beta != 0.0) {
                    x = fma(beta, dst[2 * u], x);
                    y = fma(beta, dst[2 * u + 1], y);
                }
                if (vec) {
                    *reinterpret_cast<double2*>(dst + 2 * u) = make_double2(x, y);
                } else {
                    dst[2 * u] = x;
                    dst[2 * u + 1] = y;
                }
            }
        } else {
            double* dst = C + i * ldc + j0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (j0 + u >= cols) break;
                if (beta != 0.0) o[u] = fma(beta, dst[u], o[u]);
                if (!vec) dst[u] = o[u];
            }
            if (vec) {
                *reinterpret_cast<double2*>(dst) = make_double2(o[0], o[1]);
                *reinterpret_cast<double2*>(dst + 2) = make_double2(o[2], o[3]);
            }
        }
    }
}

}  // namespace fg

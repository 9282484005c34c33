// tc_rows.cuh -- split SGEMM (3xBF16) for few rows: C (M <= MP rows) = A B with
// B split into its bf16 slices on the way to the tensor core.
//
// With one row tile, B (K x N, f32) is used once, so what the shape cannot do
// without is reading B once from HBM.  The general path cuts B into bf16
// planes in a pass of its own and reads those back: three times the bytes (32
// x 8192 x 8192: 82 us for the pass + 57 us for the product, of 148; HBM floor
// 41).  Here the products run transposed, C^T = B^T A^T, with a tile of 128
// columns of B as the M side of tcgen05.mma and A's rows as its N side, and the M
// side comes from tensor memory: a converter thread owns one column of the
// tile, takes 64 consecutive k of it from shared memory (where TMA laid the rows
// of B as they are; lanes read neighbouring columns), cuts them into hi =
// bf16(x) and lo = bf16(x - hi), packs neighbouring k and stores them with
// tcgen05.st.  So the transpose costs nothing, the slices never touch shared
// memory, and MMA work shrinks with M (N = 16, 32 or 64).
//
// Warps 0-7 convert (two groups of four, a warp per TMEM lane quarter, on
// alternate K blocks of 64), 8-11 sum the K chunks in FP32 registers (round to
// nearest, as the other split kernels) and store, 12 loads B and A's bf16 planes
// by TMA, 13 issues the MMAs.  TMEM: 4 operand stages of 64 columns (32 hi, 32
// lo), then 4 accumulator buffers of MP columns.  Persistent; a unit is a column
// tile and a K range (split-K partials go to a workspace).  All waits are
// bounded, as in tc_gemm.cuh.
//
// Bound by HBM through bytes in flight: with each converter loading its column
// to registers a block ahead (64 KB in flight per SM) 32 x 8192 x 8192 took 67.5
// us, with six 32 KB TMA stages 48 us = 5.6 TB/s.  B whose rows are not 16-byte
// aligned comes by cp.async as aligned granules into four stages (32 x 8191 x 8191:
// 81 us a call, 64 aligned, 176 with the split pass; 4-byte cp.async of each
// thread's own column took 103).
#pragma once
#include "tc_gemm.cuh"

namespace fg {

struct TcRowsArgs {
    const float* B;
    long long ldb;
    float* C;              // output, or split-K partials (ldc = N, split_stride apart)
    long long ldc, split_stride;
    int M, N, K;
    int tiles, splits;     // column tiles of 128; K ranges
    int k_blocks, kb_per_split;
    int kchunk;            // K blocks per TMEM accumulation chunk
    float alpha, beta;
    DevStatus* status;
    unsigned long long timeout_ns;
};

// TMA: B's rows are 16-byte aligned and reach the converters through shared
// memory.
template <int MP_, bool TMA_>
struct TcRowsCfg {
    static constexpr int MP = MP_;              // rows of A (MMA N)
    static constexpr bool TMA = TMA_;
    static constexpr int BN = 128, BK = 64;
    static constexpr int STAGES = 4;            // TMEM operand stages
    static constexpr int B_STAGES = MP == 64 ? 3 : 4;  // shared stages of A's planes
    static constexpr int F_STAGES = !TMA ? 4 : MP < 64 ? 6 : 5;  // shared stages of B
    static constexpr int F_PITCH = TMA ? BN : BN + 4;            // floats per row
    static constexpr int F_BYTES = BK * F_PITCH * 4;
    static constexpr int PLANE = MP * 128;      // bytes of one plane's K block
    static constexpr int ACC_BUFS = 4;
    static constexpr int ACC0 = STAGES * 64;    // first accumulator column
    static constexpr int THREADS = 448;
    static_assert(ACC0 + ACC_BUFS * MP <= 512, "TMEM columns");
    static_assert(MP % 16 == 0, "UMMA N at M = 128");
};

template <class Cfg>
struct TcRowsSmem {
    alignas(1024) uint8_t a[Cfg::B_STAGES][2][Cfg::PLANE];
    alignas(128) uint8_t f[Cfg::F_STAGES][Cfg::F_BYTES];     // B as it lies: [64 k][128 columns] of f32
    uint64_t f_full[Cfg::F_STAGES], f_empty[Cfg::F_STAGES];
    uint64_t op_full[Cfg::STAGES], op_empty[Cfg::STAGES];    // TMEM operand stages
    uint64_t a_full[Cfg::B_STAGES], a_empty[Cfg::B_STAGES];  // A planes
    uint64_t acc_full[Cfg::ACC_BUFS], acc_empty[Cfg::ACC_BUFS];
    uint64_t drain;
    uint32_t tmem_base;
    int abort;
};

template <class Cfg>
constexpr size_t tc_rows_smem_bytes() {
    return sizeof(TcRowsSmem<Cfg>) + 1024;
}

// D[tmem] (+)= A[tmem] * B[smem], kind::f16, M = 128.
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 32 lanes x 8 consecutive 32-bit columns, thread t of the warp writing lane t.
__device__ __forceinline__ void tmem_st_32x32b_x8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// bf16 slices of two f32, packed (x0 in the low half): hi = bf16(x), lo =
// bf16(x - hi), both round-to-nearest-even (split_n of prep_kernels.cuh).
__device__ __forceinline__ void split_bf16_pair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(x1), "f"(x0));
    const float r0 = x0 - __uint_as_float(hi << 16);
    const float r1 = x1 - __uint_as_float(hi & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(r1), "f"(r0));
}

// Walks the K blocks of a CTA's units in order.
struct TcRowsWalk {
    int t, kb, kb1;
    __device__ __forceinline__ void unit(const TcRowsArgs& p) {
        const int s = t / p.tiles;
        kb = s * p.kb_per_split;
        kb1 = min(p.k_blocks, kb + p.kb_per_split);
    }
    __device__ __forceinline__ void start(const TcRowsArgs& p, int first) {
        t = first;
        kb = kb1 = 0;
        if (t < p.tiles * p.splits) unit(p);
    }
    __device__ __forceinline__ bool more(const TcRowsArgs& p) const { return t < p.tiles * p.splits; }
    __device__ __forceinline__ void next(const TcRowsArgs& p) {
        if (++kb == kb1) {
            t += gridDim.x;
            if (more(p)) unit(p);
        }
    }
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
    tc_rows_kernel(const __grid_constant__ CUtensorMap map_hi, const __grid_constant__ CUtensorMap map_lo,
                   const __grid_constant__ CUtensorMap map_b, const __grid_constant__ TcRowsArgs p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    TcRowsSmem<Cfg>& s = *reinterpret_cast<TcRowsSmem<Cfg>*>(base);
    constexpr int MP = Cfg::MP;

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    volatile int* abort = &s.abort;
    const int total = p.tiles * p.splits;

    if (threadIdx.x == 0) {
        for (int i = 0; i < Cfg::STAGES; ++i) {
            mbar_init(&s.op_full[i], 4);  // the four warps of a converter group
            mbar_init(&s.op_empty[i], 1);
        }
        for (int i = 0; i < Cfg::B_STAGES; ++i) {
            mbar_init(&s.a_full[i], 1);
            mbar_init(&s.a_empty[i], 1);
        }
        for (int i = 0; i < Cfg::F_STAGES; ++i) {
            mbar_init(&s.f_full[i], Cfg::TMA ? 1 : 128);  // else every thread of a group
            mbar_init(&s.f_empty[i], 4);
        }
        for (int i = 0; i < Cfg::ACC_BUFS; ++i) {
            mbar_init(&s.acc_full[i], 1);
            mbar_init(&s.acc_empty[i], 4);
        }
        mbar_init(&s.drain, 1);
        s.abort = 0;
        fence_mbar_init();
    }
    if (warp == 12 && lane == 0) {
        tma_prefetch_desc(&map_hi);
        tma_prefetch_desc(&map_lo);
        if (Cfg::TMA) tma_prefetch_desc(&map_b);
    }
    if (warp == 13) {
        tmem_alloc(&s.tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s.tmem_base;

    if (warp < 8) {
        // ------------------------------------------------ converters
        const int group = warp / 4, quad = warp % 4;
        TcRowsWalk w;
        w.start(p, blockIdx.x);
        if (group == 1 && w.more(p)) w.next(p);
        // Without TMA a group copies its own blocks, DEPTH ahead, as the aligned
        // 16-byte granules that hold each row (one more than a row has; the row
        // starts `float address mod 4` floats into its shared row).  A warp takes
        // 16 of the 64 rows.
        constexpr int DEPTH = Cfg::F_STAGES / 2;
        auto copy_block = [&](const TcRowsWalk& u, int slot) {
            const int n0 = u.t % p.tiles * Cfg::BN;
            auto granule = [&](int r, int j) {
                const int k = u.kb * Cfg::BK + r;
                const uintptr_t a = reinterpret_cast<uintptr_t>(p.B + (long long)k * p.ldb + n0);
                const int left = p.N - n0 + static_cast<int>(a / 4 % 4) - 4 * j;  // floats to the row's end
                const int f = k < p.K ? min(max(left, 0), 4) : 0;
                const uintptr_t src = f ? (a & ~uintptr_t(15)) + 16 * j : reinterpret_cast<uintptr_t>(p.B) & ~uintptr_t(15);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                 smem_u32(s.f[slot]) + (r * Cfg::F_PITCH + 4 * j) * 4),
                             "l"(src), "r"(f * 4)
                             : "memory");
            };
#pragma unroll 4
            for (int i = 0; i < 16; ++i) granule(quad + 4 * i, lane);
            if (lane < 16) granule(quad + 4 * lane, 32);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&s.f_full[slot]))
                         : "memory");
        };
        TcRowsWalk ahead = w;  // next block to copy
        auto ahead_next = [&] {
            ahead.next(p);
            if (ahead.more(p)) ahead.next(p);
        };
        if constexpr (!Cfg::TMA) {
#pragma unroll 1
            for (int d = 0; d < DEPTH && ahead.more(p); ++d) {
                copy_block(ahead, group + 2 * d);
                ahead_next();
            }
        }
        int it = group;  // K blocks of this CTA before this one
        bool ok = true;
        while (w.more(p)) {
            const int stage = it % Cfg::STAGES;
            const uint32_t par = static_cast<uint32_t>((it / Cfg::STAGES) & 1);
            const int fs = Cfg::TMA ? it % Cfg::F_STAGES : group + 2 * (it / 2 % DEPTH);
            if (!mbar_wait(&s.op_empty[stage], par ^ 1u, p.timeout_ns, p.status, 0x31, abort)) ok = false;
            const uint32_t fpar = static_cast<uint32_t>((Cfg::TMA ? it / Cfg::F_STAGES : it / 2 / DEPTH) & 1);
            if (ok && !mbar_wait(&s.f_full[fs], fpar, p.timeout_ns, p.status, 0x32, abort)) ok = false;
            if (!__all_sync(0xFFFFFFFFu, ok)) break;
            tc_fence_after();
            const uint32_t dst = tmem + (static_cast<uint32_t>(quad * 32) << 16) + stage * 64;
            const float* col = reinterpret_cast<const float*>(s.f[fs]) + quad * 32 + lane;
            // float address mod 4 of the block's first row, and its step per row
            const int sh0 = Cfg::TMA ? 0
                                     : static_cast<int>((reinterpret_cast<uintptr_t>(p.B) / 4 +
                                                         static_cast<uintptr_t>(w.kb) * Cfg::BK * p.ldb) % 4);
            const int dsh = Cfg::TMA ? 0 : static_cast<int>(p.ldb % 4);
            auto at = [&](int k) { return col[k * Cfg::F_PITCH + (Cfg::TMA ? 0 : (sh0 + k * dsh) & 3)]; };
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    split_bf16_pair(at(16 * c + 2 * i), at(16 * c + 2 * i + 1), hi[i], lo[i]);
                tmem_st_32x32b_x8(dst + c * 8, hi);
                tmem_st_32x32b_x8(dst + 32 + c * 8, lo);
            }
            __syncwarp();  // every lane has read its column
            if (lane == 0) mbar_arrive(&s.f_empty[fs]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s.op_full[stage]);
            if constexpr (!Cfg::TMA) {
                if (ahead.more(p)) {  // refill the stage once the whole group has read it
                    if (!mbar_wait(&s.f_empty[fs], fpar, p.timeout_ns, p.status, 0x33, abort)) ok = false;
                    if (!__all_sync(0xFFFFFFFFu, ok)) break;
                    copy_block(ahead, fs);
                    ahead_next();
                }
            }
            w.next(p);
            if (w.more(p)) w.next(p);
            it += 2;
        }
        if constexpr (!Cfg::TMA) asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < 12) {
        // ------------------------------------------------ epilogue
        const int quad = warp % 4;
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
            const int split = t / p.tiles, n = t % p.tiles * Cfg::BN + quad * 32 + lane;
            const int kb0 = split * p.kb_per_split, kb1 = min(p.k_blocks, kb0 + p.kb_per_split);
            float run[MP];
#pragma unroll
            for (int j = 0; j < MP; ++j) run[j] = 0.f;
            for (int kc0 = kb0; kc0 < kb1; kc0 += p.kchunk, ++it) {
                const int buf = it % Cfg::ACC_BUFS;
                const uint32_t par = static_cast<uint32_t>((it / Cfg::ACC_BUFS) & 1);
                if (!mbar_wait(&s.acc_full[buf], par, p.timeout_ns, p.status, 0x21, abort)) ok = false;
                ok = __all_sync(0xFFFFFFFFu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint32_t src = tmem + (static_cast<uint32_t>(quad * 32) << 16) + Cfg::ACC0 + buf * MP;
#pragma unroll
                for (int c = 0; c < MP / 16; ++c) {
                    uint32_t x[16];
                    tmem_ld_32x32b_x16(src + c * 16, x);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) run[c * 16 + j] = __fadd_rn(run[c * 16 + j], __uint_as_float(x[j]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s.acc_empty[buf]);
            }
            if (!ok) break;
            if (n < p.N) {
                float* dst = p.C + split * p.split_stride + n;
                if (p.beta != 0.f) {
#pragma unroll
                    for (int j = 0; j < MP; ++j)
                        if (j < p.M) dst[j * p.ldc] = fmaf(p.beta, dst[j * p.ldc], p.alpha * run[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < MP; ++j)
                        if (j < p.M) dst[j * p.ldc] = p.alpha * run[j];
                }
            }
        }
    } else if (warp == 12) {
        // ------------------------------------------------ TMA: A's planes, B
        if (elect_one()) {
            // One walk each: B's ring runs further ahead than the planes'.
            TcRowsWalk wa, wb;
            wa.start(p, blockIdx.x);
            wb.start(p, blockIdx.x);
            uint32_t na = 0, nb = 0;  // blocks issued
            bool ok = true;
            while (ok && (wa.more(p) || (Cfg::TMA && wb.more(p)))) {
                if (Cfg::TMA && wb.more(p) && nb < na + Cfg::F_STAGES) {
                    const uint32_t st = nb % Cfg::F_STAGES, ph = nb / Cfg::F_STAGES & 1;
                    if (!(ok = mbar_wait(&s.f_empty[st], ph ^ 1u, p.timeout_ns, p.status, 0x02, abort))) break;
                    mbar_arrive_expect_tx(&s.f_full[st], Cfg::F_BYTES);
                    tma_load_2d(s.f[st], &map_b, wb.t % p.tiles * Cfg::BN, wb.kb * Cfg::BK, &s.f_full[st]);
                    ++nb;
                    wb.next(p);
                    if (nb < na + Cfg::F_STAGES && wb.more(p)) continue;
                }
                if (wa.more(p)) {
                    const uint32_t st = na % Cfg::B_STAGES, ph = na / Cfg::B_STAGES & 1;
                    if (!(ok = mbar_wait(&s.a_empty[st], ph ^ 1u, p.timeout_ns, p.status, 0x01, abort))) break;
                    mbar_arrive_expect_tx(&s.a_full[st], 2 * Cfg::PLANE);
                    tma_load_2d(s.a[st][0], &map_hi, wa.kb * Cfg::BK, 0, &s.a_full[st]);
                    tma_load_2d(s.a[st][1], &map_lo, wa.kb * Cfg::BK, 0, &s.a_full[st]);
                    ++na;
                    wa.next(p);
                }
            }
            if (!ok) {  // every load issued lands before the CTA exits
                volatile int never = 0;
                for (uint32_t i = na > Cfg::B_STAGES ? na - Cfg::B_STAGES : 0; i < na; ++i)
                    mbar_wait(&s.a_full[i % Cfg::B_STAGES], i / Cfg::B_STAGES & 1, p.timeout_ns, nullptr, 0, &never);
                for (uint32_t i = nb > Cfg::F_STAGES ? nb - Cfg::F_STAGES : 0; i < nb; ++i)
                    mbar_wait(&s.f_full[i % Cfg::F_STAGES], i / Cfg::F_STAGES & 1, p.timeout_ns, nullptr, 0, &never);
            }
        }
    } else {
        // ------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(1u, 1u, 1u, 0u, 0u, 128, MP);
            int ib = 0, it = 0, stage = 0;  // K blocks, accumulator chunks, plane stage
            uint32_t phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
                const int split = t / p.tiles;
                const int kb0 = split * p.kb_per_split, kb1 = min(p.k_blocks, kb0 + p.kb_per_split);
                for (int kc0 = kb0; kc0 < kb1 && ok; kc0 += p.kchunk, ++it) {
                    const int buf = it % Cfg::ACC_BUFS;
                    const uint32_t apar = static_cast<uint32_t>((it / Cfg::ACC_BUFS) & 1);
                    if (!mbar_wait(&s.acc_empty[buf], apar ^ 1u, p.timeout_ns, p.status, 0x11, abort)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t acc = tmem + Cfg::ACC0 + buf * MP;
                    for (int kb = kc0; kb < min(kb1, kc0 + p.kchunk); ++kb, ++ib) {
                        const int os = ib % Cfg::STAGES;
                        const uint32_t opar = static_cast<uint32_t>((ib / Cfg::STAGES) & 1);
                        if (!mbar_wait(&s.a_full[stage], phase, p.timeout_ns, p.status, 0x12, abort) ||
                            !mbar_wait(&s.op_full[os], opar, p.timeout_ns, p.status, 0x14, abort)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t op = tmem + os * 64;  // hi, then lo 32 columns on
                        const uint32_t a_hi = smem_u32(s.a[stage][0]), a_lo = smem_u32(s.a[stage][1]);
                        // lo(A) hi(B) + hi(A) lo(B) + hi(A) hi(B), smallest first
#pragma unroll
                        for (int o = 0; o < 3; ++o) {
                            const uint32_t bop = op + (o == 1 ? 32 : 0);
                            const uint32_t aop = o == 0 ? a_lo : a_hi;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                tc_mma_f16_ts(acc, bop + kk * 8, umma_desc_sw128(aop + kk * 32, 16, 1024), idesc,
                                              (kb > kc0 || o > 0 || kk > 0) ? 1u : 0u);
                        }
                        tc_commit(&s.op_empty[os]);
                        tc_commit(&s.a_empty[stage]);
                        if (++stage == Cfg::B_STAGES) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                    if (!ok) break;
                    tc_commit(&s.acc_full[buf]);
                }
            }
            tc_commit(&s.drain);
            volatile int never = 0;
            mbar_wait(&s.drain, 0, p.timeout_ns, ok ? p.status : nullptr, 0x13, &never);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace fg

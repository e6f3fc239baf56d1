// Spectral Poisson solve as dense DCT / IDCT / IDXST matrix contractions on the
// 5th-generation tensor cores (tcgen05), in two precisions:
//   * TF32: fp32 operands read as TF32 by kind::tf32, FP32 accumulation;
//   * BF16x3: each operand split into bf16 hi + lo (x = hi + lo to ~16 bits),
//     three products hi.hi + hi.lo + lo.hi per k-step (kind::f16, bf16 inputs),
//     FP32 accumulation.
// The closed forms are those of the FFT path (src/dct2d.rs, src/idct2.rs,
// src/idct_idxst.rs, src/idxst_idct.rs, src/frequencies.rs):
//   A   = (4 / mn) C_m rho C_n^T,   C[k][i] = cos(pi k (2i+1) / 2N)
//   f_x = S_m (W_x . A) D_n^T,  f_y = D_m (W_y . A) S_n^T,  psi = D_m (W_p . A) D_n^T
//   D[i][u] = c_u cos(pi u (2i+1) / 2N), S[i][u] = c_u sin(pi u (2i+1) / 2N), c = (1, 2, 2, ...)
//   W_x = wu / 2k^2, W_y = wv / 2k^2, W_p = 1 / k^2, k^2 = wu^2 + wv^2, [0,0] -> 0.
// Every contraction is written C = A B^T with both operands K-major (row-major,
// K contiguous): the first GEMM of each 2-D transform stores its result
// transposed, which is the K-major operand of the second.
//
// A launch whose result is wanted transposed (the K-major operand of the next one)
// exchanges its operands instead: (A B^T)^T = B A^T, so every result is stored by rows.
//
// GEMM kernel: persistent CTAs, one per SM (their registers allow no second), over
// 128 x BN output tiles (tile_width).
// Thread 0 issues TMA tile loads (128-byte swizzle) into a ring of shared-memory
// stages; thread 32 issues the tcgen05.mma instructions into one of two FP32
// accumulators of BN columns in tensor memory and releases each stage with
// tcgen05.commit; eight warps read the other accumulator (tcgen05.ld, a row per
// thread) and store it meanwhile.  Every mbarrier wait is bounded (status bit
// kStatusWaitTimeout).
//
// What bounds it: up to 1024^2 the latency of the operands' way from L2 through the ring
// (0.3 us per 32 columns of K with 24 KB per CTA and step; at 1024^2 the L2 is at 14 to
// 19 % of its rate and the tensor pipe active for 12 to 56 % of the cycles); at 2048^2 the tensor cores with
// their last wave (2.5 waves of 128 x 256 tiles for three maps).  Measured against one
// CTA of 128 threads per tile with a shared-memory transpose in its epilogue, us per
// solve on the device: 2048^2 BF16x3 with the potential 476 -> 317, TF32 290 -> 229;
// 1024^2 96 -> 80 and 66 -> 64; 1024 x 512 TF32 56 -> 50; 512^2 BF16x3 50 -> 39.  Same bits.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "bf16_split.cuh"
#include "bulk_copy.cuh"
#include "erp_internal.cuh"

namespace erp {

namespace {

constexpr int kTile = 128;   // rows of an output tile (TMEM lanes); its columns are BN

struct GemmMaps {            // per z: A (hi, lo) and B (hi, lo); lo only for BF16x3
    CUtensorMap a[3][2];
    CUtensorMap b[3][2];
};

struct GemmEpi {
    int mode;                // 0: plain store, 1: weighted spectra (planes)
    int split;               // store bf16 hi/lo instead of fp32
    int lo_first;            // BF16x3: the product lo.hi before hi.lo
    int unit;                // bytes per store: every output row starts on such a boundary (32, 16 or 4)
    int nplanes;             // weighted mode: planes x, y (, p)
    float alpha;             // scale applied before storing
    int ldc;                 // row stride of the stored matrix (elements)
    void *out[3][2];         // per z (plain) or per plane (weighted): fp32 or bf16 hi, bf16 lo
    const float *wu, *wv;    // weighted mode: frequencies of rows (wu) and columns (wv)
    int *status;             // bounded-wait failure flag (kStatusWaitTimeout)
    int status_on_host;      // it is page-locked host memory: only ever set, by a plain store
};

// ---- PTX wrappers (tcgen05, TMA) ----
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile in shared memory: rows of 128 bytes, 128-byte swizzle
// (as TMA writes it), 8-row groups 1024 bytes apart.  sm_100 descriptor:
// start >> 4 [0,14), leading byte offset >> 4 [16,30) (unused for swizzled
// K-major layouts: 1), stride byte offset >> 4 [32,46), version 1 [46,48),
// layout SWIZZLE_128B = 2 [61,64).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// instruction descriptor: D FP32 [4,6) = 1; A, B format [7,10), [10,13)
// (TF32 = 2 for kind::tf32, BF16 = 1 for kind::f16); K-major A and B; N >> 3
// [17,23); M >> 4 [24,29) (M = 128).
__host__ __device__ constexpr uint32_t instr_desc(uint32_t ab_format, int bn) {
    return (1u << 4) | (ab_format << 7) | (ab_format << 10) | ((uint32_t)(bn >> 3) << 17) |
           ((uint32_t)(kTile >> 4) << 24);
}

template <int KIND, int BN>
__device__ __forceinline__ void mma_issue(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
    if (KIND == 0) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(a), "l"(b), "r"(instr_desc(2, BN)), "r"(accumulate)
            : "memory");
    } else {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
            "l"(a), "l"(b), "r"(instr_desc(1, BN)), "r"(accumulate)
            : "memory");
    }
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// 32 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 bytes to a 32-byte boundary in one instruction
__device__ __forceinline__ void store_sector(void *p, const uint32_t (&r)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
// eight words, `unit` bytes at a time (the same for a whole launch)
__device__ __forceinline__ void store_words(uint32_t *p, const uint32_t (&r)[8], int unit) {
    if (unit == 32) {
        store_sector(p, r);
    } else if (unit == 16) {
        reinterpret_cast<uint4 *>(p)[0] = make_uint4(r[0], r[1], r[2], r[3]);
        reinterpret_cast<uint4 *>(p)[1] = make_uint4(r[4], r[5], r[6], r[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) p[k] = r[k];
    }
}
// 32 consecutive elements of a matrix from element `at` on: fp32, or bf16 hi and lo
__device__ __forceinline__ void store_row(void *const (&out)[2], size_t at, const float (&x)[32], int split, int unit) {
    if (!split) {
        uint32_t *o = static_cast<uint32_t *>(out[0]) + at;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) r[k] = __float_as_uint(x[8 * q + k]);
            store_words(o + 8 * q, r, unit);
        }
        return;
    }
    uint32_t *oh = static_cast<uint32_t *>(out[0]) + at / 2, *ol = static_cast<uint32_t *>(out[1]) + at / 2;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        uint32_t h[8], l[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float a = x[16 * q + 2 * k], b = x[16 * q + 2 * k + 1];
            __nv_bfloat162 hi, lo;
            split_pair(a, b, hi, lo);
            memcpy(&h[k], &hi, 4);
            memcpy(&l[k], &lo, 4);
        }
        store_words(oh + 8 * q, h, unit);
        store_words(ol + 8 * q, l, unit);
    }
}

// Stage ring: A tile 128 x 128 bytes, B tile BN x 128 bytes (+ the lo parts
// for BF16x3), as many stages as fit in 200 KB; TF32 up to 128 columns in 100 KB (more
// stages measured no faster, and launches of short grids start later with 200 KB:
// 1024 x 512 solve 52.6 against 50.3 us).  Tensor memory: 2 BN of the SM's 512 columns
// per CTA.  Its registers (320 threads of 148) leave an SM room for one CTA; by shared
// memory alone it would be two of the 100 KB form, and kMostPerSm times 2 BN columns fit
// even then, so that no allocation waits for another's.
template <int KIND, int BN>
struct GemmCfg {
    static constexpr int kABytes = kTile * 128, kBBytes = BN * 128;
    static constexpr int kStageBytes = (KIND == 0 ? 1 : 2) * (kABytes + kBBytes);
    static constexpr int kBudget = KIND == 0 && BN <= 128 ? 100 : 200;
    static constexpr int kStages = kBudget * 1024 / kStageBytes;
    static constexpr int kBK = KIND == 0 ? 32 : 64;             // K elements per stage (128 bytes)
    static constexpr size_t kSmem = (size_t)kStages * kStageBytes + 1024;
    static constexpr int kMostPerSm = (int)(227 * 1024 / kSmem);
    static_assert(kMostPerSm >= 1 && kMostPerSm * 2 * BN <= 512, "the accumulators of an SM's CTAs fit its tensor memory");
};
constexpr int kGemmThreads = 320;   // TMA warp, MMA warp, eight epilogue warps

template <int KIND, int BN>
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm_nt(const __grid_constant__ GemmMaps maps, GemmEpi epi, int K,
                                                             int tiles_m, int tiles_n, int total) {
    using Cfg = GemmCfg<KIND, BN>;
    constexpr int S = Cfg::kStages;
    extern __shared__ uint8_t dsm[];
    __shared__ __align__(8) uint64_t full[S], empty[S], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(dsm) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KT = K / Cfg::kBK;

    // stage layout: A hi | B hi | A lo | B lo
    auto tile = [&](int s, int op) {
        const size_t off = (op & 1) ? Cfg::kABytes : 0;
        return base + (size_t)s * Cfg::kStageBytes + (size_t)(op >> 1) * (Cfg::kABytes + Cfg::kBBytes) + off;
    };
    // this CTA's output tiles: blockIdx.x, blockIdx.x + gridDim.x, ... of z-major rows of tiles
    struct Tile {
        int z, m, n;
    };
    auto tile_at = [&](int t) {
        const int z = t / (tiles_m * tiles_n), r = t - z * tiles_m * tiles_n;
        const int tm = r / tiles_n;
        return Tile{z, tm * kTile, (r - tm * tiles_n) * BN};
    };

    auto load_stage = [&](const Tile &tl, int kt, int s) {
        mbar_expect_tx(&full[s], (uint32_t)Cfg::kStageBytes);
        const int k0 = kt * Cfg::kBK;
        tma_load_2d(tile(s, 0), &maps.a[tl.z][0], k0, tl.m, &full[s]);
        tma_load_2d(tile(s, 1), &maps.b[tl.z][0], k0, tl.n, &full[s]);
        if (KIND == 1) {
            tma_load_2d(tile(s, 2), &maps.a[tl.z][1], k0, tl.m, &full[s]);
            tma_load_2d(tile(s, 3), &maps.b[tl.z][1], k0, tl.n, &full[s]);
        }
    };

    // The first tile's first stages are on their way while the tensor memory is being
    // allocated (more of them would hold up the barrier below).
    const int ahead = min(2, KT);
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < 2; ++k) {
            mbar_init(&acc_full[k], 1);
            mbar_init(&acc_empty[k], 8);   // one arrival per epilogue warp
        }
        failed = 0;
        const Tile first = tile_at(blockIdx.x);
        for (int kt = 0; kt < ahead; ++kt) load_stage(first, kt, kt);
    }
    if (warp == 1) {   // two accumulators of BN columns (GemmCfg: they fit)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base)),
                     "r"(2 * BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (tid == 0) {   // TMA producer
        int it = ahead, kt = ahead;
        bool ok = true;
        for (int t = blockIdx.x; t < total && ok; t += gridDim.x, kt = 0) {
            const Tile tl = tile_at(t);
            for (; kt < KT; ++kt, ++it) {
                const int s = it % S;
                ok = mbar_wait(&empty[s], ((uint32_t)(it / S) & 1u) ^ 1u);
                if (!ok) break;
                load_stage(tl, kt, s);
            }
        }
        if (!ok) {   // a wait ran out: the copies in flight land before the block leaves
            failed = 1;
            for (int k = it > S ? it - S : 0; k < it; ++k) mbar_wait(&full[k % S], (uint32_t)(k / S) & 1u);
        }
    } else if (tid == 32) {   // MMA issuer
        int it = 0, lt = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++lt) {
            const int buf = lt & 1;
            if (!mbar_wait(&acc_empty[buf], (((uint32_t)lt >> 1) & 1u) ^ 1u)) { failed = 1; break; }
            tc_fence_after();
            const uint32_t acc_at = tmem + (uint32_t)(buf * BN);
            bool ok = true;
            for (int kt = 0; kt < KT; ++kt, ++it) {
                const int s = it % S;
                const uint32_t ph = (uint32_t)(it / S) & 1u;
                if (!mbar_wait(&full[s], ph)) { failed = 1; ok = false; break; }
                tc_fence_after();
                const uint32_t a0 = smem_addr(tile(s, 0)), b0 = smem_addr(tile(s, 1));
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {   // 4 x 32 bytes of K per 128-byte row
                    const uint32_t acc = (kt > 0 || kk > 0) ? 1u : 0u;
                    if (KIND == 0) {
                        mma_issue<0, BN>(acc_at, sw128_desc(a0 + 32 * kk), sw128_desc(b0 + 32 * kk), acc);
                    } else {
                        const uint32_t a1 = smem_addr(tile(s, 2)), b1 = smem_addr(tile(s, 3));
                        const uint32_t ax = epi.lo_first ? a1 : a0, bx = epi.lo_first ? b0 : b1;
                        const uint32_t ay = epi.lo_first ? a0 : a1, by = epi.lo_first ? b1 : b0;
                        mma_issue<1, BN>(acc_at, sw128_desc(a0 + 32 * kk), sw128_desc(b0 + 32 * kk), acc);   // hi.hi
                        mma_issue<1, BN>(acc_at, sw128_desc(ax + 32 * kk), sw128_desc(bx + 32 * kk), 1u);    // hi.lo
                        mma_issue<1, BN>(acc_at, sw128_desc(ay + 32 * kk), sw128_desc(by + 32 * kk), 1u);    // lo.hi
                    }
                }
                mma_commit(&empty[s]);   // the stage is free once these MMAs have read it
            }
            mma_commit(&acc_full[buf]);
            if (!ok) break;
        }
    } else if (warp >= 2) {
        // Epilogue: warps w and w + 4 share the TMEM lanes of quarter w mod 4 and take
        // alternate blocks of 32 columns.  Each thread holds 32 columns of its row at a
        // time and stores them itself, a 32-byte sector per instruction (16 or 4 bytes
        // where a caller's buffer allows no more): no staging, and the weights of a row share
        // its wu.  The next tile's products run meanwhile in the other accumulator.
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const float al = epi.alpha;
        int lt = 0;
        for (int t = blockIdx.x; t < total; t += gridDim.x, ++lt) {
            const Tile tl = tile_at(t);
            const int buf = lt & 1;
            const int gr = tl.m + quarter * 32 + lane;   // this thread's row
            const float wu = epi.mode == 1 ? epi.wu[gr] : 0.0f;
            const bool ready = mbar_wait(&acc_full[buf], ((uint32_t)lt >> 1) & 1u);
            if (!__all_sync(0xffffffffu, ready)) {   // one decision per warp
                failed = 1;
                break;
            }
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 32 * half; c0 < BN; c0 += 64) {
                float v[32];
                tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * BN + c0), v);
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] *= al;
                const size_t at = (size_t)gr * epi.ldc + tl.n + c0;
                if (epi.mode == 0) {
                    store_row(epi.out[tl.z], at, v, epi.split, epi.unit);
                    continue;
                }
                // weighted spectra: row u = gr, column gc (planes x, y, p)
                float px[32], py[32];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float4 w4 = __ldg(reinterpret_cast<const float4 *>(epi.wv + tl.n + c0) + q);
                    const float wv4[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = 4 * q + e;
                        const float wv = wv4[e];
                        const float k2 = __fadd_rn(__fmul_rn(wu, wu), __fmul_rn(wv, wv));
                        const float ik = (gr | (tl.n + c0 + j)) == 0 ? 0.0f : __frcp_rn(k2);
                        const float x = v[j];
                        px[j] = x * (0.5f * wu * ik);
                        py[j] = x * (0.5f * wv * ik);
                        v[j] = x * ik;
                    }
                }
                store_row(epi.out[0], at, px, epi.split, epi.unit);
                store_row(epi.out[1], at, py, epi.split, epi.unit);
                if (epi.nplanes > 2) store_row(epi.out[2], at, v, epi.split, epi.unit);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (failed && tid == 0 && epi.status) {
        if (epi.status_on_host) *(volatile int *)epi.status = kStatusWaitTimeout;
        else atomicOr(epi.status, kStatusWaitTimeout);
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
    }
}

// hi and lo of the caller's input; VEC: four elements per thread from a 16-byte boundary
template <bool VEC>
__global__ void k_split_bf16(size_t count, const float *__restrict__ src, __nv_bfloat16 *__restrict__ hi,
                             __nv_bfloat16 *__restrict__ lo) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    if (VEC) {
        for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count / 4; i += step) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(src) + i);
            __nv_bfloat162 h[2], l[2];
            split_pair(v.x, v.y, h[0], l[0]);
            split_pair(v.z, v.w, h[1], l[1]);
            uint2 ph, pl;
            memcpy(&ph, h, 8);
            memcpy(&pl, l, 8);
            reinterpret_cast<uint2 *>(hi)[i] = ph;
            reinterpret_cast<uint2 *>(lo)[i] = pl;
        }
        return;
    }
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += step) {
        const float v = src[i];
        const __nv_bfloat16 h = __float2bfloat16_rn(v);
        hi[i] = h;
        lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
    }
}

// ---- host side ----
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_encode_mu;

bool get_encode() {
    std::lock_guard<std::mutex> lk(g_encode_mu);
    if (g_encode) return true;
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
        return false;
    g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    return true;
}

// row-major [rows][cols] matrix, box_rows x 128-byte boxes, 128-byte swizzle
bool make_map(CUtensorMap *map, const void *ptr, int rows, int cols, bool bf16, int box_rows = kTile) {
    const size_t es = bf16 ? 2 : 4;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * es};
    cuuint32_t box[2] = {(cuuint32_t)(128 / es), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return g_encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                    const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// A matrix operand: fp32 (TF32) or bf16 hi + lo (BF16x3)
struct GemmOperand {
    void *p[2] = {nullptr, nullptr};
};

struct DctGemmPlan {
    int m = 0, n = 0, kind = 0;   // kind 0: TF32, 1: BF16x3
    cudaStream_t stream = nullptr;
    GemmOperand Cn, Cm, Dn, Sn, Sm, Dm;   // transform matrices
    GemmOperand rho2;                     // BF16x3: split input
    GemmOperand Zt;                       // [n][m] after the first forward contraction
    GemmOperand Aw[3];                    // [m][n] weighted spectra x, y, p
    GemmOperand Zkt[3];                   // [n][m] after the first inverse contraction
    float *wu = nullptr, *wv = nullptr;
    int *h_status = nullptr;              // page-locked: set by a launch whose bounded wait ran out
    std::vector<void *> owned;
    const void *rho_cached = nullptr;     // TF32: the rho the first map was built for
    GemmMaps g1, g2, g3[2], g4[2];        // G3, G4: without and with the potential
    int bn[2], bn3[2], bn4[2];            // their output tiles' widths
};

static bool alloc_operand(DctGemmPlan &P, GemmOperand &o, size_t count) {
    const size_t es = P.kind == 0 ? sizeof(float) : sizeof(__nv_bfloat16);
    for (int h = 0; h < (P.kind == 0 ? 1 : 2); ++h) {
        if (cudaMalloc(&o.p[h], es * count) != cudaSuccess) return false;
        P.owned.push_back(o.p[h]);
    }
    return true;
}

static bool upload_operand(DctGemmPlan &P, GemmOperand &o, const std::vector<double> &v) {
    if (!alloc_operand(P, o, v.size())) return false;
    if (P.kind == 0) {
        std::vector<float> f(v.begin(), v.end());
        return cudaMemcpy(o.p[0], f.data(), sizeof(float) * f.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    }
    std::vector<__nv_bfloat16> hi(v.size()), lo(v.size());
    for (size_t i = 0; i < v.size(); ++i) {
        const float f = (float)v[i];
        hi[i] = __float2bfloat16_rn(f);
        lo[i] = __float2bfloat16_rn(f - __bfloat162float(hi[i]));
    }
    return cudaMemcpy(o.p[0], hi.data(), 2 * hi.size(), cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(o.p[1], lo.data(), 2 * lo.size(), cudaMemcpyHostToDevice) == cudaSuccess;
}

static bool set_maps(const DctGemmPlan &P, CUtensorMap (&dst)[2], const GemmOperand &o, int rows, int cols,
                     int box_rows = kTile) {
    for (int h = 0; h < (P.kind == 0 ? 1 : 2); ++h)
        if (!make_map(&dst[h], o.p[h], rows, cols, P.kind == 1, box_rows)) return false;
    if (P.kind == 0) dst[1] = dst[0];
    return true;
}

void dctgemm_destroy(DctGemmPlan *P) {
    if (!P) return;
    if (P->stream) cudaStreamSynchronize(P->stream);
    for (void *p : P->owned) cudaFree(p);
    if (P->h_status) cudaFreeHost(P->h_status);
    delete P;
}

// Width of the output tiles of a launch: the narrowest for which every tile has an SM
// of its own; else 256, whose operand reads from shared memory keep up with the tensor
// cores (per 16 columns of K, 128 bytes a cycle at 128 columns, 96 at 256).
// Measured, us per launch at widths 32 / 64 / 128 / 256:
//   BF16x3 512^2, K 512 (32 has 64 tiles)       8.8 / 9.3 / 10.4 / 14.7
//   TF32 1024^2 (64 has 128 tiles)               23.8 / 14.7 / 15.4 / 17.3
//   BF16x3 2048 x 1024 (128 has 128 tiles)       40.2 / 23.1 / 15.4 / 23.7
//   BF16x3 2048^2 (256 has 128 tiles)            128 / 76 / 42.5 / 40.4, three maps 376 / 201 / 117 / 108
static int tile_width(int M, int N, int Z) {
    for (int bn : {32, 64, 128})
        if ((long long)(M / kTile) * (N / bn) * Z <= 152) return bn;
    return N % 256 ? 128 : 256;
}

template <int KIND, int BN>
static bool prepare_gemm() {
    return cudaFuncSetAttribute(k_gemm_nt<KIND, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)GemmCfg<KIND, BN>::kSmem) == cudaSuccess;
}
static bool prepare_gemms() {
    return prepare_gemm<0, 32>() && prepare_gemm<0, 64>() && prepare_gemm<0, 128>() && prepare_gemm<0, 256>() &&
           prepare_gemm<1, 32>() && prepare_gemm<1, 64>() && prepare_gemm<1, 128>() && prepare_gemm<1, 256>();
}

// transform matrices (FP64 closed forms), buffers and the tensor maps that do
// not depend on the caller's input
DctGemmPlan *dctgemm_create(int m, int n, float bin_w, float bin_h, int kind, cudaStream_t stream,
                            std::string &err) {
    if (m % kTile || n % kTile || m < kTile || n < kTile) {
        err = "the tensor-core solve needs bin counts that are multiples of 128";
        return nullptr;
    }
    if (!get_encode()) {
        err = "cuTensorMapEncodeTiled is not available from the driver";
        return nullptr;
    }
    if (!prepare_gemms()) {
        err = "cudaFuncSetAttribute failed";
        return nullptr;
    }
    DctGemmPlan *P = new DctGemmPlan();
    P->m = m; P->n = n; P->kind = kind; P->stream = stream;
    const double pi = 3.14159265358979323846;
    auto dct2 = [&](int N) {   // C[k][i] = cos(pi k (2i+1) / 2N)
        std::vector<double> v((size_t)N * N);
        for (int k = 0; k < N; ++k)
            for (int i = 0; i < N; ++i) v[(size_t)k * N + i] = cos(pi * k * (2.0 * i + 1) / (2.0 * N));
        return v;
    };
    auto inv = [&](int N, bool sine) {   // [i][u] = c_u cos|sin(pi u (2i+1) / 2N)
        std::vector<double> v((size_t)N * N);
        for (int i = 0; i < N; ++i)
            for (int u = 0; u < N; ++u) {
                const double a = pi * u * (2.0 * i + 1) / (2.0 * N), c = u == 0 ? 1.0 : 2.0;
                v[(size_t)i * N + u] = c * (sine ? sin(a) : cos(a));
            }
        return v;
    };
    const size_t mn = (size_t)m * n;
    bool ok = upload_operand(*P, P->Cn, dct2(n)) && upload_operand(*P, P->Cm, dct2(m)) &&
              upload_operand(*P, P->Dn, inv(n, false)) && upload_operand(*P, P->Sn, inv(n, true)) &&
              upload_operand(*P, P->Sm, inv(m, true)) && upload_operand(*P, P->Dm, inv(m, false)) &&
              alloc_operand(*P, P->Zt, mn);
    for (int k = 0; ok && k < 3; ++k) ok = alloc_operand(*P, P->Aw[k], mn) && alloc_operand(*P, P->Zkt[k], mn);
    if (ok && kind == 1) ok = alloc_operand(*P, P->rho2, mn);
    std::vector<float> hu(m), hv(n);   // frequencies as the FFT path builds them
    const float tpm = (float)(2.0 * pi) / (float)m, tpn = (float)(2.0 * pi) / (float)n, wv_div = bin_w / bin_h;
    for (int i = 0; i < m; ++i) hu[i] = (float)i * tpm;
    for (int j = 0; j < n; ++j) hv[j] = ((float)j * tpn) * wv_div;
    ok = ok && cudaMalloc(&P->wu, sizeof(float) * m) == cudaSuccess;
    if (ok) P->owned.push_back(P->wu);
    ok = ok && cudaMalloc(&P->wv, sizeof(float) * n) == cudaSuccess;
    if (ok) P->owned.push_back(P->wv);
    ok = ok && cudaMallocHost((void **)&P->h_status, sizeof(int)) == cudaSuccess;
    if (ok) *P->h_status = 0;
    ok = ok && cudaMemcpy(P->wu, hu.data(), sizeof(float) * m, cudaMemcpyHostToDevice) == cudaSuccess &&
         cudaMemcpy(P->wv, hv.data(), sizeof(float) * n, cudaMemcpyHostToDevice) == cudaSuccess;
    // maps: G1 A = C_n, B = rho (per call for TF32, rho2 for BF16x3);  G2 A = C_m, B = Zt;
    // G3 A = D_n / S_n / D_n, B = Aw[k];  G4 A = S_m / D_m / D_m, B = Zkt[k].  G1 and G3
    // give their results transposed.
    P->bn[0] = tile_width(n, m, 1);
    P->bn[1] = tile_width(m, n, 1);
    ok = ok && set_maps(*P, P->g1.a[0], P->Cn, n, n) && set_maps(*P, P->g2.a[0], P->Cm, m, m) &&
         set_maps(*P, P->g2.b[0], P->Zt, n, m, P->bn[1]);
    if (ok && kind == 1) ok = set_maps(*P, P->g1.b[0], P->rho2, m, n, P->bn[0]);
    const GemmOperand *b3[3] = {&P->Dn, &P->Sn, &P->Dn}, *a4[3] = {&P->Sm, &P->Dm, &P->Dm};
    for (int v = 0; v < 2; ++v) {   // without and with the potential
        P->bn3[v] = tile_width(n, m, 2 + v);
        P->bn4[v] = tile_width(m, n, 2 + v);
        for (int k = 0; ok && k < 2 + v; ++k)
            ok = set_maps(*P, P->g3[v].a[k], *b3[k], n, n) && set_maps(*P, P->g3[v].b[k], P->Aw[k], m, n, P->bn3[v]) &&
                 set_maps(*P, P->g4[v].a[k], *a4[k], m, m) && set_maps(*P, P->g4[v].b[k], P->Zkt[k], n, m, P->bn4[v]);
    }
    if (!ok) {
        err = "tensor-core solve set-up failed";
        dctgemm_destroy(P);
        return nullptr;
    }
    return P;
}

template <int KIND, int BN>
static cudaError_t launch_gemm(const GemmMaps &maps, const GemmEpi &epi, int M, int N, int K, int Z, cudaStream_t s) {
    const int tm = M / kTile, tn = N / BN, total = tm * tn * Z;
    k_gemm_nt<KIND, BN><<<std::min(total, 152), kGemmThreads, GemmCfg<KIND, BN>::kSmem, s>>>(maps, epi, K, tm, tn, total);
    return cudaGetLastError();
}

static cudaError_t run_gemm(const DctGemmPlan &P, const GemmMaps &maps, const GemmEpi &epi, int M, int N, int K,
                            int Z, int bn, cudaStream_t s) {
#define G(B) P.kind == 0 ? launch_gemm<0, B>(maps, epi, M, N, K, Z, s) : launch_gemm<1, B>(maps, epi, M, N, K, Z, s)
    if (bn == 32) return G(32);
    if (bn == 64) return G(64);
    if (bn == 128) return G(128);
    return G(256);
}

// Where a BF16x3 solve reads its input's hi and lo parts from; a caller that writes them
// itself passes rho = nullptr to dctgemm_solve.  False: the plan is TF32.
bool dctgemm_input_parts(const DctGemmPlan &P, void **hi, void **lo) {
    *hi = P.rho2.p[0];
    *lo = P.rho2.p[1];
    return P.kind == 1;
}

// fx, fy (, psi) = Poisson solve of rho: four contraction launches (+ the split
// of rho).  Returns cudaErrorTimeout when a bounded wait of an earlier solve
// on this plan ran out.
//
// status: where the contractions report a bounded wait that ran out; nullptr
// uses the plan's own word, in page-locked host memory that the device writes (a
// placement context passes its DevState status, read by the host with the rest of
// the state).
cudaError_t dctgemm_solve(DctGemmPlan &P, const float *rho, float *fx, float *fy, float *psi, int *status, cudaStream_t s) {
    if (!status && *(volatile int *)P.h_status) return cudaErrorTimeout;
    const int m = P.m, n = P.n, nk = psi ? 3 : 2;
    const size_t mn = (size_t)m * n;
    const bool split = P.kind == 1;
    cudaError_t e = cudaSuccess;
    if (split) {
        if (rho) {   // else the caller has filled the parts (dctgemm_input_parts)
            const bool vec = (reinterpret_cast<uintptr_t>(rho) & 15) == 0;   // mn is a multiple of 4
            (vec ? k_split_bf16<true> : k_split_bf16<false>)<<<152 * 8, 256, 0, s>>>(
                mn, rho, (__nv_bfloat16 *)P.rho2.p[0], (__nv_bfloat16 *)P.rho2.p[1]);
            if ((e = cudaGetLastError()) != cudaSuccess) return e;
        }
    } else if (rho != P.rho_cached) {
        if (!make_map(&P.g1.b[0][0], rho, m, n, false, P.bn[0])) return cudaErrorInvalidValue;
        P.g1.b[0][1] = P.g1.b[0][0];
        P.rho_cached = rho;
    }
    GemmEpi ep;
    memset(&ep, 0, sizeof ep);
    ep.status = status ? status : P.h_status;
    ep.status_on_host = status ? 0 : 1;
    ep.split = split ? 1 : 0;
    ep.unit = 32;   // the plan's own buffers
    // G1: Z^T = C_n rho^T [n][m] (the operands' order gives the transpose; lo_first keeps
    // the order of the products rho hi . C_n lo, rho lo . C_n hi)
    ep.mode = 0; ep.lo_first = 1; ep.alpha = 1.0f; ep.ldc = m;
    ep.out[0][0] = P.Zt.p[0]; ep.out[0][1] = P.Zt.p[1];
    if ((e = run_gemm(P, P.g1, ep, n, m, n, 1, P.bn[0], s)) != cudaSuccess) return e;
    // G2: A = (4/mn) C_m Z, written as the weighted spectra [m][n]
    ep.mode = 1; ep.lo_first = 0; ep.alpha = (float)(4.0 / ((double)m * (double)n)); ep.ldc = n;
    ep.nplanes = nk; ep.wu = P.wu; ep.wv = P.wv;
    for (int k = 0; k < 3; ++k) { ep.out[k][0] = P.Aw[k].p[0]; ep.out[k][1] = P.Aw[k].p[1]; }
    if ((e = run_gemm(P, P.g2, ep, m, n, m, 1, P.bn[1], s)) != cudaSuccess) return e;
    // G3: Z_k^T = (D_n | S_n | D_n) Aw_k^T [n][m]
    ep.mode = 0; ep.lo_first = 1; ep.alpha = 1.0f; ep.ldc = m; ep.nplanes = 0;
    for (int k = 0; k < 3; ++k) { ep.out[k][0] = P.Zkt[k].p[0]; ep.out[k][1] = P.Zkt[k].p[1]; }
    if ((e = run_gemm(P, P.g3[nk - 2], ep, n, m, n, nk, P.bn3[nk - 2], s)) != cudaSuccess) return e;
    // G4: field_x = S_m Z_x, field_y = D_m Z_y, psi = D_m Z_p, fp32 [m][n], the caller's buffers
    ep.split = 0; ep.lo_first = 0; ep.ldc = n;
    float *outs[3] = {fx, fy, psi};
    uintptr_t low = 0;
    for (int k = 0; k < nk; ++k) {
        ep.out[k][0] = outs[k];
        ep.out[k][1] = nullptr;
        low |= reinterpret_cast<uintptr_t>(outs[k]);
    }
    ep.unit = low & 15 ? 4 : (low & 31 ? 16 : 32);
    if ((e = run_gemm(P, P.g4[nk - 2], ep, m, n, m, nk, P.bn4[nk - 2], s)) != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace erp

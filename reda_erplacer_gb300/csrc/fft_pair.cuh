// FFT of one complex sequence of N = 64 .. 4096 points by N / R1 threads with R1
// points each, in registers; the spectral passes (k_spectral.cu) pack two real
// sequences into each complex one.
//
// N = R1 R2 R3, decimation in frequency: a DFT of R1 points per thread (stride
// M = N / R1), the twiddles W_N^(t q), then per q a transform of M = R2 R3 points
// by the same rule.  With z[n], n = t + M j:
//   after stage 1   slot (q1, t)      t < M
//   after stage 2   slot (q1, q2, o)  o < R3
//   result          Z[q1 + R1 (q2 + R2 q3)]
// so two exchanges through shared memory carry a whole transform.  8 or 16 points
// per thread (4 at side 64, where a grid has too few threads otherwise): the exchanges and their barriers were
// what bounded the four-warp radix-4 / shuffle form this replaced (barrier and
// short-scoreboard stalls 3.6 to 5 of 8 to 11 cycles per issue at 1024^2, 16
// shared-memory words per point against 6).
//
// Shared layout: P sequences of a block interleave point by point (slot f of
// sequence p at f P + p), and threads run over p first, then q1, so every access
// of a half-warp (16 words of 8 bytes) covers P x q1 lanes.  Slot offsets within a
// q1 row are XORed with a function of q1 that spreads those lanes over the banks:
// all accesses are conflict-free, but for two-way ones of the last read at P = 1,
// N = 256 and 512, and P = 2, N = 64.
#pragma once

#include <stdint.h>

namespace erp {

// The split of each length, also for the host's tables.
__host__ __device__ constexpr int fft_r1(int n) { return n == 64 ? 4 : (n <= 512 ? 8 : 16); }
__host__ __device__ constexpr int fft_r2(int n) { return n == 64 ? 4 : (n <= 1024 ? 8 : 16); }
__host__ __device__ constexpr int fft_r3(int n) { return n / (fft_r1(n) * fft_r2(n)); }
// Twiddles of a length in stage order: W_N^(t q) at (q - 1) M + t for 1 <= q < R1,
// t < M, then W_M^(o q) at (q - 1) R3 + o for 1 <= q < R2, o < R3; fewer than n.
__host__ __device__ constexpr int fft_tw1(int n) { return (fft_r1(n) - 1) * (n / fft_r1(n)); }
__host__ __device__ constexpr int fft_tw_len(int n) { return fft_tw1(n) + (fft_r2(n) - 1) * fft_r3(n); }
// The angle of twiddle k < fft_tw_len(n) as a fraction num / n of a turn (clockwise).
__host__ __device__ constexpr int fft_tw_num(int n, int k) {
    const int m = n / fft_r1(n), r3 = fft_r3(n), k2 = k - fft_tw1(n);
    return k2 < 0 ? (k / m + 1) * (k % m) : (k2 / r3 + 1) * (k2 % r3) * fft_r1(n);
}

#if defined(__CUDACC__)

// Every product below is an explicit intrinsic, so the compiler contracts nothing
// and each instantiation of a pass computes the same bits.
__device__ __forceinline__ float2 c_add(float2 a, float2 b) {
    return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y));
}
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) {
    return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y));
}
// a w (forward) or a conj(w) (inverse)
template <bool INV>
__device__ __forceinline__ float2 c_mul(float2 a, float2 w) {
    if (INV) return make_float2(__fmaf_rn(a.x, w.x, __fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, -__fmul_rn(a.x, w.y)));
    return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
}
// a W_4 (forward: -i a; inverse: i a)
template <bool INV>
__device__ __forceinline__ float2 c_quarter(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// a W_8 and a W_8^3
template <bool INV>
__device__ __forceinline__ float2 c_eighth(float2 a) {
    constexpr float r = 0.70710678118654752440f;
    const float s = __fadd_rn(a.x, a.y), d = __fsub_rn(a.y, a.x);
    return INV ? make_float2(__fmul_rn(-r, d), __fmul_rn(r, s)) : make_float2(__fmul_rn(r, s), __fmul_rn(r, d));
}
template <bool INV>
__device__ __forceinline__ float2 c_eighth3(float2 a) {
    constexpr float r = 0.70710678118654752440f;
    const float s = __fadd_rn(a.x, a.y), d = __fsub_rn(a.y, a.x);
    return INV ? make_float2(__fmul_rn(-r, s), __fmul_rn(-r, d)) : make_float2(__fmul_rn(r, d), __fmul_rn(-r, s));
}

template <bool INV>
__device__ __forceinline__ void dft4(float2 &a0, float2 &a1, float2 &a2, float2 &a3) {
    const float2 s0 = c_add(a0, a2), s1 = c_sub(a0, a2), s2 = c_add(a1, a3), s3 = c_quarter<INV>(c_sub(a1, a3));
    a0 = c_add(s0, s2);
    a1 = c_add(s1, s3);
    a2 = c_sub(s0, s2);
    a3 = c_sub(s1, s3);
}

// R-point DFT of v[0..R), in place, natural order in and out
template <int R, bool INV>
__device__ __forceinline__ void dft(float2 *v) {
    if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = c_add(a, b);
        v[1] = c_sub(a, b);
    } else if constexpr (R == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        dft4<INV>(v[0], v[2], v[4], v[6]);
        dft4<INV>(v[1], v[3], v[5], v[7]);
        const float2 o0 = v[1], o1 = c_eighth<INV>(v[3]), o2 = c_quarter<INV>(v[5]), o3 = c_eighth3<INV>(v[7]);
        const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
        v[0] = c_add(e0, o0); v[1] = c_add(e1, o1); v[2] = c_add(e2, o2); v[3] = c_add(e3, o3);
        v[4] = c_sub(e0, o0); v[5] = c_sub(e1, o1); v[6] = c_sub(e2, o2); v[7] = c_sub(e3, o3);
    } else {
        static_assert(R == 16, "radix");
        const float2 w1 = make_float2(0.92387953251128675613f, -0.38268343236508977173f);   // W_16
        const float2 w3 = make_float2(0.38268343236508977173f, -0.92387953251128675613f);   // W_16^3
        const float2 w9 = make_float2(-0.92387953251128675613f, 0.38268343236508977173f);   // W_16^9
#pragma unroll
        for (int b = 0; b < 4; ++b) dft4<INV>(v[b], v[b + 4], v[b + 8], v[b + 12]);   // over a of x[4 a + b]
        v[5] = c_mul<INV>(v[5], w1);        // slot b + 4 k1 holds k1 of column b: twiddle W_16^(b k1)
        v[6] = c_eighth<INV>(v[6]);
        v[7] = c_mul<INV>(v[7], w3);
        v[9] = c_eighth<INV>(v[9]);
        v[10] = c_quarter<INV>(v[10]);
        v[11] = c_eighth3<INV>(v[11]);
        v[13] = c_mul<INV>(v[13], w3);
        v[14] = c_eighth3<INV>(v[14]);
        v[15] = c_mul<INV>(v[15], w9);
        float2 u[16];
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            dft4<INV>(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) u[k1 + 4 * k2] = v[4 * k1 + k2];
        }
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = u[k];
    }
}

// A read-only load that stays where it is written.  Up to side 1024 a pass is one wave
// of few warps, so it issues all its loads before the first use (left to itself the
// compiler saves registers and waits several times: rows inverse at 1024^2 7.7 us,
// 5.4 us this way); larger sides have warps enough, and registers matter more.
__device__ __forceinline__ float2 ld_now(const float2 *p) {
    float2 v;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_now(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

template <int N, int P>
struct PairFft {
    static constexpr int R1 = fft_r1(N), R2 = fft_r2(N), R3 = fft_r3(N), M = N / R1, T = M;
    static constexpr int THREADS = P * T;
    static_assert(THREADS >= 32 && THREADS <= 1024 && R1 % R2 == 0 && R1 % R3 == 0 && R2 * R3 == M, "shape");
    static __device__ __forceinline__ void sync() {
        if (THREADS == 32) __syncwarp();
        else __syncthreads();
    }
    // bank spread of row q1 (see above); stays below M
    static __device__ __forceinline__ constexpr int spread(int q1) {
        constexpr int SLOT = P >= 16 ? 1 : 16 / P;
        return (R1 >= SLOT ? (q1 & (SLOT - 1)) : q1 * (SLOT / R1)) & (M - 1);
    }
    // Index of the result that v[e] holds after run().
    static __device__ __forceinline__ int out_index(int t, int e) {
        return t % R1 + R1 * (t / R1 + (e / R3) * (T / R1) + R2 * (e % R3));
    }
    static constexpr bool kEarly = N <= 1024;
    // This thread's stage-1 twiddles, loaded ahead of the transform (kEarly).
    static __device__ __forceinline__ void load_tw1(float2 (&w)[R1], const float2 *__restrict__ tw, int t) {
#pragma unroll
        for (int q = 1; kEarly && q < R1; ++q) w[q] = ld_now(tw + (q - 1) * M + t);
    }
    template <typename V>
    static __device__ __forceinline__ V load(const V *p) {
        if constexpr (kEarly) return ld_now(p);
        else return __ldg(p);
    }
    // An element that the same kernel writes later (WRITTEN), or that no pass of it does.
    template <bool WRITTEN>
    static __device__ __forceinline__ float load_elem(const float *p) {
        if constexpr (WRITTEN) {
            float v;
            asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
            return v;
        } else {
            return load(p);
        }
    }
    // A pair of the pass before: WRITTEN in the same kernel, or by an earlier one.
    template <bool WRITTEN>
    static __device__ __forceinline__ float2 load_pair(const float2 *p) {
        if constexpr (WRITTEN) {
            float2 v;
            asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
            return v;
        } else {
            return load(p);
        }
    }
    // v[j] = z[t + M j] in, v[e] = Z[out_index(t, e)] out.  A: N P slots, free on
    // entry (every thread of the block past its last use) and still being read by
    // other threads on return.  tw: this length's stage twiddles; w1: load_tw1's.
    template <bool INV>
    static __device__ __forceinline__ void run(float2 (&v)[R1], const float2 (&w1)[R1], float2 *A,
                                               const float2 *__restrict__ tw, int t, int p) {
        dft<R1, INV>(v);
#pragma unroll
        for (int q = 0; q < R1; ++q)
            A[(q * M + (t ^ spread(q))) * P + p] = q ? c_mul<INV>(v[q], kEarly ? w1[q] : __ldg(tw + (q - 1) * M + t)) : v[0];
        sync();
        const int q1 = t % R1, x = spread(q1);
        float2 *row = A + q1 * M * P + p;
#pragma unroll
        for (int i = 0; i < R1 / R2; ++i) {
            const int o = t / R1 + i * (T / R1);
            float2 *w = v + i * R2;
#pragma unroll
            for (int j = 0; j < R2; ++j) w[j] = row[((o + j * R3) ^ x) * P];
            dft<R2, INV>(w);
            // the butterfly's own slots: no other thread reads them before the barrier
#pragma unroll
            for (int q = 0; q < R2; ++q)
                row[((q * R3 + o) ^ x) * P] =
                    q ? c_mul<INV>(w[q], __ldg(tw + fft_tw1(N) + (q - 1) * R3 + o)) : w[0];
        }
        sync();
#pragma unroll
        for (int i = 0; i < R1 / R3; ++i) {
            const int q2 = t / R1 + i * (T / R1);
            float2 *w = v + i * R3;
#pragma unroll
            for (int j = 0; j < R3; ++j) w[j] = row[((q2 * R3 + j) ^ x) * P];
            dft<R3, INV>(w);
        }
    }
};

#endif  // __CUDACC__

}  // namespace erp

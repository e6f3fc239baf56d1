// Spectral Poisson solve of compute_potential (src/epotential.rs:284-343) as
// three shared-memory FFT passes over the bin grid (row index = x bin, m rows;
// column index = y bin, n columns; src/epotential.rs:237-238):
//
//   R1  rows, length n:    t1 = DCT-II_n(rho)                 (rho fused from the
//                          int64 density map + fixed-cell map, with the overflow sum)
//   C1  columns, length m: A  = (4/(mn)) DCT-II_m(t1); then per column the
//                          weighted spectra A*wu/2k^2, A*wv/2k^2 (and A/k^2) go
//                          through IDXST_m / IDCT_m (/ IDCT_m)       -> tx, ty (tp)
//   R2  rows, length n:    field_x = IDCT_n(tx), field_y = IDXST_n(ty), psi = IDCT_n(tp)
//
// The per-axis transforms are the closed forms of the reference pipelines
// (dct2_fft2 / idxst_idct / idct_idxst / idct2, src/dct2d.rs, src/idct2.rs,
// src/idct_idxst.rs, src/idxst_idct.rs, checked separable by impulse probing):
//   DCT-II  y[k] = sum_i x[i] cos(pi k (2i+1) / 2N)                 (x 2/N per axis)
//   IDCT    y[i] = sum_u c_u X[u] cos(pi u (2i+1) / 2N),  c = (1, 2, 2, ...)
//   IDXST   y[i] = sum_u c_u X[u] sin(pi u (2i+1) / 2N) = (-1)^i IDCT(X')[i],
//           X'[0] = 0, X'[u] = X[N-u]
// Each is computed with Makhoul's length-N complex FFT; two real rows (or
// columns) share one complex FFT (real + imaginary part), since the forward
// input is real and the inverse spectra are Hermitian.  Sides 64..4096 run the
// register FFT of fft_pair.cuh; sides 16 and 32 an in-place radix-2
// decimation-in-frequency pass in shared memory (natural order in, bit-reversed
// order out).  Twiddles come from FP64-computed tables.
#include <algorithm>

#include "erp_internal.cuh"
#include "bf16_split.cuh"
#include "bulk_copy.cuh"
#include "fft_pair.cuh"
#include "fixedpoint.h"
#include "reduce.cuh"

namespace erp {

__device__ __forceinline__ int brev(int k, int logN) { return (int)(__brev((unsigned)k) >> (32 - logN)); }

// In-place radix-2 DIF over nseq sequences of length N (buf[q*N + i]).
template <bool INV>
__device__ __forceinline__ void fft_dif(float2 *buf, int nseq, int N, int logN, const float2 *tw) {
    const int half = N >> 1;
    const int nbf = nseq * half;
    for (int s = 0; s < logN; ++s) {
        const int lh = logN - 1 - s;
        const int h = 1 << lh;
        for (int b = threadIdx.x; b < nbf; b += blockDim.x) {
            const int q = b >> (logN - 1);
            const int r = b & (half - 1);
            const int j = r & (h - 1);
            const int i0 = (q << logN) + ((r >> lh) << (lh + 1)) + j;
            const int i1 = i0 + h;
            const float2 a = buf[i0], c = buf[i1];
            float2 w = tw[j << s];
            if (INV) w.y = -w.y;
            const float dx = a.x - c.x, dy = a.y - c.y;
            buf[i0] = make_float2(a.x + c.x, a.y + c.y);
            buf[i1] = make_float2(dx * w.x - dy * w.y, dx * w.y + dy * w.x);
        }
        __syncthreads();
    }
}

__device__ __forceinline__ int makhoul_pos(int i, int N) { return (i & 1) ? (N - 1 - (i >> 1)) : (i >> 1); }

// IDCT spectrum Vi[u] = e^{i pi u / 2N} (X[u] - i X[N-u]); e = ek[u] = (cos, -sin)
__device__ __forceinline__ float2 idct_spec(float xu, float xnu, float2 e) {
    const float c = e.x, s = -e.y;
    return make_float2(c * xu + s * xnu, s * xu - c * xnu);
}

// The maps between the passes (t1, tx, ty, tp) keep two rows interleaved: rows at
// Makhoul positions 2 q and 2 q + 1 of the column transform form row q of n pairs.
// The pair passes below read and write both rows with one 8-byte access.
__device__ __forceinline__ size_t pair_at(int i, int j, int m, int n) {
    const int k = makhoul_pos(i, m);
    return ((size_t)(k >> 1) * n + j) * 2 + (k & 1);
}

// ---------------- R1: rows forward DCT-II ----------------
// PAIRS row pairs per block.  Input either the density map (int64 fixed point +
// fixed-cell map, converted exactly as the oracle replays it) or rho directly.
template <int PAIRS>
__global__ void __launch_bounds__(kThreads) k_rows_dct_r2(
    int m, int n, int logn, const float2 *__restrict__ tw_g, const float2 *__restrict__ ek_n,
    const float *__restrict__ rho_in, unsigned long long *__restrict__ dmap,
    const float *__restrict__ initial, float fixed_inv, float coef, float inv_area, int zero_map,
    float *__restrict__ rho_out, float *__restrict__ t1, double *__restrict__ partials,
    DevState *__restrict__ st, double movable_area, int step) {
    if (st && st->done) return;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm;
    float2 *buf = sm + (n >> 1);
    __shared__ double shr[kThreads / 32];
    for (int k = threadIdx.x; k < (n >> 1); k += blockDim.x) tw[k] = tw_g[k];
    const int row0 = blockIdx.x * 2 * PAIRS;
    Df ovf = df_zero();
    for (int idx = threadIdx.x; idx < PAIRS * n; idx += blockDim.x) {
        const int p = idx >> logn, i = idx & (n - 1);
        float v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r = row0 + 2 * p + h;
            const size_t k = (size_t)r * n + i;
            if (rho_in) {
                v[h] = rho_in[k];
            } else {
                const unsigned long long q = dmap[k];
                if (zero_map) dmap[k] = 0ull;
                // d = (float)sum * 2^-S + initial  (src/density.rs:231-236, fixed point)
                const float d = __fadd_rn(__fmul_rn(fxp_u64_to_float(q), fixed_inv), initial[k]);
                const float o = __fsub_rn(d, coef);
                ovf = df_add(ovf, o > 0.0f ? o : 0.0f);    // src/epotential.rs:274-276
                v[h] = __fmul_rn(d, inv_area);               // src/epotential.rs:284-285
                if (rho_out) rho_out[k] = v[h];
            }
        }
        buf[(p << logn) + makhoul_pos(i, n)] = make_float2(v[0], v[1]);
    }
    __syncthreads();
    fft_dif<false>(buf, PAIRS, n, logn, tw);
    for (int idx = threadIdx.x; idx < PAIRS * n; idx += blockDim.x) {
        const int p = idx >> logn, k = idx & (n - 1);
        const int kk = (n - k) & (n - 1);
        const float2 A = buf[(p << logn) + brev(k, logn)];
        float2 B = buf[(p << logn) + brev(kk, logn)];
        B.y = -B.y;
        const float2 e = ek_n[k];
        const float sx = A.x + B.x, sy = A.y + B.y, dx = A.x - B.x, dy = A.y - B.y;
        const int r = row0 + 2 * p;
        t1[pair_at(r, k, m, n)] = 0.5f * (e.x * sx - e.y * sy);
        t1[pair_at(r + 1, k, m, n)] = 0.5f * (e.x * dy + e.y * dx);
    }
    if (!rho_in && partials) {
        const Df vals[1] = {block_sum(ovf, shr)};
        if (step) {
            leave_partial(partials, blockIdx.x, vals[0]);
            return;
        }
        if (arrive_last(partials, blockIdx.x, 1, vals, &st->ctr[CTR_OVF], gridDim.x)) {
            const double tot = sum_partials(partials, gridDim.x, 1, 0, shr);
            if (threadIdx.x == 0) {
                st->overflow = tot;
                st->overflow_f = (float)(tot / movable_area);
                st->ctr[CTR_OVF] = 0;
            }
        }
    }
}

// weights of src/frequencies.rs:4-72 evaluated exactly as the oracle does
__device__ __forceinline__ float inv_k2(int u, int j, const float *wu, const float *wv) {
    if (u == 0 && j == 0) return 0.0f;
    const float s = __fadd_rn(__fmul_rn(wu[u], wu[u]), __fmul_rn(wv[j], wv[j]));
    return __fdiv_rn(1.0f, s);
}

// ---------------- C1: columns DCT-II, weights, inverse along m ----------------
template <int CP>
__global__ void __launch_bounds__(kThreads) k_cols_r2(
    int m, int n, int logm, const float2 *__restrict__ tw_g, const float2 *__restrict__ ek_m,
    const float *__restrict__ wu, const float *__restrict__ wv, const float *__restrict__ t1,
    float *__restrict__ tx, float *__restrict__ ty, float *__restrict__ tp, float scale4,
    const DevState *__restrict__ st) {
    if (st && st->done) return;
    constexpr int CB = 2 * CP;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm;
    float2 *buf = sm + (m >> 1);
    float *A = reinterpret_cast<float *>(buf + CP * m);
    const int j0 = blockIdx.x * CB;
    for (int k = threadIdx.x; k < (m >> 1); k += blockDim.x) tw[k] = tw_g[k];
    float *bf = reinterpret_cast<float *>(buf);
    for (int idx = threadIdx.x; idx < m * CB; idx += blockDim.x) {
        const int i = idx / CB, c = idx - i * CB;
        const float v = t1[pair_at(i, j0 + c, m, n)];
        bf[2 * (((c >> 1) << logm) + makhoul_pos(i, m)) + (c & 1)] = v;
    }
    __syncthreads();
    fft_dif<false>(buf, CP, m, logm, tw);
    for (int idx = threadIdx.x; idx < CP * m; idx += blockDim.x) {
        const int p = idx >> logm, u = idx & (m - 1);
        const int uu = (m - u) & (m - 1);
        const float2 Az = buf[(p << logm) + brev(u, logm)];
        float2 Bz = buf[(p << logm) + brev(uu, logm)];
        Bz.y = -Bz.y;
        const float2 e = ek_m[u];
        const float sx = Az.x + Bz.x, sy = Az.y + Bz.y, dx = Az.x - Bz.x, dy = Az.y - Bz.y;
        A[(2 * p) * m + u] = scale4 * (0.5f * (e.x * sx - e.y * sy));
        A[(2 * p + 1) * m + u] = scale4 * (0.5f * (e.x * dy + e.y * dx));
    }
    __syncthreads();
    const int nkinds = tp ? 3 : 2;
    for (int kind = 0; kind < nkinds; ++kind) {
        // kind 0: field_x  IDXST_m of A*wu_half; kind 1: field_y IDCT_m of A*wv_half;
        // kind 2: potential IDCT_m of A*inv
        const bool sine = kind == 0;
        for (int idx = threadIdx.x; idx < CP * ((m >> 1) + 1); idx += blockDim.x) {
            const int p = idx / ((m >> 1) + 1), u = idx - p * ((m >> 1) + 1);
            const int un = (m - u) & (m - 1);   // partner index (u = 0 pairs with "m", i.e. zero)
            float2 z_u = make_float2(0.f, 0.f), z_n = make_float2(0.f, 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 2 * p + h, j = j0 + c;
                const float a_u = A[c * m + u], a_n = A[c * m + un];
                float wgt_u, wgt_n;
                const float iu = inv_k2(u, j, wu, wv), in_ = inv_k2(un, j, wu, wv);
                if (kind == 0) {
                    wgt_u = __fmul_rn(__fmul_rn(wu[u], iu), 0.5f);
                    wgt_n = __fmul_rn(__fmul_rn(wu[un], in_), 0.5f);
                } else if (kind == 1) {
                    wgt_u = __fmul_rn(__fmul_rn(wv[j], iu), 0.5f);
                    wgt_n = __fmul_rn(__fmul_rn(wv[j], in_), 0.5f);
                } else {
                    wgt_u = iu;
                    wgt_n = in_;
                }
                const float xu = __fmul_rn(a_u, wgt_u);
                const float xn = (u == 0) ? 0.0f : __fmul_rn(a_n, wgt_n);   // X[m] := 0
                float2 vu, vn;
                if (!sine) {
                    vu = idct_spec(xu, xn, ek_m[u]);
                    vn = idct_spec(xn, xu, ek_m[un]);
                } else {
                    vu = (u == 0) ? make_float2(0.f, 0.f) : idct_spec(xn, xu, ek_m[u]);
                    vn = idct_spec(xu, xn, ek_m[un]);
                }
                if (h == 0) {
                    z_u.x += vu.x; z_u.y += vu.y; z_n.x += vn.x; z_n.y += vn.y;
                } else {  // + i * V_b
                    z_u.x -= vu.y; z_u.y += vu.x; z_n.x -= vn.y; z_n.y += vn.x;
                }
            }
            buf[(p << logm) + u] = z_u;
            if (u != 0 && u != (m >> 1)) buf[(p << logm) + un] = z_n;
        }
        __syncthreads();
        fft_dif<true>(buf, CP, m, logm, tw);
        float *out = kind == 0 ? tx : (kind == 1 ? ty : tp);
        for (int idx = threadIdx.x; idx < m * CB; idx += blockDim.x) {
            const int i = idx / CB, c = idx - i * CB;
            const int t = i >> 1, src = (i & 1) ? (m - 1 - t) : t;
            const float2 w = buf[((c >> 1) << logm) + brev(src, logm)];
            float v = (c & 1) ? w.y : w.x;
            if (sine && (i & 1)) v = -v;
            out[pair_at(i, j0 + c, m, n)] = v;
        }
        __syncthreads();
    }
}

// ---------------- R2: rows inverse along n ----------------
template <int PAIRS>
__global__ void __launch_bounds__(kThreads) k_rows_inv_r2(
    int m, int n, int logn, const float2 *__restrict__ tw_g, const float2 *__restrict__ ek_n,
    const float *__restrict__ tx, const float *__restrict__ ty, const float *__restrict__ tp,
    float *__restrict__ fx, float *__restrict__ fy, float *__restrict__ psi, int field_stride,
    const DevState *__restrict__ st) {
    if (st && st->done) return;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm;
    float2 *buf = sm + (n >> 1);
    for (int k = threadIdx.x; k < (n >> 1); k += blockDim.x) tw[k] = tw_g[k];
    const int row0 = blockIdx.x * 2 * PAIRS;
    const int nkinds = tp ? 3 : 2;
    for (int kind = 0; kind < nkinds; ++kind) {
        // kind 0: field_x = IDCT_n(tx); kind 1: field_y = IDXST_n(ty); kind 2: psi = IDCT_n(tp)
        const float *in = kind == 0 ? tx : (kind == 1 ? ty : tp);
        float *out = kind == 0 ? fx : (kind == 1 ? fy : psi);
        const size_t fs = kind == 2 ? 1 : field_stride;
        const bool sine = kind == 1;
        for (int idx = threadIdx.x; idx < PAIRS * n; idx += blockDim.x) {
            const int p = idx >> logn, i = idx & (n - 1);
            const int r = row0 + 2 * p;
            buf[idx] = make_float2(in[pair_at(r, i, m, n)], in[pair_at(r + 1, i, m, n)]);
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < PAIRS * ((n >> 1) + 1); idx += blockDim.x) {
            const int p = idx / ((n >> 1) + 1), u = idx - p * ((n >> 1) + 1);
            const int un = (n - u) & (n - 1);
            const float2 xu2 = buf[(p << logn) + u];
            const float2 xn2 = (u == 0) ? make_float2(0.f, 0.f) : buf[(p << logn) + un];
            float2 z_u = make_float2(0.f, 0.f), z_n = make_float2(0.f, 0.f);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float xu = h ? xu2.y : xu2.x, xn = h ? xn2.y : xn2.x;
                float2 vu, vn;
                if (!sine) {
                    vu = idct_spec(xu, xn, ek_n[u]);
                    vn = idct_spec(xn, xu, ek_n[un]);
                } else {
                    vu = (u == 0) ? make_float2(0.f, 0.f) : idct_spec(xn, xu, ek_n[u]);
                    vn = idct_spec(xu, xn, ek_n[un]);
                }
                if (h == 0) {
                    z_u.x += vu.x; z_u.y += vu.y; z_n.x += vn.x; z_n.y += vn.y;
                } else {
                    z_u.x -= vu.y; z_u.y += vu.x; z_n.x -= vn.y; z_n.y += vn.x;
                }
            }
            buf[(p << logn) + u] = z_u;
            if (u != 0 && u != (n >> 1)) buf[(p << logn) + un] = z_n;
        }
        __syncthreads();
        fft_dif<true>(buf, PAIRS, n, logn, tw);
        for (int idx = threadIdx.x; idx < PAIRS * n; idx += blockDim.x) {
            const int p = idx >> logn, i = idx & (n - 1);
            const int t = i >> 1, src = (i & 1) ? (n - 1 - t) : t;
            const float2 w = buf[(p << logn) + brev(src, logn)];
            float va = w.x, vb = w.y;
            if (sine && (i & 1)) { va = -va; vb = -vb; }
            const int r = row0 + 2 * p;
            out[((size_t)r * n + i) * fs] = va;
            out[((size_t)(r + 1) * n + i) * fs] = vb;
        }
        __syncthreads();
    }
}

// ===================================================================
// Sides 64..4096: pair transforms.  Two real sequences of one kind -- adjacent
// rows, or adjacent columns -- are the real and imaginary part of one complex
// sequence, transformed by the register FFT of fft_pair.cuh.  (Sequences of two
// kinds would do too, but a field much smaller than the other, as on an oblong
// grid, would then carry the larger one's rounding; neighbours of one kind have
// one scale.)
//
// Forward, Z = FFT(v_a + i v_b) of the Makhoul-ordered sequences:
//   y_a[k] = Re(e_k (Z[k] + conj Z[N-k]) / 2),  y_b[k] = Im-part likewise
// Inverse, from the spectra X_a, X_b (X[N] := 0), e^{i theta_u} = conj e_u:
//   cosine  z[u] = e^{i theta} ((X_a[u] + X_b[N-u]) + i (X_b[u] - X_a[N-u]))
//   sine    X'[u] = X[N-u], X'[0] = 0:  the two roles swapped, z[0] = 0
// and v_a = Re, v_b = Im of the inverse FFT, un-permuted to the output order: no
// half-length folding and two multiplications per point, where the half-length
// form spent most of its instructions.
//
// What bounds the passes: latency and issue up to 1024^2 (every map sits in L2; one
// wave of 8 to 14 warps per SM), L2 traffic and occupancy above.  Measured per pass,
// L2-warm, against four warps per half-length sequence (sides 512..2048) and radix-2
// in shared memory (side 4096):
//   1024 x 1024 solve              rows forward 7.3 -> 4.1, columns 23.3 -> 12.3, rows inverse 12.6 -> 5.9 us
//   4096 x 2048 with the potential rows forward 48 -> 18, columns 637 -> 108, rows inverse 111 -> 48 us
//   in the step, 1M cells, 1024^2  rows forward 13.9 -> 10.5, columns 24.2 -> 16.8, rows inverse 12.3 -> 6.4 us
//   in the step, 64^2              rows forward 5.1 -> 5.3, columns 4.0 -> 3.5, rows inverse 2.1 -> 2.2 us
// ===================================================================

// Makhoul position of a sequence's element, and back: v[s] = x[elem(s)]
__device__ __forceinline__ int makhoul_elem(int s, int N) { return s < (N >> 1) ? 2 * s : 2 * (N - 1 - s) + 1; }

// y_a, y_b of the forward transform at the index of Z1 = Z[k], Z2 = Z[N-k] (e = e_k)
__device__ __forceinline__ float2 dct2_pair(float2 z1, float2 z2, float2 e) {
    const float sx = __fadd_rn(z1.x, z2.x), sy = __fsub_rn(z1.y, z2.y);
    const float dx = __fsub_rn(z1.x, z2.x), dy = __fadd_rn(z1.y, z2.y);
    // e = (cos, -sin): Re(e (s_x + i s_y)) / 2 and Re(e (d_y - i d_x)) / 2
    return make_float2(__fmul_rn(0.5f, __fmaf_rn(e.x, sx, -__fmul_rn(e.y, sy))),
                       __fmul_rn(0.5f, __fmaf_rn(e.x, dy, __fmul_rn(e.y, dx))));
}

// e_{N-u} of e_u = (cos, -sin): the angle's complement to pi / 2
__device__ __forceinline__ float2 ek_mirror(float2 e) { return make_float2(-e.y, -e.x); }

// z[u] of the inverse from (X_a, X_b)[u] and (X_a, X_b)[N-u] (zero at u = 0).  The
// products with P are the rounded ones, those with Q go into the fused operation.  Other
// orders are as accurate (eight were tried), but a placement's loop grows a difference of
// one rounding: they spread the 20,000-cell run's HPWL at its least overflow over 2.3651e6
// to 2.3767e6, about the two oracle forms' own 2.3698e6 and 2.3812e6, and the end-to-end
// test asks for 0.5 % of either.  This order is the one furthest inside that bar
// (+0.29 % and -0.19 %); another may fail the test without being wrong.
__device__ __forceinline__ float2 inv_pair(float2 xu, float2 xn, float2 e) {
    const float P = __fadd_rn(xu.x, xn.y), Q = __fsub_rn(xu.y, xn.x);
    return make_float2(__fmaf_rn(e.y, Q, __fmul_rn(e.x, P)), __fmaf_rn(-e.y, P, __fmul_rn(e.x, Q)));
}

// R1: rows forward DCT-II, P row pairs per block.  From the fixed-point map, one
// thread first issues two bulk copies (the block's rows of int64 sums and of the
// fixed-cell map) on the block's mbarrier; every thread then converts the elements
// of its own FFT positions, so each bin is converted once and goes straight into
// registers, and the rows are zeroed with 16-byte stores.
struct RowsFwdP {
    int m;
    const float2 * tw_n;
    const float2 * ek_n;
    const float * rho_in;
    unsigned long long * dmap;
    const float * initial;
    float fixed_inv;
    float coef;
    float inv_area;
    int zero_map;
    float * rho_out;
    float * t1;
    double * partials;
    DevState * st;
    double movable_area;
    int step;   // 1: inside a whole step, the overflow's block sums are left for its tail (k_nesterov_update)
};
// INNER (all three passes below): the whole solve is one kernel.  What a pass reads was
// written earlier in it, or (the density, where a caller's output takes its place) is
// written later, which rules the read-only path out.
template <int N, int P, bool INNER = false>
__device__ __forceinline__ void rows_fwd_body(const RowsFwdP &a, int bid, int nblk) {
    using F = PairFft<N, P>;
    DevState *__restrict__ st = a.st;
    if (st && st->done) return;
    extern __shared__ __align__(16) float2 sm[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ double shr[F::THREADS / 32];
    const int p = threadIdx.x % P, t = threadIdx.x / P;
    const int pair = bid * P + p;   // rows at positions 2 pair and 2 pair + 1
    const size_t ra = (size_t)makhoul_elem(2 * pair, a.m) * N, rb = (size_t)makhoul_elem(2 * pair + 1, a.m) * N;
    const bool from_map = a.rho_in == nullptr;
    float2 v[F::R1], w1[F::R1];
    Df ovf = df_zero();
    if (from_map) {
        unsigned long long *q_s = reinterpret_cast<unsigned long long *>(sm);
        float *ini_s = reinterpret_cast<float *>(q_s + 2 * P * N);
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, 24u * P * N);
            for (int k = 0; k < 2 * P; ++k) {
                const size_t r = (size_t)makhoul_elem(2 * P * bid + k, a.m) * N;
                bulk_load(q_s + k * N, a.dmap + r, 8u * N, &bar);
                bulk_load(ini_s + k * N, a.initial + r, 4u * N, &bar);
            }
        }
        F::load_tw1(w1, a.tw_n, t);
        F::sync();   // the barrier's initialisation
        if (!mbar_wait(&bar, 0, (st && st->expire_waits) ? 0u : kWaitTries)) {
            if (st) {
                atomicOr(&st->status, kStatusWaitTimeout);
                st->done = 1;
            }
            mbar_wait(&bar, 0);   // the copy must land before the area is reused
        }
        Df ov[4] = {df_zero(), df_zero(), df_zero(), df_zero()};   // four independent chains
#pragma unroll
        for (int j = 0; j < F::R1; ++j) {
            const int i = makhoul_elem(t + j * F::M, N);
            float x[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = (2 * p + h) * N + i;
                // d = (float)sum * 2^-S + initial  (src/density.rs:231-236, fixed point)
                const float d = __fadd_rn(__fmul_rn(fxp_u64_to_float(q_s[k]), a.fixed_inv), ini_s[k]);
                const float o = __fsub_rn(d, a.coef);
                ov[(2 * j + h) & 3] = df_add(ov[(2 * j + h) & 3], o > 0.0f ? o : 0.0f);   // src/epotential.rs:274-276
                x[h] = __fmul_rn(d, a.inv_area);                                         // src/epotential.rs:284-285
                if (a.rho_out) a.rho_out[(h ? rb : ra) + i] = x[h];
            }
            v[j] = make_float2(x[0], x[1]);
        }
        ovf = df_add(df_add(ov[0], ov[1]), df_add(ov[2], ov[3]));
        if (a.zero_map) {
#pragma unroll
            for (int k = 0; k < F::R1 / 2; ++k) {
                reinterpret_cast<ulonglong2 *>(a.dmap + ra)[t + F::T * k] = make_ulonglong2(0ull, 0ull);
                reinterpret_cast<ulonglong2 *>(a.dmap + rb)[t + F::T * k] = make_ulonglong2(0ull, 0ull);
            }
        }
        F::sync();   // the staged rows are consumed: the FFT may overwrite them
    } else {
#pragma unroll
        for (int j = 0; j < F::R1; ++j) {
            const int i = makhoul_elem(t + j * F::M, N);
            v[j] = make_float2(F::template load_elem<INNER>(a.rho_in + ra + i), F::template load_elem<INNER>(a.rho_in + rb + i));
        }
        F::load_tw1(w1, a.tw_n, t);
    }
    F::template run<false>(v, w1, sm, a.tw_n, t, p);
    F::sync();
#pragma unroll
    for (int e = 0; e < F::R1; ++e) sm[F::out_index(t, e) * P + p] = v[e];
    F::sync();
    float2 *out = reinterpret_cast<float2 *>(a.t1) + (size_t)pair * N;
#pragma unroll
    for (int j = 0; j < F::R1 / 2; ++j) {
        const int u = t + j * F::T, u2 = u ? N - u : N / 2;   // u = 0 is done with the self-paired N / 2
        const float2 zu = sm[u * P + p], zn = sm[u2 * P + p];
        const float2 eu = __ldg(a.ek_n + u), en = u ? ek_mirror(eu) : __ldg(a.ek_n + N / 2);
        out[u] = dct2_pair(zu, u ? zn : zu, eu);
        out[u2] = dct2_pair(zn, u ? zu : zn, en);
    }
    if (from_map && a.partials) {
        const Df vals[1] = {block_sum(ovf, shr)};
        if (a.step) {
            leave_partial(a.partials, bid, vals[0]);
            return;
        }
        if (arrive_last(a.partials, bid, 1, vals, &st->ctr[CTR_OVF], nblk)) {
            const double tot = sum_partials(a.partials, nblk, 1, 0, shr);
            if (threadIdx.x == 0) {
                st->overflow = tot;
                st->overflow_f = (float)(tot / a.movable_area);
                st->ctr[CTR_OVF] = 0;
            }
        }
    }
}
template <int N, int P>
__global__ void __launch_bounds__(PairFft<N, P>::THREADS) k_rows_fwd(const __grid_constant__ RowsFwdP p) {
    rows_fwd_body<N, P>(p, blockIdx.x, gridDim.x);
}

// C1: P column pairs per block.  Forward DCT-II along x, then A / (2 k^2) per bin
// (kept as pairs in natural order), then for each output kind the weighted inverse
// along x.  Runs of 2 P pairs are read and written straight from registers.
struct ColsP {
    int n;
    const float2 * tw_m;
    const float2 * ek_m;
    const float * wu;
    const float * wv;
    const float * t1;
    float * tx;
    float * ty;
    float * tp;
    float scale4;
    const DevState * st;
};
template <int N, int P, bool INNER = false>
__device__ __forceinline__ void cols_body(const ColsP &a, int bid, int nblk) {
    using F = PairFft<N, P>;
    if (a.st && a.st->done) return;
    extern __shared__ __align__(16) float2 sm[];
    float2 *A = sm, *B = sm + N * P;   // FFT exchanges; spectra
    const int p = threadIdx.x % P, t = threadIdx.x / P;
    const int j0 = bid * (2 * P) + 2 * p;
    const size_t n = (size_t)a.n;
    const bool odd = t & 1;
    // Positions s and s ^ 1 of a column pair are one row of interleaved pairs; the
    // threads t and t ^ 1 (P lanes apart) move one column each and swap halves.
    auto swap = [&](float2 x) -> float2 {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? x.x : x.y, P);
        return odd ? make_float2(got, x.y) : make_float2(x.x, got);
    };
    const size_t at0 = (size_t)(j0 + odd);
    float2 v[F::R1], w1[F::R1];
#pragma unroll
    for (int j = 0; j < F::R1; ++j)
        v[j] = F::template load_pair<INNER>(reinterpret_cast<const float2 *>(a.t1) + ((t + j * F::M) >> 1) * n + at0);
    F::load_tw1(w1, a.tw_m, t);
#pragma unroll
    for (int j = 0; j < F::R1; ++j) v[j] = swap(v[j]);
    F::template run<false>(v, w1, A, a.tw_m, t, p);
#pragma unroll
    for (int e = 0; e < F::R1; ++e) B[F::out_index(t, e) * P + p] = v[e];
    F::sync();
    const float wv0 = __ldg(a.wv + j0), wv1 = __ldg(a.wv + j0 + 1);
    const float wv0s = __fmul_rn(wv0, wv0), wv1s = __fmul_rn(wv1, wv1);
    // A (4 / mn) / (2 (wu^2 + wv^2)), [0, 0] -> 0 (src/frequencies.rs:4-72)
    auto weigh = [&](float2 y, int u) -> float2 {
        const float w = __ldg(a.wu + u), ws = __fmul_rn(w, w);
        const float s0 = __fadd_rn(ws, wv0s), s1 = __fadd_rn(ws, wv1s);
        const float i0 = (u | j0) == 0 ? 0.0f : __fmul_rn(0.5f, __frcp_rn(s0));
        const float i1 = __fmul_rn(0.5f, __frcp_rn(s1));
        return make_float2(__fmul_rn(__fmul_rn(a.scale4, y.x), i0), __fmul_rn(__fmul_rn(a.scale4, y.y), i1));
    };
#pragma unroll
    for (int j = 0; j < F::R1 / 2; ++j) {
        const int u = t + j * F::T, u2 = u ? N - u : N / 2;
        const float2 zu = B[u * P + p], zn = B[u2 * P + p];
        const float2 eu = __ldg(a.ek_m + u), en = u ? ek_mirror(eu) : __ldg(a.ek_m + N / 2);
        B[u * P + p] = weigh(dct2_pair(zu, u ? zn : zu, eu), u);
        B[u2 * P + p] = weigh(dct2_pair(zn, u ? zu : zn, en), u2);
    }
    const int nkinds = a.tp ? 3 : 2;
#pragma unroll 1
    for (int kind = 0; kind < nkinds; ++kind) {
        // kind 0: field_x  IDXST_x of A * wu / 2k^2   (src/idxst_idct.rs, src/frequencies.rs:52-58)
        // kind 1: field_y  IDCT_x  of A * wv / 2k^2   (src/idct_idxst.rs, src/frequencies.rs:60-66)
        // kind 2: potential IDCT_x of A / k^2          (src/idct2.rs)
        F::sync();   // the spectra are complete; A is free
        const float c0 = kind == 1 ? wv0 : 2.0f, c1 = kind == 1 ? wv1 : 2.0f;
#pragma unroll
        for (int j = 0; j < F::R1; ++j) {
            const int u = t + j * F::M, un = (N - u) & (N - 1);
            float2 xu = B[u * P + p], xn = B[un * P + p];
            if (kind == 0) {
                const float wu = __ldg(a.wu + u), wn = __ldg(a.wu + un);
                xu = make_float2(__fmul_rn(xu.x, wu), __fmul_rn(xu.y, wu));
                xn = make_float2(__fmul_rn(xn.x, wn), __fmul_rn(xn.y, wn));
                const float2 s = xu;
                xu = xn;
                xn = s;
            } else {
                xu = make_float2(__fmul_rn(xu.x, c0), __fmul_rn(xu.y, c1));
                xn = make_float2(__fmul_rn(xn.x, c0), __fmul_rn(xn.y, c1));
            }
            if (u == 0) {
                xn = make_float2(0.0f, 0.0f);
                if (kind == 0) xu = xn;
            }
            v[j] = inv_pair(xu, xn, __ldg(a.ek_m + u));
        }
        F::template run<true>(v, w1, A, a.tw_m, t, p);
        float2 *out = reinterpret_cast<float2 *>(kind == 0 ? a.tx : (kind == 1 ? a.ty : a.tp)) + at0;
#pragma unroll
        for (int e = 0; e < F::R1; ++e) {
            const int k = F::out_index(t, e);   // k ^ 1 is in thread t ^ 1
            if (kind == 0 && k >= N / 2) v[e] = make_float2(-v[e].x, -v[e].y);   // odd rows of the sine form
            out[(k >> 1) * n] = swap(v[e]);
        }
    }
}
template <int N, int P>
__global__ void __launch_bounds__(PairFft<N, P>::THREADS) k_cols(const __grid_constant__ ColsP p) {
    cols_body<N, P>(p, blockIdx.x, gridDim.x);
}

// R2: rows inverse along y.  A block takes P (row pair, kind) tasks: the two fields
// (field_x = IDCT_y(tx), field_y = IDXST_y(ty)) of a row pair are neighbouring tasks
// in the first m / P blocks; when the potential is asked for, each of m / 2P more
// takes P row pairs of psi = IDCT_y(tp).
struct RowsInvP {
    int m;   // rows
    const float2 * tw_n;
    const float2 * ek_n;
    const float * tx;
    const float * ty;
    const float * tp;
    float * fx;
    float * fy;
    float * psi;
    int pairs;   // 1: the outputs start on 8-byte boundaries (a caller's buffer may not)
    int field_stride;   // elements between neighbouring bins of a field: 2 when interleaved
    const DevState * st;
};
template <int N, int P, bool INNER = false>
__device__ __forceinline__ void rows_inv_body(const RowsInvP &a, int bid, int nblk) {
    using F = PairFft<N, P>;
    if (a.st && a.st->done) return;
    extern __shared__ __align__(16) float2 sm[];
    const int p = threadIdx.x % P, t = threadIdx.x / P;
    const int nxy = a.m / P;   // blocks of the two fields
    const bool fields = bid < nxy;
    const int task = (fields ? bid : bid - nxy) * P + p;
    const int kind = fields ? (task & 1) : 2;
    const int pair = fields ? task >> 1 : task;   // rows at positions 2 pair and 2 pair + 1
    const float2 *in = reinterpret_cast<const float2 *>(kind == 0 ? a.tx : (kind == 1 ? a.ty : a.tp)) + (size_t)pair * N;
    float *out = kind == 0 ? a.fx : (kind == 1 ? a.fy : a.psi);
    const int fs = kind == 2 ? 1 : a.field_stride;
    float *oa = out + (size_t)makhoul_elem(2 * pair, a.m) * N * fs, *ob = out + (size_t)makhoul_elem(2 * pair + 1, a.m) * N * fs;
    const bool sine = kind == 1;
    float2 v[F::R1], w1[F::R1], xn[F::R1], ek[F::R1];
#pragma unroll
    for (int j = 0; j < F::R1; ++j) {
        const int u = t + j * F::M, un = (N - u) & (N - 1);
        v[j] = F::template load_pair<INNER>(in + (sine ? un : u));
        xn[j] = F::template load_pair<INNER>(in + (sine ? u : un));
    }
#pragma unroll
    for (int j = 0; j < F::R1; ++j) ek[j] = F::load(a.ek_n + t + j * F::M);
    F::load_tw1(w1, a.tw_n, t);
#pragma unroll
    for (int j = 0; j < F::R1; ++j) {
        if (j == 0 && t == 0) {   // u = 0
            xn[j] = make_float2(0.0f, 0.0f);
            if (sine) v[j] = xn[j];
        }
        v[j] = inv_pair(v[j], xn[j], ek[j]);
    }
    F::template run<true>(v, w1, sm, a.tw_n, t, p);
    F::sync();
#pragma unroll
    for (int e = 0; e < F::R1; ++e) sm[F::out_index(t, e) * P + p] = v[e];
    F::sync();
#pragma unroll
    for (int j = 0; j < F::R1 / 2; ++j) {
        const int s = t + j * F::T;   // elements 2 s and 2 s + 1
        float2 z0 = sm[s * P + p], z1 = sm[(N - 1 - s) * P + p];
        if (sine) z1 = make_float2(-z1.x, -z1.y);
        if (a.pairs && fs == 1) {
            reinterpret_cast<float2 *>(oa)[s] = make_float2(z0.x, z1.x);
            reinterpret_cast<float2 *>(ob)[s] = make_float2(z0.y, z1.y);
        } else {
            oa[2 * s * fs] = z0.x;
            oa[(2 * s + 1) * fs] = z1.x;
            ob[2 * s * fs] = z0.y;
            ob[(2 * s + 1) * fs] = z1.y;
        }
    }
}
template <int N, int P>
__global__ void __launch_bounds__(PairFft<N, P>::THREADS) k_rows_inv(const __grid_constant__ RowsInvP p) {
    rows_inv_body<N, P>(p, blockIdx.x, gridDim.x);
}

// The isolated solve of a small grid (both sides 64 or 128) as one launch of one
// cluster: the three passes with cluster barriers between them, each pass's blocks
// dealt out to the CTAs.  Its bound is latency: 16 KB to 64 KB per array, and of three
// launches back to back each took 4 to 5 us where its kernel works for about 2.
// Per solve, three launches and this (us): 64 x 64 13.3, 8.2; 64 x 128 14.3, 10.2;
// 128 x 64 15.4, 12.0; 128 x 128 16.4, 12.3; with the potential 14.3, 10.2 and 16.4,
// 14.3 at the ends.  CTAs x pairs per block at 64 x 64: 8 x 8 and 8 x 4 8.2, 4 x 8
// 10.2, 8 x 2 and 2 x 16 12.3, 1 x 16 18.4; at 128 x 128 8 x 8 12.3, 8 x 4 16.4,
// 4 x 16 20.5.  Not for 256 x 256 (16.4, 31.6 this way: eight SMs are too few) and not
// in the step, where the graph's launches cost less than the barriers (a pass of 8
// steps at 64 x 64 bins 347, 350 with this).
constexpr int kSmallCtas = 8, kSmallPairs = 8;
struct SmallP {
    RowsFwdP fwd;
    ColsP cols;
    RowsInvP inv;
};
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
template <int M, int N>
__global__ void __cluster_dims__(kSmallCtas, 1, 1) __launch_bounds__(PairFft<N, kSmallPairs>::THREADS)
    k_solve_small(const __grid_constant__ SmallP p) {
    constexpr int P = kSmallPairs, ROWS = M / (2 * P), COLS = N / (2 * P);
    static_assert(PairFft<N, P>::THREADS == PairFft<M, P>::THREADS, "one block shape for all passes");
    static_assert(ROWS <= kSmallCtas && COLS <= kSmallCtas, "at most one block per CTA");
    const int cta = blockIdx.x;
    if (cta < ROWS) rows_fwd_body<N, P, true>(p.fwd, cta, ROWS);
    cluster_barrier();
    if (cta < COLS) cols_body<M, P, true>(p.cols, cta, COLS);
    cluster_barrier();
    const int blocks = M / P + (p.inv.psi ? M / (2 * P) : 0);
    for (int b = cta; b < blocks; b += kSmallCtas) {
        rows_inv_body<N, P, true>(p.inv, b, blocks);
        __syncthreads();   // the exchange area is free for the next block
    }
}

// The density map as rho for the tensor-core solve: the conversion of R1 (same
// float rules, so rho is bit-identical to what the FFT path transforms), the
// double-float overflow sum, and the map zeroing, two bins per thread; with hi and lo
// also the BF16x3 solve's split of rho, which was a launch of its own.  512^2 bins: this
// kernel (with its own reduction tail) and the split 8.2 + 1.8 us, now 4.8 us.
__global__ void __launch_bounds__(kThreads) k_map_rho(size_t pairs, ulonglong2 *__restrict__ dmap,
                                                      const float2 *__restrict__ initial, float fixed_inv, float coef,
                                                      float inv_area, int zero_map, float2 *__restrict__ rho,
                                                      __nv_bfloat162 *__restrict__ hi, __nv_bfloat162 *__restrict__ lo,
                                                      double *__restrict__ partials, DevState *__restrict__ st,
                                                      double movable_area, int step) {
    __shared__ double shr[kThreads / 32];
    if (st->done) return;
    Df ovf = df_zero();
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < pairs; idx += (size_t)gridDim.x * blockDim.x) {
        const ulonglong2 q = dmap[idx];
        const float2 ini = initial[idx];
        if (zero_map) dmap[idx] = make_ulonglong2(0ull, 0ull);
        float r[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // d = (float)sum * 2^-S + initial  (src/density.rs:231-236, fixed point)
            const float d = __fadd_rn(__fmul_rn(fxp_u64_to_float(h ? q.y : q.x), fixed_inv), h ? ini.y : ini.x);
            const float o = __fsub_rn(d, coef);
            ovf = df_add(ovf, o > 0.0f ? o : 0.0f);  // src/epotential.rs:274-276
            r[h] = __fmul_rn(d, inv_area);             // src/epotential.rs:284-285
        }
        rho[idx] = make_float2(r[0], r[1]);
        if (hi) {
            __nv_bfloat162 a, b;
            split_pair(r[0], r[1], a, b);
            hi[idx] = a;
            lo[idx] = b;
        }
    }
    const Df vals[1] = {block_sum(ovf, shr)};
    if (step) {
        leave_partial(partials, blockIdx.x, vals[0]);
        return;
    }
    if (arrive_last(partials, blockIdx.x, 1, vals, &st->ctr[CTR_OVF], gridDim.x)) {
        const double tot = sum_partials(partials, gridDim.x, 1, 0, shr);
        if (threadIdx.x == 0) {
            st->overflow = tot;
            st->overflow_f = (float)(tot / movable_area);
            st->ctr[CTR_OVF] = 0;
        }
    }
}

// mn is even: both sides are multiples of 128
int map_rho_blocks(size_t mn) { return (int)std::min<size_t>((mn / 2 + kThreads - 1) / kThreads, 152 * 8); }

void launch_map_rho(const SpectralArgs &a, size_t mn, float *rho, void *hi, void *lo, cudaStream_t s) {
    k_map_rho<<<map_rho_blocks(mn), kThreads, 0, s>>>(
        mn / 2, reinterpret_cast<ulonglong2 *>(a.dmap), reinterpret_cast<const float2 *>(a.initial), a.fixed_inv, a.coef,
        a.inv_bin_area, a.zero_map ? 1 : 0, reinterpret_cast<float2 *>(rho), static_cast<__nv_bfloat162 *>(hi),
        static_cast<__nv_bfloat162 *>(lo), a.partials, a.st, a.movable_area, a.step ? 1 : 0);
}

int ilog2(int v) {
    int l = 0;
    while ((1 << l) < v) ++l;
    return l;
}

static size_t rows_smem(int n, int pairs) { return sizeof(float2) * ((size_t)(n >> 1) + (size_t)pairs * n); }
static size_t cols_smem(int m, int cp) {
    return sizeof(float2) * ((size_t)(m >> 1) + (size_t)cp * m) + sizeof(float) * (size_t)(2 * cp) * m;
}

constexpr int kRowPairs = 2, kColPairs = 4;   // the radix-2 kernels (sides 16 and 32)

static bool pair_side(int v) { return v >= 64; }

// Host-computed tables (FP64 angles rounded to FP32) uploaded to the given
// arrays; pageable copies, so the host buffers can go as soon as the calls return.
void spectral_tables_fill(int m, int n, float bin_w, float bin_h, float2 *tw_m, float2 *tw_n, float2 *ek_m,
                          float2 *ek_n, float *wu, float *wv, cudaStream_t s) {
    auto tw = [](int N) {   // pair FFT: stage twiddles; radix-2 FFT: W_N^k, k < N / 2
        const int len = pair_side(N) ? fft_tw_len(N) : N / 2;
        std::vector<float2> h(len);
        for (int k = 0; k < len; ++k) {
            double a = -2.0 * 3.14159265358979323846 * (double)(pair_side(N) ? fft_tw_num(N, k) : k) / (double)N;
            h[k] = make_float2((float)cos(a), (float)sin(a));
        }
        return h;
    };
    auto ek = [](int N) {
        std::vector<float2> h(N);
        for (int k = 0; k < N; ++k) {
            double a = 3.14159265358979323846 * (double)k / (2.0 * N);
            h[k] = make_float2((float)cos(a), (float)-sin(a));
        }
        return h;
    };
    const std::vector<float2> h_twm = tw(m), h_twn = tw(n), h_ekm = ek(m), h_ekn = ek(n);
    std::vector<float> h_wu(m), h_wv(n);
    const float tpm = (float)(2.0 * 3.14159265358979323846) / (float)m;
    for (int i = 0; i < m; ++i) h_wu[i] = (float)i * tpm;
    const float wv_div = bin_w / bin_h;
    const float tpn = (float)(2.0 * 3.14159265358979323846) / (float)n;
    for (int j = 0; j < n; ++j) h_wv[j] = ((float)j * tpn) * wv_div;
    cudaMemcpyAsync(tw_m, h_twm.data(), sizeof(float2) * h_twm.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(tw_n, h_twn.data(), sizeof(float2) * h_twn.size(), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(ek_m, h_ekm.data(), sizeof(float2) * m, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(ek_n, h_ekn.data(), sizeof(float2) * n, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(wu, h_wu.data(), sizeof(float) * m, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(wv, h_wv.data(), sizeof(float) * n, cudaMemcpyHostToDevice, s);
}

void spectral_tables(int m, int n, float bin_w, float bin_h, float2 **tw_m, float2 **tw_n,
                     float2 **ek_m, float2 **ek_n, float **wu, float **wv, cudaStream_t s) {
    ctx_alloc((void **)tw_m, sizeof(float2) * m, s);
    ctx_alloc((void **)tw_n, sizeof(float2) * n, s);
    ctx_alloc((void **)ek_m, sizeof(float2) * m, s);
    ctx_alloc((void **)ek_n, sizeof(float2) * n, s);
    ctx_alloc((void **)wu, sizeof(float) * m, s);
    ctx_alloc((void **)wv, sizeof(float) * n, s);
    spectral_tables_fill(m, n, bin_w, bin_h, *tw_m, *tw_n, *ek_m, *ek_n, *wu, *wv, s);
    cudaStreamSynchronize(s);
}

// ---- shapes of the pair passes: P pairs per block ----
// Dynamic shared memory: rows forward 8 N P bytes of exchange, inside the 24 N P
// that stage the map when there is one; columns exchange + spectra.
template <int N, int P>
static size_t rows_fwd_smem(bool from_map) { return (from_map ? 24 : 8) * (size_t)N * P; }
template <int N, int P>
static size_t cols_pair_smem() { return 16 * (size_t)N * P; }
template <int N, int P>
static size_t rows_inv_smem() { return 8 * (size_t)N * P; }

// Pairs per block.  A block is at least one warp, where a barrier costs least.
// Measured on square grids (us per pass, L2-warm; rows forward from the map; below 256
// one pair is less than a warp):
//   rows forward   P = 1 / 2 / 4   64: - / 6.0 / 6.4   128: - / 6.5 / 6.9   256: 7.7 / 6.8 / 7.4   512: 7.9 / 7.1 / 8.2
//                                  1024: 11.4 / 10.1 / 10.7   2048: 22.9 / 23.9 / 28.4   4096: 84 / 102
//   columns        P = 1 / 2 / 4   64: - / 3.5 / 3.2   128: - / 5.1 / 4.8   256: 5.2 / 5.3 / 5.2   512: 6.6 / 5.5 / 6.5
//                                  1024: 15.7 / 13.1 / 11.9   2048: 54 / 43 / 34   4096: 208 / 153
//   rows inverse   P = 1 / 2 / 4   64: - / 1.8 / 2.5   128: - / 2.1 / 3.1   256: 2.2 / 2.7 / 3.3   512: 3.5 / 3.2 / 3.9
//                                  1024: 5.4 / 6.4 / 7.3   2048: 14.7 / 18.6 / 26.5   4096: 69 / 103
// (P = 8: rows forward 7.4 and 8.3, columns 3.3 and 4.9, rows inverse 2.4 and 3.2 at 64
// and 128.)  Side 64 keeps four pairs in the rows forward, 0.4 us a pass more than two:
// eight steps at 2,003 cells take 309 us, 307 with two, and the overflow's block sums
// would be grouped otherwise.
// The column pass reads and writes runs of 16 P bytes; large grids, where L2 traffic
// counts, want long ones, small grids a block for every SM.  Side 4096 has room for
// P = 2 (two arrays of 8 N P bytes).
constexpr int min_pairs(int N) { return 32 / (N / fft_r1(N)) > 1 ? 32 / (N / fft_r1(N)) : 1; }
constexpr int rows_fwd_pairs(int N) { return N == 64 ? 4 : (N >= 256 && N <= 1024 ? 2 : min_pairs(N)); }
constexpr int rows_inv_pairs(int N) { return N == 512 ? 2 : min_pairs(N); }
constexpr int cols_pairs(int N) { return N == 256 || N == 512 || N == 4096 ? 2 : 4; }
// A batch's autotuner times `seqs` sequences per block (2 or 8, at least one warp)
// against the shapes above, for sides 64..256.
constexpr int seq_pairs(int N, int seqs) { return seqs / 2 > min_pairs(N) ? seqs / 2 : min_pairs(N); }
// Calls f.operator()<N, P>() for a pass's side and the plan's shape.
enum PairPass { PASS_ROWS_FWD, PASS_COLS, PASS_ROWS_INV };
template <PairPass PASS>
constexpr int fixed_pairs(int N) {
    return PASS == PASS_ROWS_FWD ? rows_fwd_pairs(N) : (PASS == PASS_COLS ? cols_pairs(N) : rows_inv_pairs(N));
}
template <PairPass PASS, int N, typename F>
static void pair_shape(int seqs, F &&f) {
    if constexpr (N <= 256) {
        if (seqs == kSeqCandidates[0]) return f.template operator()<N, seq_pairs(N, kSeqCandidates[0])>();
        if (seqs == kSeqCandidates[1]) return f.template operator()<N, seq_pairs(N, kSeqCandidates[1])>();
    }
    f.template operator()<N, fixed_pairs<PASS>(N)>();
}
template <PairPass PASS, typename F>
static void pair_dispatch(int side, int seqs, F &&f) {
    switch (side) {
    case 64: return pair_shape<PASS, 64>(seqs, f);
    case 128: return pair_shape<PASS, 128>(seqs, f);
    case 256: return pair_shape<PASS, 256>(seqs, f);
    case 512: return pair_shape<PASS, 512>(seqs, f);
    case 1024: return pair_shape<PASS, 1024>(seqs, f);
    case 2048: return pair_shape<PASS, 2048>(seqs, f);
    default: return pair_shape<PASS, 4096>(seqs, f);
    }
}

// One pass of a plan, as a launch of its own.
struct LaunchRowsFwd {
    const SpectralPlan &p;
    const SpectralArgs &a;
    static RowsFwdP params(const SpectralPlan &p, const SpectralArgs &a) {
        return RowsFwdP{p.m, p.tw_n, p.ek_n, a.rho_in, a.dmap, a.initial, a.fixed_inv, a.coef, a.inv_bin_area,
                        a.zero_map ? 1 : 0, a.rho_out, p.t1, a.rho_in == nullptr ? a.partials : nullptr, a.st,
                        a.movable_area, a.step ? 1 : 0};
    }
    template <int N, int P>
    void operator()() const {
        k_rows_fwd<N, P><<<p.m / (2 * P), PairFft<N, P>::THREADS, rows_fwd_smem<N, P>(a.rho_in == nullptr), p.stream>>>(
            params(p, a));
    }
};
struct LaunchCols {
    const SpectralPlan &p;
    const SpectralArgs &a;
    static ColsP params(const SpectralPlan &p, const SpectralArgs &a) {
        return ColsP{p.n, p.tw_m, p.ek_m, p.wu, p.wv, p.t1, p.tx, p.ty, a.psi ? p.tp : nullptr,
                     4.0f / (float)((double)p.m * (double)p.n), a.st};
    }
    template <int N, int P>
    void operator()() const {
        k_cols<N, P><<<p.n / (2 * P), PairFft<N, P>::THREADS, cols_pair_smem<N, P>(), p.stream>>>(params(p, a));
    }
};
struct LaunchRowsInv {
    const SpectralPlan &p;
    const SpectralArgs &a;
    static RowsInvP params(const SpectralPlan &p, const SpectralArgs &a) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(a.fx) | reinterpret_cast<uintptr_t>(a.fy) |
                             reinterpret_cast<uintptr_t>(a.psi);
        return RowsInvP{p.m,  p.tw_n, p.ek_n, p.tx, p.ty, a.psi ? p.tp : nullptr, a.fx, a.fy, a.psi, (at & 7) == 0,
                        a.field_stride, a.st};
    }
    static int blocks(int m, int P, bool psi) { return m / P + (psi ? m / (2 * P) : 0); }
    template <int N, int P>
    void operator()() const {
        k_rows_inv<N, P><<<blocks(p.m, P, a.psi != nullptr), PairFft<N, P>::THREADS, rows_inv_smem<N, P>(), p.stream>>>(
            params(p, a));
    }
};

static bool small_grid(int m, int n) { return (m == 64 || m == 128) && (n == 64 || n == 128); }
template <int M, int N>
static void launch_small_as(const SpectralPlan &p, const SpectralArgs &a) {
    constexpr int P = kSmallPairs;
    const size_t smem = std::max(rows_fwd_smem<N, P>(false), std::max(cols_pair_smem<M, P>(), rows_inv_smem<N, P>()));
    k_solve_small<M, N><<<kSmallCtas, PairFft<N, P>::THREADS, smem, p.stream>>>(
        SmallP{LaunchRowsFwd::params(p, a), LaunchCols::params(p, a), LaunchRowsInv::params(p, a)});
}
static void launch_small(const SpectralPlan &p, const SpectralArgs &a) {
    if (p.m == 64) (p.n == 64 ? launch_small_as<64, 64> : launch_small_as<64, 128>)(p, a);
    else (p.n == 64 ? launch_small_as<128, 64> : launch_small_as<128, 128>)(p, a);
}

// Opt the spectral kernels into large dynamic shared memory on the current device.
struct PrepareRowsFwd {
    cudaError_t &e;
    template <int N, int P>
    void operator()() const {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_rows_fwd<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)rows_fwd_smem<N, P>(true));
    }
};
struct PrepareCols {
    cudaError_t &e;
    template <int N, int P>
    void operator()() const {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_cols<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)cols_pair_smem<N, P>());
    }
};
struct PrepareRowsInv {
    cudaError_t &e;
    template <int N, int P>
    void operator()() const {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_rows_inv<N, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)rows_inv_smem<N, P>());
    }
};
cudaError_t spectral_prepare() {
    cudaError_t e = cudaSuccess;
    for (int side = 64; side <= 4096; side *= 2)
        for (int seqs : {0, kSeqCandidates[0], kSeqCandidates[1]}) {
            if (seqs && side > 256) continue;
            pair_dispatch<PASS_ROWS_FWD>(side, seqs, PrepareRowsFwd{e});
            pair_dispatch<PASS_COLS>(side, seqs, PrepareCols{e});
            pair_dispatch<PASS_ROWS_INV>(side, seqs, PrepareRowsInv{e});
        }
    return e;
}

void launch_spectral_plan(const SpectralPlan &p, const SpectralArgs &a) {
    const int m = p.m, n = p.n;
    const bool from_map = a.rho_in == nullptr;
    const int rb = m / (2 * kRowPairs);
    if (small_grid(m, n) && !from_map) return launch_small(p, a);   // an isolated solve
    if (pair_side(n)) {
        pair_dispatch<PASS_ROWS_FWD>(n, p.seqs, LaunchRowsFwd{p, a});
    } else {
        k_rows_dct_r2<kRowPairs><<<rb, kThreads, rows_smem(n, kRowPairs), p.stream>>>(
            m, n, p.logn, p.tw_n, p.ek_n, a.rho_in, a.dmap, a.initial, a.fixed_inv, a.coef,
            a.inv_bin_area, a.zero_map ? 1 : 0, a.rho_out, p.t1, from_map ? a.partials : nullptr, a.st,
            a.movable_area, a.step ? 1 : 0);
    }
    float *tp = a.psi ? p.tp : nullptr;
    if (pair_side(m)) {
        pair_dispatch<PASS_COLS>(m, p.seqs, LaunchCols{p, a});
    } else {
        k_cols_r2<kColPairs><<<n / (2 * kColPairs), kThreads, cols_smem(m, kColPairs), p.stream>>>(
            m, n, p.logm, p.tw_m, p.ek_m, p.wu, p.wv, p.t1, p.tx, p.ty, tp,
            4.0f / (float)((double)m * (double)n), a.st);
    }
    if (pair_side(n)) {
        pair_dispatch<PASS_ROWS_INV>(n, p.seqs, LaunchRowsInv{p, a});
    } else {
        k_rows_inv_r2<kRowPairs><<<rb, kThreads, rows_smem(n, kRowPairs), p.stream>>>(
            m, n, p.logn, p.tw_n, p.ek_n, p.tx, p.ty, tp, a.fx, a.fy, a.psi, a.field_stride, a.st);
    }
}

// Blocks of the forward row pass: the overflow's block sums.
struct RowBlocks {
    int m;
    int &blocks;
    template <int N, int P>
    void operator()() const { blocks = m / (2 * P); }
};
int spectral_row_blocks(const SpectralPlan &p) {
    int blocks = p.m / (2 * kRowPairs);
    if (pair_side(p.n)) pair_dispatch<PASS_ROWS_FWD>(p.n, p.seqs, RowBlocks{p.m, blocks});
    return blocks;
}

// ---- packed launches of the pair passes (batches) ----
// Sides 64..256: each pass of many solves in one launch per shape (N, P) in use.
constexpr int shape_id(int N, int P) { return N * 16 + P; }
struct ShapeOf {
    int &id;
    template <int N, int P>
    void operator()() const { id = shape_id(N, P); }
};

template <typename P, typename F>
static void plan_spectral(PackKind k, int variant, const std::vector<const SpectralJob *> &js, PackedArena &ar,
                          std::vector<PackedLaunch> &out, size_t smem, int threads, F params) {
    std::vector<P> tab;
    std::vector<int32_t> block0(1, 0);
    for (const SpectralJob *j : js) {
        int g = 0;
        tab.push_back(params(*j, g));
        block0.push_back(block0.back() + g);
    }
    if (tab.empty()) return;
    PackedLaunch l;
    l.kind = k;
    l.variant = variant;
    l.tab = ar.put(tab.data(), sizeof(P) * tab.size());
    l.block0 = ar.put(block0.data(), sizeof(int32_t) * block0.size());
    l.n = (int)tab.size();
    l.blocks = block0.back();
    l.threads = threads;
    l.smem = smem;
    out.push_back(l);
}

struct PlanPass {
    PackKind k;
    const std::vector<const SpectralJob *> &js;
    PackedArena &ar;
    std::vector<PackedLaunch> &out;
    template <int N, int P>
    void operator()() const {
        const int id = shape_id(N, P), threads = PairFft<N, P>::THREADS;
        if (k == PK_ROWS_DCT_W)
            plan_spectral<RowsFwdP>(k, id, js, ar, out, rows_fwd_smem<N, P>(true), threads,
                                    [](const SpectralJob &j, int &g) {
                                        g = j.p.m / (2 * P);
                                        return LaunchRowsFwd::params(j.p, j.a);
                                    });
        else if (k == PK_COLS_W)
            plan_spectral<ColsP>(k, id, js, ar, out, cols_pair_smem<N, P>(), threads, [](const SpectralJob &j, int &g) {
                g = j.p.n / (2 * P);
                return LaunchCols::params(j.p, j.a);
            });
        else
            plan_spectral<RowsInvP>(k, id, js, ar, out, rows_inv_smem<N, P>(), threads, [](const SpectralJob &j, int &g) {
                g = LaunchRowsInv::blocks(j.p.m, P, j.a.psi != nullptr);
                return LaunchRowsInv::params(j.p, j.a);
            });
    }
};

template <PairPass PASS>
static void plan_pass(PackKind k, const std::vector<SpectralJob> &v, PackedArena &ar, std::vector<PackedLaunch> &out) {
    auto side = [&](const SpectralJob &j) { return PASS == PASS_COLS ? j.p.m : j.p.n; };
    std::vector<int> done;
    for (const SpectralJob &first : v) {
        int id = 0;
        pair_dispatch<PASS>(side(first), first.p.seqs, ShapeOf{id});
        if (std::find(done.begin(), done.end(), id) != done.end()) continue;
        done.push_back(id);
        std::vector<const SpectralJob *> js;
        for (const SpectralJob &j : v) {
            int other = 0;
            pair_dispatch<PASS>(side(j), j.p.seqs, ShapeOf{other});
            if (other == id) js.push_back(&j);
        }
        pair_dispatch<PASS>(side(first), first.p.seqs, PlanPass{k, js, ar, out});
    }
}

void packed_spectral_stage(PackKind k, const std::vector<SpectralJob> &v, PackedArena &ar,
                           std::vector<PackedLaunch> &out) {
    if (k == PK_ROWS_DCT_W) plan_pass<PASS_ROWS_FWD>(k, v, ar, out);
    else if (k == PK_COLS_W) plan_pass<PASS_COLS>(k, v, ar, out);
    else plan_pass<PASS_ROWS_INV>(k, v, ar, out);
}

struct LaunchPacked {
    const PackedLaunch &l;
    const unsigned char *dev;
    cudaStream_t s;
    template <int N, int P>
    void operator()() const {
        if constexpr (N <= 256) {
            constexpr int TH = PairFft<N, P>::THREADS;
            if (l.kind == PK_ROWS_DCT_W)
                k_packed<RowsFwdP, rows_fwd_body<N, P>, TH, 1><<<l.blocks, TH, l.smem, s>>>(packed_args<RowsFwdP>(l, dev));
            else if (l.kind == PK_COLS_W)
                k_packed<ColsP, cols_body<N, P>, TH, 1><<<l.blocks, TH, l.smem, s>>>(packed_args<ColsP>(l, dev));
            else
                k_packed<RowsInvP, rows_inv_body<N, P>, TH, 1><<<l.blocks, TH, l.smem, s>>>(packed_args<RowsInvP>(l, dev));
        }
    }
};

bool packed_spectral_launch(const PackedLaunch &l, const unsigned char *dev, cudaStream_t s) {
    if (l.kind != PK_ROWS_DCT_W && l.kind != PK_COLS_W && l.kind != PK_ROWS_INV_W) return false;
    const LaunchPacked f{l, dev, s};
    switch (l.variant) {   // the shapes pair_shape() gives for sides 64..256
    case shape_id(64, 2): f.operator()<64, 2>(); break;
    case shape_id(64, 4): f.operator()<64, 4>(); break;
    case shape_id(128, 2): f.operator()<128, 2>(); break;
    case shape_id(128, 4): f.operator()<128, 4>(); break;
    case shape_id(256, 1): f.operator()<256, 1>(); break;
    case shape_id(256, 2): f.operator()<256, 2>(); break;
    case shape_id(256, 4): f.operator()<256, 4>(); break;
    default: return false;
    }
    return true;
}

}  // namespace erp

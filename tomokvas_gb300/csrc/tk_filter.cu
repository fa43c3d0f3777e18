// tk_filter.cu -- fused preprocessing + ramp filter for GB300 (sm_103a).
//
// Replaces three stages of the reference FDK (Lukas-kV/TomoKvas):
//   * raw uint16 -> line integral, rsq::FlatFieldCorrection (FBPG/rsq_load.cpp:299-325);
//   * cosine pre-weight, RB_comma3DKernel (FBPG/kernel.cu:179-201);
//   * row-wise ramp filter, fConvolution (FBPG/kernel.cu:557-781): per detector
//     row, zero-pad to p = 2*nextpow2(W), R2C, multiply by tau*|R2C(h)|, C2R
//     unnormalised.
//
// GB300 design: one pass over HBM.  Each CTA streams pairs of detector rows
// straight from the raw input, applies log + cosine weight while loading,
// packs the two real rows as one complex signal z = a + i b, and runs a
// radix-16 Stockham FFT in registers and shared memory.  Because the filter
// spectrum is real and even, IFFT(FFT(z) * Hf) = (a*k) + i (b*k), so one forward
// and one inverse complex FFT filter two rows.  The inverse is computed as
// conj(FFT(conj(Z) * Hf)).  Results are written once, projection-major, in
// FP32/FP16/BF16.  No cuFFT, no staging copies, no per-row plans.
#include "tk_common.cuh"
#include "tk_fft_shape.h"
#include "tk_filter_core.cuh"
#include "tk_internal.h"

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace tk {

constexpr int kMaxHf = 4097;  // p/2 + 1 for p <= 8192
constexpr float kScaleTarget = 16384.f;  // bound of |stored value| for 16-bit storage

// ---------------------------------------------------------------------------
// Mixed-radix Stockham FFT.
//
// A pass with span Ns and radix R maps butterfly j (k = j mod Ns) as
//   v[r] = x[j + r p/R] * w^(r k p/(R Ns)),  y[(j-k) R + k + s Ns] = DFT_R(v)[s],
// one butterfly per thread, the R points in registers.  The length p = 2^lg
// forward transform runs radix 16 passes and one last pass of radix
// RL = 16, 8, 4 or 2; the inverse runs the RL pass first.  Then three of the
// joints need no shared memory: the first forward pass (Ns = 1) takes the
// samples x[j + r p/16] from registers, its upper half being the zero padding;
// the last forward pass ends on X[j + s p/RL], which are just the inputs of the
// inverse's first pass, so spectrum product and both butterflies run on the
// same registers; and the last inverse pass (Ns = p/16) ends on the output
// columns j + s p/16, of which s < 8 are wanted.  A row pair of p = 2048 takes
// four passes through shared memory and five barriers (eight and nine with a
// separate load, product and output pass): 90 frames of 1024^2 uint16 into FP16
// coefficients 830 -> 668 us, 411 x 300 FP32 rows of 1501 (p = 4096)
// 1971 -> 1310 us.
//
// Buffers are padded by one element per 16 (pidx), which makes every pass's
// loads and stores conflict-free; twiddles come from per-pass tables laid out
// [k][r] (one thread reads R-1 consecutive entries).

struct FiltParams {
    LoadParams L;
    void *out;
    const float *q_scale;  // device storage scale (16-bit) or null (= 1)
    long long nrows, npairs;
    int Wp, p, lg, precision;
    int rc, nchunks;        // coefficient image: rows per work unit, units per projection
    long long nunits;
    int fgrp, fstride;      // coefficient image, frames in groups (> 0): frame f is f/fgrp*fstride + f%fgrp
    int out_layout;         // raw output: TK_LAYOUT_PROJECTION [N][H][Wp] or TK_LAYOUT_SINOGRAM [H][N][Wp]
    int weight_out;         // multiply the output by the cosine weight (the filter's transpose)
    float Hf[kMaxHf];  // tau * |R2C_p(h)| * window, k = 0..p/2
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// Complex sum and difference as one packed FP32 instruction each.
__device__ __forceinline__ float2 cadd(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 A, B;\n\tmov.b64 A, {%2, %3};\n\tmov.b64 B, {%4, %5};\n\t"
        "add.rn.f32x2 A, A, B;\n\tmov.b64 {%0, %1}, A;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 A, B;\n\tmov.b64 A, {%2, %3};\n\tmov.b64 B, {%4, %5};\n\t"
        "sub.rn.f32x2 A, A, B;\n\tmov.b64 {%0, %1}, A;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// Padded index of element i of a transform buffer.
__host__ __device__ __forceinline__ int pidx(int i) { return i + (i >> 4); }

// Twiddle table of a pass: entry (k, r) is exp(-2 pi i r k / (R Ns)), r = 1..R-1, k < Ns.  All threads of the CTA.
__device__ __forceinline__ void fill_table(float2 *tw, int R, int Ns)
{
    for (int i = threadIdx.x; i < Ns * (R - 1); i += blockDim.x) {
        const int k = i / (R - 1), r = i - k * (R - 1) + 1;
        float sn, cs;
        sincospif(-2.0f * (float)(r * k) / (float)(R * Ns), &sn, &cs);  // exact argument: R Ns is 2^n
        tw[i] = make_float2(cs, sn);
    }
}
template <int LG> __device__ __forceinline__ void fill_twiddles(float2 *tw)
{
    using F = Fft<LG>;
#pragma unroll
    for (int m = 1; m < F::NP; ++m) fill_table(tw + F::fwd_off(m), m == F::NP - 1 ? F::RL : 16, 1 << (4 * m));
    if constexpr (F::OWN_INV) {
#pragma unroll
        for (int m = 0; m < F::NP - 1; ++m) fill_table(tw + F::inv_off(m), 16, F::inv_span(m));
    }
}

// Forward DFTs of 2, 4, 8 and 16 points in registers (natural order).
__device__ __forceinline__ void dft2(float2 &a, float2 &b)
{
    const float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}
__device__ __forceinline__ void dft4(float2 &x0, float2 &x1, float2 &x2, float2 &x3)
{
    const float2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = csub(x1, x3);
    x0 = cadd(a, c);
    x2 = csub(a, c);
    x1 = make_float2(b.x + d.y, b.y - d.x);  // b - i d
    x3 = make_float2(b.x - d.y, b.y + d.x);  // b + i d
}
constexpr float kR2 = 0.70710678118654752440f;  // cos(pi/4)
constexpr float kC8 = 0.92387953251128675613f;  // cos(pi/8)
constexpr float kS8 = 0.38268343236508977173f;  // sin(pi/8)

template <int R> __device__ __forceinline__ void dft(float2 (&v)[R]);
template <> __device__ __forceinline__ void dft<2>(float2 (&v)[2]) { dft2(v[0], v[1]); }
template <> __device__ __forceinline__ void dft<4>(float2 (&v)[4]) { dft4(v[0], v[1], v[2], v[3]); }
// 8 = 2 x 4: X[k + 4h] = E0[k] + (-1)^h W8^k E1[k], E_e = DFT4(x[e], x[e+2], x[e+4], x[e+6]).
template <> __device__ __forceinline__ void dft<8>(float2 (&v)[8])
{
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const float2 t1 = make_float2(kR2 * (v[3].x + v[3].y), kR2 * (v[3].y - v[3].x));   // W8^1 = (r, -r)
    const float2 t2 = make_float2(v[5].y, -v[5].x);                                     // W8^2 = -i
    const float2 t3 = make_float2(kR2 * (v[7].y - v[7].x), -kR2 * (v[7].x + v[7].y));  // W8^3 = (-r, -r)
    const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = cadd(e0, v[1]);
    v[4] = csub(e0, v[1]);
    v[1] = cadd(e1, t1);
    v[5] = csub(e1, t1);
    v[2] = cadd(e2, t2);
    v[6] = csub(e2, t2);
    v[3] = cadd(e3, t3);
    v[7] = csub(e3, t3);
}
// 16 = 4 x 4: E_e = DFT4(x[e], x[e+4], x[e+8], x[e+12]); T_e[k] = W16^(e k) E_e[k];
// X[k + 4h] = DFT4_h(T_0[k], T_1[k], T_2[k], T_3[k]).
// DFT_4 of (x0, x1, 0, 0).
__device__ __forceinline__ void dft4_half(float2 x0, float2 x1, float2 &o0, float2 &o1, float2 &o2, float2 &o3)
{
    o0 = cadd(x0, x1);
    o2 = csub(x0, x1);
    o1 = make_float2(x0.x + x1.y, x0.y - x1.x);
    o3 = make_float2(x0.x - x1.y, x0.y + x1.x);
}
// The W16^(e k) of dft<16> on E_e[k] in v[e + 4k], then its second stage; LOW: outputs 0 .. 7 only.
template <bool LOW> __device__ __forceinline__ void dft16_second(float2 (&v)[16])
{
    const float2 w1 = make_float2(kC8, -kS8), w2 = make_float2(kR2, -kR2), w3 = make_float2(kS8, -kC8);
    const float2 w6 = make_float2(-kR2, -kR2), w9 = make_float2(-kC8, kS8);
    v[5] = cmul(v[5], w1);                          // e=1,k=1
    v[9] = cmul(v[9], w2);                          // e=1,k=2
    v[13] = cmul(v[13], w3);                        // e=1,k=3
    v[6] = cmul(v[6], w2);                          // e=2,k=1
    v[10] = make_float2(v[10].y, -v[10].x);         // e=2,k=2: W16^4 = -i
    v[14] = cmul(v[14], w6);                        // e=2,k=3
    v[7] = cmul(v[7], w3);                          // e=3,k=1
    v[11] = cmul(v[11], w6);                        // e=3,k=2
    v[15] = cmul(v[15], w9);                        // e=3,k=3
    float2 o[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 x0 = v[4 * k], x1 = v[4 * k + 1], x2 = v[4 * k + 2], x3 = v[4 * k + 3];
        const float2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), d = csub(x1, x3);
        o[k] = cadd(a, c);
        o[k + 4] = make_float2(b.x + d.y, b.y - d.x);
        if constexpr (!LOW) {
            o[k + 8] = csub(a, c);
            o[k + 12] = make_float2(b.x - d.y, b.y + d.x);
        }
    }
#pragma unroll
    for (int i = 0; i < (LOW ? 8 : 16); ++i) v[i] = o[i];
}
template <> __device__ __forceinline__ void dft<16>(float2 (&v)[16])
{
#pragma unroll
    for (int e = 0; e < 4; ++e) dft4(v[e], v[e + 4], v[e + 8], v[e + 12]);
    dft16_second<false>(v);
}
// Outputs 0 .. 7 of DFT_16.
__device__ __forceinline__ void dft16_low(float2 (&v)[16])
{
#pragma unroll
    for (int e = 0; e < 4; ++e) dft4(v[e], v[e + 4], v[e + 8], v[e + 12]);
    dft16_second<true>(v);
}
// DFT_R of R/2 values followed by R/2 zeros.
template <int R> __device__ __forceinline__ void dft_half(float2 (&v)[R])
{
    if constexpr (R == 2) {
        v[1] = v[0];
    } else if constexpr (R == 4) {
        dft4_half(v[0], v[1], v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        v[4] = v[5] = v[6] = v[7] = make_float2(0.f, 0.f);
        dft<8>(v);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) dft4_half(v[e], v[e + 4], v[e], v[e + 4], v[e + 8], v[e + 12]);
        dft16_second<false>(v);
    }
}

// Barrier of the TPF threads of transform group grp (named barrier 1 + grp, or
// the warp's own where groups share a warp): the groups of a CTA share only
// read-only tables, so none waits on another.
template <int TPF>
__device__ __forceinline__ void group_sync(int grp)
{
    if constexpr (TPF < 32)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(TPF) : "memory");
}

// Loads of butterfly j of a radix-R pass: x[j + r Q] times its twiddles.
template <int R, int P, int NS, bool FROM_HALF>
__device__ __forceinline__ void load_butterfly(float2 (&v)[R], const float2 *x, const float2 *tw, int j)
{
    constexpr int Q = P / R;
    const int k = j & (NS - 1);
    if constexpr (Q % 16 == 0) {  // pidx(j + r Q) = pidx(j) + r (Q + Q/16)
        const float2 *xs = x + pidx(j);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = xs[r * (Q + Q / 16)];
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = x[pidx(j + r * Q)];
    }
    if constexpr (NS > 1 && FROM_HALF) {  // tw[m] = w_P^m, m < P/2; w_P^(m + P/2) = -w_P^m
#pragma unroll
        for (int r = 1; r < R; ++r) {
            const int m = r * k * (P / (R * NS));
            float2 w = tw[m & (P / 2 - 1)];
            if (m & (P / 2)) w = make_float2(-w.x, -w.y);
            v[r] = cmul(v[r], w);
        }
    } else if constexpr (NS > 1) {
        const float2 *w = tw + k * (R - 1) - 1;
#pragma unroll
        for (int r = 1; r < R; ++r) v[r] = cmul(v[r], w[r]);
    }
}
// Its stores: y[(j - k) R + k + s Ns].
template <int R, int NS> __device__ __forceinline__ void store_butterfly(const float2 (&v)[R], float2 *y, int j)
{
    const int k = j & (NS - 1);
    const int o = (j - k) * R + k;
    if constexpr (NS % 16 == 0) {
        float2 *ys = y + pidx(o);
#pragma unroll
        for (int s2 = 0; s2 < R; ++s2) ys[s2 * (NS + NS / 16)] = v[s2];
    } else if constexpr (NS == 1 && R == 16) {  // o is a multiple of 16: o + s stays in one padding group
        float2 *ys = y + pidx(o);
#pragma unroll
        for (int s2 = 0; s2 < R; ++s2) ys[s2] = v[s2];
    } else {
#pragma unroll
        for (int s2 = 0; s2 < R; ++s2) y[pidx(o + s2 * NS)] = v[s2];
    }
}

// A radix-16 pass of span NS from x to y and the group's barrier.
template <int LG, int NS, bool FROM_HALF>
__device__ __forceinline__ void pass16(const float2 *x, float2 *y, const float2 *tw, int t, int grp)
{
    using F = Fft<LG>;
    constexpr int Q = F::P / 16, ITER = (Q + F::TPF - 1) / F::TPF;
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
        const int j = t + i * F::TPF;
        if ((Q % F::TPF) != 0 && j >= Q) break;
        float2 v[16];
        load_butterfly<16, F::P, NS, FROM_HALF>(v, x, tw, j);
        dft<16>(v);
        store_butterfly<16, NS>(v, y, j);
    }
    group_sync<F::TPF>(grp);
}
// Forward passes m = M .. NP - 2.
template <int LG, int M>
__device__ __forceinline__ void forward_passes(float2 *&x, float2 *&y, const float2 *tw, int t, int grp)
{
    using F = Fft<LG>;
    if constexpr (M <= F::NP - 2) {
        pass16<LG, (1 << (4 * M)), false>(x, y, tw + F::fwd_off(M), t, grp);
        float2 *z = x;
        x = y;
        y = z;
        forward_passes<LG, M + 1>(x, y, tw, t, grp);
    }
}
// Inverse radix-16 passes m = M .. NP - 3 (all but the last).
template <int LG, int M>
__device__ __forceinline__ void inverse_passes(float2 *&x, float2 *&y, const float2 *tw, int t, int grp)
{
    using F = Fft<LG>;
    if constexpr (M <= F::NP - 3) {
        if constexpr (LG == 13)
            pass16<LG, F::inv_span(M), true>(x, y, tw + F::fwd_off(F::NP - 1), t, grp);
        else
            pass16<LG, F::inv_span(M), false>(x, y, tw + F::inv_off(M), t, grp);
        float2 *z = x;
        x = y;
        y = z;
        inverse_passes<LG, M + 1>(x, y, tw, t, grp);
    }
}

// Filters one row pair.  in[i][r] is the packed sample x = j + r Q1 of butterfly j = t + i TPF (the caller's
// registers; 0 at x >= W), out[i][s] the filtered pair (a, -b) at column j + s QC of butterfly j = t + i TPF.  Every
// thread of the group calls it.  Buffer A is free again when it returns, B once the group has passed another barrier.
template <int LG>
__device__ __forceinline__ void filter_pair(const float2 (&in)[Fft<LG>::ITIN][Fft<LG>::IN],
                                            float2 (&out)[Fft<LG>::ITC][Fft<LG>::NC], float2 *A, float2 *B,
                                            const float2 *tw, const float *hf, int t, int grp)
{
    using F = Fft<LG>;
    constexpr int P = F::P, RL = F::RL, NS = P / RL;  // NS: span and butterflies of the last forward pass
    float2 *x = A, *y = B;
    // spectrum product and the inverse's first pass on the outputs X[j + s NS] of the last forward pass
    auto middle = [&](float2 (&v)[RL], int j) {
        dft<RL>(v);
#pragma unroll
        for (int s2 = 0; s2 < RL; ++s2) {
            const int k = j + s2 * NS;
            const float h = hf[k <= (P >> 1) ? k : P - k];
            v[s2] = make_float2(v[s2].x * h, -v[s2].y * h);  // conj(Z) * Hf
        }
        dft<RL>(v);
    };
    if constexpr (F::NP > 1) {
#pragma unroll
        for (int i = 0; i < F::ITIN; ++i) {
            const int j = t + i * F::TPF;
            if ((F::Q1 % F::TPF) != 0 && j >= F::Q1) break;
            float2 v[16];
#pragma unroll
            for (int r = 0; r < 8; ++r) v[r] = in[i][r];
            dft_half<16>(v);
            store_butterfly<16, 1>(v, x, j);
        }
        group_sync<F::TPF>(grp);
        forward_passes<LG, 1>(x, y, tw, t, grp);
        constexpr int ITER = (NS + F::TPF - 1) / F::TPF;
#pragma unroll(ITER <= 4 ? ITER : 4)
        for (int i = 0; i < ITER; ++i) {
            const int j = t + i * F::TPF;
            if ((NS % F::TPF) != 0 && j >= NS) break;
            float2 v[RL];
            load_butterfly<RL, P, NS, false>(v, x, tw + F::fwd_off(F::NP - 1), j);
            middle(v, j);
            store_butterfly<RL, 1>(v, y, j);
        }
        group_sync<F::TPF>(grp);
        float2 *z = x;
        x = y;
        y = z;
        inverse_passes<LG, 0>(x, y, tw, t, grp);
#pragma unroll
        for (int i = 0; i < F::ITC; ++i) {
            const int j = t + i * F::TPF;
            if ((F::QC % F::TPF) != 0 && j >= F::QC) break;
            float2 v[16];
            if constexpr (LG == 13)
                load_butterfly<16, P, P / 16, true>(v, x, tw + F::fwd_off(F::NP - 1), j);
            else
                load_butterfly<16, P, P / 16, false>(v, x, tw + F::inv_off(F::NP - 2), j);
            dft16_low(v);
#pragma unroll
            for (int s2 = 0; s2 < 8; ++s2) out[i][s2] = v[s2];
        }
    } else {  // p <= 16: one butterfly
        if (t == 0) {
            float2 v[RL];
#pragma unroll
            for (int r = 0; r < RL / 2; ++r) v[r] = in[0][r];
            dft_half<RL>(v);
#pragma unroll
            for (int s2 = 0; s2 < RL; ++s2) {
                const float h = hf[s2 <= (P >> 1) ? s2 : P - s2];
                v[s2] = make_float2(v[s2].x * h, -v[s2].y * h);
            }
            dft<RL>(v);
            store_butterfly<RL, 1>(v, x, 0);
        }
        group_sync<F::TPF>(grp);
        if (t < F::QC) out[0][0] = x[pidx(t)];
        group_sync<F::TPF>(grp);
    }
}

// Element offset of output row `row` (= b*H + r) of the raw-sample output.
__device__ __forceinline__ long long out_row_offset(const FiltParams &P, long long row, int &r)
{
    const long long b = row / P.L.H;
    r = (int)(row - b * P.L.H);
    return P.out_layout == TK_LAYOUT_SINOGRAM ? ((long long)r * P.L.N + b) * P.Wp : row * (long long)P.Wp;
}

// Shared memory of the filter kernels: twiddle tables, the spectrum, then per group two transform buffers and the
// first columns of its warps.
template <int LG> struct FiltSmem {
    float2 *tw, *A, *B, *edge;
    float *hf;
    __device__ __forceinline__ FiltSmem(float2 *base, int grp)
    {
        using F = Fft<LG>;
        tw = base;
        hf = reinterpret_cast<float *>(base + F::TW);
        A = reinterpret_cast<float2 *>(reinterpret_cast<char *>(hf + F::HF) + (size_t)grp * F::group_bytes());
        B = A + F::P + F::P / 16;
        edge = B + F::P + F::P / 16;
    }
};

// Raw samples of one row at a thread's inputs x = j + r Q1 (0 at x >= W and where not valid), as they are stored
// (a conversion here would wait for the load).
template <int LG>
__device__ __forceinline__ void load_inputs(const LoadParams &L, long long off, bool valid, int t,
                                            uint32_t (&v)[Fft<LG>::ITIN][Fft<LG>::IN])
{
    using F = Fft<LG>;
#pragma unroll
    for (int i = 0; i < F::ITIN; ++i)
#pragma unroll
        for (int r = 0; r < F::IN; ++r) {
            const int j = t + i * F::TPF, x = j + r * F::Q1;
            v[i][r] = 0u;
            if (valid && j < F::Q1 && x < L.W)
                v[i][r] = L.input_type == TK_INPUT_U16 ? __ldg(static_cast<const uint16_t *>(L.in) + off + x)
                                                       : __ldg(static_cast<const uint32_t *>(L.in) + off + x);
        }
}
// Preprocesses both rows' raw samples and packs them.
template <int LG>
__device__ __forceinline__ void pack_inputs(const LoadParams &L, int r_a, int r_b, bool valid, bool hasb, int t,
                                            const uint32_t (&a)[Fft<LG>::ITIN][Fft<LG>::IN],
                                            const uint32_t (&b)[Fft<LG>::ITIN][Fft<LG>::IN],
                                            float2 (&in)[Fft<LG>::ITIN][Fft<LG>::IN])
{
    using F = Fft<LG>;
    auto value = [&](uint32_t v) { return L.input_type == TK_INPUT_U16 ? (float)v : __uint_as_float(v); };
    const float rta = weight_row_term(L, r_a), rtb = weight_row_term(L, r_b);
    const bool maps = has_maps(L);
#pragma unroll
    for (int i = 0; i < F::ITIN; ++i) {
        const int j = t + i * F::TPF;
        // (r_a is a row of the detector only where valid, r_b only with hasb)
        auto one = [&](bool ok, int row, float rt, const uint32_t(&raw)[F::IN], float(&v)[F::IN]) {
            ok = ok && j < F::Q1;
            if (ok && maps) {
                float dk[F::IN], fl[F::IN];
                load_maps<F::IN>(L, row, j, F::Q1, dk, fl);
#pragma unroll
                for (int r = 0; r < F::IN; ++r)
                    v[r] = j + r * F::Q1 < L.W ? pre_maps(L, j + r * F::Q1, value(raw[r]), dk[r], fl[r], rt) : 0.f;
            } else {
#pragma unroll
                for (int r = 0; r < F::IN; ++r)
                    v[r] = ok && j + r * F::Q1 < L.W ? pre_scalar(L, j + r * F::Q1, value(raw[r]), rt) : 0.f;
            }
        };
        float va[F::IN], vb[F::IN];
        one(valid, r_a, rta, a[i], va);
        one(hasb, r_b, rtb, b[i], vb);
#pragma unroll
        for (int r = 0; r < F::IN; ++r) in[i][r] = make_float2(va[r], vb[r]);
    }
}

template <int LG>
__global__ void __launch_bounds__(Fft<LG>::NT, Fft<LG>::MINB) filter_fft_kernel(const __grid_constant__ FiltParams P)
{
    extern __shared__ __align__(16) float2 fsm[];
    using F = Fft<LG>;
    const int grp = threadIdx.x / F::TPF, t = threadIdx.x - grp * F::TPF;
    const FiltSmem<LG> S(fsm, grp);
    fill_twiddles<LG>(S.tw);
    for (int k = threadIdx.x; k <= F::P / 2; k += F::NT) S.hf[k] = P.Hf[k];
    const int W = P.L.W;
    float *out = static_cast<float *>(P.out);
    __syncthreads();

    // Raw samples of a pair group's two rows, fetched one group ahead so that
    // their latency overlaps the transforms of the current one.
    uint32_t raw_a[F::ITIN][F::IN], raw_b[F::ITIN][F::IN];
    auto fetch = [&](long long pgf) {
        const long long pr = pgf * F::G + grp;
        const bool vl = pr < P.npairs;
        const bool hb = vl && 2 * pr + 1 < P.nrows;
        int rr;
        const long long oa = vl ? in_row_offset(P.L, 2 * pr, rr) : 0;
        const long long ob = hb ? in_row_offset(P.L, 2 * pr + 1, rr) : 0;
        load_inputs<LG>(P.L, oa, vl, t, raw_a);
        load_inputs<LG>(P.L, ob, hb, t, raw_b);
    };
    if ((long long)blockIdx.x * F::G < P.npairs) fetch(blockIdx.x);
    for (long long pg = blockIdx.x; pg * F::G < P.npairs; pg += gridDim.x) {
        const long long pair = pg * F::G + grp;
        const bool valid = pair < P.npairs;
        const long long ra = 2 * pair, rb = 2 * pair + 1;
        const bool hasb = valid && rb < P.nrows;
        int r_a = 0, r_b = 0;
        const long long qa = valid ? out_row_offset(P, ra, r_a) : 0, qb = hasb ? out_row_offset(P, rb, r_b) : 0;
        float2 in[F::ITIN][F::IN], q[F::ITC][F::NC];
        pack_inputs<LG>(P.L, r_a, r_b, valid, hasb, t, raw_a, raw_b, in);
        if ((pg + gridDim.x) * F::G < P.npairs) fetch(pg + gridDim.x);
        filter_pair<LG>(in, q, S.A, S.B, S.tw, S.hf, t, grp);
        if (valid) {
            const float rta = weight_row_term(P.L, r_a), rtb = weight_row_term(P.L, r_b);
#pragma unroll
            for (int i = 0; i < F::ITC; ++i)
#pragma unroll
                for (int s2 = 0; s2 < F::NC; ++s2) {
                    const int j = t + i * F::TPF, c = j + s2 * F::QC;
                    if (j >= F::QC || c >= W) continue;
                    out[qa + c] = q[i][s2].x * (P.weight_out ? cosine_weight_rt(P.L, rta, c) : 1.f);
                    if (hasb) out[qb + c] = -q[i][s2].y * (P.weight_out ? cosine_weight_rt(P.L, rtb, c) : 1.f);
                }
        }
    }
}

// ---------------------------------------------------------------------------
// Filter straight into a bilinear coefficient image.
//
// A work unit is RC consecutive detector rows of one projection.  The group
// filters the unit's rows two at a time (plus the first row of the next unit,
// which the last coefficient row needs) and keeps the previous filtered row in
// registers (each thread holds it at its own columns), so every coefficient
// row r is formed from filtered rows r and r+1 without another pass over HBM.
// Rows 2i and 2i + 1 of a frame always share a transform, the next unit's first
// row and its partner too (the partner is used there only): a transform's
// rounding depends on both of its rows, and RC on the number of frames in the
// call, which a frame's entries must not follow.
// A thread's columns are j + s QC; column c + 1 sits in the next lane, or, for
// the last lane of a warp, in the next warp's first columns, which pass through
// shared memory.  Samples outside the detector are 0.

template <int MODE, int LG>
__global__ void __launch_bounds__(Fft<LG>::NT, Fft<LG>::MINB) filter_coef_kernel(const __grid_constant__ FiltParams P)
{
    extern __shared__ __align__(16) float2 fsm[];
    using F = Fft<LG>;
    static_assert(F::ITC == 1 && F::ITIN == 1, "one butterfly per thread (p <= 4096)");
    constexpr int NC = F::NC;
    const int grp = threadIdx.x / F::TPF, t = threadIdx.x - grp * F::TPF;
    const FiltSmem<LG> S(fsm, grp);
    fill_twiddles<LG>(S.tw);
    for (int k = threadIdx.x; k <= F::P / 2; k += F::NT) S.hf[k] = P.Hf[k];
    const float sigma = P.q_scale ? *P.q_scale : 1.f;
    const int W = P.L.W, H = P.L.H, RC = P.rc;
    const int Wc = MODE == TK_F32_COEF ? W : ((W + 1) & ~1);
    __syncthreads();

    for (long long ug = blockIdx.x; ug * F::G < P.nunits; ug += gridDim.x) {
        const long long unit = ug * F::G + grp;
        const bool valid = unit < P.nunits;
        const long long b = valid ? unit / P.nchunks : 0;
        const int r0 = valid ? (int)(unit - b * P.nchunks) * RC : 0;
        // the frame of the input and of the output (frame groups: fgrp frames every fstride)
        const long long bf = P.fgrp > 0 ? b / P.fgrp * P.fstride + b % P.fgrp : b;
        const int r1 = min(r0 + RC, H);         // coefficient rows [r0, r1)
        const int rend = min(r0 + RC, H - 1);   // last filtered row (includes the next unit's first)
        const int npair = valid ? (rend - r0 + 2) / 2 : 0;
        // every group runs the same number of pair steps
        const int steps = (min(RC, H - 1) + 2) / 2;
        // Raw samples of the next step's two rows, fetched one step ahead so that their latency
        // overlaps the transforms.
        uint32_t raw_a[1][F::IN], raw_b[1][F::IN];
        auto fetch = [&](int kk) {
            const bool lv = valid && kk < npair;
            const int qa = r0 + 2 * kk, qb = qa + 1;
            const bool hb = lv && qb < H;
            int rr;
            const long long oa = lv ? in_row_offset(P.L, bf * H + qa, rr) : 0;
            const long long ob = hb ? in_row_offset(P.L, bf * H + qb, rr) : 0;
            load_inputs<LG>(P.L, oa, lv, t, raw_a);
            load_inputs<LG>(P.L, ob, hb, t, raw_b);
        };
        float pq[NC], pd[NC];  // the previous filtered row (ra - 1) at this thread's columns: value, difference to c + 1
#pragma unroll
        for (int s2 = 0; s2 < NC; ++s2) pq[s2] = pd[s2] = 0.f;
        fetch(0);
        for (int k = 0; k < steps; ++k) {
            const bool live = valid && k < npair;
            const int ra = r0 + 2 * k, rb = ra + 1;
            const bool hasb = live && rb < H;
            float2 in[1][F::IN], q[1][NC];
            pack_inputs<LG>(P.L, ra, rb, live, hasb, t, raw_a, raw_b, in);
            if (k + 1 < steps) fetch(k + 1);
            filter_pair<LG>(in, q, S.A, S.B, S.tw, S.hf, t, grp);
            // rows ra (x) and rb (y); columns past W read as 0
#pragma unroll
            for (int s2 = 0; s2 < NC; ++s2) {
                const bool in_row = t < F::QC && t + s2 * F::QC < W;
                q[0][s2] = in_row ? make_float2(q[0][s2].x * sigma, hasb ? -q[0][s2].y * sigma : 0.f)
                                  : make_float2(0.f, 0.f);
            }
            if (t % 32 == 0) {
#pragma unroll
                for (int s2 = 0; s2 < NC; ++s2) S.edge[(t >> 5) * (NC + 1) + s2] = q[0][s2];
            }
            group_sync<F::TPF>(grp);
            const int next = F::next_edge(t);
            const size_t base = ((size_t)bf * H + ra) * Wc;
#pragma unroll
            for (int s2 = 0; s2 < NC; ++s2) {
                const int c = t + s2 * F::QC;
                const float2 v = q[0][s2];
                float2 n;
                n.x = __shfl_down_sync(0xffffffffu, v.x, 1);
                n.y = __shfl_down_sync(0xffffffffu, v.y, 1);
                if (next >= 0) n = c + 1 < W ? S.edge[next + s2] : make_float2(0.f, 0.f);
                const float da = n.x - v.x, db = n.y - v.y;
                if (live && t < F::QC && c < Wc) {
                    if (ra - 1 >= r0)  // the previous row, followed by row ra
                        store_coef<MODE>(P.out, base - Wc + c, pq[s2], pd[s2], v.x - pq[s2], da - pd[s2]);
                    if (ra < r1)  // followed by row rb, or 0 below the detector's last row
                        store_coef<MODE>(P.out, base + c, v.x, da, v.y - v.x, db - da);
                    if (hasb && rb < r1 && rb == rend)  // detector's last row, nothing follows
                        store_coef<MODE>(P.out, base + Wc + c, v.y, db, 0.f - v.y, 0.f - db);
                }
                pq[s2] = v.y;
                pd[s2] = db;
            }
        }
    }
}

// max(m, |v|); a NaN sample leaves the bound unchanged.
__device__ __forceinline__ float bound_of(float m, float v)
{
    v = fabsf(v);
    return v == v ? fmaxf(m, v) : m;
}
// max |preprocessed sample| over the whole input, as float bits in *maxbits.
// Each warp takes whole detector rows (lanes on consecutive columns), so the
// row's offset is formed once per row rather than by a division per sample.
// With dark and flat maps up to eight samples per lane are loaded with their
// pixels before the first is used: 301 x 389 x 500 uint16 135 -> 124 us.  Rows
// of up to 128 samples take runs of four, of up to 64 of two: of eight, most
// would lie past the row (19392 rows of 33 into FP16, with the filter, 45.1 us
// with runs of eight, 41.1 so).
// (Skipping samples that cannot pass the lane's maximum, by two compares, cost
// more in divergence than the logarithms it saved: 164 us.)
template <int RUN>
__device__ __forceinline__ float prescan_maps_row(const LoadParams &L, long long off, int r, float rt, int lane, float m)
{
    for (int x0 = lane; x0 < L.W; x0 += 32 * RUN) {
        float raw[RUN], dk[RUN], fl[RUN];
#pragma unroll
        for (int i = 0; i < RUN; ++i) raw[i] = x0 + 32 * i < L.W ? load_raw(L, off, x0 + 32 * i) : 0.f;
        load_maps<RUN>(L, r, x0, 32, dk, fl);
#pragma unroll
        for (int i = 0; i < RUN; ++i)
            if (x0 + 32 * i < L.W) m = bound_of(m, pre_maps(L, x0 + 32 * i, raw[i], dk[i], fl[i], rt));
    }
    return m;
}
__global__ void __launch_bounds__(256) prescan_kernel(const __grid_constant__ LoadParams L, long long nrows,
                                                      unsigned *maxbits)
{
    const bool maps = has_maps(L);
    float m = 0.f;
    const int lane = threadIdx.x & 31;
    const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; row < nrows; row += nwarps) {
        int r;
        const long long off = in_row_offset(L, row, r);
        const float rt = weight_row_term(L, r);
        if (maps) {
            m = L.W <= 64    ? prescan_maps_row<2>(L, off, r, rt, lane, m)
                : L.W <= 128 ? prescan_maps_row<4>(L, off, r, rt, lane, m)
                             : prescan_maps_row<8>(L, off, r, rt, lane, m);
        } else {
            for (int x = lane; x < L.W; x += 32) m = bound_of(m, pre_scalar(L, x, load_raw(L, off, x), rt));
        }
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ float wm[8];
    if ((threadIdx.x & 31) == 0) wm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, wm[w]);
        atomicMax(maxbits, __float_as_uint(m));
    }
}

// Turns the bound into a power-of-two storage scale: |q| <= max * L1K.  With
// bound = f 2^eb (f in [0.5, 1)), 2^(14 - eb) is the largest power of two s
// with s bound <= 2^14 = kScaleTarget (exact exponent arithmetic, FP32).
__global__ void scale_finalize_kernel(float *scale, float L1K)
{
    const float m = __uint_as_float(*reinterpret_cast<unsigned *>(scale));
    float s = 1.f;
    const float bound = m * L1K * (1.f + 0x1p-20f);  // rounded up past the two FP32 roundings
    if (bound > 0.f && isfinite(bound)) {
        int eb = 0;
        (void)frexpf(bound, &eb);
        const int e = max(-100, min(100, 14 - eb));
        s = ldexpf(1.f, e);
    }
    *scale = s;
}

__global__ void set_scale_kernel(float *scale, float v) { *scale = v; }

// ---------------------------------------------------------------------------
// host: filter spectrum (FP64), cached per (W, tau, window, p)

struct Spectrum {
    int p;
    std::vector<float> Hf;  // p/2 + 1
    double L1K;             // sum_n |K[n]|, K = unnormalised spatial kernel, |n| < W
};

// FilteredBackProjection::RamLak (kernel.cu:792-802), float result.
static float ramlak_ref(int v, float sm)
{
    if (v == 0) return (float)(1. / (4. * sm * sm));
    if ((v % 2) == 0) return 0.f;
    return (float)(-1. / (v * v * M_PI * M_PI * sm * sm));
}

static double window_gain(int window, int k, int p)
{
    const double f = (double)k / (double)p;
    if (window == TK_WINDOW_SHEPP_LOGAN) return k == 0 ? 1.0 : std::sin(M_PI * f) / (M_PI * f);
    if (window == TK_WINDOW_HANN) return 0.5 * (1.0 + std::cos(2.0 * M_PI * f));
    return 1.0;
}

static const Spectrum &spectrum(int W, float tau, int window, int p)
{
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, int, int>, Spectrum> cache;
    uint32_t tb;
    std::memcpy(&tb, &tau, 4);
    const auto key = std::make_tuple(W, tb, window, p);
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    Spectrum sp;
    sp.p = p;
    // h[i] = RamLak(i - W/2)/2 for i < W, zero padded (FillFilter, kernel.cu:783-790)
    std::vector<float> h(W);
    for (int i = 0; i < W; ++i) h[i] = ramlak_ref(i - W / 2, tau) / 2;
    std::vector<double> ct(p), st(p);
    for (int m = 0; m < p; ++m) {
        ct[m] = std::cos(2.0 * M_PI * m / p);
        st[m] = std::sin(2.0 * M_PI * m / p);
    }
    std::vector<double> Hd(p / 2 + 1);
    for (int k = 0; k <= p / 2; ++k) {
        double sr = 0, si = 0;
        for (int i = 0; i < W; ++i) {
            const int m = (int)(((long long)k * i) % p);
            sr += h[i] * ct[m];
            si -= h[i] * st[m];
        }
        // AbsKernel: sampling * |X| (kernel.cu:55-64)
        Hd[k] = (double)tau * std::sqrt(sr * sr + si * si) * window_gain(window, k, p);
    }
    sp.Hf.resize(p / 2 + 1);
    for (int k = 0; k <= p / 2; ++k) sp.Hf[k] = (float)Hd[k];
    double L1 = 0;
    for (int n = 0; n < W; ++n) {
        double s = Hd[0] + Hd[p / 2] * ((n & 1) ? -1.0 : 1.0);
        for (int k = 1; k < p / 2; ++k) s += 2.0 * Hd[k] * ct[(int)(((long long)k * n) % p)];
        L1 += (n == 0 ? 1.0 : 2.0) * std::fabs(s);
    }
    sp.L1K = L1;
    return cache.emplace(key, std::move(sp)).first->second;
}

// The kernel instantiated for storage `precision` and pad length 2^lg
// (2 <= lg <= 13; coefficient storage up to lg = 12, i.e. W <= 2048).
struct FiltKernel {
    const void *fn = nullptr;
    size_t smem = 0;
    int groups = 1, threads = 0;
};
template <int LG> static FiltKernel filter_kernel_lg(int precision)
{
    FiltKernel k;
    k.smem = Fft<LG>::smem();
    k.groups = Fft<LG>::G;
    k.threads = Fft<LG>::NT;
    switch (precision) {
    case TK_F32: k.fn = reinterpret_cast<const void *>(&filter_fft_kernel<LG>); break;
    case TK_F16: if constexpr (LG <= 12) k.fn = reinterpret_cast<const void *>(&filter_coef_kernel<TK_F16, LG>); break;
    case TK_BF16: if constexpr (LG <= 12) k.fn = reinterpret_cast<const void *>(&filter_coef_kernel<TK_BF16, LG>); break;
    case TK_F32_COEF:
        if constexpr (LG <= 12) k.fn = reinterpret_cast<const void *>(&filter_coef_kernel<TK_F32_COEF, LG>);
        break;
    }
    return k;
}

static FiltKernel filter_kernel(int precision, int lg)
{
    switch (lg) {
    case 2: return filter_kernel_lg<2>(precision);
    case 3: return filter_kernel_lg<3>(precision);
    case 4: return filter_kernel_lg<4>(precision);
    case 5: return filter_kernel_lg<5>(precision);
    case 6: return filter_kernel_lg<6>(precision);
    case 7: return filter_kernel_lg<7>(precision);
    case 8: return filter_kernel_lg<8>(precision);
    case 9: return filter_kernel_lg<9>(precision);
    case 10: return filter_kernel_lg<10>(precision);
    case 11: return filter_kernel_lg<11>(precision);
    case 12: return filter_kernel_lg<12>(precision);
    case 13: return filter_kernel_lg<13>(precision);
    }
    return FiltKernel{};
}

// Rows per work unit of a coefficient image: each of the `slots` resident groups takes ceil(units / slots) units of
// (rc + 2) / 2 pair steps (the first row of the next unit is filtered too), so unit sizes that leave the last round
// nearly empty cost up to a round.  Picks the number of units per projection with the fewest steps; 90 x 1024 rows on
// 608 groups: 54 rows, 84 steps, against 64 rows, 99 steps (that filter 668 -> 622 us).
static int rows_per_unit(int N, int H, long long slots)
{
    long long best = -1;
    int rc = 64;
    for (int n = 1; n <= std::max(1, H / 8); ++n) {
        const int r = ((H + n - 1) / n + 1) & ~1;  // even: the same row pairs whatever the unit
        const long long units = (long long)N * ((H + r - 1) / r);
        const long long cost = (units + slots - 1) / slots * ((std::min(r, H - 1) + 2) / 2);
        if (best < 0 || cost < best) {
            best = cost;
            rc = r;
        }
    }
    return rc;
}

static int launch_filter_typed(FiltParams &P, int p, cudaStream_t stream, int precision)
{
    const FiltKernel k = filter_kernel(precision, P.lg);
    const void *fn = k.fn;
    TK_CHECK(fn, TK_ERR_UNSUPPORTED, "filter: no kernel for pad length %d with this storage", p);
    const int G = k.groups;
    const size_t smem = k.smem;
    TK_CHECK(smem <= 227 * 1024, TK_ERR_UNSUPPORTED, "filter: pad length %d needs too much shared memory", p);
    TK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int dev = 0, sms = 0, per_sm = 0;
    TK_CUDA(cudaGetDevice(&dev));
    TK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, k.threads, smem));
    if (per_sm < 1) per_sm = 1;
    if (is_coef(precision)) {
        P.rc = rows_per_unit(P.L.N, P.L.H, (long long)sms * per_sm * G);
        P.nchunks = (P.L.H + P.rc - 1) / P.rc;
        P.nunits = (long long)P.L.N * P.nchunks;
    }
    const long long work = is_coef(precision) ? P.nunits : P.npairs;
    const long long groups = (work + G - 1) / G;
    const long long grid = std::min<long long>(groups, (long long)sms * per_sm);
    void *args[] = {&P};
    TK_CUDA(cudaLaunchKernel(fn, dim3((unsigned)std::max<long long>(grid, 1)), dim3(k.threads), args, smem,
                             stream));
    count_launch();
    return TK_OK;
}

int launch_filter(const tk_geometry &g, const void *d_in, int input_type, int layout, const tk_flatfield *ff,
                  int window, void *d_q, int precision, float *d_q_scale, cudaStream_t stream, int fgrp, int fstride,
                  int form)
{
    if (int rc = validate_geometry(&g)) return rc;
    TK_CHECK(fgrp <= 0 || (is_coef(precision) && layout == TK_LAYOUT_PROJECTION && fstride >= fgrp), TK_ERR_INVALID,
             "filter: frame groups need a coefficient image from detector frames");
    TK_CHECK(d_in && d_q, TK_ERR_INVALID, "filter: null device pointer");
    TK_CHECK(input_type == TK_INPUT_F32 || input_type == TK_INPUT_U16, TK_ERR_INVALID, "filter: bad input type");
    TK_CHECK(layout == TK_LAYOUT_SINOGRAM || layout == TK_LAYOUT_PROJECTION, TK_ERR_INVALID, "filter: bad layout");
    TK_CHECK(window >= TK_WINDOW_RAMLAK && window <= TK_WINDOW_HANN, TK_ERR_INVALID, "filter: bad window");
    TK_CHECK(valid_precision(precision), TK_ERR_INVALID, "filter: bad precision");
    const bool sixteen = precision == TK_F16 || precision == TK_BF16;
    TK_CHECK(!sixteen || d_q_scale, TK_ERR_INVALID, "filter: 16-bit storage needs d_q_scale");
    TK_CHECK(fgrp <= 0 || !sixteen || (input_type == TK_INPUT_U16 && ff && !ff->dark && !ff->flat), TK_ERR_INVALID,
             "filter: frame groups need a storage scale known without a scan of the data");
    TK_CHECK(input_type == TK_INPUT_F32 || ff, TK_ERR_INVALID, "filter: raw input needs flat-field parameters");
    const int p = reference_pad_length(g.W);
    TK_CHECK(p <= 2 * (kMaxHf - 1), TK_ERR_UNSUPPORTED, "filter: W = %d exceeds the supported 4096", g.W);
    TK_CHECK(!is_coef(precision) || p <= 4096, TK_ERR_UNSUPPORTED,
             "filter: coefficient storage supports W <= 2048 (W = %d)", g.W);

    static thread_local FiltParams P;  // ~16 KB: keep off the stack
    std::memset(&P, 0, sizeof(P));
    LoadParams &L = P.L;
    L.in = d_in;
    L.W = g.W;
    L.N = g.N;
    L.H = g.H;
    L.layout = layout;
    L.input_type = input_type;
    L.in_pitch = g.W;
    L.weight_in = 1;
    L.cX = g.cX;
    L.cZ = g.cZ;
    L.D = g.D;
    L.A = 1.f;
    if (input_type == TK_INPUT_U16) {
        TK_CHECK(ff->floor_counts > 0.f, TK_ERR_INVALID, "filter: floor_counts must be > 0");
        TK_CHECK(ff->flat || ff->flat_value > 0.f, TK_ERR_INVALID, "filter: flat field missing");
        L.dark = ff->dark;
        L.flat = ff->flat;
        L.dark_v = ff->dark_value;
        L.flat_v = ff->flat_value;
        L.A = ff->A;
        L.B = ff->B;
        L.invert = ff->invert ? 1 : 0;
        L.floor_counts = ff->floor_counts;
    }
    finish_load_params(L);
    const Spectrum &sp = spectrum(g.W, g.tau, window, p);
    P.out = d_q;
    P.out_layout = TK_LAYOUT_PROJECTION;
    P.weight_out = 0;
    P.nrows = (long long)g.N * g.H;
    P.npairs = (P.nrows + 1) / 2;
    P.Wp = row_pitch(g.W);
    P.p = p;
    int lg = 0;
    while ((1 << lg) < p) ++lg;
    P.lg = lg;
    P.precision = precision;
    P.fgrp = fgrp > 0 ? fgrp : 0;
    P.fstride = fgrp > 0 ? fstride : 0;
    std::memcpy(P.Hf, sp.Hf.data(), sizeof(float) * sp.Hf.size());

    if (!sixteen) {
        P.q_scale = nullptr;
        if (d_q_scale) {
            set_scale_kernel<<<1, 1, 0, stream>>>(d_q_scale, 1.f);
            count_launch();
        }
    } else if (input_type == TK_INPUT_U16 && !ff->dark && !ff->flat) {
        // Scalar flat/dark: |A log(num/den) + B| is bounded without looking at the
        // data, since num in [floor, 65535] and den = max(flat - dark, floor).
        const double fl = ff->floor_counts, den = std::fmax((double)ff->flat_value - ff->dark_value, fl);
        const double lg = std::fmax(std::fabs(std::log(fl / den)), std::fabs(std::log(65535.0 / fl)));
        const double bound = (std::fabs((double)ff->A) * lg + std::fabs((double)ff->B)) * sp.L1K;
        int e = bound > 0 ? (int)std::floor(std::log2((double)kScaleTarget / bound)) : 0;
        e = std::max(-100, std::min(100, e));
        set_scale_kernel<<<1, 1, 0, stream>>>(d_q_scale, (float)std::ldexp(1.0, e));
        count_launch();
        P.q_scale = d_q_scale;
    } else {
        TK_CUDA(cudaMemsetAsync(d_q_scale, 0, sizeof(float), stream));
        int dev = 0, sms = 0;
        TK_CUDA(cudaGetDevice(&dev));
        TK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        prescan_kernel<<<sms * 4, 256, 0, stream>>>(L, P.nrows, reinterpret_cast<unsigned *>(d_q_scale));
        scale_finalize_kernel<<<1, 1, 0, stream>>>(d_q_scale, (float)sp.L1K);
        count_launch(2);  // prescan + finalize
        P.q_scale = d_q_scale;
    }
    TK_CUDA(cudaGetLastError());
    const int use = form <= TK_FILTER_AUTO ? filter_form_for(g.W, precision)
                    : (form == TK_FILTER_TOEPLITZ && toeplitz_supported(g.W, precision, TK_LAYOUT_PROJECTION))
                        ? TK_FILTER_TOEPLITZ
                        : TK_FILTER_FFT;
    if (use == TK_FILTER_TOEPLITZ)
        return launch_filter_toeplitz(L, P.Hf, p, d_q, precision, P.q_scale, P.nrows, storage_pitch(g.W, precision),
                                      P.fgrp, P.fstride, stream);
    return launch_filter_typed(P, p, stream, precision);
}

// Filter form selection (tk_filter_select_form).  TK_FILTER_AUTO takes the
// tensor-core Toeplitz product for 16-bit storage up to kToeplitzAutoMaxW,
// where it measured faster than the FFT (360 uint16 frames into FP16
// coefficients: 2.2x at W = 128, 1.5x at 192, 1.4x at 256 and 384, 1.1x at
// 512), and the FFT otherwise.  FP32 storage keeps the FFT: the split-BF16
// product carries about 2e-5 relative error on the filtered values, below
// 16-bit storage rounding (2^-12 or coarser) but above the FP32 forms' 1e-5
// reconstruction bound.
static int g_filter_form = TK_FILTER_AUTO;
constexpr int kToeplitzAutoMaxW = 512;

int filter_form_for(int W, int precision)
{
    const bool ok = toeplitz_supported(W, precision, TK_LAYOUT_PROJECTION);
    if (g_filter_form == TK_FILTER_TOEPLITZ) return ok ? TK_FILTER_TOEPLITZ : TK_FILTER_FFT;
    if (g_filter_form == TK_FILTER_FFT) return TK_FILTER_FFT;
    const bool sixteen = precision == TK_F16 || precision == TK_BF16;
    return ok && sixteen && W <= kToeplitzAutoMaxW ? TK_FILTER_TOEPLITZ : TK_FILTER_FFT;
}

// Transpose of the filter stage for the adjoint: the ramp filter is a
// symmetric Toeplitz operator (its spectrum is real and even) and the cosine
// weight is diagonal, so (F W)^T = W F.  Reads a [N][H][Wp] FP32 gradient,
// filters each row with the same spectrum and unnormalised scale, multiplies
// by the cosine weight and writes FP32 in `layout` with row pitch W.
int launch_filter_transpose(const tk_geometry &g, const float *d_qbar, int window, float *d_pbar, int layout,
                            cudaStream_t stream)
{
    if (int rc = validate_geometry(&g)) return rc;
    TK_CHECK(d_qbar && d_pbar, TK_ERR_INVALID, "filter transpose: null device pointer");
    TK_CHECK(layout == TK_LAYOUT_SINOGRAM || layout == TK_LAYOUT_PROJECTION, TK_ERR_INVALID, "bad layout");
    TK_CHECK(window >= TK_WINDOW_RAMLAK && window <= TK_WINDOW_HANN, TK_ERR_INVALID, "bad window");
    const int p = reference_pad_length(g.W);
    TK_CHECK(p <= 2 * (kMaxHf - 1), TK_ERR_UNSUPPORTED, "filter: W = %d exceeds the supported 4096", g.W);
    static thread_local FiltParams P;
    std::memset(&P, 0, sizeof(P));
    LoadParams &L = P.L;
    L.in = d_qbar;
    L.W = g.W;
    L.N = g.N;
    L.H = g.H;
    L.layout = TK_LAYOUT_PROJECTION;
    L.input_type = TK_INPUT_F32;
    L.in_pitch = row_pitch(g.W);
    L.weight_in = 0;
    L.cX = g.cX;
    L.cZ = g.cZ;
    L.D = g.D;
    L.A = 1.f;
    finish_load_params(L);
    const Spectrum &sp = spectrum(g.W, g.tau, window, p);
    P.out = d_pbar;
    P.out_layout = layout;
    P.weight_out = 1;
    P.q_scale = nullptr;
    P.nrows = (long long)g.N * g.H;
    P.npairs = (P.nrows + 1) / 2;
    P.Wp = g.W;  // dense output rows
    P.p = p;
    int lg = 0;
    while ((1 << lg) < p) ++lg;
    P.lg = lg;
    P.precision = TK_F32;
    std::memcpy(P.Hf, sp.Hf.data(), sizeof(float) * sp.Hf.size());
    return launch_filter_typed(P, p, stream, TK_F32);
}

}  // namespace tk

extern "C" int tk_filter_select_form(int form)
{
    if (form < TK_FILTER_AUTO || form > TK_FILTER_TOEPLITZ) {
        tk::set_error("no filter form %d", form);
        return TK_ERR_INVALID;
    }
    tk::g_filter_form = form;
    return TK_OK;
}

extern "C" int tk_filter_form_for(int W, int precision) { return tk::filter_form_for(W, precision); }

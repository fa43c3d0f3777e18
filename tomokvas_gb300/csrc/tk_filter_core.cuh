// tk_filter_core.cuh -- device pieces shared by the ramp-filter kernels
// (the shared-memory FFT in tk_filter.cu, the tensor-core Toeplitz product in
// tk_toeplitz.cu): the raw-input description, the fused preprocessing of a
// sample (flat field + log, cosine weight) and the coefficient-entry writer.
#pragma once

#include "tk_common.cuh"

namespace tk {

struct LoadParams {
    const void *in;
    const float *dark, *flat;
    float dark_v, flat_v, A, B, floor_counts;
    int invert;
    int W, N, H, layout, input_type;
    int in_pitch;   // elements between consecutive input rows of one layout line (W, or Wp)
    int weight_in;  // apply the cosine weight while loading (forward); 0 for the transpose
    float cX, cZ, D;
    float D2;       // D * D
    float inv_den;  // 1 / max(flat - dark, floor) for scalar flat/dark
    int gran;       // rows start aligned to and span whole units of 16, 8 or 4 bytes; 0: none of these
    int map_vec;    // dark and flat rows start 16-byte aligned and span whole 16-byte chunks
};

// Element offset of the first sample of output row `row` (= b*H + r) in the input.
__device__ __forceinline__ long long in_row_offset(const LoadParams &L, long long row, int &r)
{
    const long long b = row / L.H;
    r = (int)(row - b * L.H);
    return L.layout == TK_LAYOUT_SINOGRAM ? ((long long)r * L.N + b) * L.in_pitch : row * (long long)L.in_pitch;
}

// row[x] *= distance / sqrt(ce*ce + distance*distance + cs*cs)  (kernel.cu:195-199),
// evaluated as D rsqrt(ce^2 + (cs^2 + D^2)) with the row term cs^2 + D^2
// formed once per row (within 2 ulp of the IEEE divide and square root).
__device__ __forceinline__ float weight_row_term(const LoadParams &L, int r)
{
    const float cs = (float)r - L.cZ;
    return fmaf(cs, cs, L.D2);
}
__device__ __forceinline__ float cosine_weight_rt(const LoadParams &L, float rt, int x)
{
    const float ce = (float)x - L.cX;
    return L.D * rsqrtf(fmaf(ce, ce, rt));
}

// Raw sample x of the row at element offset off (counts as float for u16).
__device__ __forceinline__ float load_raw(const LoadParams &L, long long off, int x)
{
    return L.input_type == TK_INPUT_U16 ? (float)static_cast<const uint16_t *>(L.in)[off + x]
                                        : static_cast<const float *>(L.in)[off + x];
}

// Preprocessing of a raw sample: flat-field + log if raw counts
// (rsq_load.cpp:299-325: A log(num / den) + B, num = max(I - dark, floor),
// den = max(flat - dark, floor); here in FP32 with __logf, absolute error
// below 4e-7 for transmissions near 1), then the cosine weight (kernel.cu:
// 195-199).  rt is the row's weight_row_term.
__host__ __device__ __forceinline__ bool has_maps(const LoadParams &L)
{
    return L.input_type == TK_INPUT_U16 && (L.dark || L.flat);
}
// Transmission -> line integral, weighted.
__device__ __forceinline__ float pre_finish(const LoadParams &L, int x, float t, float rt)
{
    float val = fmaf(L.A, __logf(t), L.B);
    if (L.invert) val = -val;
    return L.weight_in ? val * cosine_weight_rt(L, rt, x) : val;
}
// With maps: dk and fl are the pixel's dark and flat.
__device__ __forceinline__ float pre_maps(const LoadParams &L, int x, float raw, float dk, float fl, float rt)
{
    return pre_finish(L, x, __fdividef(fmaxf(raw - dk, L.floor_counts), fmaxf(fl - dk, L.floor_counts)), rt);
}
// Without: FP32 line integrals, or counts with a scalar dark and flat.
__device__ __forceinline__ float pre_scalar(const LoadParams &L, int x, float raw, float rt)
{
    if (L.input_type == TK_INPUT_U16)
        return pre_finish(L, x, fmaxf(raw - L.dark_v, L.floor_counts) * L.inv_den, rt);
    return L.weight_in ? raw * cosine_weight_rt(L, rt, x) : raw;
}
// Dark and flat of the pixels x0, x0 + step, ... of row r (N of them, those below W).  A caller loads a run of
// them before it uses the first: one by one, each sample would wait for its own two loads.
template <int N>
__device__ __forceinline__ void load_maps(const LoadParams &L, int r, int x0, int step, float (&dk)[N], float (&fl)[N])
{
    const size_t row = (size_t)r * L.W;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int x = x0 + i * step;
        dk[i] = L.dark && x < L.W ? __ldg(L.dark + row + x) : L.dark_v;
        fl[i] = L.flat && x < L.W ? __ldg(L.flat + row + x) : L.flat_v;
    }
}
// Preprocesses the eight counts x0 .. x0 + 7 (x0 a multiple of 8, below W) of row r in place, with maps, which are
// read four pixels at a time, in 16-byte loads where they allow it; samples at or past W become 0.
__device__ __forceinline__ void pre8_maps(const LoadParams &L, int r, int x0, float rt, float (&v)[8])
{
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        float dk[4], fl[4];
        if (L.map_vec && x0 + h < L.W) {
            const size_t at = (size_t)r * L.W + x0 + h;
            const float4 d = L.dark ? __ldg(reinterpret_cast<const float4 *>(L.dark + at))
                                    : make_float4(L.dark_v, L.dark_v, L.dark_v, L.dark_v);
            const float4 f = L.flat ? __ldg(reinterpret_cast<const float4 *>(L.flat + at))
                                    : make_float4(L.flat_v, L.flat_v, L.flat_v, L.flat_v);
            dk[0] = d.x, dk[1] = d.y, dk[2] = d.z, dk[3] = d.w;
            fl[0] = f.x, fl[1] = f.y, fl[2] = f.z, fl[3] = f.w;
        } else {
            load_maps<4>(L, r, x0 + h, 1, dk, fl);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            v[h + e] = x0 + h + e < L.W ? pre_maps(L, x0 + h + e, v[h + e], dk[e], fl[e], rt) : 0.f;
    }
}

// Coefficient entries of columns c and c+1 of one row (c even, c < W) from
// the row's filtered values a and the next row's b at c, c+1, c+2 (0 at
// columns >= W).  The 16-bit formats store both entries with one 16-byte
// store: their rows hold an even number of entries (Wc), so entry c+1 exists
// and c starts a 16-byte unit; the FP32 format writes entry c+1 only below W.
template <int MODE>
__device__ __forceinline__ void emit_coef_pair(void *img, size_t row_base, int c, int W, const float *a,
                                               const float *b)
{
    const float dU0 = a[1] - a[0], dU1 = a[2] - a[1];
    const float Q0 = a[0], dV0 = b[0] - a[0], dUV0 = (b[1] - b[0]) - dU0;
    const float Q1 = a[1], dV1 = b[1] - a[1], dUV1 = (b[2] - b[1]) - dU1;
    if constexpr (MODE == TK_F32_COEF) {
        float4 *e = static_cast<float4 *>(img) + row_base + c;
        e[0] = make_float4(Q0, dU0, dV0, dUV0);
        if (c + 1 < W) e[1] = make_float4(Q1, dU1, dV1, dUV1);
    } else {
        uint4 e;
        if constexpr (MODE == TK_F16) {
            const __half2 l0 = __floats2half2_rn(Q0, dV0), h0 = __floats2half2_rn(dU0, dUV0);
            const __half2 l1 = __floats2half2_rn(Q1, dV1), h1 = __floats2half2_rn(dU1, dUV1);
            e = make_uint4(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&h0),
                           *reinterpret_cast<const uint32_t *>(&l1), *reinterpret_cast<const uint32_t *>(&h1));
        } else {
            const __nv_bfloat162 l0 = __floats2bfloat162_rn(Q0, dV0), h0 = __floats2bfloat162_rn(dU0, dUV0);
            const __nv_bfloat162 l1 = __floats2bfloat162_rn(Q1, dV1), h1 = __floats2bfloat162_rn(dU1, dUV1);
            e = make_uint4(*reinterpret_cast<const uint32_t *>(&l0), *reinterpret_cast<const uint32_t *>(&h0),
                           *reinterpret_cast<const uint32_t *>(&l1), *reinterpret_cast<const uint32_t *>(&h1));
        }
        *reinterpret_cast<uint4 *>(static_cast<uint2 *>(img) + row_base + c) = e;
    }
}

// One coefficient entry (see tk_precision) at entry offset `at`.
template <int MODE>
__device__ __forceinline__ void store_coef(void *img, size_t at, float Q, float dU, float dV, float dUV)
{
    if constexpr (MODE == TK_F32_COEF) {
        static_cast<float4 *>(img)[at] = make_float4(Q, dU, dV, dUV);
    } else if constexpr (MODE == TK_F16) {
        const __half2 l = __floats2half2_rn(Q, dV), h = __floats2half2_rn(dU, dUV);
        static_cast<uint2 *>(img)[at] =
            make_uint2(*reinterpret_cast<const uint32_t *>(&l), *reinterpret_cast<const uint32_t *>(&h));
    } else {
        const __nv_bfloat162 l = __floats2bfloat162_rn(Q, dV), h = __floats2bfloat162_rn(dU, dUV);
        static_cast<uint2 *>(img)[at] =
            make_uint2(*reinterpret_cast<const uint32_t *>(&l), *reinterpret_cast<const uint32_t *>(&h));
    }
}

// Derived load parameters: D^2, the scalar flat-field reciprocal, and the
// largest unit that rows can be read in (aligned base, row pitch a multiple of
// it, so every unit that starts below W lies inside its row).
inline void finish_load_params(LoadParams &L)
{
    L.D2 = L.D * L.D;
    L.inv_den = 1.f;
    if (L.input_type == TK_INPUT_U16 && !L.dark && !L.flat)
        L.inv_den = 1.f / std::fmax(L.flat_v - L.dark_v, L.floor_counts);
    const int es = L.input_type == TK_INPUT_U16 ? 2 : 4;
    L.gran = 0;
    for (int b = 16; b >= 4 && !L.gran; b /= 2)
        if (reinterpret_cast<uintptr_t>(L.in) % b == 0 && ((long long)L.in_pitch * es) % b == 0) L.gran = b;
    L.map_vec = L.W % 4 == 0 && reinterpret_cast<uintptr_t>(L.dark) % 16 == 0 &&
                reinterpret_cast<uintptr_t>(L.flat) % 16 == 0;
}

}  // namespace tk

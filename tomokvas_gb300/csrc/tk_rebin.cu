// tk_rebin.cu -- offset-detector (half-fan) sinogram completion and fan to
// parallel rebinning on the GPU: rsq::Half2FullFan and rsq::Half2Para /
// rsq::Fan2Para of Lukas-kV/TomoKvas (FBPG/rsq_load.cpp:327-487).
//
// A half-fan scan measures, per detector row, N angles x W columns with the
// rotation axis at column `axis_move`; the columns left of the axis are never
// measured.  Completion fills them from the conjugate rays; rebinning
// resamples the fan rays onto parallel ones.  One thread per output column.
// The angle shift of an output column depends on the column only: the host
// forms it in FP64 as the reference does (atan / asin of the column offset)
// and passes it per column as an integer angle step plus an FP32 fraction, so
// the kernels take the two neighbouring angles exactly and interpolate in
// FP32 (the samples are FP32).
#include "tk_common.cuh"
#include "tk_internal.h"

#include <algorithm>
#include <cmath>

namespace tk {

constexpr double kPiD = 3.14159265358979323846;

// Angle index modulo N, clamped into [0, N-1].
__device__ __forceinline__ int wrap_angle(int a, int N)
{
    if (a > N - 1) a -= N;
    if (a < 0) a += N;
    return min(max(a, 0), N - 1);
}

constexpr int kRebinMaxCols = 2048;  // output columns left of (fan) or around (parallel) the axis

// Per-column angle shifts: shift = k + frac with k an integer number of angle
// steps and frac in [0, 1) (FP32), formed on the host in FP64.
struct RebinShifts {
    short k[2][kRebinMaxCols];
    float frac[2][kRebinMaxCols];
};

// Both kernels: a thread owns one output column (its shifts, from the kernel
// parameters, are read once) and walks a chunk of angles of one
// detector row.  Neighbouring threads read neighbouring samples of the same
// one or two fan angles, and the lower angle of an output is the upper angle
// of the output before it, so a step costs one global load and one store;
// the loads of kRebinBatch angles are issued together.  Bound by HBM: 256 rows
// of 720 x 520 samples into 720 x 997 take 1930 us with one thread per output
// sample in flat order (64-bit divisions, a divergent parameter read and two
// loads per sample) and 213 us in this form (1.12 GB moved).
// Where a batch's angles neither wrap nor change conjugate (all but a few
// batches) its samples lie one row apart and need no index arithmetic, which
// otherwise bounds the kernel (ALU pipe 78 %, 61 instructions per sample).
constexpr int kRebinThreads = 128;
constexpr int kRebinBatch = 8;

// One such batch: upper samples at rows hi, hi + 1, ... of img, lower samples one row above them, the lower one's
// weight q (0: the upper sample alone).  `held` is the row whose sample `last` is.
__device__ __forceinline__ void rebin_rows(const float *__restrict__ img, int W, int hi, float q, int &held, float &last,
                                           float *&dst, long long ostep)
{
    const float *p = img + (long long)hi * W;
    float A[kRebinBatch];
#pragma unroll
    for (int j = 0; j < kRebinBatch; ++j) {
        A[j] = __ldg(p);
        p += W;
    }
    if (q != 0.f) {
        if (held != hi - 1) last = __ldg(img + (long long)(hi - 1) * W);
#pragma unroll
        for (int j = 0; j < kRebinBatch; ++j) {
            *dst = A[j] + (last - A[j]) * q;
            last = A[j];
            dst += ostep;
        }
    } else {
#pragma unroll
        for (int j = 0; j < kRebinBatch; ++j) {
            *dst = A[j];
            dst += ostep;
        }
        last = A[kRebinBatch - 1];
    }
    held = hi + kRebinBatch - 1;
}

// Half2FullFan (rsq_load.cpp:327-380): output row width Wc = 2W - 1 - 2am.
// Columns c >= W-1-am copy the measured half (from the axis column on);
// column c < W-1-am is the ray at detector offset t = c - (W-1-am) < 0, taken
// from the conjugate ray at offset -t and angle nf = f - (2 atan(t/D) + pi)/dfi,
// or f - (2 atan(t/D) - pi)/dfi when the first lies outside [0, N-1]; with the
// shift (2 atan(t/D) +- pi)/dfi = k + frac, nf = (f - k) - frac, so the
// two angles are f - k - 1 and f - k (one angle when frac = 0) and the weight
// of the lower is frac.  `flip` stores the angles in reverse order.
__global__ void __launch_bounds__(kRebinThreads)
    half2fullfan_kernel(const float *__restrict__ in, float *__restrict__ out, int W, int N, int rows, int am, int flip,
                        int chunk, const __grid_constant__ RebinShifts S)
{
    const int Wc = 2 * W - 1 - 2 * am;
    const int c0 = W - 1 - am;  // output column of the axis
    const int c = blockIdx.x * kRebinThreads + threadIdx.x;
    if (c >= Wc) return;
    const bool copy = c >= c0;
    const int k0 = copy ? 0 : S.k[0][c], k1 = copy ? 0 : S.k[1][c];
    const float fr0 = copy ? 0.f : S.frac[0][c], fr1 = copy ? 0.f : S.frac[1][c];
    const int col = copy ? c - c0 + am : c0 - c + am;  // -t + am
    const int f0 = blockIdx.y * chunk, f1 = min(f0 + chunk, N);
    const long long ostep = flip ? -(long long)Wc : Wc;
    for (int r = blockIdx.z; r < rows; r += gridDim.z) {
        const float *img = in + (long long)r * N * W + col;
        float *dst = out + ((long long)r * N + (flip ? N - 1 - f0 : f0)) * Wc + c;
        int held = -1;  // the angle whose sample `last` is
        float last = 0.f;
        for (int f = f0; f < f1; f += kRebinBatch) {
            {  // whole batch copied, or from the first, or from the other conjugate, inside [1, N - 1]
                const int a = f - k0, b = f - k1, n1 = N - kRebinBatch;
                const bool first = a >= 1 && a <= n1, other = (a + kRebinBatch <= 0 || a > N) && b >= 1 && b <= n1;
                if (f + kRebinBatch <= f1 && (copy || first || other)) {
                    rebin_rows(img, W, copy ? f : first ? a : b, copy ? 0.f : first ? fr0 : fr1, held, last, dst, ostep);
                    continue;
                }
            }
            int hi[kRebinBatch], lo[kRebinBatch];
            float fr[kRebinBatch], A[kRebinBatch];
#pragma unroll
            for (int j = 0; j < kRebinBatch; ++j) {
                // nf = (f - k) - frac; outside [0, N-1] the other conjugate (shift - 2 pi / dfi)
                int fk = f + j - k0;
                fr[j] = fr0;
                // nf < 0 or nf > N - 1, decided on the integer part (nf = fk - fr, fr in [0, 1))
                const bool below = fr0 > 0.f ? fk <= 0 : fk < 0;
                const bool above = fr0 > 0.f ? fk >= N : fk > N - 1;
                if (!copy && (below || above)) {
                    fk = f + j - k1;
                    fr[j] = fr1;
                }
                // the angle past the last one wraps to the first (rsq_load.cpp:361-366); indices are
                // also wrapped and clamped for angle steps not exactly 2 pi / N
                hi[j] = wrap_angle(fk, N);      // ceil(nf)
                lo[j] = wrap_angle(fk - 1, N);  // floor(nf)
                if (f + j < f1) A[j] = __ldg(img + (long long)hi[j] * W);
            }
#pragma unroll
            for (int j = 0; j < kRebinBatch; ++j) {
                if (f + j >= f1) break;
                float v = A[j];
                if (fr[j] != 0.f) {
                    const float B = lo[j] == held ? last : __ldg(img + (long long)lo[j] * W);
                    v = A[j] + (B - A[j]) * fr[j];  // (a - nf) = frac
                }
                last = A[j];
                held = hi[j];
                *dst = v;
                dst += ostep;
            }
        }
    }
}

// Half2Para + Fan2Para (rsq_load.cpp:382-470): N/2 parallel angles x Wc
// columns.  Parallel column u at offset s = u - (W-1-am) samples the fan ray
// through detector column |s| + am at fan angle beta = f + asin(s/D)/dfi
// (s >= 0) or f - (asin(s/D) - pi)/dfi (s < 0), wrapped into [0, N), linearly
// interpolated between the two neighbouring fan angles.  With the shift =
// k + frac, beta = (f + k) + frac: the angles are f + k and f + k + 1 (one
// when frac = 0), the weight of the upper is frac.  As in the reference, both
// column taps use the ceiling index, so the column is never interpolated (the
// offsets are integers).
__global__ void __launch_bounds__(kRebinThreads)
    half2para_kernel(const float *__restrict__ in, float *__restrict__ out, int W, int N, int rows, int am, int chunk,
                     const __grid_constant__ RebinShifts S)
{
    const int Wc = 2 * W - 1 - 2 * am, Np = N / 2;
    const int u = blockIdx.x * kRebinThreads + threadIdx.x;
    if (u >= Wc) return;
    const int ui = u - (W - 1 - am);
    const int k = S.k[0][u];
    const float fr = S.frac[0][u];
    const int col = min(max((ui < 0 ? -ui : ui) + am, 0), W - 1);
    const int f0 = blockIdx.y * chunk, f1 = min(f0 + chunk, Np);
    for (int r = blockIdx.z; r < rows; r += gridDim.z) {
        const float *img = in + (long long)r * N * W + col;
        float *dst = out + ((long long)r * Np + f0) * Wc + u;
        int held = -1;  // the angle whose sample `last` is
        float last = 0.f;
        for (int f = f0; f < f1; f += kRebinBatch) {
            {
                int fb = f + k;
                if (fb < 0) fb += N;
                if (fr > 0.f ? fb >= N - 1 : fb > N - 1) fb -= N;
                if (f + kRebinBatch <= f1 && fb >= 0 && fb + kRebinBatch <= N - 1) {
                    rebin_rows(img, W, fr != 0.f ? fb + 1 : fb, fr != 0.f ? 1.f - fr : 0.f, held, last, dst, Wc);
                    continue;
                }
            }
            int up[kRebinBatch], dn[kRebinBatch];
            float A[kRebinBatch];
#pragma unroll
            for (int j = 0; j < kRebinBatch; ++j) {
                int fb = f + j + k;
                // beta = fb + fr, fr in [0, 1): beta < 0 iff fb < 0; beta > N - 1 decided on the integer part
                if (fb < 0) fb += N;
                if (fr > 0.f ? fb >= N - 1 : fb > N - 1) fb -= N;
                dn[j] = wrap_angle(fb, N);                              // floor(beta)
                up[j] = fr != 0.f ? wrap_angle(fb + 1, N) : dn[j];  // ceil(beta)
                if (f + j < f1) A[j] = __ldg(img + (long long)up[j] * W);
            }
#pragma unroll
            for (int j = 0; j < kRebinBatch; ++j) {
                if (f + j >= f1) break;
                float v = A[j];
                if (fr != 0.f) {
                    const float vb = dn[j] == held ? last : __ldg(img + (long long)dn[j] * W);
                    v = A[j] + (vb - A[j]) * (1.f - fr);  // (ba - beta) = 1 - frac
                }
                last = A[j];
                held = up[j];
                *dst = v;
                dst += Wc;
            }
        }
    }
}

// shift = k + frac, k = floor(shift), frac in [0, 1)
static void split_shift(double shift, short &k, float &frac)
{
    const double fl = std::floor(shift);
    k = (short)fl;
    frac = (float)(shift - fl);
    if (frac >= 1.f) {  // rounding to FP32 reached the next step
        k = (short)(k + 1);
        frac = 0.f;
    }
}

static int rebin_check(const float *d_in, float *d_out, int W, int N, int rows, int am, double D, double dfi)
{
    TK_CHECK(d_in && d_out, TK_ERR_INVALID, "rebin: null device pointer");
    TK_CHECK(W > 1 && N > 1 && rows > 0, TK_ERR_INVALID, "rebin: bad sizes %d x %d x %d", W, N, rows);
    TK_CHECK(am >= 0 && am < W - 1, TK_ERR_INVALID, "rebin: axis_move %d outside [0, W-1)", am);
    TK_CHECK(std::isfinite(D) && D > W && std::isfinite(dfi) && dfi > 0, TK_ERR_INVALID,
             "rebin: need D > W (pixels) and dfi > 0");
    TK_CHECK(std::fabs(dfi * N - 2 * kPiD) < 1e-3, TK_ERR_UNSUPPORTED, "rebin: needs a full 360-degree scan");
    TK_CHECK(N <= 16384 && 2 * W - 1 - 2 * am <= kRebinMaxCols, TK_ERR_UNSUPPORTED,
             "rebin: at most 16384 angles and %d output columns", kRebinMaxCols);
    return TK_OK;
}

// Column blocks x angle chunks x rows.  Chunks of 64 angles (one extra load each); shorter ones,
// down to one batch, where that would leave fewer than 16 blocks per SM.
static dim3 rebin_grid(int Wc, int angles, int rows, int *chunk)
{
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int bx = (Wc + kRebinThreads - 1) / kRebinThreads, bz = std::min(rows, 65535);
    int c = 64;
    while (c > kRebinBatch && (long long)bx * ((angles + c - 1) / c) * bz < 16ll * sms) c /= 2;
    *chunk = c;
    return dim3((unsigned)bx, (unsigned)((angles + c - 1) / c), (unsigned)bz);
}

}  // namespace tk

using namespace tk;

extern "C" int tk_half_to_full_fan(const float *d_in, int W, int N, int rows, int axis_move, double D, double dfi,
                                   int flip, float *d_out, void *stream)
{
    if (int rc = rebin_check(d_in, d_out, W, N, rows, axis_move, D, dfi)) return rc;
    static thread_local RebinShifts S;
    const int c0 = W - 1 - axis_move;
    for (int c = 0; c < c0; ++c) {  // rsq_load.cpp:329-333, 352-355
        const double at = std::atan((double)(c - c0) / D);
        split_shift((2 * at + kPiD) / dfi, S.k[0][c], S.frac[0][c]);
        split_shift((2 * at - kPiD) / dfi, S.k[1][c], S.frac[1][c]);
    }
    int chunk = 0;
    const dim3 grid = rebin_grid(2 * W - 1 - 2 * axis_move, N, rows, &chunk);
    half2fullfan_kernel<<<grid, kRebinThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        d_in, d_out, W, N, rows, axis_move, flip ? 1 : 0, chunk, S);
    count_launch();
    TK_CUDA(cudaGetLastError());
    return TK_OK;
}

extern "C" int tk_half_to_parallel(const float *d_in, int W, int N, int rows, int axis_move, double D, double dfi,
                                   float *d_out, void *stream)
{
    if (int rc = rebin_check(d_in, d_out, W, N, rows, axis_move, D, dfi)) return rc;
    TK_CHECK(N % 2 == 0, TK_ERR_INVALID, "rebin: parallel rebinning needs an even number of angles");
    static thread_local RebinShifts S;
    const int Wc = 2 * W - 1 - 2 * axis_move;
    for (int u = 0; u < Wc; ++u) {  // rsq_load.cpp:409-413
        const double ui = (double)u - (double)(W - 1 - axis_move);
        const double g = ui >= 0. ? std::asin(ui / D) / dfi : -(std::asin(ui / D) - kPiD) / dfi;
        split_shift(g, S.k[0][u], S.frac[0][u]);
    }
    int chunk = 0;
    const dim3 grid = rebin_grid(Wc, N / 2, rows, &chunk);
    half2para_kernel<<<grid, kRebinThreads, 0, static_cast<cudaStream_t>(stream)>>>(d_in, d_out, W, N, rows, axis_move,
                                                                                    chunk, S);
    count_launch();
    TK_CUDA(cudaGetLastError());
    return TK_OK;
}

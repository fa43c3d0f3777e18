// tk_fp_plan.h -- which form a forward projection takes: the shape of the row lanes (fp_rows_kernel in tk_bp.cu) and
// their estimated time beside that of the slice lanes (fp_scatter_col_kernel).  Plain C++, so that the rule can be checked
// on a host.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>

#include "tk_fdk.h"

namespace tk {

constexpr int kFpTX = 16, kFpTY = 8, kFpCols = kFpTX * kFpTY, kFpHalf = kFpCols / 2, kFpWarps = 8, kFpMaxRows = 64;

// Shape of a row-lane forward projection (fp_rows_kernel), or K = 0 where it does not apply: the source
// inside the field of view (U has no bound there), row steps below 1/2 (more than four slices per row), or
// footprints too large for two CTAs per SM.
struct FpRowsPlan {
    int K = 0, TZ = 0, GP = 0, zchunks = 0, BW = 0, BH = 0, stage_elems = 0;
    size_t smem = 0;
};

// The box of a 16 x 8 x TZ tile measured from the smallest row and column that its columns inside the field of
// view reach: columns 0 .. floor(du) + 1 (plus the second tap, plus 3 for the TMA alignment of the origin),
// rows 0 .. floor(dv) + 2, with du, dv bounded as in bp_box_dims for radii up to W/2.
inline FpRowsPlan fp_rows_plan(const tk_geometry &g, int nz, float zoff)
{
    FpRowsPlan p;
    const double s = std::fabs((double)g.scale), D = g.D;
    const double ex = s * std::fmax(std::fabs((double)g.cx), std::fabs((double)(g.X - 1) - g.cx));
    const double ey = s * std::fmax(std::fabs((double)g.cy), std::fabs((double)(g.Y - 1) - g.cy));
    const double R = std::fmin(0.5 * g.W, std::sqrt(ex * ex + ey * ey) + 1.0);
    if (!(D - R > 1e-3 * D)) return p;
    const double dv_min = s * D / (D + R);
    const int K = dv_min >= 1.0001 ? 2 : dv_min >= 2.0001 / 3.0 ? 3 : dv_min >= 0.50005 ? 4 : 0;
    if (!K) return p;
    const double Umax = D / (D - R), dU = D / ((D - R) * (D - R));
    const double dxy = s * std::sqrt((double)((kFpTX - 1) * (kFpTX - 1) + (kFpTY - 1) * (kFpTY - 1)));
    const double azmax = s * std::fmax(std::fabs((double)zoff), std::fabs((double)(nz - 1) + zoff));
    const int BW = (((int)std::floor(dxy * Umax + R * dU * dxy + 0.01) + 6 + 3) / 4 | 1) * 4;  // BW / 4 odd
    if (BW > 256) return p;
    auto shape = [&](int TZ) {
        p.TZ = TZ;
        p.GP = (TZ + (K == 2 ? 3 : 2 * K)) | 1;
        p.BW = BW;
        p.BH = (int)std::floor(s * (TZ - 1) * Umax + azmax * dU * dxy + 0.01) + 3;
        p.stage_elems = BW * kFpMaxRows;  // per warp a box, and 32 bytes for each of half the columns
        p.smem = kFpWarps * ((size_t)p.stage_elems * 4 + 2 * kFpHalf * 16) + (size_t)kFpCols * p.GP * 4;
        return p.BH <= kFpMaxRows && p.smem <= 112 * 1024;  // two CTAs per SM
    };
    int TZ = std::min(nz, kFpMaxRows);
    while (TZ >= 1 && !shape(TZ)) --TZ;
    if (TZ < std::min(nz, 8) || (nz + TZ - 1) / TZ > 65535) return p;  // (a grid's y)
    p.zchunks = (nz + TZ - 1) / TZ;
    shape((nz + p.zchunks - 1) / p.zchunks);  // even chunks
    p.K = K;
    return p;
}

// CTAs that share a tile's projections (at least 4 per warp): small volumes, until the chip has about four waves of CTAs.
inline int fp_rows_split(long long ctas, int N, int sms)
{
    return (int)std::max(1ll, std::min<long long>((8ll * sms + ctas - 1) / ctas, N / (4 * kFpWarps)));
}

// Whether the row lanes are the faster form for a volume of nz slices and N projections; the slice lanes' box has
// slice_cells cells, and two of their CTAs fit an SM or one.  A row-lane CTA works through 64 rows per column and
// projection however few slices its chunk has, so its time follows the chunks, not the voxels: footprints that leave
// little shared memory for voxels cut the chunks short.  Its warps take whole projections, so few projections leave warps
// idle.  Estimates in us from CTAs per SM: row lanes 1.12, 1.35 and 1.6 per CTA and projection for K = 2, 3, 4; slice
// lanes 2.2 and 0.2 per 1000 cells per CTA and projection (a quarter more with one CTA per SM), whole rounds of CTAs, and
// the loading of a tile as 1.6 projections; each has a floor where the GPU is not full.  Of 402 geometries (48^3 to
// 700 x 600 x 100, scales 0.5 to 2.5, D = 2 W to 8 W, 1 to 300 projections) two take the form that is slower by more than
// 1 % (by 5 and 6 %).  512^3 into 60 projections, slice lanes / row lanes (slices per chunk): scale 1.5, D = 5.2 W 16.3 /
// 12.7 ms (36), D = 4 W 17.1 / 36.1 (12); scale 1.35, D = 3 W 17.4 / 35.6 (12); scale 2, D = 8 W 20.0 / 37.3 (12).
inline bool fp_rows_faster(const FpRowsPlan &p, int X, int Y, int nz, int N, int slice_cells, bool two_slice_ctas,
                           int sms)
{
    const auto up = [](int n, int d) { return (long long)(n + d - 1) / d; };
    const long long ctas = up(X, kFpTX) * up(Y, kFpTY) * p.zchunks;
    const int warps = kFpWarps * fp_rows_split(ctas, N, sms);  // that share a tile's projections
    const double row_cta = p.K == 2 ? 1.12 : p.K == 3 ? 1.35 : 1.6;
    const double rows = std::max(row_cta * ctas / sms * warps * up(N, warps), 14.0) + 0.4 * N;
    const double x = (double)(up(X, 16) * up(Y, 16) * up(nz, 32)) / sms;
    const double slice_cta = (2.2 + 2e-4 * slice_cells) * (two_slice_ctas ? 1.0 : 1.25);
    return rows <= std::max(x <= 1.0 ? 5.0 : 6.4, slice_cta * std::ceil(x)) * (N + 1.6);
}

}  // namespace tk

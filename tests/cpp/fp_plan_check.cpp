// The forward projector's choice of form (csrc/tk_fp_plan.h): one line per geometry given as
// W H N X Y Z D scale cells two (the slice lanes' box and whether two of their CTAs fit an SM), K TZ zchunks faster.
#include <cstdio>

#include "tk_fp_plan.h"

int main()
{
    int W, H, N, X, Y, Z, cells, two;
    double D, scale;
    while (std::scanf("%d %d %d %d %d %d %lf %lf %d %d", &W, &H, &N, &X, &Y, &Z, &D, &scale, &cells, &two) == 10) {
        tk_geometry g{};
        g.W = W, g.H = H, g.N = N, g.X = X, g.Y = Y, g.Z = Z;
        g.cX = 0.5f * (W - 1), g.cZ = 0.5f * (H - 1), g.cx = 0.5f * (X - 1), g.cy = 0.5f * (Y - 1);
        g.D = (float)D, g.scale = (float)scale, g.dfi = 6.2831853f / N, g.tau = 0.02f;
        const tk::FpRowsPlan p = tk::fp_rows_plan(g, Z, -0.5f * (Z - 1));
        std::printf("%d %d %d %d\n", p.K, p.TZ, p.zchunks, p.K && tk::fp_rows_faster(p, X, Y, Z, N, cells, two != 0, 152));
    }
    return 0;
}

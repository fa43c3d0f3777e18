// tk_fft_shape.h -- shape of the FFT filter's transforms (tk_filter.cu): passes, threads, twiddle tables and shared
// memory of a length-2^LG row filter.  Plain C++, so that the index rules can be checked on a host.
#pragma once

#include <cstddef>

namespace tk {

constexpr int kFiltThreads = 256;  // of a CTA, and the most of a transform

// Threads per transform: one radix-16 butterfly each (a single butterfly serves p <= 16, whose outputs p/2 threads
// write), at most a CTA.  Transforms of p <= 256 share warps: on a warp each, most of its lanes would own nothing.  20000
// FP32 rows into FP32 samples, W = 64 / 128: 20.6 / 26.8 us with the passes apart, 28.8 / 32.8 with joined passes on a
// warp, 14.4 / 18.5 so.
constexpr int fft_threads_c(int p)
{
    return p <= 16 ? p / 2 : (p >> 4) < kFiltThreads ? (p >> 4) : kFiltThreads;
}

// Shape of the length-2^LG filter.
template <int LG> struct Fft {
    static constexpr int P = 1 << LG, NP = (LG + 3) / 4;              // passes of one transform
    static constexpr int RL = LG % 4 ? 1 << (LG % 4) : 16;            // radix of the last forward pass
    static constexpr int R1 = NP > 1 ? 16 : RL, Q1 = P / R1;          // first pass: radix and butterflies
    // Threads of a transform, of a CTA and transforms of a CTA.  Small CTAs where transforms share warps: short inputs
    // still reach every SM.
    static constexpr int TPF = fft_threads_c(P), NT = TPF < 32 ? 64 : kFiltThreads, G = NT / TPF;
    static constexpr int MINB = NT == 64 ? 8 : 0;  // CTAs per SM that registers must leave room for (0: not stated)
    static constexpr int IN = R1 / 2, ITIN = (Q1 + TPF - 1) / TPF;    // samples j + r Q1, r < IN, per butterfly
    // output columns j + s QC, s < NC, of butterfly j of the last pass
    static constexpr int NC = NP > 1 ? 8 : 1, QC = NP > 1 ? P / 16 : P / 2, ITC = (QC + TPF - 1) / TPF;
    // twiddle tables: forward passes m >= 1 (span 16^m), then the inverse's radix-16 passes (span RL 16^m).
    // RL = 16: the same tables.  LG = 13: the last forward table, w^k for k < p/2, serves the inverse.
    static constexpr int fwd_off(int m) { return m >= 1 ? (1 << (4 * m)) - 16 : 0; }
    static constexpr int FWD = NP > 1 ? fwd_off(NP - 1) + (P / RL) * (RL - 1) : 0;
    static constexpr bool OWN_INV = RL != 16 && LG < 13 && NP > 1;
    static constexpr int inv_span(int m) { return RL << (4 * m); }    // m = 0 .. NP - 2
    static constexpr int inv_off(int m)
    {
        int o = OWN_INV ? FWD : 0;
        for (int i = 0; i < m; ++i) o += inv_span(i) * 15;
        return o;
    }
    static constexpr int TW = OWN_INV ? inv_off(NP - 1) : FWD;        // entries of all tables
    static constexpr int HF = ((P / 2 + 1) + 3) & ~3;                 // spectrum, floats
    static constexpr int EDGE = (TPF + 31) / 32 * (NC + 1);           // first columns of each warp, float2
    // Where thread t of a group finds the column after its column t + s QC: entry next_edge(t) + s of the edge array
    // (the first columns 32 w + s QC of the group's w-th 32 threads are entries w (NC + 1) + s), or -1: in the next lane,
    // or t has no column.
    static constexpr int next_edge(int t)
    {
        return t == QC - 1 ? 1 : t < QC && t % 32 == 31 ? (t / 32 + 1) * (NC + 1) : -1;
    }
    // Transform buffers and edge of a group, in float2; groups that share a warp start TPF banks of 8 bytes apart.
    static constexpr int USED = 2 * (P + P / 16) + EDGE;
    static constexpr int STRIDE = TPF >= 16 ? USED : USED + (16 + TPF - USED % 16) % 16;
    static constexpr size_t group_bytes() { return (size_t)STRIDE * 8; }
    static constexpr size_t smem() { return (size_t)TW * 8 + HF * 4 + G * group_bytes(); }
};

}  // namespace tk

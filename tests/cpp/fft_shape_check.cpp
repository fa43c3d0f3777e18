// Index rules of the FFT filter's coefficient form, by enumeration: for every transform length and every row width
// that takes it, each edge entry that a thread reads lies in its group's array, was written there, and holds the column
// after the thread's own; every other column that is stored finds the next one in the next lane.
#include <cstdio>
#include <vector>

#include "tk_fft_shape.h"

template <int LG> static int check()
{
    using F = tk::Fft<LG>;
    // entry e of the edge array: the column it holds, -1 where no thread writes it
    std::vector<int> holds(F::EDGE, -1);
    for (int t = 0; t < F::TPF; t += 32)
        for (int s = 0; s < F::NC; ++s) holds[t / 32 * (F::NC + 1) + s] = t < F::QC ? t + s * F::QC : -1;
    int bad = 0;
    for (int W = F::P / 4 + 1; W <= F::P / 2; ++W)
        for (int t = 0; t < F::TPF; ++t)
            for (int s = 0; s < F::NC; ++s) {
                const int c = t + s * F::QC, next = F::next_edge(t);
                if (next >= 0 && c + 1 < W) {  // the kernel's read
                    const int e = next + s;
                    if (e >= F::EDGE || holds[e] != c + 1) ++bad;
                } else if (next < 0 && t < F::QC && c + 1 < W) {  // the next lane's column
                    if (t % 32 == 31 || t + 1 >= F::QC) ++bad;
                }
            }
    if (bad) std::printf("p = %d: %d wrong reads\n", F::P, bad);
    return bad;
}

int main()
{
    const int bad = check<2>() + check<3>() + check<4>() + check<5>() + check<6>() + check<7>() + check<8>() +
                    check<9>() + check<10>() + check<11>() + check<12>();
    return bad ? 1 : 0;
}

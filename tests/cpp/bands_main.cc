// Host check of the small-level kernel's row bands (mg_window.cuh, mg_plan.h):
// for every grid height, cut of the levels and cluster size that layout_small
// accepts, the bands of each level follow one another from row 0 to its end,
// and a band's rows are where its arrays have room for them.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "mg_plan.h"

using namespace stzg;
using namespace stzg::mgw;

template <typename S> static long check(int m, int n, int yp) {
    int M[kMaxLevels], N[kMaxLevels], nl = 1;
    M[0] = m;
    N[0] = n;
    while ((long)M[nl - 1] * N[nl - 1] > 10 && M[nl - 1] > 4 && nl < kMaxLevels) {
        if (yp && (N[nl - 1] & 1)) break;
        M[nl] = (M[nl - 1] + 1) >> 1;
        N[nl] = yp ? N[nl - 1] >> 1 : (N[nl - 1] + 2) >> 1;
        nl++;
    }
    long bad = 0;
    for (int d = 1; d < nl; d++)
        for (int t = 0; t < d; t++)
            for (int c = 1; c <= 16; c <<= 1) {
                small_plan<S> P;
                std::memset(&P, 0, sizeof(P));
                for (int l = t; l <= d; l++) {
                    P.lv[l].m = M[l];
                    P.lv[l].n = N[l];
                    P.lv[l].homog = 1;
                    P.lv[l].nst = 5;
                    P.lv[l].ncls = N[l];
                }
                P.top = t == 0 && !yp;
                if (!layout_small(P, t, d, c, 227 * 1024)) continue;
                for (int l = t; l <= d; l++)
                    for (int k = 0; k < c; k++) {
                        const int y0 = band_row(P, l, k), y1 = band_row(P, l, k + 1);
                        if (y0 < 0 || y1 < y0 || y1 > N[l] || (k == 0 && y0) || (k + 1 == c && y1 != N[l])) bad++;
                        if (l < d && (long)(y1 - y0 + band_below(P, l) + band_above(P, l)) * M[l] > P.lv[l].ps) bad++;
                    }
            }
    return bad;
}

int main() {
    long bad = 0;
    for (int n = 5; n <= 700; n++)
        for (int m : {8, 24, 46, 90}) bad += check<ff>(m, n, 0) + check<float>(m, n, 0) + check<ff>(m, n, 1);
    std::printf("%ld bands out of place\n", bad);
    return bad ? 1 : 0;
}

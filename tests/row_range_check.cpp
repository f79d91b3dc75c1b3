// Check of the gridding rows' pixel ranges (bsoft_b200/csrc/row_range.h): for
// views at random and a hair off an axis, the range that the FP32 bounds call
// sure is the one of the FP64 bounds.  Prints the numbers of rows, of sure rows
// and of wrong ones.
#include "../bsoft_b200/csrc/row_range.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>

int main(int argc, char** argv) {
    const long rows = argc > 1 ? atol(argv[1]) : 1000000;
    std::mt19937_64 rng(3);
    std::uniform_real_distribution<double> u(-1, 1);
    const double tiny[] = {5e-9, 1e-10, 2e-12, 1e-6};
    const int T = 8, hf = 256;
    long sure = 0, wrong = 0, empty = 0;
    for (long i = 0; i < rows; ++i) {
        // steps along h of the three axes, the row's coordinate at pixel hc
        double ad[3], b[3];
        for (int k = 0; k < 3; ++k) {
            ad[k] = 0.5 * u(rng);
            if (rng() % 2) ad[k] = tiny[rng() % 4] * (rng() % 2 ? 1 : -1);
            b[k] = 3.5 + 9 * u(rng);
        }
        const int hc = (int)(200 * u(rng)), h_lo = hc - 1 - (int)(rng() % 40), h_hi = hc + 1 + (int)(rng() % 40);
        // FP64: pixels whose tents reach the tile along every axis
        double lo = std::max(h_lo, -hf) - hc, hi = std::min(h_hi, hf - 1) - hc;
        float la = -1e9f, lb = -1e9f, ha = 1e9f, hb = 1e9f;
        for (int k = 0; k < 3; ++k) {
            double p = (-1.0 - b[k]) / ad[k], q = (T - b[k]) / ad[k];
            if (p > q) std::swap(p, q);
            lo = std::max(lo, p);
            hi = std::min(hi, q);
            // setup_pair's and walk_groups' FP32 forms
            const float ia = (float)(1.0 / ad[k]), err = 5e-5f * fabsf(ia) + 1e-5f;
            const float p0 = -1.0f * ia, p1 = (float)T * ia, s = -(float)b[k] * ia;
            la = fmaxf(la, s + (fminf(p0, p1) - err));
            lb = fmaxf(lb, s + (fminf(p0, p1) + err));
            ha = fminf(ha, s + (fmaxf(p0, p1) - err));
            hb = fminf(hb, s + (fmaxf(p0, p1) + err));
        }
        const bool some = lo <= hi;
        const long l = some ? hc + (long)ceil(lo) : 0, h = some ? hc + (long)floor(hi) : -1;
        const bsg::RowRange r = bsg::row_range(hc, std::max(h_lo, -hf), std::min(h_hi, hf - 1), la, lb, ha, hb);
        if (!r.sure) continue;
        ++sure;
        const bool none = h < l;
        empty += none;
        if (none ? r.lo <= r.hi : (r.lo != l || r.hi != h)) ++wrong;
    }
    printf("rows %ld sure %ld empty %ld wrong %ld\n", rows, sure, empty, wrong);
    return wrong != 0;
}

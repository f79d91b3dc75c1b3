// Check of the order in which lattice.cu tries the phase lattices
// (bsoft_b200/csrc/lattice.h): the candidates are choose_lattice's loops in
// their order, and the first safe one of the first 32 that hold any is
// choose_lattice's, for random views, steps and curvatures.  Prints the numbers
// of candidates out of order, of views and of differing choices.
#include "../bsoft_b200/csrc/lattice.h"

#include <cstdio>
#include <cstdlib>
#include <random>

using namespace bsg;

static bool same(const PhaseLattice& a, const PhaseLattice& b) { return a.lh == b.lh && a.lk == b.lk && a.sh == b.sh; }

int main(int argc, char** argv) {
    const int views = argc > 1 ? atoi(argv[1]) : 1000;
    int c = 0, order = 0;
    for (int d = 1; d <= LATTICE_PHASES; ++d)
        for (int lk = 1; lk <= d; ++lk)
            for (int sh = 0; d % lk == 0 && sh < d / lk; ++sh, ++c)
                order += !same(lattice_candidate(c), {d / lk, lk, sh});
    order += c != LATTICE_CANDIDATES;
    order += lattice_candidate(c).lh != 0;

    std::mt19937_64 rng(5);
    std::normal_distribution<double> nd;
    const double steps[] = {0.5, 0.4, 0.25, 0.7, 1.0, 0.1, 0.02}, curves[] = {0.0, 0.0, 0.01, 0.1, 0.6};
    int differ = 0, n = 0;
    for (double step : steps)
        for (double curve : curves)
            for (int v = 0; v < views; ++v, ++n) {
                double a[3], b[3], aa = 0, ab = 0, bb = 0;
                for (int i = 0; i < 3; ++i) { a[i] = nd(rng); aa += a[i] * a[i]; }
                if (v == 0) { a[0] = aa = 1; a[1] = a[2] = 0; }
                for (int i = 0; i < 3; ++i) a[i] /= sqrt(aa);
                for (int i = 0; i < 3; ++i) { b[i] = v ? nd(rng) : i == 1; ab += a[i] * b[i]; }
                for (int i = 0; i < 3; ++i) { b[i] -= ab * a[i]; bb += b[i] * b[i]; }
                double ad[3], bd[3];
                for (int i = 0; i < 3; ++i) { ad[i] = step * a[i]; bd[i] = step * b[i] / sqrt(bb); }
                const double reach = lattice_reach(ad, bd, curve * step);
                PhaseLattice best = square_lattice(reach);
                bool found = false;
                for (int c0 = 0; reach < 64.0 && c0 < LATTICE_CANDIDATES && !found; c0 += 32)
                    for (int lane = 0; lane < 32 && !found; ++lane) {
                        const PhaseLattice l = lattice_candidate(c0 + lane);
                        if (l.lh > 0 && lattice_ok(ad, bd, l.lh, l.lk, l.sh, reach, curve * step)) { best = l; found = true; }
                    }
                differ += !same(best, choose_lattice(ad, bd, LATTICE_PHASES, curve * step));
            }
    printf("out_of_order %d views %d differ %d\n", order, n, differ);
    return order != 0 || differ != 0;
}

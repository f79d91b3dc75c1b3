// lattice.h - the phase lattice of the gridding scatter, chosen per particle, on
// the device (lattice.cu) or, for a few, on the host; plain C++ there.
//
// The gridding kernel walks a particle's pixels phase by phase: the pixels
// (h0 + lh i + sh j, k0 + lk j) of one phase are gridded by the 32 lanes of
// a warp at once, each lane adding to the corners of its pixel's unit cell
// of the map with a plain shared-memory read-modify-write.  That is only
// correct if two pixels of one phase never fall in the same cell.  Two
// pixels whose pixel-step difference is (dh, dk) sit d = dh ad + dk bd apart
// in the map (ad, bd: the map displacement of one pixel step along h and k);
// they can share a cell only if |d_x|, |d_y| and |d_z| are all below 1.  So
// a lattice is safe when every nonzero lattice vector has max_c |d_c| >= 1
// (with a margin above the rounding of the per-pixel coordinates: the
// kernel forms them in FP32 relative to its tile, < 5e-6 voxel).
//
// A lattice safe for every orientation needs vectors of length >= sqrt(3)
// voxels (12 phases at half-voxel pixel steps); for one orientation the
// smallest safe lattice usually has 4 to 6 phases (the cube's section by the
// particle's plane has area 4 to 3 sqrt(3) voxels^2, and a lattice with no
// point inside a symmetric convex region needs at least a quarter of its
// area per point).  Fewer phases means fewer per-phase scans and fuller warps.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define BSG_LATTICE_FN __host__ __device__ inline
#else
#define BSG_LATTICE_FN inline
#endif

namespace bsg {

struct PhaseLattice {
    int lh, lk, sh;
};

// Products and sums rounded one by one: the device would contract them, and a
// vector within rounding of the margin would then get another lattice (and a
// particle another order of its sums) than the host's.
BSG_LATTICE_FN double lat_mul(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
BSG_LATTICE_FN double lat_add(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}

// Length (in pixel steps) beyond which a pixel-step vector cannot fail:
// sqrt(3) / (smallest singular value of [ad bd]), since max_c |d_c| >=
// |d| / sqrt(3).  Infinite when ad, bd are degenerate.
BSG_LATTICE_FN double lattice_reach(const double ad[3], const double bd[3], double curve = 0.0) {
    double aa = 0, ab = 0, bb = 0;
    for (int c = 0; c < 3; ++c) {
        aa = lat_add(aa, lat_mul(ad[c], ad[c]));
        ab = lat_add(ab, lat_mul(ad[c], bd[c]));
        bb = lat_add(bb, lat_mul(bd[c], bd[c]));
    }
    const double tr = aa + bb, det = lat_add(lat_mul(aa, bb), -lat_mul(ab, ab));
    const double d2 = lat_add(lat_mul(tr, tr), -lat_mul(4.0, det));
    const double disc = sqrt(d2 > 0.0 ? d2 : 0.0);
    const double smin2 = lat_mul(0.5, tr - disc);
    if (!(smin2 > 0)) return HUGE_VAL;
    // a curved surface (Ewald sphere) moves two points |v| pixel steps apart
    // by at most curve |v| voxels more: |d| >= |v| (sigma_min - curve)
    const double smin = sqrt(smin2) - curve;
    if (!(smin > 0)) return HUGE_VAL;
    return lat_add(lat_mul(1.7320508075688772 / smin, 1.0 + 1e-9), 1e-9);
}

// True when no nonzero vector of the lattice {(lh i + sh j, lk j)} maps to a
// displacement with all three |d_c| < 1 + margin.  Only vectors shorter than
// `reach` pixel steps need checking, and of each pair +-v only one.
BSG_LATTICE_FN bool lattice_ok(const double ad[3], const double bd[3], int lh, int lk, int sh, double reach,
                               double curve = 0.0) {
    const double margin = 2e-5, r2 = lat_mul(reach, reach);
    const int jmax = (int)floor(reach / lk);
    for (int j = 0; j <= jmax; ++j) {
        const double dk = (double)lk * j, x = (double)sh * j;
        const int ilo = j == 0 ? 1 : (int)ceil((-reach - x) / lh);
        const int ihi = (int)floor((reach - x) / lh);
        for (int i = ilo; i <= ihi; ++i) {
            const double dh = (double)lh * i + x;              // (whole numbers: exact)
            const double v2 = lat_add(lat_mul(dh, dh), lat_mul(dk, dk));
            if (v2 > r2) continue;
            double m = 0;
            for (int c = 0; c < 3; ++c) {
                const double d = fabs(lat_add(lat_mul(dh, ad[c]), lat_mul(dk, bd[c])));
                if (d > m) m = d;
            }
            if (m < lat_add(1.0 + margin, lat_mul(curve, sqrt(v2)))) return false;
        }
    }
    return true;
}

// The square lattice of side ceil(reach), which no vector shorter than `reach`
// belongs to; {0, 0, 0} when that side would not fit the 12-bit fields of
// pack_lattice.
BSG_LATTICE_FN PhaseLattice square_lattice(double reach) {
    if (!(reach < 4095.0)) return {0, 0, 0};
    const int L = (int)ceil(reach);
    return {L > 1 ? L : 1, L > 1 ? L : 1, 0};
}

constexpr int LATTICE_PHASES = 16;           // most phases lh * lk tried
constexpr int LATTICE_CANDIDATES = 220;      // lattices (lh, lk, sh) with lh lk <= 16

// Lattice number c in the order of preference: fewest phases lh lk, then
// fewest rows lk, then the smallest shift ({0, 0, 0} past the last).
BSG_LATTICE_FN PhaseLattice lattice_candidate(int c) {
    for (int d = 1; d <= LATTICE_PHASES; ++d)
        for (int lk = 1; lk <= d; ++lk) {
            if (d % lk) continue;
            const int lh = d / lk;
            if (c < lh) return {lh, lk, c};
            c -= lh;
        }
    return {0, 0, 0};
}

// The safe lattice with the fewest phases (up to max_phases; lattice_candidate's
// order), else the square one.  lattice.cu makes this choice on the device, 32
// candidates at a time; this is the host's form, and what the tests hold that to.
// curve: bound on the extra displacement (voxels per pixel step of the
// lattice vector) of a curved insertion surface; 0 for the plane.
inline PhaseLattice choose_lattice(const double ad[3], const double bd[3], int max_phases = LATTICE_PHASES,
                                   double curve = 0.0) {
    const double reach = lattice_reach(ad, bd, curve);
    if (reach < 64.0) {
        for (int d = 1; d <= max_phases; ++d)
            for (int lk = 1; lk <= d; ++lk) {
                if (d % lk) continue;
                const int lh = d / lk;
                for (int sh = 0; sh < lh; ++sh)
                    if (lattice_ok(ad, bd, lh, lk, sh, reach, curve)) return {lh, lk, sh};
            }
    }
    return square_lattice(reach);
}

// lh | lk << 12 | sh << 24 (0: no lattice chosen).
BSG_LATTICE_FN int pack_lattice(const PhaseLattice& l) {
    if (l.lh <= 0 || l.lk <= 0 || l.lh > 4095 || l.lk > 4095 || l.sh < 0 || l.sh > 127) return 0;
    return l.lh | (l.lk << 12) | (l.sh << 24);
}

}  // namespace bsg

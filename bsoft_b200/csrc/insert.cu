// insert.cu - central-section insertion (fspace_pack_2D +
// fspace_2D_interpolate, bsoft/src/img/Bimage_reconstruct.cpp:25-174).
//
// The reference scatters every pixel q = (h, k) of each padded particle
// transform, q in [-ft/2, ft/2-1]^2, to the map frequency
// m = R (h, k, 0) * inv * mscale and adds F(q) * w to the 1 (nearest) or 8
// (trilinear) voxels around m, with index wrap-around, on a full complex
// N^3 map, plus w to the weight map (and w |F|^2, w^2 to the FOM channels).
//
// Decomposition: one warp owns one tile of the map (8 x 8 x 8, 16 x 16 x 4,
// 16 x 8 x 8 or 16 x 16 x 8 voxels; the autotuner picks the shape) and keeps its
// sums in shared memory in FP32 (each contribution is the float product
// F * w, as the reference forms it), adding them to the FP64 accumulators in
// HBM at the end of the batch.  Nothing else writes the tile, so there are
// no atomics and no block-wide barriers.  The warp tests 32 particles at a
// time against its tile (plane slab and reach, per wrap-around alias) and
// walks the pixels of each particle that reaches it, in particle order.
//
// Conflict-free lanes: the pixels of a particle's footprint are visited on
// a lattice whose points never share a unit cell of the map, one phase
// after another.  Each particle record carries the smallest such lattice
// for its orientation (lattice.h; 5 to 9 phases at step 0.5); without one,
// a lattice safe for every orientation is used (points at least sqrt(3)
// voxels apart: L x L pixels with L = ceil(sqrt(3)/step), step = voxels per
// pixel, or at step 0.5 the 12-phase lattice spanned by (4, 0) and (2, 3)
// pixels).  Two points of a phase have different base voxels floor(m), so
// for any one corner offset the lanes of a warp touch distinct voxels: a
// plain read-modify-write of shared memory is exact.
// The order of every voxel's sum (particle, alias, phase, lattice point,
// corner) is fixed, so results are bitwise reproducible.  Tiles are visited
// heaviest first (nearest to the Fourier origin, where every particle's
// plane passes) so the long ones do not trail the launch, and each tile has
// R replica warps that take consecutive slices of the particle list into
// private partial sums, added in replica order by the last of them to arrive
// (grid4_kernel) or, with the FOM channels, by a combine pass.
//
// A row's pixels are found exactly from the three slab constraints of the tile
// box.  grid4_kernel bounds them in FP32 where that settles the integers, gives
// each lane a group of a row's pixels, one of each column phase, and steps
// through the phases together (walk_groups).  The FOM path enumerates phase by
// phase: lane j computes the h-interval of lattice row j (once for all phases
// that walk it), a warp scan turns the row counts into offsets, and lanes take
// points in order (walk_pair).
#include "context.cuh"
#include "row_range.h"

#include <math.h>

namespace bsg {

constexpr int WARPS = 4;                  // warps (tiles) per block

struct InsertArgs {
    const float2* spec;        // batch x (ft+1) x (ft+2), centred
    const DevParticle* part;   // particles of this launch
    const TileTest* test;      // their tile tests
    int np;
    int half;                  // only particles of this half map (-1: all)
    int N, ft, pitch;
    int ntx, nty, ntz;         // tiles per axis
    const int* order;          // tile visiting order (heaviest first)
    int R;                     // replicas per tile (each takes a slice of the particles)
    int nlow;                  // tiles below the split (grid4_kernel)
    float* psum;               // R > 1: replica partial sums, tiles x R x 3 x tile voxels
    unsigned* arrived;         // per tile: replicas done (bits 0-7) and which stored sums (8 + rep)
    double* fsum;              // FOM path, R > 1: replica partial sums, R x 5 x N^3
    int zsplit;                // > 0: half-space gridding (walk_edges)
    double2* evol;             // half-space: unpaired pixels' sums below zsplit (zsplit x N^2)
    double* ew;
    float edge_rmin;           // unpaired pixels lie at least this far from the origin (voxels)
    float edge_rmax;           // and no pixel farther than this
    float rmax;                // nor, with its tent and an Ewald surface's curvature, than this
    int interp;
    double maxs2, mins2, mscale;
    double2* vol;
    double* w;
    double* pow;
    double* w2;
};

// The alias combinations (bit i: axis i shifted by -N) under which a pixel at
// most rmax voxels from the origin can reach the tile: for most tiles one or two
// of the eight that tile_mask then has to test for every record.
template <int TX, int TY, int TZ>
__device__ __forceinline__ unsigned tile_aliases(int x0, int y0, int z0, int N, float rmax) {
    const float ex = 0.5f * (TX - 1), ey = 0.5f * (TY - 1), ez = 0.5f * (TZ - 1);
    unsigned set = 0;
    for (int a = 0; a < 8; ++a) {
        const float dx = fmaxf(0.f, fabsf(x0 - ((a & 1) ? N : 0) + ex) - ex);
        const float dy = fmaxf(0.f, fabsf(y0 - ((a & 2) ? N : 0) + ey) - ey);
        const float dz = fmaxf(0.f, fabsf(z0 - ((a & 4) ? N : 0) + ez) - ez);
        if (dx * dx + dy * dy + dz * dz <= rmax * rmax) set |= 1u << a;
    }
    return set;
}

// Does the record's plane come within reach of the tile for the alias
// combinations in `aliases`?  Bitmask over the 8.
template <int TX, int TY, int TZ>
__device__ __forceinline__ unsigned tile_mask(const TileTest& t, unsigned aliases, int x0, int y0, int z0, int N) {
    unsigned mask = 0;
    const float ex = 0.5f * (TX - 1), ey = 0.5f * (TY - 1), ez = 0.5f * (TZ - 1);
    const float slack = t.slab + fabsf(t.n[0]) * ex + fabsf(t.n[1]) * ey + fabsf(t.n[2]) * ez;
#pragma unroll 1
    for (unsigned left = aliases; left; left &= left - 1) {
        const int a = __ffs(left) - 1;
        const float cx = x0 - ((a & 1) ? N : 0) + ex;
        const float cy = y0 - ((a & 2) ? N : 0) + ey;
        const float cz = z0 - ((a & 4) ? N : 0) + ez;
        if (fabsf(cx) - ex > t.reach[0] || fabsf(cy) - ey > t.reach[1] || fabsf(cz) - ez > t.reach[2]) continue;
        if (fabsf(t.n[0] * cx + t.n[1] * cy + t.n[2] * cz) > slack) continue;
        mask |= 1u << a;
    }
    return mask;
}

__device__ __forceinline__ float pixel_weight_gate(const InsertArgs& a, const DevParticle& P, int h, int k,
                                                   bool& keep) {
    // s2 as fspace_pack_2D forms it: s = (h, k) * inv in double
    const double inv = sqrt(P.inv2);
    const double sx = h * inv, sy = k * inv;
    const double s2 = sx * sx + sy * sy;
    keep = (s2 >= a.mins2 && s2 <= a.maxs2);
    const double d = (a.maxs2 - s2) * a.mscale;
    return d < 1.0 ? (float)sqrt(d > 0 ? d : 0.0) : 1.0f;
}

// Tile sums are FP32: one batch adds at most a few thousand contributions
// to a voxel, each the float product F * w the reference forms; the batch's
// sums are folded into the FP64 map accumulators, which carry the long
// reduction over all particles.
typedef float tacc_t;

struct TileAcc {
    tacc_t* re;
    tacc_t* im;
    tacc_t* w;
    tacc_t* p;
    tacc_t* q;
};

__device__ __forceinline__ void add_voxel(const TileAcc& A, int i, float2 f, float w) {
    A.re[i] += f.x * w;
    A.im[i] += f.y * w;
    A.w[i] += w;
    A.p[i] += w * (f.x * f.x + f.y * f.y);
    A.q[i] += w * w;
}

// One pixel (h, k) of particle P against the tile at alias origin o.  All
// lanes of the warp call this together (`act` false for idle lanes); the
// __syncwarp after each corner orders the shared-memory updates of
// different corner offsets, which may touch the same voxel from different
// lanes.
template <bool GATE, int TX, int TY, int TZ>
__device__ __forceinline__ void pixel(const InsertArgs& a, const DevParticle& P, const float2* S, const TileAcc& A,
                                      double ox, double oy, double oz, int h, int k, bool act) {
    const int hf = a.ft / 2;
    float wt = P.pw;
    if (GATE && act) {
        bool keep;
        const float tw = pixel_weight_gate(a, P, h, k, keep);
        if (!keep) act = false;
        wt *= tw;
    }
    // map frequency relative to the tile origin, in double as the reference
    // forms it
    double mx = h * P.ad[0] + k * P.bd[0] - ox;
    double my = h * P.ad[1] + k * P.bd[1] - oy;
    double mz = h * P.ad[2] + k * P.bd[2] - oz;
    if (P.ewh != 0.0) {
        // Ewald surface: s_z = +-(lambda/2) s2 along R[:,2] (Bimage_reconstruct.cpp:157-168)
        const double sx = h * P.inv, sy = k * P.inv, sz = P.ewh * (sx * sx + sy * sy);
        mx += sz * P.cd[0];
        my += sz * P.cd[1];
        mz += sz * P.cd[2];
    }
    const float2 f = act ? __ldg(S + (size_t)(k + hf) * a.pitch + (h + hf)) : make_float2(0.f, 0.f);
    if (a.interp != 2) {
        const double fx = floor(mx + 0.5), fy = floor(my + 0.5), fz = floor(mz + 0.5);
        const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
        float w = wt;
        if (a.interp == 1) {
            const double dx = mx - fx, dy = my - fy, dz = mz - fz;
            w = (float)((double)wt * (1.0 - sqrt(dx * dx + dy * dy + dz * dz)));
        }
        if (act && (unsigned)ix < TX && (unsigned)iy < TY && (unsigned)iz < TZ && w > 0.f)
            add_voxel(A, (iz * TY + iy) * TX + ix, f, w);
        __syncwarp();
        return;
    }
    const double flx = floor(mx), fly = floor(my), flz = floor(mz);
    const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
    const float rx = (float)(mx - flx), ry = (float)(my - fly), rz = (float)(mz - flz);
#pragma unroll
    for (int dz = 0; dz < 2; ++dz) {
        const int z = iz + dz;
        const float wz = dz ? rz : 1.f - rz;
#pragma unroll
        for (int dy = 0; dy < 2; ++dy) {
            const int y = iy + dy;
            const float wyz = (dy ? ry : 1.f - ry) * wz * wt;
#pragma unroll
            for (int dx = 0; dx < 2; ++dx) {
                const int x = ix + dx;
                if (act && (unsigned)x < TX && (unsigned)y < TY && (unsigned)z < TZ)
                    add_voxel(A, (z * TY + y) * TX + x, f, (dx ? rx : 1.f - rx) * wyz);
                __syncwarp();
            }
        }
    }
}

// Walk the pixels of particle P (alias origin o) whose contributions can
// reach the tile, phase by phase of the lattice, calling pix(h, k, act) with
// all lanes of the warp together (act false for idle lanes).
template <int TX, int TY, int TZ, class Pix>
__device__ __forceinline__ void walk_pair(const DevParticle& P, int hf, double ox, double oy, double oz, int lane,
                                          int* s_row, Pix&& pix) {
    // open box of map frequencies whose tent touches the tile (an Ewald
    // surface adds up to P.ezmax voxels to every coordinate)
    const double e = P.ezmax;
    const double lo[3] = {ox - 1.0 - e, oy - 1.0 - e, oz - 1.0 - e};
    const double hi[3] = {ox + TX + e, oy + TY + e, oz + TZ + e};
    double vc = 0, hv = 0, uc = 0, hu = 0;
    for (int i = 0; i < 3; ++i) {
        const double c = 0.5 * (lo[i] + hi[i]), e = 0.5 * (hi[i] - lo[i]);
        vc += P.bd[i] * c; hv += fabs(P.bd[i]) * e;
        uc += P.ad[i] * c; hu += fabs(P.ad[i]) * e;
    }
    vc *= P.inv_st2; hv *= P.inv_st2; uc *= P.inv_st2; hu *= P.inv_st2;
    const int k_lo = max((int)ceil(vc - hv), -hf), k_hi = min((int)floor(vc + hv), hf - 1);
    const int h_lo = max((int)ceil(uc - hu), -hf), h_hi = min((int)floor(uc + hu), hf - 1);
    if (k_lo > k_hi || h_lo > h_hi) return;
    // Conflict-free lattice: two points of one phase never share a unit cell
    // of the map.  P.lat, when set, is the smallest such lattice for this
    // particle's orientation (lattice.h; 5 to 9 phases at step 0.5).  Else
    // one safe for every orientation, whose points are >= sqrt(3) voxels
    // apart: the square lattice of L x L pixels (L = ceil(sqrt(3)/step)), or,
    // where it has fewer phases, the lattice spanned by (4, 0) and (2, 3)
    // pixels (shortest vector sqrt(13) pixels; 12 phases at step 0.5).
    // Row j of phase (ph, pk) is k = k_lo + pk + Lk j, its points
    // h = h_lo + ph + sh j + Lh i.
    int Lh, Lk, sh;
    if (P.lat) {
        Lh = P.lat & 0xfff; Lk = (P.lat >> 12) & 0xfff; sh = (P.lat >> 24) & 0x7f;
    } else {
        const int L = max(1, (int)ceilf(1.7320508f * 1.0001f * P.inv_step));
        if (L * L > 12 && 3.6055513f * P.step >= 1.7320508f * 1.0001f) { Lh = 4; Lk = 3; sh = 2; }
        else { Lh = L; Lk = L; sh = 0; }
    }
    // per-axis 1 / ad (0 when the axis does not vary along h)
    const double* ia = P.iad;
    for (int pk = 0; pk < Lk; ++pk) {
        const int k0 = k_lo + pk;
        if (k0 > k_hi) break;
        const int nrows = (k_hi - k0) / Lk + 1;
        for (int jb = 0; jb < nrows; jb += 32) {
            // lane j: the exact h range [hl, hh] of row k = k0 + Lk (jb + j),
            // shared by the Lh phases that walk this row
            const int j = jb + lane;
            const int k = k0 + Lk * j;
            double hl = h_lo, hh = h_hi;
            bool live = j < nrows;
            if (live) {
                for (int i = 0; i < 3; ++i) {
                    const double base = k * P.bd[i];
                    if (ia[i] != 0.0) {
                        double p0 = (lo[i] - base) * ia[i], p1 = (hi[i] - base) * ia[i];
                        if (p0 > p1) { const double t = p0; p0 = p1; p1 = t; }
                        hl = fmax(hl, p0);
                        hh = fmin(hh, p1);
                    } else if (!(base > lo[i] && base < hi[i])) {
                        live = false;
                    }
                }
                live = live && hl <= hh;
            }
            for (int ph = 0; ph < Lh; ++ph) {
                if (sh == 0 && h_lo + ph > h_hi) break;
                int hfirst = 0, cnt = 0;
                if (live) {
                    // lattice h = h0 + Lh i inside [hl, hh]
                    const int h0 = h_lo + ph + sh * j;
                    const int i0 = (int)ceil((hl - h0) / Lh), i1 = (int)floor((hh - h0) / Lh);
                    if (i1 >= i0) { hfirst = h0 + Lh * i0; cnt = i1 - i0 + 1; }
                }
                // exclusive scan of the row counts
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(0xffffffffu, incl, 31);
                if (total == 0) continue;
                s_row[lane] = incl;                        // inclusive end of row j
                s_row[32 + lane] = hfirst;
                s_row[64 + lane] = k;
                __syncwarp();
                for (int t0 = 0; t0 < total; t0 += 32) {
                    const int t = t0 + lane;
                    const bool act = t < total;
                    int r = 0;                              // row holding point t
#pragma unroll
                    for (int sft = 16; sft > 0; sft >>= 1)
                        if (s_row[r + sft - 1] <= t) r += sft;
                    r = min(r, 31);
                    const int before = r ? s_row[r - 1] : 0;
                    const int h = s_row[32 + r] + Lh * (t - before);
                    pix(h, s_row[64 + r], act);
                }
                __syncwarp();
            }
        }
    }
}

// floor(x / d) for 0 < d and |x| < 2^20, from an approximate reciprocal of
// d: the float quotient is within one of the answer, and the remainder
// corrects it (the integers a division would give, without one per row).
__device__ __forceinline__ int floor_div(int x, int d, float inv_d) {
    int q = __float2int_rd((float)x * inv_d);
    int r = x - q * d;
    if (r < 0) { --q; r += d; }
    if (r >= d) ++q;
    return q;
}

// One (tile, particle, alias) pair of the gridding walk, set up by one lane
// (setup_pair) and read by the whole warp: pixel ranges, the anchor pixel and
// its tile-relative map coordinate, and the particle's constants.
struct __align__(16) Pair {
    int h_lo, h_hi, k_lo, k_hi;       // edge walk: t0, t1 of line 0 and line 1
    int hc, kc;                       // anchor pixel
    int part, lat;
    float bx, by, bz, pw;             // coordinate of the anchor; particle weight
    float ax, ay, az, inv_step;       // map step per pixel along h
    float cx, cy, cz;                 // and along k
    int spec;
};

// The FP32 form of a row's pixel bounds: along axis i, a row whose coordinate
// at h = hc is b has its tents inside the tile for h - hc between
// -b ia + lo and -b ia + hi, each with its error bound taken off and added on.
struct __align__(16) RowBounds {
    float ia[3], lo_a[3], lo_b[3], hi_a[3], hi_b[3];
    int exact;                        // an axis does not vary along h: the FP64 form only
};
constexpr int QN = 8;                 // pairs set up at a time

// The pixels [hmin, hmax] of row k whose tents reach the tile box, in FP64:
// the set of pixels that a tile grids is defined by these bounds.
template <int TX, int TY, int TZ>
__device__ __noinline__ int2 row_bounds(const DevParticle& P, int k, int h_lo, int h_hi, double ox, double oy,
                                        double oz, double e) {
    const double lo[3] = {ox - 1.0 - e, oy - 1.0 - e, oz - 1.0 - e};
    const double hi[3] = {ox + TX + e, oy + TY + e, oz + TZ + e};
    double hl = h_lo, hh = h_hi;
    bool live = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double base = k * P.bd[i], ia = P.iad[i];
        if (ia != 0.0) {
            double p0 = (lo[i] - base) * ia, p1 = (hi[i] - base) * ia;
            if (p0 > p1) { const double t = p0; p0 = p1; p1 = t; }
            hl = fmax(hl, p0);
            hh = fmin(hh, p1);
        } else if (!(base > lo[i] && base < hi[i])) {
            live = false;
        }
    }
    return live && hl <= hh ? make_int2((int)ceil(hl), (int)floor(hh)) : make_int2(0, -1);
}

// Walk the pixels of pair Q that can reach the tile, on the particle's phase
// lattice: lane t takes a group of Lh consecutive pixels of one lattice row
// (h = g, g + 1, ..., g + Lh - 1 with g = h_lo + sh j + Lh i), one pixel of
// each column phase, and the warp steps through the phases together: at step
// ph every lane holds a point of phase (ph, pk), so the conflict-free property
// of a phase holds, and pix() ends each step with __syncwarp.  Each pixel's
// value is fetched one step before it is gridded (fetch(h, k, act), then
// pix(value, h, k, act)).  (Groups that start at a row's first pixel instead
// of on the lattice fill the lanes better, 10.5 against 11.4 thousand steps a
// particle, but add a voxel's contributions in another order.)
//
// The rows' bounds are FP32 with an error bound; where that does not settle
// the integers (1 to 2% of the walks) the warp evaluates them in FP64, so the
// pixels are the FP64 ones always.  A lane finds its group's row from the
// groups' starts in a bit mask.  The FP64 bounds, a shuffle scan and a binary
// search in shared memory took 2.8 of 6.0 ms per 953 particles at 256^3.
template <int TX, int TY, int TZ, class Fetch, class Pix>
__device__ __forceinline__ void walk_groups(const DevParticle& P, const Pair& Q, const RowBounds& B, double e,
                                             double ox, double oy, double oz, int lane, int4* s_row, Fetch&& fetch,
                                             Pix&& pix) {
    const int k_lo = Q.k_lo, k_hi = Q.k_hi, h_lo = Q.h_lo, h_hi = Q.h_hi;
    int Lh, Lk, sh;
    if (Q.lat) {
        Lh = Q.lat & 0xfff; Lk = (Q.lat >> 12) & 0xfff; sh = (Q.lat >> 24) & 0x7f;
    } else {
        const int L = max(1, (int)ceilf(1.7320508f * 1.0001f * Q.inv_step));
        if (L * L > 12 && 3.6055513f * P.step >= 1.7320508f * 1.0001f) { Lh = 4; Lk = 3; sh = 2; }
        else { Lh = L; Lk = L; sh = 0; }
    }
    const float iLh = __fdividef(1.0f, (float)Lh);
    const unsigned lt = (1u << lane) - 1u;
    for (int pk = 0; pk < Lk; ++pk) {
        const int k0 = k_lo + pk;
        if (k0 > k_hi) break;
        for (int jb = 0; k0 + Lk * jb <= k_hi; jb += 32) {
            const int j = jb + lane, k = k0 + Lk * j;
            const bool row = k <= k_hi;
            int hmin = 0, hmax = -1;
            bool sure = !row;
            if (row && !B.exact) {
                const float dk = (float)(k - Q.kc);
                const float b[3] = {fmaf(dk, Q.cx, Q.bx), fmaf(dk, Q.cy, Q.by), fmaf(dk, Q.cz, Q.bz)};
                float la = -1e9f, lb = -1e9f, ha = 1e9f, hb = 1e9f;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const float q = -b[i] * B.ia[i];
                    la = fmaxf(la, q + B.lo_a[i]);
                    lb = fmaxf(lb, q + B.lo_b[i]);
                    ha = fminf(ha, q + B.hi_a[i]);
                    hb = fminf(hb, q + B.hi_b[i]);
                }
                const RowRange r = row_range(Q.hc, h_lo, h_hi, la, lb, ha, hb);
                hmin = r.lo;
                hmax = r.hi;
                sure = r.sure;
            }
            if (__any_sync(0xffffffffu, !sure) && row) {
                const int2 r = row_bounds<TX, TY, TZ>(P, k, h_lo, h_hi, ox, oy, oz, e);
                hmin = r.x;
                hmax = r.y;
            }
            // the row's groups; cnt < 16 in all but extreme geometries
            int gfirst = 0, cnt = 0;
            if (hmax >= hmin) {
                const int g0 = h_lo + sh * j, i0 = floor_div(hmin - g0, Lh, iLh);
                gfirst = g0 + Lh * i0;
                cnt = floor_div(hmax - g0, Lh, iLh) - i0 + 1;
            }
            int off, total;
            if (!__any_sync(0xffffffffu, cnt > 15)) {
                const unsigned b0 = __ballot_sync(0xffffffffu, cnt & 1), b1 = __ballot_sync(0xffffffffu, cnt & 2),
                               b2 = __ballot_sync(0xffffffffu, cnt & 4), b3 = __ballot_sync(0xffffffffu, cnt & 8);
                off = __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt) + 8 * __popc(b3 & lt);
                total = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2) + 8 * __popc(b3);
            } else {
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                off = incl - cnt;
                total = __shfl_sync(0xffffffffu, incl, 31);
            }
            if (total == 0) continue;
            const unsigned some = __ballot_sync(0xffffffffu, cnt > 0);
            if (cnt > 0) s_row[__popc(some & lt)] = make_int4(gfirst - Lh * off, k, hmin, hmax);
            __syncwarp();
            for (int t0 = 0; t0 < total; t0 += 32) {
                const bool here = cnt > 0 && (unsigned)(off - t0) < 32u;
                const unsigned starts = __reduce_or_sync(0xffffffffu, here ? 1u << (off - t0) : 0u);
                const int before = __popc(__ballot_sync(0xffffffffu, cnt > 0 && off < t0));
                const int t = t0 + lane;
                const bool in = t < total;
                const int4 r = s_row[max(0, before + __popc(starts & (lt | (1u << lane))) - 1)];
                const int g = r.x + Lh * t;
                bool act = in && g >= r.z && g <= r.w;
                float2 f = fetch(g, r.y, act);
#pragma unroll 1
                for (int ph = 0; ph < Lh; ++ph) {
                    const int h = g + ph + 1;
                    const bool next = in && ph + 1 < Lh && h >= r.z && h <= r.w;
                    const float2 fn = fetch(h, r.y, next);
                    pix(f, h - 1, r.y, act);
                    f = fn;
                    act = next;
                }
            }
            __syncwarp();
        }
    }
}

// Half-space gridding.  A real image's transform is Hermitian, F(-q) =
// conj(F(q)), and a pixel q and its mate -q land at mirrored map positions
// m and -m (m is linear in q) with mirrored trilinear corners of equal
// weights.  So the sums P of the pixels that have their mate in the stored
// transform (q in [-ft/2, ft/2 - 1]^2) satisfy P(-v) = conj(P(v)),
// P_w(-v) = P_w(v); the others - the row k = -ft/2 and the column
// h = -ft/2 - make sums U of their own.  With zsplit > N/2 (so every voxel
// or its mirror lies below it), the tiles below zsplit grid P (walk_groups
// without the unpaired pixels) into the map accumulators and U into evol /
// ew; the tiles at or above zsplit grid only U, into the map accumulators.
// Reading the map gives P(v) + U(v) below the split and conj(P(-v)) + U(v)
// above it: sums of the same contributions as the full map's, none of them
// subtracted, so a voxel that nothing reaches reads exactly zero.
// walk_edges visits the unpaired pixels whose tents reach the tile, one
// line at a time, points L pixels apart (L step >= sqrt(3) voxels) so that
// the lanes of a call touch distinct cells; edge_range gives a line's pixels
// (line 0: (t, -hf), t in [-hf, hf - 1]; line 1: (-hf, t), t in [-hf + 1,
// hf - 1]; t0 > t1: none).
template <int TX, int TY, int TZ>
__device__ __noinline__ void edge_range(const DevParticle& P, int hf, double ox, double oy, double oz, int line,
                                           int& t0, int& t1) {
    const double lo[3] = {ox - 1.0, oy - 1.0, oz - 1.0};
    const double hi[3] = {ox + TX, oy + TY, oz + TZ};
    const bool along_h = line == 0;
    double tl = line == 0 ? -hf : -hf + 1;
    double th = hf - 1;
    bool live = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double idir = along_h ? P.iad[i] : P.ibd[i];
        const double base = -hf * (along_h ? P.bd[i] : P.ad[i]);
        if (idir != 0.0) {
            double p0 = (lo[i] - base) * idir, p1 = (hi[i] - base) * idir;
            if (p0 > p1) { const double t = p0; p0 = p1; p1 = t; }
            tl = fmax(tl, p0);
            th = fmin(th, p1);
        } else if (!(base >= lo[i] && base <= hi[i])) {
            live = false;
        }
    }
    t0 = 0;
    t1 = -1;
    if (live && tl <= th) {
        t0 = (int)ceil(tl);
        t1 = (int)floor(th);
    }
}

template <class Fetch, class Pix>
__device__ __forceinline__ void walk_edges(const Pair& Q, int hf, int lane, Fetch&& fetch, Pix&& pix) {
    const int L = max(1, (int)ceilf(1.7320508f * 1.0001f * Q.inv_step));
#pragma unroll 1
    for (int line = 0; line < 2; ++line) {
        const int t0 = line ? Q.k_lo : Q.h_lo, t1 = line ? Q.k_hi : Q.h_hi;
        for (int ph = 0; ph < L; ++ph) {
            const int first = t0 + ph;
            if (first > t1) break;
            for (int tb = first; tb <= t1; tb += 32 * L) {
                const int t = tb + L * lane;
                const int h = line ? -hf : t, k = line ? t : -hf;
                const bool act = t <= t1;
                pix(fetch(h, k, act), h, k, act);
            }
        }
    }
}

// Of the aliases in `mask`, those whose tile box (grown by a voxel) comes
// near a line of unpaired pixels: the box's enclosing sphere against the
// segment, in FP32 with a margin above its rounding (a superset; edge_range
// decides).  A plane reaches some 1,400 (tile, alias) pairs below the split of
// a 256^3 map, its two lines about 130: setting all of them up took 2.9 of
// 13.3 ms per 2,000 particles.
template <int TX, int TY, int TZ>
__device__ __forceinline__ unsigned edge_mask(const DevParticle& P, unsigned mask, int x0, int y0, int z0, int N,
                                              int ft) {
    const float hf = 0.5f * ft;
    const float ex = 0.5f * (TX + 1), ey = 0.5f * (TY + 1), ez = 0.5f * (TZ + 1);
    const float R = sqrtf(ex * ex + ey * ey + ez * ez) + 0.05f;
    const float ax = P.af[0], ay = P.af[1], az = P.af[2], bx = P.bf[0], by = P.bf[1], bz = P.bf[2];
    const float ia = 1.0f / (ax * ax + ay * ay + az * az), ib = 1.0f / (bx * bx + by * by + bz * bz);
    unsigned out = 0;
    while (mask) {
        const int al = __ffs(mask) - 1;
        mask &= mask - 1;
        const float cx = x0 - ((al & 1) ? N : 0) + 0.5f * (TX - 1), cy = y0 - ((al & 2) ? N : 0) + 0.5f * (TY - 1),
                    cz = z0 - ((al & 4) ? N : 0) + 0.5f * (TZ - 1);
        // d = centre - (the line's offset -hf v); the nearest point is t u
        float dx = fmaf(hf, bx, cx), dy = fmaf(hf, by, cy), dz = fmaf(hf, bz, cz);
        float t = fminf(fmaxf((dx * ax + dy * ay + dz * az) * ia, -hf), hf);
        dx -= t * ax; dy -= t * ay; dz -= t * az;
        bool near = dx * dx + dy * dy + dz * dz <= R * R;
        dx = fmaf(hf, ax, cx); dy = fmaf(hf, ay, cy); dz = fmaf(hf, az, cz);
        t = fminf(fmaxf((dx * bx + dy * by + dz * bz) * ib, -hf), hf);
        dx -= t * bx; dy -= t * by; dz -= t * bz;
        near = near || dx * dx + dy * dy + dz * dz <= R * R;
        if (near) out |= 1u << al;
    }
    return out;
}

// Can an unpaired pixel (at least rmin voxels from the origin, and no pixel
// beyond rmax) reach the tile, under some wrap-around alias?  (FP32 with a
// margin: a superset.)
template <int TX, int TY, int TZ>
__device__ __forceinline__ bool tile_reaches_edges(int x0, int y0, int z0, int N, float rmin, float rmax) {
    const int o[3] = {x0, y0, z0}, T[3] = {TX, TY, TZ};
    for (int a = 0; a < 8; ++a) {
        float nr = 0, fr = 0;
        for (int i = 0; i < 3; ++i) {
            const float lo = o[i] - (((a >> i) & 1) ? N : 0) - 1.0f, hi = lo + T[i] + 1.0f;
            const float n = fmaxf(0.f, fmaxf(lo, -hi)), f = fmaxf(fabsf(lo), fabsf(hi));
            nr += n * n;
            fr += f * f;
        }
        if (nr <= rmax * rmax * 1.00001f && fr * 1.00001f >= rmin * rmin) return true;
    }
    return false;
}

template <bool GATE, int TX, int TY, int TZ>
__device__ __forceinline__ void scatter_particle(const InsertArgs& a, const DevParticle& P, const float2* S,
                                                 const TileAcc& A, double ox, double oy, double oz, int lane,
                                                 int* s_row) {
    walk_pair<TX, TY, TZ>(P, a.ft / 2, ox, oy, oz, lane, s_row, [&](int h, int k, bool act) {
        pixel<GATE, TX, TY, TZ>(a, P, S, A, ox, oy, oz, h, k, act);
    });
}

// Tile sums -> HBM: added to the map accumulators (one replica), or stored
// into this replica's partial buffer (combined later in replica order).
template <int TX, int TY, int TZ>
__device__ __forceinline__ void fold_tile(const InsertArgs& a, const TileAcc& A, int x0, int y0, int z0, int r,
                                          int lane) {
    const int N = a.N;
    constexpr int TV = TX * TY * TZ;
    const size_t N3 = (size_t)N * N * N;
    for (int i = lane; i < TV; i += 32) {
        const int lx = i % TX, ly = (i / TX) % TY, lz = i / (TX * TY);
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        if (x < N && y < N && z < N) {
            const size_t idx = ((size_t)z * N + y) * N + x;
            if (a.R > 1) {
                double* pb = a.fsum + (size_t)r * 5 * N3 + idx;
                pb[0] = A.re[i];
                pb[N3] = A.im[i];
                pb[2 * N3] = A.w[i];
                pb[3 * N3] = A.p[i]; pb[4 * N3] = A.q[i];
            } else {
                double2 o = a.vol[idx];
                o.x += A.re[i];
                o.y += A.im[i];
                a.vol[idx] = o;
                a.w[idx] += A.w[i];
                a.pow[idx] += A.p[i]; a.w2[idx] += A.q[i];
            }
        }
        A.re[i] = 0; A.im[i] = 0; A.w[i] = 0;
        A.p[i] = 0; A.q[i] = 0;
    }
    __syncwarp();
}

template <bool GATE, int TX, int TY, int TZ>
__global__ void __launch_bounds__(WARPS * 32) insert_kernel(InsertArgs a) {
    constexpr int NCH = 5;
    constexpr int TV = TX * TY * TZ;
    extern __shared__ tacc_t s_dacc[];                 // WARPS x NCH x TV
    tacc_t* const my_acc = s_dacc + (size_t)(threadIdx.x >> 5) * NCH * TV;
    __shared__ int s_rows[WARPS][96];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gw = blockIdx.x * WARPS + warp;
    const int slot = gw / a.R, rep = gw % a.R;       // replicas of a tile are adjacent
    if (slot >= a.ntx * a.nty * a.ntz) return;
    const int tile = a.order[slot];
    // this replica's slice of the particles
    const int p_lo = (int)((long)a.np * rep / a.R), p_hi = (int)((long)a.np * (rep + 1) / a.R);
    const int x0 = (tile % a.ntx) * TX, y0 = ((tile / a.ntx) % a.nty) * TY, z0 = (tile / (a.ntx * a.nty)) * TZ;
    const int N = a.N;
    const int hf = a.ft / 2;
    const size_t spec_stride = (size_t)(2 * hf + 1) * a.pitch;
    TileAcc A;
    A.re = my_acc; A.im = A.re + TV; A.w = A.im + TV;
    A.p = A.w + TV; A.q = A.p + TV;
    for (int i = lane; i < NCH * TV; i += 32) my_acc[i] = 0;
    __syncwarp();

    const unsigned aliases = tile_aliases<TX, TY, TZ>(x0, y0, z0, N, a.rmax);
    for (int base = p_lo; base < p_hi; base += 32) {
        const int p = base + lane;
        unsigned mask = 0;
        if (p < p_hi) {
            const TileTest t = a.test[p];
            if (t.half == a.half || a.half < 0) mask = tile_mask<TX, TY, TZ>(t, aliases, x0, y0, z0, N);
        }
        unsigned todo = __ballot_sync(0xffffffffu, mask != 0);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const unsigned am = __shfl_sync(0xffffffffu, mask, src);
            const int pi = base + src;
            const DevParticle& P = a.part[pi];
            const float2* S = a.spec + (size_t)P.spec * spec_stride;
            for (int al = 0; al < 8; ++al)
                if ((am >> al) & 1u)
                    scatter_particle<GATE, TX, TY, TZ>(a, P, S, A, (double)(x0 - ((al & 1) ? N : 0)),
                                                (double)(y0 - ((al & 2) ? N : 0)),
                                                (double)(z0 - ((al & 4) ? N : 0)), lane, s_rows[warp]);
        }
    }
    fold_tile<TX, TY, TZ>(a, A, x0, y0, z0, rep, lane);
}

// ---- gridding without the FOM channels -----------------------------------
//
// The map tile is an array of float2 cells {F re * w, F im * w} and one of
// float weights, so a corner's read-modify-write is an 8-byte and a 4-byte
// load, three adds and the two stores.  Cell (x, y, z) of the tile sits at
// index x + PX y + PP z: the plane pitch PP (PX TY plus a few unused cells)
// spreads the cells that a warp's lattice points touch over the banks, and the
// corner offsets stay compile-time constants.  The shared-memory pipe is what
// bounds the scatter: as one float4 cell a corner took 4 + 4 wavefronts at
// best where this takes 3 + 3 (5.47 -> 4.90 ms per 953 particles at 256^3;
// pitches 64 to 102 measured between 4.90 and 5.44).
//
// Map frequencies are formed in FP32 relative to the tile: per (tile,
// particle) pair an anchor pixel (hc, kc) near the tile's projection has its
// frequency hc ad + kc bd - o formed in FP64, and a point (h, k) adds
// (h - hc) af + (k - kc) bf to it.  The offsets are at most ~25 pixel steps
// at these tile sizes, so the coordinates carry < 5e-6 voxel of rounding;
// the trilinear weights are continuous in the coordinates, so a floor that
// lands on the other side of a cell boundary because of it moves a
// contribution by that much, and the phase lattices keep a margin above it
// (lattice.h).
// A corner's read-modify-write: the cell at byte address `at` + 8 OFF and its
// weight at `wt` + 4 OFF.  A corner outside the tile (on = false) is loaded all
// the same - its address lies within the guards around the arrays (GridSmem) -
// and not stored, so the eight corners are constant offsets from two registers
// (953 particles at 256^3: a branch per corner 6.53, a select of its address
// 5.47 ms with float4 cells; with split cells 256 particles took 1.63 with the
// select and take 1.56 ms so, with the tile tests read from 32-byte entries).
template <int OFF>
__device__ __forceinline__ void cell_add(unsigned at, unsigned wt, float2 f, float w, bool on) {
    float x, y, z;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(x), "=f"(y) : "r"(at), "n"(8 * OFF) : "memory");
    asm volatile("ld.shared.f32 %0, [%1+%2];" : "=f"(z) : "r"(wt), "n"(4 * OFF) : "memory");
    x = fmaf(f.x, w, x);
    y = fmaf(f.y, w, y);
    z += w;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t"
        "@p st.shared.v2.f32 [%0+%6], {%1, %2};\n\t@p st.shared.f32 [%3+%7], %4;\n\t}" ::"r"(at),
        "f"(x), "f"(y), "r"(wt), "f"(z), "r"((int)on), "n"(8 * OFF), "n"(4 * OFF)
        : "memory");
}

// Shared memory of a gridding warp: the queue of pairs, the cells, their
// weights and what the loads of corners outside the tile can reach.  The first
// corner of a pixel with a corner in the tile is cell FIRST .. LAST (coordinates
// -1 .. T - 1), and pixel4 limits it to that, so loads reach from cell FIRST to
// the eighth corner of cell LAST.
template <int TX, int TY, int TZ, int PX, int PP>
struct GridSmem {
    static constexpr int SLOTS = PP * TZ, CORNER = 1 + PX + PP;
    static constexpr int FIRST = -CORNER, LAST = (TX - 1) + PX * (TY - 1) + PP * (TZ - 1);
    static constexpr int PAST = LAST + CORNER + 1 > SLOTS ? LAST + CORNER + 1 - SLOTS : 0;
    static constexpr int round16(int n) { return (n + 15) & ~15; }
    static constexpr int larger(int m, int n) { return m > n ? m : n; }
    static constexpr int QUEUE = 32 * (int)sizeof(int4) + QN * (int)(sizeof(Pair) + sizeof(RowBounds) + sizeof(int));
    static constexpr int CELLS = round16(larger(QUEUE, 8 * CORNER));       // byte offset of the cells
    static constexpr int WEIGHTS = CELLS + round16(8 * SLOTS);             // byte offset of the weights
    static constexpr int BYTES = larger(WEIGHTS + 4 * (SLOTS + PAST), CELLS + 8 * (SLOTS + PAST));
    static_assert(WEIGHTS - 4 * CORNER >= 0, "loads before the first weight");
    static_assert(4 * SLOTS % 16 == 0, "cleared in 16-byte pieces");
    static_assert(sizeof(Pair) % 16 == 0 && sizeof(RowBounds) % 8 == 0, "alignment in the queue");
};

// the corners (0, y, z) and (1, y, z) at cell offset OFF
template <int OFF, int PX, int PP>
__device__ __forceinline__ void corner_row(unsigned at, unsigned wt, float2 f, float rx, float wyz, const bool* vx, bool on,
                                           unsigned lanes) {
    cell_add<OFF>(at, wt, f, (1.f - rx) * wyz, vx[0] && on);
    __syncwarp(lanes);
    cell_add<OFF + 1>(at, wt, f, rx * wyz, vx[1] && on);
    __syncwarp(lanes);
}

template <bool GATE, bool EW, int TX, int TY, int TZ, int PX, int PP>
__device__ __forceinline__ void pixel4(const InsertArgs& a, const DevParticle& P, const Pair& Q, unsigned cells,
                                       unsigned weights, float2 f, int h, int k, bool act) {
    float wt_ = Q.pw;
    if (GATE && act) {
        bool keep;
        const float tw = pixel_weight_gate(a, P, h, k, keep);
        if (!keep) act = false;
        wt_ *= tw;
    }
    const float dh = (float)(h - Q.hc), dk = (float)(k - Q.kc);
    float mx = fmaf(dh, Q.ax, fmaf(dk, Q.cx, Q.bx));
    float my = fmaf(dh, Q.ay, fmaf(dk, Q.cy, Q.by));
    float mz = fmaf(dh, Q.az, fmaf(dk, Q.cz, Q.bz));
    if (EW && P.ewh != 0.0) {
        // Ewald surface: s_z = +-(lambda/2) s2 along R[:,2] (Bimage_reconstruct.cpp:
        // 157-168), at most P.ezmax voxels, added in FP32 to the tile-relative
        // coordinate (the lattice keeps a margin for its variation)
        const double sx = h * P.inv, sy = k * P.inv, sz = P.ewh * (sx * sx + sy * sy);
        mx += (float)(sz * P.cd[0]);
        my += (float)(sz * P.cd[1]);
        mz += (float)(sz * P.cd[2]);
    }
    if (a.interp != 2) {
        const float fx = floorf(mx + 0.5f), fy = floorf(my + 0.5f), fz = floorf(mz + 0.5f);
        const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
        float w = wt_;
        if (a.interp == 1) {
            const float dx = mx - fx, dy = my - fy, dz = mz - fz;
            w = wt_ * (1.0f - sqrtf(dx * dx + dy * dy + dz * dz));
        }
        const bool on = act && (unsigned)ix < TX && (unsigned)iy < TY && (unsigned)iz < TZ && w > 0.f;
        const int i = on ? ix + PX * iy + PP * iz : 0;
        cell_add<0>(cells + 8 * i, weights + 4 * i, f, w, on);
        __syncwarp();
        return;
    }
    // only the lanes with a pixel (4 of 32 on average) go on: the others would
    // load too, and a load's two half warps cost a wavefront each
    const unsigned lanes = __ballot_sync(0xffffffffu, act);
    if (act) {
        const float flx = floorf(mx), fly = floorf(my), flz = floorf(mz);
        const int ix = (int)flx, iy = (int)fly, iz = (int)flz;
        const float rx = mx - flx, ry = my - fly, rz = mz - flz;
        const bool vx[2] = {(unsigned)ix < TX, (unsigned)(ix + 1) < TX};
        const bool vy[2] = {(unsigned)iy < TY, (unsigned)(iy + 1) < TY};
        const bool vz[2] = {(unsigned)iz < TZ, (unsigned)(iz + 1) < TZ};
        typedef GridSmem<TX, TY, TZ, PX, PP> Smem;
        const int cell = min(max(ix + PX * iy + PP * iz, Smem::FIRST), Smem::LAST);
        const unsigned at = cells + 8 * cell, wt = weights + 4 * cell;
        const float z0 = (1.f - rz) * wt_, z1 = rz * wt_;
        corner_row<0, PX, PP>(at, wt, f, rx, (1.f - ry) * z0, vx, vy[0] && vz[0], lanes);
        corner_row<PX, PX, PP>(at, wt, f, rx, ry * z0, vx, vy[1] && vz[0], lanes);
        corner_row<PP, PX, PP>(at, wt, f, rx, (1.f - ry) * z1, vx, vy[0] && vz[1], lanes);
        corner_row<PP + PX, PX, PP>(at, wt, f, rx, ry * z1, vx, vy[1] && vz[1], lanes);
    }
    __syncwarp();
}

// The pair's set-up by one lane: the pixels whose tents can reach the tile at
// alias origin (ox, oy, oz) lie in [h_lo, h_hi] x [k_lo, k_hi] (excl = 1
// leaves out the row k = -hf and the column h = -hf, which half-space gridding
// grids separately), or, for the edge walk, the two lines' ranges; the anchor
// is the tile centre's projection on the plane.  False: no pixel.
template <int TX, int TY, int TZ>
__device__ __noinline__ bool setup_pair(const DevParticle& P, int part, int hf, double ox, double oy, double oz,
                                           bool edge, int excl, Pair& Q, RowBounds& B) {
    if (edge) {
        edge_range<TX, TY, TZ>(P, hf, ox, oy, oz, 0, Q.h_lo, Q.h_hi);
        edge_range<TX, TY, TZ>(P, hf, ox, oy, oz, 1, Q.k_lo, Q.k_hi);
        if (Q.h_lo > Q.h_hi && Q.k_lo > Q.k_hi) return false;
    } else {
        const double e = P.ezmax;
        const double lo[3] = {ox - 1.0 - e, oy - 1.0 - e, oz - 1.0 - e};
        const double hi[3] = {ox + TX + e, oy + TY + e, oz + TZ + e};
        double vc = 0, hv = 0, uc = 0, hu = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double c = 0.5 * (lo[i] + hi[i]), e2 = 0.5 * (hi[i] - lo[i]);
            vc += P.bd[i] * c; hv += fabs(P.bd[i]) * e2;
            uc += P.ad[i] * c; hu += fabs(P.ad[i]) * e2;
        }
        vc *= P.inv_st2; hv *= P.inv_st2; uc *= P.inv_st2; hu *= P.inv_st2;
        Q.k_lo = max((int)ceil(vc - hv), -hf + excl);
        Q.k_hi = min((int)floor(vc + hv), hf - 1);
        Q.h_lo = max((int)ceil(uc - hu), -hf + excl);
        Q.h_hi = min((int)floor(uc + hu), hf - 1);
        if (Q.k_lo > Q.k_hi || Q.h_lo > Q.h_hi) return false;
    }
    const double cx = ox + 0.5 * (TX - 1), cy = oy + 0.5 * (TY - 1), cz = oz + 0.5 * (TZ - 1);
    Q.hc = (int)rint((P.ad[0] * cx + P.ad[1] * cy + P.ad[2] * cz) * P.inv_st2);
    Q.kc = (int)rint((P.bd[0] * cx + P.bd[1] * cy + P.bd[2] * cz) * P.inv_st2);
    Q.bx = (float)(Q.hc * P.ad[0] + Q.kc * P.bd[0] - ox);
    Q.by = (float)(Q.hc * P.ad[1] + Q.kc * P.bd[1] - oy);
    Q.bz = (float)(Q.hc * P.ad[2] + Q.kc * P.bd[2] - oz);
    Q.part = part;
    Q.lat = P.lat;
    Q.pw = P.pw;
    Q.inv_step = P.inv_step;
    Q.ax = P.af[0]; Q.ay = P.af[1]; Q.az = P.af[2];
    Q.cx = P.bf[0]; Q.cy = P.bf[1]; Q.cz = P.bf[2];
    Q.spec = P.spec;
    if (edge) return true;
    // Errors of -b ia + bound: b is off by its own rounding, the steps' and
    // the sum's (|b| < 64 voxels: < 1e-5), and each product and sum by 2^-24
    // of at most 64 |ia|; together < 3e-5 |ia|, and the integers' own sum.
    B.exact = 0;
    const int T[3] = {TX, TY, TZ};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float ia = (float)P.iad[i], err = 5e-5f * fabsf(ia) + 1e-5f;
        const float p0 = (-1.0f - P.ezmax) * ia, p1 = ((float)T[i] + P.ezmax) * ia;
        if (ia == 0.f) B.exact = 1;
        B.ia[i] = ia;
        B.lo_a[i] = fminf(p0, p1) - err;
        B.lo_b[i] = fminf(p0, p1) + err;
        B.hi_a[i] = fmaxf(p0, p1) - err;
        B.hi_b[i] = fmaxf(p0, p1) + err;
    }
    return true;
}

// Work items: R replicas of a tile, each on its slice of the particles, and
// with half-space gridding one more per tile below the split for the unpaired
// pixels (all particles).  The pairs that reach the tile are queued QN at a
// time, in (particle, alias) order, and set up by one lane each: the FP64
// set-up of a pair cost the warp ~850 instructions of the ~3,900 a pair
// takes when every lane did it.  One warp per CTA: the items' times differ, and
// in CTAs of four the early ones' shared memory waited for the last (11 of 20
// warps resident on average).
template <bool GATE, bool EW, int TX, int TY, int TZ, int PX, int PP>
__global__ void __launch_bounds__(32, 20) grid4_kernel(InsertArgs a) {
    constexpr int SLOTS = PP * TZ;
    constexpr int TV = TX * TY * TZ;
    typedef GridSmem<TX, TY, TZ, PX, PP> Smem;
    extern __shared__ __align__(16) unsigned char s_grid[];
    int4* const s_rows = reinterpret_cast<int4*>(s_grid);
    Pair* const s_pairs = reinterpret_cast<Pair*>(s_rows + 32);
    RowBounds* const s_bounds = reinterpret_cast<RowBounds*>(s_pairs + QN);
    int* const s_ids = reinterpret_cast<int*>(s_bounds + QN);
    float2* const s_sum = reinterpret_cast<float2*>(s_grid + Smem::CELLS);
    float* const s_wt = reinterpret_cast<float*>(s_grid + Smem::WEIGHTS);
    const int lane = threadIdx.x;
    const bool hs = a.zsplit > 0;
    // per tile: R items, and one for the unpaired pixels below the split (those
    // tiles come first)
    int slot, rep;
    if (hs && blockIdx.x < (unsigned)a.nlow * (a.R + 1)) {
        slot = blockIdx.x / (a.R + 1);
        rep = blockIdx.x - slot * (a.R + 1);
    } else {
        const unsigned b = blockIdx.x - (hs ? (unsigned)a.nlow * (a.R + 1) : 0u);
        slot = b / a.R;
        rep = b - slot * a.R;
        if (hs) slot += a.nlow;
    }
    const int tile = a.order[slot];
    const int x0 = (tile % a.ntx) * TX, y0 = ((tile / a.ntx) % a.nty) * TY, z0 = (tile / (a.ntx * a.nty)) * TZ;
    const int N = a.N;
    const int hf = a.ft / 2;
    const size_t spec_stride = (size_t)(2 * hf + 1) * a.pitch;
    const unsigned cells = (unsigned)__cvta_generic_to_shared(s_sum), weights = (unsigned)__cvta_generic_to_shared(s_wt);
    // half-space gridding (walk_edges): tiles at or above zsplit grid only
    // the unpaired pixels; those below it grid the others, and the extra item
    // the unpaired ones into evol / ew
    const bool upper = hs && z0 >= a.zsplit;
    const bool extra = rep == a.R;
    const bool edge_walk = extra || upper;
    // (a tile that no unpaired pixel reaches skips the edge walks)
    const bool none = edge_walk && !tile_reaches_edges<TX, TY, TZ>(x0, y0, z0, N, a.edge_rmin, a.edge_rmax);
    if (extra && none) return;
    const int p_lo = extra ? 0 : (int)((long)a.np * rep / a.R);
    const int p_hi = none ? p_lo : extra ? a.np : (int)((long)a.np * (rep + 1) / a.R);
    for (int i = lane; i < (Smem::WEIGHTS - Smem::CELLS + 4 * SLOTS) / 16; i += 32)
        reinterpret_cast<float4*>(s_grid + Smem::CELLS)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();

    bool any = false;                // some pair reached the tile
    const unsigned aliases = tile_aliases<TX, TY, TZ>(x0, y0, z0, N, a.rmax);
    TileTest ahead;                  // this lane's next test, on its way
    if (p_lo + lane < p_hi) ahead = a.test[p_lo + lane];
    int base = p_lo - 32, qn = 0;
    unsigned mask = 0;               // this lane's particle's aliases still to be queued
    for (;;) {
        const unsigned todo = __ballot_sync(0xffffffffu, mask != 0);
        if (todo) {
            const int cnt = __popc(mask);
            int off = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, off, o);
                if (lane >= o) off += v;
            }
            const int total = __shfl_sync(0xffffffffu, off, 31);
            for (int at = qn + off - cnt; mask && at < QN; ++at) {
                const int al = __ffs(mask) - 1;
                mask &= mask - 1;
                s_ids[at] = (base + lane) * 8 + al;
            }
            qn = min(QN, qn + total);
        } else {
            base += 32;
            if (base < p_hi) {
                const int p = base + lane;
                if (p < p_hi) {
                    const TileTest t = ahead;
                    if (p + 32 < p_hi) ahead = a.test[p + 32];
                    if (t.half == a.half || a.half < 0) mask = tile_mask<TX, TY, TZ>(t, aliases, x0, y0, z0, N);
                    if (edge_walk && mask) mask = edge_mask<TX, TY, TZ>(a.part[p], mask, x0, y0, z0, N, a.ft);
                }
                continue;
            }
            if (qn == 0) break;
        }
        if (qn < QN && base < p_hi) continue;
        __syncwarp();
        bool ok = false;
        if (lane < qn) {
            const int id = s_ids[lane], al = id & 7;
            ok = setup_pair<TX, TY, TZ>(a.part[id >> 3], id, hf, (double)(x0 - ((al & 1) ? N : 0)),
                                        (double)(y0 - ((al & 2) ? N : 0)), (double)(z0 - ((al & 4) ? N : 0)),
                                        edge_walk, hs ? 1 : 0, s_pairs[lane], s_bounds[lane]);
        }
        unsigned go = __ballot_sync(0xffffffffu, ok);
        __syncwarp();
        any = any || go;
        while (go) {
            const int at = __ffs(go) - 1;
            const Pair Q = s_pairs[at];
            go &= go - 1;
            const int al = Q.part & 7;
            const DevParticle& P = a.part[Q.part >> 3];
            const float2* S = a.spec + (size_t)Q.spec * spec_stride + (size_t)hf * a.pitch + hf;
            auto fetch = [&](int h, int k, bool act) {
                return act ? __ldg(S + (long)k * a.pitch + h) : make_float2(0.f, 0.f);
            };
            auto pix = [&](float2 f, int h, int k, bool act) {
                pixel4<GATE, EW, TX, TY, TZ, PX, PP>(a, P, Q, cells, weights, f, h, k, act);
            };
            if (edge_walk) walk_edges(Q, hf, lane, fetch, pix);
            else walk_groups<TX, TY, TZ>(P, Q, s_bounds[at], EW ? (double)P.ezmax : 0.0,
                                          (double)(x0 - ((al & 1) ? N : 0)), (double)(y0 - ((al & 2) ? N : 0)),
                                          (double)(z0 - ((al & 4) ? N : 0)), lane, s_rows, fetch, pix);
        }
        qn = 0;
        __syncwarp();
    }
    // tile sums -> HBM.  One replica (and the unpaired pixels' item) adds to
    // the map; of several, the one that arrives last adds the FP32 partial sums
    // in replica order: its own from shared memory, the others', which they
    // stored, while they are still in L2 (a separate pass over FP64 partial sums
    // took 0.86 ms of a 256^3 map's 14.9 ms and 0.93 ms per batch and half map
    // at 384^3).  Replicas that no pair reached store nothing.  Four voxels at a
    // time where the map's rows allow it: a voxel at a time left one warp
    // waiting for 16 trips to L2 and HBM in turn (0.29 of the 1.56 ms of 256
    // particles at 256^3; now 0.11 of 1.35).
    const bool sole = extra || a.R == 1;
    unsigned have = 0;               // whose partial sums there are
    float* const mine = a.psum + ((size_t)tile * a.R + rep) * 3 * TV;
    if (sole) {
        if (!any) return;
    } else {
        const unsigned self = any ? 256u << rep : 0u;
        unsigned old = 0;
        if (lane == 0) old = *(volatile unsigned*)&a.arrived[tile];
        old = __shfl_sync(0xffffffffu, old, 0);
        if ((int)(old & 255u) != a.R - 1) {            // the others are not all done
            if (any) {
#pragma unroll 2
                for (int i = 4 * lane; i < TV; i += 128) {
                    const int ci = i % TX + PX * ((i / TX) % TY) + PP * (i / (TX * TY));
                    const float2 c0 = s_sum[ci], c1 = s_sum[ci + 1], c2 = s_sum[ci + 2], c3 = s_sum[ci + 3];
                    *reinterpret_cast<float4*>(mine + i) = make_float4(c0.x, c1.x, c2.x, c3.x);
                    *reinterpret_cast<float4*>(mine + TV + i) = make_float4(c0.y, c1.y, c2.y, c3.y);
                    *reinterpret_cast<float4*>(mine + 2 * TV + i) = make_float4(s_wt[ci], s_wt[ci + 1], s_wt[ci + 2], s_wt[ci + 3]);
                }
                __threadfence();
            }
            __syncwarp();
            if (lane == 0) old = atomicAdd(&a.arrived[tile], 1u | self);
            old = __shfl_sync(0xffffffffu, old, 0);
            if ((int)(old & 255u) != a.R - 1) return;
        }
        have = (old | self) >> 8;
        if (lane == 0) a.arrived[tile] = 0;           // for the next launch
        if (!have) return;
        __threadfence();
    }
    const size_t N2 = (size_t)N * N;
    const float* const all = a.psum + (size_t)tile * a.R * 3 * TV;
    double2* const vol = extra ? a.evol : a.vol;
    double* const wgt = extra ? a.ew : a.w;
    if ((N & 3) == 0) {
#pragma unroll 1
        for (int i = 4 * lane; i < TV; i += 128) {
            const int lx = i % TX, ly = (i / TX) % TY, lz = i / (TX * TY);
            if (x0 + lx >= N || y0 + ly >= N || z0 + lz >= N) continue;
            const size_t idx = (size_t)(z0 + lz) * N2 + (size_t)(y0 + ly) * N + x0 + lx;
            const int ci = lx + PX * ly + PP * lz;
            double2* const wq = reinterpret_cast<double2*>(wgt + idx);
            double2 o[4] = {vol[idx], vol[idx + 1], vol[idx + 2], vol[idx + 3]}, w0 = wq[0], w1 = wq[1];
            if (sole) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    o[k].x += s_sum[ci + k].x;
                    o[k].y += s_sum[ci + k].y;
                }
                w0.x += s_wt[ci]; w0.y += s_wt[ci + 1];
                w1.x += s_wt[ci + 2]; w1.y += s_wt[ci + 3];
            } else {
                double re[4] = {}, im[4] = {}, w[4] = {};
#pragma unroll 2
                for (int r = 0; r < a.R; ++r) {
                    if (!((have >> r) & 1u)) continue;
                    float4 p, q, v;
                    if (r == rep) {
                        p = make_float4(s_sum[ci].x, s_sum[ci + 1].x, s_sum[ci + 2].x, s_sum[ci + 3].x);
                        q = make_float4(s_sum[ci].y, s_sum[ci + 1].y, s_sum[ci + 2].y, s_sum[ci + 3].y);
                        v = make_float4(s_wt[ci], s_wt[ci + 1], s_wt[ci + 2], s_wt[ci + 3]);
                    } else {
                        const float* src = all + (size_t)r * 3 * TV + i;
                        p = __ldcg(reinterpret_cast<const float4*>(src));
                        q = __ldcg(reinterpret_cast<const float4*>(src + TV));
                        v = __ldcg(reinterpret_cast<const float4*>(src + 2 * TV));
                    }
                    re[0] += p.x; re[1] += p.y; re[2] += p.z; re[3] += p.w;
                    im[0] += q.x; im[1] += q.y; im[2] += q.z; im[3] += q.w;
                    w[0] += v.x; w[1] += v.y; w[2] += v.z; w[3] += v.w;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) { o[k].x += re[k]; o[k].y += im[k]; }
                w0.x += w[0]; w0.y += w[1];
                w1.x += w[2]; w1.y += w[3];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) vol[idx + k] = o[k];
            wq[0] = w0;
            wq[1] = w1;
        }
        return;
    }
#pragma unroll 1
    for (int i = lane; i < TV; i += 32) {
        const int lx = i % TX, ly = (i / TX) % TY, lz = i / (TX * TY);
        if (x0 + lx >= N || y0 + ly >= N || z0 + lz >= N) continue;
        const size_t idx = (size_t)(z0 + lz) * N2 + (size_t)(y0 + ly) * N + x0 + lx;
        const int ci = lx + PX * ly + PP * lz;
        double re = 0, im = 0, w = 0;
        if (sole) {
            re = s_sum[ci].x;
            im = s_sum[ci].y;
            w = s_wt[ci];
        } else {
            for (int r = 0; r < a.R; ++r) {
                if (!((have >> r) & 1u)) continue;
                const float* q = all + (size_t)r * 3 * TV + i;
                re += r == rep ? s_sum[ci].x : __ldcg(q);
                im += r == rep ? s_sum[ci].y : __ldcg(q + TV);
                w += r == rep ? s_wt[ci] : __ldcg(q + 2 * TV);
            }
        }
        double2 o = vol[idx];
        o.x += re;
        o.y += im;
        vol[idx] = o;
        wgt[idx] += w;
    }
}

// FOM path: map += sum over replicas, in replica order.
__global__ void combine_kernel(InsertArgs a) {
    const size_t N3 = (size_t)a.N * a.N * a.N;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N3; i += (size_t)gridDim.x * blockDim.x) {
        double re = 0, im = 0, w = 0, p = 0, q = 0;
        for (int r = 0; r < a.R; ++r) {
            const double* pb = a.fsum + (size_t)r * 5 * N3 + i;
            re += pb[0]; im += pb[N3]; w += pb[2 * N3];
            p += pb[3 * N3]; q += pb[4 * N3];
        }
        double2 o = a.vol[i];
        o.x += re; o.y += im;
        a.vol[i] = o;
        a.w[i] += w;
        a.pow[i] += p; a.w2[i] += q;
    }
}

// Tile shapes the autotuner chooses from (map voxels per warp).  The cell
// pitches (PX, PP) of each shape are the template
// arguments of its grid4_kernel launch below.
struct Shape { int tx, ty, tz; };
static const Shape kShapes[] = {{8, 8, 8}, {16, 16, 4}, {16, 8, 8}, {16, 16, 8}};
constexpr int kNumShapes = 4;

int insert_num_shapes() { return kNumShapes; }
void insert_shape(int i, int* tx, int* ty, int* tz) { *tx = kShapes[i].tx; *ty = kShapes[i].ty; *tz = kShapes[i].tz; }

template <int TX, int TY, int TZ>
static cudaError_t set_smem_shape() {
    const int smem = (int)(WARPS * 5 * TX * TY * TZ * sizeof(tacc_t));
    cudaError_t e = cudaFuncSetAttribute(insert_kernel<true, TX, TY, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(insert_kernel<false, TX, TY, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

template <int TX, int TY, int TZ, int PX, int PP>
static cudaError_t set_smem_shape4() {
    const int smem = GridSmem<TX, TY, TZ, PX, PP>::BYTES;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(grid4_kernel<true, false, TX, TY, TZ, PX, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(grid4_kernel<false, false, TX, TY, TZ, PX, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(grid4_kernel<true, true, TX, TY, TZ, PX, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    return cudaFuncSetAttribute(grid4_kernel<false, true, TX, TY, TZ, PX, PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

cudaError_t prepare_insert_attributes() {
    cudaError_t e;
    if ((e = set_smem_shape4<8, 8, 8, 8, 67>()) != cudaSuccess) return e;
    if ((e = set_smem_shape4<16, 16, 4, 17, 277>()) != cudaSuccess) return e;
    if ((e = set_smem_shape4<16, 8, 8, 16, 134>()) != cudaSuccess) return e;
    if ((e = set_smem_shape4<16, 16, 8, 16, 262>()) != cudaSuccess) return e;
    if ((e = set_smem_shape<8, 8, 8>()) != cudaSuccess) return e;
    if ((e = set_smem_shape<16, 16, 4>()) != cudaSuccess) return e;
    return set_smem_shape<16, 8, 8>();
}

template <int TX, int TY, int TZ>
static cudaError_t launch_shape(const InsertArgs& a0, const Context& c, cudaStream_t s) {
    InsertArgs a = a0;
    const int N = c.g.map;
    a.ntx = (N + TX - 1) / TX;
    a.nty = (N + TY - 1) / TY;
    a.ntz = (N + TZ - 1) / TZ;
    const int ntiles = a.ntx * a.nty * a.ntz;
    const unsigned blocks = (unsigned)(((long)ntiles * a.R + WARPS - 1) / WARPS);
    const size_t smem = (size_t)WARPS * 5 * TX * TY * TZ * sizeof(tacc_t);
    if (c.g.gate) insert_kernel<true, TX, TY, TZ><<<blocks, WARPS * 32, smem, s>>>(a);
    else insert_kernel<false, TX, TY, TZ><<<blocks, WARPS * 32, smem, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || a.R == 1) return e;
    combine_kernel<<<148 * 8, 256, 0, s>>>(a);
    return cudaGetLastError();
}

template <int TX, int TY, int TZ, int PX, int PP>
static cudaError_t launch_shape4(const InsertArgs& a0, const Context& c, cudaStream_t s) {
    InsertArgs a = a0;
    const int N = c.g.map;
    a.ntx = (N + TX - 1) / TX;
    a.nty = (N + TY - 1) / TY;
    a.ntz = (N + TZ - 1) / TZ;
    const int ntiles = a.ntx * a.nty * a.ntz;
    a.nlow = a.zsplit > 0 ? a.ntx * a.nty * ((a.zsplit + TZ - 1) / TZ) : 0;
    const long items = (long)ntiles * a.R + a.nlow;
    const size_t smem = GridSmem<TX, TY, TZ, PX, PP>::BYTES;
    if (c.g.ewald) {
        if (c.g.gate) grid4_kernel<true, true, TX, TY, TZ, PX, PP><<<(unsigned)items, 32, smem, s>>>(a);
        else grid4_kernel<false, true, TX, TY, TZ, PX, PP><<<(unsigned)items, 32, smem, s>>>(a);
    } else {
        if (c.g.gate) grid4_kernel<true, false, TX, TY, TZ, PX, PP><<<(unsigned)items, 32, smem, s>>>(a);
        else grid4_kernel<false, false, TX, TY, TZ, PX, PP><<<(unsigned)items, 32, smem, s>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_insert(const Context& c, const float2* spectra, const DevParticle* parts, const TileTest* tests,
                          int np, int half, cudaStream_t s) {
    InsertArgs a;
    a.spec = spectra;
    a.part = parts;
    a.test = tests;
    a.np = np;
    a.half = half;
    a.N = c.g.map;
    a.ft = c.g.ft;
    a.pitch = c.g.ft + 2;
    a.interp = c.g.interp;
    a.maxs2 = c.g.maxs2;
    a.mins2 = c.g.mins2;
    a.mscale = c.g.mscale;
    const int h = half < 0 ? 0 : half;
    a.vol = c.d_vol[h];
    a.w = c.d_w[h];
    a.pow = c.d_pow[h];
    a.w2 = c.d_w2[h];
    a.order = c.d_tile_order;
    a.R = c.replicas;
    a.psum = reinterpret_cast<float*>(c.d_part_sums);
    a.fsum = reinterpret_cast<double*>(c.d_part_sums);
    a.arrived = c.d_arrived;
    a.zsplit = c.g.fom ? 0 : c.zsplit;
    a.evol = c.d_evol[h];
    a.ew = c.d_ew[h];
    a.edge_rmin = (float)c.edge_rmin;
    a.edge_rmax = (float)c.edge_rmax;
    a.rmax = c.rmax;
    if (!c.g.fom) {
        switch (c.shape) {
            case 0: return launch_shape4<8, 8, 8, 8, 67>(a, c, s);
            case 2: return launch_shape4<16, 8, 8, 16, 134>(a, c, s);
            case 3: return launch_shape4<16, 16, 8, 16, 262>(a, c, s);
            default: return launch_shape4<16, 16, 4, 17, 277>(a, c, s);
        }
    }
    switch (c.shape) {
        case 0: return launch_shape<8, 8, 8>(a, c, s);
        case 2: return launch_shape<16, 8, 8>(a, c, s);
        default: return launch_shape<16, 16, 4>(a, c, s);
    }
}

}  // namespace bsg

// lattice.cu - the phase lattices of a batch's gridding records (lattice.h) and
// their tile-test entries, one warp per record: the lanes test 32 candidates at a time, in
// choose_lattice's order, and the first safe one is the record's.  On the host
// the search took 0.5 to 0.7 us a record before the batch's first kernel could
// start (1.1 of 2.7 ms for 2,000 particles of 64^2); here 12 us for all.  (A batch
// of a few particles stays on the host: capi.cu, upload_params.)
#include "context.cuh"
#include "lattice.h"

namespace bsg {

__global__ void __launch_bounds__(128) lattice_kernel(DevParticle* part, TileTest* tests, long n,
                                                       double mscale, int ft) {
    const long r = blockIdx.x * 4L + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    DevParticle& P = part[r];
    // bound on the Ewald surface's extra displacement per pixel step
    // (make_dev_particle)
    double curve = lat_mul(lat_mul(lat_mul(fabs(P.ewh), P.inv2), mscale), (double)ft);
    curve = lat_mul(lat_mul(curve, 1.4142135623730951), 1.0001);
    const double ad[3] = {P.ad[0], P.ad[1], P.ad[2]}, bd[3] = {P.bd[0], P.bd[1], P.bd[2]};
    const double reach = lattice_reach(ad, bd, curve);
    PhaseLattice best = square_lattice(reach);
    if (reach < 64.0)
        for (int c0 = 0; c0 < LATTICE_CANDIDATES; c0 += 32) {
            const PhaseLattice l = lattice_candidate(c0 + lane);
            const bool ok = l.lh > 0 && lattice_ok(ad, bd, l.lh, l.lk, l.sh, reach, curve);
            const unsigned some = __ballot_sync(0xffffffffu, ok);
            if (!some) continue;
            const int src = __ffs(some) - 1;
            best = {__shfl_sync(0xffffffffu, l.lh, src), __shfl_sync(0xffffffffu, l.lk, src),
                    __shfl_sync(0xffffffffu, l.sh, src)};
            break;
        }
    if (lane == 0) {
        P.lat = pack_lattice(best);
        tests[r] = tile_test(P, ft);
    }
}

cudaError_t launch_lattices(const Context& c, DevParticle* parts, TileTest* tests, long n, cudaStream_t s) {
    lattice_kernel<<<(unsigned)((n + 3) / 4), 128, 0, s>>>(parts, tests, n, c.g.mscale, c.g.ft);
    return cudaGetLastError();
}

}  // namespace bsg

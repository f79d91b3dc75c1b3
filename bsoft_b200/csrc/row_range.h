// row_range.h - the pixels of a gridding row from its FP32 bounds (insert.cu,
// walk_groups; plain C++ on the host, where tests/row_range_check.cpp runs it).
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define BSG_ROW_FN __host__ __device__ inline
#else
#define BSG_ROW_FN inline
#endif

namespace bsg {

struct RowRange {
    int lo, hi;       // pixels lo .. hi (none: hi < lo)
    bool sure;        // the exact bounds give these integers too
};

BSG_ROW_FN int row_ceil(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_ru(x);
#else
    return (int)ceilf(x);
#endif
}
BSG_ROW_FN int row_floor(float x) {
#ifdef __CUDA_ARCH__
    return __float2int_rd(x);
#else
    return (int)floorf(x);
#endif
}

// The row's pixels within [h_lo, h_hi], their exact bounds relative to pixel hc
// lying between lo_a and lo_b below and hi_a and hi_b above.  A view a hair off
// an axis (a step of 1e-9 voxels) has bounds beyond any integer: they are cut
// at 1e9 on both sides, so that the sum with hc cannot wrap round and a row
// outside the tile stays empty.
BSG_ROW_FN RowRange row_range(int hc, int h_lo, int h_hi, float lo_a, float lo_b, float hi_a, float hi_b) {
    const float far = 1e9f;
    lo_a = fminf(fmaxf(lo_a, -far), far);
    lo_b = fminf(fmaxf(lo_b, -far), far);
    hi_a = fminf(fmaxf(hi_a, -far), far);
    hi_b = fminf(fmaxf(hi_b, -far), far);
    const int l0 = hc + row_ceil(lo_a), l1 = hc + row_ceil(lo_b), h0 = hc + row_floor(hi_a), h1 = hc + row_floor(hi_b);
    RowRange r;
    r.lo = l0 > h_lo ? l0 : h_lo;
    r.hi = h1 < h_hi ? h1 : h_hi;
    r.sure = r.lo > r.hi || (r.lo == (l1 > h_lo ? l1 : h_lo) && r.hi == (h0 < h_hi ? h0 : h_hi));
    return r;
}

}  // namespace bsg

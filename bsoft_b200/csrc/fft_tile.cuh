// fft_tile.cuh - transforms of a tile of 16 or 8 lines by one CTA, for the 3-D map
// transform.
//
// The tile sits in shared memory as [element][line], so the 16 lines of an
// element are adjacent: a half warp runs one butterfly of 16 lines, its loads
// and stores fall in distinct banks and its twiddles are one broadcast.
// Mixed-radix Stockham autosort (natural order in and out) with the radices
// compiled in: each butterfly is R loads, an R-point transform in registers
// and R stores, so an edge of 384 = 8 8 6 takes three round trips through
// shared memory.
#pragma once

#include <cuda_runtime.h>

namespace bsg {

constexpr int TILE_LINES = 16;
constexpr int MAX_STAGES = 12;

struct TilePlan {
    int n;                       // transform length
    int nstage;
    int radix[MAX_STAGES];
    int ns[MAX_STAGES];          // product of the radices before the stage
    int magic[MAX_STAGES];       // j / ns = j magic >> 20 for j <= 512
};

// Radices 8, 6, 4, 2, 7, 5, 3 of n (a product of 2, 3, 5 and 7, at most 512):
// as few stages as this greedy split gives.  False for other lengths.
inline bool tile_plan(int n, TilePlan* p) {
    p->n = n;
    p->nstage = 0;
    int two = 0, three = 0, m = n;
    while (m % 2 == 0) { m /= 2; ++two; }
    while (m % 3 == 0) { m /= 3; ++three; }
    int r[MAX_STAGES], ns = 0;
    auto put = [&](int v) { if (ns < MAX_STAGES) r[ns] = v; ++ns; };
    while (m % 7 == 0) { m /= 7; put(7); }
    while (m % 5 == 0) { m /= 5; put(5); }
    if (m != 1) return false;
    // a left-over factor of 2 or 4 pairs with 3s as 6
    while (three > 0 && two % 3 == 1) { put(6); --three; --two; }
    while (three > 1 && two % 3 == 2) { put(6); put(6); three -= 2; two -= 2; }
    while (three-- > 0) put(3);
    while (two >= 3 && two != 4) { put(8); two -= 3; }
    while (two >= 2) { put(4); two -= 2; }
    if (two) put(2);
    if (ns > MAX_STAGES) return false;
    int prod = 1;
    for (int i = 0; i < ns; ++i) {
        p->radix[i] = r[i];
        p->ns[i] = prod;
        p->magic[i] = ((1 << 20) + prod - 1) / prod;
        prod *= r[i];
    }
    p->nstage = ns;
    return prod == n;
}

__device__ __forceinline__ float2 tadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 tsub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 tmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a times -i (forward) or i (inverse)
template <bool INV>
__device__ __forceinline__ float2 trot(float2 a) { return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x); }

template <bool INV>
__device__ __forceinline__ void dft2(float2& a, float2& b) {
    const float2 t = tsub(a, b);
    a = tadd(a, b);
    b = t;
}

template <bool INV>
__device__ __forceinline__ void dft3(float2& a, float2& b, float2& c) {
    const float s = 0.8660254037844386f;
    const float2 t = tadd(b, c), d = trot<INV>(tsub(b, c));
    const float2 m = make_float2(a.x - 0.5f * t.x, a.y - 0.5f * t.y);
    a = tadd(a, t);
    b = make_float2(m.x + s * d.x, m.y + s * d.y);
    c = make_float2(m.x - s * d.x, m.y - s * d.y);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& a, float2& b, float2& c, float2& d) {
    const float2 s0 = tadd(a, c), s1 = tsub(a, c), s2 = tadd(b, d), s3 = trot<INV>(tsub(b, d));
    a = tadd(s0, s2);
    b = tadd(s1, s3);
    c = tsub(s0, s2);
    d = tsub(s1, s3);
}

// odd R by pairs: cos / sin of 2 pi k / R, k = 1 .. (R - 1) / 2
template <int R, bool INV>
__device__ __forceinline__ void dft_odd(float2* v, const float* cs, const float* sn) {
    constexpr int H = (R - 1) / 2;
    float2 s[H], d[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
        s[j] = tadd(v[1 + j], v[R - 1 - j]);
        d[j] = trot<INV>(tsub(v[1 + j], v[R - 1 - j]));
    }
    float2 e[H], o[H];
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 a = v[0], b = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            const int m = (j * k) % R, q = m <= H ? m : R - m;
            const float c = cs[q - 1], t = m <= H ? sn[q - 1] : -sn[q - 1];
            a.x += c * s[j - 1].x;
            a.y += c * s[j - 1].y;
            b.x += t * d[j - 1].x;
            b.y += t * d[j - 1].y;
        }
        e[k - 1] = a;
        o[k - 1] = b;
    }
    float2 t = v[0];
#pragma unroll
    for (int j = 0; j < H; ++j) t = tadd(t, s[j]);
    v[0] = t;
#pragma unroll
    for (int k = 0; k < H; ++k) {
        v[1 + k] = tadd(e[k], o[k]);
        v[R - 1 - k] = tsub(e[k], o[k]);
    }
}

// R-point transform in registers, natural order in and out
template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
    if (R == 2) dft2<INV>(v[0], v[1]);
    if (R == 3) dft3<INV>(v[0], v[1], v[2]);
    if (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
    if (R == 5) {
        const float c[2] = {0.30901699437494745f, -0.8090169943749475f};
        const float s[2] = {0.9510565162951535f, 0.5877852522924731f};
        dft_odd<R == 5 ? 5 : 3, INV>(v, c, s);
    }
    if (R == 7) {
        const float c[3] = {0.6234898018587336f, -0.2225209339563144f, -0.9009688679024191f};
        const float s[3] = {0.7818314824680298f, 0.9749279121818236f, 0.4338837391175581f};
        dft_odd<R == 7 ? 7 : 3, INV>(v, c, s);
    }
    if (R == 6) {
        // 2 x 3 by the Chinese remainder theorem: no twiddles
        float2 a0 = v[0], a1 = v[2], a2 = v[4], b0 = v[3], b1 = v[5], b2 = v[1];
        dft3<INV>(a0, a1, a2);
        dft3<INV>(b0, b1, b2);
        v[0] = tadd(a0, b0);
        v[3] = tsub(a0, b0);
        v[4] = tadd(a1, b1);
        v[1] = tsub(a1, b1);
        v[2] = tadd(a2, b2);
        v[5] = tsub(a2, b2);
    }
    if (R == 8) {
        const float h = 0.7071067811865476f;
        dft4<INV>(v[0], v[2], v[4], v[6]);
        dft4<INV>(v[1], v[3], v[5], v[7]);
        // odd half times exp(-+ 2 pi i k / 8)
        const float2 t1 = INV ? make_float2(h * (v[3].x - v[3].y), h * (v[3].x + v[3].y))
                              : make_float2(h * (v[3].x + v[3].y), h * (v[3].y - v[3].x));
        const float2 t2 = trot<INV>(v[5]);
        const float2 t3 = INV ? make_float2(h * (-v[7].x - v[7].y), h * (v[7].x - v[7].y))
                              : make_float2(h * (v[7].y - v[7].x), h * (-v[7].x - v[7].y));
        const float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
        v[0] = tadd(e0, o0);
        v[4] = tsub(e0, o0);
        v[1] = tadd(e1, t1);
        v[5] = tsub(e1, t1);
        v[2] = tadd(e2, t2);
        v[6] = tsub(e2, t2);
        v[3] = tadd(e3, t3);
        v[7] = tsub(e3, t3);
    }
}

template <int R, bool INV, int LINES>
__device__ __forceinline__ void tile_stage(const float2* src, float2* dst, int n, int ns, int magic,
                                           const float2* roots, int rstride, int pitch) {
    const int nr = n / R, tstep = n / (ns * R) * rstride;
    for (int i = threadIdx.x; i < nr * LINES; i += blockDim.x) {
        const int c = i & (LINES - 1), j = i / LINES;
        const int q = (j * magic) >> 20, k = j - q * ns;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[(j + r * nr) * pitch + c];
        if (k) {
#pragma unroll
            for (int r = 1; r < R; ++r) {
                float2 w = roots[r * k * tstep];
                if (INV) w.y = -w.y;
                v[r] = tmul(v[r], w);
            }
        }
        dft<R, INV>(v);
        const int base = q * ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) dst[(base + r * ns) * pitch + c] = v[r];
    }
}

// Transform the tile in a (p.n x LINES, element pitch `pitch`) with b as the
// other buffer; all threads of the CTA, which have synchronised after filling
// a.  roots: exp(-2 pi i t / (p.n rstride)), t < p.n rstride, in shared
// memory.  Returns the buffer holding the result (synchronised).
template <bool INV, int LINES = TILE_LINES>
__device__ __forceinline__ float2* tile_fft(float2* a, float2* b, const TilePlan& p, const float2* roots, int rstride,
                                            int pitch) {
    for (int s = 0; s < p.nstage; ++s) {
        const int ns = p.ns[s], mg = p.magic[s];
        switch (p.radix[s]) {
            case 2: tile_stage<2, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            case 3: tile_stage<3, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            case 4: tile_stage<4, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            case 5: tile_stage<5, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            case 6: tile_stage<6, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            case 7: tile_stage<7, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
            default: tile_stage<8, INV, LINES>(a, b, p.n, ns, mg, roots, rstride, pitch); break;
        }
        __syncthreads();
        float2* t = a;
        a = b;
        b = t;
    }
    return a;
}

}  // namespace bsg

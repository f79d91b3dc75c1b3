// fft2d.cu - the 2-D half of particle_reconstruct on the GPU: background,
// padding, forward FFT (1/ft scale), origin phase shift and CTF, for a batch
// of particles.  Reference steps (bsoft/src):
//   calculate_background  img/Bimage_background.cpp:27-80
//   pad(ft, FILL_BACKGROUND)  img/Bimage_resize.cpp:28-110, 347-357
//   fft(plan, 1)          img/Bimage_fft.cpp:176-234
//   phase_shift_to_origin img/Bimage_complex.cpp:490-534
//   img_ctf_apply_complex mg/mg_ctf.cpp:661-676 with img_ctf_calculate :46-122
//
// Three kernels per batch:
//   background_kernel  one CTA per image: background mean (FP64 sum) and the
//                      separable phase-shift tables exp(i h shx), exp(i k shy)
//                      evaluated in double;
//   rows_kernel        pairs of image rows: the pair is packed as one complex
//                      line (row a + i row b), padded with the background,
//                      transformed, and split into the two real-input half
//                      spectra (h = 0..ft/2);
//   cols_kernel        16 columns per CTA: column transforms of the row
//                      spectra (rows >= n are the constant background rows,
//                      whose transform is ft*bkg at h = 0 and 0 elsewhere),
//                      then the fused epilogue 1/ft * shift * CTF, written for
//                      pixel (h, k) and its mate (-h, -k) (conjugate symmetry
//                      of a real image's transform), i.e. the full ft x ft
//                      spectrum, stored centred and padded as
//                      [k + ft/2][h + ft/2] with row pitch ft + 2 and ft + 1
//                      rows (the extra row/columns stay zero).
//
// Each thread holds 16 elements of a line in registers and runs up to four
// radix-2 stages on them (the stages and products of an in-place
// decimation-in-time transform of bit-reversed input, so the results are those
// bit for bit); the line changes hands through shared memory once (up to 256
// elements) or twice.  Lines in shared memory with a round trip per two stages
// took 3.59 (columns) and 0.99 ms (rows) per 2,000 particles of 256^2 at ft
// 512, bound by those trips; now 1.81 and 0.65.
#include "context.cuh"
#include "fft_dev.cuh"

#include <math.h>

namespace bsg {

// ------------------------------------------------------------------ background
__global__ void background_kernel(const float* __restrict__ img, const DevParticle* __restrict__ part,
                                  int n, int ft, double* __restrict__ bkg, float2* __restrict__ phase) {
    const int b = blockIdx.x;
    const float* im = img + (size_t)b * n * n;
    const DevParticle& P = part[b];
    const int hn = n / 2;
    const double h = (double)hn;
    // dividing by a power of two is multiplying by its exact reciprocal:
    // the same doubles without the division sequence
    const bool pow2 = (hn & (hn - 1)) == 0;
    const double ih = 1.0 / h;
    double sum = 0.0;
    int cnt = 0;
    // pixel i = y n + x, stepped by blockDim.x without a division per pixel
    int y = threadIdx.x / n, x = threadIdx.x - y * n;
    const int dy = blockDim.x / n, dx = blockDim.x - dy * n;
    // eight pixels' loads in flight at a time (one at a time, behind its test,
    // the pass took 0.97 ms per 2,000 images of 256^2: now 0.38)
    constexpr int AHEAD = 8;
    const double bx = P.bx, by = P.by, na = P.na, nb = P.nb;
    for (int i0 = threadIdx.x; i0 < n * n; i0 += AHEAD * blockDim.x) {
        float v[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int i = i0 + u * blockDim.x;
            v[u] = i < n * n ? im[i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            double x2, y2;
            if (pow2) { x2 = (x - bx) * ih; y2 = (y - by) * ih; }
            else { x2 = (x - bx) / h; y2 = (y - by) / h; }
            if (i0 + u * (int)blockDim.x < n * n && x2 * x2 + y2 * y2 - 1 > 0) {
                sum += (float)(v[u] * na + nb);
                ++cnt;
            }
            x += dx;
            y += dy;
            if (x >= n) { x -= n; ++y; }
        }
    }
    // deterministic block reduction (fixed tree)
    __shared__ double ssum[256];
    __shared__ int scnt[256];
    ssum[threadIdx.x] = sum;
    scnt[threadIdx.x] = cnt;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            ssum[threadIdx.x] += ssum[threadIdx.x + o];
            scnt[threadIdx.x] += scnt[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) bkg[b] = scnt[0] ? ssum[0] / scnt[0] : 0.0;
    // separable origin shift factors, phi = h*shx + k*shy (double)
    float2* ex = phase + (size_t)b * 2 * ft;
    float2* ey = ex + ft;
    for (int i = threadIdx.x; i < ft; i += blockDim.x) {
        double f = (double)sfreq(i, ft);
        double s, c;
        sincos(f * P.shx, &s, &c);
        ex[i] = make_float2((float)c, (float)s);
        sincos(f * P.shy, &s, &c);
        ey[i] = make_float2((float)c, (float)s);
    }
}

// ------------------------------------------------------------------ lines
constexpr int E = 16;            // elements of a line per thread

// two radix-2 stages on (a0, a1, a2, a3), the inputs at distance half, 2 half
// and 3 half: w1 the first stage's twiddle, w2a / w2b the second's
__device__ __forceinline__ void radix4(float2& a0, float2& a1, float2& a2, float2& a3, float2 w1, float2 w2a,
                                       float2 w2b) {
    const float2 t1 = cmul(a1, w1), t3 = cmul(a3, w1);
    const float2 b0 = make_float2(a0.x + t1.x, a0.y + t1.y);
    const float2 b1 = make_float2(a0.x - t1.x, a0.y - t1.y);
    const float2 b2 = make_float2(a2.x + t3.x, a2.y + t3.y);
    const float2 b3 = make_float2(a2.x - t3.x, a2.y - t3.y);
    const float2 u2 = cmul(b2, w2a), u3 = cmul(b3, w2b);
    a0 = make_float2(b0.x + u2.x, b0.y + u2.y);
    a2 = make_float2(b0.x - u2.x, b0.y - u2.y);
    a1 = make_float2(b1.x + u3.x, b1.y + u3.y);
    a3 = make_float2(b1.x - u3.x, b1.y - u3.y);
}

__device__ __forceinline__ void radix2(float2& a0, float2& a1, float2 w) {
    const float2 u = a0, t = cmul(a1, w);
    a0 = make_float2(u.x + t.x, u.y + t.y);
    a1 = make_float2(u.x - t.x, u.y - t.y);
}

// Stages FIRST + 1 .. FIRST + M of a line of 2^LOG elements on the group
// v[0 .. 2^M), elements at distance 2^FIRST from position j + (a multiple of
// 2^(FIRST + M)); stages in pairs, a last one alone.  tw: the line's ft / 2
// twiddles, stored swizzled.
template <int LOG, int FIRST, int M>
__device__ __forceinline__ void group_stages(float2* v, int j, const float2* tw) {
    constexpr int L = 1 << LOG, G = 1 << M;
#pragma unroll
    for (int m = 0; m < M; m += 2) {
        const int s = FIRST + m + 1;                  // the stage
        const int d = 1 << m;                         // its distance within the group
        if (m + 1 < M) {
#pragma unroll
            for (int q = 0; q < G / 4; ++q) {
                const int lo = q & (d - 1), i = ((q - lo) << 2) + lo;
                const int jj = j + (lo << FIRST);     // position within the half-group of stage s
                radix4(v[i], v[i + d], v[i + 2 * d], v[i + 3 * d], tw[swz(jj * (L >> s))], tw[swz(jj * (L >> (s + 1)))],
                       tw[swz((jj + (1 << (s - 1))) * (L >> (s + 1)))]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < G / 2; ++q) {
                const int lo = q & (d - 1), i = ((q - lo) << 1) + lo;
                radix2(v[i], v[i + d], tw[swz((j + (lo << FIRST)) * (L >> s))]);
            }
        }
    }
}

// A line of 2^LOG elements by 2^LOG / 16 threads (t: this one's number).  On
// entry v[q] is the input element line_input<LOG>(t, q); `put(i, v)` and
// `get(i)` exchange through shared memory around `sync()`.  On return v[q] is
// output element line_output<LOG>(t, q).
template <int LOG>
__device__ __forceinline__ int line_input(int t, int q) {
    return (int)(__brev((unsigned)q) >> 28 << (LOG - 4)) + (LOG > 4 ? (int)(__brev((unsigned)t) >> (36 - LOG)) : 0);
}

// elements held after the second (LOG <= 8) or third phase
template <int LOG>
__device__ __forceinline__ int line_output(int t, int q) {
    constexpr int T = 1 << (LOG - 4);
    if constexpr (LOG <= 8) {
        constexpr int U = E / T;                      // groups of T elements per thread
        return t * U + q / T + 16 * (q % T);
    } else {
        constexpr int R = 1 << (LOG - 8);             // group of the third phase
        return t + T * (q / R) + 256 * (q % R);
    }
}

template <int LOG, class Put, class Get, class Sync>
__device__ __forceinline__ void line_fft(float2* v, int t, const float2* tw, Put&& put, Get&& get, Sync&& sync) {
    group_stages<LOG, 0, 4>(v, 0, tw);
#pragma unroll
    for (int q = 0; q < E; ++q) put(16 * t + q, v[q]);
    sync();
    if constexpr (LOG <= 8) {
        constexpr int M = LOG - 4, G = 1 << M, U = E / G;
#pragma unroll
        for (int q = 0; q < E; ++q) v[q] = get(line_output<LOG>(t, q));
#pragma unroll
        for (int u = 0; u < U; ++u) group_stages<LOG, 4, M>(v + u * G, t * U + u, tw);
    } else {
        const int j = t & 15, b = 256 * (t >> 4) + j;
#pragma unroll
        for (int q = 0; q < E; ++q) v[q] = get(b + 16 * q);
        group_stages<LOG, 4, 4>(v, j, tw);
        sync();
#pragma unroll
        for (int q = 0; q < E; ++q) put(b + 16 * q, v[q]);
        sync();
        constexpr int T = 1 << (LOG - 4), M = LOG - 8, R = 1 << M;
#pragma unroll
        for (int q = 0; q < E; ++q) v[q] = get(line_output<LOG>(t, q));
#pragma unroll
        for (int u = 0; u < E / R; ++u) group_stages<LOG, 8, M>(v + u * R, t + T * u, tw);
    }
}

// ------------------------------------------------------------------ rows
// (a box of 32 has 16 pairs: 64 threads at ft 64, where 256 left three quarters
// idle; 500 particles 13.2 -> 7.3 us)
template <int LOG>
constexpr int ROW_THREADS = LOG <= 6 ? 64 : 256;

// ROW_THREADS / T row pairs per CTA, T = ft / 16 threads each; at most 32 KB of lines.
template <int LOG>
__global__ void __launch_bounds__(ROW_THREADS<LOG>)
rows_kernel(const float* __restrict__ img, const double* __restrict__ bkg, const float2* __restrict__ tw,
            const DevParticle* __restrict__ part, int n, float2* __restrict__ rows) {
    constexpr int ft = 1 << LOG, T = ft / E, THREADS = ROW_THREADS<LOG>, LINES = THREADS / T;
    __shared__ float2 stw[ft / 2];
    __shared__ float2 lines[LINES * ft];
    for (int i = threadIdx.x; i < ft / 2; i += THREADS) stw[swz(i)] = tw[i];
    __syncthreads();
    const int b = blockIdx.y, t = threadIdx.x % T;
    const int pair = blockIdx.x * LINES + threadIdx.x / T;
    const bool live = pair < (n + 1) / 2;
    float2* buf = lines + (threadIdx.x / T) * ft;
    const int y0 = 2 * pair, y1 = y0 + 1;
    const float fill = (float)bkg[b];
    const float* r0 = img + ((size_t)b * n + y0) * n;
    const float* r1 = r0 + n;
    // the particle's normalisation (rescale_to_avg_std, stored as float)
    const double na = part[b].na, nb = part[b].nb;
    float2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int x = line_input<LOG>(t, q);
        v[q].x = (live && x < n) ? (float)(r0[x] * na + nb) : fill;
        v[q].y = (live && y1 < n && x < n) ? (float)(r1[x] * na + nb) : fill;
    }
    line_fft<LOG>(v, t, stw, [&](int i, float2 a) { buf[swz(i)] = a; }, [&](int i) { return buf[swz(i)]; },
                  [] { __syncthreads(); });
    __syncthreads();
#pragma unroll
    for (int q = 0; q < E; ++q) buf[swz(line_output<LOG>(t, q))] = v[q];
    __syncthreads();
    if (!live) return;
    constexpr int hw = ft / 2 + 1;
    float2* o0 = rows + ((size_t)b * n + y0) * hw;
    float2* o1 = o0 + hw;
#pragma unroll
    for (int q = 0; q <= E / 2; ++q) {
        const int h = t + T * q;
        if (h >= hw) break;
        float2 z = buf[swz(h)], zm = buf[swz((ft - h) & (ft - 1))];
        o0[h] = make_float2(0.5f * (z.x + zm.x), 0.5f * (z.y - zm.y));
        if (y1 < n) o1[h] = make_float2(0.5f * (z.y + zm.y), -0.5f * (z.x - zm.x));
    }
}

// ------------------------------------------------------------------ columns + epilogue
constexpr int COL_W = 16;   // columns per CTA

struct ColArgs {
    const float2* rows;
    const double* bkg;
    const float2* phase;
    const DevParticle* part;
    const float2* tw;
    float2* spec;
    int n;
    int ctf_action;
    double wiener;
    double shi2;
};

// The particle's CTF terms, held in registers for the epilogue: read through
// the record in global memory they would be loaded again after every store
// of the spectrum (the compiler cannot tell that the stores leave them alone).
struct CtfTerms {
    double fs, c00, c20, c22, c2m2, c40, c11, c1m1;
};

__device__ __forceinline__ CtfTerms ctf_terms(const DevParticle& P) {
    CtfTerms t;
    t.fs = P.fs; t.c00 = P.c00; t.c20 = P.c20; t.c22 = P.c22; t.c2m2 = P.c2m2; t.c40 = P.c40;
    t.c11 = P.c11; t.c1m1 = P.c1m1;
    return t;
}

// CTF weight of one pixel from its reduced even aberration r in (-pi, pi].
__device__ __forceinline__ float ctf_weight(const ColArgs& a, double r) {
    if (a.ctf_action == 1) return (r < 0.0) ? -1.f : 1.f;
    float w = sinf((float)r);
    if (a.wiener != 0.0) w = (float)((a.wiener + 1.0) * w / ((double)w * w + a.wiener));
    return w;
}

// CTF factor of pixel (h, k) without the odd aberrations: img_ctf_calculate:
// s = (h, k) * fs, inside [0, shi2]; even aberration chi = c00 + s2 (c20 + c22
// cos2a + c2m2 sin2a) + c40 s2^2 with s2 cos2a = sx^2 - sy^2, s2 sin2a = 2 sx
// sy (ctf.h:321-334), in double.  The same for (-h, -k).
__device__ __forceinline__ float even_ctf(const ColArgs& a, const CtfTerms& P, double sx, double sy) {
    const double s2 = sx * sx + sy * sy;
    if (!(s2 <= a.shi2)) return 0.f;
    const double even = P.c00 + P.c20 * s2 + P.c22 * (sx * sx - sy * sy) + P.c40 * s2 * s2;
    const double chi = even + P.c2m2 * (2.0 * sx * sy);
    // reduce to (-pi, pi] in double so the sign of sin(chi) is exact
    return ctf_weight(a, chi - 6.283185307179586 * rint(chi * 0.15915494309189535));
}

// The epilogue's products, each rounding written out, so that a pixel's value
// does not depend on which product the compiler contracts: the phase factor
// ex ey, its mate conj(ex) ey, and the value times the factor.
__device__ __forceinline__ float2 phase_of(float2 ex, float2 ey) {
    return make_float2(__fmaf_rn(ex.x, ey.x, -__fmul_rn(ex.y, ey.y)), __fmaf_rn(ex.y, ey.x, __fmul_rn(ex.x, ey.y)));
}
__device__ __forceinline__ float2 mate_phase_of(float2 ex, float2 ey) {
    return make_float2(__fmaf_rn(ey.x, ex.x, __fmul_rn(ey.y, ex.y)), __fmaf_rn(-ey.x, ex.y, __fmul_rn(ey.y, ex.x)));
}
__device__ __forceinline__ float2 value_times(float2 g, float2 f) {
    return make_float2(__fmaf_rn(g.x, f.x, -__fmul_rn(g.y, f.y)), __fmaf_rn(g.x, f.y, __fmul_rn(g.y, f.x)));
}

// Factor 1/ft * phase * CTF of a pixel from its phase factor, even CTF factor
// and frequency (the odd, beam-tilt aberration is psi = c1m1 sy + c11 sx).
__device__ __forceinline__ float2 pixel_factor(const ColArgs& a, const CtfTerms& P, float sc, float2 ph, float w,
                                               double sx, double sy) {
    float2 f = make_float2(ph.x * sc, ph.y * sc);
    if (!a.ctf_action) return f;
    if (w == 0.f) return make_float2(0.f, 0.f);
    f.x *= w;
    f.y *= w;
    if (P.c11 != 0.0 || P.c1m1 != 0.0) {
        float sp, cp;
        sincosf((float)(P.c1m1 * sy + P.c11 * sx), &sp, &cp);
        f = cmulc(f, make_float2(cp, sp));
    }
    return f;
}

// 16 adjacent columns per CTA, ft / 16 threads each, a column's elements 16
// apart in shared memory so that the columns of one element are adjacent.
// A thread's outputs are 16 pixels (h, k) of one column: it writes each and
// its mate (-h, -k) = conj, whose even CTF factor is the same, so the FP64
// aberration is evaluated once for the two.  Four pixels of the epilogue at a
// time: with all 16 unrolled a launch waited for the instructions to arrive, 21 us
// for the smallest, now 10 (500 particles of ft 512 480 -> 452 us, of ft 64 23 ->
// 14; two at a time 458 and 15, one 474 and 15).
template <int LOG>
__global__ void __launch_bounds__(COL_W * (1 << (LOG - 4)), LOG <= 9 ? 1024 / (COL_W * (1 << (LOG - 4))) : 1)
cols_kernel(ColArgs a) {
    constexpr int ft = 1 << LOG, T = ft / E, THREADS = COL_W * T, hw = ft / 2 + 1, hf = ft / 2;
    extern __shared__ float2 smem[];
    float2* stw = smem;                          // ft / 2 twiddles
    float2* sey = smem + ft / 2;                 // exp(i k shy)
    float2* buf = sey + ft;                      // ft x COL_W
    const int b = blockIdx.y, c = threadIdx.x % COL_W, t = threadIdx.x / COL_W;
    const int hidx = blockIdx.x * COL_W + c;
    const float2* ex = a.phase + (size_t)b * 2 * ft;
    for (int i = threadIdx.x; i < ft / 2; i += THREADS) stw[swz(i)] = a.tw[i];
    for (int i = threadIdx.x; i < ft; i += THREADS) sey[i] = ex[ft + i];
    const float dc = (float)(a.bkg[b] * ft);
    const float2* rows = a.rows + (size_t)b * a.n * hw + hidx;
    float2 v[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        const int y = line_input<LOG>(t, q);
        v[q] = make_float2(0.f, 0.f);
        if (hidx < hw) {
            if (y < a.n) v[q] = rows[(size_t)y * hw];
            else if (hidx == 0) v[q] = make_float2(dc, 0.f);
        }
    }
    __syncthreads();
    line_fft<LOG>(v, t, stw, [&](int i, float2 z) { buf[i * COL_W + c] = z; },
                  [&](int i) { return buf[i * COL_W + c]; }, [] { __syncthreads(); });
    if (hidx >= hw) return;
    const CtfTerms P = ctf_terms(a.part[b]);
    // centred, padded layout: [k + ft/2][h + ft/2], row pitch ft + 2
    constexpr int pitch = ft + 2;
    float2* out = a.spec + (size_t)b * (ft + 1) * pitch + (size_t)hf * pitch + hf;
    const float sc = 1.0f / (float)ft;
    const int h = sfreq(hidx, ft);               // hidx == ft/2 -> -ft/2
    const bool mate = hidx >= 1 && hidx < hf;
    const float2 exh = ex[hidx];
    const double sx = (double)h * P.fs;
    // (back to the places in shared memory that this thread read last, so that
    // the loop below need not be unrolled)
#pragma unroll
    for (int q = 0; q < E; ++q) buf[line_output<LOG>(t, q) * COL_W + c] = v[q];
#pragma unroll 4
    for (int q = 0; q < E; ++q) {
        const int kk = line_output<LOG>(t, q), k = sfreq(kk, ft);
        const float2 g = buf[kk * COL_W + c];
        const double sy = (double)k * P.fs;
        const float w = a.ctf_action ? even_ctf(a, P, sx, sy) : 0.f;
        out[(long)k * pitch + h] = value_times(g, pixel_factor(a, P, sc, phase_of(exh, sey[kk]), w, sx, sy));
        if (mate) {
            // F(-h, -k) = conj(G(h, k)) * factor(-h, -k); -(-ft/2) is -ft/2
            const int km = (ft - kk) & (ft - 1), k2 = sfreq(km, ft);
            const double sy2 = (double)k2 * P.fs;
            const float w2 = k2 == -k || !a.ctf_action ? w : even_ctf(a, P, -sx, sy2);
            out[(long)k2 * pitch - h] = value_times(
                make_float2(g.x, -g.y), pixel_factor(a, P, sc, mate_phase_of(exh, sey[km]), w2, -sx, sy2));
        }
    }
}

cudaError_t launch_background(const Context& c, const float* img, int nimg, cudaStream_t s) {
    background_kernel<<<nimg, 256, 0, s>>>(img, c.d_part, c.g.n, c.g.ft, c.d_bkg, c.d_phase);
    return cudaGetLastError();
}

// f.operator()<LOG>() for the transform's log2 (bsg_recon_create admits 32 .. 1024)
template <class F>
static cudaError_t for_log(int log, F&& f) {
    switch (log) {
        case 5: return f.template operator()<5>();
        case 6: return f.template operator()<6>();
        case 7: return f.template operator()<7>();
        case 8: return f.template operator()<8>();
        case 9: return f.template operator()<9>();
        case 10: return f.template operator()<10>();
        default: return cudaErrorInvalidValue;
    }
}

struct RowsLaunch {
    const Context& c;
    const float* img;
    int nimg;
    cudaStream_t s;
    template <int LOG>
    cudaError_t operator()() const {
        constexpr int LINES = ROW_THREADS<LOG> / ((1 << LOG) / E);
        const int npairs = (c.g.n + 1) / 2;
        const dim3 grid((npairs + LINES - 1) / LINES, nimg);
        rows_kernel<LOG><<<grid, ROW_THREADS<LOG>, 0, s>>>(img, c.d_bkg, c.d_tw, c.d_part, c.g.n, c.d_rows);
        return cudaGetLastError();
    }
};

cudaError_t launch_rows(const Context& c, const float* img, int nimg, cudaStream_t s) {
    return for_log(c.g.logft, RowsLaunch{c, img, nimg, s});
}

template <int LOG>
static constexpr size_t cols_smem() {
    return sizeof(float2) * ((1 << LOG) / 2 + (1 << LOG) + (size_t)COL_W * (1 << LOG));
}

struct ColsLaunch {
    const Context& c;
    const ColArgs& a;
    int nimg;
    cudaStream_t s;
    template <int LOG>
    cudaError_t operator()() const {
        constexpr int hw = (1 << LOG) / 2 + 1;
        const dim3 grid((hw + COL_W - 1) / COL_W, nimg);
        cols_kernel<LOG><<<grid, COL_W * ((1 << LOG) / E), cols_smem<LOG>(), s>>>(a);
        return cudaGetLastError();
    }
};

cudaError_t launch_cols(const Context& c, int nimg, float2* spectra, cudaStream_t s) {
    ColArgs a;
    a.rows = c.d_rows; a.bkg = c.d_bkg; a.phase = c.d_phase; a.part = c.d_part; a.tw = c.d_tw;
    a.spec = spectra; a.n = c.g.n;
    a.ctf_action = c.g.ctf_action; a.wiener = c.g.wiener; a.shi2 = c.g.ctf_shi2;
    return for_log(c.g.logft, ColsLaunch{c, a, nimg, s});
}

struct ColsAttribute {
    template <int LOG>
    cudaError_t operator()() const {
        return cudaFuncSetAttribute(cols_kernel<LOG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cols_smem<LOG>());
    }
};

cudaError_t prepare_fft2d_attributes() {
    for (int log = 5; log <= 10; ++log) {
        const cudaError_t e = for_log(log, ColsAttribute{});
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace bsg

// cnn.cu - the learned orientation proposer: a small convolutional network
// that maps a particle image to a rotation (6-D representation, made
// orthonormal by Gram-Schmidt) and an in-plane shift, trained on the GPU by
// the kernels below.  It has no counterpart in the reference; it proposes
// poses for a local search whose scores are the reference's figure of merit.
//
// Network (activations NHWC, FP32; weights kept as FP32 masters and used
// rounded to BF16, products accumulated in FP32):
//   input  box x box x 1, normalised to zero mean and unit variance per image
//   6 x    3x3 convolution, stride 2, padding 1, bias, ReLU
//   fc1    (box/64)^2 * C6 -> hidden, ReLU
//   fc2    hidden -> 8 = a1(3), a2(3), shift(2)
//   head   b1 = a1/|a1|, b2 = normalised a2 - (b1.a2) b1, b3 = b1 x b2;
//          R = [b1 b2 b3] (columns), t = shift (pixels)
//   loss   mean over the batch of |R - R*|_F^2 + lambda |t - t*|^2
//
// Convolutions are implicit GEMMs on the tensor cores (BF16 mma.sync with the
// operands split into two BF16 terms, FP32 accumulation): the operand rows
// are fetched from the activation planes as a tap needs them, in the forward
// pass, the input gradient and the weight gradient (over pixel ranges whose
// partial sums are added in order).  Every reduction has a fixed order, so
// training is bitwise reproducible for a given seed.
#include "common.cuh"

#include <cuda_bf16.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <random>
#include <vector>

namespace bsg {

namespace {

constexpr int NCONV = 6;
constexpr int NOUT = 8;     // a1, a2, shift
constexpr int NRES = 11;    // R (9, row-major) and shift (2)

using bf16 = __nv_bfloat16;

// ---- operands ---------------------------------------------------------------
//
// Every value that enters a product is held as two BF16 terms, hi = bf16(v)
// and lo = bf16(v - hi), in two planes; a product adds hi hi, hi lo and lo hi
// (the lo x lo term is below 2^-16 of it), so it keeps ~17 significant bits.
// The weights are BF16 values already: their lo terms are zero and left out.
// The planes are written by the kernel that produces the value (32 bits a
// value, as the float would take), so no consumer splits again, and they are
// NHWC with the channels padded to a multiple of 32 (zeros), so every operand
// row is copied in aligned 16-byte pieces.
constexpr int CPAD = 32;
__host__ __device__ constexpr int cpad(int c) { return (c + CPAD - 1) / CPAD * CPAD; }

__device__ __forceinline__ void mma_bf16(float* c, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// 16 bytes global -> shared, zeros when !ok
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void split_bf16(float v, bf16& hi, bf16& lo) {
    hi = __float2bfloat16_rn(v);
    lo = __float2bfloat16_rn(v - __bfloat162float(hi));
}
__device__ __forceinline__ uint32_t pack2(bf16 a, bf16 b) {
    return (uint32_t)__bfloat16_as_ushort(a) | ((uint32_t)__bfloat16_as_ushort(b) << 16);
}
__device__ __forceinline__ void split2(float v0, float v1, uint32_t& hi, uint32_t& lo) {
    bf16 h0, h1, l0, l1;
    split_bf16(v0, h0, l0);
    split_bf16(v1, h1, l1);
    hi = pack2(h0, h1);
    lo = pack2(l0, l1);
}

// ---- convolution as an implicit GEMM ----------------------------------------
//
// C[m][n] = sum over taps and channels of A(m, tap, c) W(n, tap, c): row m is
// an output pixel (b, y, x), A its input pixel (stride y + dy, stride x + dx)
// of the tap (zero outside the image), fetched straight from the activation
// planes by cp.async, so no column matrix is written.  The forward pass is
// stride 2 with nine taps; the input gradient is one GEMM per parity class
// of the input pixel (stride 1 over the output gradient, 4, 2, 2 and 1 taps,
// blockIdx.z the class); a dense layer is one tap on a 1 x 1 image.
// The epilogue adds the bias and applies the ReLU (forward) or the ReLU's
// mask (gradient) and writes the two planes of the result.
//
// Column matrices and separate bias, ReLU and mask passes bounded this path
// before (a K-deep FP32 copy of every input pixel: 302 MB for the second
// layer of 256 images of 128^2, written, read and split again); a layer now
// reads its input about 9 / 4 times through L2 and writes its output once.
// 2,048 images of 128^2: 14.5 -> 1.66 ms, the same bits; loss and gradient of
// 256 images 11.3 -> 2.1 ms, of which 1.0 ms is the host copies.  Block tile BM x BN with K-steps of 32 in a 4-deep ring, 8 warps of
// 32 rows.  mma.sync keeps the accumulation order of every product sum (k in
// steps of 16; hi, then lo), so results do not depend on the tile.
// Column j of a warp's n-tile t is channel 2 NT (j / 2) + 2 t + (j & 1): a
// lane's accumulators are then 2 NT consecutive channels of its row and
// leave in 16-byte stores.
struct ConvClass {
    int ntap;
    signed char dy[9], dx[9], w[9];   // input offset and weight slice of each tap
    int oy, ox;                       // output pixel = ostride (y, x) + (oy, ox)
};

struct ConvArgs {
    const bf16 *ah, *al;              // input planes, pitch C
    const bf16* w;                    // weights: n wrow + slice wtap + c
    long wrow, wtap;
    int M, N, logw, logh;             // rows: m = (b, y, x), 2^logh x 2^logw per image
    int H, W, C, stride;              // input image
    bf16 *oh, *ol;                    // output planes, pitch N
    int OH, OW, ostride;
    const float* bias;                // or null
    int nbias;
    int relu;
    const bf16* mask;                 // output kept where mask > 0 (laid out as the output), or null
    ConvClass cls[4];
};

constexpr int CBK = 32, CST = 4;

template <int BM, int BN>
constexpr int conv_smem() { return CST * (2 * BM + BN) * CBK * 2; }

template <int BM, int BN>
__global__ void __launch_bounds__(256) conv_gemm_kernel(const __grid_constant__ ConvArgs a) {
    constexpr int WMS = BM / 32, WNS = 8 / WMS, WN = BN / WNS, NT = WN / 8;
    constexpr int LOGR = NT == 8 ? 4 : NT == 4 ? 3 : 2;            // log2(2 NT)
    static_assert(NT == 2 || NT == 4 || NT == 8, "warp tile");
    constexpr int APL = BM * CBK * 2, STAGE = 2 * APL + BN * CBK * 2;
    extern __shared__ __align__(128) unsigned char csm[];
    const uint32_t base = smem_addr(csm);
    const ConvClass& k = a.cls[blockIdx.z];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int wm = (warp / WNS) * 32, wn = (warp % WNS) * WN;

    // this thread's copies: 16-byte piece ch of rows r0 + 64 i
    const int ch = tid & 3, r0 = tid >> 2;
    constexpr int AR = (BM + 63) / 64, BR = (BN + 63) / 64;
    int iy[AR], ix[AR];
    long ib[AR];
    bool iv[AR];
#pragma unroll
    for (int i = 0; i < AR; ++i) {
        const int r = r0 + 64 * i, m = m0 + r;
        iv[i] = r < BM && m < a.M;
        const int x = m & ((1 << a.logw) - 1), y = (m >> a.logw) & ((1 << a.logh) - 1), b = m >> (a.logw + a.logh);
        iy[i] = y * a.stride;
        ix[i] = x * a.stride;
        ib[i] = (long)b * a.H * a.W;
    }
    const int kch = a.C / CBK, T = k.ntap * kch;
    auto load = [&](int it) {
        const int tap = it / kch, c0 = (it - tap * kch) * CBK + ch * 8;
        const uint32_t st = base + (it % CST) * STAGE;
        const int dy = k.dy[tap], dx = k.dx[tap];
#pragma unroll
        for (int i = 0; i < AR; ++i) {
            const int r = r0 + 64 * i;
            if (BM >= 64 || r < BM) {
                const int yy = iy[i] + dy, xx = ix[i] + dx;
                const bool ok = iv[i] && (unsigned)yy < (unsigned)a.H && (unsigned)xx < (unsigned)a.W;
                const long off = ok ? (ib[i] + (long)yy * a.W + xx) * a.C + c0 : 0;
                const uint32_t d = st + r * 64 + ((ch ^ ((r >> 1) & 3)) << 4);
                cp16(d, a.ah + off, ok);
                cp16(d + APL, a.al + off, ok);
            }
        }
#pragma unroll
        for (int i = 0; i < BR; ++i) {
            const int r = r0 + 64 * i;
            if (BN >= 64 || r < BN)
                cp16(st + 2 * APL + r * 64 + ((ch ^ ((r >> LOGR) & 3)) << 4),
                     a.w + (n0 + r) * a.wrow + k.w[tap] * a.wtap + c0, true);
        }
    };

    float acc[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;

#pragma unroll
    for (int s = 0; s < CST - 1; ++s) {
        if (s < T) load(s);
        cp_commit();
    }
    for (int it = 0; it < T; ++it) {
        cp_wait<CST - 2>();
        __syncthreads();
        if (it + CST - 1 < T) load(it + CST - 1);
        cp_commit();
        const uint32_t st = base + (it % CST) * STAGE;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            uint32_t ah[2][4], al[2][4], b[NT][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int r = wm + mt * 16 + (lane & 15), c = kk * 2 + (lane >> 4);
                const uint32_t ad = st + r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
                ldsm4(ah[mt], ad);
                ldsm4(al[mt], ad + APL);
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2) {
                const int q = lane >> 3, j = lane & 7;
                const int r = wn + 2 * NT * (j >> 1) + 2 * (nt + (q >> 1)) + (j & 1), c = kk * 2 + (q & 1);
                ldsm4(b[nt], st + 2 * APL + r * 64 + ((c ^ ((r >> LOGR) & 3)) << 4));
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    mma_bf16(acc[mt][nt], ah[mt], b[nt]);
                    mma_bf16(acc[mt][nt], al[mt], b[nt]);
                }
        }
    }
    cp_wait<0>();

    const int g = lane >> 2, t = lane & 3;
    const int nc = n0 + wn + 2 * NT * t;                      // this lane's first channel
    float bias[2 * NT];
#pragma unroll
    for (int j = 0; j < 2 * NT; ++j) bias[j] = a.bias && nc + j < a.nbias ? a.bias[nc + j] : 0.f;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int m = m0 + wm + mt * 16 + hr * 8 + g;
            if (m >= a.M) continue;
            const int x = m & ((1 << a.logw) - 1), y = (m >> a.logw) & ((1 << a.logh) - 1), bb = m >> (a.logw + a.logh);
            const long o = (((long)bb * a.OH + y * a.ostride + k.oy) * a.OW + x * a.ostride + k.ox) * a.N + nc;
            uint32_t h[NT], l[NT], mk[NT];
            if (a.mask) {
#pragma unroll
                for (int j = 0; j < NT; j += 2) {
                    const uint2 v = *reinterpret_cast<const uint2*>(a.mask + o + 2 * j);
                    mk[j] = v.x;
                    mk[j + 1] = v.y;
                }
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                float v0 = acc[mt][j][2 * hr] + bias[2 * j], v1 = acc[mt][j][2 * hr + 1] + bias[2 * j + 1];
                if (a.relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
                if (a.mask) {
                    // BF16 terms of a ReLU output: positive or zero
                    if (!(mk[j] & 0xffffu)) v0 = 0.f;
                    if (!(mk[j] >> 16)) v1 = 0.f;
                }
                split2(v0, v1, h[j], l[j]);
            }
#pragma unroll
            for (int j = 0; j < NT; j += 4) {
                if (NT >= 4) {
                    *reinterpret_cast<uint4*>(a.oh + o + 2 * j) = make_uint4(h[j], h[j + 1], h[j + 2], h[j + 3]);
                    *reinterpret_cast<uint4*>(a.ol + o + 2 * j) = make_uint4(l[j], l[j + 1], l[j + 2], l[j + 3]);
                } else {
                    *reinterpret_cast<uint2*>(a.oh + o) = make_uint2(h[0], h[1]);
                    *reinterpret_cast<uint2*>(a.ol + o) = make_uint2(l[0], l[1]);
                }
            }
        }
}

// ---- first convolution: one input channel -----------------------------------

// per image: mean and 1 / population standard deviation (FP64 sums in a
// fixed order); idx: the images of the batch within the data set, or null
__global__ void __launch_bounds__(256) image_norm_kernel(const float* __restrict__ data, const int* __restrict__ idx,
                                                         int npix, float2* __restrict__ norm) {
    __shared__ double s1[256], s2[256];
    const long src = idx ? idx[blockIdx.x] : blockIdx.x;
    const float* p = data + src * (long)npix;
    double a = 0, b = 0;
    for (int i = threadIdx.x; i < npix; i += 256) { const double v = p[i]; a += v; b += v * v; }
    s1[threadIdx.x] = a;
    s2[threadIdx.x] = b;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if (threadIdx.x < o) { s1[threadIdx.x] += s1[threadIdx.x + o]; s2[threadIdx.x] += s2[threadIdx.x + o]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double mean = s1[0] / npix;
        const double var = s2[0] / npix - mean * mean;
        norm[blockIdx.x] = make_float2((float)mean, var > 1e-30 ? (float)(1.0 / sqrt(var)) : 1.f);
    }
}

// A CTA's patch of the normalised image: output pixels [p0, p0 + 256) of the
// wo x wo grid and their 3 x 3 input pixels, row pitch 2 wo + 4, column 0
// holding x = -1 (zeros outside the image).  Rows of wo are split when wo
// exceeds 256 (never: wo <= 256).
constexpr int C1PIX = 256;
__device__ __forceinline__ int c1_rows(int wo) { return 2 * (C1PIX / wo) + 1; }
__device__ __forceinline__ int c1_pitch(int wo) { return 2 * wo + 4; }

__device__ __forceinline__ void c1_load(float* patch, const float* img, float2 nm, int wo, int y0) {
    const int rows = c1_rows(wo), pitch = c1_pitch(wo), w = 2 * wo;
    for (int i = threadIdx.x; i < rows * pitch; i += blockDim.x) {
        const int r = i / pitch, x = i - r * pitch - 1, y = 2 * y0 - 1 + r;
        float v = 0.f;
        if (y >= 0 && y < w && x >= 0 && x < w) v = (img[(long)y * w + x] - nm.x) * nm.y;
        patch[i] = v;
    }
}

// input value of output pixel p (relative to the CTA's first) at tap (ky, kx)
__device__ __forceinline__ float c1_tap(const float* patch, int pitch, int logw, int p, int tap) {
    const int y = p >> logw, x = p & ((1 << logw) - 1);
    const int ky = tap / 3, kx = tap - 3 * ky;
    return patch[(2 * y + ky) * pitch + 2 * x + kx];
}

// 256 output pixels of one image per CTA; the nine taps are one K-step of 16
// whose A fragments are built from the patch in registers.  Bound by its
// output (two BF16 planes).  w: [cout padded][16] BF16, blockIdx.y the block
// of 32 channels.
__global__ void __launch_bounds__(256) conv1_kernel(const float* __restrict__ data, const int* __restrict__ idx,
                                                    const float2* __restrict__ norm, int logw,
                                                    const bf16* __restrict__ w, const float* __restrict__ bias,
                                                    int nbias, int pitch_out, bf16* __restrict__ oh,
                                                    bf16* __restrict__ ol) {
    extern __shared__ float patch[];
    const int wo = 1 << logw, pitch = c1_pitch(wo);
    const int perimg = (wo * wo) / C1PIX;
    const int b = blockIdx.x / perimg, p0 = (blockIdx.x - b * perimg) * C1PIX;
    const long src = idx ? idx[b] : b;
    c1_load(patch, data + src * (4L << (2 * logw)), norm[b], wo, p0 >> logw);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.y * 32;
    // weight fragments: column j of n-tile q is channel 8 (j / 2) + 2 q + (j & 1)
    uint32_t bw[4][2];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t* r = reinterpret_cast<const uint32_t*>(w + (n0 + 8 * (g >> 1) + 2 * q + (g & 1)) * 16);
        bw[q][0] = r[t];
        bw[q][1] = r[t + 4];
    }
    float bs[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) bs[j] = n0 + 8 * t + j < nbias ? bias[n0 + 8 * t + j] : 0.f;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        const int pr = warp * 32 + mt * 16 + g;
        uint32_t ah[4], al[4];
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int p = pr + 8 * hr;
            split2(c1_tap(patch, pitch, logw, p, 2 * t), c1_tap(patch, pitch, logw, p, 2 * t + 1), ah[hr], al[hr]);
            split2(t == 0 ? c1_tap(patch, pitch, logw, p, 8) : 0.f, 0.f, ah[2 + hr], al[2 + hr]);
        }
        float acc[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[q][e] = 0.f;
            mma_bf16(acc[q], ah, bw[q]);
            mma_bf16(acc[q], al, bw[q]);
        }
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const long o = (((long)b << (2 * logw)) + p0 + pr + 8 * hr) * pitch_out + n0 + 8 * t;
            uint32_t h[4], l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                split2(fmaxf(acc[q][2 * hr] + bs[2 * q], 0.f), fmaxf(acc[q][2 * hr + 1] + bs[2 * q + 1], 0.f), h[q], l[q]);
            *reinterpret_cast<uint4*>(oh + o) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(ol + o) = make_uint4(l[0], l[1], l[2], l[3]);
        }
    }
}

// ---- weight gradients ---------------------------------------------------------
//
// dW[n][tap][c] = sum over output pixels of gY(pixel, n) X(pixel's input at
// tap, c): a GEMM over the pixels whose operands are rows of the planes
// (fragments by ldmatrix.trans), one tap per CTA.  Three products per step
// (both operands are split).  The pixels are divided over blockIdx.z ranges
// whose partial sums are added in a fixed order afterwards; the bias gradient
// (the column sums of gY) is one more product with a fragment of ones, in the
// CTAs of the centre tap.
struct WgradArgs {
    const bf16 *yh, *yl;              // gY planes: pixels x N
    const bf16 *xh, *xl;              // X planes, pitch C
    int M, N, C, logw, logh, H, W, stride, ntap;
    int steps, per;                   // K-steps of 32 pixels, steps per range
    float* part;                      // ranges x (N x ntap x C), then ranges x N bias sums
    float* bpart;
};

constexpr int GST = 3;

template <int BN>
constexpr int wgrad_smem() { return GST * 32 * (64 + BN) * 2 * 2; }

// 16-byte piece c of row r in a tile of rows of RB bytes
template <int RB>
__device__ __forceinline__ int tswz(int r, int c) {
    return r * RB + ((RB == 128 ? c ^ (r & 7) : c ^ ((r >> 1) & 3)) << 4);
}

// grid: x = tap, y = (block of 64 of N) + (blocks of N) (block of BN of C), z = range
template <int BN>
__global__ void __launch_bounds__(128) wgrad_kernel(const __grid_constant__ WgradArgs a) {
    constexpr int NT = BN / 16;                          // n-tiles per warp (2 x 2 warps)
    constexpr int YB = 128, XB = BN * 2;                 // row bytes
    constexpr int YPL = 32 * YB, XPL = 32 * XB, STAGE = 2 * (YPL + XPL);
    extern __shared__ __align__(128) unsigned char gsm[];
    const uint32_t base = smem_addr(gsm);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tap = blockIdx.x, nb = (a.N + 63) / 64;
    const int n0 = (blockIdx.y % nb) * 64, c0 = (blockIdx.y / nb) * BN;
    const int dy = a.ntap == 9 ? tap / 3 - 1 : 0, dx = a.ntap == 9 ? tap % 3 - 1 : 0;
    const int s0 = blockIdx.z * a.per, s1 = min(a.steps, s0 + a.per);
    const bool dobias = tap == a.ntap / 2 && c0 == 0;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * (BN / 2);
    auto load = [&](int s, int slot) {
        const uint32_t st = base + slot * STAGE;
#pragma unroll
        for (int i = 0; i < 2; ++i) {                    // gY: 32 rows x 8 pieces
            const int e = tid + 128 * i, r = e >> 3, c = e & 7, m = s * 32 + r;
            const bool ok = m < a.M && n0 + c * 8 < a.N;
            const long off = ok ? (long)m * a.N + n0 + c * 8 : 0;
            cp16(st + tswz<YB>(r, c), a.yh + off, ok);
            cp16(st + YPL + tswz<YB>(r, c), a.yl + off, ok);
        }
#pragma unroll
        for (int i = 0; i < BN / 32; ++i) {              // X: 32 rows x BN / 8 pieces
            const int e = tid + 128 * i, r = e / (BN / 8), c = e % (BN / 8), m = s * 32 + r;
            const int x = m & ((1 << a.logw) - 1), y = (m >> a.logw) & ((1 << a.logh) - 1), b = m >> (a.logw + a.logh);
            const int yy = y * a.stride + dy, xx = x * a.stride + dx;
            const bool ok = m < a.M && (unsigned)yy < (unsigned)a.H && (unsigned)xx < (unsigned)a.W && c0 + c * 8 < a.C;
            const long off = ok ? (((long)b * a.H + yy) * a.W + xx) * a.C + c0 + c * 8 : 0;
            cp16(st + 2 * YPL + tswz<XB>(r, c), a.xh + off, ok);
            cp16(st + 2 * YPL + XPL + tswz<XB>(r, c), a.xl + off, ok);
        }
    };
    float acc[2][NT][4], bacc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int q = 0; q < 4; ++q) bacc[i][q] = 0.f;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
    }
    const uint32_t ones[2] = {0x3f803f80u, 0x3f803f80u};
#pragma unroll
    for (int s = 0; s < GST - 1; ++s) {
        if (s0 + s < s1) load(s0 + s, s);
        cp_commit();
    }
    int slot = 0;
    for (int s = s0; s < s1; ++s) {
        cp_wait<GST - 2>();
        __syncthreads();
        if (s + GST - 1 < s1) load(s + GST - 1, slot == 0 ? GST - 1 : slot - 1);
        cp_commit();
        const uint32_t st = base + slot * STAGE;
        slot = slot + 1 == GST ? 0 : slot + 1;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            uint32_t ah[2][4], al[2][4], bh[NT][2], bl[NT][2];
            const int q = lane >> 3, j = lane & 7;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                // matrices (k, m): (lo, lo), (lo, hi), (hi, lo), (hi, hi) of 8 pixels x 8 channels
                const int r = kk * 16 + (q >> 1) * 8 + j, c = (wm + mt * 16) / 8 + (q & 1);
                ldsm4t(ah[mt], st + tswz<YB>(r, c));
                ldsm4t(al[mt], st + YPL + tswz<YB>(r, c));
            }
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2) {
                const int r = kk * 16 + (q & 1) * 8 + j, c = wn / 8 + nt + (q >> 1);
                ldsm4t(bh[nt], st + 2 * YPL + tswz<XB>(r, c));
                ldsm4t(bl[nt], st + 2 * YPL + XPL + tswz<XB>(r, c));
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    mma_bf16(acc[mt][nt], ah[mt], bh[nt]);
                    mma_bf16(acc[mt][nt], ah[mt], bl[nt]);
                    mma_bf16(acc[mt][nt], al[mt], bh[nt]);
                }
                if (dobias) { mma_bf16(bacc[mt], ah[mt], ones); mma_bf16(bacc[mt], al[mt], ones); }
            }
        }
    }
    cp_wait<0>();
    const int g = lane >> 2, t = lane & 3;
    float* out = a.part + (long)blockIdx.z * a.N * a.ntap * a.C;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
            const int n = n0 + wm + mt * 16 + hr * 8 + g;
            if (n >= a.N) continue;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                const int c = c0 + wn + nt * 8 + 2 * t;
                if (c < a.C)
                    *reinterpret_cast<float2*>(out + ((long)n * a.ntap + tap) * a.C + c) =
                        make_float2(acc[mt][nt][2 * hr], acc[mt][nt][2 * hr + 1]);
            }
            if (dobias && t == 0 && (warp & 1) == 0) a.bpart[(long)blockIdx.z * a.N + n] = bacc[mt][2 * hr];
        }
}

// The first layer's gradient: 32 channels (blockIdx.y) x (nine taps and a
// column of ones, the bias) over the pixels of C1PER CTA patches per block.
// Bound by reading the gradient planes once.  part: blocks x N x 16.
__global__ void __launch_bounds__(256) wgrad1_kernel(const float* __restrict__ data, const int* __restrict__ idx,
                                                     const float2* __restrict__ norm, int logw,
                                                     const bf16* __restrict__ yh, const bf16* __restrict__ yl, int N,
                                                     int patches, int per, float* __restrict__ part) {
    extern __shared__ __align__(16) float patch[];
    __shared__ __align__(16) bf16 ys[2][C1PIX * 32];
    float (*red)[32 * 16] = reinterpret_cast<float (*)[32 * 16]>(&ys[0][0]);   // the warps' sums, at the end
    const int wo = 1 << logw, pitch = c1_pitch(wo), perimg = (wo * wo) / C1PIX;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.y * 32;
    const uint32_t yb = smem_addr(ys);
    float acc[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
    const int q0 = blockIdx.x * per, q1 = min(patches, q0 + per);
    for (int pt = q0; pt < q1; ++pt) {
        const int b = pt / perimg, p0 = (pt - b * perimg) * C1PIX;
        const long src = idx ? idx[b] : b;
        __syncthreads();
        const long row = ((long)b << (2 * logw)) + p0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + 256 * i, r = e >> 2, c = e & 3;
            const long off = (row + r) * N + n0 + c * 8;
            cp16(yb + tswz<64>(r, c), yh + off, true);
            cp16(yb + C1PIX * 64 + tswz<64>(r, c), yl + off, true);
        }
        cp_commit();
        c1_load(patch, data + src * (4L << (2 * logw)), norm[b], wo, p0 >> logw);
        cp_wait<0>();
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const int k0 = warp * 32 + kk * 16;
            uint32_t ah[2][4], al[2][4], bh[2][2], bl[2][2];
            const int q = lane >> 3, j = lane & 7;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int r = k0 + (q >> 1) * 8 + j, c = mt * 2 + (q & 1);
                ldsm4t(ah[mt], yb + tswz<64>(r, c));
                ldsm4t(al[mt], yb + C1PIX * 64 + tswz<64>(r, c));
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int p = k0 + 8 * h + 2 * t;
                split2(c1_tap(patch, pitch, logw, p, g), c1_tap(patch, pitch, logw, p + 1, g), bh[0][h], bl[0][h]);
                float v0 = 0.f, v1 = 0.f;
                if (g == 0) { v0 = c1_tap(patch, pitch, logw, p, 8); v1 = c1_tap(patch, pitch, logw, p + 1, 8); }
                else if (g == 1) v0 = v1 = 1.f;
                split2(v0, v1, bh[1][h], bl[1][h]);
            }
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    mma_bf16(acc[mt][nt], ah[mt], bh[nt]);
                    mma_bf16(acc[mt][nt], ah[mt], bl[nt]);
                    mma_bf16(acc[mt][nt], al[mt], bh[nt]);
                }
        }
    }
    // the warps' sums, in warp order
    __syncthreads();
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                red[warp][(mt * 16 + g + (q >> 1) * 8) * 16 + nt * 8 + 2 * t + (q & 1)] = acc[mt][nt][q];
    __syncthreads();
    for (int i = tid; i < 512; i += 256) {
        float s = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += red[w][i];
        part[((long)blockIdx.x * N + n0) * 16 + i] = s;
    }
}

// ---- the last dense layer -----------------------------------------------------

// o = h W^T + bias: one warp per 16 rows, the eight outputs one n-tile
__global__ void __launch_bounds__(32) fc2_kernel(const bf16* __restrict__ hh, const bf16* __restrict__ hl, int B, int K,
                                                 const bf16* __restrict__ w, const float* __restrict__ bias,
                                                 float* __restrict__ o) {
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
    const int r0 = blockIdx.x * 16 + g, r1 = r0 + 8;
    const uint32_t* h0 = reinterpret_cast<const uint32_t*>(hh + (long)min(r0, B - 1) * K);
    const uint32_t* h1 = reinterpret_cast<const uint32_t*>(hh + (long)min(r1, B - 1) * K);
    const uint32_t* l0 = reinterpret_cast<const uint32_t*>(hl + (long)min(r0, B - 1) * K);
    const uint32_t* l1 = reinterpret_cast<const uint32_t*>(hl + (long)min(r1, B - 1) * K);
    const uint32_t* wr = reinterpret_cast<const uint32_t*>(w + (long)g * K);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = t; k < K / 2; k += 8) {
        const uint32_t ah[4] = {h0[k], h1[k], h0[k + 4], h1[k + 4]};
        const uint32_t al[4] = {l0[k], l1[k], l0[k + 4], l1[k + 4]};
        const uint32_t b[2] = {wr[k], wr[k + 4]};
        mma_bf16(acc, ah, b);
        mma_bf16(acc, al, b);
    }
    const float b0 = bias[2 * t], b1 = bias[2 * t + 1];
    if (r0 < B) { o[r0 * NOUT + 2 * t] = acc[0] + b0; o[r0 * NOUT + 2 * t + 1] = acc[1] + b1; }
    if (r1 < B) { o[r1 * NOUT + 2 * t] = acc[2] + b0; o[r1 * NOUT + 2 * t + 1] = acc[3] + b1; }
}

// its gradients in FP32: dh = go W masked by the ReLU (planes of pitch Kp),
// one thread per (row, hidden unit)
__global__ void __launch_bounds__(256) fc2_dgrad_kernel(const float* __restrict__ go, int B, int K, int Kp,
                                                        const float* __restrict__ w, const bf16* __restrict__ hh,
                                                        bf16* __restrict__ gh, bf16* __restrict__ gl) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= (long)B * Kp) return;
    const int b = (int)(i / Kp), j = (int)(i - (long)b * Kp);
    float s = 0.f;
    if (j < K && __bfloat162float(hh[i]) > 0.f)
#pragma unroll
        for (int q = 0; q < NOUT; ++q) s = fmaf(go[b * NOUT + q], w[(long)q * K + j], s);
    split_bf16(s, gh[i], gl[i]);
}

// dW = go^T h and db = sum go: 32 hidden units per CTA, the rows over 8
// groups of lanes that are added in order
__global__ void __launch_bounds__(256) fc2_wgrad_kernel(const float* __restrict__ go, int B, int K, int Kp,
                                                        const bf16* __restrict__ hh, const bf16* __restrict__ hl,
                                                        float* __restrict__ dw, float* __restrict__ db) {
    __shared__ float red[8][NOUT][33];
    const int jl = threadIdx.x & 31, sl = threadIdx.x >> 5, j = blockIdx.x * 32 + jl;
    float s[NOUT], sb = 0.f;
#pragma unroll
    for (int q = 0; q < NOUT; ++q) s[q] = 0.f;
#pragma unroll 4
    for (int b = sl; b < B; b += 8) {
        const long i = (long)b * Kp + j;
        const float h = __bfloat162float(hh[i]) + __bfloat162float(hl[i]);
#pragma unroll
        for (int q = 0; q < NOUT; ++q) s[q] = fmaf(go[b * NOUT + q], h, s[q]);
        if (jl < NOUT) sb += go[b * NOUT + jl];
    }
#pragma unroll
    for (int q = 0; q < NOUT; ++q) red[sl][q][jl] = s[q];
    if (jl < NOUT) red[sl][jl][32] = sb;
    __syncthreads();
    float v = 0.f;
#pragma unroll
    for (int z = 0; z < 8; ++z) v += red[z][sl][jl];      // warp sl takes output sl
    if (j < K) dw[(long)sl * K + j] = v;
    if (blockIdx.x == 0 && jl == 0) {
        float u = 0.f;
#pragma unroll
        for (int z = 0; z < 8; ++z) u += red[z][sl][32];
        db[sl] = u;
    }
}

// ---- packed weights and gradient sums -----------------------------------------

// A layer's weights in the parameter vector, [cout][taps][cin], and the
// packed forms: forward [coutp][tapsp][cinp] (row n, K contiguous) and, for
// the input gradient, [taps][cinp][coutp].
struct PackLayer {
    long woff, boff;
    int cin, cout, cinp, coutp, taps, tapsp;
    long f, fn, b, bn;                // offset and count of the two forms (bn = 0: none)
    const float* part;                // weight-gradient partials: [ranges][coutp][tapsp][cinp]
    const float* bpart;               // bias partials: [ranges][coutp] (null: column cin of the weights')
    int ranges;
};
constexpr int NPACK = NCONV + 2;
struct PackArgs {
    PackLayer l[NPACK];
    int n;
};

// Packs the masters w, rounded to BF16 (blockIdx.y the layer); for new parameters
// one more block row writes the rounded values themselves into weff and clears
// the optimiser's moments m, v.  The transposed form goes
// through 32 x 32 tiles: read with its stride, with 64-bit divisions, packing the
// 8.5 M parameters of a 512-pixel network took 0.2 of a training step's 1.24 ms
// (now 1.04); set_params of the small networks 37 and 50 us in four launches,
// now 29 and 39 in one.  A layer's forms have less than 2^31 elements.
constexpr int PACK_BLOCKS = 148, PACK_THREADS = 256;

__global__ void __launch_bounds__(PACK_THREADS) pack_kernel(const __grid_constant__ PackArgs p,
                                                            const float* __restrict__ w, bf16* __restrict__ out,
                                                            float* __restrict__ weff, float* __restrict__ m,
                                                            float* __restrict__ v, long nparams) {
    if (blockIdx.y == NPACK) {
        for (long i = blockIdx.x * (long)PACK_THREADS + threadIdx.x; i < nparams; i += (long)gridDim.x * PACK_THREADS) {
            weff[i] = __bfloat162float(__float2bfloat16_rn(w[i]));
            m[i] = 0.f;
            v[i] = 0.f;
        }
        return;
    }
    const PackLayer& L = p.l[blockIdx.y];
    const float* src = w + L.woff;
    const unsigned cin = L.cin, cout = L.cout, taps = L.taps, cinp = L.cinp, coutp = L.coutp, tapsp = L.tapsp;
    for (unsigned i = blockIdx.x * PACK_THREADS + threadIdx.x; i < (unsigned)L.fn; i += gridDim.x * PACK_THREADS) {
        const unsigned q = i / cinp, c = i - q * cinp, n = q / tapsp, tap = q - n * tapsp;
        const bool ok = n < cout && tap < taps && c < cin;
        out[L.f + i] = __float2bfloat16_rn(ok ? src[((long)n * taps + tap) * cin + c] : 0.f);
    }
    if (!L.bn) return;
    // [taps][cinp][coutp]: tiles of 32 channels c by 32 rows n (both padded to 32)
    __shared__ float tile[32][33];
    const unsigned tx = threadIdx.x & 31, ty = threadIdx.x >> 5, tc = cinp / 32, tn = coutp / 32;
    for (unsigned t = blockIdx.x; t < taps * tc * tn; t += gridDim.x) {
        const unsigned q = t / tn, n0 = (t - q * tn) * 32, tap = q / tc, c0 = (q - tap * tc) * 32;
        __syncthreads();
#pragma unroll
        for (unsigned r = 0; r < 32; r += PACK_THREADS / 32) {
            const unsigned n = n0 + ty + r, c = c0 + tx;
            tile[ty + r][tx] = n < cout && c < cin ? src[((long)n * taps + tap) * cin + c] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (unsigned r = 0; r < 32; r += PACK_THREADS / 32)
            out[L.b + ((long)tap * cinp + c0 + ty + r) * coutp + n0 + tx] = __float2bfloat16_rn(tile[tx][ty + r]);
    }
}

// the layers' partial sums, ranges in order, into the gradient vector
__global__ void grad_sum_kernel(const __grid_constant__ PackArgs p, float* __restrict__ g) {
    const PackLayer& L = p.l[blockIdx.y];
    const long nw = (long)L.cout * L.taps * L.cin, slab = (long)L.coutp * L.tapsp * L.cinp;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nw + L.cout; i += (long)gridDim.x * blockDim.x) {
        float s = 0.f;
        if (i < nw) {
            const int c = (int)(i % L.cin), tap = (int)(i / L.cin % L.taps), n = (int)(i / ((long)L.cin * L.taps));
            const float* q = L.part + ((long)n * L.tapsp + tap) * L.cinp + c;
#pragma unroll 4
            for (int z = 0; z < L.ranges; ++z) s += q[z * slab];
            g[L.woff + i] = s;
        } else {
            const int n = (int)(i - nw);
            if (L.bpart)
                for (int z = 0; z < L.ranges; ++z) s += L.bpart[(long)z * L.coutp + n];
            else
                for (int z = 0; z < L.ranges; ++z) s += L.part[z * slab + n * 16 + 9];
            g[L.boff + n] = s;
        }
    }
}

// rows idx[b] of a (n x width) table
__global__ void gather_rows_kernel(const float* __restrict__ src, const int* __restrict__ idx, int rows, int width,
                                   float* __restrict__ dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * width) return;
    const int r = i / width, c = i - r * width;
    dst[i] = src[(long)idx[r] * width + c];
}

__device__ __forceinline__ void cross3(const float* a, const float* b, float* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// head: outputs (B x 8) -> R (row-major, columns b1 b2 b3) and shift;
// with targets: per-sample loss and d loss / d outputs (mean over B)
__global__ void head_kernel(const float* __restrict__ o, int B, const float* __restrict__ tgt, float lambda,
                            float* __restrict__ res, float* __restrict__ go, float* __restrict__ loss) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const float* a1 = o + b * NOUT;
    const float* a2 = a1 + 3;
    const float n1 = sqrtf(a1[0] * a1[0] + a1[1] * a1[1] + a1[2] * a1[2]) + 1e-12f;
    float b1[3] = {a1[0] / n1, a1[1] / n1, a1[2] / n1};
    const float d = b1[0] * a2[0] + b1[1] * a2[1] + b1[2] * a2[2];
    float u2[3] = {a2[0] - d * b1[0], a2[1] - d * b1[1], a2[2] - d * b1[2]};
    const float n2 = sqrtf(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]) + 1e-12f;
    float b2[3] = {u2[0] / n2, u2[1] / n2, u2[2] / n2};
    float b3[3];
    cross3(b1, b2, b3);
    const float t0 = o[b * NOUT + 6], t1 = o[b * NOUT + 7];
    if (res) {
        float* r = res + b * NRES;
        for (int i = 0; i < 3; ++i) { r[3 * i + 0] = b1[i]; r[3 * i + 1] = b2[i]; r[3 * i + 2] = b3[i]; }
        r[9] = t0;
        r[10] = t1;
    }
    if (!tgt) return;
    const float* T = tgt + b * NRES;    // R* row-major, t*
    float r1[3] = {T[0], T[3], T[6]}, r2[3] = {T[1], T[4], T[7]}, r3[3] = {T[2], T[5], T[8]};
    float L = 0.f, gb1[3], gb2[3], gb3[3];
    for (int i = 0; i < 3; ++i) {
        gb1[i] = 2.f * (b1[i] - r1[i]);
        gb2[i] = 2.f * (b2[i] - r2[i]);
        gb3[i] = 2.f * (b3[i] - r3[i]);
        L += (b1[i] - r1[i]) * (b1[i] - r1[i]) + (b2[i] - r2[i]) * (b2[i] - r2[i]) + (b3[i] - r3[i]) * (b3[i] - r3[i]);
    }
    const float dt0 = t0 - T[9], dt1 = t1 - T[10];
    L += lambda * (dt0 * dt0 + dt1 * dt1);
    // b3 = b1 x b2: d/db1 (g.b3) = b2 x g, d/db2 (g.b3) = g x b1
    float c[3];
    cross3(b2, gb3, c);
    for (int i = 0; i < 3; ++i) gb1[i] += c[i];
    cross3(gb3, b1, c);
    for (int i = 0; i < 3; ++i) gb2[i] += c[i];
    // b2 = u2 / n2
    const float gb2b2 = gb2[0] * b2[0] + gb2[1] * b2[1] + gb2[2] * b2[2];
    float gu2[3];
    for (int i = 0; i < 3; ++i) gu2[i] = (gb2[i] - gb2b2 * b2[i]) / n2;
    // u2 = a2 - (b1.a2) b1
    const float gu2b1 = gu2[0] * b1[0] + gu2[1] * b1[1] + gu2[2] * b1[2];
    float ga2[3];
    for (int i = 0; i < 3; ++i) {
        ga2[i] = gu2[i] - gu2b1 * b1[i];
        gb1[i] += -d * gu2[i] - a2[i] * gu2b1;
    }
    // b1 = a1 / n1
    const float gb1b1 = gb1[0] * b1[0] + gb1[1] * b1[1] + gb1[2] * b1[2];
    const float sc = 1.f / B;
    float* g = go + b * NOUT;
    for (int i = 0; i < 3; ++i) {
        g[i] = sc * (gb1[i] - gb1b1 * b1[i]) / n1;
        g[3 + i] = sc * ga2[i];
    }
    g[6] = sc * 2.f * lambda * dt0;
    g[7] = sc * 2.f * lambda * dt1;
    loss[b] = L;
}

__global__ void mean_kernel(const float* __restrict__ v, int n, float* __restrict__ out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double s = 0;
        for (int i = 0; i < n; ++i) s += v[i];
        *out = (float)(s / n);
    }
}

// Adam on the FP32 masters; the working copy is the BF16 rounding
__global__ void adam_kernel(float* __restrict__ w, float* __restrict__ weff, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, long n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
        w[i] = wi;
        weff[i] = __bfloat162float(__float2bfloat16_rn(wi));
    }
}

struct Layer {
    int cin, cout, h, w, ho, wo;   // convolution geometry (fc: h = w = ho = wo = 1)
    long woff, boff, k;            // weight / bias offsets, K = 9 cin (conv) or cin (fc)
};

}  // namespace

struct Cnn {
    bsg_cnn_config cfg;
    int device = 0;
    cudaStream_t stream = nullptr;
    Layer conv[NCONV], fc1, fc2;
    long nparams = 0;
    float *d_w = nullptr, *d_weff = nullptr, *d_g = nullptr, *d_m = nullptr, *d_v = nullptr;
    int cap = 0;                       // images the forward buffers hold
    int gcap = 0;                      // images the gradient buffers hold
    float2* d_norm = nullptr;          // mean and 1 / standard deviation of each image
    bf16 *d_ah[NCONV + 1] = {}, *d_al[NCONV + 1] = {};   // activation planes after ReLU, NHWC (1 .. NCONV)
    bf16 *d_hh = nullptr, *d_hl = nullptr;               // fc1 output planes
    float* d_o = nullptr;              // fc2 output
    bf16 *d_gh[2] = {}, *d_gl[2] = {}; // activation gradient planes (two, in turn)
    bf16 *d_dh = nullptr, *d_dl = nullptr;               // gradient of the fc1 output
    float* d_go = nullptr;
    float* d_part = nullptr;           // weight-gradient partial sums of every layer
    bf16* d_pack = nullptr;            // packed weights
    PackArgs pack{};
    float* d_src = nullptr;            // host images' copy
    size_t src_elems = 0;
    float* d_res = nullptr;            // cap x 11
    float* d_tgt = nullptr;            // cap x 11
    float* d_loss = nullptr;           // cap
    long step = 0;                     // Adam steps taken
};

}  // namespace bsg

using namespace bsg;

namespace {

int cfail(int code, const char* fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    set_error("%s", buf);
    return code;
}

#define CCK(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return cfail(BSG_ERR_CUDA, "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

unsigned grid_for(long n) { return (unsigned)std::max(1L, std::min(148L * 16, (n + 255) / 256)); }

int ilog2(int v) { int l = 0; while ((1 << l) < v) ++l; return l; }

template <int BM, int BN>
cudaError_t launch_conv(const ConvArgs& a, int nclass, cudaStream_t s) {
    const dim3 grid((unsigned)((a.M + BM - 1) / BM), (unsigned)(a.N / BN), (unsigned)nclass);
    conv_gemm_kernel<BM, BN><<<grid, 256, conv_smem<BM, BN>(), s>>>(a);
    return cudaGetLastError();
}

// Widest column tile that divides the channels; then the tallest row tile
// that still gives every SM a block (the deep layers have few pixels: at 256
// images of 128^2 the last convolution has 1,024 rows, 8 blocks of 128 but
// 32 of 32).
cudaError_t conv_gemm(const ConvArgs& a, int nclass, cudaStream_t s) {
    const long n128 = a.N / 128, rows = a.M;
    if (a.N % 128 == 0) {
        if ((rows + 127) / 128 * n128 * nclass >= 148) return launch_conv<128, 128>(a, nclass, s);
        if ((rows + 63) / 64 * n128 * nclass >= 148) return launch_conv<64, 128>(a, nclass, s);
        return launch_conv<32, 128>(a, nclass, s);
    }
    if (a.N % 64 == 0) {
        if ((rows + 127) / 128 * (a.N / 64) * nclass >= 148) return launch_conv<128, 64>(a, nclass, s);
        return launch_conv<64, 64>(a, nclass, s);
    }
    return launch_conv<128, 32>(a, nclass, s);
}

template <int BM, int BN>
cudaError_t conv_attr() {
    return cudaFuncSetAttribute(conv_gemm_kernel<BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, conv_smem<BM, BN>());
}

cudaError_t cnn_attributes() {
    cudaError_t e = conv_attr<128, 128>();
    if (e == cudaSuccess) e = conv_attr<64, 128>();
    if (e == cudaSuccess) e = conv_attr<32, 128>();
    if (e == cudaSuccess) e = conv_attr<128, 64>();
    if (e == cudaSuccess) e = conv_attr<64, 64>();
    if (e == cudaSuccess) e = conv_attr<128, 32>();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wgrad_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, wgrad_smem<64>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(wgrad_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, wgrad_smem<32>());
    return e;
}

// forward and input-gradient forms of the layers' weights, from the masters;
// for new parameters (fresh) the working copy and the optimiser's state too
cudaError_t pack_weights(Cnn& c, bool fresh, cudaStream_t s) {
    pack_kernel<<<dim3(PACK_BLOCKS, NPACK + (fresh ? 1 : 0)), PACK_THREADS, 0, s>>>(c.pack, c.d_w, c.d_pack, c.d_weff,
                                                                                   c.d_m, c.d_v, c.nparams);
    return cudaGetLastError();
}

void plan_pack(Cnn& c) {
    long off = 0;
    auto take = [&](long n) { const long o = off; off += (n + 7) / 8 * 8; return o; };
    c.pack.n = NPACK;
    for (int l = 0; l < NPACK; ++l) {
        PackLayer& P = c.pack.l[l];
        const Layer& L = l < NCONV ? c.conv[l] : l == NCONV ? c.fc1 : c.fc2;
        P.woff = L.woff;
        P.boff = L.boff;
        P.cout = L.cout;
        P.coutp = l == NCONV + 1 ? NOUT : cpad(L.cout);
        if (l < NCONV) {
            P.cin = L.cin;
            P.taps = 9;
            P.cinp = l ? cpad(L.cin) : 1;
            P.tapsp = l ? 9 : 16;
        } else if (l == NCONV) {
            // (pixel, channel) of the last activation
            P.cin = c.conv[NCONV - 1].cout;
            P.cinp = cpad(P.cin);
            P.taps = P.tapsp = (int)(L.k / P.cin);
        } else {
            P.cin = (int)L.k;
            P.cinp = cpad(P.cin);
            P.taps = P.tapsp = 1;
        }
        P.fn = (long)P.coutp * P.tapsp * P.cinp;
        P.f = take(P.fn);
        P.bn = l > 0 && l <= NCONV ? P.fn : 0;
        P.b = take(P.bn);
    }
}

long pack_elems(const Cnn& c) {
    const PackLayer& P = c.pack.l[NPACK - 1];
    return P.b + P.bn + 8;
}

// planes of one image's activations, in elements of one plane
size_t act_elems(const Cnn& c, int l) { return (size_t)c.conv[l].ho * c.conv[l].wo * cpad(c.conv[l].cout); }

size_t image_bytes(const Cnn& c) {
    size_t b = 4 * (size_t)cpad(c.cfg.hidden);
    for (int l = 0; l < NCONV; ++l) b += 4 * act_elems(c, l);
    return b;
}

void free_forward(Cnn& c) {
    auto F = [](auto*& p) { cudaFree(p); p = nullptr; };
    for (int l = 1; l <= NCONV; ++l) { F(c.d_ah[l]); F(c.d_al[l]); }
    F(c.d_hh); F(c.d_hl); F(c.d_o); F(c.d_norm); F(c.d_res);
    c.cap = 0;
}

int ensure_batch(Cnn& c, int B) {
    if (B <= c.cap) return BSG_OK;
    free_forward(c);
    const size_t n = (size_t)B;
    for (int l = 0; l < NCONV; ++l) {
        CCK(cudaMalloc(&c.d_ah[l + 1], sizeof(bf16) * act_elems(c, l) * n));
        CCK(cudaMalloc(&c.d_al[l + 1], sizeof(bf16) * act_elems(c, l) * n));
    }
    CCK(cudaMalloc(&c.d_hh, sizeof(bf16) * cpad(c.cfg.hidden) * n));
    CCK(cudaMalloc(&c.d_hl, sizeof(bf16) * cpad(c.cfg.hidden) * n));
    CCK(cudaMalloc(&c.d_o, sizeof(float) * NOUT * n));
    CCK(cudaMalloc(&c.d_norm, sizeof(float2) * n));
    CCK(cudaMalloc(&c.d_res, sizeof(float) * NRES * n));
    c.cap = B;
    return BSG_OK;
}

// pixel ranges of a layer's weight gradient: about four CTAs per SM, each
// with at least eight K-steps (a function of the sizes only: the sums'
// order is fixed)
int wgrad_ranges(long ctas, int steps) {
    return (int)std::max<long>(1, std::min<long>((4 * 148 + ctas - 1) / ctas, steps / 8));
}

struct WgradPlan {
    int steps, per, ranges, bn;
    unsigned gy;
};

WgradPlan wgrad_plan(long M, int N, int C, int ntap) {
    WgradPlan p;
    p.steps = (int)((M + 31) / 32);
    p.bn = C % 64 == 0 ? 64 : 32;
    p.gy = (unsigned)((N + 63) / 64) * (unsigned)((C + p.bn - 1) / p.bn);
    const int want = wgrad_ranges((long)ntap * p.gy, p.steps);
    p.per = (p.steps + want - 1) / want;
    p.ranges = (p.steps + p.per - 1) / p.per;
    return p;
}

constexpr int W1_PER = 8;      // first layer: patches of 256 pixels per CTA

void free_grad(Cnn& c) {
    auto F = [](auto*& p) { cudaFree(p); p = nullptr; };
    for (int i = 0; i < 2; ++i) { F(c.d_gh[i]); F(c.d_gl[i]); }
    F(c.d_dh); F(c.d_dl); F(c.d_go); F(c.d_tgt); F(c.d_loss); F(c.d_part);
    c.gcap = 0;
}

// gradient buffers, and room for the layers' partial sums
int ensure_grad(Cnn& c, int B) {
    if (B > c.gcap) {
        free_grad(c);
        size_t act = 0;
        for (int l = 0; l < NCONV; ++l) act = std::max(act, act_elems(c, l));
        for (int i = 0; i < 2; ++i) {
            CCK(cudaMalloc(&c.d_gh[i], sizeof(bf16) * act * B));
            CCK(cudaMalloc(&c.d_gl[i], sizeof(bf16) * act * B));
        }
        CCK(cudaMalloc(&c.d_dh, sizeof(bf16) * cpad(c.cfg.hidden) * (size_t)B));
        CCK(cudaMalloc(&c.d_dl, sizeof(bf16) * cpad(c.cfg.hidden) * (size_t)B));
        CCK(cudaMalloc(&c.d_go, sizeof(float) * NOUT * B));
        CCK(cudaMalloc(&c.d_tgt, sizeof(float) * NRES * B));
        CCK(cudaMalloc(&c.d_loss, sizeof(float) * B));
        // the most any batch up to B needs: the ranges grow with the batch
        size_t elems = 0;
        for (int l = 0; l <= NCONV; ++l) {
            const PackLayer& P = c.pack.l[l];
            if (l == 0) {
                const long patches = (long)B * ((c.conv[0].ho * c.conv[0].wo) / C1PIX);
                elems += (size_t)((patches + W1_PER - 1) / W1_PER) * P.coutp * 16;
                continue;
            }
            const long M = l < NCONV ? (long)B * c.conv[l].ho * c.conv[l].wo : B;
            const int ntap = l < NCONV ? 9 : 1, C = l < NCONV ? P.cinp : P.tapsp * P.cinp;
            const WgradPlan w = wgrad_plan(M, P.coutp, C, ntap);
            elems += (size_t)wgrad_ranges((long)ntap * w.gy, w.steps) * (P.fn + P.coutp);
        }
        CCK(cudaMalloc(&c.d_part, sizeof(float) * elems));
        c.gcap = B;
    }
    return BSG_OK;
}

int ensure_src(Cnn& c, size_t elems) {
    if (elems <= c.src_elems) return BSG_OK;
    cudaFree(c.d_src);
    c.d_src = nullptr;
    c.src_elems = 0;
    CCK(cudaMalloc(&c.d_src, sizeof(float) * elems));
    c.src_elems = elems;
    return BSG_OK;
}

size_t patch_bytes(int wo) { return sizeof(float) * (2 * (C1PIX / wo) + 1) * (2 * wo + 4); }

// forward pass of B images: data (and idx, the batch's images within it, or
// null) on the device; outputs in c.d_o
cudaError_t forward(Cnn& c, const float* data, const int* idx, int B, cudaStream_t s) {
    const int box = c.cfg.box;
    image_norm_kernel<<<B, 256, 0, s>>>(data, idx, box * box, c.d_norm);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    {
        const Layer& L = c.conv[0];
        const PackLayer& P = c.pack.l[0];
        const dim3 grid((unsigned)((long)B * ((L.ho * L.wo) / C1PIX)), (unsigned)(P.coutp / 32));
        conv1_kernel<<<grid, 256, patch_bytes(L.wo), s>>>(data, idx, c.d_norm, ilog2(L.wo), c.d_pack + P.f,
                                                          c.d_weff + L.boff, L.cout, P.coutp, c.d_ah[1], c.d_al[1]);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    for (int l = 1; l <= NCONV; ++l) {
        const PackLayer& P = c.pack.l[l];
        const bool fc = l == NCONV;
        const Layer& L = fc ? c.fc1 : c.conv[l];
        ConvArgs a{};
        a.ah = c.d_ah[l];
        a.al = c.d_al[l];
        a.w = c.d_pack + P.f;
        a.C = fc ? P.tapsp * P.cinp : P.cinp;
        a.wrow = (long)P.tapsp * P.cinp;
        a.wtap = P.cinp;
        a.M = B * L.ho * L.wo;
        a.N = P.coutp;
        a.logw = a.logh = ilog2(L.wo);
        a.H = a.W = L.h;
        a.stride = fc ? 1 : 2;
        a.oh = fc ? c.d_hh : c.d_ah[l + 1];
        a.ol = fc ? c.d_hl : c.d_al[l + 1];
        a.OH = a.OW = L.ho;
        a.ostride = 1;
        a.bias = c.d_weff + P.boff;
        a.nbias = P.cout;
        a.relu = 1;
        ConvClass& k = a.cls[0];
        k.ntap = fc ? 1 : 9;
        for (int t = 0; t < k.ntap; ++t) {
            k.dy[t] = (signed char)(fc ? 0 : t / 3 - 1);
            k.dx[t] = (signed char)(fc ? 0 : t % 3 - 1);
            k.w[t] = (signed char)t;
        }
        if ((e = conv_gemm(a, 1, s)) != cudaSuccess) return e;
    }
    const PackLayer& P = c.pack.l[NCONV + 1];
    fc2_kernel<<<(B + 15) / 16, 32, 0, s>>>(c.d_hh, c.d_hl, B, P.cinp, c.d_pack + P.f, c.d_weff + P.boff, c.d_o);
    return cudaGetLastError();
}

// gradients of the batch loss into c.d_g (overwritten), from c.d_go; the
// batch as given to forward
cudaError_t backward(Cnn& c, const float* data, const int* idx, int B, cudaStream_t s) {
    const int Hp = cpad(c.cfg.hidden);
    const PackLayer& P2 = c.pack.l[NCONV + 1];
    fc2_wgrad_kernel<<<Hp / 32, 256, 0, s>>>(c.d_go, B, c.cfg.hidden, Hp, c.d_hh, c.d_hl, c.d_g + P2.woff,
                                             c.d_g + P2.boff);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    fc2_dgrad_kernel<<<(unsigned)(((long)B * Hp + 255) / 256), 256, 0, s>>>(c.d_go, B, c.cfg.hidden, Hp,
                                                                            c.d_weff + P2.woff, c.d_hh, c.d_dh, c.d_dl);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    PackArgs sums = c.pack;
    float* part = c.d_part;
    const bf16 *yh = c.d_dh, *yl = c.d_dl;                    // gradient of layer l's output
    for (int l = NCONV; l >= 1; --l) {
        PackLayer& P = sums.l[l];
        const bool fc = l == NCONV;
        const Layer& L = fc ? c.fc1 : c.conv[l];
        WgradArgs w{};
        w.yh = yh;
        w.yl = yl;
        w.xh = c.d_ah[l];
        w.xl = c.d_al[l];
        w.M = B * L.ho * L.wo;
        w.N = P.coutp;
        w.C = fc ? P.tapsp * P.cinp : P.cinp;
        w.logw = w.logh = ilog2(L.wo);
        w.H = w.W = L.h;
        w.stride = fc ? 1 : 2;
        w.ntap = fc ? 1 : 9;
        const WgradPlan p = wgrad_plan(w.M, w.N, w.C, w.ntap);
        w.steps = p.steps;
        w.per = p.per;
        w.part = part;
        w.bpart = part + (size_t)p.ranges * P.fn;
        part = w.bpart + (size_t)p.ranges * P.coutp;
        P.part = w.part;
        P.bpart = w.bpart;
        P.ranges = p.ranges;
        const dim3 grid((unsigned)w.ntap, p.gy, (unsigned)p.ranges);
        if (p.bn == 64) wgrad_kernel<64><<<grid, 128, wgrad_smem<64>(), s>>>(w);
        else wgrad_kernel<32><<<grid, 128, wgrad_smem<32>(), s>>>(w);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        // input gradient, masked by the ReLU of the layer below
        ConvArgs a{};
        a.ah = yh;
        a.al = yl;
        a.w = c.d_pack + P.b;
        a.wrow = P.coutp;
        a.wtap = (long)P.cinp * P.coutp;
        a.C = P.coutp;
        a.N = fc ? P.tapsp * P.cinp : P.cinp;
        a.M = B * L.ho * L.wo;
        a.logw = a.logh = ilog2(L.wo);
        a.H = a.W = L.ho;
        a.stride = 1;
        a.oh = c.d_gh[l & 1];
        a.ol = c.d_gl[l & 1];
        a.OH = a.OW = fc ? 1 : L.h;
        a.ostride = fc ? 1 : 2;
        a.mask = c.d_ah[l];
        int ncls = 0;
        if (fc) {
            a.cls[0].ntap = 1;
            ncls = 1;
        } else {
            // input pixel 2 y + py takes the taps ky = py + 1 (mod 2) from
            // output row y + (py + 1 - ky) / 2; the class with most taps first
            for (int py = 1; py >= 0; --py)
                for (int px = 1; px >= 0; --px) {
                    ConvClass& k = a.cls[ncls++];
                    k.oy = py;
                    k.ox = px;
                    for (int ky = 0; ky < 3; ++ky)
                        for (int kx = 0; kx < 3; ++kx) {
                            if (((py + 1 - ky) & 1) || ((px + 1 - kx) & 1)) continue;
                            k.dy[k.ntap] = (signed char)((py + 1 - ky) / 2);
                            k.dx[k.ntap] = (signed char)((px + 1 - kx) / 2);
                            k.w[k.ntap++] = (signed char)(ky * 3 + kx);
                        }
                }
        }
        if ((e = conv_gemm(a, ncls, s)) != cudaSuccess) return e;
        yh = a.oh;
        yl = a.ol;
    }
    {
        PackLayer& P = sums.l[0];
        const Layer& L = c.conv[0];
        const int patches = B * ((L.ho * L.wo) / C1PIX);
        P.ranges = (patches + W1_PER - 1) / W1_PER;
        P.part = part;
        P.bpart = nullptr;
        wgrad1_kernel<<<dim3((unsigned)P.ranges, (unsigned)(P.coutp / 32)), 256, patch_bytes(L.wo), s>>>(
            data, idx, c.d_norm, ilog2(L.wo), yh, yl, P.coutp, patches, W1_PER, part);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    grad_sum_kernel<<<dim3(148, NCONV + 1), 256, 0, s>>>(sums, c.d_g);
    return cudaGetLastError();
}

uint64_t splitmix(uint64_t& x) {
    uint64_t z = (x += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

}  // namespace

extern "C" int bsg_cnn_create(const bsg_cnn_config* cfg, bsg_cnn** out) {
    if (!cfg || !out) return cfail(BSG_ERR_ARG, "bsg_cnn_create: null argument");
    *out = nullptr;
    const int box = cfg->box;
    if (box < 64 || box > 512 || (box & (box - 1)))
        return cfail(BSG_ERR_ARG, "bsg_cnn_create: box %d must be a power of two in 64..512", box);
    for (int l = 0; l < NCONV; ++l)
        if (cfg->channels[l] < 1 || cfg->channels[l] > 1024) return cfail(BSG_ERR_ARG, "bsg_cnn_create: bad channel count");
    if (cfg->hidden < 1 || cfg->hidden > 8192) return cfail(BSG_ERR_ARG, "bsg_cnn_create: bad hidden width");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || cfg->device < 0 || cfg->device >= ndev)
        return cfail(BSG_ERR_NODEV, "bsg_cnn_create: no CUDA device %d", cfg->device);
    CCK(cudaSetDevice(cfg->device));
    Cnn* c = new (std::nothrow) Cnn();
    if (!c) return cfail(BSG_ERR_NOMEM, "bsg_cnn_create: out of host memory");
    c->cfg = *cfg;
    c->device = cfg->device;
    long off = 0;
    int h = box, cin = 1;
    for (int l = 0; l < NCONV; ++l) {
        Layer& L = c->conv[l];
        L.cin = cin; L.cout = cfg->channels[l]; L.h = L.w = h; L.ho = L.wo = h / 2; L.k = 9L * cin;
        L.woff = off; off += (long)L.cout * L.k;
        L.boff = off; off += L.cout;
        cin = L.cout;
        h /= 2;
    }
    c->fc1 = Layer{h * h * cin, cfg->hidden, 1, 1, 1, 1, off, 0, (long)h * h * cin};
    off += (long)c->fc1.cout * c->fc1.k;
    c->fc1.boff = off; off += c->fc1.cout;
    c->fc2 = Layer{cfg->hidden, NOUT, 1, 1, 1, 1, off, 0, cfg->hidden};
    off += (long)NOUT * cfg->hidden;
    c->fc2.boff = off; off += NOUT;
    c->nparams = off;
    // He initialisation from a seeded generator; biases zero
    std::vector<float> w(off, 0.f);
    uint64_t st = cfg->seed ? cfg->seed : 0x5EEDull;
    auto normal = [&]() {
        const double u1 = ((splitmix(st) >> 11) + 1.0) / 9007199254740993.0, u2 = (splitmix(st) >> 11) / 9007199254740992.0;
        return sqrt(-2.0 * log(u1)) * cos(2 * M_PI * u2);
    };
    auto init = [&](const Layer& L) {
        const double sd = sqrt(2.0 / L.k);
        for (long i = 0; i < (long)L.cout * L.k; ++i) w[L.woff + i] = (float)(sd * normal());
    };
    for (int l = 0; l < NCONV; ++l) init(c->conv[l]);
    init(c->fc1);
    {
        const double sd = sqrt(1.0 / c->fc2.k);
        for (long i = 0; i < (long)NOUT * c->fc2.k; ++i) w[c->fc2.woff + i] = (float)(sd * normal());
    }
    cudaError_t e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_w, sizeof(float) * off);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_weff, sizeof(float) * off);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_g, sizeof(float) * off);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_m, sizeof(float) * off);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_v, sizeof(float) * off);
    plan_pack(*c);
    if (e == cudaSuccess) e = cudaMalloc(&c->d_pack, sizeof(bf16) * pack_elems(*c));
    if (e == cudaSuccess) e = cnn_attributes();
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d_w, w.data(), sizeof(float) * off, cudaMemcpyHostToDevice, c->stream);
    if (e == cudaSuccess) e = pack_weights(*c, true, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
        bsg_cnn_destroy(reinterpret_cast<bsg_cnn*>(c));
        return cfail(BSG_ERR_CUDA, "bsg_cnn_create: %s", cudaGetErrorString(e));
    }
    *out = reinterpret_cast<bsg_cnn*>(c);
    return BSG_OK;
}

extern "C" void bsg_cnn_destroy(bsg_cnn* h) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c) return;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    free_forward(*c);
    free_grad(*c);
    float* fp[] = {c->d_w, c->d_weff, c->d_g, c->d_m, c->d_v, c->d_src};
    for (float* p : fp) if (p) cudaFree(p);
    if (c->d_pack) cudaFree(c->d_pack);
    if (c->stream) cudaStreamDestroy(c->stream);
    delete c;
}

extern "C" long bsg_cnn_num_params(const bsg_cnn* h) {
    const Cnn* c = reinterpret_cast<const Cnn*>(h);
    return c ? c->nparams : 0;
}

extern "C" int bsg_cnn_get_params(bsg_cnn* h, float* out) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c || !out) return cfail(BSG_ERR_ARG, "bsg_cnn_get_params: null argument");
    CCK(cudaSetDevice(c->device));
    CCK(cudaMemcpy(out, c->d_w, sizeof(float) * c->nparams, cudaMemcpyDeviceToHost));
    return BSG_OK;
}

extern "C" int bsg_cnn_set_params(bsg_cnn* h, const float* in) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c || !in) return cfail(BSG_ERR_ARG, "bsg_cnn_set_params: null argument");
    CCK(cudaSetDevice(c->device));
    CCK(cudaMemcpyAsync(c->d_w, in, sizeof(float) * c->nparams, cudaMemcpyHostToDevice, c->stream));
    CCK(pack_weights(*c, true, c->stream));
    c->step = 0;
    CCK(cudaStreamSynchronize(c->stream));
    return BSG_OK;
}

extern "C" int bsg_cnn_predict(bsg_cnn* h, const float* images, long n, float* out, int flags) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c || !images || !out || n < 1) return cfail(BSG_ERR_ARG, "bsg_cnn_predict: bad argument");
    CCK(cudaSetDevice(c->device));
    // images per pass: at least the context's batch; as many as 1.5 GB of
    // activations hold when they fit (each image's result is its own).  2,048
    // images of 128^2 in passes of 256 leave the deep layers with 8 to 32
    // blocks for 148 SMs.
    int B = std::max(1, std::min<int>(c->cfg.batch > 0 ? c->cfg.batch : 256, (int)std::min<long>(n, 1 << 20)));
    const long wide = std::min<long>(std::min<long>(n, 16384), (long)(1500000000 / image_bytes(*c)));
    const size_t npix = (size_t)c->cfg.box * c->cfg.box;
    const bool dev = (flags & BSG_DEVICE_PTR) != 0;
    // the activations of b images, and host images' copy
    auto room = [&](int b) {
        const int rc = ensure_batch(*c, b);
        return rc || dev ? rc : ensure_src(*c, npix * b);
    };
    if (wide > B && room((int)wide) == BSG_OK) {
        B = (int)wide;
    } else {
        if (wide > B) {                          // they did not fit together
            cudaGetLastError();
            free_forward(*c);
        }
        const int rc = room(B);
        if (rc) return rc;
    }
    cudaStream_t s = c->stream;
    cudaError_t e = cudaSuccess;
    for (long b0 = 0; e == cudaSuccess && b0 < n; b0 += B) {
        const int cnt = (int)std::min<long>(B, n - b0);
        const float* src = images + (size_t)b0 * npix;
        if (!dev) {
            e = cudaMemcpyAsync(c->d_src, src, sizeof(float) * (size_t)npix * cnt, cudaMemcpyHostToDevice, s);
            src = c->d_src;
        }
        if (e == cudaSuccess) e = forward(*c, src, nullptr, cnt, s);
        float* res = dev ? out + (size_t)b0 * NRES : c->d_res;
        if (e == cudaSuccess) {
            head_kernel<<<(cnt + 127) / 128, 128, 0, s>>>(c->d_o, cnt, nullptr, 0.f, res, nullptr, nullptr);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess && !dev)
            e = cudaMemcpyAsync(out + (size_t)b0 * NRES, res, sizeof(float) * NRES * cnt, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess && !dev) e = cudaStreamSynchronize(s);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cfail(BSG_ERR_CUDA, "bsg_cnn_predict: %s", cudaGetErrorString(e));
    return BSG_OK;
}

extern "C" int bsg_cnn_loss_grad(bsg_cnn* h, const float* images, const float* targets, long n, double* loss,
                                 float* grads) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c || !images || !targets || n < 1) return cfail(BSG_ERR_ARG, "bsg_cnn_loss_grad: bad argument");
    CCK(cudaSetDevice(c->device));
    const int B = (int)n;
    int rc = ensure_batch(*c, B);
    if (!rc) rc = ensure_grad(*c, B);
    if (rc) return rc;
    const int npix = c->cfg.box * c->cfg.box;
    cudaStream_t s = c->stream;
    if ((rc = ensure_src(*c, (size_t)npix * B))) return rc;
    cudaError_t e = cudaMemcpyAsync(c->d_src, images, sizeof(float) * (size_t)npix * B, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d_tgt, targets, sizeof(float) * NRES * B, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = forward(*c, c->d_src, nullptr, B, s);
    if (e == cudaSuccess) {
        head_kernel<<<(B + 127) / 128, 128, 0, s>>>(c->d_o, B, c->d_tgt, c->cfg.shift_weight, c->d_res, c->d_go, c->d_loss);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = backward(*c, c->d_src, nullptr, B, s);
    std::vector<float> l(B);
    if (e == cudaSuccess) e = cudaMemcpyAsync(l.data(), c->d_loss, sizeof(float) * B, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && grads) e = cudaMemcpyAsync(grads, c->d_g, sizeof(float) * c->nparams, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cfail(BSG_ERR_CUDA, "bsg_cnn_loss_grad: %s", cudaGetErrorString(e));
    if (loss) {
        double t = 0;
        for (float v : l) t += v;
        *loss = t / B;
    }
    return BSG_OK;
}

extern "C" int bsg_cnn_train(bsg_cnn* h, const float* images, const float* targets, long ndata, int steps, float lr,
                             float* losses, int flags) {
    Cnn* c = reinterpret_cast<Cnn*>(h);
    if (!c || !images || !targets || ndata < 1 || steps < 1)
        return cfail(BSG_ERR_ARG, "bsg_cnn_train: bad argument");
    if (!(flags & BSG_DEVICE_PTR))
        return cfail(BSG_ERR_ARG, "bsg_cnn_train: the training set must be on the device (BSG_DEVICE_PTR)");
    CCK(cudaSetDevice(c->device));
    const int B = std::max(1, c->cfg.batch > 0 ? c->cfg.batch : 256);
    int rc = ensure_batch(*c, B);
    if (!rc) rc = ensure_grad(*c, B);
    if (rc) return rc;
    cudaStream_t s = c->stream;
    // mini-batch indices for every step (seeded, sampled without replacement
    // within each pass over the data)
    std::vector<int> idx((size_t)steps * B);
    std::mt19937_64 rng(c->cfg.seed + 7919ull * (uint64_t)c->step);
    std::vector<int> perm(ndata);
    long pos = ndata;
    for (size_t i = 0; i < idx.size(); ++i) {
        if (pos >= ndata) {
            for (long j = 0; j < ndata; ++j) perm[j] = (int)j;
            std::shuffle(perm.begin(), perm.end(), rng);
            pos = 0;
        }
        idx[i] = perm[pos++];
    }
    int* d_all = nullptr;
    float* d_losses = nullptr;
    CCK(cudaMalloc(&d_all, sizeof(int) * idx.size()));
    CCK(cudaMalloc(&d_losses, sizeof(float) * steps));
    cudaError_t e = cudaMemcpyAsync(d_all, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, s);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int t = 0; e == cudaSuccess && t < steps; ++t) {
        const int* bi = d_all + (size_t)t * B;
        gather_rows_kernel<<<(B * NRES + 255) / 256, 256, 0, s>>>(targets, bi, B, NRES, c->d_tgt);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = forward(*c, images, bi, B, s);
        if (e == cudaSuccess) {
            head_kernel<<<(B + 127) / 128, 128, 0, s>>>(c->d_o, B, c->d_tgt, c->cfg.shift_weight, c->d_res, c->d_go,
                                                        c->d_loss);
            mean_kernel<<<1, 32, 0, s>>>(c->d_loss, B, d_losses + t);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = backward(*c, images, bi, B, s);
        if (e == cudaSuccess) {
            ++c->step;
            const float c1 = 1.f / (1.f - powf(b1, (float)c->step)), c2 = 1.f / (1.f - powf(b2, (float)c->step));
            adam_kernel<<<grid_for(c->nparams), 256, 0, s>>>(c->d_w, c->d_weff, c->d_g, c->d_m, c->d_v, c->nparams, lr,
                                                             b1, b2, eps, c1, c2);
            e = cudaGetLastError();
            if (e == cudaSuccess) e = pack_weights(*c, false, s);
        }
    }
    if (e == cudaSuccess && losses) e = cudaMemcpyAsync(losses, d_losses, sizeof(float) * steps, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d_all);
    cudaFree(d_losses);
    if (e != cudaSuccess) return cfail(BSG_ERR_CUDA, "bsg_cnn_train: %s", cudaGetErrorString(e));
    return BSG_OK;
}

namespace bsg {
namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// per image: variance of the signal inside the inscribed circle, then
// Gaussian noise of variance var / snr (Box-Muller on a counter-based hash
// of seed, image and pixel, so the result does not depend on the launch)
__global__ void __launch_bounds__(256) add_noise_kernel(float* __restrict__ img, int box, double snr, uint64_t seed) {
    __shared__ double s1[256], s2[256], s3[256];
    float* p = img + (size_t)blockIdx.x * box * box;
    const double c = box / 2.0, r2 = c * c;
    double a = 0, b = 0, n = 0;
    for (int i = threadIdx.x; i < box * box; i += 256) {
        const double dx = i % box - c, dy = i / box - c;
        if (dx * dx + dy * dy <= r2) { const double v = p[i]; a += v; b += v * v; n += 1; }
    }
    s1[threadIdx.x] = a; s2[threadIdx.x] = b; s3[threadIdx.x] = n;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if (threadIdx.x < o) {
            s1[threadIdx.x] += s1[threadIdx.x + o]; s2[threadIdx.x] += s2[threadIdx.x + o]; s3[threadIdx.x] += s3[threadIdx.x + o];
        }
        __syncthreads();
    }
    const double mean = s1[0] / s3[0], var = s2[0] / s3[0] - mean * mean;
    const double sd = var > 0 ? sqrt(var / snr) : 0.0;
    for (int i = threadIdx.x; i < box * box; i += 256) {
        const uint64_t h = mix64(seed ^ mix64(((uint64_t)blockIdx.x << 32) + (uint64_t)i + 0x9E3779B97F4A7C15ull));
        const double u1 = ((h >> 11) + 1.0) / 9007199254740993.0;
        const double u2 = (mix64(h) >> 11) / 9007199254740992.0;
        p[i] += (float)(sd * sqrt(-2.0 * log(u1)) * cos(2 * M_PI * u2));
    }
}

}  // namespace
}  // namespace bsg

extern "C" int bsg_add_noise(float* d_images, long n, int box, double snr, unsigned long long seed, void* stream) {
    if (!d_images || n < 1 || box < 2 || !(snr > 0)) return cfail(BSG_ERR_ARG, "bsg_add_noise: bad argument");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    for (long b0 = 0; b0 < n; b0 += 65535) {
        const long cnt = std::min(65535L, n - b0);
        add_noise_kernel<<<(unsigned)cnt, 256, 0, s>>>(d_images + (size_t)b0 * box * box, box, snr, seed + (uint64_t)b0);
        CCK(cudaGetLastError());
    }
    CCK(cudaStreamSynchronize(s));
    return BSG_OK;
}

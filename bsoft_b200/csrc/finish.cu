// finish.cu - from accumulated central sections to the real-space map.
// Reference steps (bsoft/src):
//   sum of partial maps + weigh   mg/mg_reconstruct.cpp:306-331,
//                                 img/Bimage_reconstruct.cpp:486-515
//   SNR (FOM) map                 img/Bimage_reconstruct.cpp:610-634
//   phase_shift_to_center         img/Bimage_complex.cpp:545-552 (= (-1)^(h+k+l))
//   fft_back (1/sqrt(N^3)), real  img/Bimage.h:903-908, Bimage_complex.cpp:170-186
//   filter_sinc (trilinear)       img/Bimage_filter.cpp:484-509
//
// Only the real part of the inverse transform is kept, and the real part of
// a transform is the transform of the Hermitian part G(v) = (F(v) +
// conj(F(-v))) / 2.  So the finish works on the half volume x = 0 .. N/2 of
// G: y lines (weighing the sums as it loads them), z lines, then x lines as
// a complex-to-real transform of half the length with the scale and the sinc
// weight.  One pass over the sums, then 8 N^3 bytes a pass.
#include "context.cuh"
#include "fft_tile.cuh"

#include <math.h>

#include <algorithm>

namespace bsg {

// Sums of one half map (vol, w), their unpaired pixels' sums below zsplit
// (e, ew; half-space accumulators) and the FOM channels (p, q).
struct HalfSums {
    const double2* vol;
    const double* w;
    const double2* e;
    const double* ew;
    const double* p;
    const double* q;
};

struct WeighArgs {
    HalfSums h[2];
    int nh;           // halves that are added
    int N;
    int zsplit;       // > 0: half-space accumulators (insert.cu walk_edges)
    float* fom;       // SNR map (snr_kernel)
};

// Index of the voxel at minus the frequency of voxel (x, y, z) (wrap-around).
__device__ __forceinline__ size_t mirror_index(size_t x, size_t y, size_t z, size_t N) {
    return ((((N - z) % N) * N + (N - y) % N) * N + (N - x) % N);
}

// One half map's sums at voxel v = (x, y, z) and at its mirror -v = (xm, ym, zm).
// Half-space accumulators (zsplit > 0) hold the paired pixels' sums P below
// zsplit, with the unpaired pixels' sums U there in (e, ew), and U alone at and
// above zsplit: the map is P(v) + U(v) below the split and conj(P(-v)) + U(v)
// above it.  Of v and -v one at least lies below (zsplit > N/2).
struct VoxelPair {
    double2 v, vm;
    double w, wm;
};

__device__ __forceinline__ VoxelPair half_pair(const HalfSums& h, int x, int y, int z, int xm, int ym, int zm, int N,
                                               int zsplit) {
    const size_t i = ((size_t)z * N + y) * N + x, m = ((size_t)zm * N + ym) * N + xm;
    VoxelPair s{h.vol[i], h.vol[m], h.w[i], h.w[m]};
    if (zsplit <= 0) return s;
    const bool low = z < zsplit, lowm = zm < zsplit;
    const double2 p = s.v, pm = s.vm;
    const double wp = s.w, wpm = s.wm;
    if (low) {
        const double2 u = h.e[i];
        s.v.x += u.x;
        s.v.y += u.y;
        s.w += h.ew[i];
    } else {
        s.v.x += pm.x;
        s.v.y -= pm.y;
        s.w += wpm;
    }
    if (lowm) {
        const double2 u = h.e[m];
        s.vm.x += u.x;
        s.vm.y += u.y;
        s.wm += h.ew[m];
    } else {
        s.vm.x += p.x;
        s.vm.y -= p.y;
        s.wm += wp;
    }
    return s;
}

// The pair's sums over the halves that are added.
__device__ __forceinline__ VoxelPair voxel_pair(const WeighArgs& a, int x, int y, int z, int xm, int ym, int zm) {
    VoxelPair s = half_pair(a.h[0], x, y, z, xm, ym, zm, a.N, a.zsplit);
    if (a.nh > 1) {
        const VoxelPair t = half_pair(a.h[1], x, y, z, xm, ym, zm, a.N, a.zsplit);
        s.v.x += t.v.x;
        s.v.y += t.v.y;
        s.w += t.w;
        s.vm.x += t.vm.x;
        s.vm.y += t.vm.y;
        s.wm += t.wm;
    }
    return s;
}

// fspace_reconstruction_weigh: the sum over the weight, as float
__device__ __forceinline__ float2 weighed(double2 v, double w) {
    if (!(w > 1e-30)) return make_float2(0.f, 0.f);
    return make_float2((float)(v.x / w), (float)(v.y / w));
}

// fspace_reconstruction_snr on the weighed channels (full-map sums: the FOM
// channels switch half-space gridding off)
__global__ void snr_kernel(WeighArgs a) {
    const size_t N = a.N, N3 = N * N * N;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N3; i += (size_t)gridDim.x * blockDim.x) {
        double2 v = a.h[0].vol[i];
        double w = a.h[0].w[i];
        if (a.nh > 1) {
            const double2 u = a.h[1].vol[i];
            v.x += u.x;
            v.y += u.y;
            w += a.h[1].w[i];
        }
        double p = a.h[0].p[i], q = a.h[0].q[i];
        if (a.nh > 1) { p += a.h[1].p[i]; q += a.h[1].q[i]; }
        const float2 F = weighed(v, w);
        if (w > 1e-30) {
            q = w - q / w;
            if (q > 1.0) p /= q;
            else if (w > 1.0) p /= w;
            if (p < 0.0) p = 0.0;
        } else {
            p = 0.0;
            w = 1e-30;
        }
        const double signal = (double)F.x * F.x + (double)F.y * F.y;
        double noise = p - signal;
        if (noise < signal) noise = signal;
        float f = 0.f;
        if (w > 1.0 && signal > 1e-30 && noise > 1e-30) f = (float)((w * signal - p) / noise);
        a.fom[i] = (i == 0) ? 1.f : f;
    }
}

// ---- 3-D inverse transform ----------------------------------------------------
//
// 384^3, both half maps and their FSC: 24.8 -> 4.3 ms; the passes were
// full complex volumes through runtime-radix line transforms (an index
// division per element and local-memory butterflies) at 1.4 TB/s.

constexpr int FIN_THREADS = 256;
// float2 between the elements of a strided tile (16 lines side by side) and
// of a transposed x tile (odd, so that a warp's consecutive elements of one
// line fall in distinct banks)
constexpr int YZ_PITCH = TILE_LINES, X_PITCH = TILE_LINES + 1;
// weigh_y's tiles: 8 lines leave room for twice the CTAs, whose loads of the
// sums it waits for, and a pitch of 9 spreads the radix-8 stages' stores over
// the banks (384^3: 16 lines 0.86, 8 lines 0.97, with the pitch 0.65 ms a map)
constexpr int W_LINES = 8, W_PITCH = 9;

struct IfftArgs {
    float2* g;         // N x N x pitch: the half volume
    const float2* tw;  // N roots
    int N, pitch;
    TilePlan plan;     // N (y, z) or N / 2 (x)
    float* out;        // x pass: the real map
    float scale;
    const double* sinc;   // weight by squared distance from the map centre, or null
};

// y lines: 8 adjacent x of one z, G formed from the sums on the way in.  Bound
// by the reads of the sums' two ends: 1.25 -> 0.65 ms a map at 384^3, half of it
// from the coordinates of -v, which 64-bit divisions of the index gave.
__global__ void __launch_bounds__(FIN_THREADS) weigh_y_kernel(const __grid_constant__ WeighArgs w,
                                                              const __grid_constant__ IfftArgs a) {
    extern __shared__ float2 sm[];
    const int N = a.N, XH = N / 2 + 1;
    float2* roots = sm;
    float2* t0 = sm + N;
    float2* t1 = t0 + N * W_PITCH;
    for (int i = threadIdx.x; i < N; i += FIN_THREADS) roots[i] = a.tw[i];
    const int x0 = blockIdx.x * W_LINES, z = blockIdx.y, zm = z ? N - z : 0;
    for (int i = threadIdx.x; i < N * W_LINES; i += FIN_THREADS) {
        const int c = i & (W_LINES - 1), y = i / W_LINES, x = x0 + c;
        float2 g = make_float2(0.f, 0.f);
        if (x < XH) {
            const int ym = y ? N - y : 0, xm = x ? N - x : 0;
            const VoxelPair q = voxel_pair(w, x, y, z, xm, ym, zm);
            const float2 f = weighed(q.v, q.w), m = weighed(q.vm, q.wm);
            // half the sum; phase_shift_to_center is (-1)^(h+k+l), the same
            // for both (signed and unsigned indices share parity for even N)
            const float s = ((x + y + z) & 1) ? -0.5f : 0.5f;
            g = make_float2(s * (f.x + m.x), s * (f.y - m.y));
        }
        t0[y * W_PITCH + c] = g;
    }
    __syncthreads();
    const float2* r = tile_fft<true, W_LINES>(t0, t1, a.plan, roots, 1, W_PITCH);
    for (int i = threadIdx.x; i < N * W_LINES; i += FIN_THREADS) {
        const int c = i & (W_LINES - 1), y = i / W_LINES, x = x0 + c;
        if (x < XH) a.g[((size_t)z * N + y) * a.pitch + x] = r[y * W_PITCH + c];
    }
}

// z lines: 16 adjacent x of one y, in place
__global__ void __launch_bounds__(FIN_THREADS) fft_z_kernel(const __grid_constant__ IfftArgs a) {
    extern __shared__ float2 sm[];
    const int N = a.N, XH = N / 2 + 1;
    float2* roots = sm;
    float2* t0 = sm + N;
    float2* t1 = t0 + N * YZ_PITCH;
    for (int i = threadIdx.x; i < N; i += FIN_THREADS) roots[i] = a.tw[i];
    const int x0 = blockIdx.x * TILE_LINES, y = blockIdx.y;
    const size_t zs = (size_t)N * a.pitch;
    float2* g = a.g + (size_t)y * a.pitch + x0;
    for (int i = threadIdx.x; i < N * TILE_LINES; i += FIN_THREADS) {
        const int c = i & (TILE_LINES - 1), z = i / TILE_LINES;
        t0[z * YZ_PITCH + c] = x0 + c < XH ? g[z * zs + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const float2* r = tile_fft<true>(t0, t1, a.plan, roots, 1, YZ_PITCH);
    for (int i = threadIdx.x; i < N * TILE_LINES; i += FIN_THREADS) {
        const int c = i & (TILE_LINES - 1), z = i / TILE_LINES;
        if (x0 + c < XH) g[z * zs + c] = r[z * YZ_PITCH + c];
    }
}

// x lines, complex to real: x[2j] + i x[2j+1] is the N/2-point transform of
// E_k + i O_k, E_k = G_k + conj(G_{N/2-k}), O_k = (G_k - conj(G_{N/2-k}))
// exp(2 pi i k / N); then the scale and the sinc weight.  16 consecutive rows
// (z, y) per CTA, a warp reading and writing one row at a time.
__global__ void __launch_bounds__(FIN_THREADS) fft_x_real_kernel(const __grid_constant__ IfftArgs a) {
    extern __shared__ float2 sm[];
    const int N = a.N, M = N / 2;
    float2* roots = sm;
    float2* t0 = sm + N;
    float2* t1 = t0 + (M + 1) * X_PITCH;
    for (int i = threadIdx.x; i < N; i += FIN_THREADS) roots[i] = a.tw[i];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long rows = (long)N * N, r0 = (long)blockIdx.x * TILE_LINES;
    for (int c = warp; c < TILE_LINES; c += FIN_THREADS / 32) {
        const float2* src = a.g + (r0 + c) * a.pitch;
        for (int k = lane; k <= M; k += 32) {
            float2 v = r0 + c < rows ? src[k] : make_float2(0.f, 0.f);
            if (k == 0 || k == M) v.y = 0.f;       // real up to rounding
            t1[k * X_PITCH + c] = v;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < M * TILE_LINES; i += FIN_THREADS) {
        const int c = i & (TILE_LINES - 1), k = i / TILE_LINES;
        const float2 p = t1[k * X_PITCH + c], q = t1[(M - k) * X_PITCH + c], w = roots[k];
        const float2 e = make_float2(p.x + q.x, p.y - q.y), d = make_float2(p.x - q.x, p.y + q.y);
        const float2 o = make_float2(d.x * w.x + d.y * w.y, d.y * w.x - d.x * w.y);   // d conj(w)
        t0[k * X_PITCH + c] = make_float2(e.x - o.y, e.y + o.x);
    }
    __syncthreads();
    const float2* r = tile_fft<true>(t0, t1, a.plan, roots, 2, X_PITCH);
    for (int c = warp; c < TILE_LINES; c += FIN_THREADS / 32) {
        const long row = r0 + c;
        if (row >= rows) break;
        const int z = (int)(row / N), y = (int)(row - (long)z * N);
        const int dy = y - M, dz = z - M, d2 = dy * dy + dz * dz;
        float2* dst = reinterpret_cast<float2*>(a.out + row * N);
        for (int j = lane; j < M; j += 32) {
            float2 v = r[j * X_PITCH + c];
            v.x *= a.scale;
            v.y *= a.scale;
            if (a.sinc) {
                const int x = 2 * j - M;
                v.x = (float)(a.sinc[d2 + x * x] * v.x);
                v.y = (float)(a.sinc[d2 + (x + 1) * (x + 1)] * v.y);
            }
            dst[j] = v;
        }
    }
}

// filter_sinc: r = pi |d|, d = (index - N/2) / N, weight (r / sin r)^2, by
// the squared distance in voxels (0 .. 3 (N/2)^2)
__global__ void sinc_table_kernel(double* t, int N) {
    const int n = 3 * (N / 2) * (N / 2) + 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double rr = 3.14159265358979323846 * (sqrt((double)i) / N);
        const double w = i ? rr / sin(rr) : 1.0;
        t[i] = w * w;
    }
}

cudaError_t launch_sinc_table(double* t, int N, cudaStream_t s) {
    sinc_table_kernel<<<64, 256, 0, s>>>(t, N);
    return cudaGetLastError();
}

static HalfSums half_sums(const Context& c, int h) {
    return HalfSums{c.d_vol[h], c.d_w[h], c.d_evol[h], c.d_ew[h], c.d_pow[h], c.d_w2[h]};
}

static WeighArgs weigh_args(const Context& c, int imap) {
    WeighArgs w{};
    w.N = c.g.map;
    w.zsplit = c.zsplit;
    w.nh = 1;
    w.h[0] = half_sums(c, c.nhalves == 2 && imap > 0 ? imap - 1 : 0);
    if (c.nhalves == 2 && imap == 0) {
        w.h[1] = half_sums(c, 1);
        w.nh = 2;
    }
    return w;
}

static size_t yz_smem(int N) { return sizeof(float2) * ((size_t)N + 2 * (size_t)N * YZ_PITCH); }
static size_t weigh_smem(int N) { return sizeof(float2) * ((size_t)N + 2 * (size_t)N * W_PITCH); }
static size_t x_smem(int N) { return sizeof(float2) * ((size_t)N + 2 * (size_t)(N / 2 + 1) * X_PITCH); }

// Map imap (0: the halves added) of the context's sums: weighed, transformed,
// scaled and, with sinc, weighted, into map_out; the SNR map into d_fom when
// the context keeps its channels.  *launches: kernels launched.
cudaError_t launch_finish(const Context& c, int imap, float* map_out, bool sinc, int* launches, cudaStream_t s) {
    const int N = c.g.map, XH = N / 2 + 1;
    WeighArgs w = weigh_args(c, imap);
    *launches = 3;
    cudaError_t e;
    if (c.g.fom) {
        w.fom = c.d_fom;
        snr_kernel<<<148 * 8, 256, 0, s>>>(w);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *launches = 4;
    }
    IfftArgs a{};
    a.g = c.d_work;
    a.tw = c.d_twmap;
    a.N = N;
    // whole 32-byte sectors per row
    a.pitch = (XH + 3) / 4 * 4;
    if (!tile_plan(N, &a.plan)) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)((XH + TILE_LINES - 1) / TILE_LINES), (unsigned)N);
    weigh_y_kernel<<<dim3((unsigned)((XH + W_LINES - 1) / W_LINES), (unsigned)N), FIN_THREADS, weigh_smem(N), s>>>(w, a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    fft_z_kernel<<<grid, FIN_THREADS, yz_smem(N), s>>>(a);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (!tile_plan(N / 2, &a.plan)) return cudaErrorInvalidValue;
    a.out = map_out;
    a.scale = (float)(1.0 / sqrt((double)N * N * N));
    a.sinc = sinc ? c.d_sinc : nullptr;
    fft_x_real_kernel<<<(unsigned)(((long)N * N + TILE_LINES - 1) / TILE_LINES), FIN_THREADS, x_smem(N), s>>>(a);
    return cudaGetLastError();
}

// Half-space accumulators -> the map's sums (half_pair), into (dv, dw); in
// place (dv == vol) too: the voxels at and above zsplit are written first,
// from the paired sums below it, then (e, ew) is added below it.
__global__ void map_sums_upper_kernel(double2* dv, double* dw, const double2* vol, const double* w, int N,
                                      int zsplit) {
    const size_t n = N, n2 = n * n, first = (size_t)zsplit * n2, N3 = n2 * n;
    for (size_t i = first + blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N3;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t m = mirror_index(i % n, (i / n) % n, i / n2, n);
        const double2 u = vol[m];
        double2 v = vol[i];
        v.x += u.x;
        v.y -= u.y;
        dv[i] = v;
        dw[i] = w[i] + w[m];
    }
}

__global__ void map_sums_lower_kernel(double2* dv, double* dw, const double2* vol, const double* w,
                                      const double2* e, const double* ew, size_t count) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x) {
        double2 v = vol[i];
        const double2 u = e[i];
        v.x += u.x;
        v.y += u.y;
        dv[i] = v;
        dw[i] = w[i] + ew[i];
    }
}

cudaError_t launch_map_sums(double2* dv, double* dw, const double2* vol, const double* w, const double2* e,
                            const double* ew, int N, int zsplit, cudaStream_t s) {
    if (zsplit <= 0) return cudaSuccess;
    map_sums_upper_kernel<<<148 * 8, 256, 0, s>>>(dv, dw, vol, w, N, zsplit);
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    map_sums_lower_kernel<<<148 * 8, 256, 0, s>>>(dv, dw, vol, w, e, ew, (size_t)zsplit * N * N);
    return cudaGetLastError();
}

// FSC partial sums as Bimage::fsc(Bimage*) forms them
// (bsoft/src/img/Bimage_resolution.cpp:330-406 with fspace_radial_power,
// Bimage_fspace.cpp:848-958): radius = real * |index / real| (wrapped at
// (N-1)/2), a voxel adds (1 - f) to shell floor(radius) and f to the next,
// only voxels with floor(radius) < maxrad count.  The weighed values come
// straight from the sums (the centre shift's sign leaves F1 conj(F2) and
// |F|^2 unchanged).
//
// A warp takes rows (z, y), 32 values of h >= 0 at a time with their mates
// -(h, k, l), which have the same radius.  Along a row the radius grows by
// less than 1 a step, so the lanes of a shell are consecutive: a segmented
// scan sums them and the last lane of a run adds it to the warp's shells in
// shared memory.  Rows, warps and CTAs in fixed order: deterministic, FP64
// throughout.  Bound by the FP64 pipe and the reads of the sums; a thread per
// shell scanning a whole plane (384 CTAs, every voxel's square root two to
// four times) took 5.4 ms at 384^3 after 2.0 ms of weighing, now 1.7.
__device__ __forceinline__ double fsc_radius(int h, int k, int l, double real) {
    const double fs = 1.0 / real;
    double rx = h * fs, ry = k * fs, rz = l * fs;
    rx *= rx; ry *= ry; rz *= rz;
    return real * sqrt(rx + ry + rz);
}

constexpr int FSC_WARPS = 8;

struct FscArgs {
    WeighArgs w[2];
    int N, ns, maxrad;     // ns: shells kept
    double real;
    double* part;          // CTAs x ns x 3
};

__global__ void __launch_bounds__(FSC_WARPS * 32) fsc_rows_kernel(const __grid_constant__ FscArgs a) {
    extern __shared__ double shells[];        // FSC_WARPS x ns x 3
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* my = shells + (size_t)warp * a.ns * 3;
    for (int i = lane; i < a.ns * 3; i += 32) my[i] = 0.0;
    __syncwarp();
    const int N = a.N, rows = N * N, H = N / 2;
    for (int row = blockIdx.x * FSC_WARPS + warp; row < rows; row += gridDim.x * FSC_WARPS) {
        const int z = row / N, y = row - z * N, zm = z ? N - z : 0, ym = y ? N - y : 0;
        const int k = sfreq(y, N), l = sfreq(z, N);
        for (int h0 = 0; h0 <= H; h0 += 32) {
            const int h = h0 + lane;
            const double rad = fsc_radius(h, k, l, a.real);
            int ir = (int)rad;
            const bool in = h <= H && ir < a.maxrad;
            if (!__any_sync(0xffffffffu, in)) break;            // the radius only grows
            double num = 0, d1 = 0, d2 = 0;
            if (in) {
                const int hm = h ? N - h : 0;
                const VoxelPair q1 = voxel_pair(a.w[0], h, y, z, hm, ym, zm), q2 = voxel_pair(a.w[1], h, y, z, hm, ym, zm);
                for (int m = 0; m < 2; ++m) {
                    if (m && (h == 0 || h == H)) continue;       // its mate is another row's
                    const float2 f1 = m ? weighed(q1.vm, q1.wm) : weighed(q1.v, q1.w);
                    const float2 f2 = m ? weighed(q2.vm, q2.wm) : weighed(q2.v, q2.w);
                    num += (double)f1.x * f2.x + (double)f1.y * f2.y;
                    d1 += (double)f1.x * f1.x + (double)f1.y * f1.y;
                    d2 += (double)f2.x * f2.x + (double)f2.y * f2.y;
                }
            } else {
                ir = -1;
            }
            const double f = rad - ir;
            double s[6] = {num * (1.0 - f), d1 * (1.0 - f), d2 * (1.0 - f), num * f, d1 * f, d2 * f};
            if (!in)
#pragma unroll
                for (int q = 0; q < 6; ++q) s[q] = 0.0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int other = __shfl_up_sync(0xffffffffu, ir, o);
                const bool add = lane >= o && other == ir;
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const double t = __shfl_up_sync(0xffffffffu, s[q], o);
                    if (add) s[q] += t;
                }
            }
            const int next = __shfl_down_sync(0xffffffffu, ir, 1);
            const bool last = in && (lane == 31 || next != ir);
            if (last && ir < a.ns)
#pragma unroll
                for (int q = 0; q < 3; ++q) my[ir * 3 + q] += s[q];
            __syncwarp();
            if (last && ir + 1 < a.ns)
#pragma unroll
                for (int q = 0; q < 3; ++q) my[(ir + 1) * 3 + q] += s[3 + q];
            __syncwarp();
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.ns * 3; i += FSC_WARPS * 32) {
        double t = 0;
        for (int w = 0; w < FSC_WARPS; ++w) t += shells[(size_t)w * a.ns * 3 + i];
        a.part[(size_t)blockIdx.x * a.ns * 3 + i] = t;
    }
}

// FSC[0] = 1 (the reference sets it), FSC[r] = num / sqrt(d1 d2), 0 where
// not finite or beyond maxrad.  One warp per shell: the CTAs' sums lane by
// lane, then a fixed tree.
__global__ void fsc_reduce_kernel(const double* part, int parts, int ns, int nshell, int maxrad, double* fsc) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= nshell) return;
    double num = 0, d1 = 0, d2 = 0;
    if (r < ns)
        for (int z = lane; z < parts; z += 32) {
            const double* o = part + ((size_t)z * ns + r) * 3;
            num += o[0]; d1 += o[1]; d2 += o[2];
        }
    for (int o = 16; o; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        d1 += __shfl_xor_sync(0xffffffffu, d1, o);
        d2 += __shfl_xor_sync(0xffffffffu, d2, o);
    }
    if (lane) return;
    double v = 0;
    if (r == 0) v = 1;
    else if (r < maxrad) {
        v = num / sqrt(d1 * d2);
        if (!isfinite(v)) v = 0;
    }
    fsc[r] = v;
}

// shells that a voxel can reach: at most sqrt(3) N / 2, and the next
static int fsc_shells(const Context& c, int nshell) { return std::min(nshell, (int)(0.8661 * c.g.map) + 2); }
static int fsc_ctas(const Context& c) { return std::min(148 * 2, (c.g.map * c.g.map + FSC_WARPS - 1) / FSC_WARPS); }

size_t fsc_part_elems(const Context& c, int nshell) { return (size_t)fsc_ctas(c) * fsc_shells(c, nshell) * 3; }

cudaError_t launch_fsc(const Context& c, int nshell, double* part, double* out_dev, cudaStream_t s) {
    FscArgs a{};
    a.w[0] = weigh_args(c, 1);
    a.w[1] = weigh_args(c, 2);
    a.N = c.g.map;
    a.ns = fsc_shells(c, nshell);
    // fspace_maximum_radius (Bimage_fspace.cpp:26-38), sampling ratio 1
    a.real = c.g.map * c.cfg.map_sampling;
    a.maxrad = c.cfg.hi_res > 0.1 ? (int)(long)(a.real / c.cfg.hi_res) : c.g.map / 2;
    a.part = part;
    const int ctas = fsc_ctas(c);
    fsc_rows_kernel<<<ctas, FSC_WARPS * 32, sizeof(double) * 3 * FSC_WARPS * a.ns, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    fsc_reduce_kernel<<<(nshell + 7) / 8, 256, 0, s>>>(part, ctas, a.ns, nshell, a.maxrad, out_dev);
    return cudaGetLastError();
}

cudaError_t prepare_finish_attributes() {
    const int most = 512;
    cudaError_t e = cudaFuncSetAttribute(weigh_y_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)yz_smem(most));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fft_z_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)yz_smem(most));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fft_x_real_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x_smem(most));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fsc_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double) * 3 * FSC_WARPS * 512));
    return e;
}

}  // namespace bsg

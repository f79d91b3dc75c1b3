// search.cu - exhaustive orientation search on sm_100a: every held particle
// image (at every trial origin) against a panel of central sections, scored
// by a BF16 correlation on the tensor cores (tcgen05, FP32 accumulators in
// TMEM), the best candidates of each image rescored with the exact FRC
// figure of merit of the reference (img_recip_space_fom).
//
// The reference refines locally (img_refine_grid, bsoft/src/mg/mg_refine.cpp:
// 1086-1195) and scores each hypothesis with img_recip_space_fom (:660-781):
//   FRC = (1/n_f) sum_j  sum_{p in j} Re(X_p conj(R_p) c_p)
//                        / sqrt(sum_{p in j} |X_p|^2  sum_{p in j} |R_p c_p|^2)
// over shells j < max_rad.  Written as one dot product per (image, section)
// pair it becomes a GEMM when the mixed term sum |R_p|^2 c_p^2 is split as
// (sum |R_p|^2) * mean_j(c_p^2), exact when the CTF is constant on a shell:
//   A[row = (image, origin)][p] = X_p e^{i phi_origin(p)} c_p / (n_f sqrt(D_j C_j))
//   B[col = section][p]         = R_p / sqrt(M_j)
// with D_j, C_j, M_j the shell sums of |X|^2, mean c^2, |R|^2 over the
// Hermitian half plane (the full-plane sums are twice these).  Complex
// products are real dot products of interleaved (re, im) pairs, so K = 2 x
// the half-plane pixels below max_rad, padded to 64.
//
// GEMM (C = A B^T, both K-major BF16): 128 x 256 output tiles, K-blocks of
// 64 staged by TMA (128-byte swizzle) through a 4-deep shared-memory ring;
// one elected thread issues tcgen05.mma (M=128, N=256, K=16) into one of two
// 256-column TMEM accumulators while four epilogue warps read the other with
// tcgen05.ld and keep each row's 8 best columns in registers.  The M tiles
// are taken in groups (search_runs.h; short panels are cut into runs instead); the CTAs of a group are a grid of its M tiles by
// stretches of N, so that those of one stretch read the same B tiles at the
// same time and all share the group's A tiles through L2.  Groups of 21, seven
// and four M tiles (7, 21 and 37 stretches) keep 147 and 148 of the 148 SMs at
// work, and the stretches' lengths, which differ by one tile, alternate from
// group to group.  Larger groups read B from HBM fewer times, which the power
// cap rewards; the A tiles of 21 fit L2 at 128^2.  256 images x 25 origins
// against 68,520 sections, the whole call: ten M tiles x 15 stretches as 150
// work items a group (the last of six rounds nearly empty) 7.70, sevens and
// fours 7.21, with 21s 7.04 ms; 2,048 images against 550,320 sections: 523,
// 568 and 522 ms of GEMM.  One run of tiles per CTA regardless of the
// stretches, evener still, 7.70: B is then read by one CTA at a time.  A CTA
// carries its rows' top-8 along its stretch.  Every wait is bounded (2 s) and reports through a status word.
#include "match.cuh"
#include "search_runs.h"

#include <cuda.h>
#include <cuda_bf16.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

namespace bsg {

namespace {

constexpr int BM = 128, BN = 256, BK = 64, STAGES = 4, TOPK = 8;
constexpr int A_STAGE = BM * BK * 2;          // 16 KB
constexpr int B_STAGE = BN * BK * 2;          // 32 KB
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int GEMM_THREADS = 192;             // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
constexpr int GEMM_SMEM = STAGES * STAGE_BYTES + 1024;
constexpr uint64_t WAIT_NS = 2000000000ull;   // bounded waits: 2 s

// instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t gtime() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// wait for the phase of `parity` to complete; false after WAIT_NS or when
// another role has given up
__device__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = gtime();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try(bar, parity)) return true;
        if ((it & 127) == 0) {
            if (*abort_flag) return false;
            if (gtime() - t0 > WAIT_NS) { *abort_flag = 1; return false; }
        }
    }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
        "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(IDESC), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms
// 1024 bytes apart (SBO), version 1, base offset 0 (stage buffers are
// 1024-byte aligned)
__device__ __forceinline__ uint64_t sdesc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

struct GemmArgs {
    int kblocks;          // K / 64
    int ncols;            // valid columns (sections)
    Runs runs;            // the batch's M tiles by ceil(ncols / 256) N tiles
    long prow;            // row stride of the partial buffers (batch height)
    float* part_score;    // [slot][prow][TOPK]
    int* part_idx;
    int* status;
};

// keep the 8 largest (value, column) of a row, sorted descending
struct Top8 {
    float s[TOPK];
    int i[TOPK];
    __device__ __forceinline__ void reset() {
#pragma unroll
        for (int t = 0; t < TOPK; ++t) { s[t] = -3.0e38f; i[t] = -1; }
    }
    __device__ __forceinline__ void push(float v, int c) {
        if (!(v > s[TOPK - 1])) return;
        s[TOPK - 1] = v;
        i[TOPK - 1] = c;
#pragma unroll
        for (int t = TOPK - 1; t > 0; --t) {
            if (s[t] > s[t - 1]) {
                const float ts = s[t]; s[t] = s[t - 1]; s[t - 1] = ts;
                const int ti = i[t]; i[t] = i[t - 1]; i[t - 1] = ti;
            }
        }
    }
};

__global__ void __launch_bounds__(GEMM_THREADS, 1)
search_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs a) {
    extern __shared__ uint8_t gsm_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], tfull_bar[2], tempty_bar[2], drain_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(gsm_raw) + 1023u) & ~1023u;   // 1024-aligned stage ring
    const Runs runs = a.runs;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(smem_u32(&full_bar[s]), 1); mbar_init(smem_u32(&empty_bar[s]), 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(smem_u32(&tfull_bar[s]), 1); mbar_init(smem_u32(&tempty_bar[s]), 4); }
        mbar_init(smem_u32(&drain_bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {   // TMEM: two 256-column fp32 accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    volatile int* abort_v = &abort_flag;

    if (warp == 0) {
        // ---- TMA producer ----
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmA) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&tmB) : "memory");
            uint32_t stage = 0, phase = 0;
            uint32_t issued_mask = 0, last_parity = 0;   // per stage: ever issued, parity of its last load
            bool ok = true;
            for (int g = 0; ok && g < runs.groups; ++g) {
                int mtile, n0, n1;
                if (!runs.work(g, blockIdx.x, mtile, n0, n1)) continue;
                for (int nt = n0; ok && nt < n1; ++nt) {
                    for (int kb = 0; kb < a.kblocks; ++kb) {
                        if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, abort_v)) { ok = false; break; }
                        const uint32_t fb = smem_u32(&full_bar[stage]);
                        mbar_expect_tx(fb, STAGE_BYTES);
                        const uint32_t sa = base + stage * STAGE_BYTES;
                        tma_load_2d(sa, &tmA, fb, kb * BK, mtile * BM);
                        tma_load_2d(sa + A_STAGE, &tmB, fb, kb * BK, nt * BN);
                        issued_mask |= 1u << stage;
                        last_parity = (last_parity & ~(1u << stage)) | (phase << stage);
                        if (++stage == STAGES) { stage = 0; phase ^= 1; }
                    }
                }
            }
            if (!ok) {
                // let the copies already issued land before the CTA can exit:
                // the phase of each stage's last load completes with its bytes
                for (int s = 0; s < STAGES; ++s) {
                    if (!(issued_mask >> s & 1)) continue;
                    const uint32_t par = (last_parity >> s) & 1;
                    const uint64_t t0 = gtime();
                    while (!mbar_try(smem_u32(&full_bar[s]), par) && gtime() - t0 < WAIT_NS) {
                    }
                }
                atomicOr(a.status, 1);
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer (one thread) ----
        if (lane == 0) {
            uint32_t stage = 0, phase = 0, acc = 0, aphase = 0;
            bool ok = true;
            for (int g = 0; ok && g < runs.groups; ++g) {
                int mtile, n0, n1;
                if (!runs.work(g, blockIdx.x, mtile, n0, n1)) continue;
                for (int nt = n0; ok && nt < n1; ++nt) {
                    if (!mbar_wait(smem_u32(&tempty_bar[acc]), aphase ^ 1, abort_v)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t d = tmem + acc * BN;
                    for (int kb = 0; kb < a.kblocks; ++kb) {
                        if (!mbar_wait(smem_u32(&full_bar[stage]), phase, abort_v)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t sa = base + stage * STAGE_BYTES, sb = sa + A_STAGE;
#pragma unroll
                        for (int kk = 0; kk < BK / 16; ++kk)
                            tc_mma(d, sdesc(sa + kk * 32), sdesc(sb + kk * 32), (kb | kk) ? 1u : 0u);
                        tc_commit(smem_u32(&empty_bar[stage]));   // frees the stage when these MMAs finish
                        if (++stage == STAGES) { stage = 0; phase ^= 1; }
                    }
                    if (!ok) break;
                    tc_commit(smem_u32(&tfull_bar[acc]));         // accumulator ready
                    if (++acc == 2) { acc = 0; aphase ^= 1; }
                }
            }
            if (!ok) {
                // every MMA issued so far must finish before TMEM is released
                tc_commit(smem_u32(&drain_bar));
                const uint64_t t0 = gtime();
                while (!mbar_try(smem_u32(&drain_bar), 0) && gtime() - t0 < WAIT_NS) {
                }
                atomicOr(a.status, 2);
            }
        }
    } else {
        // ---- epilogue: warps 2..5, TMEM lane quarter = warp % 4 ----
        const int quarter = warp & 3;
        const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
        uint32_t acc = 0, aphase = 0;
        Top8 top;
        bool ok = true;
        for (int g = 0; ok && g < runs.groups; ++g) {
            int mtile, n0, n1;
            if (!runs.work(g, blockIdx.x, mtile, n0, n1)) continue;
            top.reset();
            for (int nt = n0; nt < n1; ++nt) {
                // one lane waits, the warp follows it (tcgen05.ld is warp-collective)
                int w = 1;
                if (lane == 0) w = mbar_wait(smem_u32(&tfull_bar[acc]), aphase, abort_v) ? 1 : 0;
                w = __shfl_sync(0xffffffffu, w, 0);
                if (!w) { ok = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem + lane_off + acc * BN;
                for (int c = 0; c < BN; c += 32) {
                    uint32_t v[32];
                    tc_ld32(taddr + c, v);
                    const int col0 = nt * BN + c;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (col0 + j < a.ncols) top.push(__uint_as_float(v[j]), col0 + j);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tempty_bar[acc]));
                if (++acc == 2) { acc = 0; aphase ^= 1; }
            }
            if (!ok) break;
            const long row = (long)mtile * BM + quarter * 32 + lane;
            const long o = ((long)runs.slot(g, blockIdx.x) * a.prow + row) * TOPK;
#pragma unroll
            for (int t = 0; t < TOPK; ++t) { a.part_score[o + t] = top.s[t]; a.part_idx[o + t] = top.i[t]; }
        }
        if (!ok && lane == 0) atomicOr(a.status, 4);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---- panel and rows ---------------------------------------------------------

// one CTA per section: FSI-kernel gather of the coarse pixels (FP64
// accumulation), per-shell norms, BF16 row of interleaved (re, im)
__global__ void __launch_bounds__(256) panel_kernel(cudaTextureObject_t tex, int D,
                                                    const float* __restrict__ lut_g, int wd,
                                                    const MPix* __restrict__ cpix, int ncpix,
                                                    const int* __restrict__ cstart, int nf,
                                                    const MHyp* __restrict__ secs, double inv, double real, int kpad,
                                                    __nv_bfloat16* __restrict__ panel) {
    extern __shared__ float psm[];
    float* lut = psm;                                                // (NDIV+1)*MAXW
    float2* vals = reinterpret_cast<float2*>(psm + (NDIV + 1) * MAXW);   // ncpix
    float* gn = reinterpret_cast<float*>(vals + ncpix);              // nf
    for (int i = threadIdx.x; i < (NDIV + 1) * wd; i += blockDim.x) lut[i] = lut_g[i];
    __syncthreads();
    const MHyp& V = secs[blockIdx.x];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int p = warp; p < ncpix; p += 8) {
        const MPix q = cpix[p];
        const double ix = q.h * inv, iy = q.k * inv;
        const double mx = (V.m[0] * ix + V.m[1] * iy) * real;
        const double my = (V.m[3] * ix + V.m[4] * iy) * real;
        const double mz = (V.m[6] * ix + V.m[7] * iy) * real;
        float vr, vi;
        fsi_gather<float>(TexSrc{tex}, D, mx, my, mz, lut, wd, lane, vr, vi);
        if (lane == 0) vals[p] = make_float2(vr, vi);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < nf; j += blockDim.x) {
        float m = 0.f;
        for (int p = cstart[j]; p < cstart[j + 1]; ++p) m += vals[p].x * vals[p].x + vals[p].y * vals[p].y;
        gn[j] = m > 0.f ? rsqrtf(m) : 0.f;
    }
    __syncthreads();
    __nv_bfloat162* row = reinterpret_cast<__nv_bfloat162*>(panel + (size_t)blockIdx.x * kpad);
    for (int p = threadIdx.x; p < kpad / 2; p += blockDim.x) {
        float2 v = make_float2(0.f, 0.f);
        if (p < ncpix) {
            const float g = gn[cpix[p].shell];
            v = make_float2(vals[p].x * g, vals[p].y * g);
        }
        row[p] = __floats2bfloat162_rn(v.x, v.y);
    }
}

// per image of the batch: 1 / (n_f sqrt(D_j C_j)) per coarse shell.  All threads
// fetch the pixels' terms, NORM_PIX at a time, and a thread per shell adds them
// in pixel order (a thread per shell that fetched them itself waited for each
// pixel in turn: 512 images of 128^2 32 us, now 20).
constexpr int NORM_PIX = 1024;
constexpr int NORM_SHELLS = 2;             // shells per thread and pass (up to box 512 there are fewer than 512)

__global__ void __launch_bounds__(256) coarse_norm_kernel(const float2* __restrict__ spec, int D,
                                                          const float* __restrict__ ctf, int npix,
                                                          const MPix* __restrict__ cpix, const int* __restrict__ cstart,
                                                          int nf, long img0, float* __restrict__ gA) {
    __shared__ double2 term[NORM_PIX];
    const long img = img0 + blockIdx.x;
    const float2* X = spec + img * (long)D * D;
    const float* C = ctf + img * (long)npix;
    const int total = cstart[nf];
    for (int j0 = 0; j0 < nf; j0 += 256 * NORM_SHELLS) {
        int lo[NORM_SHELLS], hi[NORM_SHELLS];
        double d[NORM_SHELLS], c2[NORM_SHELLS];
#pragma unroll
        for (int i = 0; i < NORM_SHELLS; ++i) {
            const int j = j0 + threadIdx.x + 256 * i;
            lo[i] = j < nf ? cstart[j] : 0;
            hi[i] = j < nf ? cstart[j + 1] : 0;
            d[i] = c2[i] = 0;
        }
        for (int b = 0; b < total; b += NORM_PIX) {
            const int m = min(NORM_PIX, total - b);
#pragma unroll 4
            for (int p = threadIdx.x; p < m; p += 256) {
                const MPix q = cpix[b + p];
                const float2 x = X[q.idx];
                const double c = C[q.pad];
                term[p] = make_double2((double)x.x * x.x + (double)x.y * x.y, c * c);
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < NORM_SHELLS; ++i) {
                const int p1 = min(hi[i] - b, m);
#pragma unroll 8
                for (int p = max(lo[i] - b, 0); p < p1; ++p) {
                    const double2 t = term[p];
                    d[i] += t.x;
                    c2[i] += t.y;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < NORM_SHELLS; ++i) {
            const int j = j0 + threadIdx.x + 256 * i, n = hi[i] - lo[i];
            if (j >= nf) continue;
            const double den = n > 0 ? d[i] * (c2[i] / n) : 0.0;
            gA[(long)blockIdx.x * nf + j] = den > 0 ? (float)(1.0 / (nf * sqrt(den))) : 0.f;
        }
    }
}

// one CTA per row (image, origin): X e^{i phi} c g as BF16 (re, im) pairs
__global__ void __launch_bounds__(256) rows_kernel(const float2* __restrict__ spec, int D, const float* __restrict__ ctf,
                                                   int npix, const MPix* __restrict__ cpix, int ncpix, int nf,
                                                   const float* __restrict__ gA, const double2* __restrict__ slopes,
                                                   int nshift, long img0, int kpad, __nv_bfloat16* __restrict__ A) {
    const int row = blockIdx.x;
    const int b = row / nshift, s = row - b * nshift;
    const long img = img0 + b;
    const float2* X = spec + img * (long)D * D;
    const float* C = ctf + img * (long)npix;
    const float* g = gA + (long)b * nf;
    const double2 sl = slopes[s];
    __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(A + (size_t)row * kpad);
    for (int p = threadIdx.x; p < kpad / 2; p += blockDim.x) {
        float2 v = make_float2(0.f, 0.f);
        if (p < ncpix) {
            const MPix q = cpix[p];
            const float2 x = X[q.idx];
            double phi = q.h * sl.x + q.k * sl.y;
            phi -= 6.283185307179586 * rint(phi * 0.15915494309189535);
            float sn, cs;
            sincosf((float)phi, &sn, &cs);
            const float f = C[q.pad] * g[q.shell];
            v = make_float2((x.x * cs - x.y * sn) * f, (x.x * sn + x.y * cs) * f);
        }
        out[p] = __floats2bfloat162_rn(v.x, v.y);
    }
}

// One CTA per image: the topk best of the partial candidates of its nshift rows
// in (score descending, section, origin) order.  A candidate is one number
// that sorts that way (64 bits; 128 when sections x origins exceed 32).  Each
// thread reads its share once and keeps the TOPK best of it in registers, in
// order; a pick is the largest of the threads' first ones.  Bound by the reads'
// latency, hence 1,024 threads for a few images.  (256 images of 25 origins:
// read again for every pick by one warp per image 0.42 ms, by 256 threads from
// shared memory 0.07, now 0.04; 5 images against 8,580 sections, 0.84 by the
// warp, 0.08 with 148 places a row, most of them empty, now 34 and 0.02.)
constexpr int MERGE_MOST = 1024;

typedef unsigned __int128 wide_t;

__device__ __forceinline__ unsigned long long shfl_xor_key(unsigned long long v, int o) {
    return __shfl_xor_sync(0xffffffffu, v, o);
}
__device__ __forceinline__ wide_t shfl_xor_key(wide_t v, int o) {
    return (wide_t)__shfl_xor_sync(0xffffffffu, (unsigned long long)(v >> 64), o) << 64 |
           __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
}

// K: score in the upper half, the inverted section x origin number in the lower
template <class K>
__global__ void __launch_bounds__(sizeof(K) == 8 ? MERGE_MOST : MERGE_MOST / 2)
    merge_kernel(const float* __restrict__ ps, const int* __restrict__ pi, Runs runs, long mrows, int nshift, int topk,
                 long img0, int* __restrict__ cand_sec, int* __restrict__ cand_org, float* __restrict__ cand_score) {
    constexpr int HALF = 4 * sizeof(K);
    constexpr K LOW = ((K)1 << HALF) - 1;
    __shared__ K best[2][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    K top[TOPK];                                 // this thread's best, largest first
#pragma unroll
    for (int i = 0; i < TOPK; ++i) top[i] = 0;
    // a row's slots and places, a row after the other: thread t takes every
    // blockDim.x-th of the image's candidates
    int e = threadIdx.x, s = 0;
    long row = (long)blockIdx.x * nshift;
    int n = runs.slots((int)(row / BM)) * TOPK;
    while (s < nshift) {
        if (e >= n) {
            e -= n;
            if (++s == nshift) break;
            ++row;
            if (row % BM == 0) n = runs.slots((int)(row / BM)) * TOPK;
            continue;
        }
        const int r = e / TOPK;
        const long o = ((long)r * mrows + row) * TOPK + e % TOPK;
        const int sec = __ldg(pi + o);
        const float score = __ldg(ps + o);
        if (sec >= 0) {
            unsigned u = __float_as_uint(score);
            u ^= (u >> 31) ? 0xffffffffu : 0x80000000u;         // sorts as the float does
            K v = (K)u << HALF | (LOW - ((K)sec * nshift + s));
            if (v > top[TOPK - 1]) {
#pragma unroll
                for (int i = 0; i < TOPK; ++i)
                    if (v > top[i]) { const K w = top[i]; top[i] = v; v = w; }
            }
        }
        e += blockDim.x;
    }
    for (int t = 0; t < topk; ++t) {
        K b = top[0];
        for (int o = 16; o; o >>= 1) {
            const K v = shfl_xor_key(b, o);
            if (v > b) b = v;
        }
        if (lane == 0) best[t & 1][warp] = b;
        __syncthreads();
        b = lane < nwarps ? best[t & 1][lane] : (K)0;
        for (int o = 16; o; o >>= 1) {
            const K v = shfl_xor_key(b, o);
            if (v > b) b = v;
        }
        if (b && top[0] == b) {
#pragma unroll
            for (int i = 0; i + 1 < TOPK; ++i) top[i] = top[i + 1];
            top[TOPK - 1] = 0;
        }
        if (threadIdx.x == 0) {
            const long c = (img0 + blockIdx.x) * topk + t;
            const long key = (long)(LOW - (b & LOW));
            unsigned u = (unsigned)(b >> HALF);
            u ^= (u >> 31) ? 0x80000000u : 0xffffffffu;
            cand_sec[c] = b ? (int)(key / nshift) : -1;
            cand_org[c] = b ? (int)(key % nshift) : -1;
            cand_score[c] = b ? __uint_as_float(u) : -3.0e38f;
        }
    }
}


// ---- local search around proposals -----------------------------------------

constexpr int LOCAL_MAXC = 1024;    // candidate sections per image
constexpr int LOCAL_MAXO = 9;       // trial origins per image

// IMG images per CTA: the panel sections whose rotation lies within the angle
// whose cosine bound is `tr_min` of trace(R_p^T R_s), in panel order.  rots: nine
// rows of nsec elements.  The warps take 32 sections each in turn and leave a
// bit per section and image; then WPI warps per image count their words and
// write the sections out, a segment of SEL_WORDS words at a time.  Bound by the
// loads of the rotations: as 36-byte records, one image per CTA and a barrier
// per 256 sections, 512 images against 68,520 sections took 0.21 ms (now
// 0.06).
constexpr int SEL_THREADS = 1024;
constexpr int SEL_WORDS = 4096;

template <int IMG>
__global__ void __launch_bounds__(SEL_THREADS) local_select_kernel(const float* __restrict__ prop,
                                                                   const float* __restrict__ rots, long nsec,
                                                                   float tr_min, long img0, int nimg, int words,
                                                                   int* __restrict__ cand, int* __restrict__ count) {
    constexpr int WARPS = SEL_THREADS / 32, WPI = WARPS / IMG;
    extern __shared__ unsigned s_bits[];               // IMG x words
    __shared__ int s_sum[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int first = blockIdx.x * IMG;
    float R[IMG][9];
#pragma unroll
    for (int i = 0; i < IMG; ++i)
#pragma unroll
        for (int k = 0; k < 9; ++k) R[i][k] = prop[(img0 + min(first + i, nimg - 1)) * 11 + k];
    const int mine = warp / WPI, part = warp - mine * WPI;
    int* out = cand + (long)(first + mine) * LOCAL_MAXC;
    int base = 0;                                      // sections of earlier segments
    for (long seg = 0; seg < nsec; seg += 32L * words) {
        const int here = (int)min((long)words, (nsec - seg + 31) / 32);
#pragma unroll 2
        for (int w = warp; w < here; w += WARPS) {
            const long j = seg + 32L * w + lane;
            const bool live = j < nsec;
            float r[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) r[k] = live ? __ldg(rots + k * nsec + j) : 0.f;
#pragma unroll
            for (int i = 0; i < IMG; ++i) {
                float t = 0.f;
#pragma unroll
                for (int k = 0; k < 9; ++k) t = fmaf(R[i][k], r[k], t);
                const unsigned b = __ballot_sync(0xffffffffu, live && t >= tr_min);
                if (lane == 0) s_bits[i * words + w] = b;
            }
        }
        __syncthreads();
        const unsigned* bits = s_bits + mine * words;
        const int per = (here + WPI - 1) / WPI, w0 = min(here, part * per), w1 = min(here, w0 + per);
        int n = 0;
        for (int w = w0 + lane; w < w1; w += 32) n += __popc(bits[w]);
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) s_sum[warp] = n;
        __syncthreads();
        int at = base;
        for (int q = 0; q < WPI; ++q) {
            const int v = s_sum[mine * WPI + q];
            if (q < part) at += v;
            base += v;
        }
        if (n > 0 && first + mine < nimg)
            for (int wb = w0; wb < w1; wb += 32) {
                unsigned word = wb + lane < w1 ? bits[wb + lane] : 0u;
                const int c = __popc(word);
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                for (int pos = at + incl - c; word && pos < LOCAL_MAXC; ++pos) {
                    out[pos] = (int)(seg + 32L * (wb + lane) + __ffs(word) - 1);
                    word &= word - 1;
                }
                at += __shfl_sync(0xffffffffu, incl, 31);
            }
        __syncthreads();                               // before the next segment's bits
    }
    if (part == 0 && lane == 0 && first + mine < nimg) count[first + mine] = base;
}

__device__ __forceinline__ float2 bf2f(uint32_t u) {
    return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}

// per image: its A rows at its local origins in shared memory (BF16, as
// rows_kernel writes them), then the candidate sections' panel rows dotted with
// them, a warp taking two sections and LOCAL_O origins at a time; the topk
// (section, origin) pairs by score go to the candidate arrays in (score desc,
// section, origin) order.  A lane's products of one pair are added in the order
// of the row, whatever the split.  The A rows fill an SM's shared memory for
// large boxes (115 KB at 128^2 and half the Nyquist frequency), so one CTA has
// to bring enough warps: 256 threads, one section at a time with all nine
// origins and a single warp's search for the best pairs took 0.77 ms for 512
// images of 128^2 (now 0.18).
constexpr int LOCAL_O = 3;
constexpr int LOCAL_THREADS = 1024;
constexpr int LOCAL_SMEM = 227 * 1024 - 512;       // dynamic, beside the picks' 512 bytes (rows of 10,816 values at most)

__global__ void __launch_bounds__(LOCAL_THREADS, 1) local_score_kernel(
    const float2* __restrict__ spec, int D, const float* __restrict__ ctf, int npix, const MPix* __restrict__ cpix,
    int ncpix, int nf, const float* __restrict__ gA, const double2* __restrict__ slopes,
    const int* __restrict__ lorg, const int* __restrict__ nlorg, const int* __restrict__ cand,
    const int* __restrict__ count, const __nv_bfloat16* __restrict__ panel, int kpad, int topk, long img0,
    int* __restrict__ out_sec, int* __restrict__ out_org, float* __restrict__ out_score) {
    extern __shared__ uint4 lsm[];
    __shared__ unsigned long long best[64];
    const int b = blockIdx.x;
    const long img = img0 + b;
    const int no = nlorg[b];
    const int nc = min(count[b], LOCAL_MAXC);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    __nv_bfloat162* A = reinterpret_cast<__nv_bfloat162*>(lsm);           // no x kpad/2
    float* sc = reinterpret_cast<float*>(A + (size_t)LOCAL_MAXO * (kpad / 2));   // LOCAL_MAXC x LOCAL_MAXO
    double2* s_slope = reinterpret_cast<double2*>(sc);                    // before the scores
    if (threadIdx.x < no) s_slope[threadIdx.x] = slopes[lorg[b * LOCAL_MAXO + threadIdx.x]];
    __syncthreads();
    const float2* X = spec + img * (long)D * D;
    const float* C = ctf + img * (long)npix;
    const float* g = gA + (long)b * nf;
    for (int p = threadIdx.x; p < kpad / 2; p += blockDim.x) {
        MPix q = {};
        float2 x = make_float2(0.f, 0.f);
        float f = 0.f;
        const bool live = p < ncpix;
        if (live) {
            q = cpix[p];
            x = X[q.idx];
            f = C[q.pad] * g[q.shell];
        }
        for (int o = 0; o < no; ++o) {
            float2 v = make_float2(0.f, 0.f);
            if (live) {
                const double2 sl = s_slope[o];
                double phi = q.h * sl.x + q.k * sl.y;
                phi -= 6.283185307179586 * rint(phi * 0.15915494309189535);
                float sn, cs;
                sincosf((float)phi, &sn, &cs);
                v = make_float2((x.x * cs - x.y * sn) * f, (x.x * sn + x.y * cs) * f);
            }
            A[(size_t)o * (kpad / 2) + p] = __floats2bfloat162_rn(v.x, v.y);
        }
    }
    __syncthreads();
    const int n = nc * LOCAL_MAXO;
    for (int e = threadIdx.x; e < n; e += blockDim.x) sc[e] = __int_as_float(0x7fffffff);    // no such origin
    __syncthreads();
    const uint4* As = reinterpret_cast<const uint4*>(A);
    const int k8 = kpad / 8;                 // 16-byte chunks per row
    const int og = (no + LOCAL_O - 1) / LOCAL_O, items = (nc + 1) / 2 * og;
    for (int it = warp; it < items; it += nwarps) {
        const int pair = it / og, o0 = (it - pair * og) * LOCAL_O;
        const int c0 = 2 * pair, c1 = min(c0 + 1, nc - 1);
        const uint4* r0 = reinterpret_cast<const uint4*>(panel + (size_t)cand[(long)b * LOCAL_MAXC + c0] * kpad);
        const uint4* r1 = reinterpret_cast<const uint4*>(panel + (size_t)cand[(long)b * LOCAL_MAXC + c1] * kpad);
        float acc[2][LOCAL_O];
#pragma unroll
        for (int o = 0; o < LOCAL_O; ++o) acc[0][o] = acc[1][o] = 0.f;
#pragma unroll 2
        for (int p = lane; p < k8; p += 32) {
            const uint4 p0 = __ldg(r0 + p), p1 = __ldg(r1 + p);
            const float2 b0[4] = {bf2f(p0.x), bf2f(p0.y), bf2f(p0.z), bf2f(p0.w)};
            const float2 b1[4] = {bf2f(p1.x), bf2f(p1.y), bf2f(p1.z), bf2f(p1.w)};
#pragma unroll
            for (int o = 0; o < LOCAL_O; ++o) {
                const uint4 ab = As[(size_t)min(o0 + o, no - 1) * k8 + p];
                const float2 a[4] = {bf2f(ab.x), bf2f(ab.y), bf2f(ab.z), bf2f(ab.w)};
                float t = acc[0][o], u = acc[1][o];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t = fmaf(a[k].x, b0[k].x, t); t = fmaf(a[k].y, b0[k].y, t);
                    u = fmaf(a[k].x, b1[k].x, u); u = fmaf(a[k].y, b1[k].y, u);
                }
                acc[0][o] = t;
                acc[1][o] = u;
            }
        }
#pragma unroll
        for (int o = 0; o < LOCAL_O; ++o) {
            float t = acc[0][o], u = acc[1][o];
#pragma unroll
            for (int k = 16; k; k >>= 1) {
                t += __shfl_xor_sync(0xffffffffu, t, k);
                u += __shfl_xor_sync(0xffffffffu, u, k);
            }
            if (lane == 0 && o0 + o < no) {
                sc[c0 * LOCAL_MAXO + o0 + o] = t;
                if (c1 > c0) sc[c1 * LOCAL_MAXO + o0 + o] = u;
            }
        }
    }
    __syncthreads();
    // A pair as one number that sorts in the order of the picks (the candidates
    // are in section order), 0 for none; each pick is the largest below the last.
    auto key = [&](int e) -> unsigned long long {
        const float v = sc[e];
        if (!(v >= -3.0e38f && v <= 3.0e38f)) return 0ull;
        unsigned u = __float_as_uint(v + 0.f);
        u ^= (u >> 31) ? 0xffffffffu : 0x80000000u;
        return (unsigned long long)u << 32 | (0xffffffffu - (unsigned)e);
    };
    unsigned long long prev = ~0ull;
    for (int t = 0; t < topk; ++t) {
        unsigned long long top = 0;
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const unsigned long long v = key(e);
            if (v < prev && v > top) top = v;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, top, o);
            if (v > top) top = v;
        }
        if (lane == 0) best[(t & 1) * 32 + warp] = top;
        __syncthreads();
        top = lane < nwarps ? best[(t & 1) * 32 + lane] : 0ull;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const unsigned long long v = __shfl_xor_sync(0xffffffffu, top, o);
            if (v > top) top = v;
        }
        if (threadIdx.x == 0) {
            const long c = img * topk + t;
            const int e = (int)(0xffffffffu - (unsigned)top);
            out_sec[c] = top ? cand[(long)b * LOCAL_MAXC + e / LOCAL_MAXO] : -1;
            out_org[c] = top ? lorg[b * LOCAL_MAXO + e % LOCAL_MAXO] : -1;
            out_score[c] = top ? sc[e] : -3.0e38f;
        }
        prev = top;                                    // (0: nothing is left)
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// K-major BF16 matrix [rows][kpad] with a box of 64 x box_rows, 128B swizzle
bool make_map(CUtensorMap* m, const void* ptr, long rows, int kpad, int box_rows) {
    EncodeTiledFn f = encode_fn();
    if (!f) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)kpad * 2};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

std::once_flag g_search_attr;
cudaError_t g_search_attr_err = cudaSuccess;

}  // namespace

// the coarse pixel list: half plane (k > 0, or k == 0 and h > 0), shells
// 1 .. n_f - 1, inside the section limit; .pad = index in the full list
static void coarse_pixels(Match& M) {
    M.h_cpix.clear();
    M.h_cstart.assign(M.nf + 1, 0);
    for (size_t i = 0; i < M.h_pix.size(); ++i) {
        MPix q = M.h_pix[i];
        if (q.shell < 1 || q.shell >= M.nf || !q.insec) continue;
        if (!(q.k > 0 || (q.k == 0 && q.h > 0))) continue;
        q.pad = (int)i;
        M.h_cpix.push_back(q);
        M.h_cstart[q.shell + 1]++;
    }
    for (int j = 0; j < M.nf; ++j) M.h_cstart[j + 1] += M.h_cstart[j];
    M.ncpix = (int)M.h_cpix.size();
    M.kpad = ((2 * M.ncpix + BK - 1) / BK) * BK;
}


// exact rescoring of the candidates in d_csec / d_corg / d_cscore (topk per
// held image): candidates of one image that share a section form one group
// (one gather, several origins); out gets each image's candidates ordered
// by the exact figure of merit
static cudaError_t rescore_candidates(Match& Mr, int topk, const std::vector<double2>& sl, double* out, float* tres,
                                      long* ngroups) {
    Match* M = &Mr;
    cudaStream_t s = M->stream;
    cudaError_t e = cudaSuccess;
    const long ncand = M->nimg * topk;
    std::vector<int> csec(ncand), corg(ncand);
    std::vector<float> cscore(ncand);
    e = cudaMemcpyAsync(csec.data(), M->d_csec, sizeof(int) * ncand, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(corg.data(), M->d_corg, sizeof(int) * ncand, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(cscore.data(), M->d_cscore, sizeof(float) * ncand, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    // groups of one image and one section (up to MAXORG origins), built per
    // image from the section index (the candidates of an image are adjacent)
    std::vector<MHypG> groups;
    std::vector<int> gsec;
    std::vector<long> cslot(ncand, -1);
    groups.reserve(ncand);
    for (long i = 0; i < M->nimg; ++i) {
        const size_t g0 = groups.size();
        for (int t = 0; t < topk; ++t) {
            const long c = i * topk + t;
            if (csec[c] < 0) continue;
            size_t g = groups.size();
            for (size_t q = g0; q < groups.size(); ++q)
                if (gsec[q] == csec[c] && groups[q].norg < MAXORG) { g = q; break; }
            if (g == groups.size()) {
                MHypG ng;
                memset(&ng, 0, sizeof(ng));
                memcpy(ng.m, M->h_secs[csec[c]].m, sizeof(ng.m));
                ng.img = (int)i;
                ng.ctf = (int)i;
                ng.sec = csec[c];          // row of the panel's exact sections
                groups.push_back(ng);
                gsec.push_back(csec[c]);
            }
            MHypG& G = groups[g];
            G.sx[G.norg] = sl[corg[c]].x;
            G.sy[G.norg] = sl[corg[c]].y;
            cslot[c] = (long)g * MAXORG + G.norg;
            G.norg++;
        }
    }
    const long ng = (long)groups.size();
    *ngroups = ng;
    std::vector<double> cf(2 * ncand, 0.0);
    *tres = 0;
    if (ng > 0) {
        if (ensure_groups(*M, ng) != BSG_OK) return cudaErrorMemoryAllocation;
        std::vector<double> go(2 * ng * MAXORG);
        cudaEvent_t e0, e1;
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        e = cudaMemcpyAsync(M->d_grp, groups.data(), sizeof(MHypG) * ng, cudaMemcpyHostToDevice, s);
        cudaEventRecord(e0, s);
        if (e == cudaSuccess)
            e = launch_fom(*M, M->d_grp, ng, M->d_gout, M->d_gout + ng * MAXORG, s, false, nullptr, nullptr, false,
                           M->d_pexact);
        cudaEventRecord(e1, s);
        if (e == cudaSuccess) e = cudaMemcpyAsync(go.data(), M->d_gout, sizeof(double) * go.size(), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        cudaEventElapsedTime(tres, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (e != cudaSuccess) return e;
        for (long c = 0; c < ncand; ++c) {
            if (cslot[c] < 0) continue;
            cf[c] = go[cslot[c]];
            cf[ncand + c] = go[ng * MAXORG + cslot[c]];
        }
    }
    for (long i = 0; i < M->nimg; ++i) {
        int ord[TOPK];
        const long b = i * topk;
        auto before = [&](int x, int y) {
            const bool vx = csec[b + x] >= 0, vy = csec[b + y] >= 0;
            if (vx != vy) return vx;
            return cf[b + x] > cf[b + y];
        };
        for (int t = 0; t < topk; ++t) {
            int j = t;
            for (; j > 0 && before(t, ord[j - 1]); --j) ord[j] = ord[j - 1];
            ord[j] = t;
        }
        for (int t = 0; t < topk; ++t) {
            const long c = b + ord[t];
            double* o = out + (b + t) * BSG_MATCH_RESULT_DOUBLES;
            o[0] = csec[c];
            o[1] = corg[c];
            o[2] = cscore[c];
            o[3] = csec[c] >= 0 ? cf[c] : 0.0;
            o[4] = csec[c] >= 0 ? cf[ncand + c] : 0.0;
        }
    }
    return cudaSuccess;
}

}  // namespace bsg

using namespace bsg;

extern "C" int bsg_match_set_panel(bsg_match* h, const double* mats, long nsec, int flags) {
    Match* M = reinterpret_cast<Match*>(h);
    if (!M || !mats || nsec < 1) return match_fail(BSG_ERR_ARG, "bsg_match_set_panel: bad argument");
    if (!M->have_ref) return match_fail(BSG_ERR_STATE, "bsg_match_set_panel: set the reference first");
    cudaError_t e = cudaSetDevice(M->device);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_set_panel: %s", cudaGetErrorString(e));
    std::call_once(g_search_attr, [] {
        g_search_attr_err = cudaFuncSetAttribute(search_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM);
        if (g_search_attr_err == cudaSuccess)
            g_search_attr_err = cudaFuncSetAttribute(panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    });
    if (g_search_attr_err != cudaSuccess)
        return match_fail(BSG_ERR_CUDA, "bsg_match_set_panel: %s", cudaGetErrorString(g_search_attr_err));
    coarse_pixels(*M);
    const size_t psmem = sizeof(float) * (NDIV + 1) * MAXW + sizeof(float2) * M->ncpix + sizeof(float) * M->nf;
    if (psmem > 200 * 1024) return match_fail(BSG_ERR_ARG, "bsg_match_set_panel: %d coarse pixels exceed the panel kernel's shared memory", M->ncpix);
    cudaStream_t s = M->stream;
    // release an older panel first
    cudaFree(M->d_panel); M->d_panel = nullptr;
    cudaFree(M->d_secs); M->d_secs = nullptr;
    cudaFree(M->d_cpix); M->d_cpix = nullptr;
    cudaFree(M->d_cstart); M->d_cstart = nullptr;
    cudaFree(M->d_rots); M->d_rots = nullptr;
    cudaFree(M->d_pexact); M->d_pexact = nullptr;
    M->nsec = 0;
    std::vector<MHyp> sv(nsec);
    for (long v = 0; v < nsec; ++v) {
        memset(&sv[v], 0, sizeof(MHyp));
        match_view_rows(*M, mats + 9 * v, sv[v].m);
    }
    e = cudaMalloc(&M->d_panel, sizeof(__nv_bfloat16) * (size_t)nsec * M->kpad);
    if (e == cudaSuccess) e = cudaMalloc(&M->d_secs, sizeof(MHyp) * nsec);
    if (e == cudaSuccess) e = cudaMalloc(&M->d_cpix, sizeof(MPix) * std::max(1, M->ncpix));
    if (e == cudaSuccess) e = cudaMalloc(&M->d_cstart, sizeof(int) * (M->nf + 1));
    if (e == cudaSuccess) e = cudaMalloc(&M->d_rots, sizeof(float) * 9 * nsec);
    if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_set_panel: %ld sections: %s", nsec, cudaGetErrorString(e));
    e = cudaMemcpyAsync(M->d_secs, sv.data(), sizeof(MHyp) * nsec, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(M->d_cpix, M->h_cpix.data(), sizeof(MPix) * M->ncpix, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(M->d_cstart, M->h_cstart.data(), sizeof(int) * (M->nf + 1), cudaMemcpyHostToDevice, s);
    {
        std::vector<float> rf((size_t)9 * nsec);
        for (long i = 0; i < nsec; ++i)
            for (int k = 0; k < 9; ++k) rf[k * nsec + i] = (float)mats[9 * i + k];
        if (e == cudaSuccess) e = cudaMemcpyAsync(M->d_rots, rf.data(), sizeof(float) * rf.size(), cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    for (long v0 = 0; e == cudaSuccess && v0 < nsec; v0 += 1L << 20) {
        const long cnt = std::min(nsec - v0, 1L << 20);
        panel_kernel<<<(unsigned)cnt, 256, psmem, s>>>(M->ref_tex, M->D, M->d_lutf, M->wd, M->d_cpix, M->ncpix, M->d_cstart,
                                                       M->nf, M->d_secs + v0, 1.0 / M->real_map, M->real_map, M->kpad,
                                                       M->d_panel + (size_t)v0 * M->kpad);
        e = cudaGetLastError();
    }
    cudaEventRecord(e1, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_set_panel: %s", cudaGetErrorString(e));
    M->nsec = nsec;
    M->h_secs.swap(sv);
    M->sstats.panel_ms += ms;
    M->sstats.launches += (nsec + (1L << 20) - 1) >> 20;
    // the panel's FP32 sections at the figure-of-merit pixels, kept for the
    // exact rescoring when they fit with 8 GB to spare (else the rescoring
    // gathers them per candidate)
    if (!(flags & BSG_MATCH_PANEL_GATHER)) {
        const size_t bytes = sizeof(float2) * (size_t)nsec * M->h_pix.size();
        size_t freeb = 0, total = 0;
        if (cudaMemGetInfo(&freeb, &total) == cudaSuccess && bytes + (8ull << 30) < freeb &&
            cudaMalloc(&M->d_pexact, bytes) == cudaSuccess) {
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
            cudaEventRecord(e0, s);
            e = launch_panel_exact(*M, M->d_secs, nsec, M->d_pexact, s);
            cudaEventRecord(e1, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            float xms = 0;
            cudaEventElapsedTime(&xms, e0, e1);
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            if (e != cudaSuccess) {
                cudaFree(M->d_pexact);
                M->d_pexact = nullptr;
                return match_fail(BSG_ERR_CUDA, "bsg_match_set_panel: exact sections: %s", cudaGetErrorString(e));
            }
            M->sstats.panel_exact_ms += xms;
            M->sstats.panel_exact_bytes = (double)bytes;
            M->sstats.launches += (nsec + (1L << 20) - 1) >> 20;
        } else {
            cudaGetLastError();     // a failed allocation leaves no sticky error; clear the last one
            M->sstats.panel_exact_bytes = 0;
        }
    }
    return BSG_OK;
}

extern "C" int bsg_match_search(bsg_match* h, const double* origins, int norigin, int topk, double* out, int flags) {
    (void)flags;
    Match* M = reinterpret_cast<Match*>(h);
    if (!M || !origins || !out || norigin < 1 || topk < 1 || topk > TOPK)
        return match_fail(BSG_ERR_ARG, "bsg_match_search: bad argument (topk must be 1..%d)", TOPK);
    if (M->nsec < 1 || M->nimg < 1) return match_fail(BSG_ERR_STATE, "bsg_match_search: set the panel and the images first");
    cudaError_t e = cudaSetDevice(M->device);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search: %s", cudaGetErrorString(e));
    cudaStream_t s = M->stream;
    const int nf = M->nf, kpad = M->kpad;
    // images per batch: rows of A (image x origin) up to ~256 MB
    const long row_bytes = 2L * kpad;
    long nb = std::max(1L, std::min<long>(M->nimg, (256L << 20) / (row_bytes * norigin)));
    if (M->cfg.batch > 0) nb = std::min<long>(nb, M->cfg.batch);
    const long rows_max = nb * norigin;
    const long mrows = ((rows_max + BM - 1) / BM) * BM;
    const int mtiles_max = (int)(mrows / BM);
    const int ntiles = (int)((M->nsec + BN - 1) / BN);
    const Runs full = Runs::plan(mtiles_max, ntiles);
    const long tail_rows = ((M->nimg - 1) % nb + 1) * norigin;             // the last batch
    const Runs tail = Runs::plan((int)((tail_rows + BM - 1) / BM), ntiles);
    long slots = 1;
    for (const Runs* r : {&full, &tail})
        for (int m = 0; m < r->mtiles; ++m) slots = std::max(slots, (long)r->slots(m));

    // scratch (kept between calls)
    const size_t need_A = (size_t)mrows * kpad;
    const size_t need_part = (size_t)slots * mrows * TOPK;
    const size_t need_cand = (size_t)M->nimg * topk;
    if (need_A > M->a_elems) {
        cudaFree(M->d_A); M->d_A = nullptr; M->a_elems = 0;
        e = cudaMalloc(&M->d_A, sizeof(__nv_bfloat16) * need_A);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
        M->a_elems = need_A;
    }
    if (need_part > M->part_elems) {
        cudaFree(M->d_pscore); cudaFree(M->d_pidx); M->d_pscore = nullptr; M->d_pidx = nullptr; M->part_elems = 0;
        e = cudaMalloc(&M->d_pscore, sizeof(float) * need_part);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_pidx, sizeof(int) * need_part);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
        M->part_elems = need_part;
    }
    if (need_cand > M->cand_elems) {
        cudaFree(M->d_csec); cudaFree(M->d_corg); cudaFree(M->d_cscore);
        M->d_csec = nullptr; M->d_corg = nullptr; M->d_cscore = nullptr;
        M->cand_elems = 0;
        e = cudaMalloc(&M->d_csec, sizeof(int) * need_cand);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_corg, sizeof(int) * need_cand);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_cscore, sizeof(float) * need_cand);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
        M->cand_elems = need_cand;
    }
    if (M->gA_elems < (size_t)nb * nf) {
        cudaFree(M->d_gA); M->d_gA = nullptr;
        e = cudaMalloc(&M->d_gA, sizeof(float) * nb * nf);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
        M->gA_elems = (size_t)nb * nf;
    }
    if (M->slope_elems < (size_t)norigin) {
        cudaFree(M->d_slopes); M->d_slopes = nullptr;
        e = cudaMalloc(&M->d_slopes, sizeof(double2) * norigin);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
        M->slope_elems = norigin;
    }
    if (!M->d_status) {
        e = cudaMalloc(&M->d_status, sizeof(int));
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search: %s", cudaGetErrorString(e));
    }
    // phase slopes of each trial origin (pixels of the uncut image, scaled
    // with the cut as change_transform_size does, then 2 pi o / diam)
    std::vector<double2> sl(norigin);
    for (int i = 0; i < norigin; ++i)
        sl[i] = make_double2(M->cut_scale * origins[2 * i] / M->D * 2 * M_PI, M->cut_scale * origins[2 * i + 1] / M->D * 2 * M_PI);
    e = cudaMemcpyAsync(M->d_slopes, sl.data(), sizeof(double2) * norigin, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(M->d_status, 0, sizeof(int), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(M->d_A, 0, sizeof(__nv_bfloat16) * need_A, s);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search: %s", cudaGetErrorString(e));

    CUtensorMap tmA, tmB;
    if (!make_map(&tmA, M->d_A, mrows, kpad, BM) || !make_map(&tmB, M->d_panel, M->nsec, kpad, BN))
        return match_fail(BSG_ERR_CUDA, "bsg_match_search: cuTensorMapEncodeTiled failed");

    cudaEvent_t ev[5];
    for (auto& x : ev) cudaEventCreate(&x);
    double agen = 0, gemm = 0, merge = 0;
    long launches = 0;
    for (long i0 = 0; e == cudaSuccess && i0 < M->nimg; i0 += nb) {
        const long cnt = std::min(nb, M->nimg - i0);
        const long rows = cnt * norigin;
        cudaEventRecord(ev[0], s);
        coarse_norm_kernel<<<(unsigned)cnt, 256, 0, s>>>(M->d_spec, M->D, M->d_ctf, (int)M->h_pix.size(), M->d_cpix,
                                                         M->d_cstart, nf, i0, M->d_gA);
        rows_kernel<<<(unsigned)rows, 256, 0, s>>>(M->d_spec, M->D, M->d_ctf, (int)M->h_pix.size(), M->d_cpix, M->ncpix,
                                                    nf, M->d_gA, M->d_slopes, norigin, i0, kpad, M->d_A);
        if (rows < mrows && i0 > 0)
            cudaMemsetAsync(M->d_A + (size_t)rows * kpad, 0, sizeof(__nv_bfloat16) * (mrows - rows) * kpad, s);
        cudaEventRecord(ev[1], s);
        GemmArgs ga{};
        ga.kblocks = kpad / BK;
        ga.ncols = (int)M->nsec;
        ga.runs = Runs::plan((int)((rows + BM - 1) / BM), ntiles);
        ga.prow = mrows;
        ga.part_score = M->d_pscore;
        ga.part_idx = M->d_pidx;
        ga.status = M->d_status;
        search_gemm_kernel<<<ga.runs.ctas, GEMM_THREADS, GEMM_SMEM, s>>>(tmA, tmB, ga);
        cudaEventRecord(ev[2], s);
        // two CTAs of half the threads share an SM (256 images 38 against 45 us, 16 images 29 against 26)
        const int half = MERGE_MOST / 2, threads = cnt > 148 ? half : MERGE_MOST;
        if (M->nsec * (long)norigin < 0xffffffffL)
            merge_kernel<unsigned long long><<<(unsigned)cnt, threads, 0, s>>>(
                M->d_pscore, M->d_pidx, ga.runs, mrows, norigin, topk, i0, M->d_csec, M->d_corg, M->d_cscore);
        else
            merge_kernel<wide_t><<<(unsigned)cnt, half, 0, s>>>(
                M->d_pscore, M->d_pidx, ga.runs, mrows, norigin, topk, i0, M->d_csec, M->d_corg, M->d_cscore);
        cudaEventRecord(ev[3], s);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaEventSynchronize(ev[3]);
        float t01 = 0, t12 = 0, t23 = 0;
        cudaEventElapsedTime(&t01, ev[0], ev[1]);
        cudaEventElapsedTime(&t12, ev[1], ev[2]);
        cudaEventElapsedTime(&t23, ev[2], ev[3]);
        agen += t01;
        gemm += t12;
        merge += t23;
        launches += 4;
        int st = 0;
        if (e == cudaSuccess) e = cudaMemcpy(&st, M->d_status, sizeof(int), cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && st) {
            for (auto& x : ev) cudaEventDestroy(x);
            return match_fail(BSG_ERR_CUDA, "bsg_match_search: the correlation kernel gave up waiting (status %d)", st);
        }
        M->sstats.gemm_flops += 2.0 * (double)rows * (double)M->nsec * (double)(2 * M->ncpix);
    }
    for (auto& x : ev) cudaEventDestroy(x);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search: %s", cudaGetErrorString(e));
    float tres = 0;
    long ng = 0;
    e = rescore_candidates(*M, topk, sl, out, &tres, &ng);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search: %s", cudaGetErrorString(e));
    const long ncand = M->nimg * topk;
    M->sstats.agen_ms += agen;
    M->sstats.gemm_ms += gemm;
    M->sstats.merge_ms += merge;
    M->sstats.rescore_ms += tres;
    M->sstats.launches += launches + (ng > 0 ? 1 : 0);
    M->sstats.gemm_launches += launches / 4;
    M->sstats.images += M->nimg;
    M->sstats.hypotheses += (double)M->nimg * norigin * (double)M->nsec;
    M->sstats.rescored += ncand;
    return BSG_OK;
}

extern "C" int bsg_match_get_stats(bsg_match* h, bsg_match_stats* st) {
    Match* M = reinterpret_cast<Match*>(h);
    if (!M || !st) return match_fail(BSG_ERR_ARG, "bsg_match_get_stats: null argument");
    *st = M->sstats;
    st->coarse_k = 2 * M->ncpix;
    st->kpad = M->kpad;
    return BSG_OK;
}

extern "C" int bsg_match_reset_stats(bsg_match* h) {
    Match* M = reinterpret_cast<Match*>(h);
    if (!M) return match_fail(BSG_ERR_ARG, "bsg_match_reset_stats: null argument");
    memset(&M->sstats, 0, sizeof(M->sstats));
    return BSG_OK;
}

extern "C" void* bsg_match_stream(bsg_match* h) {
    Match* M = reinterpret_cast<Match*>(h);
    return M ? static_cast<void*>(M->stream) : nullptr;
}

extern "C" int bsg_match_search_local(bsg_match* h, const float* proposals, double radius, const double* origins,
                                      int norigin, double origin_radius, int topk, double* out, int flags) {
    (void)flags;
    Match* M = reinterpret_cast<Match*>(h);
    if (!M || !proposals || !origins || !out || norigin < 1 || topk < 1 || topk > TOPK || !(radius > 0))
        return match_fail(BSG_ERR_ARG, "bsg_match_search_local: bad argument (topk must be 1..%d)", TOPK);
    if (M->nsec < 1 || M->nimg < 1) return match_fail(BSG_ERR_STATE, "bsg_match_search_local: set the panel and the images first");
    cudaError_t e = cudaSetDevice(M->device);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search_local: %s", cudaGetErrorString(e));
    static std::once_flag once;
    static cudaError_t attr = cudaSuccess;
    std::call_once(once, [] {
        attr = cudaFuncSetAttribute(local_score_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LOCAL_SMEM);
        if (attr == cudaSuccess)
            attr = cudaFuncSetAttribute(local_select_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(unsigned) * 4 * SEL_WORDS);
    });
    const size_t lsmem = sizeof(__nv_bfloat16) * (size_t)LOCAL_MAXO * M->kpad + sizeof(float) * LOCAL_MAXC * LOCAL_MAXO;
    if (attr != cudaSuccess || lsmem > LOCAL_SMEM)
        return match_fail(BSG_ERR_ARG, "bsg_match_search_local: %d coarse values per row exceed the kernel's shared memory",
                          M->kpad);
    cudaStream_t s = M->stream;
    const long nimg = M->nimg;
    const int nf = M->nf;
    // (the proposals are on the host too, for the choice of the trial origins)
    std::vector<float> prop((size_t)nimg * 11);
    e = cudaMemcpy(prop.data(), proposals, sizeof(float) * prop.size(),
                   (flags & BSG_DEVICE_PTR) ? cudaMemcpyDeviceToHost : cudaMemcpyHostToHost);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search_local: %s", cudaGetErrorString(e));
    std::vector<double2> sl(norigin);
    for (int i = 0; i < norigin; ++i)
        sl[i] = make_double2(M->cut_scale * origins[2 * i] / M->D * 2 * M_PI, M->cut_scale * origins[2 * i + 1] / M->D * 2 * M_PI);
    const long nb = std::max(1L, std::min<long>(nimg, M->cfg.batch > 0 ? M->cfg.batch : 4096));
    // scratch
    const size_t need_cand = (size_t)nimg * topk;
    if (need_cand > M->cand_elems) {
        cudaFree(M->d_csec); cudaFree(M->d_corg); cudaFree(M->d_cscore);
        M->d_csec = nullptr; M->d_corg = nullptr; M->d_cscore = nullptr;
        M->cand_elems = 0;
        e = cudaMalloc(&M->d_csec, sizeof(int) * need_cand);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_corg, sizeof(int) * need_cand);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_cscore, sizeof(float) * need_cand);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search_local: %s", cudaGetErrorString(e));
        M->cand_elems = need_cand;
    }
    if (M->gA_elems < (size_t)nb * nf) {
        cudaFree(M->d_gA); M->d_gA = nullptr;
        e = cudaMalloc(&M->d_gA, sizeof(float) * nb * nf);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search_local: %s", cudaGetErrorString(e));
        M->gA_elems = (size_t)nb * nf;
    }
    if (M->slope_elems < (size_t)norigin) {
        cudaFree(M->d_slopes); M->d_slopes = nullptr;
        e = cudaMalloc(&M->d_slopes, sizeof(double2) * norigin);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search_local: %s", cudaGetErrorString(e));
        M->slope_elems = norigin;
    }
    // scratch kept in the context (grow-only): no allocation per call
    if (M->lscr_img < nimg) {
        cudaFree(M->d_lprop); cudaFree(M->d_lorg); cudaFree(M->d_nlorg);
        M->d_lprop = nullptr; M->d_lorg = nullptr; M->d_nlorg = nullptr;
        M->lscr_img = 0;
        e = cudaMalloc(&M->d_lprop, sizeof(float) * 11 * nimg);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_lorg, sizeof(int) * LOCAL_MAXO * nimg);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_nlorg, sizeof(int) * nimg);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search_local: %s", cudaGetErrorString(e));
        M->lscr_img = nimg;
    }
    if (M->lscr_nb < nb) {
        cudaFree(M->d_lcand); cudaFree(M->d_lcount);
        M->d_lcand = nullptr; M->d_lcount = nullptr;
        M->lscr_nb = 0;
        e = cudaMalloc(&M->d_lcand, sizeof(int) * nb * LOCAL_MAXC);
        if (e == cudaSuccess) e = cudaMalloc(&M->d_lcount, sizeof(int) * nb);
        if (e != cudaSuccess) return match_fail(BSG_ERR_NOMEM, "bsg_match_search_local: %s", cudaGetErrorString(e));
        M->lscr_nb = nb;
    }
    float* d_prop = M->d_lprop;
    int *d_lorg = M->d_lorg, *d_nlorg = M->d_nlorg, *d_cand = M->d_lcand, *d_count = M->d_lcount;
    e = cudaMemcpyAsync(d_prop, prop.data(), sizeof(float) * prop.size(), cudaMemcpyHostToDevice, s);
    const float tr_min = (float)(1.0 + 2.0 * cos(radius));
    cudaEvent_t ev[2];
    cudaEventCreate(&ev[0]);
    cudaEventCreate(&ev[1]);
    cudaEventRecord(ev[0], s);
    // Four images per CTA once that fills the SMs: the rotations are read once
    // for them (512 images against 68,520 sections 176 us with one, 61
    // with four; 64 images 34 and 54).
    const int words = (int)std::min<long>(SEL_WORDS, (M->nsec + 31) / 32);
    auto select = [&](long i0, long cnt) {
        if (cnt > 148)
            local_select_kernel<4><<<(unsigned)((cnt + 3) / 4), SEL_THREADS, sizeof(unsigned) * 4 * words, s>>>(
                d_prop, M->d_rots, M->nsec, tr_min, i0, (int)cnt, words, d_cand, d_count);
        else
            local_select_kernel<1><<<(unsigned)cnt, SEL_THREADS, sizeof(unsigned) * words, s>>>(
                d_prop, M->d_rots, M->nsec, tr_min, i0, (int)cnt, words, d_cand, d_count);
        coarse_norm_kernel<<<(unsigned)cnt, 256, 0, s>>>(M->d_spec, M->D, M->d_ctf, (int)M->h_pix.size(), M->d_cpix,
                                                         M->d_cstart, nf, i0, M->d_gA);
        return cudaGetLastError();
    };
    if (e == cudaSuccess) e = select(0, std::min(nb, nimg));
    // meanwhile, the local trial origins of each image: those within
    // origin_radius of the proposed origin (box centre + proposed shift), nearest
    // first, at most LOCAL_MAXO
    std::vector<int> lorg((size_t)nimg * LOCAL_MAXO, 0), nlorg(nimg, 0);
    for (long i = 0; i < nimg; ++i) {
        const double px = M->n / 2 + prop[i * 11 + 9], py = M->n / 2 + prop[i * 11 + 10];
        double d[LOCAL_MAXO];
        int* at = &lorg[i * LOCAL_MAXO];
        int k = 0;
        for (int o = 0; o < norigin; ++o) {
            const double dx = origins[2 * o] - px, dy = origins[2 * o + 1] - py, v = dx * dx + dy * dy;
            if (k == LOCAL_MAXO && !(v < d[k - 1])) continue;
            int j = k < LOCAL_MAXO ? k++ : k - 1;
            for (; j > 0 && v < d[j - 1]; --j) { d[j] = d[j - 1]; at[j] = at[j - 1]; }
            d[j] = v;
            at[j] = o;
        }
        int within = 1;
        while (within < k && !(d[within] > origin_radius * origin_radius)) ++within;
        for (int j = within; j < k; ++j) at[j] = 0;
        nlorg[i] = within;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_lorg, lorg.data(), sizeof(int) * lorg.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d_nlorg, nlorg.data(), sizeof(int) * nimg, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(M->d_slopes, sl.data(), sizeof(double2) * norigin, cudaMemcpyHostToDevice, s);
    long launches = 0, considered = 0;
    std::vector<int> cnt_h(nb);
    // (as many threads as an SM's registers hold beside what its shared memory does)
    const int threads = lsmem > 75 * 1024 ? LOCAL_THREADS : LOCAL_THREADS / 2;
    for (long i0 = 0; e == cudaSuccess && i0 < nimg; i0 += nb) {
        const long cnt = std::min(nb, nimg - i0);
        if (i0 > 0 && (e = select(i0, cnt)) != cudaSuccess) break;
        local_score_kernel<<<(unsigned)cnt, threads, lsmem, s>>>(
            M->d_spec, M->D, M->d_ctf, (int)M->h_pix.size(), M->d_cpix, M->ncpix, nf, M->d_gA, M->d_slopes,
            d_lorg + i0 * LOCAL_MAXO, d_nlorg + i0, d_cand, d_count, M->d_panel, M->kpad, topk, i0, M->d_csec,
            M->d_corg, M->d_cscore);
        e = cudaGetLastError();
        launches += 3;
        if (e == cudaSuccess) e = cudaMemcpyAsync(cnt_h.data(), d_count, sizeof(int) * cnt, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        for (long i = 0; i < cnt; ++i) considered += (long)std::min(cnt_h[i], LOCAL_MAXC) * nlorg[i0 + i];
    }
    cudaEventRecord(ev[1], s);
    if (e == cudaSuccess) e = cudaEventSynchronize(ev[1]);
    float lms = 0;
    cudaEventElapsedTime(&lms, ev[0], ev[1]);
    cudaEventDestroy(ev[0]);
    cudaEventDestroy(ev[1]);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search_local: %s", cudaGetErrorString(e));
    float tres = 0;
    long ng = 0;
    e = rescore_candidates(*M, topk, sl, out, &tres, &ng);
    if (e != cudaSuccess) return match_fail(BSG_ERR_CUDA, "bsg_match_search_local: %s", cudaGetErrorString(e));
    M->sstats.local_ms += lms;
    M->sstats.rescore_ms += tres;
    M->sstats.launches += launches + (ng > 0 ? 1 : 0);
    M->sstats.images += nimg;
    M->sstats.hypotheses += (double)considered;
    M->sstats.rescored += nimg * topk;
    return BSG_OK;
}

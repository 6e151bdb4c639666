// k_corr.cu -- FP32 correlation cost volume with the unary fused in.
//
// Restates kCorrelation_NHWC / kCorrelation_NHWC_interpolation
// (stereo/operators/stereocorrelation.cu:66-142, rectCorr = 0) followed by the
// channel softmax over D and the negation (stereo/operators/softmax.cpp:30-38,
// stereo/utils.cu:289-292), or by 1 - <fL,fR> for L2-normalised features.
// Compiled with --fmad=false; the dot products use explicit fmaf in channel
// order and the softmax sum follows the lane layout below, so the output is
// bit-identical to the CPU oracle.
//
// Block = one image row y, 32 pixels; the left tile and the band of right
// pixels those pixels can see are staged in shared memory (odd row stride:
// lanes read consecutive rows without bank conflicts).  One warp per pixel;
// lane j owns disparity indices k = j + 32 r.
#include <algorithm>
#include <cfloat>

#include <cuda_bf16.h>

#include "../../include/cnncrf_fmath.h"
#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

namespace {

constexpr int PIX = 32;
constexpr int MAXP = 16; // D <= 512

__device__ __forceinline__ float to_f(float v) { return v; }
__device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }

// TIN: feature element type (float: the bit-exact path; bf16: the tensor-core
// path's features); cs = channel stride of a pixel (>= C)
template <typename TIN>
__global__ void __launch_bounds__(256)
    k_corr(const TIN *__restrict__ fl, const TIN *__restrict__ fr, int H, int W, int C, int cs,
           const float *__restrict__ list, int D, int omin, int omax, int interp, int unary,
           float *__restrict__ out, long fps)
{
    extern __shared__ float sm[];
    fl += blockIdx.z * fps; // pair of the batch
    fr += blockIdx.z * fps;
    out += (long)blockIdx.z * H * W * D;
    const int y = blockIdx.y;
    const int x0 = blockIdx.x * PIX;
    const int CS = C + 1;
    const int xlo = max(0, x0 + omin);
    const int xhi = min(W - 1, x0 + PIX - 1 + omax);
    const int R = max(0, xhi - xlo + 1);
    const int npx = min(PIX, W - x0);
    float *sl = sm;                     // [PIX][CS]
    float *sr = sl + PIX * CS;          // [R][CS]
    float *sd = sr + (size_t)R * CS;    // [D]
    for (int i = threadIdx.x; i < npx * C; i += blockDim.x) {
        int p = i / C, c = i - p * C;
        sl[p * CS + c] = to_f(fl[((long)y * W + x0 + p) * cs + c]);
    }
    for (int i = threadIdx.x; i < R * C; i += blockDim.x) {
        int p = i / C, c = i - p * C;
        sr[p * CS + c] = to_f(fr[((long)y * W + xlo + p) * cs + c]);
    }
    for (int i = threadIdx.x; i < D; i += blockDim.x) sd[i] = list[i];
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = (D + 31) >> 5;
    for (int pi = warp; pi < npx; pi += 8) {
        const int x = x0 + pi;
        const float *a = sl + pi * CS;
        float cv[MAXP];
#pragma unroll
        for (int r = 0; r < MAXP; ++r) {
            cv[r] = 0.0f;
            int kk = lane + 32 * r;
            if (r < P && kk < D) {
                float s = sd[kk];
                float w2 = (float)x + s;
                float acc = 0.0f;
                if (!interp) {
                    if (w2 >= 0.0f) {
                        int xs = x + (int)s;
                        if (xs <= W - 1) {
                            const float *b = sr + (xs - xlo) * CS;
                            for (int c = 0; c < C; ++c) acc = __fmaf_rn(a[c], b[c], acc);
                        }
                    }
                } else if (w2 >= 0.0f) {
                    int xa = (int)floorf(w2);
                    int xb = (int)(w2 + 1.0f);
                    float num = w2 - (float)xa;
                    float den = (float)xb - (float)xa;
                    // taps stay inside the staged band [xlo, xhi] (float rounding of
                    // w2 + 1 cannot step past it); xhi <= W - 1 also clamps the right edge
                    const float *b0 = sr + (min(max(xa, xlo), xhi) - xlo) * CS;
                    const float *b1 = sr + (min(max(xb, xlo), xhi) - xlo) * CS;
                    for (int c = 0; c < C; ++c) {
                        float y0 = b0[c], y1 = b1[c];
                        float it = y0 + ((y1 - y0) * num) / den;
                        acc = __fmaf_rn(a[c], it, acc);
                    }
                }
                cv[r] = acc;
            }
        }
        float *o = out + ((long)y * W + x) * D;
        if (unary == 0) {
            float m = -FLT_MAX;
#pragma unroll
            for (int r = 0; r < MAXP; ++r)
                if (r < P && lane + 32 * r < D) m = fmaxf(m, cv[r]);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
            float s = 0.0f;
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                if (r < P) {
                    int kk = lane + 32 * r;
                    float e = kk < D ? cnncrf_expf(cv[r] - m) : 0.0f;
                    cv[r] = e;
                    s = (r == 0) ? e : s + e;
                }
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = -(cv[r] / s);
            }
        } else {
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = unary == 1 ? 1.0f - cv[r] : cv[r];
            }
        }
    }
}

// Integer disparities of the other cases (BF16 features, ragged channel
// counts, wide bands) as a banded GEMM: for the 32 pixels x0.. of row y and
// every right pixel j of their band, T[p][j] = sum_c fL[c][p] * fR[c][j]
// (ascending c, one fmaf per term from 0: the same value as the per-pixel
// loop above), register-blocked 4 pixels x NJ band columns per thread; then
// one warp per pixel picks its D taps out of T and applies the unary.
constexpr int MAXNJ = 16;

template <typename TIN>
__global__ void __launch_bounds__(256)
    k_corr_band(const TIN *__restrict__ fl, const TIN *__restrict__ fr, int H, int W, int C, int cs,
                const float *__restrict__ list, int D, int omin, int omax, int NJ, int unary,
                float *__restrict__ out, long fps)
{
    extern __shared__ float sm[];
    fl += blockIdx.z * fps; // pair of the batch
    fr += blockIdx.z * fps;
    out += (long)blockIdx.z * H * W * D;
    const int y = blockIdx.y;
    const int x0 = blockIdx.x * PIX;
    const int RB = NJ * 32;                  // band columns computed (>= PIX + omax - omin)
    const int xlo = x0 + omin;               // band column 0 (may be < 0: zero filled)
    const int LS = PIX + 1, RS = RB + 1;     // odd row strides
    float *sl = sm;                          // [C][LS]
    float *sr = sl + (size_t)C * LS;         // [C][RS]
    float *sd = sr + (size_t)C * RS;         // [D]
    const int npx = min(PIX, W - x0);
    for (int i = threadIdx.x; i < PIX * C; i += blockDim.x) {
        int p = i / C, c = i - p * C;
        sl[c * LS + p] = p < npx ? to_f(fl[((long)y * W + x0 + p) * cs + c]) : 0.0f;
    }
    for (int i = threadIdx.x; i < RB * C; i += blockDim.x) {
        int j = i / C, c = i - j * C;
        int xr = xlo + j;
        sr[c * RS + j] = (xr >= 0 && xr < W) ? to_f(fr[((long)y * W + xr) * cs + c]) : 0.0f;
    }
    for (int i = threadIdx.x; i < D; i += blockDim.x) sd[i] = list[i];
    __syncthreads();

    const int tp = threadIdx.x & 7, tj = threadIdx.x >> 3;
    float acc[4][MAXNJ];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < MAXNJ; ++j) acc[i][j] = 0.0f;
    for (int c = 0; c < C; ++c) {
        const float *a = sl + c * LS + tp * 4;
        const float a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3];
        const float *b = sr + c * RS + tj * NJ;
#pragma unroll
        for (int j = 0; j < MAXNJ; ++j) {
            if (j < NJ) {
                const float bv = b[j];
                acc[0][j] = __fmaf_rn(a0, bv, acc[0][j]);
                acc[1][j] = __fmaf_rn(a1, bv, acc[1][j]);
                acc[2][j] = __fmaf_rn(a2, bv, acc[2][j]);
                acc[3][j] = __fmaf_rn(a3, bv, acc[3][j]);
            }
        }
    }
    __syncthreads(); // the tiles are dead: T reuses their storage
    float *T = sm;   // [PIX][RS]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < MAXNJ; ++j)
            if (j < NJ) T[(tp * 4 + i) * RS + tj * NJ + j] = acc[i][j];
    float *sd2 = T + (size_t)PIX * RS;
    for (int i = threadIdx.x; i < D; i += blockDim.x) sd2[i] = list[i];
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = (D + 31) >> 5;
    for (int pi = warp; pi < npx; pi += 8) {
        const int x = x0 + pi;
        float cv[MAXP];
#pragma unroll
        for (int r = 0; r < MAXP; ++r) {
            cv[r] = 0.0f;
            int kk = lane + 32 * r;
            if (r < P && kk < D) {
                float s = sd2[kk];
                float w2 = (float)x + s;
                if (w2 >= 0.0f) {
                    int xs = x + (int)s;
                    if (xs <= W - 1) cv[r] = T[pi * RS + (xs - xlo)];
                }
            }
        }
        float *o = out + ((long)y * W + x) * D;
        if (unary == 0) {
            float m = -FLT_MAX;
#pragma unroll
            for (int r = 0; r < MAXP; ++r)
                if (r < P && lane + 32 * r < D) m = fmaxf(m, cv[r]);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
            float sum = 0.0f;
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                if (r < P) {
                    int kk = lane + 32 * r;
                    float e = kk < D ? cnncrf_expf(cv[r] - m) : 0.0f;
                    cv[r] = e;
                    sum = (r == 0) ? e : sum + e;
                }
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) sum = sum + __shfl_xor_sync(0xffffffffu, sum, off);
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = -(cv[r] / sum);
            }
        } else {
#pragma unroll
            for (int r = 0; r < MAXP; ++r) {
                int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = unary == 1 ? 1.0f - cv[r] : cv[r];
            }
        }
    }
}

// FP32 features with channel counts in multiples of 4: the band without its
// corners.  A CTA holds PX = 8 PG pixels of a row and the PX + 8 KG right
// columns that offsets smax, smax - 1, .. of them reach, both as
// [channel][column]; a thread computes 8 pixels x 8 offsets, whose 64 products
// per channel need only 8 left and 15 right values (pixel i, offset smax - j:
// right column i + 7 - j of its window).
// Per output the terms in ascending channel, one fmaf each from 0, so the
// costs equal k_corr_band's; they then go through shared memory to one warp
// per pixel for the unary, in k_corr_band's order.
//
// Column px lies at px ^ 8 (c / 4 mod 4), which spreads the transposing stores
// (8 pixels x 4 channel groups per warp) over the banks, and ^ 4 in every
// other group of 32, which does the same for eight lanes' 16-byte loads.
// Bound by the latency of its phases: two CTAs per SM (shared memory), 8 warps,
// load their whole tile, then compute, then gather and normalise, and issue in
// 46 % of the cycles (FMA pipe 27 %, shared memory 38 % of its rate, DRAM 7 %).
// A thread takes 24 floats from shared memory per 64 fmas: 24 wavefronts per
// warp and channel, 96 of an SM's cycles for 77 of its fmas.  A KITTI pair at D = 128, C
// = 100 with the softmax: 3.44 -> 1.04 ms; a 720 x 480 pair at D = 96 plus the
// refinement's three labels 2.98 -> 0.81 ms; 256 x 192 at D = 32 0.214 ->
// 0.066 ms (k_corr_band: scalar loads, 9 wavefronts per 20 fmas, its band's
// corners computed).
template <int PG> // 16: up to 128 threads, 8: up to 256
__global__ void __launch_bounds__(2048 / PG, 2)
    k_corr_unit(const float *__restrict__ fl, const float *__restrict__ fr, int H, int W, int C, const float *__restrict__ list, int D,
                int KG, int smax, int unary, float *__restrict__ out, long fps)
{
    constexpr int PX = 8 * PG;
    extern __shared__ float4 sm4[];
    fl += blockIdx.z * fps; // pair of the batch
    fr += blockIdx.z * fps;
    out += (long)blockIdx.z * H * W * D;
    const int y = blockIdx.y, x0 = blockIdx.x * PX;
    const int RP = (PX + 8 * KG + 31) & ~31; // columns of the right window, whole swizzle groups
    const int cb = x0 + smax - (8 * KG - 1); // its first column
    float *Ls = (float *)sm4, *Rs = Ls + C * PX; // [C][PX], [C][RP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const int npx = min(PX, W - x0), NQ = C / 4, NB = (NQ + 3) / 4;
    auto stage = [&](const float *f, int first, int width, float *dst, int pitch) {
        constexpr int U = 8; // loads in flight per thread
        const int pl = lane >> 2, ql = lane & 3, nt = (width / 8) * NB;
        for (int t0 = warp; t0 < nt; t0 += nw * U) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = t0 + nw * u, p8 = t / NB, q = (t - p8 * NB) * 4 + ql, x = first + p8 * 8 + pl;
                v[u] = t < nt && q < NQ && x >= 0 && x < W ? __ldg((const float4 *)(f + ((long)y * W + x) * C + 4 * q))
                                                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int t = t0 + nw * u, p8 = t / NB, q = (t - p8 * NB) * 4 + ql;
                if (t < nt && q < NQ) {
                    float *d = dst + 4 * q * pitch + ((p8 * 8 + pl) ^ (8 * ql) ^ (p8 & 4));
                    d[0] = v[u].x, d[pitch] = v[u].y, d[2 * pitch] = v[u].z, d[3 * pitch] = v[u].w;
                }
            }
        }
    };
    stage(fl, x0, PX, Ls, PX);
    stage(fr, cb, RP, Rs, RP);
    __syncthreads();

    const int pg = tid % PG, kg = tid / PG;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    if (kg < KG) {
        const float *lp = Ls, *rp = Rs;
        const int p0 = 8 * pg, lc = 8 * (pg + KG - 1 - kg);
        const int fl4 = pg & 4, fr4 = (lc >> 3) & 4, fs4 = ((lc >> 3) + 1) & 4;
        for (int c4 = 0; c4 < NQ; ++c4) {
            const int swz = 8 * (c4 & 3), lo = p0 ^ swz, r0 = lc ^ swz, r1 = (lc + 8) ^ swz;
#pragma unroll
            for (int e = 0; e < 4; ++e, lp += PX, rp += RP) {
                float l[8], r[16];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 a = *(const float4 *)(lp + lo + (4 * h ^ fl4)), b = *(const float4 *)(rp + r0 + (4 * h ^ fr4)),
                                 d = *(const float4 *)(rp + r1 + (4 * h ^ fs4));
                    l[4 * h] = a.x, l[4 * h + 1] = a.y, l[4 * h + 2] = a.z, l[4 * h + 3] = a.w;
                    r[4 * h] = b.x, r[4 * h + 1] = b.y, r[4 * h + 2] = b.z, r[4 * h + 3] = b.w;
                    r[8 + 4 * h] = d.x, r[9 + 4 * h] = d.y, r[10 + 4 * h] = d.z, r[11 + 4 * h] = d.w;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = __fmaf_rn(l[i], r[i + 7 - j], acc[i][j]);
            }
        }
    }
    __syncthreads(); // the tiles are dead: T reuses their storage
    const int TP = 8 * KG + 4;
    float *T = (float *)sm4; // [PX][TP]
    if (kg < KG) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float *t = T + (8 * pg + i) * TP + 8 * kg;
            *(float4 *)t = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            *(float4 *)(t + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
        }
    }
    __syncthreads();

    // the stored disparities of this lane's labels; label s reads T's column smax - s
    constexpr int MP = 8; // D <= 256
    const int P = (D + 31) >> 5;
    float sv[MP];
#pragma unroll
    for (int r = 0; r < MP; ++r) sv[r] = r < P && lane + 32 * r < D ? __ldg(list + lane + 32 * r) : 0.0f;
#pragma unroll 2
    for (int pi = warp; pi < npx; pi += nw) {
        const int x = x0 + pi;
        float cv[MP];
#pragma unroll
        for (int r = 0; r < MP; ++r) {
            const int s = (int)sv[r];
            cv[r] = r < P && lane + 32 * r < D && (float)x + sv[r] >= 0.0f && x + s <= W - 1 ? T[pi * TP + smax - s] : 0.0f;
        }
        float *o = out + ((long)y * W + x0 + pi) * D;
        if (unary == 0) {
            float m = -FLT_MAX;
#pragma unroll
            for (int r = 0; r < MP; ++r)
                if (r < P && lane + 32 * r < D) m = fmaxf(m, cv[r]);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
            float sum = 0.0f;
#pragma unroll
            for (int r = 0; r < MP; ++r) {
                if (r < P) {
                    const int kk = lane + 32 * r;
                    const float e = kk < D ? cnncrf_expf(cv[r] - m) : 0.0f;
                    cv[r] = e;
                    sum = (r == 0) ? e : sum + e;
                }
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) sum = sum + __shfl_xor_sync(0xffffffffu, sum, off);
#pragma unroll
            for (int r = 0; r < MP; ++r) {
                const int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = -(cv[r] / sum);
            }
        } else {
#pragma unroll
            for (int r = 0; r < MP; ++r) {
                const int kk = lane + 32 * r;
                if (r < P && kk < D) o[kk] = unary == 1 ? 1.0f - cv[r] : cv[r];
            }
        }
    }
}

// shared memory of k_corr_unit at 8 PG pixels and KB right columns per pixel
size_t unit_smem(int PG, int C, int KB)
{
    const int KG = (KB + 7) / 8, PX = 8 * PG;
    return sizeof(float) * std::max((size_t)C * (PX + ((PX + 8 * KG + 31) & ~31)), (size_t)PX * (8 * KG + 4));
}

template <int PG>
int launch_unit(const float *fl, const float *fr, int H, int W, int C, const float *d_list, int D, int KB, int smax, int unary,
                float *out, cudaStream_t st, int npairs, long fps)
{
    const int KG = (KB + 7) / 8, PX = 8 * PG;
    const int threads = std::max(128, (PG * KG + 31) & ~31); // narrow bands: more warps load than compute
    const size_t sm = unit_smem(PG, C, KB);
    CNNCRF_CUDA(allow_smem(k_corr_unit<PG>));
    CNNCRF_PROF("corr", st);
    k_corr_unit<PG><<<dim3(ceil_div(W, PX), H, npairs), threads, sm, st>>>(fl, fr, H, W, C, d_list, D, KG, smax, unary, out,
                                                                           fps);
    return CNNCRF_OK;
}

} // namespace

template <typename TIN>
static int corr_launch(const TIN *fl, const TIN *fr, int H, int W, int C, int cs, const float *d_list, int D,
                       int omin, int omax, bool interp, int unary, float *out, cudaStream_t st, int npairs,
                       long fps)
{
    if (D < 1 || D > 32 * MAXP) return fail(CNNCRF_EINVAL, "correlation: D=%d outside [1,%d]", D, 32 * MAXP);
    dim3 grid(ceil_div(W, PIX), H, npairs);
    const int NJ = ceil_div(PIX + omax - omin, 32);
    // phase 1 holds the two feature tiles, phase 2 the result tile T in the
    // same storage: allocate the larger of the two
    const size_t tiles = (size_t)C * (PIX + 1) + (size_t)C * (NJ * 32 + 1) + D;
    const size_t tres = (size_t)PIX * (NJ * 32 + 1) + D;
    const size_t band_smem = sizeof(float) * std::max(tiles, tres);
    if (!interp && NJ <= MAXNJ && band_smem <= SMEM_MAX) {
        CNNCRF_CUDA(allow_smem(k_corr_band<TIN>));
        {
            CNNCRF_PROF("corr", st);
            k_corr_band<TIN><<<grid, 256, band_smem, st>>>(fl, fr, H, W, C, cs, d_list, D, omin, omax, NJ, unary, out,
                                                             fps);
        }
        CNNCRF_CHECK_LAUNCH();
        return CNNCRF_OK;
    }
    int R = PIX + omax - omin + 1;
    size_t smem = sizeof(float) * ((size_t)(PIX + R) * (C + 1) + D);
    if (smem > SMEM_MAX)
        return fail(CNNCRF_EINVAL, "correlation: disparity band too wide (%zu bytes of shared memory)", smem);
    CNNCRF_CUDA(allow_smem(k_corr<TIN>));
    {
        CNNCRF_PROF("corr", st);
        k_corr<TIN><<<grid, 256, smem, st>>>(fl, fr, H, W, C, cs, d_list, D, omin, omax, interp ? 1 : 0, unary, out,
                                              fps);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int correlation(const float *fl, const float *fr, int H, int W, int C, const float *d_list, int D, int omin,
                int omax, bool interp, int unary, float *out, cudaStream_t st, int npairs, long fps)
{
    // k_corr_unit: integer taps, 16-byte aligned pixels, up to 256 labels and right columns per pixel (its threads),
    // tiles that fit; 128 pixels per CTA for up to 64 columns (as many threads), else 64
    const int KB = omax - omin + 1;
    const bool al16 = (((uintptr_t)fl | (uintptr_t)fr) & 15) == 0 && C % 4 == 0 && fps % 4 == 0;
    if (!interp && al16 && D <= 256 && KB <= 256 && npairs <= 65535 && H <= 65535) {
        if (KB <= 64 && unit_smem(16, C, KB) <= SMEM_MAX) {
            CNNCRF_TRY(launch_unit<16>(fl, fr, H, W, C, d_list, D, KB, omax, unary, out, st, npairs, fps));
            CNNCRF_CHECK_LAUNCH();
            return CNNCRF_OK;
        }
        if (unit_smem(8, C, KB) <= SMEM_MAX) {
            CNNCRF_TRY(launch_unit<8>(fl, fr, H, W, C, d_list, D, KB, omax, unary, out, st, npairs, fps));
            CNNCRF_CHECK_LAUNCH();
            return CNNCRF_OK;
        }
    }
    return corr_launch<float>(fl, fr, H, W, C, C, d_list, D, omin, omax, interp, unary, out, st, npairs, fps);
}

int correlation_bf16(const void *fl, const void *fr, int H, int W, int C, int cs, const float *d_list, int D,
                     int omin, int omax, bool interp, int unary, float *out, cudaStream_t st, int npairs, long fps)
{
    return corr_launch<__nv_bfloat16>((const __nv_bfloat16 *)fl, (const __nv_bfloat16 *)fr, H, W, C, cs, d_list,
                                      D, omin, omax, interp, unary, out, st, npairs, fps);
}

} // namespace k
} // namespace cnncrf

// k_conv_simt.cu -- the FP32 convolution of the bit-exact path.
//
// Implicit GEMM on the CUDA cores: out[p][co] = act(bias[co] + sum_k A[p][k] W[k][co])
// with p = output pixel, k = (ky, kx, ci) ci fastest.  Each output is
// accumulated in ascending k with one fmaf per term, so it equals the CPU
// oracle bit for bit (reference: cudnnConvolutionForward in
// CUDNN_CONVOLUTION mode + cudnnAddTensor + tanh, stereo/operators/
// convolution.cpp:141-152, bias.cpp:58-67, activation.cpp:33-41).
//
// k_conv_px and k_conv_patch carry the nets' layers; k_conv_nt and k_conv_simt
// (CTA = 128 pixels of one output row x up to 128 output channels, k-slices
// double-buffered in shared memory, 8x8 register tiles) the other shapes.
#include <algorithm>
#include <type_traits>

#include <cuda_bf16.h>

#include "../../include/cnncrf_fmath.h"
#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

namespace {

constexpr int BM = 128, BN = 128, BK = 8, APAD = 4;

__device__ __forceinline__ float act_fn(float v, int act)
{
    if (act == 1) return cnncrf_tanhf(v);
    if (act == 2) return fabsf(v);
    if (act == 3) return fabsf(cnncrf_tanhf(v));
    return v;
}

__global__ void __launch_bounds__(256) k_conv_simt(ConvArgs a, int Ho, int Wo, int K)
{
    __shared__ __align__(16) float As[2][BK][BM + APAD];
    __shared__ __align__(16) float Bs[2][BK][BN];
    const int tid = threadIdx.x;
    const int oy = blockIdx.y;
    const int ox0 = blockIdx.x * BM;
    a.in += (long)blockIdx.z * a.in_img; // image of the batch
    if (a.out16) a.out16 = (char *)a.out16 + (long)blockIdx.z * a.out_img * 2;
    else a.out += (long)blockIdx.z * a.out_img;
    const int a_kk = tid & 7, a_p = tid >> 3;
    const int b_kk = tid >> 5, b_n = (tid & 31) * 4;
    const int tx = tid & 15, ty = tid >> 4;
    const int nsl = (K + BK - 1) / BK;

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;

    float ra[4];
    float4 rb;
    auto loadA = [&](int s) {
        int kk = s * BK + a_kk;
        bool kv = kk < K;
        int ky = 0, kx = 0, ci = 0;
        if (kv) {
            int tap = kk / a.Cin;
            ci = kk - tap * a.Cin;
            ky = tap / a.kw;
            kx = tap - ky * a.kw;
        }
        const float *rowp = a.in + (long)(oy + ky) * a.in_row + (long)kx * a.in_pix + ci;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int ox = ox0 + a_p + 32 * e;
            ra[e] = (kv && ox < Wo) ? __ldg(rowp + (long)ox * a.in_pix) : 0.0f;
        }
    };
    auto loadB = [&](int s) {
        int kk = s * BK + b_kk;
        rb = kk < K ? __ldg((const float4 *)(a.wt + (long)kk * BN + b_n)) : make_float4(0, 0, 0, 0);
    };
    auto storeAB = [&](int buf) {
#pragma unroll
        for (int e = 0; e < 4; ++e) As[buf][a_kk][a_p + 32 * e] = ra[e];
        *(float4 *)&Bs[buf][b_kk][b_n] = rb;
    };

    loadA(0);
    loadB(0);
    storeAB(0);
    __syncthreads();
    for (int s = 0; s < nsl; ++s) {
        const int cur = s & 1;
        if (s + 1 < nsl) {
            loadA(s + 1);
            loadB(s + 1);
        }
        const int kmax = min(BK, K - s * BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            if (kk < kmax) {
                float4 a0 = *(const float4 *)&As[cur][kk][ty * 4];
                float4 a1 = *(const float4 *)&As[cur][kk][64 + ty * 4];
                float4 b0 = *(const float4 *)&Bs[cur][kk][tx * 4];
                float4 b1 = *(const float4 *)&Bs[cur][kk][64 + tx * 4];
                float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = __fmaf_rn(av[i], bv[j], acc[i][j]);
            }
        }
        if (s + 1 < nsl) storeAB(cur ^ 1);
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 8; ++i) {
        int p = (i < 4) ? ty * 4 + i : 64 + ty * 4 + (i - 4);
        int ox = ox0 + p;
        if (ox >= Wo) continue;
        float *dst = a.out16 ? nullptr : a.out + (long)oy * a.out_row + (long)ox * a.out_pix;
        __nv_bfloat16 *dst16 = a.out16 ? (__nv_bfloat16 *)a.out16 + ((long)oy * Wo + ox) * a.out_cs : nullptr;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int co = (j < 4) ? tx * 4 + j : 64 + tx * 4 + (j - 4);
            if (co < a.Cout) {
                float v = acc[i][j];
                if (a.bias) v = __fadd_rn(v, a.bias[co]);
                v = act_fn(v, a.act);
                if (dst16) dst16[co] = __float2bfloat16_rn(v);
                else dst[(long)co * a.out_ch] = v;
            }
        }
    }
}

// Packed FP32: two IEEE fmas, each rounded once (fma.rn.f32x2), on a pair of
// floats held in one 64-bit register -- the same values as two __fmaf_rn at
// half the instruction issue.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// The layers that k_conv_px does not take (thin or oddly aligned inputs, up to
// 32 or over 104 channels, BF16 outputs).  The same convolution with the channel tile cut to the layer's width (TN =
// 32, 64 or 112 output channels, for Cout <= TN) and the index arithmetic
// taken out of the k loop.  2 TN threads, each an 8 x 8 register tile (8
// pixels x 8 channels); k-slices of TK (7 at TN = 112, else 8), so that every
// thread loads one fixed k offset of each slice, for 128 TK / (2 TN) pixels
// whose offsets it computes once, and steps its (ky, kx, ci) from slice to
// slice without a division.  Per output the terms are accumulated in
// ascending k with one fmaf each, then + bias and the activation, as in
// k_conv_simt: the same bits.
template <int TN, int TK>
__global__ void __launch_bounds__(2 * TN, 2) k_conv_nt(ConvArgs a, int Ho, int Wo, int K)
{
    constexpr int NT = 2 * TN;      // threads
    constexpr int PA = BM * TK / NT; // pixels a thread loads per slice
    constexpr int PS = NT / TK;      // their stride
    constexpr int B4 = TK * TN / 4;  // float4 of a weight slice
    constexpr int BR = (B4 + NT - 1) / NT; // of them per thread
    static_assert(NT % TK == 0 && (BM * TK) % NT == 0, "k_conv_nt tile");
    __shared__ __align__(16) float As[2][TK][BM + APAD];
    __shared__ __align__(16) float Bs[2][TK][TN];
    const int tid = threadIdx.x;
    const int oy = blockIdx.y, ox0 = blockIdx.x * BM;
    a.in += (long)blockIdx.z * a.in_img; // image of the batch
    if (a.out16) a.out16 = (char *)a.out16 + (long)blockIdx.z * a.out_img * 2;
    else a.out += (long)blockIdx.z * a.out_img;
    const float *inb = a.in + (long)oy * a.in_row;
    // loader roles: k offset lk of every slice at pixels lp + PS j; weight float4s tid + NT r
    const int lk = tid % TK, lp = tid / TK;
    // compute roles: 16 pixel groups x TN / 8 channel groups, the pixel group
    // fastest, so that a quarter warp's 128-bit fragment loads read 128
    // contiguous bytes of the pixel row and the channel fragments are broadcasts
    const int ty = tid % 16, tx = tid / 16;
    long poff[PA];
    uint32_t pvalid = 0;
#pragma unroll
    for (int j = 0; j < PA; ++j) {
        const int ox = ox0 + lp + PS * j;
        poff[j] = (long)ox * a.in_pix;
        if (ox < Wo) pvalid |= 1u << j;
    }
    // (ky, kx, ci) of this thread's k in the current slice
    int kk = lk, ci = 0, kx = 0, ky = 0;
    if (kk < K) {
        const int tap = kk / a.Cin;
        ci = kk - tap * a.Cin;
        ky = tap / a.kw;
        kx = tap - ky * a.kw;
    }
    const int nfull = K / TK, nsl = (K + TK - 1) / TK;

    // accumulators of 8 pixels x 4 channel pairs (channels 2m, 2m+1 of the thread's 8)
    unsigned long long acc2[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int m = 0; m < 4; ++m) acc2[i][m] = 0ull;

    float ra[PA];
    float4 rb[BR];
    auto loadA = [&]() {
        const bool kv = kk < K;
        const float *src = inb + (long)ky * a.in_row + (long)kx * a.in_pix + ci;
#pragma unroll
        for (int j = 0; j < PA; ++j) ra[j] = (kv && (pvalid >> j & 1u)) ? __ldg(src + poff[j]) : 0.0f;
    };
    auto loadB = [&](int s) {
#pragma unroll
        for (int r = 0; r < BR; ++r) {
            const int f = tid + NT * r, k = s * TK + f / (TN / 4), n = (f % (TN / 4)) * 4;
            rb[r] = (f < B4 && k < K) ? __ldg((const float4 *)(a.wt + (long)k * BN + n)) : make_float4(0, 0, 0, 0);
        }
    };
    auto storeAB = [&](int buf) {
#pragma unroll
        for (int j = 0; j < PA; ++j) As[buf][lk][lp + PS * j] = ra[j];
#pragma unroll
        for (int r = 0; r < BR; ++r) {
            const int f = tid + NT * r;
            if (f < B4) *(float4 *)&Bs[buf][f / (TN / 4)][(f % (TN / 4)) * 4] = rb[r];
        }
    };
    auto advance = [&]() { // this thread's k of the next slice
        kk += TK;
        ci += TK;
        while (ci >= a.Cin) {
            ci -= a.Cin;
            if (++kx == a.kw) kx = 0, ++ky;
        }
    };
    auto step = [&](int cur, int k) {
        const float4 a0 = *(const float4 *)&As[cur][k][ty * 4];
        const float4 a1 = *(const float4 *)&As[cur][k][64 + ty * 4];
        const ulonglong2 b0 = *(const ulonglong2 *)&Bs[cur][k][tx * 4];
        const ulonglong2 b1 = *(const ulonglong2 *)&Bs[cur][k][TN / 2 + tx * 4];
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const unsigned long long bp[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned long long ap = pack2(av[i], av[i]);
#pragma unroll
            for (int m = 0; m < 4; ++m) fma2(acc2[i][m], ap, bp[m]);
        }
    };

    loadA();
    loadB(0);
    storeAB(0);
    __syncthreads();
    for (int s = 0; s < nsl; ++s) {
        const int cur = s & 1;
        if (s + 1 < nsl) {
            advance();
            loadA();
            loadB(s + 1);
        }
        if (s < nfull) {
#pragma unroll
            for (int k = 0; k < TK; ++k) step(cur, k);
        } else {
            for (int k = 0; k < K - nfull * TK; ++k) step(cur, k);
        }
        if (s + 1 < nsl) storeAB(cur ^ 1);
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int ox = ox0 + ((i < 4) ? ty * 4 + i : 64 + ty * 4 + (i - 4));
        if (ox >= Wo) continue;
        float *dst = a.out16 ? nullptr : a.out + (long)oy * a.out_row + (long)ox * a.out_pix;
        __nv_bfloat16 *dst16 = a.out16 ? (__nv_bfloat16 *)a.out16 + ((long)oy * Wo + ox) * a.out_cs : nullptr;
        float accf[8];
#pragma unroll
        for (int m = 0; m < 4; ++m) asm("mov.b64 {%0, %1}, %2;" : "=f"(accf[2 * m]), "=f"(accf[2 * m + 1]) : "l"(acc2[i][m]));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int co = (j < 4) ? tx * 4 + j : TN / 2 + tx * 4 + (j - 4);
            if (co < a.Cout) {
                float v = accf[j];
                if (a.bias) v = __fadd_rn(v, a.bias[co]);
                v = act_fn(v, a.act);
                if (dst16) dst16[co] = __float2bfloat16_rn(v);
                else dst[(long)co * a.out_ch] = v;
            }
        }
    }
}

// The wide layers (Cin a multiple of 16 or 20, 16-byte aligned pixels): a CTA
// of four warps computes 128 output pixels, taken in row order across row
// ends so that narrow images leave no part of a tile idle; lane l has pixels
// l, l + 32, l + 64, l + 96 of it, warp w CPW channels (w_pitch).
// Four k steps of a warp are four 16-byte loads of its pixels' inputs
// (conflict-free at a pitch of 20 floats), broadcast loads of its weights and
// 8 CPW packed fmas; every scheduler carries the same two warps.  k-slices of
// TK, which divides Cin: a slice lies inside one tap and its input offset is
// the same for every pixel.  Inputs and weights come by cp.async, PXS slices
// deep.  Per output the terms in ascending k, one fmaf each: the same bits as
// k_conv_nt.
//
// Bound by the FMA pipe: fma.rn.f32x2 issues every 2.2 cycles where it shares
// an operand register with the one before it (else 2.5 to 3), 114 cycles per
// warp and k step at CPW = 26; the 3x3 layers of a 720 x 480 pair take about
// 140, a tenth of it for the copies.  All FP32 convolutions of that pair with
// its re-match: 33.4 ms in k_conv_nt (14 warps per SM on four schedulers, 8
// pack moves per 32 fmas, a row's last tile), now 22.5; of a KITTI pair in 2x2
// layers 14.5 and 9.7 ms; of a 256 x 192 grey pair 4.58 and 2.55 ms.  Of that
// the order of the fmas and the operands loaded a step ahead gave 4 % and
// tanh_pair 7 to 15 %.  Measured and left out: three CTAs at 160 to 168
// registers (23.0 to 23.2 ms), scalar fmas, exactly 25 channels per warp with
// one unpaired (2 % slower).
constexpr int PXT = 128, PXS = 3, PXP = 20; // pixels per CTA, slices in flight, floats of a pixel's slice
// a k row of weights in shared memory: warp w's channels are wmain = CPW / 4 * 4 from wmain w on and, where CPW is not a
// multiple of 4, the pair from 4 wmain + 2 w on: 16- and 8-byte loads out of rows copied as they lie in memory
__host__ __device__ constexpr int w_main(int CPW) { return CPW / 4 * 4; }
__host__ __device__ constexpr int w_pitch(int CPW) { return CPW > 16 ? BN : 64; }
__host__ __device__ constexpr int epi_pitch(int CPW) { return CPW / 2 % 2 ? CPW : CPW + 2; } // floats of a pixel in the epilogue
__host__ __device__ constexpr int px_stage(int CPW, int TK) { return PXT * PXP + TK * w_pitch(CPW); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// shared-memory loads that stay where they are written in the k loop
__device__ __forceinline__ void lds_f4(const float *p, float (&v)[4])
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void lds_u2(const float *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// accumulators of 4 pixels x CPW / 2 channel pairs, and k steps on them: A the lane's pixel, B the warp's run of weights,
// Bt the pair beyond it
template <int CPW> struct PxAcc {
    unsigned long long v[4][CPW / 2];
    __device__ __forceinline__ PxAcc()
    {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int m = 0; m < CPW / 2; ++m) v[i][m] = 0ull;
    }
    // ap: the pixels' input of this k, duplicated.  The pixel index snakes, so that every fma shares an operand register
    // with the one before it
    __device__ __forceinline__ void step(const unsigned long long (&ap)[4], const float *b, const float *bt)
    {
        unsigned long long bv[CPW / 2];
#pragma unroll
        for (int m = 0; m + 1 < CPW / 2; m += 2) {
            const ulonglong2 t = *(const ulonglong2 *)(b + 2 * m);
            bv[m] = t.x, bv[m + 1] = t.y;
        }
        if (CPW / 2 % 2) bv[CPW / 2 - 1] = *(const unsigned long long *)bt;
#pragma unroll
        for (int m = 0; m < CPW / 2; ++m)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = m % 2 ? 3 - j : j;
                fma2(v[i][m], ap[i], bv[m]);
            }
    }
    // NK k steps, the operands of a step loaded during the one before it
    template <int PITCH, int NK> __device__ __forceinline__ void slice(const float *A, const float *B, const float *Bt)
    {
        constexpr int WB = w_pitch(CPW), M = CPW / 2;
        float av[2][4][4];
        unsigned long long bv[2][M];
        auto loadA = [&](int q) {
#pragma unroll
            for (int i = 0; i < 4; ++i) lds_f4(A + 32 * PITCH * i + 4 * q, av[q & 1][i]);
        };
        auto loadB = [&](int k) {
#pragma unroll
            for (int m = 0; m + 1 < M; m += 2) lds_u2(B + k * WB + 2 * m, bv[k & 1][m], bv[k & 1][m + 1]);
            if (M % 2) bv[k & 1][M - 1] = *(const unsigned long long *)(Bt + k * WB);
        };
        loadA(0);
        loadB(0);
#pragma unroll
        for (int k = 0; k < NK; ++k) {
            if (k + 1 < NK) loadB(k + 1);
            if (k % 4 == 1 && k / 4 + 1 < NK / 4) loadA(k / 4 + 1);
            unsigned long long ap[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) ap[i] = pack2(av[k / 4 & 1][i][k % 4], av[k / 4 & 1][i][k % 4]);
#pragma unroll
            for (int m = 0; m < M; ++m)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int i = m % 2 ? 3 - j : j;
                    fma2(v[i][m], ap[i], bv[k & 1][m]);
                }
        }
    }
    template <int PITCH> __device__ __forceinline__ void steps(const float *A, const float *B, const float *Bt, int kn = 4)
    {
        constexpr int WB = w_pitch(CPW);
        float av[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = *(const float4 *)(A + 32 * PITCH * i);
            av[i][0] = t.x, av[i][1] = t.y, av[i][2] = t.z, av[i][3] = t.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= kn) break;
            unsigned long long ap[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) ap[i] = pack2(av[i][k], av[i][k]);
            step(ap, B + k * WB, Bt + k * WB);
        }
    }
};

__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long vfma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long vadd2(unsigned long long a, unsigned long long b)
{
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long vmul2(unsigned long long a, unsigned long long b)
{
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// cnncrf_tanhf of two values, the same bits, without branches and on packed operations where it has two of them:
//   rint of 0 <= y < 2^22 is (y + 1.5 2^23) - 1.5 2^23, and the sum's low bits are the integer;
//   2 |x| <= 18 needs no range case of expm1, 2^0 em1 + (2^0 - 1) is em1, and the quotient at |x| = 9 rounds to 1;
//   the quotient E / (E + 2) by Markstein's correctly rounded division ("Computation of elementary functions on the
//   IBM RISC System/6000 processor", 1990): a reciprocal y refined by one Newton step, q = E y, q + y (E - q (E + 2)).
//   Its operands are those of the 2^27 or so floats between 2^-12 and 9; selftest_tanh compares every float with cnncrf_tanhf.
__device__ __forceinline__ float2 tanh_pair(float2 x)
{
    auto both = [](float c) { return pack2(c, c); };
    float ax, ay; // |x|, at most 9; NaN stays
    asm("min.NaN.f32 %0, %1, 0f41100000;" : "=f"(ax) : "f"(fabsf(x.x)));
    asm("min.NaN.f32 %0, %1, 0f41100000;" : "=f"(ay) : "f"(fabsf(x.y)));
    const unsigned long long a = pack2(ax, ay), v = vadd2(a, a);
    const unsigned long long z = vadd2(vmul2(v, both(CNNCRF_INV_LN2)), both(12582912.0f));
    const unsigned long long n = vadd2(z, both(-12582912.0f));
    unsigned long long r = vfma2(n, both(-CNNCRF_LN2_HI), v);
    r = vfma2(n, both(-CNNCRF_LN2_LO), r);
    float zx, zy;
    unpack2(z, zx, zy);
    const unsigned long long s = pack2(__int_as_float((__float_as_int(zx) << 23) + 0x3f800000),
                                       __int_as_float((__float_as_int(zy) << 23) + 0x3f800000)); // 2^n
    unsigned long long q = vfma2(both(CNNCRF_C8), r, both(CNNCRF_C7));
    q = vfma2(q, r, both(CNNCRF_C6));
    q = vfma2(q, r, both(CNNCRF_C5));
    q = vfma2(q, r, both(CNNCRF_C4));
    q = vfma2(q, r, both(CNNCRF_C3));
    q = vfma2(q, r, both(CNNCRF_C2));
    const unsigned long long em1 = vfma2(vmul2(r, r), q, r);
    const unsigned long long e = vfma2(s, em1, vadd2(s, both(-1.0f)));
    const unsigned long long d = vadd2(e, both(2.0f)), nd = vfma2(e, both(-1.0f), both(-2.0f));
    float dx, dy, yx, yy;
    unpack2(d, dx, dy);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yx) : "f"(dx));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yy) : "f"(dy));
    unsigned long long y = pack2(yx, yy);
    y = vfma2(vfma2(nd, y, both(1.0f)), y, y);
    const unsigned long long t0 = vmul2(e, y), t = vfma2(vfma2(nd, t0, e), y, t0);
    float tx, ty;
    unpack2(t, tx, ty);
    tx = ax < 2.44140625e-4f ? x.x : copysignf(tx, x.x);
    ty = ay < 2.44140625e-4f ? x.y : copysignf(ty, x.y);
    return make_float2(tx, ty);
}

// The warp's 128 pixels x CPW channels through shared memory, then a rolled loop of bias, activation and store on
// channel pairs, a pixel's channels as one run (unrolled on the registers, the activations were 66 KB of code that
// every CTA ran through once).  The pitch makes a column of pairs conflict-free
template <int CPW>
__device__ __forceinline__ void px_epilogue(const ConvArgs &a, const PxAcc<CPW> &acc, float *sm, float *outp, int p0, int npx,
                                            int Wo, int lane, int warp)
{
    constexpr int EP = epi_pitch(CPW);
    constexpr int NM = w_main(CPW) / 2, NP = CPW / 2; // channel pairs of the warp's run, and with the one beyond it
    float *st = sm + warp * PXT * EP;
    const int c0 = warp * w_main(CPW), ct = 4 * w_main(CPW) + 2 * warp;
    if (c0 >= a.Cout) return;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int m = 0; m < NP; ++m) *(unsigned long long *)(st + (lane + 32 * i) * EP + 2 * m) = acc.v[i][m];
    __syncwarp();
    const bool dense = a.out_ch == 1 && a.out_row == Wo * a.out_pix;
    const bool pairs = dense && a.out_pix % 2 == 0 && ((uintptr_t)outp & 7) == 0;
    constexpr int DQ = 32 / NP, DM = 32 - DQ * NP; // a lane's stride in pixels and pairs
    int q = lane / NP, m = lane - q * NP;
    constexpr int U = 4; // pairs of a lane at a time
    static_assert(PXT * NP % (32 * U) == 0, "px_epilogue rounds");
#pragma unroll 1
    for (int e = 0; e < PXT * NP / 32; e += U) {
        float2 t[U];
        int pp[U], cc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            pp[u] = p0 + q, cc[u] = m < NM ? c0 + 2 * m : ct;
            t[u] = *(const float2 *)(st + q * EP + 2 * m);
            if (a.bias) t[u].x = __fadd_rn(t[u].x, __ldg(a.bias + cc[u])), t[u].y = __fadd_rn(t[u].y, __ldg(a.bias + cc[u] + 1));
            m += DM, q += DQ;
            if (m >= NP) m -= NP, ++q;
        }
        if (a.act & 1)
#pragma unroll
            for (int u = 0; u < U; ++u) t[u] = tanh_pair(t[u]);
        if (a.act & 2)
#pragma unroll
            for (int u = 0; u < U; ++u) t[u].x = fabsf(t[u].x), t[u].y = fabsf(t[u].y);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int p = pp[u], c = cc[u];
            if (p >= npx || c >= a.Cout) continue;
            const bool both = c + 1 < a.Cout;
            if (pairs && both) {
                *(float2 *)(outp + (long)p * a.out_pix + c) = t[u];
            } else {
                const int y = dense ? 0 : p / Wo, x = p - y * Wo;
                float *o = outp + (long)y * a.out_row + (long)x * a.out_pix + (long)c * a.out_ch;
                o[0] = t[u].x;
                if (both) o[a.out_ch] = t[u].y;
            }
        }
    }
}

template <int CPW, int TK>
__global__ void __launch_bounds__(128, 2) k_conv_px(ConvArgs a, int npx, int Wo, int K)
{
    constexpr int NQ = TK / 4;         // 16-byte pieces of a pixel's slice
    constexpr int WB = w_pitch(CPW);   // a k row of weights
    constexpr int SF = px_stage(CPW, TK);
    static_assert(CPW % 2 == 0 && TK % 4 == 0 && TK <= PXP && 4 * CPW <= BN, "k_conv_px tile");
    extern __shared__ float4 sm4[];
    float *sm = (float *)sm4; // [PXS][PXT][PXP] inputs and [TK][WB] weights
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p0 = blockIdx.x * PXT;
    const float *in = a.in + (long)blockIdx.y * a.in_img; // image of the batch
    float *outp = a.out + (long)blockIdx.y * a.out_img;
    // loader: piece q of a pixel, 128 NQ pieces over 128 threads, the piece fastest; its input offset without the
    // slice's, and its place in a stage
    int poff[NQ];
    uint32_t pdst[NQ];
    const uint32_t sm_s = (uint32_t)__cvta_generic_to_shared(sm);
#pragma unroll
    for (int j = 0; j < NQ; ++j) {
        const int f = tid + 128 * j, px = f / NQ, q = f - px * NQ;
        const int p = min(p0 + px, npx - 1), y = p / Wo, x = p - y * Wo; // the last tile's idle pixels repeat the last one
        poff[j] = y * (int)a.in_row + x * (int)a.in_pix + 4 * q;
        pdst[j] = sm_s + 4 * (px * PXP + 4 * q);
    }
    const int nsl = K / TK;
    // the slice being loaded: tap column kx, first channel ci
    int kx = 0, ci = 0, ls = 0, lbuf = 0;
    const float *src = in, *wsrc = a.wt;
    auto load = [&]() {
        if (ls < nsl) {
            const uint32_t o = 4u * SF * lbuf;
#pragma unroll
            for (int j = 0; j < NQ; ++j) cp_async16(pdst[j] + o, src + poff[j]);
            const uint32_t d = sm_s + o + 4 * PXT * PXP + 16 * tid;
#pragma unroll
            for (int f = 0; f < TK * WB / 4; f += 128)
                if (f + 128 <= TK * WB / 4 || f + tid < TK * WB / 4)
                    cp_async16(d + 16 * f, WB == BN ? wsrc + 4 * (f + tid) : wsrc + (f + tid) / (WB / 4) * BN + (f + tid) % (WB / 4) * 4);
            wsrc += TK * BN;
            ci += TK, src += TK;
            if (ci == a.Cin) {
                ci = 0, src += a.in_pix - a.Cin;
                if (++kx == a.kw) kx = 0, src += a.in_row - a.kw * a.in_pix;
            }
            ++ls, lbuf = lbuf + 1 == PXS ? 0 : lbuf + 1;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    PxAcc<CPW> acc;
    for (int s = 0; s < PXS - 1; ++s) load();
    for (int s = 0, cur = 0; s < nsl; ++s, cur = cur + 1 == PXS ? 0 : cur + 1) {
        asm volatile("cp.async.wait_group %0;" ::"n"(PXS - 2) : "memory");
        __syncthreads(); // slice s is there; everyone is done with slice s - 1
        load();
        const float *A = sm + cur * SF + lane * PXP, *B = sm + cur * SF + PXT * PXP + warp * w_main(CPW);
        const float *Bt = sm + cur * SF + PXT * PXP + 4 * w_main(CPW) + 2 * warp;
        acc.template slice<PXP, TK>(A, B, Bt);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    px_epilogue<CPW>(a, acc, sm, outp, p0, npx, Wo, lane, warp);
}

// First layers (thin inputs): the same tile, with the 128 pixels' patches of K
// = kh kw Cin <= KP values gathered whole, [pixel][KP] at a conflict-free
// pitch, and all K rows of the weights in shared memory.  Bound by the tanh
// epilogue and the output's bytes; a thread per pixel with all channels in
// registers stored 4 bytes at a 400-byte stride and took 1.42 ms for a KITTI
// pair's three first layers, this 0.41 (0.75 with cnncrf_tanhf as it stands).
template <int CPW, int KP>
__global__ void __launch_bounds__(128, 3) k_conv_patch(ConvArgs a, int npx, int Wo, int K)
{
    constexpr int WB = w_pitch(CPW);
    static_assert(KP % 8 == 4, "conflict-free pixel pitch");
    extern __shared__ float4 sm4[];
    float *A = (float *)sm4, *B = A + PXT * KP; // [PXT][KP], [K][WB]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int p0 = blockIdx.x * PXT;
    float *outp = a.out + (long)blockIdx.y * a.out_img;
    {
        const int p = min(p0 + tid, npx - 1), y = p / Wo, x = p - y * Wo; // this thread's pixel (idle ones repeat the last)
        const float *src = a.in + (long)blockIdx.y * a.in_img + (long)y * a.in_row + (long)x * a.in_pix;
        float *d = A + tid * KP;
        for (int ky = 0; ky < a.kh; ++ky)
            for (int kx = 0; kx < a.kw; ++kx)
                for (int ci = 0; ci < a.Cin; ++ci) *d++ = __ldg(src + (long)ky * a.in_row + (long)kx * a.in_pix + ci);
    }
    for (int i = tid; i < K * CPW; i += 128) {
        const int k = i / CPW, c = i - k * CPW;
        *(float4 *)(B + k * WB + 4 * c) = __ldg((const float4 *)(a.wt + (long)k * BN + 4 * c));
    }
    __syncthreads();
    PxAcc<CPW> acc;
    const float *Ap = A + lane * KP, *Bp = B + warp * w_main(CPW), *Bt = B + 4 * w_main(CPW) + 2 * warp;
#pragma unroll 1
    for (int k = 0; k < K; k += 4, Ap += 4, Bp += 4 * WB, Bt += 4 * WB) acc.template steps<KP>(Ap, Bp, Bt, K - k);
    __syncthreads();
    px_epilogue<CPW>(a, acc, A, outp, p0, npx, Wo, lane, warp);
}

template <int CPW, int TK> int launch_px(const ConvArgs &a, int Ho, int Wo, int K, cudaStream_t st)
{
    const int sm = 4 * std::max(PXS * px_stage(CPW, TK), 4 * PXT * epi_pitch(CPW));
    CNNCRF_CUDA(allow_smem(k_conv_px<CPW, TK>));
    CNNCRF_PROF("conv_simt", st);
    k_conv_px<CPW, TK><<<dim3(ceil_div((long)Ho * Wo, PXT), a.n_img), 128, sm, st>>>(a, Ho * Wo, Wo, K);
    return CNNCRF_OK;
}

template <int CPW, int KP> int launch_patch(const ConvArgs &a, int Ho, int Wo, int K, cudaStream_t st)
{
    const int sm = 4 * std::max(PXT * KP + K * w_pitch(CPW), 4 * PXT * epi_pitch(CPW));
    CNNCRF_CUDA(allow_smem(k_conv_patch<CPW, KP>));
    CNNCRF_PROF("conv_first", st);
    k_conv_patch<CPW, KP><<<dim3(ceil_div((long)Ho * Wo, PXT), a.n_img), 128, sm, st>>>(a, Ho * Wo, Wo, K);
    return CNNCRF_OK;
}

// the floats of bit patterns first .. first + 2 npairs - 1 for which tanh_pair is not cnncrf_tanhf, counted (NaN equals NaN)
__global__ void __launch_bounds__(256) k_tanh_sweep(uint32_t first, uint32_t npairs, unsigned long long *differing)
{
    uint32_t bad = 0;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < npairs; i += (long)gridDim.x * blockDim.x) {
        const uint32_t b = first + 2 * (uint32_t)i;
        const float x[2] = {__uint_as_float(b), __uint_as_float(b + 1)};
        const float2 t = tanh_pair(make_float2(x[0], x[1]));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float got = k ? t.y : t.x, want = cnncrf_tanhf(x[k]);
            bad += __float_as_uint(got) != __float_as_uint(want) && !(got != got && want != want);
        }
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(differing, (unsigned long long)bad);
}

__global__ void k_head2(const float *__restrict__ in, int npx, int Cin, const float *__restrict__ w,
                        float *__restrict__ out)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npx) return;
    in += (long)blockIdx.y * npx * Cin; // image of the batch
    out += (long)blockIdx.y * 2 * npx;
    const float *x = in + (long)p * Cin;
    float a0 = 0.0f, a1 = 0.0f;
    for (int ci = 0; ci < Cin; ++ci) {
        float v = x[ci];
        a0 = __fmaf_rn(w[ci], v, a0);
        a1 = __fmaf_rn(w[Cin + ci], v, a1);
    }
    out[p] = fabsf(a0);
    out[(long)npx + p] = fabsf(a1);
}

// Per pixel x / |x|, |x| = sqrt of the channel sum of squares in ascending c
// (one fmaf per term).  A CTA stages L2N pixels' channels in shared memory
// (row stride C + 1, odd: the per-pixel reads hit distinct banks) so the
// global reads and writes are contiguous, and one thread per pixel keeps the
// sequential sum.
constexpr int L2N = 64;
__global__ void __launch_bounds__(L2N) k_l2norm(float *__restrict__ f, long npx, int C)
{
    extern __shared__ float xs[]; // [L2N][C + 1]
    const long p0 = (long)blockIdx.x * L2N;
    const int n = (int)min((long)L2N, npx - p0), CS = C + 1;
    float *g = f + p0 * C;
    for (int i = threadIdx.x; i < n * C; i += L2N) {
        const int q = i / C;
        xs[q * CS + (i - q * C)] = g[i];
    }
    __syncthreads();
    if (threadIdx.x < n) {
        float *x = xs + threadIdx.x * CS;
        float s = 0.0f;
        for (int c = 0; c < C; ++c) s = __fmaf_rn(x[c], x[c], s);
        const float nr = __fsqrt_rn(s);
        for (int c = 0; c < C; ++c) x[c] = nr > 0.0f ? __fdiv_rn(x[c], nr) : 0.0f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * C; i += L2N) {
        const int q = i / C;
        g[i] = xs[q * CS + (i - q * C)];
    }
}

} // namespace

int conv_simt(const ConvArgs &args, cudaStream_t st)
{
    ConvArgs a = args;
    if (a.Cout > BN) return fail(CNNCRF_EINVAL, "conv_simt: Cout %d > %d", a.Cout, BN);
    int Ho = a.H - a.kh + 1, Wo = a.W - a.kw + 1;
    if (Ho <= 0 || Wo <= 0) return fail(CNNCRF_ESHAPE, "conv_simt: empty output");
    int K = a.kh * a.kw * a.Cin;
    const bool dense = a.out_pix == 0;
    if (dense) a.out_pix = a.Cout, a.out_row = (long)Wo * a.Cout, a.out_ch = 1;
    // k_conv_patch: K = 9 (grey), 27 (RGB), 45 (RGB and coordinates) of a first 3x3 layer
    if (!a.out16 && K <= 52 && a.Cout > 32 && a.Cout <= 104 && (long)Ho * Wo < (1L << 31) && a.n_img <= 65535) {
        auto launch = [&](auto cpw) {
            constexpr int CPW = decltype(cpw)::value;
            return K <= 12   ? launch_patch<CPW, 12>(a, Ho, Wo, K, st)
                   : K <= 28 ? launch_patch<CPW, 28>(a, Ho, Wo, K, st)
                             : launch_patch<CPW, 52>(a, Ho, Wo, K, st);
        };
        CNNCRF_TRY(a.Cout <= 64 ? launch(std::integral_constant<int, 16>()) : launch(std::integral_constant<int, 26>()));
        CNNCRF_CHECK_LAUNCH();
        return CNNCRF_OK;
    }
    // k_conv_px: 16-byte pixels, slices inside a tap, 32-bit offsets within an image
    const bool al16 = (((uintptr_t)a.in | (uintptr_t)a.wt) & 15) == 0 && a.in_pix % 4 == 0 && a.in_row % 4 == 0 &&
                      a.in_img % 4 == 0 && a.Cin % 4 == 0;
    const bool off32 = (long)a.H * a.in_row < (1L << 31) && (long)Ho * Wo < (1L << 31);
    if (al16 && off32 && !a.out16 && a.n_img <= 65535 && (a.Cin % 20 == 0 || a.Cin % 16 == 0)) {
        const bool t20 = a.Cin % 20 == 0;
        if (a.Cout > 64 && a.Cout <= 104) {
            CNNCRF_TRY((t20 ? launch_px<26, 20>(a, Ho, Wo, K, st) : launch_px<26, 16>(a, Ho, Wo, K, st)));
            CNNCRF_CHECK_LAUNCH();
            return CNNCRF_OK;
        }
        if (a.Cout > 32 && a.Cout <= 64) {
            CNNCRF_TRY((t20 ? launch_px<16, 20>(a, Ho, Wo, K, st) : launch_px<16, 16>(a, Ho, Wo, K, st)));
            CNNCRF_CHECK_LAUNCH();
            return CNNCRF_OK;
        }
    }
    dim3 grid(ceil_div(Wo, BM), Ho, a.n_img);
    {
        CNNCRF_PROF("conv_simt", st);
        if (a.Cout <= 32) k_conv_nt<32, 8><<<grid, 64, 0, st>>>(a, Ho, Wo, K);
        else if (a.Cout <= 64) k_conv_nt<64, 8><<<grid, 128, 0, st>>>(a, Ho, Wo, K);
        else if (a.Cout <= 112) k_conv_nt<112, 14><<<grid, 224, 0, st>>>(a, Ho, Wo, K);
        else k_conv_simt<<<grid, 256, 0, st>>>(a, Ho, Wo, K);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int selftest_tanh(uint32_t first, uint64_t count, uint64_t *differing, cudaStream_t st)
{
    if (!differing || count < 2 || count % 2 || first + count > (1ull << 32))
        return fail(CNNCRF_EINVAL, "selftest: floats %u .. + %llu", first, (unsigned long long)count);
    DevBuf n;
    CNNCRF_TRY(n.reserve(sizeof(unsigned long long)));
    CNNCRF_CUDA(cudaMemsetAsync(n.get(), 0, sizeof(unsigned long long), st));
    {
        CNNCRF_PROF("tanh_sweep", st);
        k_tanh_sweep<<<(int)std::min<uint64_t>((count / 2 + 255) / 256, 8 * 152), 256, 0, st>>>(first, (uint32_t)(count / 2),
                                                                                            n.as<unsigned long long>());
    }
    CNNCRF_CHECK_LAUNCH();
    CNNCRF_CUDA(cudaMemcpyAsync(differing, n.get(), sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    CNNCRF_CUDA(cudaStreamSynchronize(st));
    return CNNCRF_OK;
}

int conv_head2(const float *in, int npx, int Cin, const float *w, float *out, cudaStream_t st, int n_img)
{
    {
        CNNCRF_PROF("head2", st);
        k_head2<<<dim3(ceil_div(npx, 256), n_img), 256, 0, st>>>(in, npx, Cin, w, out);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int l2norm(float *f, long npx, int C, cudaStream_t st)
{
    {
        CNNCRF_PROF("l2norm", st);
        const size_t sm = sizeof(float) * L2N * (size_t)(C + 1);
        if (sm > 48 * 1024) return fail(CNNCRF_EINVAL, "l2norm: %d channels", C);
        k_l2norm<<<ceil_div(npx, L2N), L2N, sm, st>>>(f, npx, C);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

} // namespace k
} // namespace cnncrf

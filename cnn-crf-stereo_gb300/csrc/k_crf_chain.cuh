// k_crf_chain.cuh -- the chain pass of the CRF solve (k_crf.cu), shared by
// the translation units that instantiate it for their label counts per lane
// (k_crf.cu: 4, k_crf_p12.cu: 1 and 2, k_crf_p6.cu, k_crf_p8.cu), so they
// compile in parallel.  Everything device-side has internal linkage; each
// unit exports launchers, crf_pass_p<P>.
#ifndef CNNCRF_K_CRF_CHAIN_CUH
#define CNNCRF_K_CRF_CHAIN_CUH

#include <cfloat>
#include <math_constants.h>

#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

// pairwise term: rho[t] for |t| = 0..8 (t > delta: L2), slack fraction
struct Rho {
    float rho[9];
    float L2;
    float slack;
};

// one pass over all chains of one direction (see k_crf_chain)
struct CrfPassArgs {
    const float *theta; // the cost volume [np][H][W][D]
    const uint16_t *thetaq; // its 16-bit fixed-point copy, read by the H pass instead of theta when set
    float qscale, qoffset;  // theta = q * qscale + qoffset (exact in FP32)
    float qoffset23;        // qoffset - 2^23 qscale, exact: theta = (2^23 + q) * qscale + qoffset23
    float *phi;         // H/V split of the unary [np][H][W][DP]
    const float *wgt;   // wx (H pass) or wy (V pass), pair stride wps
    float *lbuf;        // each block's first forward message, [np][H][blocks][DP] in an H pass, [np][blocks][W][DP] in a V pass
    int W, H, D, np;
    int DP;              // labels from one vector of phi and lbuf to the next: D rounded up to 4, or D (layout, k_crf.cu)
    long wps;
    Rho rp;
    int first;           // H pass of the first iteration: phi = 0, not read
    int store_phi;       // 0: the pass's phi is dead (the last V pass when no caller reads C1), not written
    int32_t *labels;     // V pass of the last iteration: argmin labels, else null
    double *cmin;        // per chain minimum [np][chains]
};

// how a pass runs: every choice gives the same bits
struct CrfForm {
    bool paired; // two warps per chain, else one
    int buffers; // blocks of BLK nodes in shared memory (2 or 3)
    int wpb;     // chains per CTA (paired: always one)
};

constexpr int BLK = 8; // chain nodes per block

// launch one pass; EUNSUPPORTED when the CTA's shared memory would exceed the limit
int crf_pass_p1(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st);
int crf_pass_p2(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st);
int crf_pass_p4(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st);
int crf_pass_p6(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st);
int crf_pass_p8(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st);

// how a pass's vectors lie in memory: on 16 bytes throughout; the cost volume's on any float and phi's on 16 bytes (an H
// pass whose D is no multiple of 4); both on any float
enum : int { ALIGNED = 0, SPREAD = 1, RAGGED = 2 };
inline int vec_mode(const CrfPassArgs &a, bool hpass)
{
    return a.D % 4 == 0 ? ALIGNED : (a.DP % 4 ? RAGGED : (hpass ? SPREAD : ALIGNED));
}

// a chain's shared memory in floats: per block buffer two planes of BLK node vectors, the unary (H pass; 16-bit codes
// take half the floats) and phi (RAGGED vectors carry up to 3 floats of their neighbours at either end); one block of
// messages and of edge costs, or two with paired warps
__host__ __device__ constexpr int vec_floats(int P, int mode) { return 32 * P + (mode == RAGGED ? 4 : 0); }
__host__ __device__ constexpr int theta_floats(int P, bool hpass, bool t16, int mode)
{
    return hpass ? BLK * (t16 ? 16 * P : vec_floats(P, mode)) : 0;
}
__host__ __device__ constexpr int block_floats(int P, bool hpass, bool t16, int mode)
{
    return theta_floats(P, hpass, t16, mode) + BLK * vec_floats(P, mode);
}
constexpr int EDGE = 8;                // EDGE: floats of an edge's costs (w rho_1 .. w rho_4, w L2)
constexpr int EDGES = (BLK + 1) * EDGE;       // of the edges a block uses
__host__ __device__ constexpr int chain_floats(int P, bool hpass, bool t16, int mode, bool paired, int buffers)
{
    return buffers * block_floats(P, hpass, t16, mode) + (paired ? 2 : 1) * (BLK * 32 * P + EDGES);
}

namespace {

#define INF CUDART_INF_F

// Exact two-lane IEEE operations (add/sub/mul/fma.rn.f32x2) and three-input
// minimum (min.f32 with three sources): the same values as two __fadd_rn and
// two fminf, in fewer instructions.
__device__ __forceinline__ void add2(float a0, float a1, float b0, float b1, float &d0, float &d1)
{
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void sub2(float a0, float a1, float b0, float b1, float &d0, float &d1)
{
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}
__device__ __forceinline__ void mul2(float a0, float a1, float b, float &d0, float &d1)
{
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %4};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b));
}
__device__ __forceinline__ void fma2(float a0, float a1, float b, float c, float &d0, float &d1)
{
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %4};\n\t"
        "mov.b64 rc, {%5, %5};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d0), "=f"(d1)
        : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ float min3(float a, float b, float c)
{
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// element-wise over a lane's P labels, in pairs
template <int P> __device__ __forceinline__ void vadd(const float (&a)[P], const float (&b)[P], float (&d)[P])
{
#pragma unroll
    for (int r = 0; r + 1 < P; r += 2) add2(a[r], a[r + 1], b[r], b[r + 1], d[r], d[r + 1]);
    if constexpr (P % 2) d[P - 1] = __fadd_rn(a[P - 1], b[P - 1]);
}
template <int P> __device__ __forceinline__ void vsub(const float (&a)[P], const float (&b)[P], float (&d)[P])
{
#pragma unroll
    for (int r = 0; r + 1 < P; r += 2) sub2(a[r], a[r + 1], b[r], b[r + 1], d[r], d[r + 1]);
    if constexpr (P % 2) d[P - 1] = __fsub_rn(a[P - 1], b[P - 1]);
}
template <int P> __device__ __forceinline__ void vsub1(const float (&a)[P], float b, float (&d)[P])
{
#pragma unroll
    for (int r = 0; r + 1 < P; r += 2) sub2(a[r], a[r + 1], b, b, d[r], d[r + 1]);
    if constexpr (P % 2) d[P - 1] = __fsub_rn(a[P - 1], b);
}
template <int P> __device__ __forceinline__ void vmul1(const float (&a)[P], float b, float (&d)[P])
{
#pragma unroll
    for (int r = 0; r + 1 < P; r += 2) mul2(a[r], a[r + 1], b, d[r], d[r + 1]);
    if constexpr (P % 2) d[P - 1] = __fmul_rn(a[P - 1], b);
}

// The warp minimum of the lanes' minima: one redux.sync.min.f32 (sm_100 and
// later), exact like a float min.  A zero may come back with either sign,
// which no later operation distinguishes (the labels compare values, the
// bound adds them).  `none`: what pad labels stand for, +inf or NaN
// (pad_value); it turns a lane of pads, which the slack hand-over leaves at
// NaN, back into +inf.
template <int P> __device__ __forceinline__ float warp_min(const float (&v)[P], float none)
{
    float m;
    if constexpr (P == 1) m = fminf(v[0], none);
    else if constexpr (P == 2) m = min3(v[0], v[1], none);
    else {
        m = min3(v[0], v[1], v[2]);
#pragma unroll
        for (int r = 3; r + 1 < P; r += 2) m = min3(m, v[r], v[r + 1]);
        if constexpr (P % 2 == 0) m = min3(m, v[P - 1], none);
    }
    float w;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(w) : "f"(m));
    return w;
}

// The value of pad labels.  A minimum takes its other operand either way; where no label has a finite cost, +inf makes the
// minimum +inf, and NaN leaves it NaN as it is without pads.  So the label counts that fill their lanes at 1, 2, 3, 4, 6 or
// 8 labels each have NaN (96 labels run in lanes of 4)
__device__ __forceinline__ float pad_value(int D) { return D % 32 == 0 && D != 160 && D != 224 ? CUDART_NAN_F : INF; }

// Lane constants: 0, or +inf in the lanes whose neighbour `o` lanes below
// (lo) or above (hi) is outside the warp.  Added to a neighbour's value they
// put +inf beyond label 0 and label 32 P - 1; labels D..32 P - 1 carry +inf
// or NaN themselves (a minimum takes its other operand).
template <int P, int DELTA> struct Edge {
    static constexpr int NO = (DELTA + P - 1) / P;
    float lo[NO + 1], hi[NO + 1];
    float none; // warp_min's
    __device__ __forceinline__ Edge(int lane, float pad) : none(pad)
    {
#pragma unroll
        for (int o = 1; o <= NO; ++o) lo[o] = lane < o ? INF : 0.0f, hi[o] = lane + o > 31 ? INF : 0.0f;
    }
};

// out = minconv(v) - g with out_k = min(v_k, v_{k+-t} + w rho_t (t <= DELTA), g + w L2) - g; returns g = min v.  cw: the
// edge's w L2, w rho_1, ..  This is the chain's critical path: the neighbours' labels are sent off first, the minimum and
// what a lane's own labels give are worked out while they travel, and an arriving label takes one addition, of its cost
// with the edge constant in it, and one minimum.
template <int P, int DELTA>
__device__ __forceinline__ float minconv(const float (&v)[P], const float (&cw)[EDGE], const Edge<P, DELTA> &ed, float (&out)[P])
{
    float lo[DELTA + 1], hi[DELTA + 1]; // labels lane P - t and lane P + P - 1 + t
#pragma unroll
    for (int t = 1; t <= DELTA; ++t) {
        const int ol = (t + P - 1) / P, rl = (P - t % P) % P;
        const int oh = (P - 1 + t) / P, rh = (P - 1 + t) % P;
        lo[t] = __shfl_up_sync(0xffffffffu, v[rl], ol);
        hi[t] = __shfl_down_sync(0xffffffffu, v[rh], oh);
    }
    const float g = warp_min<P>(v, ed.none), base = __fadd_rn(g, cw[0]);
    float o[P], pend[P]; // pend: a value not yet in the minimum o, so that they go in by pairs
    bool has[P];
#pragma unroll
    for (int r = 0; r < P; ++r) o[r] = v[r], pend[r] = INF, has[r] = false;
    auto put = [&](int r, float x) {
        if (has[r]) o[r] = min3(o[r], pend[r], x);
        else pend[r] = x;
        has[r] = !has[r];
    };
#pragma unroll
    for (int t = 1; t <= DELTA; ++t) {
        float S[P + 1];
#pragma unroll
        for (int i = 0; i < P; i += 2) {
            if (i + 1 < P) add2(v[i], v[i + 1], cw[t], cw[t], S[i], S[i + 1]);
            else S[i] = __fadd_rn(v[i], cw[t]);
        }
#pragma unroll
        for (int r = 0; r < P; ++r) {
            if (r - t >= 0) put(r, S[r - t]);
            if (r + t < P) put(r, S[r + t]);
        }
    }
#pragma unroll
    for (int r = 0; r < P; ++r) put(r, base);
#pragma unroll
    for (int t = 1; t <= DELTA; ++t)
#pragma unroll
        for (int q = 1; q <= t; ++q) { // the label q beyond the lane's, t from label r
            const int ol = (q + P - 1) / P, oh = (P - 1 + q) / P;
            if (t - q < P) put(t - q, __fadd_rn(lo[q], __fadd_rn(cw[t], ed.lo[ol])));
            if (t - q < P) put(P - 1 - (t - q), __fadd_rn(hi[q], __fadd_rn(cw[t], ed.hi[oh])));
        }
#pragma unroll
    for (int r = 0; r < P; ++r)
        if (has[r]) o[r] = fminf(o[r], pend[r]);
    vsub1<P>(o, g, out);
    return g;
}

// ---------------------------------------------------------------- copies
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// the first `bytes` of a 16-byte chunk (zeros after them)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// all but the newest `left` groups (0 or 1) are complete
__device__ __forceinline__ void cp_wait_left(int left)
{
    if (left == 0) cp_wait<0>();
    else cp_wait<1>();
}

// `cnt` consecutive vectors of 32 P labels of EB bytes that lie one after the
// other, into a plane: one flat run of 16-byte chunks
template <int P, int EB> __device__ __forceinline__ void copy_run(uint32_t dst, const void *src, int lane, int cnt)
{
    constexpr int NC = BLK * 2 * P * EB; // chunks of a whole block
    const char *g = (const char *)src + 16 * lane;
    const uint32_t d = dst + 16 * lane;
    if (cnt == BLK) {
#pragma unroll
        for (int c = 0; c < NC; c += 32)
            if (c + 32 <= NC || lane + c < NC) cp_async16(d + 16 * c, g + 16 * c);
    } else {
        for (int c = 0; lane + c < cnt * (NC / BLK); c += 32) cp_async16(d + 16 * c, g + 16 * c);
    }
}
// `cnt` vectors of D labels (a multiple of 4) at a stride of ns labels, into a
// plane.  A vector of 32 or 64 labels takes 8 or 16 lanes, so that a copy
// instruction then carries 4 or 2 nodes.
template <int P> __device__ __forceinline__ void copy_nodes(uint32_t dst, const float *src, long ns, int lane, int cnt, int D)
{
    if (P <= 2 && D == 32 * P) {
        constexpr int LN = 8 * (P <= 2 ? P : 4), NI = 32 / LN; // lanes per node, nodes per instruction
        const float *g = src + (lane / LN) * ns + 4 * (lane % LN);
        const uint32_t d = dst + 16 * lane;
#pragma unroll
        for (int j = 0; j < BLK; j += NI, g += NI * ns)
            if (j + lane / LN < cnt) cp_async16(d + 16 * LN * j, g);
    } else {
        const float *g = src + 4 * lane;
        uint32_t d = dst + 16 * lane;
        auto node = [&]() {
#pragma unroll
            for (int c = 0; c < 8 * P; c += 32)
                if (4 * (lane + c) < D) cp_async16(d + 16 * c, g + 4 * c);
            g += ns, d += 128 * P;
        };
        if (cnt == BLK) {
#pragma unroll
            for (int j = 0; j < BLK; ++j) node();
        } else {
            for (int j = 0; j < cnt; ++j) node();
        }
    }
}

// `cnt` vectors of any D labels from element o0 of a 16-byte aligned array of `total` elements, at a stride of ns: the
// 16-byte chunks that hold each one (element o lands o % 4 floats into its slot), cut off at the array's end
template <int P> __device__ __forceinline__ void copy_ragged(uint32_t dst, const float *base, long o0, long ns, long total, int lane,
                                                             int cnt, int D)
{
    uint32_t d = dst + 16 * lane;
    long o = o0;
    auto node = [&]() {
        const int mis = (int)(o & 3);
        const long c0 = o - mis + 4 * lane; // this lane's chunk
#pragma unroll
        for (int c = 0; c < 8 * P + 1; c += 32)
            if (4 * (lane + c) < D + mis) cp_async16(d + 16 * c, base + c0 + 4 * c, 4 * (int)min(4L, total - c0 - 4 * c));
        o += ns, d += 4 * vec_floats(P, RAGGED);
    };
    if (cnt == BLK) {
#pragma unroll
        for (int j = 0; j < BLK; ++j) node();
    } else {
        for (int j = 0; j < cnt; ++j) node();
    }
}

// `cnt` vectors of any D labels that lie one after the other, into slots of 32 P labels, float by float
template <int P> __device__ __forceinline__ void copy_spread(uint32_t dst, const float *src, int lane, int cnt, int D)
{
    const float *g = src + lane;
    uint32_t d = dst + 4 * lane;
    auto node = [&]() {
#pragma unroll
        for (int c = 0; c < P; ++c)
            if (lane + 32 * c < D) cp_async4(d + 128 * c, g + 32 * c);
        g += D, d += 128 * P;
    };
    if (cnt == BLK) {
#pragma unroll
        for (int j = 0; j < BLK; ++j) node();
    } else {
        for (int j = 0; j < cnt; ++j) node();
    }
}

// dequantise: q * scale + offset is exact (q < 2^16, scale a power of two,
// the sum a multiple of scale below 2^9 in magnitude).  The code goes into
// the low mantissa bits of 2^23 by one byte permute, which makes the float
// 2^23 + q exactly, and offset23 = offset - 2^23 scale (exact, checked on the
// host) takes the 2^23 back out inside the one rounding of the fma:
// (2^23 + q) scale + offset23 = q scale + offset.
template <int P>
__device__ __forceinline__ void read16(const float *slot, int lane, float scale, float offset23, float (&v)[P])
{
    uint32_t w[P / 2];
    const uint32_t *q = (const uint32_t *)slot + lane * (P / 2);
    if constexpr (P == 4) {
        const uint2 t = *(const uint2 *)q;
        w[0] = t.x, w[1] = t.y;
    } else if constexpr (P == 8) {
        const uint4 t = *(const uint4 *)q;
        w[0] = t.x, w[1] = t.y, w[2] = t.z, w[3] = t.w;
    } else {
#pragma unroll
        for (int i = 0; i < P / 2; ++i) w[i] = q[i];
    }
#pragma unroll
    for (int i = 0; i < P / 2; ++i) {
        const float lo = __int_as_float((int)__byte_perm(w[i], 0x4B000000u, 0x7410)); // bytes w0, w1, 0x00, 0x4B
        const float hi = __int_as_float((int)__byte_perm(w[i], 0x4B000000u, 0x7432)); // bytes w2, w3, 0x00, 0x4B
        fma2(lo, hi, scale, offset23, v[2 * i], v[2 * i + 1]);
    }
}

// a lane's P labels of a vector in shared memory (slots are 16-byte aligned)
template <int P> __device__ __forceinline__ void read_vec(const float *slot, int lane, float (&v)[P])
{
    const float *q = slot + lane * P;
    if constexpr (P % 4 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 4) {
            const float4 t = *(const float4 *)(q + i);
            v[i] = t.x, v[i + 1] = t.y, v[i + 2] = t.z, v[i + 3] = t.w;
        }
    } else if constexpr (P % 2 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 2) {
            const float2 t = *(const float2 *)(q + i);
            v[i] = t.x, v[i + 1] = t.y;
        }
    } else {
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = q[r];
    }
}

template <int P> __device__ __forceinline__ void read_raw(const float *slot, int lane, float (&v)[P])
{
#pragma unroll
    for (int r = 0; r < P; ++r) v[r] = slot[lane * P + r];
}

// store a lane's P labels to p (shared or global; the labels below D); ALIGNED: 16-byte aligned vectors, D a multiple of 4
template <int P, bool ALIGNED> __device__ __forceinline__ void write_vec(float *p, int lane, int D, const float (&v)[P])
{
    const int k0 = lane * P;
    if constexpr (ALIGNED && P % 4 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 4)
            if (k0 + i < D) *(float4 *)(p + k0 + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else if constexpr (ALIGNED && P % 2 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 2)
            if (k0 + i < D) *(float2 *)(p + k0 + i) = make_float2(v[i], v[i + 1]);
    } else {
#pragma unroll
        for (int r = 0; r < P; ++r)
            if (k0 + r < D) p[k0 + r] = v[r];
    }
}
// load a lane's P labels from global memory (0 from label D on)
template <int P, bool ALIGNED> __device__ __forceinline__ void load_vec(const float *p, int lane, int D, float (&v)[P])
{
    const int k0 = lane * P;
#pragma unroll
    for (int r = 0; r < P; ++r) v[r] = 0.0f;
    if constexpr (ALIGNED && P % 4 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 4)
            if (k0 + i < D) {
                const float4 t = *(const float4 *)(p + k0 + i);
                v[i] = t.x, v[i + 1] = t.y, v[i + 2] = t.z, v[i + 3] = t.w;
            }
    } else if constexpr (ALIGNED && P % 2 == 0) {
#pragma unroll
        for (int i = 0; i < P; i += 2)
            if (k0 + i < D) {
                const float2 t = *(const float2 *)(p + k0 + i);
                v[i] = t.x, v[i + 1] = t.y;
            }
    } else {
#pragma unroll
        for (int r = 0; r < P; ++r)
            if (k0 + r < D) v[r] = p[k0 + r];
    }
}

// One pass over the chains of one direction; one or two warps per chain.
//   HPASS: chain = row y over x (weights wx[y][x] on edge x -> x+1), unary
//          theta - phi, the handed-over slack is added to phi.
//   !HPASS: chain = column x over y (weights wy[y][x] on edge y -> y+1),
//          unary phi, the handed-over slack is subtracted from phi; labels
//          (if given) = first argmin of the min-marginals.
// A chain is walked in blocks of BLK nodes.  The block's pixel vectors come
// from a ring of block buffers in shared memory, filled `buffers` - 1 blocks
// ahead, so that the chain's dependent arithmetic does not wait on DRAM:
//   ALIGNED     16-byte cp.async by the whole warp, several nodes per
//               instruction where they are small or contiguous
//   SPREAD      D not a multiple of 4: phi as above, the volume's vectors
//               float by float into the same slots
//   RAGGED      the 16-byte chunks that hold each vector, where the workspace
//               does not hold phi at a pitch of whole chunks (k_crf.cu)
// Vectors at a pitch DP > D carry pad labels D..DP - 1 along.  The H pass
// that starts a solve stores them as +inf, a V pass turns that into NaN, and
// neither ever wins a minimum.  D = 75, of a 619 x 271 solve, against RAGGED
// vectors (four-way bank conflicts on each, masks, single-float stores): the H
// pass 196 -> 107 us, the V pass 106 -> 81 us, as D = 76; D = 255 of a KITTI
// pair 1354 -> 511 and 828 -> 377 us.  Measured and left out: the volume's
// block as one run of 16-byte copies, each lane shifting its labels into place
// (150 us) or the copying warp doing so once (155 us).
// An edge's costs w rho_t and w L2 are multiplied out once per block, an edge
// per lane, and read back as broadcasts.
//
// The forward sweep makes every node's message and the backward sweep needs
// them again in reverse.  Only each block's first message goes to memory; the
// others are recomputed from it, in shared memory, out of the pixel vectors
// the backward sweep reads anyway: a third sweep of arithmetic for 2 - 2/BLK
// fewer vectors moved per node (of the 16-bit H pass's 6 N D floats 4.25
// remain, of the V pass's 5, 3.25).
//   !PAIRED: one warp does it all; many chains hide its latencies.
//   PAIRED: a second warp per chain copies the blocks in and recomputes the
//     messages one block ahead of the first, which walks the chain: for few
//     chains, whose time is the sweeps' latency.  The two meet at a barrier
//     once per block; one chain per CTA.
//
// What bounds it: many chains, DRAM (eight KITTI pairs at D = 128: the H pass
// 7.98 GB by the counters in 1.22 ms, 6.56 TB/s, and the V pass 5.94 GB in 0.92
// ms, 6.46 TB/s; with all messages stored and read back 1.72 and 1.38 ms).  Few chains, the latency of
// a node's step, about 420 cycles for both sweeps of a KITTI pair's row: four
// halo shuffles issue 4.3 cycles apart and return after 24, the warp minimum
// after 18, and the copies of a block cost 18 cycles per instruction, which is
// why they are few and on the second warp (one pair's H pass 470 -> 252 us,
// its V pass 208 -> 154 us; the 256 x 192, D = 32 solve's 89 -> 39 and 70 ->
// 32 us).  The first warp's sweeps bound it: the forward one takes 160 to 185
// cycles a node, the backward one 200 to 230, as long without the second
// warp's recomputation.  Sending the halo off before the warp minimum gave 2
// to 5 % (256 x 192, D = 128: 48.6 -> 46.2 and 39.9 -> 38.5 us).  Measured and left out: bulk copies on mbarriers for the H blocks
// (a wait costs 150 cycles, cp.async's 43; 338 against 316 us for one pair),
// and keeping all messages for few chains (276 against 258 us).
template <int P, int DELTA, bool HPASS, bool T16, int MODE, bool PAIRED>
__global__ void __launch_bounds__(PAIRED ? 64 : 128) k_crf_chain(const CrfPassArgs a, const int NB)
{
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool walks = !PAIRED || warp == 0, helps = !PAIRED || warp == 1; // roles: walk the chain; copy and recompute
    const int wib = PAIRED ? 0 : warp; // the chain within the CTA
    const int gchain = PAIRED ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + wib;
    constexpr bool RAG = MODE == RAGGED, VEC = !RAG; // VEC: phi and lbuf in whole 16-byte chunks
    const int W = a.W, H = a.H, D = T16 ? 32 * P : a.D, DP = T16 ? 32 * P : (RAG ? a.D : a.DP);
    const int n = HPASS ? W : H;
    const int nch = HPASS ? H : W;
    if (gchain >= nch * a.np) return;
    // pair of the batch and chain within it
    const int pair = gchain / nch, chain = gchain - pair * nch;
    // element offset of the chain's node 0 and the stride between its nodes
    const long ns = (HPASS ? 1L : (long)W) * DP;
    const long cn = (long)W * H * pair + (HPASS ? (long)chain * W : (long)chain);
    const long cb = cn * DP, tcb = cn * D; // of phi; of theta (H passes: its nodes are D apart)
    const uint16_t *thetaq = T16 ? a.thetaq + tcb : nullptr;
    float *phi = a.phi + cb;
    const int nblk = (n + BLK - 1) / BLK;
    const long ls = (HPASS ? 1L : (long)W) * DP; // from a block's first message to the next block's
    float *lbuf = a.lbuf + (HPASS ? ((long)pair * H + chain) * nblk : (long)pair * nblk * W + chain) * DP;
    const float *wgt = a.wgt + a.wps * pair + (HPASS ? (long)chain * W : (long)chain);
    const long wst = HPASS ? 1 : W; // weight of edge e (node e to e + 1) at wgt[e wst]

    constexpr int LP = 32 * P, VF = vec_floats(P, MODE), TF = T16 ? 16 * P : VF; // TF: of a node's unary
    constexpr int OP = theta_floats(P, HPASS, T16, MODE); // planes of a buffer: the unary at 0, phi at OP
    constexpr int BF = block_floats(P, HPASS, T16, MODE), MF = BLK * LP + EDGES;
    float *ring = (float *)smem4 + (size_t)wib * chain_floats(P, HPASS, T16, MODE, PAIRED, NB);
    float *msg = ring + NB * BF; // the block's messages and edge costs (PAIRED: of even and odd blocks of the sweep)
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    const bool use_phi = !(HPASS && a.first);

    // Labels DP..32 P - 1 (of a SPREAD unary D..) are pads: set once,
    // the copies never write them (RAGGED slots hold other vectors' labels
    // there, and read_node masks them).  The first H pass copies no phi: zero.
    const float none = pad_value(D);
    if (helps && (D < LP || !use_phi)) {
        for (int i = lane; i < NB * BLK * VF; i += 32) {
            const int nd = i / VF, k = i - nd * VF, q = nd / BLK, j = nd - q * BLK;
            float *s = ring + q * BF;
            const bool pad = k >= DP;
            if (HPASS) {
                if (!T16 && (pad || (MODE == SPREAD && k >= D))) s[j * TF + k] = none;
                if (pad || !use_phi) s[OP + j * VF + k] = 0.0f;
            } else if (pad) {
                s[OP + j * VF + k] = none;
            }
        }
    }
    __syncwarp();

    int ibuf = 0; // the buffer of the next copied block
    // copy block b into the next buffer
    auto issue = [&](int b) {
        if (b >= 0 && b < nblk) {
            const int i0 = b * BLK, cnt = min(BLK, n - i0);
            const uint32_t d = ring_s + (uint32_t)(ibuf * BF) * 4u;
            const long o = (long)i0 * ns;
            if constexpr (!RAG) {
                if constexpr (HPASS) {
                    const long to = tcb + (long)i0 * D;
                    if constexpr (T16) copy_run<P, 2>(d, thetaq + (long)i0 * D, lane, cnt);
                    else if constexpr (MODE == SPREAD) copy_spread<P>(d, a.theta + to, lane, cnt, D);
                    else if (D == LP) copy_run<P, 4>(d, a.theta + to, lane, cnt);
                    else copy_nodes<P>(d, a.theta + to, D, lane, cnt, D);
                }
                if (HPASS && DP == LP) {
                    if (use_phi) copy_run<P, 4>(d + OP * 4, phi + o, lane, cnt);
                } else {
                    if (use_phi) copy_nodes<P>(d + OP * 4, phi + o, ns, lane, cnt, DP);
                }
            } else {
                const long total = (long)W * H * D * a.np;
                if (HPASS) copy_ragged<P>(d, a.theta, cb + o, ns, total, lane, cnt, D);
                if (use_phi) copy_ragged<P>(d + OP * 4, a.phi, cb + o, ns, total, lane, cnt, D);
            }
            ibuf = ibuf + 1 == NB ? 0 : ibuf + 1;
        }
        cp_commit();
    };
    // the next block is in its buffer, every lane is done with the one before it
    int buf = 0;
    auto arrived = [&]() {
        cp_wait_left(NB - 2);
        __syncwarp();
    };
    // PAIRED: the two warps of the chain (the CTA) meet
    auto meet = [&]() {
        if constexpr (PAIRED) __syncthreads();
    };
    auto next_buf = [&]() -> const float * {
        const float *p = ring + buf * BF;
        buf = buf + 1 == NB ? 0 : buf + 1;
        return p;
    };
    // lane l < BLK + 1: the weight of edge BLK b - 1 + l
    auto weights = [&](int b) -> float {
        const int e = b * BLK - 1 + lane;
        return (b >= 0 && lane <= BLK && e >= 0 && e < n - 1) ? __ldg(wgt + (long)e * wst) : 0.0f;
    };
    // that edge's costs: w L2, w rho_1, .., w rho_DELTA
    auto edge_costs = [&](float w, float *ec) {
        float c[EDGE];
        c[0] = __fmul_rn(w, a.rp.L2);
#pragma unroll
        for (int t = 1; t < EDGE; ++t) c[t] = t <= DELTA ? __fmul_rn(w, a.rp.rho[t]) : 0.0f;
        if (lane <= BLK) {
            *(float4 *)(ec + lane * EDGE) = make_float4(c[0], c[1], c[2], c[3]);
            if (DELTA > 3) ec[lane * EDGE + 4] = c[4];
        }
    };
    // a node's inputs: the subproblem's unary (theta - phi, or phi), phi, and the costs of the edge its message crosses.
    // Every sweep reads them one node ahead of the chain's arithmetic, which so waits neither on shared memory nor on
    // the dequantisation
    struct Node {
        float un[P], ph[P], vm[P], cw[EDGE];
    };
    auto read_plane = [&](const float *bs, int j, long o, float (&x)[P]) {
        if constexpr (RAG) read_raw<P>(bs + j * VF + (int)(o & 3), lane, x);
        else read_vec<P>(bs + j * VF, lane, x);
    };
    auto read_node = [&](const float *bs, int i0, int j, Node &nd) {
        const long o = RAG ? cb + (long)(i0 + j) * ns : 0;
        if constexpr (HPASS) {
            float th[P];
            if constexpr (T16) read16<P>(bs + j * TF, lane, a.qscale, a.qoffset23, th);
            else read_plane(bs, j, o, th);
            read_plane(bs + OP, j, o, nd.ph);
            vsub<P>(th, nd.ph, nd.un);
        } else {
            read_plane(bs + OP, j, o, nd.un);
        }
        if constexpr (RAG)
#pragma unroll
            for (int r = 0; r < P; ++r) nd.un[r] = lane * P + r < D ? nd.un[r] : INF;
    };
    auto read_edge = [&](const float *ec, int j, Node &nd) { // slot j: edge i0 - 1 + j
        const float4 t = *(const float4 *)(ec + j * EDGE);
        nd.cw[0] = t.x, nd.cw[1] = t.y, nd.cw[2] = t.z, nd.cw[3] = t.w;
        if (DELTA > 3) nd.cw[4] = ec[j * EDGE + 4];
    };

    const Edge<P, DELTA> ed(lane, none);
    float L[P], v[P];
    Node cur, nxt;
#pragma unroll
    for (int r = 0; r < P; ++r) L[r] = 0.0f;

    double cmin = 0.0;
    float R[P], m[P], Lc[P];
#pragma unroll
    for (int r = 0; r < P; ++r) R[r] = 0.0f, Lc[r] = 0.0f;

    // block b again from its first message, Lc: message plus unary of every node, into ms; the first message of the
    // sweep's next block loads meanwhile
    auto recompute = [&](int b, const float *bs, float *ms) {
        const int i0 = b * BLK, cnt = min(BLK, n - i0);
        const float *ec = ms + BLK * LP;
#pragma unroll
        for (int r = 0; r < P; ++r) L[r] = b > 0 ? Lc[r] : 0.0f;
        if (b > 1) load_vec<P, VEC>(lbuf + (b - 1) * ls, lane, DP, Lc);
        read_node(bs, i0, 0, nxt);
        read_edge(ec, 1, nxt);
        auto again = [&](int j, bool more) { // more: another node follows in the block
            cur = nxt;
            if (more) {
                read_node(bs, i0, j + 1, nxt);
                read_edge(ec, j + 2, nxt);
            }
            vadd<P>(L, cur.un, v);
            write_vec<P, true>(ms + j * LP, lane, LP, v);
            if (more) {
                minconv<P, DELTA>(v, cur.cw, ed, L);
            }
        };
        if (cnt == BLK) {
#pragma unroll
            for (int j = 0; j < BLK; ++j) again(j, j < BLK - 1);
        } else {
#pragma unroll 1
            for (int j = 0; j < cnt; ++j) again(j, j < cnt - 1);
        }
    };

    if (PAIRED && !walks) { // ---- the second warp: copies, and the messages of the backward sweep
        float wn = weights(0), *ms = msg;
        for (int b = 0; b < NB - 1; ++b) issue(b);
        for (int b = 0; b < nblk; ++b) {
            edge_costs(wn, ms + BLK * LP);
            wn = weights(b + 1);
            ms = ms == msg ? msg + MF : msg;
            arrived();
            meet(); // block b is there; block b - 1's buffer is free
            issue(b + NB - 1);
            next_buf();
        }
        cp_wait<0>();
        meet(); // the first messages are in memory
        for (int q = 0; q < NB - 1; ++q) issue(nblk - 1 - q);
        if (nblk > 1) load_vec<P, VEC>(lbuf + (nblk - 1) * ls, lane, DP, Lc);
        wn = weights(nblk - 1), ms = msg;
        for (int b = nblk - 1; b >= 0; --b) {
            edge_costs(wn, ms + BLK * LP);
            wn = weights(b - 1);
            arrived();
            recompute(b, next_buf(), ms);
            meet(); // block b and its messages are there; block b + 1's buffers are free
            issue(b - (NB - 1));
            ms = ms == msg ? msg + MF : msg;
        }
        cp_wait<0>();
        return;
    }

    // ---- forward: messages into each node.  The chain's minimum in FP64:
    // lane l sums the node minima g_i of i = l mod 32 in ascending i, and the
    // 32 partial sums are added in lane order at the end of the sweep.  Lane l
    // keeps node 32 b + l's minimum as a float (gb) and adds it once per 32
    // nodes: no FP64 operation on the message chain
    double acc = 0.0;
    float gb = 0.0f;
    if (!PAIRED)
        for (int b = 0; b < NB - 1; ++b) issue(b);
    float wn = PAIRED ? 0.0f : weights(0), *ms = msg;
    long so = 0; // element offset of the message being stored, then of the node's phi
    for (int b = 0; b < nblk; ++b) {
        meet();
        if (!PAIRED) {
            arrived();
            issue(b + NB - 1);
        }
        const float *bs = next_buf(), *ec = ms + BLK * LP;
        if (PAIRED) {
            ms = ms == msg ? msg + MF : msg;
        } else {
            edge_costs(wn, ms + BLK * LP);
            wn = weights(b + 1);
            __syncwarp();
        }
        const int i0 = b * BLK, cnt = min(BLK, n - i0), gl = lane - (i0 & 31);
        if (b > 0) write_vec<P, VEC>(lbuf + so, lane, DP, L);
        so += ls;
        read_node(bs, i0, 0, nxt);
        read_edge(ec, 1, nxt);
        auto step = [&](int j, bool more, bool last) { // more: node j + 1 is in the block
            cur = nxt;
            if (more) {
                read_node(bs, i0, j + 1, nxt);
                read_edge(ec, j + 2, nxt);
            }
            vadd<P>(L, cur.un, v);
            const float g = last ? warp_min<P>(v, none) : minconv<P, DELTA>(v, cur.cw, ed, L);
            gb = gl == j ? g : gb;
        };
        if (b < nblk - 1) {
#pragma unroll
            for (int j = 0; j < BLK; ++j) step(j, j < BLK - 1, false);
        } else {
#pragma unroll 1
            for (int j = 0; j < cnt; ++j) step(j, j < cnt - 1, j == cnt - 1);
        }
        if (b == nblk - 1 || (i0 & 31) == 32 - BLK) {
            if (lane < (i0 & 31) + cnt) acc += (double)gb;
        }
    }
    if (!PAIRED) cp_wait<0>();

    // ---- backward: min-marginals, slack hand-over, reduced unary propagated back.
    // The chain minimum ((p0 + p1) + p2) + ... + p31 is added up meanwhile, two
    // partial sums per block: 31 dependent FP64 adds take about 3100 cycles
    cmin = __shfl_sync(0xffffffffu, acc, 0);
    int part = 1;
    auto add_part = [&]() {
        if (part < 32) cmin += __shfl_sync(0xffffffffu, acc, part);
        ++part;
    };
    __syncwarp();
    meet();
    const int Dst = a.store_phi ? DP : 0; // labels of phi to store
    if (!PAIRED) {
        for (int q = 0; q < NB - 1; ++q) issue(nblk - 1 - q);
        if (nblk > 1) load_vec<P, VEC>(lbuf + (nblk - 1) * ls, lane, DP, Lc);
        wn = weights(nblk - 1);
    }
    ms = msg;
    for (int b = nblk - 1; b >= 0; --b) {
        meet();
        if (!PAIRED) {
            arrived();
            issue(b - (NB - 1));
        }
        const float *bs = next_buf(), *ec = ms + BLK * LP;
        const int i0 = b * BLK, cnt = min(BLK, n - i0);
        add_part();
        add_part();
        if (!PAIRED) {
            edge_costs(wn, ms + BLK * LP);
            wn = weights(b - 1);
            __syncwarp();
            recompute(b, bs, ms);
        }
        auto read_back = [&](int j) {
            read_node(bs, i0, j, nxt);
            read_vec<P>(ms + j * LP, lane, nxt.vm);
            read_edge(ec, j, nxt);
        };
        read_back(cnt - 1);
        auto back = [&](int j, bool first, bool want) { // first: node 0 of the chain; want: labels
            cur = nxt;
            if (j > 0) read_back(j - 1);
            vadd<P>(cur.vm, R, m);
            const float mu = warp_min<P>(m, none);
            if (!HPASS && want) {
                int best = 0x7fffffff;
#pragma unroll
                for (int r = P - 1; r >= 0; --r)
                    if (m[r] == mu) best = lane * P + r;
                best = __reduce_min_sync(0xffffffffu, best);
                if (lane == 0) a.labels[(long)W * H * pair + (long)(i0 + j) * W + chain] = best;
            }
            float h[P], A[P];
            vsub1<P>(m, mu, h);
            vmul1<P>(h, a.rp.slack, h);
            vsub<P>(cur.un, h, A);
            if constexpr (HPASS) vadd<P>(cur.ph, h, cur.ph);
            write_vec<P, VEC>(phi + so, lane, Dst, HPASS ? cur.ph : A);
            so -= ns;
            if (!first) {
                vadd<P>(A, R, v);
                minconv<P, DELTA>(v, cur.cw, ed, R);
            }
        };
        so = (long)(i0 + cnt - 1) * ns;
        if (cnt == BLK && b > 0 && !a.labels) {
#pragma unroll
            for (int j = BLK - 1; j >= 0; --j) back(j, false, false);
        } else {
            const bool want = a.labels != nullptr;
#pragma unroll 1
            for (int j = cnt - 1; j >= 0; --j) back(j, i0 + j == 0, want);
        }
        if (PAIRED) ms = ms == msg ? msg + MF : msg;
    }
    if (!PAIRED) cp_wait<0>();
    while (part < 32) add_part();
    if (lane == 0) a.cmin[(long)nch * pair + chain] = cmin;
}

template <int P, int DELTA, bool HPASS, bool T16, int MODE, bool PAIRED>
int launch_form_as(const CrfPassArgs &a, const CrfForm &f, cudaStream_t st)
{
    const int wpb = PAIRED ? 1 : f.wpb;
    const size_t sm = sizeof(float) * wpb * (size_t)chain_floats(P, HPASS, T16, MODE, PAIRED, f.buffers);
    if (sm > SMEM_MAX) return fail(CNNCRF_EUNSUPPORTED, "crf: %zu bytes of ring per CTA", sm);
    auto kern = k_crf_chain<P, DELTA, HPASS, T16, MODE, PAIRED>;
    CNNCRF_CUDA(allow_smem(kern));
    const long chains = (long)(HPASS ? a.H : a.W) * a.np;
    {
        CNNCRF_PROF(HPASS ? "crf_h" : "crf_v", st);
        kern<<<ceil_div(chains, wpb), (PAIRED ? 64 : 32) * wpb, sm, st>>>(a, f.buffers);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

template <int P, int DELTA, bool HPASS, bool T16, int MODE>
int launch_mode(const CrfPassArgs &a, const CrfForm &f, cudaStream_t st)
{
    return f.paired ? launch_form_as<P, DELTA, HPASS, T16, MODE, true>(a, f, st)
                    : launch_form_as<P, DELTA, HPASS, T16, MODE, false>(a, f, st);
}

template <int P, int DELTA, bool HPASS, bool T16>
int launch_form(const CrfPassArgs &a, const CrfForm &f, cudaStream_t st)
{
    // whole 16-byte chunks where the vectors allow them (the solver's arrays start on 16 bytes: the workspace's by its
    // layout, a caller's cost volume by check_args)
    const int mode = vec_mode(a, HPASS);
    if (mode == ALIGNED) return launch_mode<P, DELTA, HPASS, T16, ALIGNED>(a, f, st);
    if constexpr (T16) return fail(CNNCRF_EINVAL, "crf: 16-bit unary at depth %d", a.D); // crf_reads_q16: never
    else {
        if constexpr (HPASS)
            if (mode == SPREAD) return launch_mode<P, DELTA, HPASS, T16, SPREAD>(a, f, st);
        return launch_mode<P, DELTA, HPASS, T16, RAGGED>(a, f, st);
    }
}

template <int P, int DELTA> int launch_dir(const CrfPassArgs &a, bool hpass, const CrfForm &f, cudaStream_t st)
{
    if (!hpass) return launch_form<P, DELTA, false, false>(a, f, st);
    // the H pass on the 16-bit unary where the labels fill the lanes with an even count (aligned copies)
    if constexpr (P % 2 == 0)
        if (a.thetaq && a.D == 32 * P) return launch_form<P, DELTA, true, true>(a, f, st);
    return launch_form<P, DELTA, true, false>(a, f, st);
}

template <int P> int launch_pass(const CrfPassArgs &a, bool hpass, int delta, const CrfForm &f, cudaStream_t st)
{
    if (f.wpb < 1 || f.wpb > 4) return fail(CNNCRF_EINVAL, "crf: %d chains per CTA outside 1..4", f.wpb);
    if (f.buffers < 2 || f.buffers > 3) return fail(CNNCRF_EINVAL, "crf: %d block buffers outside 2..3", f.buffers);
    // An offset whose rho reaches L2 never wins over the truncation: v_{k+-t} >= g, and adding the same w L2 rounds
    // monotonically, so v_{k+-t} + w rho_t >= g + w L2.  Those offsets are left out (the repository's truncated linear
    // term, L1 = 0.5, L2 = 1.5 at delta 3, computes two of its three), with the same bits
    if (delta < 1 || delta > 4) return fail(CNNCRF_EUNSUPPORTED, "crf: delta %d outside 1..4", delta);
    while (delta > 1 && a.rp.rho[delta] >= a.rp.L2) --delta;
    switch (delta) {
    case 1: return launch_dir<P, 1>(a, hpass, f, st);
    case 2: return launch_dir<P, 2>(a, hpass, f, st);
    case 3: return launch_dir<P, 3>(a, hpass, f, st);
    default: return launch_dir<P, 4>(a, hpass, f, st);
    }
}

} // namespace

} // namespace k
} // namespace cnncrf

#endif

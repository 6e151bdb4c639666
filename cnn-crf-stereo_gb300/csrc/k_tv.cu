// k_tv.cu -- the TV/Huber primal-dual refinement (the inner loop of
// cuda::fuseTHuberQuadFit, stereo/stereo.cu:1141-1166) as one fused kernel.
//
// The reference runs every iteration as three full-image passes: a copy
// u_ = u, ttvqf_primal_kernel (stereo/stereo.cu:701-729) and
// thuberqf_dual_kernel (stereo/stereo.cu:773-796).  Here one launch runs K
// iterations on a 64 x 32 pixel tile held on chip.  A warp has two rows, a
// lane two columns of them: each thread keeps its 2 x 2 pixels' u, the fit's
// per-pixel constants, the weights and p, q in registers.  The values
// neighbours read -- p.x - q.x, p.y - q.y (the primal's divergence) and u_
// (the dual's gradient) -- come from the thread itself, from the next lane by
// a shuffle per row, or from the next warp through shared memory, one row of
// each per warp.  The primal at (x, y) reads (x-1, y) and (x, y-1); the dual
// reads (x+1, y) and (x, y+1), so a tile's edge corrupts one more ring of
// pixels per iteration: the tile overlaps its neighbours by a halo of K pixels
// on every side and writes only its interior (64 - 2K) x (32 - 2K) block.
// Neighbour indices are clamped to the image exactly as the reference's
// clamp-addressed texture reads are (EDGE tiles; the others touch no image
// border), so tiles on the image border see the same values as the unfused
// kernels.
//
// Tiles read the state (u, p, q) of the previous launch and write a second
// copy (a workspace ping-pong), since a tile's halo belongs to other tiles.
// The per-element arithmetic is the reference kernels', operation for
// operation -- the fused multiply-adds their default compilation contracts
// are written out as __fmaf_rn, the rest is single IEEE operations -- and the
// per-pixel constants of the primal update are the same operations hoisted
// out of the iteration loop, so the results equal both the CPU oracle and the
// reference's own kernels bit for bit.  Compiled with --fmad=false.
//
// Bound by instruction issue: three IEEE divisions, two prox operators and
// the clamps per pixel and iteration, on 1.7 times the interior's pixels at K
// = 5.  Ten iterations on 4096 x 2160: 787 -> 521 us (a thread had four pixels
// eight rows apart, every neighbour through shared memory with clamped
// indices).  Larger tiles lose to their barriers what they save in halo: 64 x
// 64 539 us, 64 x 48 566 us.
#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

namespace {

constexpr int TX = 64, TY = 32, NT = 512; // a warp: 2 rows; a lane: 2 columns of them
// Iterations per launch: a launch of K costs about 22 K (64 32) / ((64 - 2K) (32 - 2K)) + 68 us on 4096 x 2160 (the halo's
// recomputation, the state's bytes), so 5 + 5 beat one launch of 8 or more and equal 4 + 3 + 3.  A field of at most a tile
// per SM hides the recomputation and saves launches: up to 8 iterations each (a whole call of 16 on 300 x 200: 63 -> 56 us
// on the device; 480 x 320, 200 tiles: 64 -> 70).
int iterations_per_launch(int W, int H) { return (long)ceil_div(W, TX - 16) * ceil_div(H, TY - 16) <= 152 ? 8 : 5; }

__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fmaxf(lo, fminf(v, hi)); }

// prox_p with alpha = 0 (stereo/stereo.cu:752-757): v itself where |v| <= 0 w, else the shrunk |v| with v's sign,
// clamped.  The first case is v = 0 alone (w infinite or NaN apart); with beta >= 0 a zero also shrinks to a zero, but it
// must not reach the clamp, which a negative w turns into |w| (4096 x 2160, ten iterations: 521 us with the test, 515
// without; a vote per tile on whether any weight is negative 523)
template <bool BETA_POS> __device__ __forceinline__ float prox_p0(float v, float beta, float sigma, float w)
{
    if (!BETA_POS && fabsf(v) <= __fmul_rn(w, 0.0f)) return v;
    const float m = fmaxf(0.0f, __fmaf_rn(-sigma, beta, fabsf(v)));
    const float r = BETA_POS ? copysignf(m, v) : __fmul_rn(m, v > 0.0f ? 1.0f : -1.0f);
    return BETA_POS && v == 0.0f ? v : clampf(r, -w, w);
}

// a + a - b for two values, each operation rounded by itself: a fused 2 a - b would not overflow where 2 a does
__device__ __forceinline__ void twice_less(const float (&a)[2], const float (&b)[2], float (&d)[2])
{
    asm("{\n\t.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, ra;\n\t"
        "sub.rn.f32x2 rd, rd, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d[0]), "=f"(d[1])
        : "f"(a[0]), "f"(a[1]), "f"(b[0]), "f"(b[1]));
}

struct TvArgs {
    const float *u_in;
    const float2 *p_in, *q_in; // null: p = q = 0
    const float *u0;
    const float2 *qf;
    const float *wx, *wy;
    float *u_out;
    float2 *p_out, *q_out;
    float *ubar_out; // the last iteration's u_ (null: not written)
    int W, H, K;
    float tau, sigma, half, C, eps;
};

// the K iterations of a tile whose first pixel is (ex, ey)
template <bool EDGE, bool BETA_POS>
__device__ __forceinline__ void tv_tile(const TvArgs &a, int ex, int ey, float2 (*sY)[TX / 2], float2 (*sU)[TX / 2])
{
    const int W = a.W, H = a.H, K = a.K;
    const int lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
    const int gx0 = ex + 2 * lane, gy0 = ey + 2 * wr;
    const int wm = wr > 0 ? wr - 1 : 0, wp = wr + 1 < TY / 2 ? wr + 1 : wr; // the warps above and below

    // per pixel (row i, column j): the state (u, u_, p, q) and the primal's per-pixel constants, computed once per
    // launch with the operations the reference applies per iteration: inner = a - b u0, den = 1 + tau b, the box
    // u0 -+ step / 2
    float u[2][2], ub[2][2], px[2][2], py[2][2], qx[2][2], qy[2][2];
    float inn[2][2], den[2][2], lo[2][2], hi[2][2], wx[2][2], wy[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int gx = gx0 + j, gy = gy0 + i;
            float uz = 0.0f, fa = 0.0f, fb = 0.0f;
            u[i][j] = wx[i][j] = wy[i][j] = px[i][j] = py[i][j] = qx[i][j] = qy[i][j] = ub[i][j] = 0.0f;
            if (!EDGE || (gx >= 0 && gx < W && gy >= 0 && gy < H)) {
                const long o = (long)gy * W + gx;
                u[i][j] = a.u_in[o];
                uz = a.u0[o];
                const float2 f = a.qf[o];
                fa = f.x, fb = f.y;
                wx[i][j] = a.wx[o], wy[i][j] = a.wy[o];
                if (a.p_in) {
                    const float2 pp = a.p_in[o], qq = a.q_in[o];
                    px[i][j] = pp.x, py[i][j] = pp.y, qx[i][j] = qq.x, qy[i][j] = qq.y;
                }
            }
            inn[i][j] = __fmaf_rn(-fb, uz, fa);
            den[i][j] = __fmaf_rn(a.tau, fb, 1.0f);
            lo[i][j] = __fsub_rn(uz, a.half);
            hi[i][j] = __fadd_rn(uz, a.half);
        }
    const float dd = __fmaf_rn(a.sigma, a.eps, 1.0f);
    // the row below this warp's reads its lower row's p.y - q.y
    auto put_y = [&]() { sY[wr][lane] = make_float2(__fsub_rn(py[1][0], qy[1][0]), __fsub_rn(py[1][1], qy[1][1])); };
    put_y();
    __syncthreads();

#pragma unroll 1
    for (int it = 0; it < K; ++it) {
        // ---- primal (ttvqf_primal_kernel); u_ = u at the iteration's start
        const float2 above = sY[wm][lane];
        float X[2][2], Y[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                X[i][j] = __fsub_rn(px[i][j], qx[i][j]), Y[i][j] = __fsub_rn(py[i][j], qy[i][j]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float left = __shfl_up_sync(0xffffffffu, X[i][1], 1);
            float u2[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float xl = j ? X[i][0] : left, yu = i ? Y[0][j] : (j ? above.y : above.x);
                if (EDGE) {
                    if (gx0 + j <= 0) xl = X[i][j];
                    if (gy0 + i <= 0) yu = Y[i][j];
                }
                const float div = __fsub_rn(__fadd_rn(__fsub_rn(X[i][j], xl), Y[i][j]), yu);
                float un = __fmaf_rn(a.tau, div, u[i][j]);
                const float num = __fmaf_rn(-a.tau, inn[i][j], un);
                un = clampf(__fdiv_rn(num, den[i][j]), lo[i][j], hi[i][j]);
                u2[j] = un;
            }
            twice_less(u2, u[i], ub[i]);
            u[i][0] = u2[0], u[i][1] = u2[1];
        }
        sU[wr][lane] = make_float2(ub[0][0], ub[0][1]); // the warp above reads this warp's upper row
        __syncthreads();
        // ---- dual (thuberqf_dual_kernel), Huber parameter eps
        const float2 below = sU[wp][lane];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float right = __shfl_down_sync(0xffffffffu, ub[i][0], 1);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float uc = ub[i][j];
                float ur = j ? right : ub[i][1], ud = i ? (j ? below.y : below.x) : ub[1][j];
                if (EDGE) {
                    if (gx0 + j >= W - 1) ur = uc;
                    if (gy0 + i >= H - 1) ud = uc;
                }
                const float dx = __fsub_rn(ur, uc), dy = __fsub_rn(ud, uc);
                const float pnx = __fmaf_rn(a.sigma, dx, px[i][j]), pny = __fmaf_rn(a.sigma, dy, py[i][j]);
                const float qnx = __fmaf_rn(a.sigma, dx, qx[i][j]), qny = __fmaf_rn(a.sigma, dy, qy[i][j]);
                px[i][j] = clampf(__fdiv_rn(pnx, dd), -wx[i][j], wx[i][j]);
                py[i][j] = clampf(__fdiv_rn(pny, dd), -wy[i][j], wy[i][j]);
                qx[i][j] = prox_p0<BETA_POS>(qnx, a.C, a.sigma, wx[i][j]);
                qy[i][j] = prox_p0<BETA_POS>(qny, a.C, a.sigma, wy[i][j]);
            }
        }
        put_y();         // this iteration's primals read sY before the barrier above
        __syncthreads(); // every dual has read sU before the next primal rewrites it
    }

    // ---- the interior block, inside the image
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int c = 2 * lane + j, r = 2 * wr + i, gx = gx0 + j, gy = gy0 + i;
            if (c < K || c >= TX - K || r < K || r >= TY - K) continue;
            if (EDGE && (gx < 0 || gx >= W || gy < 0 || gy >= H)) continue;
            const long o = (long)gy * W + gx;
            a.u_out[o] = u[i][j];
            a.p_out[o] = make_float2(px[i][j], py[i][j]);
            a.q_out[o] = make_float2(qx[i][j], qy[i][j]);
            if (a.ubar_out) a.ubar_out[o] = ub[i][j];
        }
}

template <bool BETA_POS> __global__ void __launch_bounds__(NT, 2) k_tv_fused(const TvArgs a)
{
    __shared__ float2 sY[TY / 2][TX / 2], sU[TY / 2][TX / 2];
    const int ex = blockIdx.x * (TX - 2 * a.K) - a.K, ey = blockIdx.y * (TY - 2 * a.K) - a.K;
    // pixels 0 and W - 1 (H - 1) are the only ones whose neighbours are clamped
    if (ex > 0 && ey > 0 && ex + TX < a.W && ey + TY < a.H) tv_tile<false, BETA_POS>(a, ex, ey, sY, sU);
    else tv_tile<true, BETA_POS>(a, ex, ey, sY, sU);
}

struct TvWs {
    size_t u, p, q, total;
};

TvWs tv_ws_layout(int W, int H)
{
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t n = (size_t)W * H;
    TvWs l;
    l.u = 0;
    l.p = al(n * sizeof(float));
    l.q = al(l.p + 2 * n * sizeof(float));
    l.total = al(l.q + 2 * n * sizeof(float));
    return l;
}

} // namespace

size_t tv_workspace_bytes(int W, int H) { return tv_ws_layout(W, H).total; }

// `iters` iterations from (u, p, q), or from (u, 0, 0) when pq_zero; the
// state ends in (u, p, q) and the last iteration's u_ in u_.  Launches of at
// most kmax iterations, alternating between the caller's state and the
// workspace so that the last launch writes the caller's buffers.
int tv_iterate(float *u, float *u_, const float *u0, const float *qf, float *p, float *q, const float *wx,
               const float *wy, int W, int H, float C, float eps, float step, int iters, void *ws,
               size_t ws_bytes, bool pq_zero, cudaStream_t st)
{
    if (W < 1 || H < 1) return fail(CNNCRF_EINVAL, "tv: bad size %dx%d", W, H);
    const size_t n = (size_t)W * H;
    if (iters <= 0) {
        if (pq_zero) {
            CNNCRF_CUDA(cudaMemsetAsync(p, 0, 2 * n * sizeof(float), st));
            CNNCRF_CUDA(cudaMemsetAsync(q, 0, 2 * n * sizeof(float), st));
        }
        return CNNCRF_OK;
    }
    const TvWs l = tv_ws_layout(W, H);
    if (!ws || ws_bytes < l.total) return fail(CNNCRF_EINVAL, "tv: workspace %zu < %zu bytes", ws_bytes, l.total);
    if (((uintptr_t)ws & 255) != 0) return fail(CNNCRF_EINVAL, "tv: workspace not 256-byte aligned");
    char *w = (char *)ws;
    float *wu = (float *)(w + l.u);
    float2 *wp = (float2 *)(w + l.p), *wq = (float2 *)(w + l.q);
    // launches of near-equal iteration counts, at most kmax each (the halo,
    // and so the recomputed fringe, grows with the count)
    const int kmax = iterations_per_launch(W, H);
    const int L = (iters + kmax - 1) / kmax;
    // state sets: 0 = the caller's buffers, 1 = the workspace; launch l
    // writes set (L-1-l) % 2, so the last one writes the caller's
    int in_set = (L % 2 == 1) ? 1 : 0;
    if (in_set == 1) { // the first launch writes the caller's set: read a copy
        CNNCRF_CUDA(cudaMemcpyAsync(wu, u, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
        if (!pq_zero) {
            CNNCRF_CUDA(cudaMemcpyAsync(wp, p, 2 * n * sizeof(float), cudaMemcpyDeviceToDevice, st));
            CNNCRF_CUDA(cudaMemcpyAsync(wq, q, 2 * n * sizeof(float), cudaMemcpyDeviceToDevice, st));
        }
    }
    const float Lc = (float)sqrt(8.0);
    TvArgs a{};
    a.u0 = u0, a.qf = (const float2 *)qf, a.wx = wx, a.wy = wy;
    a.W = W, a.H = H;
    a.tau = 1.0f / Lc, a.sigma = 1.0f / Lc, a.half = 0.5f * step, a.C = C, a.eps = eps;
    int done = 0;
    for (int li = 0; li < L; ++li) {
        const int K = (iters - done + (L - li) - 1) / (L - li);
        const int out_set = (L - 1 - li) % 2;
        a.K = K;
        a.u_in = in_set ? wu : u;
        a.p_in = (li == 0 && pq_zero) ? nullptr : (in_set ? wp : (const float2 *)p);
        a.q_in = (li == 0 && pq_zero) ? nullptr : (in_set ? wq : (const float2 *)q);
        a.u_out = out_set ? wu : u;
        a.p_out = out_set ? wp : (float2 *)p;
        a.q_out = out_set ? wq : (float2 *)q;
        a.ubar_out = li == L - 1 ? u_ : nullptr;
        const dim3 grid(ceil_div(W, TX - 2 * K), ceil_div(H, TY - 2 * K));
        {
            CNNCRF_PROF("tv", st);
            if (C >= 0.0f) k_tv_fused<true><<<grid, NT, 0, st>>>(a);
            else k_tv_fused<false><<<grid, NT, 0, st>>>(a);
        }
        CNNCRF_CHECK_LAUNCH();
        in_set = out_set;
        done += K;
    }
    return CNNCRF_OK;
}

} // namespace k
} // namespace cnncrf

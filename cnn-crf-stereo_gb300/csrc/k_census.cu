// k_census.cu -- the non-CNN parts of the Stereo pipeline: grey images,
// census matching cost, image-gradient edge weights, the QuadDirect
// refinement and the left-right consistency check.
//
// Reference kernels: rgb_to_gray_kernel (stereo/stereo.cu:853-863),
// cost_vol_census_kernel (stereo/stereo.cu:306-346), calcEdgeImage =
// Gaussian(0.7) + filter_{x,y}_forward_kernel (stereo/stereo.cu:471-520,
// 1090-1095), do_fitting_kernel_volume + do_argmin_kernel_volume
// (stereo/stereo.cu:913-942, 1172-1194), leftrightcheck_kernel
// (stereo/stereo.cu:803-817).  The reference reads its images through CUDA
// textures; here every read is explicit index arithmetic:
//   clamp-addressed point reads at integer positions (the reference's texel
//   centres), and at fractional positions a linear interpolation in FP32
//   (t[i] + a * (t[i+1] - t[i]), a = position - floor(position)) where the
//   reference's texture unit interpolates with 8-bit weights.
// Compiled with --fmad=false: every result equals the CPU oracle bit for bit.
#include <algorithm>
#include <cmath>

#include "../../include/cnncrf_fmath.h"
#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

namespace {

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// linear read of row r at unnormalised texture coordinate u (texel centres at
// i + 0.5), clamp addressing
__device__ __forceinline__ float lerp_row(const float *__restrict__ r, int W, float u)
{
    const float t = __fsub_rn(u, 0.5f);
    const float f = floorf(t);
    const int i = (int)f;
    const float a = __fsub_rn(t, f);
    const float v0 = r[clampi(i, 0, W - 1)];
    if (a == 0.0f) return v0;
    const float v1 = r[clampi(i + 1, 0, W - 1)];
    return __fadd_rn(v0, __fmul_rn(a, __fsub_rn(v1, v0)));
}

__global__ void k_gray(const float *__restrict__ rgba, long n, float *__restrict__ gray)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float *px = rgba + 4 * i;
    gray[i] = (float)(0.2989 * (double)px[0] + 0.5870 * (double)px[1] + 0.1140 * (double)px[2]);
}

// any disparities: one thread per pixel, all of them; list[z] = the z-th disparity
__global__ void k_census(const float *__restrict__ g1, const float *__restrict__ g2, int W, int H, int fs,
                         const float *__restrict__ list, int D, float lambda, float *__restrict__ vol)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    const float norm = (float)(fs * fs * 4);
    const float c1 = g1[(long)y * W + x];
    const float xx = __fadd_rn((float)x, 0.5f);
    for (int z = 0; z < D; ++z) {
        const float d = list[z];
        const float c2 = lerp_row(g2 + (long)y * W, W, __fsub_rn(xx, d));
        float cnt = 0.0f;
        for (int dy = -fs; dy <= fs; ++dy) {
            const int yy = clampi(y + dy, 0, H - 1);
            const float *r1 = g1 + (long)yy * W, *r2 = g2 + (long)yy * W;
            for (int dx = -fs; dx <= fs; ++dx) {
                if (dx == 0 && dy == 0) continue;
                const float i1 = r1[clampi(x + dx, 0, W - 1)];
                const float i2 = lerp_row(r2, W, __fsub_rn(__fadd_rn((float)(x + dx), 0.5f), d));
                if ((c1 > i1) != (c2 > i2)) cnt = __fadd_rn(cnt, 1.0f);
            }
        }
        vol[((long)y * W + x) * D + z] = __fmul_rn(lambda, __fdiv_rn(cnt, norm));
    }
}

// The same volume for integer disparities, where every read is a texel: the
// other image's reads depend on x - d alone, so each pixel's comparisons are
// one bit string, computed once, and a cost is the bits in which the two
// strings differ.  A CTA takes CPX pixels of a row: the window rows of both
// images in shared memory, a bit string per left pixel and per right column
// x - d any label reaches (words [word][column]), then a warp per pixel with
// the labels across the lanes, 7 words compared and counted per label at
// filter size 7, and the (window^2 - 1)-entry table of lambda count / norm.
// k_census compared all 225 positions per pixel and label, each with its own
// two interpolation coordinates: 12.4 ms for 720 x 480 at 128 labels; this
// takes 211 us.  Bound by issue (89 % of the cycles; 223 M warp instructions);
// the population counts alone (16 per SM and cycle) are 67 us, the volume's
// bytes 26.
// NW: words per string, 0 for any.
constexpr int CPX = 64, CTH = 256;

template <int NW>
__global__ void __launch_bounds__(CTH)
    k_census_bits(const float *__restrict__ g1, const float *__restrict__ g2, int W, int H, int fs,
                  const float *__restrict__ list, int D, int dmin, int dmax, float lambda, float *__restrict__ vol)
{
    extern __shared__ float4 sm4[];
    const int side = 2 * fs + 1, bits = side * side - 1, nw = NW ? NW : (bits + 31) / 32;
    const int cols = CPX + dmax - dmin, tw1 = CPX + 2 * fs, tw2 = cols + 2 * fs;
    float *t1 = (float *)sm4, *t2 = t1 + side * tw1;                   // window rows of the two images
    uint32_t *b1 = (uint32_t *)(t2 + side * tw2), *b2 = b1 + nw * CPX; // [nw][CPX], [nw][cols]
    float *lut = (float *)(b2 + nw * cols);                            // [bits + 1]
    int *sd = (int *)(lut + bits + 1);                                 // [D]
    const int x0 = blockIdx.x * CPX, y = blockIdx.y, tid = threadIdx.x;
    const int xr = x0 - dmax; // the right column of b2[.][0]
    for (int i = tid; i < side * tw1; i += CTH) {
        const int r = i / tw1, c = i - r * tw1;
        t1[i] = __ldg(g1 + (long)clampi(y + r - fs, 0, H - 1) * W + clampi(x0 - fs + c, 0, W - 1));
    }
    for (int i = tid; i < side * tw2; i += CTH) {
        const int r = i / tw2, c = i - r * tw2;
        t2[i] = __ldg(g2 + (long)clampi(y + r - fs, 0, H - 1) * W + clampi(xr - fs + c, 0, W - 1));
    }
    const float norm = (float)(fs * fs * 4);
    for (int i = tid; i <= bits; i += CTH) lut[i] = __fmul_rn(lambda, __fdiv_rn((float)i, norm));
    for (int i = tid; i < D; i += CTH) sd[i] = (int)list[i];
    __syncthreads();
    for (int j = tid; j < CPX + cols; j += CTH) {
        const bool left = j < CPX;
        const int c = left ? j : j - CPX, tw = left ? tw1 : tw2, pitch = left ? CPX : cols;
        const float *t = (left ? t1 : t2) + c;
        uint32_t *b = (left ? b1 : b2) + c;
        const float centre = t[fs * tw + fs];
        uint32_t word = 0;
        int n = 0;
        for (int dy = 0; dy < side; ++dy, t += tw)
            for (int dx = 0; dx < side; ++dx) {
                if (dy == fs && dx == fs) continue;
                word = 2 * word + (centre > t[dx] ? 1u : 0u);
                if ((++n & 31) == 0) *b = word, b += pitch, word = 0;
            }
        if (n & 31) *b = word;
    }
    __syncthreads();
    const int lane = tid & 31;
    for (int px = tid >> 5; px < CPX && x0 + px < W; px += CTH / 32) {
        uint32_t w1[NW ? NW : 1];
        if (NW)
#pragma unroll
            for (int w = 0; w < NW; ++w) w1[w] = b1[w * CPX + px];
        float *o = vol + ((long)y * W + x0 + px) * D;
        for (int z = lane; z < D; z += 32) {
            const uint32_t *b = b2 + px + dmax - sd[z]; // right column x - d
            int cnt = 0;
            if (NW) {
#pragma unroll
                for (int w = 0; w < NW; ++w) cnt += __popc(w1[w] ^ b[w * cols]);
            } else {
                for (int w = 0; w < nw; ++w) cnt += __popc(b1[w * CPX + px] ^ b[w * cols]);
            }
            o[z] = lut[cnt];
        }
    }
}

size_t census_bits_smem(int fs, int D, int range)
{
    const size_t side = 2 * fs + 1, bits = side * side - 1, nw = (bits + 31) / 32, cols = CPX + range;
    return 4 * (side * (CPX + cols + 4 * fs) + nw * (CPX + cols) + bits + 1 + D);
}

// Whether the bit strings are the cheaper way.  A CTA's 64 pixels take 2 CPX + range strings of side^2 comparisons however
// few the labels are, k_census D times side^2 comparisons per pixel (720 x 480 at filter size 7: 112 us plus 0.5 us per
// column of range against 16 us plus 96 us per label; three labels 1000 columns apart 2514 against 303 us, four labels in a
// row at filter size 1 40 against 28 us).  The line, from filter sizes 1 to 16, 1 to 16 labels and ranges up to 8000, lies
// where no list is slower than in k_census; strings cost 1.3 and 2 times as much with two and one CTAs per SM
bool bits_pay(int fs, int D, int range, size_t smem)
{
    const double sq = (2 * fs + 1) * (2 * fs + 1);
    const size_t ctas = 228 * 1024 / (smem + 1024);
    const double strings = (2 * CPX + range) * (ctas >= 3 ? 1.0 : (ctas == 2 ? 1.3 : 2.0));
    return strings * (sq + 2) + 8000 < 140 * sq * D;
}

// separable Gaussian, radius R, clamp-to-edge; horizontal then vertical pass
__global__ void k_gauss_h(const float *__restrict__ in, int W, int H, const float *__restrict__ w, int R,
                          float *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    const float *r = in + (long)y * W;
    float s = 0.0f;
    for (int i = -R; i <= R; ++i) s = __fmaf_rn(w[i + R], r[clampi(x + i, 0, W - 1)], s);
    out[(long)y * W + x] = s;
}

__global__ void k_gauss_v(const float *__restrict__ in, int W, int H, const float *__restrict__ w, int R,
                          float *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    float s = 0.0f;
    for (int i = -R; i <= R; ++i) s = __fmaf_rn(w[i + R], in[(long)clampi(y + i, 0, H - 1) * W + x], s);
    out[(long)y * W + x] = s;
}

__device__ __forceinline__ float edge_weight(float diff, float alpha, float beta, float lambda)
{
    if (alpha > 0.0f)
        return fmaxf(__fmul_rn(lambda, cnncrf_expf(__fmul_rn(-alpha, cnncrf_powf(diff, beta)))), 1.0e-6f);
    return __fmul_rn(lambda, diff);
}

// forward differences of the smoothed image (the last column / row mirrors
// onto itself: difference 0)
__global__ void k_edges(const float *__restrict__ t, int W, int H, float alpha, float beta, float lambda,
                        float *__restrict__ wx, float *__restrict__ wy)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    const long i = (long)y * W + x;
    const float c = t[i];
    const float dxv = fabsf(__fsub_rn(t[(long)y * W + min(x + 1, W - 1)], c));
    const float dyv = fabsf(__fsub_rn(t[(long)min(y + 1, H - 1) * W + x], c));
    wx[i] = edge_weight(dxv, alpha, beta, lambda);
    wy[i] = edge_weight(dyv, alpha, beta, lambda);
}

// parabola through the three costs c (of labels z - 1, z, z + 1) around the solution's label z
__device__ __forceinline__ float quadfit(float u, float cm, float c, float cp, float dstep)
{
    const float a = __fdiv_rn(__fsub_rn(cm, cp), __fmul_rn(dstep, 2.0f));
    const float b = fmaxf(1.0e-3f, __fdiv_rn(__fsub_rn(__fadd_rn(cm, cp), __fmul_rn(2.0f, c)), __fmul_rn(dstep, dstep)));
    return __fadd_rn(u, __fdiv_rn(a, b));
}

__global__ void k_quadfit_direct(float *__restrict__ u, const float *__restrict__ c1, long npx, int D, float dmin,
                                 float dstep)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npx) return;
    const int z = (int)__fdiv_rn(__fsub_rn(u[i], dmin), dstep);
    if (z <= 0 || z >= D - 1) return; // no neighbour on one side: unchanged
    const float *c = c1 + i * D;
    u[i] = quadfit(u[i], c[z - 1], c[z], c[z + 1], dstep);
}

// The same on the solver's own arrays: its C1 is theta - phi, of which a pixel reads three values; writing out all D of
// them first took 139 us of a 720 x 480 pair at 128 labels, this kernel takes about as long as the fit on a given C1 (16 us).
__global__ void k_quadfit_solver(float *__restrict__ u, const float *__restrict__ cost, const uint16_t *__restrict__ costq,
                                 float qs, float qo, const float *__restrict__ phi, int DP, long npx, int D, float dmin,
                                 float dstep)
{
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npx) return;
    const int z = (int)__fdiv_rn(__fsub_rn(u[i], dmin), dstep);
    if (z <= 0 || z >= D - 1) return;
    auto c = [&](int k) {
        const long o = i * D + k;
        return __fsub_rn(costq ? __fmaf_rn((float)costq[o], qs, qo) : cost[o], phi[i * DP + k]);
    };
    u[i] = quadfit(u[i], c(z - 1), c(z), c(z + 1), dstep);
}

__global__ void k_lr_check(const float *__restrict__ left, const float *__restrict__ right, int W, int H, float th,
                           float *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W) return;
    const long i = (long)y * W + x;
    const float d = left[i];
    const float dr = -lerp_row(right + (long)y * W, W, __fsub_rn(__fadd_rn((float)x, 0.5f), d));
    out[i] = fabsf(__fsub_rn(d, dr)) <= th ? d : -1.0f;
}

} // namespace

int rgb_to_gray(const float *rgba, long n, float *gray, cudaStream_t st)
{
    {
        CNNCRF_PROF("gray", st);
        k_gray<<<ceil_div(n, 256), 256, 0, st>>>(rgba, n, gray);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int census_volume(const float *g1, const float *g2, int W, int H, int fs, const float *d_list, const float *h_list, int D,
                  float lambda, float *vol, cudaStream_t st)
{
    if (fs < 1 || fs > 16) return fail(CNNCRF_EINVAL, "census: filter size %d outside 1..16", fs);
    // k_census_bits: integer disparities whose coordinates x + dx + 0.5 - d are exact, tiles that fit, and lists dense enough
    bool whole = true;
    float lo = h_list[0], hi = h_list[0];
    for (int i = 0; i < D; ++i) {
        whole = whole && h_list[i] == std::floor(h_list[i]) && std::fabs(h_list[i]) < 1048576.0f;
        lo = std::min(lo, h_list[i]), hi = std::max(hi, h_list[i]);
    }
    if (whole && W < 1048576 && hi - lo < 8192.0f) {
        const size_t sm = census_bits_smem(fs, D, (int)(hi - lo));
        if (sm <= SMEM_MAX && bits_pay(fs, D, (int)(hi - lo), sm)) {
            const int side = 2 * fs + 1, nw = (side * side - 1 + 31) / 32;
            auto kern = nw == 1   ? k_census_bits<1>
                        : nw == 2 ? k_census_bits<2>
                        : nw == 3 ? k_census_bits<3>
                        : nw == 4 ? k_census_bits<4>
                        : nw == 6 ? k_census_bits<6>
                        : nw == 7 ? k_census_bits<7>
                                  : k_census_bits<0>;
            CNNCRF_CUDA(allow_smem(kern));
            {
                CNNCRF_PROF("census_bits", st);
                kern<<<dim3(ceil_div(W, CPX), H), CTH, sm, st>>>(g1, g2, W, H, fs, d_list, D, (int)lo, (int)hi, lambda, vol);
            }
            CNNCRF_CHECK_LAUNCH();
            return CNNCRF_OK;
        }
    }
    {
        CNNCRF_PROF("census", st);
        k_census<<<dim3(ceil_div(W, 128), H), 128, 0, st>>>(g1, g2, W, H, fs, d_list, D, lambda, vol);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

void gauss_weights(float sigma, int R, float *w)
{
    // exp(-i^2 / (2 sigma^2)) / sum, in double, rounded once (host; the CPU
    // oracle computes the same floats the same way)
    double s = 0.0, v[64];
    for (int i = -R; i <= R; ++i) s += (v[i + R] = std::exp(-(double)(i * i) / (2.0 * sigma * sigma)));
    for (int i = 0; i <= 2 * R; ++i) w[i] = (float)(v[i] / s);
}

int edge_weights(const float *gray, int W, int H, float alpha, float beta, float lambda, float *tmp, float *tmp2,
                 const float *d_gw, float *wx, float *wy, cudaStream_t st)
{
    const dim3 g(ceil_div(W, 128), H);
    {
        CNNCRF_PROF("gauss", st);
        k_gauss_h<<<g, 128, 0, st>>>(gray, W, H, d_gw, GAUSS_R, tmp);
        k_gauss_v<<<g, 128, 0, st>>>(tmp, W, H, d_gw, GAUSS_R, tmp2);
    }
    {
        CNNCRF_PROF("edges", st);
        k_edges<<<g, 128, 0, st>>>(tmp2, W, H, alpha, beta, lambda, wx, wy);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int quadfit_direct(float *u, const float *c1, long npx, int D, float dmin, float dstep, cudaStream_t st)
{
    {
        CNNCRF_PROF("quadfit", st);
        k_quadfit_direct<<<ceil_div(npx, 256), 256, 0, st>>>(u, c1, npx, D, dmin, dstep);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int quadfit_solver(float *u, const float *cost, const void *costq, UnaryQ16 q, const float *phi, int DP, long npx, int D, float dmin,
                   float dstep, cudaStream_t st)
{
    {
        CNNCRF_PROF("quadfit", st);
        k_quadfit_solver<<<ceil_div(npx, 256), 256, 0, st>>>(u, cost, (const uint16_t *)costq, q.scale, q.offset, phi, DP, npx, D,
                                                             dmin, dstep);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

int lr_check(const float *left, const float *right, int W, int H, float th, float *out, cudaStream_t st)
{
    {
        CNNCRF_PROF("lr_check", st);
        k_lr_check<<<dim3(ceil_div(W, 128), H), 128, 0, st>>>(left, right, W, H, th, out);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

} // namespace k
} // namespace cnncrf

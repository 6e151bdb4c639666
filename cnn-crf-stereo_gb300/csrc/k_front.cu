// k_front.cu -- mirror padding and RGB normalisation (the front end of
// ColorStereoNet::predict).  Compiled with --fmad=false: results must match
// the CPU oracle bit for bit.
#include <algorithm>

#include "common.h"
#include "kernels.h"

namespace cnncrf {
namespace k {

namespace {

// cudaAddressModeMirror at texel centres (stereo/stereo.cu:879-911): symmetric
// reflection, edge sample repeated, period 2n.
__device__ __forceinline__ int mirror_idx(int i, int n)
{
    int m = i % (2 * n);
    if (m < 0) m += 2 * n;
    return m >= n ? 2 * n - 1 - m : m;
}

__global__ void k_pad(const float4 *__restrict__ in, int W, int H, int p, float4 *__restrict__ out)
{
    int Wp = W + 2 * p, Hp = H + 2 * p;
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long)Wp * Hp) return;
    in += (long)blockIdx.y * W * H; // image of the batch
    out += (long)blockIdx.y * Wp * Hp;
    int y = (int)(i / Wp), x = (int)(i - (long)y * Wp);
    out[i] = in[(long)mirror_idx(y - p, H) * W + mirror_idx(x - p, W)];
}

// plane c of a pixel: RGB channel, or rgb_to_gray_kernel's weights
// (stereo/stereo.cu:853-863) evaluated in double and rounded once.
template <bool GRAY> __device__ __forceinline__ float plane_val(const float4 &px, int c)
{
    if (GRAY) return (float)(0.2989 * (double)px.x + 0.5870 * (double)px.y + 0.1140 * (double)px.z);
    return c == 0 ? px.x : (c == 1 ? px.y : px.z);
}

// a caller's image may start on any float
template <bool AL> __device__ __forceinline__ float4 load_px(const float4 *p)
{
    if (AL) return __ldg(p);
    const float *f = (const float *)p;
    return make_float4(__ldg(f), __ldg(f + 1), __ldg(f + 2), 0.0f);
}

// image i of the batch: the first n from a, the others from b
__device__ __forceinline__ const float4 *image(const float4 *a, const float4 *b, int n, int i, long npx)
{
    return i < n ? a + i * npx : b + (i - n) * npx;
}

// FP64 sums in a fixed order shared with the CPU oracle: lane j of a warp sums
// the elements j, j+32, j+64, ... in ascending order, then the 32 partial sums
// are combined by an xor butterfly (offsets 16, 8, 4, 2, 1).
__device__ __forceinline__ double warp_tree_sum(double s)
{
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = s + __shfl_xor_sync(0xffffffffu, s, off);
    return s;
}

// The statistic of one plane from its row sums, added by one warp in the same
// lane / butterfly order; every lane has it.  Each consumer's CTAs take it
// from the row sums themselves: a launch between them cost 8 us
__device__ __forceinline__ double plane_sum(const double *rows, int Hp, int lane)
{
    double s = 0.0;
#pragma unroll 8
    for (int y = lane; y < Hp; y += 32) s += rows[y];
    return warp_tree_sum(s);
}

// One warp per (row, plane), a few rows per CTA.  pass 0 sums the values,
// pass 1 the squares of (v - mean_c) rounded to float.  rows: [image][pass][3]
// [Hp].  Bound by the FP64 additions (conversions by integer operations took the
// same time); the warps are small and many, their loads eight pixels ahead.
// Both sides of a KITTI pair in three launches take 72 us, in the ten launches
// of one side at a time with the statistics in launches of their own 107 us.
// TALL: more rows than ROW_CTAS CTAs per image (5 per SM) take once.  Each CTA of the second pass adds up all rows' sums for
// the mean, which with a CTA per two rows grew with the square of the height: both passes of a 48 x 12000 pair 959 -> 203 us.
// The others keep their kernel without the row loop (a KITTI pair 44 us, 49 with it).
template <bool GRAY> __host__ __device__ constexpr int row_cta() { return GRAY ? 4 : 2; }
constexpr int ROW_CTAS = 760;
template <bool GRAY, bool AL, bool TALL>
__global__ void __launch_bounds__(32 * row_cta<GRAY>() * (GRAY ? 1 : 3))
    k_rowsums(const float4 *__restrict__ ia, const float4 *__restrict__ ib, int n, int Wp, int Hp, int pass,
              double *__restrict__ rowsum)
{
    constexpr int NP = GRAY ? 1 : 3;
    __shared__ float smean[NP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = warp / NP, c = warp - r * NP;
    double *rows = rowsum + (long)blockIdx.y * 6 * Hp;
    float mean = 0.0f;
    if (pass) {
        if (warp < NP) {
            const double s = plane_sum(rows + warp * Hp, Hp, lane);
            if (lane == 0) smean[warp] = (float)(s / (double)((long)Wp * Hp));
        }
        __syncthreads();
        mean = smean[c];
        rows += 3 * Hp;
    }
    const float4 *im = image(ia, ib, n, blockIdx.y, (long)Wp * Hp);
    for (int y = blockIdx.x * row_cta<GRAY>() + r; y < Hp; y += gridDim.x * row_cta<GRAY>()) {
        const float4 *px = im + (long)y * Wp;
        double s = 0.0;
#pragma unroll 8
        for (int x = lane; x < Wp; x += 32) {
            float v = plane_val<GRAY>(load_px<AL>(px + x), c);
            if (pass) v = __fsub_rn(v, mean), v = __fmul_rn(v, v);
            s += (double)v;
        }
        s = warp_tree_sum(s);
        if (lane == 0) rows[c * Hp + y] = s;
        if (!TALL) return;
    }
}

// (v - mean) / population std, and the coordinate planes.  A CTA takes the
// statistics once, so the grid is a few CTAs per SM however large the images.
template <bool GRAY, bool AL>
__global__ void __launch_bounds__(256)
    k_norm_write(const float4 *__restrict__ ia, const float4 *__restrict__ ib, int n, int Wp, int Hp, int ic,
                 const double *__restrict__ rowsum, float *__restrict__ out)
{
    constexpr int NP = GRAY ? 1 : 3;
    __shared__ float stats[2][3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long npx = (long)Wp * Hp;
    const double *rows = rowsum + (long)blockIdx.y * 6 * Hp;
    if (warp < 2 * NP) {
        const int k = warp / NP, c = warp - k * NP;
        const double s = plane_sum(rows + (3 * k + c) * Hp, Hp, lane) / (double)npx;
        if (lane == 0) stats[k][c] = (float)(k ? sqrt(s) : s);
    }
    __syncthreads();
    const float4 *px = image(ia, ib, n, blockIdx.y, npx);
    out += (long)blockIdx.y * npx * ic;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < npx; i += (long)gridDim.x * blockDim.x) {
        const float4 p = load_px<AL>(px + i);
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            const float v = __fsub_rn(plane_val<GRAY>(p, c), stats[0][c]), sd = stats[1][c];
            out[i * ic + c] = sd > 0.0f ? __fdiv_rn(v, sd) : 0.0f;
        }
        if (ic == 5) { // stereo/colorstereonet.cpp:102-121
            const int y = (int)(i / Wp), x = (int)(i - (long)y * Wp);
            out[i * ic + 3] = (float)(((double)x - (double)Wp / 2.0) / (double)Wp);
            out[i * ic + 4] = (float)(((double)y - (double)Hp / 2.0) / (double)Hp);
        }
    }
}

template <bool GRAY, bool AL>
int launch_normalize(const float4 *a, const float4 *b, int n, int nimg, int Wp, int Hp, int ic, float *out, double *rows,
                     cudaStream_t st)
{
    const long npx = (long)Wp * Hp;
    for (int pass = 0; pass < 2; ++pass) {
        CNNCRF_PROF("rowsums", st);
        const int ctas = std::min(ceil_div(Hp, row_cta<GRAY>()), ROW_CTAS);
        const auto kern = ctas * row_cta<GRAY>() < Hp ? k_rowsums<GRAY, AL, true> : k_rowsums<GRAY, AL, false>;
        kern<<<dim3(ctas, nimg), 32 * row_cta<GRAY>() * (GRAY ? 1 : 3), 0, st>>>(a, b, n, Wp, Hp, pass, rows);
    }
    {
        CNNCRF_PROF("norm_write", st);
        const long ctas = std::min<long>(ceil_div(npx, 256), std::max(8, ceil_div(608, nimg))); // 4 per SM
        k_norm_write<GRAY, AL><<<dim3((unsigned)ctas, nimg), 256, 0, st>>>(a, b, n, Wp, Hp, ic, rows, out);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

} // namespace

int pad_rgba(const float *in, int W, int H, int p, float *out, cudaStream_t st, int nimg)
{
    long n = (long)(W + 2 * p) * (H + 2 * p);
    {
        CNNCRF_PROF("pad", st);
        k_pad<<<dim3(ceil_div(n, 256), nimg), 256, 0, st>>>((const float4 *)in, W, H, p, (float4 *)out);
    }
    CNNCRF_CHECK_LAUNCH();
    return CNNCRF_OK;
}

size_t normalize_scratch_bytes(int Hp, int nimg) { return sizeof(double) * 6 * (size_t)Hp * nimg; }

int normalize(const float *rgba, const float *rgba2, int Wp, int Hp, int ic, float *out, void *scratch, cudaStream_t st,
              int nimg)
{
    const float4 *a = (const float4 *)rgba, *b = (const float4 *)rgba2;
    const int total = rgba2 ? 2 * nimg : nimg;
    const bool al = (((uintptr_t)rgba | (uintptr_t)rgba2) & 15) == 0;
    auto *launch = ic == 1 ? (al ? launch_normalize<true, true> : launch_normalize<true, false>)
                           : (al ? launch_normalize<false, true> : launch_normalize<false, false>);
    return launch(a, b, nimg, total, Wp, Hp, ic, out, (double *)scratch, st);
}

} // namespace k
} // namespace cnncrf

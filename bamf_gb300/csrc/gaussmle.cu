/*
 * gaussmle.cu - single-emitter maximum-likelihood fits of (x, y, N, bg)
 * (gaussMLE 'Basic'/'CCD': kernel_MLEFit_XYNB_, cuda_gaussMLEv2.cu:16-141,
 * with GPUgaussLib.cuh:14-258 and MatInvLib.h:15-75) for sm_103a.
 *
 * A group of 8 lanes per fit (one thread per fit in the reference).  The model
 * is separable (gaussmle_axis.cuh): the integrated PSF and its derivatives are
 * evaluated once per pixel edge and axis and Newton iteration, and the start-up
 * filter is two passes of one-dimensional sums (O(sz^3) instead of O(sz^4)).
 * Output layout as the reference: param-major P[Nfits*k + i], k = 0..3 for
 * (x along the contiguous axis, y, N, bg), CRLB likewise, LogLikelihood[i].
 */
#include <cuda_runtime.h>

#include "bamf.h"
#include "frontend_launch.h"
#include "gaussmle_axis.cuh"
#include "smem_limit.h"

namespace {

constexpr int MAXSZ = GAUSS_MLE_MAX_SIZE; /* IMSZBIG of definitions.h: largest fit window */
constexpr int GROUP_FITS_PER_BLOCK = 16;  /* 128 threads */

/* A CTA's shared memory in floats: the staged ROIs, per fit the filter's first
 * pass and the edge and axis rows, then the filter's tables and pixel p -> (ii,
 * jj) as ii << 8 | jj (no division in the pixel loops).  Axis rows first: they
 * are read 16 bytes at a time. */
constexpr int AXIS_FLOATS = 2 * 4 * MAXSZ + 2 * 2 * (MAXSZ + 2);
__host__ __device__ constexpr int mle_smem_floats(int sz)
{
    return GROUP_FITS_PER_BLOCK * (AXIS_FLOATS + 2 * sz * sz) + 3 * MAXSZ + sz * sz;
}

/* The nblk (<= GROUP_FITS_PER_BLOCK) fits from ROI `first` of `data`, by
 * the whole CTA; parameter k of fit i to P[stride * k + i] and CRLB alike,
 * the log-likelihood to LL[i].  Every thread returns here.  Lane l of a group owns pixels l, l + GL, ...:
 * the Newton sums and the Fisher information are lane partial sums; the sums
 * of an iteration are scattered over the group (group_sum_pairs), so that each
 * parameter's quotient and update run once, on its own two lanes.  SZ > 0 fixes
 * sz: the pixels' values and offsets then stay in registers.
 *
 * Issue-bound.  79,787 fits of 7x7, 10 iterations: 256 us with both edges
 * of every index evaluated, the two-dimensional filter and all four updates on
 * every lane, 143 us with these, 125 us with the quick reciprocal. */
template <int SZ>
__device__ __forceinline__ void mle_xynb_block(const float *__restrict__ data, float sigma, int sz_, int iterations,
                                               float *__restrict__ P, float *__restrict__ CRLB,
                                               float *__restrict__ LL, int64_t stride, int64_t first, int nblk)
{
    extern __shared__ __align__(16) float sm[];
    const int sz = SZ > 0 ? SZ : sz_, npx = sz * sz;
    float *rois = sm + GROUP_FITS_PER_BLOCK * AXIS_FLOATS;
    float *tmps = rois + GROUP_FITS_PER_BLOCK * npx;
    float *w = tmps + GROUP_FITS_PER_BLOCK * npx, *norm = w + 2 * MAXSZ;
    int *pix = (int *)(norm + MAXSZ);
    for (int i = threadIdx.x; i < nblk * npx; i += blockDim.x) rois[i] = data[first * npx + i];
    for (int q = threadIdx.x; q < npx; q += blockDim.x) pix[q] = (q / sz) << 8 | (q % sz);
    filter_tables(w, norm, sz, sigma);
    __syncthreads();
    const int g = threadIdx.x / GL, l = threadIdx.x % GL;
    /* a group past the batch's end fits the block's first ROI again (its
     * lanes take part in the warp's shuffles) and writes nothing */
    const bool active = g < nblk;
    const float *d = rois + (active ? g : 0) * npx;
    float4 *xr = (float4 *)(sm + g * AXIS_FLOATS), *yr = xr + MAXSZ; /* {PSF, d1, d2, 0} per index */
    float2 *xe = (float2 *)(yr + MAXSZ), *ye = xe + MAXSZ + 2;
    const int64_t fit = first + g;
    float theta[4];
    {
        float nmax, bg;
        start_values<SZ>(d, tmps + g * npx, w, norm, pix, sz, l, &theta[0], &theta[1], &nmax, &bg);
        theta[3] = bg;
        theta[2] = fmaxf(0.0f, (nmax - bg) * 2 * 2 * MLE_PI * sigma * sigma);
    }
    const float inv_s = 1.0f / sigma, erf_s = sqrtf(1.0f / 2.0f / sigma / sigma);
    const float k1 = -1.0f / sqrtf(2.0f * MLE_PI) / sigma, k2 = -1.0f / sqrtf(2.0f * MLE_PI) / (sigma * sigma * sigma);
    /* this lane's pixels: value, and (ii, jj) */
    constexpr int NP = SZ > 0 ? (SZ * SZ + GL - 1) / GL : 1;
    float dv[NP];
    int at[NP];
#pragma unroll
    for (int t = 0; t < (SZ > 0 ? NP : 0); ++t) {
        const int p = min(l + GL * t, npx - 1);
        at[t] = pix[p];
        dv[t] = d[sz * (at[t] & 255) + (at[t] >> 8)];
    }

    for (int kk = 0; kk <= iterations; kk++) {
        /* the axis terms of theta (after the last iteration: for the Fisher
         * information) */
        axis_edges(xe, sz, theta[0], inv_s, erf_s, l);
        axis_edges(ye, sz, theta[1], inv_s, erf_s, l);
        __syncwarp();
        const float n1 = k1 * theta[2], n2 = k2 * theta[2];
        for (int q = l; q < sz; q += GL) {
            const float2 x0 = xe[q], x1 = xe[q + 1], y0 = ye[q], y1 = ye[q + 1];
            const float ux = (float)q - theta[0], uy = (float)q - theta[1];
            xr[q] = make_float4(0.5f * (x1.x - x0.x), n1 * (x1.y - x0.y), n2 * ((ux + 1.0f) * x1.y - ux * x0.y), 0.0f);
            yr[q] = make_float4(0.5f * (y1.x - y0.x), n1 * (y1.y - y0.y), n2 * ((uy + 1.0f) * y1.y - uy * y0.y), 0.0f);
        }
        __syncwarp();
        if (kk == iterations) break;
        float num[4] = {0.0f, 0.0f, 0.0f, 0.0f}, den[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        auto pixel = [&](int ij, float data_v) {
            const float4 ax = xr[ij >> 8], ay = yr[ij & 255];
            const float psf = ax.x * ay.x, model = theta[3] + theta[2] * psf;
            const float u0 = ax.y * ay.x, u1 = ay.y * ax.x;
            float cf = 0.0f, df = 0.0f;
            if (model > 10e-3f) {
                /* data/model, data/model^2 as products (beyond 1e37, as at infinity, both
                 * vanish against the rest) */
                const float r = recip(fminf(model, 1e37f));
                cf = data_v * r - 1;
                df = data_v * r * r;
            }
            cf = fminf(cf, 10e4f);
            df = fminf(df, 10e4f);
            num[0] += u0 * cf;
            num[1] += u1 * cf;
            num[2] += psf * cf;
            num[3] += cf;
            den[0] = fmaf(ax.z * ay.x, cf, fmaf(-(u0 * u0), df, den[0]));
            den[1] = fmaf(ay.z * ax.x, cf, fmaf(-(u1 * u1), df, den[1]));
            den[2] = fmaf(-(psf * psf), df, den[2]);
            den[3] -= df;
        };
        if (SZ > 0) {
#pragma unroll
            for (int t = 0; t < NP; ++t)
                if (l + GL * t < npx) pixel(at[t], dv[t]);
        } else {
            for (int p = l; p < npx; p += GL) pixel(pix[p], d[sz * (pix[p] & 255) + (pix[p] >> 8)]);
        }
        group_sum_pairs(num, den, l);
        /* parameter k = l >> 1: steps bounded by 1 (positions) or by its value */
        const int k = l >> 1;
        const float th = k == 0 ? theta[0] : k == 1 ? theta[1] : k == 2 ? theta[2] : theta[3];
        const float jump = k < 2 ? 1.0f : th;
        float nt = th - fminf(fmaxf(num[0] / den[0], -jump), jump);
        if (k == 2) nt = fmaxf(nt, 1.0f);
        if (k == 3) nt = fmaxf(nt, 0.01f);
#pragma unroll
        for (int q = 0; q < 4; ++q) theta[q] = __shfl_sync(0xffffffffu, nt, 2 * q, GL);
    }

    /* Fisher information (10 distinct entries) and log-likelihood
     * (cuda_gaussMLEv2.cu:104-130) */
    float F[10] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float Div = 0.0f;
    auto fisher = [&](int ij, float data_v) {
        const float4 ax = xr[ij >> 8], ay = yr[ij & 255];
        const float psf = ax.x * ay.x, model = theta[3] + theta[2] * psf;
        const float dudt[4] = {ax.y * ay.x, ay.y * ax.x, psf, 1.0f};
        const float rm = model > 10e-3f && model < 1e37f ? recip(model) : 1.0f / model;
        int e = 0;
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = a; b < 4; b++) F[e++] += dudt[b] * dudt[a] * rm;
        if (model > 0) {
            if (data_v > 0)
                Div += data_v * logf(model) - model - data_v * logf(data_v) + data_v;
            else
                Div += -model;
        }
    };
    if (SZ > 0) {
#pragma unroll 1
        for (int p = l; p < npx; p += GL) fisher(pix[p], d[sz * (pix[p] & 255) + (pix[p] >> 8)]);
    } else {
        for (int p = l; p < npx; p += GL) fisher(pix[p], d[sz * (pix[p] & 255) + (pix[p] >> 8)]);
    }
    for (int e = 0; e < 10; ++e) F[e] = group_sum(F[e]);
    Div = group_sum(Div);
    const float crlb = inverse_diagonal<4>(F, l);
    if (!active) return;
    if (l < 4) {
        P[stride * l + fit] = l == 0 ? theta[0] : l == 1 ? theta[1] : l == 2 ? theta[2] : theta[3];
        CRLB[stride * l + fit] = crlb;
    }
    if (l == 0) LL[fit] = Div;
}

template <int SZ>
__global__ void __launch_bounds__(GL * GROUP_FITS_PER_BLOCK) mle_xynb_group_kernel(
    const float *__restrict__ data, float sigma, int sz, int iterations,
    float *__restrict__ P, float *__restrict__ CRLB, float *__restrict__ LL, int nfits)
{
    const int64_t first = (int64_t)blockIdx.x * GROUP_FITS_PER_BLOCK;
    mle_xynb_block<SZ>(data, sigma, sz, iterations, P, CRLB, LL, nfits, first,
                   (int)min((int64_t)GROUP_FITS_PER_BLOCK, (int64_t)nfits - first));
}

/* The fits of ROIs [range[0], min(range[1], capacity)) of a stack whose
 * range is known only on the device: blocks of GROUP_FITS_PER_BLOCK fits,
 * grid-stride. */
template <int SZ>
__global__ void __launch_bounds__(GL * GROUP_FITS_PER_BLOCK) mle_xynb_range_kernel(
    const float *__restrict__ data, float sigma, int sz, int iterations, float *__restrict__ P,
    float *__restrict__ CRLB, float *__restrict__ LL, int64_t stride, const int64_t *__restrict__ range,
    int64_t capacity)
{
    const int64_t f0 = range[0], f1 = min(range[1], capacity);
    for (int64_t first = f0 + (int64_t)blockIdx.x * GROUP_FITS_PER_BLOCK; first < f1;
         first += (int64_t)gridDim.x * GROUP_FITS_PER_BLOCK) {
        mle_xynb_block<SZ>(data, sigma, sz, iterations, P, CRLB, LL, stride, first,
                           (int)min((int64_t)GROUP_FITS_PER_BLOCK, f1 - first));
        __syncthreads(); /* the staged ROIs and axis rows are rewritten for the next fits */
    }
}

}  // namespace

/* dynamic shared memory of a launch; above 48 KB (sz > 15) it is asked for */
template <typename Kern>
static bool gauss_mle_smem(Kern kern, int sz, size_t *bytes)
{
    *bytes = (size_t)mle_smem_floats(sz) * sizeof(float);
    return *bytes <= 48 * 1024 || allow_smem(kern, mle_smem_floats(MAXSZ) * sizeof(float)) == cudaSuccess;
}

bamf_status launch_gauss_mle_range(const float *rois, int sz, float psf_sigma, int iterations, float *params,
                                   float *crlb, float *loglik, int64_t stride, const int64_t *range,
                                   int64_t capacity, int blocks, cudaStream_t stream)
{
    if (sz < 1 || sz > MAXSZ || iterations < 0 || blocks < 1) return BAMF_ERR_INVALID_ARG;
    /* 7 and 8 px are findROI's and findPriors' boxes, so nearly every fit: with the
     * size known 80k fits take 125 and 164 us, without 168 and 221 */
    const auto kern = sz == 7 ? mle_xynb_range_kernel<7> : sz == 8 ? mle_xynb_range_kernel<8> : mle_xynb_range_kernel<0>;
    size_t smem;
    if (!gauss_mle_smem(kern, sz, &smem)) {
        cudaGetLastError();
        return BAMF_ERR_CUDA;
    }
    kern<<<blocks, GL * GROUP_FITS_PER_BLOCK, smem, stream>>>(
        rois, psf_sigma, sz, iterations, params, crlb, loglik, stride, range, capacity);
    return cudaGetLastError() == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

extern "C" bamf_status bamf_gauss_mle_device(const float *rois, int sz, int nfits, float psf_sigma,
                                             int iterations, float *params, float *crlb,
                                             float *loglik, void *stream)
{
    if (!rois || !params || !crlb || !loglik || sz < 1 || nfits < 0 || iterations < 0)
        return BAMF_ERR_INVALID_ARG;
    if (sz > MAXSZ) return BAMF_ERR_TOO_LARGE;
    if (nfits == 0) return BAMF_OK;
    /* a group of GL lanes per fit: 16 fits per CTA of 128 threads */
    const auto kern = sz == 7 ? mle_xynb_group_kernel<7> : sz == 8 ? mle_xynb_group_kernel<8> : mle_xynb_group_kernel<0>;
    size_t smem;
    if (!gauss_mle_smem(kern, sz, &smem)) {
        cudaGetLastError();
        return BAMF_ERR_CUDA;
    }
    int blocks = (nfits + GROUP_FITS_PER_BLOCK - 1) / GROUP_FITS_PER_BLOCK;
    kern<<<blocks, GL * GROUP_FITS_PER_BLOCK, smem, (cudaStream_t)stream>>>(
        rois, psf_sigma, sz, iterations, params, crlb, loglik, nfits);
    return cudaGetLastError() == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

extern "C" bamf_status bamf_gauss_mle_host(const float *rois, int sz, int nfits, float psf_sigma,
                                           int iterations, float *params, float *crlb,
                                           float *loglik)
{
    if (!rois || !params || !crlb || !loglik || sz < 1 || nfits < 0 || iterations < 0)
        return BAMF_ERR_INVALID_ARG;
    if (sz > MAXSZ) return BAMF_ERR_TOO_LARGE;
    if (nfits == 0) return BAMF_OK;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    float *dr = nullptr, *dp = nullptr, *dc = nullptr, *dl = nullptr;
    size_t nin = (size_t)nfits * sz * sz, nout = (size_t)nfits * 4;
    bamf_status st = BAMF_OK;
    if (cudaMalloc(&dr, nin * sizeof(float)) != cudaSuccess || cudaMalloc(&dp, nout * sizeof(float)) != cudaSuccess ||
        cudaMalloc(&dc, nout * sizeof(float)) != cudaSuccess || cudaMalloc(&dl, nfits * sizeof(float)) != cudaSuccess)
        st = BAMF_ERR_CUDA;
    if (!st && cudaMemcpy(dr, rois, nin * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) st = BAMF_ERR_CUDA;
    if (!st) st = bamf_gauss_mle_device(dr, sz, nfits, psf_sigma, iterations, dp, dc, dl, nullptr);
    if (!st && cudaDeviceSynchronize() != cudaSuccess) st = BAMF_ERR_CUDA;
    if (!st && (cudaMemcpy(params, dp, nout * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(crlb, dc, nout * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(loglik, dl, nfits * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess))
        st = BAMF_ERR_CUDA;
    cudaFree(dr);
    cudaFree(dp);
    cudaFree(dc);
    cudaFree(dl);
    return st;
}

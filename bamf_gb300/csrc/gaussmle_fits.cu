/*
 * gaussmle_fits.cu - the other gaussMLE fit types (@RJ/gaussMLE.m FitType
 * 'Sigma', 'Z', 'SigmaYX', and CameraType 'SCMOS' for all four types) with
 * the reference kernels' Newton-Raphson updates, constraints, Fisher
 * information and log-likelihood (cuda_gaussMLEv2.cu:144-1125 with
 * GPUgaussLib.cuh:14-258 and MatInvLib.h:15-75).  CCD 'Basic' has its own
 * optimised kernel (gaussmle.cu).
 *
 * One group of 8 lanes per fit (four fits per warp), the block's ROIs staged
 * through shared memory; lane l of a group evaluates pixels l, l + 8, ....  As in
 * the Basic kernel the model's axis terms, the start filter and the sums are
 * those of gaussmle_axis.cuh.  Issue-bound: 20,000 Sigma fits of 8x8, 20
 * iterations, took 389 us with every pixel evaluating both axes' functions at
 * both edges (4 erf, 8 exp, some 20 divisions), 148 us with the axis rows.
 *
 * Parameters theta: 0 = position along the contiguous ROI axis (MATLAB rows:
 * Results.Y), 1 = the other axis (Results.X), 2 = photons, 3 = background, then
 *   Sigma:   4 = sigma of a symmetric PSF
 *   Z:       4 = z of an astigmatic PSF, sigma_a = sigma_a0 sqrt(alpha_a(z)),
 *            alpha_a(z) = 1 + (z'/d)^2 + A_a (z'/d)^3 + B_a (z'/d)^4 with
 *            z' = z - gamma along axis 0 and z + gamma along axis 1
 *   SigmaYX: 4, 5 = sigma along axis 0 and axis 1
 * sCMOS: every pixel's variance-to-gain ratio g (from a square map, at the
 * ROI's box corner) enters as cf = (data - model)/(model + g),
 * df = (data + g)/(model + g)^2.  The reference's CRLB / log-likelihood pass
 * does not re-read g per pixel: it uses the value left from the last pixel
 * of the last Newton iteration, (sz-1, sz-1), and so does this code (0 when
 * there are no iterations, where the reference reads an uninitialised
 * value).
 */
#include <cuda_runtime.h>

#include <algorithm>

#include "bamf.h"
#include "gaussmle_axis.cuh"
#include "smem_limit.h"

namespace {

constexpr int MAXSZ = 21;
constexpr int FITS_PER_BLOCK = 16; /* fits per CTA, 8 lanes each */

struct ZPar {
    float sx, sy, Ax, Ay, Bx, By, gamma, d;
};

/* kernel_alpha and its z-derivatives (:25-57) */
__device__ __forceinline__ float alpha_z(float z, float A, float B, float d)
{
    float t = z / d;
    return 1.0f + t * t + A * t * t * t + B * t * t * t * t;
}
__device__ __forceinline__ float dalpha_z(float z, float A, float B, float d)
{
    return 2.0f * z / (d * d) + 3.0f * A * z * z / (d * d * d) + 4.0f * B * z * z * z / (d * d * d * d);
}
__device__ __forceinline__ float d2alpha_z(float z, float A, float B, float d)
{
    return 2.0f / (d * d) + 6.0f * A * z / (d * d * d) + 12.0f * B * z * z / (d * d * d * d);
}

/* axis_rows: the terms of every index along one axis: the PSF; the first and
 * second derivative by the position (kernel_DerivativeIntGauss1D,
 * GPUgaussLib.cuh:67-87) and by the width (kernel_DerivativeIntGauss1DSigma,
 * :90-110), up to the other axis's PSF. */
/* shared memory of a fit in floats: two axes of {PSF, d1, d2, s1} rows, the edges,
 * the s2 rows */
constexpr int AXIS_FLOATS = 2 * 4 * MAXSZ + 2 * 2 * (MAXSZ + 2) + 2 * (MAXSZ + 1);
static_assert(AXIS_FLOATS % 4 == 0, "16-byte rows");

__device__ __forceinline__ void axis_rows(float4 *row, float *row2, float2 *edge, int sz, float c, float S, float N,
                                          bool width, int l)
{
    axis_edges(edge, sz, c, 1.0f / S, sqrtf(1.0f / 2.0f / S / S), l);
    __syncwarp();
    const float k = N / sqrtf(2.0f * MLE_PI) / S; /* N / sqrt(2 pi) / S */
    const float k2 = k / S, k3 = k2 / S, k5 = k3 / S / S, m2 = 2.0f / S;
    for (int q = l; q < sz; q += GL) {
        const float2 e0 = edge[q], e1 = edge[q + 1];
        const float v = (float)q - c, u = v + 1.0f;
        const float au = u * e1.y, bv = v * e0.y, g = -k2 * (au - bv);
        row[q] = make_float4(0.5f * (e1.x - e0.x), -k * (e1.y - e0.y), -k3 * (au - bv), g);
        if (width) row2[q] = -m2 * g - k5 * (au * u * u - bv * v * v);
    }
}

template <int FIT, bool SCMOS>
__global__ void __launch_bounds__(GL * FITS_PER_BLOCK) mle_fit_kernel(
    const float *__restrict__ data, float sigma, ZPar zp, const float *__restrict__ coords,
    const float *__restrict__ gmap, int mapsz, int sz, int iterations, float *__restrict__ P,
    float *__restrict__ CRLB, float *__restrict__ LL, int nfits)
{
    constexpr int NV = FIT == BAMF_FIT_BASIC ? 4 : (FIT == BAMF_FIT_SIGMAYX ? 6 : 5);
    constexpr bool WIDTH = FIT != BAMF_FIT_BASIC;
    extern __shared__ __align__(16) float sm[];
    const int npx = sz * sz;
    const int64_t first = (int64_t)blockIdx.x * FITS_PER_BLOCK;
    const int nblk = (int)min((int64_t)FITS_PER_BLOCK, (int64_t)nfits - first);
    /* per fit the axis rows, then the staged ROIs, the filter's first pass, its
     * tables, and pixel -> (ii, jj) (ii << 8 | jj) */
    float *rois = sm + FITS_PER_BLOCK * AXIS_FLOATS, *tmps = rois + FITS_PER_BLOCK * npx;
    float *w = tmps + FITS_PER_BLOCK * npx, *norm = w + 2 * MAXSZ;
    int *pix = (int *)(norm + MAXSZ);
    for (int i = threadIdx.x; i < nblk * npx; i += blockDim.x) rois[i] = data[first * npx + i];
    for (int q = threadIdx.x; q < npx; q += blockDim.x) pix[q] = (q / sz) << 8 | (q % sz);
    filter_tables(w, norm, sz, FIT == BAMF_FIT_Z ? zp.sx : sigma);
    __syncthreads();
    const int g = threadIdx.x / GL, l = threadIdx.x % GL;
    /* a group past the batch's end fits the block's first ROI again (its
     * lanes take part in the warp's shuffles) and writes nothing */
    const bool active = g < nblk;
    const float *d = rois + (active ? g : 0) * npx;
    float4 *xr = (float4 *)(sm + g * AXIS_FLOATS), *yr = xr + MAXSZ;
    float2 *xe = (float2 *)(yr + MAXSZ), *ye = xe + MAXSZ + 2;
    float *x2 = (float *)(ye + MAXSZ + 2), *y2 = x2 + MAXSZ + 1;
    const int64_t fit = first + (active ? g : 0);
    float c0 = 0.0f, c1 = 0.0f;
    if (SCMOS) {
        c0 = coords[2 * fit];
        c1 = coords[2 * fit + 1];
    }

    float th[6];
    {
        float nmax, bg;
        start_values<0>(d, tmps + g * npx, w, norm, pix, sz, l, &th[0], &th[1], &nmax, &bg);
        th[3] = bg;
        if (FIT == BAMF_FIT_Z) {
            th[2] = fmaxf(0.0f, (nmax - bg) * 2 * MLE_PI * zp.sx * zp.sy * sqrtf(2.0f));
            th[4] = 0.0f; /* z0: gaussMLE.m passes zeros */
        } else {
            th[2] = fmaxf(0.0f, (nmax - bg) * 2 * 2 * MLE_PI * sigma * sigma);
            th[4] = sigma;
        }
        th[5] = sigma;
    }

    /* Z (kernel_DerivativeIntGauss2Dz, :135-205): the widths of both axes and
     * their first two derivatives by z */
    float zx1 = 0.0f, zx2 = 0.0f, zy1 = 0.0f, zy2 = 0.0f;
    auto axes = [&]() {
        float sx = FIT == BAMF_FIT_BASIC ? sigma : th[4], sy = FIT == BAMF_FIT_SIGMAYX ? th[5] : sx;
        if (FIT == BAMF_FIT_Z) {
            const float zz = th[4], zm = zz - zp.gamma, zpl = zz + zp.gamma;
            const float ax = alpha_z(zm, zp.Ax, zp.Bx, zp.d), ay = alpha_z(zpl, zp.Ay, zp.By, zp.d);
            const float rx = sqrtf(ax), ry = sqrtf(ay);
            const float dax = dalpha_z(zm, zp.Ax, zp.Bx, zp.d), day = dalpha_z(zpl, zp.Ay, zp.By, zp.d);
            sx = zp.sx * rx;
            sy = zp.sy * ry;
            const float px = zp.sx / 2.0f / rx, py = zp.sy / 2.0f / ry;
            zx1 = px * dax;
            zy1 = py * day;
            zx2 = -zp.sx / 4.0f / (ax * rx) * dax * dax + px * d2alpha_z(zm, zp.Ax, zp.Bx, zp.d);
            zy2 = -zp.sy / 4.0f / (ay * ry) * day * day + py * d2alpha_z(zpl, zp.Ay, zp.By, zp.d);
        }
        axis_rows(xr, x2, xe, sz, th[0], sx, th[2], WIDTH, l);
        axis_rows(yr, y2, ye, sz, th[1], sy, th[2], WIDTH, l);
        __syncwarp();
    };
    /* derivatives of the model at a pixel; d2u null: first ones only */
    auto pixel = [&](int ii, int jj, float *psf, float *du, float *d2u) {
        const float4 ax = xr[ii], ay = yr[jj];
        *psf = ax.x * ay.x;
        du[0] = ax.y * ay.x;
        du[1] = ay.y * ax.x;
        du[2] = *psf;
        du[3] = 1.0f;
        const float sx1 = ax.w * ay.x, sy1 = ay.w * ax.x;
        if (FIT == BAMF_FIT_SIGMA) du[4] = sx1 + sy1;
        if (FIT == BAMF_FIT_SIGMAYX) {
            du[4] = sx1;
            du[5] = sy1;
        }
        if (FIT == BAMF_FIT_Z) du[4] = sx1 * zx1 + sy1 * zy1;
        if (d2u) {
            d2u[0] = ax.z * ay.x;
            d2u[1] = ay.z * ax.x;
            d2u[2] = 0.0f;
            d2u[3] = 0.0f;
            if (WIDTH) {
                const float sx2 = x2[ii] * ay.x, sy2 = y2[jj] * ax.x;
                if (FIT == BAMF_FIT_SIGMA) d2u[4] = sx2 + sy2;
                if (FIT == BAMF_FIT_SIGMAYX) {
                    d2u[4] = sx2;
                    d2u[5] = sy2;
                }
                if (FIT == BAMF_FIT_Z) d2u[4] = sx2 * (zx1 * zx1) + sx1 * zx2 + sy2 * (zy1 * zy1) + sy1 * zy2;
            }
        }
    };

    for (int kk = 0; kk < iterations; kk++) {
        axes();
        float num[6] = {0, 0, 0, 0, 0, 0}, den[6] = {0, 0, 0, 0, 0, 0};
        for (int p = l; p < npx; p += GL) {
            const int ii = pix[p] >> 8, jj = pix[p] & 255;
            float psf, du[6], d2u[6];
            pixel(ii, jj, &psf, du, d2u);
            float model = th[3] + th[2] * psf;
            float dv = d[sz * jj + ii];
            float cf = 0.0f, df = 0.0f;
            if (SCMOS) {
                int gi = (int)((c1 + jj) * mapsz + c0 + ii);
                gi = min(max(gi, 0), mapsz * mapsz - 1); /* corners outside the map: edge value */
                const float gRp = gmap[gi];
                if (model > 10e-3f) {
                    cf = (dv - model) / (model + gRp);
                    df = (dv + gRp) / ((model + gRp) * (model + gRp));
                }
            } else if (model > 10e-3f) {
                const float r = recip(fminf(model, 1e37f));
                cf = dv * r - 1;
                df = dv * r * r;
            }
            cf = fminf(cf, 10e4f);
            df = fminf(df, 10e4f);
#pragma unroll
            for (int q = 0; q < NV; q++) {
                num[q] += du[q] * cf;
                den[q] = fmaf(d2u[q], cf, fmaf(-(du[q] * du[q]), df, den[q]));
            }
        }
        /* parameters 0..3 on lane pairs, 4 and 5 on every lane */
#pragma unroll
        for (int q = 4; q < NV; q++) {
            num[q] = group_sum(num[q]);
            den[q] = group_sum(den[q]);
        }
        {
            float n4[4] = {num[0], num[1], num[2], num[3]}, d4[4] = {den[0], den[1], den[2], den[3]};
            group_sum_pairs(n4, d4, l);
            const int k = l >> 1;
            const float t = k == 0 ? th[0] : k == 1 ? th[1] : k == 2 ? th[2] : th[3];
            const float jump = k < 2 ? 1.0f : t;
            float nt = t - fminf(fmaxf(n4[0] / d4[0], -jump), jump);
            if (k == 2) nt = fmaxf(nt, 1.0f);
            if (k == 3) nt = fmaxf(nt, 0.01f);
#pragma unroll
            for (int q = 0; q < 4; ++q) th[q] = __shfl_sync(0xffffffffu, nt, 2 * q, GL);
        }
        if (FIT == BAMF_FIT_SIGMA || FIT == BAMF_FIT_SIGMAYX) {
            th[4] -= fminf(fmaxf(num[4] / den[4], -th[4]), th[4]);
            th[4] = fmaxf(th[4], 0.5f);
            th[4] = fminf(th[4], sz / 2.0f);
        }
        if (FIT == BAMF_FIT_SIGMAYX) {
            th[5] -= fminf(fmaxf(num[5] / den[5], -th[5]), th[5]);
            th[5] = fmaxf(th[5], 0.5f);
            th[5] = fminf(th[5], sz / 2.0f);
        }
        if (FIT == BAMF_FIT_Z) th[4] -= fminf(fmaxf(num[4] / den[4], -1e-1f), 1e-1f);
        __syncwarp(); /* every lane has read the axis rows before they change */
    }
    /* the reference's CRLB / log-likelihood pass uses the variance-gain
     * ratio left from the last pixel of the last iteration, (sz-1, sz-1) */
    float gR = 0.0f;
    if (SCMOS && iterations > 0) {
        int gi = (int)((c1 + (sz - 1)) * mapsz + c0 + (sz - 1));
        gR = gmap[min(max(gi, 0), mapsz * mapsz - 1)];
    }

    /* Fisher information (distinct entries, lane partial sums) and
     * log-likelihood */
    constexpr int NF = NV * (NV + 1) / 2;
    float F[NF];
#pragma unroll
    for (int q = 0; q < NF; ++q) F[q] = 0.0f;
    float Div = 0.0f;
    axes();
    for (int p = l; p < npx; p += GL) {
        const int ii = pix[p] >> 8, jj = pix[p] & 255;
        float psf, du[6];
        pixel(ii, jj, &psf, du, nullptr);
        float model = th[3] + th[2] * psf;
        float dv = d[sz * jj + ii];
        const float rd = 1.0f / (SCMOS ? model + gR : model);
        int e = 0;
#pragma unroll
        for (int a = 0; a < NV; a++)
#pragma unroll
            for (int b = a; b < NV; b++) F[e++] += du[b] * du[a] * rd;
        if (SCMOS) {
            if (model + gR > 0) {
                if (dv + gR > 0)
                    Div += (dv + gR) * logf(model + gR) - model - (dv + gR) * logf(dv + gR) + dv;
                else
                    Div += -model - gR;
            }
        } else if (model > 0) {
            if (dv > 0)
                Div += dv * logf(model) - model - dv * logf(dv) + dv;
            else
                Div += -model;
        }
    }
#pragma unroll
    for (int q = 0; q < NF; ++q) F[q] = group_sum(F[q]);
    Div = group_sum(Div);
    const float crlb = inverse_diagonal<NV>(F, l);
    if (!active) return;
    float t = th[0];
#pragma unroll
    for (int k = 1; k < NV; k++)
        if (l == k) t = th[k];
    if (l < NV) {
        P[(int64_t)nfits * l + fit] = t;
        CRLB[(int64_t)nfits * l + fit] = crlb;
    }
    if (l == 0) LL[fit] = Div;
}

constexpr size_t fit_smem(int sz)
{
    return ((size_t)FITS_PER_BLOCK * (AXIS_FLOATS + 2 * sz * sz) + 3 * MAXSZ + (size_t)sz * sz) * sizeof(float);
}

template <int FIT, bool SCMOS>
cudaError_t launch(const float *rois, int sz, int nfits, float sigma, const ZPar &zp, const float *coords,
                   const float *gmap, int mapsz, int iterations, float *P, float *C, float *L, cudaStream_t s)
{
    const size_t smem = fit_smem(sz);
    if (smem > 48 * 1024) {
        const cudaError_t e = allow_smem(mle_fit_kernel<FIT, SCMOS>, fit_smem(MAXSZ));
        if (e != cudaSuccess) return e;
    }
    int blocks = (nfits + FITS_PER_BLOCK - 1) / FITS_PER_BLOCK;
    mle_fit_kernel<FIT, SCMOS><<<blocks, GL * FITS_PER_BLOCK, smem, s>>>(rois, sigma, zp, coords, gmap, mapsz, sz,
                                                                         iterations, P, C, L, nfits);
    return cudaGetLastError();
}

}  // namespace

extern "C" int bamf_gauss_mle_nparams(int fit_type)
{
    switch (fit_type) {
    case BAMF_FIT_BASIC: return 4;
    case BAMF_FIT_SIGMA: return 5;
    case BAMF_FIT_Z: return 5;
    case BAMF_FIT_SIGMAYX: return 6;
    default: return -1;
    }
}

extern "C" bamf_status bamf_gauss_mle_fit_device(const float *rois, int sz, int nfits, int fit_type, float psf_sigma,
                                                 const bamf_zfit *zfit, const float *box_corners,
                                                 const float *var_gain_map, int map_size, int iterations,
                                                 float *params, float *crlb, float *loglik, void *stream)
{
    if (!rois || !params || !crlb || !loglik || sz < 1 || nfits < 0 || iterations < 0) return BAMF_ERR_INVALID_ARG;
    if (bamf_gauss_mle_nparams(fit_type) < 0) return BAMF_ERR_INVALID_ARG;
    if (fit_type == BAMF_FIT_Z && !zfit) return BAMF_ERR_INVALID_ARG;
    const bool scmos = var_gain_map != nullptr;
    if (scmos && (!box_corners || map_size < 1)) return BAMF_ERR_INVALID_ARG;
    if (sz > MAXSZ) return BAMF_ERR_TOO_LARGE;
    if (nfits == 0) return BAMF_OK;
    if (!scmos && fit_type == BAMF_FIT_BASIC)
        return bamf_gauss_mle_device(rois, sz, nfits, psf_sigma, iterations, params, crlb, loglik, stream);
    ZPar zp = {0, 0, 0, 0, 0, 0, 0, 1};
    if (zfit) zp = {zfit->sigma_x, zfit->sigma_y, zfit->Ax, zfit->Ay, zfit->Bx, zfit->By, zfit->gamma, zfit->d};
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
#define BAMF_FIT_CASE(F)                                                                                          \
    e = scmos ? launch<F, true>(rois, sz, nfits, psf_sigma, zp, box_corners, var_gain_map, map_size, iterations,  \
                                params, crlb, loglik, s)                                                          \
              : launch<F, false>(rois, sz, nfits, psf_sigma, zp, nullptr, nullptr, 0, iterations, params, crlb,   \
                                 loglik, s)
    switch (fit_type) {
    case BAMF_FIT_BASIC: BAMF_FIT_CASE(BAMF_FIT_BASIC); break;
    case BAMF_FIT_SIGMA: BAMF_FIT_CASE(BAMF_FIT_SIGMA); break;
    case BAMF_FIT_Z: BAMF_FIT_CASE(BAMF_FIT_Z); break;
    default: BAMF_FIT_CASE(BAMF_FIT_SIGMAYX); break;
    }
#undef BAMF_FIT_CASE
    return e == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

namespace {

/* fits' ROIs out of planes: in[(a * sz + b) * n + fit] (a numpy array (sz, sz, n)) to
 * out[fit * sz * sz + sz * b + a], 32 fits per CTA in tiles of 32 pixels through
 * shared memory.  Bound by its bytes (each read and written
 * once).  20,000 ROIs of 8x8: numpy's reordering on the host took 1330 of the
 * call's 2110 us; with this and one allocation the call takes 509 us. */
__global__ void __launch_bounds__(256) planes_kernel(const float *__restrict__ in, int sz, int n,
                                                     float *__restrict__ out)
{
    __shared__ float t[32][33];
    const int npx = sz * sz, x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int64_t first = (int64_t)blockIdx.x * 32;
    for (int q0 = 0; q0 < npx; q0 += 32) {
        for (int q = y; q < 32; q += 8)
            if (q0 + q < npx && first + x < n)
                t[q][x] = in[(int64_t)((q0 + q) % sz * sz + (q0 + q) / sz) * n + first + x];
        __syncthreads();
        for (int f = y; f < 32; f += 8)
            if (q0 + x < npx && first + f < n) out[(first + f) * npx + q0 + x] = t[x][f];
        __syncthreads();
    }
}

/* The planes go to the device at most so many bytes at a time (fits, in steps
 * of planes_kernel's 32), so that a stack takes no more device memory than one
 * that needs no reordering, but for these. */
constexpr size_t PLANES_BYTES = (size_t)256 << 20;

bamf_status fit_host(const float *rois, bool planes, int sz, int nfits, int fit_type, float psf_sigma,
                     const bamf_zfit *zfit, const float *box_corners, const float *var_gain_map, int map_size,
                     int iterations, float *params, float *crlb, float *loglik)
{
    const int np = bamf_gauss_mle_nparams(fit_type);
    if (!rois || !params || !crlb || !loglik || sz < 1 || nfits < 0 || np < 0) return BAMF_ERR_INVALID_ARG;
    if (var_gain_map && (!box_corners || map_size < 1)) return BAMF_ERR_INVALID_ARG;
    if (sz > MAXSZ) return BAMF_ERR_TOO_LARGE;
    if (nfits == 0) return BAMF_OK;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    /* one allocation for the call, its parts at multiples of 256 bytes */
    const size_t n = (size_t)nfits, npx = (size_t)sz * sz, nin = n * npx * 4, nout = n * np * 4;
    const size_t piece = std::min(n, std::max<size_t>(32, PLANES_BYTES / (npx * 4) / 32 * 32));
    size_t total = 0;
    auto part = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t at_r = part(nin), at_q = part(planes ? piece * npx * 4 : 0), at_p = part(nout), at_c = part(nout),
                 at_l = part(n * 4), at_co = part(var_gain_map ? n * 2 * 4 : 0),
                 at_m = part(var_gain_map ? (size_t)map_size * map_size * 4 : 0);
    char *mem = nullptr;
    if (cudaMalloc(&mem, total) != cudaSuccess) {
        cudaGetLastError();
        return BAMF_ERR_CUDA;
    }
    float *dr = (float *)(mem + at_r), *dq = (float *)(mem + at_q), *dp = (float *)(mem + at_p),
          *dc = (float *)(mem + at_c), *dl = (float *)(mem + at_l);
    float *dco = var_gain_map ? (float *)(mem + at_co) : nullptr, *dm = var_gain_map ? (float *)(mem + at_m) : nullptr;
    bamf_status st = BAMF_OK;
    if (!planes && cudaMemcpy(dr, rois, nin, cudaMemcpyHostToDevice) != cudaSuccess) st = BAMF_ERR_CUDA;
    if (!st && var_gain_map &&
        (cudaMemcpy(dco, box_corners, n * 2 * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
         cudaMemcpy(dm, var_gain_map, (size_t)map_size * map_size * 4, cudaMemcpyHostToDevice) != cudaSuccess))
        st = BAMF_ERR_CUDA;
    for (size_t f0 = 0; !st && planes && f0 < n; f0 += piece) {
        const size_t m = std::min(piece, n - f0);
        /* the planes' values of the fits f0 ..; of all fits they are one piece of memory */
        const size_t rows = m == n ? 1 : npx, row = m == n ? npx * n : m;
        for (size_t q = 0; !st && q < rows; ++q)
            if (cudaMemcpy(dq + q * m, rois + f0 + q * n, row * 4, cudaMemcpyHostToDevice) != cudaSuccess)
                st = BAMF_ERR_CUDA;
        if (st) break;
        planes_kernel<<<(unsigned)((m - 1) / 32 + 1), 256>>>(dq, sz, (int)m, dr + f0 * npx);
        if (cudaGetLastError() != cudaSuccess) st = BAMF_ERR_CUDA;
    }
    if (!st)
        st = bamf_gauss_mle_fit_device(dr, sz, nfits, fit_type, psf_sigma, zfit, dco, dm, map_size, iterations, dp,
                                       dc, dl, nullptr);
    if (!st && cudaDeviceSynchronize() != cudaSuccess) st = BAMF_ERR_CUDA;
    if (!st && (cudaMemcpy(params, dp, nout, cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(crlb, dc, nout, cudaMemcpyDeviceToHost) != cudaSuccess ||
                cudaMemcpy(loglik, dl, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess))
        st = BAMF_ERR_CUDA;
    cudaFree(mem);
    if (st) cudaGetLastError();
    return st;
}

}  // namespace

extern "C" bamf_status bamf_gauss_mle_fit_host(const float *rois, int sz, int nfits, int fit_type, float psf_sigma,
                                               const bamf_zfit *zfit, const float *box_corners,
                                               const float *var_gain_map, int map_size, int iterations,
                                               float *params, float *crlb, float *loglik)
{
    return fit_host(rois, false, sz, nfits, fit_type, psf_sigma, zfit, box_corners, var_gain_map, map_size, iterations,
                    params, crlb, loglik);
}

extern "C" bamf_status bamf_gauss_mle_fit_host_planes(const float *planes, int sz, int nfits, int fit_type,
                                                      float psf_sigma, const bamf_zfit *zfit,
                                                      const float *box_corners, const float *var_gain_map,
                                                      int map_size, int iterations, float *params, float *crlb,
                                                      float *loglik)
{
    return fit_host(planes, true, sz, nfits, fit_type, psf_sigma, zfit, box_corners, var_gain_map, map_size, iterations,
                    params, crlb, loglik);
}

/*
 * gaussmle_axis.cuh - what the gaussMLE kernels share: a group of GL lanes per
 * fit, the model's per-axis terms, the start values, and the group's sums.
 *
 * The model is separable: the integrated PSF of a pixel is a product of one
 * factor per axis, and so are its derivatives, up to the other axis's PSF.  The
 * factors of index i are differences of the same functions at the pixel edges i
 * and i + 1, so an iteration evaluates erf and exp once per edge (sz + 1 per
 * axis) instead of twice per index, and the pixel loops only multiply.
 */
#pragma once

#include <cuda_runtime.h>

namespace {

constexpr int GL = 8;     /* lanes per fit: four fits per warp */
#define MLE_PI 3.141592f  /* definitions.h:13 */

/* 1 / x for a normal x whose reciprocal is normal: the hardware's estimate and
 * one Newton step from its exact residual (within 0.51 ulp; no special cases) */
__device__ __forceinline__ float recip(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}

__device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* Sums of N pairs (N <= 4) over the group, lane pair l >> 1 = k ending with pair
 * k in a[0], b[0]: each step halves the pairs a lane carries, so it takes 8
 * shuffles for four pairs instead of 24; the additions are group_sum's. */
__device__ __forceinline__ void group_sum_pairs(float (&a)[4], float (&b)[4], int l)
{
    const bool hi = l & 4;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float sa = __shfl_xor_sync(0xffffffffu, hi ? a[k] : a[2 + k], 4);
        const float sb = __shfl_xor_sync(0xffffffffu, hi ? b[k] : b[2 + k], 4);
        a[k] = (hi ? a[2 + k] : a[k]) + sa;
        b[k] = (hi ? b[2 + k] : b[k]) + sb;
    }
    const bool odd = l & 2;
    const float sa = __shfl_xor_sync(0xffffffffu, odd ? a[0] : a[1], 2);
    const float sb = __shfl_xor_sync(0xffffffffu, odd ? b[0] : b[1], 2);
    a[0] = (odd ? a[1] : a[0]) + sa;
    b[0] = (odd ? b[1] : b[0]) + sb;
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    b[0] += __shfl_xor_sync(0xffffffffu, b[0], 1);
}

/* erf and exp at the edges q = 0..sz of an axis: erf((q - c) / (sqrt 2 sigma)),
 * exp(-(q - c)^2 / (2 sigma^2)), GL lanes */
__device__ __forceinline__ void axis_edges(float2 *edge, int sz, float c, float inv_s, float erf_s, int l)
{
    for (int q = l; q <= sz; q += GL) {
        const float u = (float)q - c, v = u * inv_s;
        edge[q] = make_float2(erff(u * erf_s), expf(-0.5f * (v * v)));
    }
}

/* kernel_CenterofMass2D and kernel_GaussFMaxMin2D (GPUgaussLib.cuh:207-258) of
 * the group's ROI d: the centre, and the largest and smallest value of the
 * Gaussian-filtered ROI.  The filter is separable, rows into tmp (sz * sz), then
 * columns; w holds the 2 sz - 1 weights of width sigma, norm the sz sums of the
 * weights that reach index k (both filled by `filter_tables` for the block). */
__device__ __forceinline__ void filter_tables(float *w, float *norm, int sz, float sigma)
{
    const float nrm = 1.0f / 2.0f / sigma / sigma;
    for (int q = threadIdx.x; q < 2 * sz - 1; q += blockDim.x) {
        const int k = q - (sz - 1);
        w[q] = expf(-(float)(k * k) * nrm);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < sz; k += blockDim.x) {
        float s = 0.0f;
        for (int i = 0; i < sz; ++i) s += w[i - k + sz - 1];
        norm[k] = s;
    }
}

template <int SZ>
__device__ __forceinline__ void start_values(const float *d, float *tmp, const float *w, const float *norm,
                                             const int *pix, int sz_, int l, float *c0, float *c1, float *fmax_,
                                             float *fmin_)
{
    const int sz = SZ > 0 ? SZ : sz_, npx = sz * sz;
    float tx = 0.0f, ty = 0.0f, ts = 0.0f;
    for (int p = l; p < npx; p += GL) {
        const int ii = pix[p] >> 8, jj = pix[p] & 255; /* pixel d[sz*jj + ii] */
        const float v = d[sz * jj + ii];
        tx += v * ii;
        ty += v * jj;
        ts += v;
        /* row jj of d filtered at ii */
        float f = 0.0f;
#pragma unroll
        for (int q = 0; q < sz; ++q) f += w[q - ii + sz - 1] * d[sz * jj + q];
        tmp[sz * jj + ii] = f;
    }
    tx = group_sum(tx);
    ty = group_sum(ty);
    ts = group_sum(ts);
    *c0 = tx / ts;
    *c1 = ty / ts;
    __syncwarp();
    float mx = 0.0f, mn = 10e10f;
    for (int p = l; p < npx; p += GL) {
        const int ii = pix[p] >> 8, jj = pix[p] & 255;
        float f = 0.0f;
#pragma unroll
        for (int q = 0; q < sz; ++q) f += w[q - jj + sz - 1] * tmp[sz * q + ii];
        f /= norm[ii] * norm[jj];
        mx = fmaxf(mx, f);
        mn = fminf(mn, f);
    }
#pragma unroll
    for (int o = GL / 2; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    }
    *fmax_ = mx;
    *fmin_ = mn;
}

/* The CRLB, the diagonal of the inverse of the Fisher matrix with the distinct
 * entries F (row by row): LU without pivoting in the order of kernel_MatInvN
 * (MatInvLib.h:15-75).  Every lane factors; lane num < NV solves for unit vector
 * num and returns its element num (the reference solves them one by one). */
template <int NV>
__device__ __forceinline__ float inverse_diagonal(const float (&F)[NV * (NV + 1) / 2], int num)
{
    float M[NV][NV]; /* row, column */
    int e = 0;
#pragma unroll
    for (int a = 0; a < NV; a++)
#pragma unroll
        for (int b = a; b < NV; b++) {
            M[a][b] = M[b][a] = F[e];
            ++e;
        }
    float rd[NV]; /* 1 / M[i][i] */
#pragma unroll
    for (int jj = 0; jj < NV; jj++) {
#pragma unroll
        for (int ii = 1; ii < NV; ii++) {
            float t = 0.0f;
#pragma unroll
            for (int q = 0; q < NV; q++)
                if (q < ii && q < jj) t += M[ii][q] * M[q][jj];
            if (ii <= jj) M[ii][jj] -= t;
        }
        rd[jj] = 1 / M[jj][jj];
#pragma unroll
        for (int ii = 1; ii < NV; ii++)
            if (ii > jj) {
                float t = 0.0f;
#pragma unroll
                for (int q = 0; q < NV; q++)
                    if (q < jj) t += M[ii][q] * M[q][jj];
                M[ii][jj] = rd[jj] * (M[ii][jj] - t);
            }
    }
    float y[NV], x[NV], out = 0.0f;
#pragma unroll
    for (int ii = 0; ii < NV; ii++) {
        float t = 0.0f;
#pragma unroll
        for (int q = 0; q < NV; q++)
            if (q < ii) t += M[ii][q] * y[q];
        y[ii] = (ii == num ? 1.0f : 0.0f) - t;
    }
#pragma unroll
    for (int ii = NV - 1; ii >= 0; ii--) {
        float t = 0.0f;
#pragma unroll
        for (int q = 0; q < NV; q++)
            if (q > ii) t += M[ii][q] * x[q];
        x[ii] = ii == NV - 1 ? y[ii] / M[ii][ii] : rd[ii] * (y[ii] - t);
        if (ii == num) out = x[ii];
    }
    return out;
}

}  // namespace

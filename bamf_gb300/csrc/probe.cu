/*
 * probe.cu - throughput probes for the sampler's roofline denominators:
 * FP32 FMA and MUFU log2 issue rates of the current device, measured with
 * independent chains so the pipes, not latency, set the rate.
 */
#include <cuda_runtime.h>

#include "bamf.h"
#include "parity_quick.cuh"

/* a failed CUDA runtime call: clear its error so that a later call on this
 * thread does not report it again */
static inline bamf_status clear_cuda_error()
{
    cudaGetLastError();
    return BAMF_ERR_CUDA;
}

namespace {

__global__ void fma_probe(float *out, int iters, float a, float b)
{
    float x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
    float x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
    for (int i = 0; i < iters; ++i) {
        x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
        x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
    }
    float s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
    if (s == 12345.678f) out[blockIdx.x] = s;
}

__global__ void mufu_probe(float *out, int iters)
{
    float x0 = 1.5f + threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
    for (int i = 0; i < iters; ++i) {
        x0 = __log2f(x0) + 2.0f; x1 = __log2f(x1) + 2.0f;
        x2 = __log2f(x2) + 2.0f; x3 = __log2f(x3) + 2.0f;
    }
    float s = x0 + x1 + x2 + x3;
    if (s == 12345.678f) out[blockIdx.x] = s;
}

}  // namespace

extern "C" bamf_status bamf_probe_peaks(double *fp32_flops, double *mufu_ops)
{
    if (!fp32_flops || !mufu_ops) return BAMF_ERR_INVALID_ARG;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return BAMF_ERR_NO_DEVICE;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    float *out = nullptr;
    if (cudaMalloc(&out, 65536 * sizeof(float)) != cudaSuccess) return clear_cuda_error();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = sms * 8, threads = 256;
    const int it_fma = 4096, it_mufu = 2048;
    cudaStream_t st;
    cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    float ms = 0.0f, best_fma = 1e30f, best_mufu = 1e30f;
    fma_probe<<<blocks, threads, 0, st>>>(out, 16, 1.0001f, 0.5f); /* warm-up */
    mufu_probe<<<blocks, threads, 0, st>>>(out, 16);
    for (int rep = 0; rep < 3; ++rep) {
        cudaEventRecord(e0, st);
        fma_probe<<<blocks, threads, 0, st>>>(out, it_fma, 1.0001f, 0.5f);
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        best_fma = ms < best_fma ? ms : best_fma;
        cudaEventRecord(e0, st);
        mufu_probe<<<blocks, threads, 0, st>>>(out, it_mufu);
        cudaEventRecord(e1, st);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        best_mufu = ms < best_mufu ? ms : best_mufu;
    }
    cudaStreamDestroy(st);
    *fp32_flops = 2.0 * 8.0 * it_fma * (double)blocks * threads / (best_fma * 1e-3);
    *mufu_ops = 4.0 * it_mufu * (double)blocks * threads / (best_mufu * 1e-3);
    cudaError_t err = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    return err == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

/* The parity math of the exact sampler (parity_quick.cuh) on the device:
 * out[i] = f(x[i]) for f = erf (0), log (1), exp (2); a host caller compares
 * with include/bamf_parity_math.h compiled for the CPU. */
__global__ void parity_math_kernel(const float *__restrict__ x, int n, int fn, float *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = x[i];
    out[i] = fn == 0 ? bamf::pq::erf_q(v) : (fn == 1 ? bamf::pq::log_q(v) : bamf::pq::exp_q(v));
}

extern "C" bamf_status bamf_parity_math_device(int fn, const float *x, int n, float *out)
{
    if (!x || !out || n < 0 || fn < 0 || fn > 2) return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    float *d = nullptr;
    if (cudaMalloc(&d, 2 * (size_t)n * sizeof(float)) != cudaSuccess) return clear_cuda_error();
    bamf_status st = BAMF_OK;
    if (cudaMemcpy(d, x, (size_t)n * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) st = BAMF_ERR_CUDA;
    if (!st) {
        parity_math_kernel<<<(n + 255) / 256, 256>>>(d, n, fn, d + n);
        if (cudaMemcpy(out, d + n, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
            st = BAMF_ERR_CUDA;
    }
    if (st) cudaGetLastError();
    cudaFree(d);
    return st;
}

/* pair i of the division check: significands, exponents and kind from a hash
 * of i (multiply and xor-shift rounds) */
__device__ __forceinline__ void division_pair(uint32_t i, float *a, float *b)
{
    uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ull + 0xD1B54A32D192ED03ull;
    for (int r = 0; r < 2; ++r) {
        h ^= h >> 32;
        h *= 0xD6E8FEB86659FD93ull;
    }
    h ^= h >> 32;
    uint32_t mb = (uint32_t)h & 0x7fffffu, mq = (uint32_t)(h >> 23) & 0x7fffffu;
    const uint32_t eb = 127u - 44u + (uint32_t)(h >> 46) % 88u; /* 2^-44 .. 2^43 */
    const uint32_t kind = (uint32_t)(h >> 54) & 3u, low = (uint32_t)(h >> 56) & 7u;
    if (kind == 2) mb = 0x7fffffu - low; /* next to the excluded significand */
    *b = __uint_as_float(eb << 23 | mb);
    const float one_b = __uint_as_float(127u << 23 | mb), q = __uint_as_float(127u << 23 | mq);
    if (kind == 0 || kind == 2) {
        *a = __uint_as_float((127u - 44u + (uint32_t)(h >> 40) % 88u) << 23 | mq);
    } else if (kind == 1) {
        /* a quotient next to the midpoint of q and the float after it */
        const float mid = (float)((double)one_b * ((double)q + 0x1p-24));
        const float t = __uint_as_float(__float_as_uint(mid) + low - 3u);
        *a = t * __uint_as_float(eb << 23); /* exact: a power of two */
    } else {
        *a = low == 0 ? *b : __uint_as_float(__float_as_uint(one_b * q) + low - 3u) * __uint_as_float(eb << 23);
    }
}

__global__ void parity_check_kernel(int fn, unsigned long long *bad)
{
    unsigned long long n = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (1ull << 32); i += stride) {
        if (fn == 3) {
            float a, b;
            division_pair((uint32_t)i, &a, &b);
            const float got = bamf::pq::div_try(a, b);
            const bool in = a >= 0x1p-40f && a < 0x1p40f && b >= 0x1p-40f && b < 0x1p40f &&
                            (__float_as_uint(b) & 0x7fffffu) != 0x7fffffu;
            n += in ? __float_as_uint(got) != __float_as_uint(__fdiv_rn(a, b)) : got == got;
        } else {
            const float x = __uint_as_float((uint32_t)i);
            const float want = fn == 0 ? bamf_pm_erff(x) : fn == 1 ? bamf_pm_logf(x) : bamf_pm_expf(x);
            const float got = fn == 0 ? bamf::pq::erf_q(x) : fn == 1 ? bamf::pq::log_q(x) : bamf::pq::exp_q(x);
            n += __float_as_uint(want) != __float_as_uint(got) && !(want != want && got != got);
        }
    }
    if (n) atomicAdd(bad, n);
}

extern "C" bamf_status bamf_parity_math_check(int fn, int64_t *mismatches)
{
    if (!mismatches || fn < 0 || fn > 3) return BAMF_ERR_INVALID_ARG;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    unsigned long long *d = nullptr, h = 0;
    if (cudaMalloc(&d, sizeof h) != cudaSuccess) return clear_cuda_error();
    bamf_status st = cudaMemset(d, 0, sizeof h) == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
    if (!st) {
        parity_check_kernel<<<sms * 8, 256>>>(fn, d);
        if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) st = BAMF_ERR_CUDA;
    }
    if (st) cudaGetLastError();
    cudaFree(d);
    *mismatches = (int64_t)h;
    return st;
}

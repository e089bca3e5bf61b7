/*
 * mapfit.cu - the chain summaries that follow the sampler in the reference's
 * analysis, on the device, from the thinned state records of the batched
 * sampler (bamf_batch_results.pos_trace):
 *
 *   findMap.m:29-111  MAP emitter count over the second half of the chain,
 *                     k-means (k = MAP count) of the positions of the states
 *                     with that count, and per-cluster mean / standard
 *                     deviation of X, Y, I; mean / std of the background
 *   mcmc.m:142-169    per-emitter mean / standard deviation over the second
 *                     half of a fixed-count (jumps-only) chain
 *
 * "Second half" is the reference's: with L = chain entries - 1 (the MEX
 * output drops the last entry), entries round(L/2) .. L (1-based) of the
 * accepted chain, i.e. 0-based entries ceil(L/2)-1 .. L-1, restricted here
 * to the recorded ones (every pos_thin-th entry).
 *
 * k-means: Lloyd iterations with squared Euclidean distance (ties to the
 * lower cluster), started from the emitters of the first qualifying state
 * (distinct points of one posterior sample), until no assignment changes
 * or max_iter; an empty cluster keeps its centre.  MATLAB's kmeans starts
 * from random k-means++ seeds, so cluster order and the last digits differ;
 * the clusters themselves are the same partition of a well-separated
 * posterior.  Standard deviations use n - 1 (MATLAB std); one point gives 0.
 */
#include <cuda_runtime.h>

#include <cmath>

#include "bamf.h"
#include "smem_limit.h"

/* a failed CUDA runtime call: clear its error so that a later call on this
 * thread does not report it again */
static inline bamf_status clear_cuda_error()
{
    cudaGetLastError();
    return BAMF_ERR_CUDA;
}

namespace {

constexpr int S = BAMF_POS_SLOTS;
constexpr int REC = BAMF_POS_RECORD;
constexpr int THREADS = 128;
constexpr int MAX_POS_LEN = 256;

__device__ __forceinline__ float nanf_() { return __int_as_float(0x7fc00000); }

constexpr int TREES = 12; /* sums per round */

/* res[i] = the sum of part[i][0 .. THREADS - 1] as a tree (halves added, 64 apart,
 * then 32, ... 1), i < n, warp w taking the sums w, w + 4, ....  The GPU adds two
 * doubles per cycle and SM, so a sum is a warp's 8 additions instead of seven
 * rounds of the whole block. */
__device__ __forceinline__ void tree_sums(const double (*part)[THREADS], int n, double *res)
{
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < n; i += THREADS / 32) {
        double v = (part[i][lane] + part[i][lane + 64]) + (part[i][lane + 32] + part[i][lane + 96]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) res[i] = v;
    }
}

/* mean and standard deviation (n - 1) from the count, sum and sum of squares */
__device__ __forceinline__ void mean_std(double n, double a, double a2, float *mean, float *std_)
{
    *mean = n > 0 ? (float)(a / n) : nanf_();
    *std_ = n > 1 ? (float)sqrt(fmax(0.0, (a2 - a * a / n) / (n - 1.0))) : (n == 1 ? 0.0f : nanf_());
}

struct Range {
    int lo, hi; /* qualifying 0-based entries lo .. hi */
};

__device__ __forceinline__ Range second_half(int n_entries)
{
    int iter = n_entries - 1;
    Range r;
    r.lo = (iter + 1) / 2 - 1;
    r.hi = iter - 1;
    return r;
}

/* records that can qualify: the entries of a chain's second half, or what of
 * them a truncated trace holds */
__host__ __device__ constexpr int max_records(int pos_len) { return pos_len / 2 + 2; }
__host__ __device__ constexpr size_t kmeans_smem(int pos_len)
{
    return (size_t)max_records(pos_len) * (S * (2 * sizeof(float) + 1) + sizeof(uint16_t));
}

/* A CTA per ROI; point p = j K + s is emitter s of qualifying record j, thread t
 * owns the points t, t + 128, ....  A round of sums takes four clusters' positions
 * or two clusters' six statistics, and only clusters that won or lost a point have
 * their centre computed again.  Bound by the double-precision additions.  3,380
 * ROIs, 200 records: 5.0 ms with room for 256 records' points of three
 * coordinates in shared memory (one CTA per SM) and every sum by the whole
 * block, 1.3 ms like this. */
__global__ void __launch_bounds__(THREADS) map_kmeans_kernel(const float *__restrict__ pos, int pos_len,
                                                             int pos_thin, const int32_t *__restrict__ n_entries,
                                                             const int32_t *__restrict__ map_n, int n,
                                                             int max_iter, float *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int cap = max_records(pos_len);
    float *PX = (float *)smem_raw;
    float *PY = PX + cap * S;
    uint16_t *recs = (uint16_t *)(PY + cap * S); /* the qualifying records */
    uint8_t *asg = (uint8_t *)(recs + cap);
    __shared__ double part[TREES][THREADS], res[TREES];
    __shared__ int cntp[4][THREADS];
    __shared__ int wcount[THREADS / 32];
    __shared__ float cx[S], cy[S];
    __shared__ unsigned dirty_sh;
    __shared__ int size[S]; /* points per cluster */
    const int roi = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (roi >= n) return;
    float *o = out + (int64_t)roi * BAMF_MAP_RECORD;
    const float *rp = pos + (int64_t)roi * pos_len * REC;
    const Range rg = second_half(n_entries[roi]);
    const int nw = min(pos_len, (n_entries[roi] + pos_thin - 1) / pos_thin); /* records written */
    const int K = min(max(map_n[roi], 0), S);
    /* the qualifying records, in order, and the background's sums */
    int nrec = 0;
    double sb = 0.0, sb2 = 0.0, sa = 0.0, sbb = 0.0;
    for (int b0 = 0; b0 < nw; b0 += THREADS) {
        const int r = b0 + t;
        const float *rec = rp + (int64_t)min(r, nw - 1) * REC;
        bool q = false;
        if (r < nw) {
            const int e = r * pos_thin;
            q = rec[1] == (float)K && e >= rg.lo && e <= rg.hi;
        }
        if (q) {
            sb += rec[2];
            sb2 += (double)rec[2] * rec[2];
            sa += rec[3];
            sbb += rec[4];
        }
        const unsigned m = __ballot_sync(0xffffffffu, q);
        if (lane == 0) wcount[warp] = __popc(m);
        __syncthreads();
        int at = nrec + __popc(m & ((1u << lane) - 1));
#pragma unroll
        for (int k = 0; k < THREADS / 32; ++k) {
            if (k < warp) at += wcount[k];
            nrec += wcount[k];
        }
        if (q && at < cap) recs[at] = (uint16_t)r;
        __syncthreads();
    }
    nrec = min(nrec, cap);
    part[0][t] = sb;
    part[1][t] = sb2;
    part[2][t] = sa;
    part[3][t] = sbb;
    for (int s = t; s < 6 * S; s += THREADS) o[6 + s] = nanf_();
    __syncthreads();
    tree_sums(part, 4, res);
    __syncthreads();
    if (t == 0) {
        const double tc = (double)nrec;
        o[0] = (float)K;
        o[1] = (float)nrec;
        mean_std(tc, res[0], res[1], o + 2, o + 3);
        o[4] = tc > 0 ? (float)(res[2] / tc) : nanf_();
        o[5] = tc > 0 ? (float)(res[3] / tc) : nanf_();
    }
    if (K == 0 || nrec == 0) return;
    const int npts = nrec * K, dj = THREADS / K, ds = THREADS % K;
    {
        int j = t / K, s = t - j * K;
        for (int p = t; p < npts; p += THREADS) {
            const float *rec = rp + (int64_t)recs[j] * REC + 5;
            PX[p] = rec[s];
            PY[p] = rec[S + s];
            asg[p] = 255;
            j += dj;
            s += ds;
            if (s >= K) {
                s -= K;
                ++j;
            }
        }
    }
    if (t < S) size[t] = 0;
    if (t == 0) dirty_sh = 0;
    __syncthreads();
    if (t < K) {
        cx[t] = PX[t];
        cy[t] = PY[t];
    }
    __syncthreads();
    /* Lloyd iterations */
    for (int it = 0; it < max_iter; ++it) {
        unsigned moved = 0; /* clusters that won or lost one of this thread's points */
        for (int p = t; p < npts; p += THREADS) {
            const float bx = PX[p], by = PY[p];
            int best = 0;
            float bd = INFINITY;
            for (int c = 0; c < K; ++c) {
                const float dx = bx - cx[c], dy = by - cy[c];
                const float d = dx * dx + dy * dy;
                if (d < bd) {
                    bd = d;
                    best = c;
                }
            }
            const int old = asg[p];
            if (old != best) {
                asg[p] = (uint8_t)best;
                moved |= 1u << best;
                if (old < S) moved |= 1u << old;
            }
        }
        moved = __reduce_or_sync(0xffffffffu, moved);
        if (lane == 0 && moved) atomicOr(&dirty_sh, moved);
        __syncthreads();
        unsigned dirty = dirty_sh;
        if (!dirty) break;
        while (dirty) {
            int cl[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                cl[k] = dirty ? __ffs(dirty) - 1 : -1;
                dirty &= dirty - 1;
                if (cl[k] < 0) continue;
                double sx = 0.0, sy = 0.0;
                int sn = 0;
                for (int p = t; p < npts; p += THREADS)
                    if (asg[p] == cl[k]) {
                        sx += PX[p];
                        sy += PY[p];
                        ++sn;
                    }
                part[2 * k][t] = sx;
                part[2 * k + 1][t] = sy;
                cntp[k][t] = sn;
            }
            __syncthreads();
            const int mine = warp == 0 ? cl[0] : warp == 1 ? cl[1] : warp == 2 ? cl[2] : cl[3];
            if (mine >= 0) {
                const int sn = __reduce_add_sync(0xffffffffu, cntp[warp][lane] + cntp[warp][lane + 32] +
                                                                  cntp[warp][lane + 64] + cntp[warp][lane + 96]);
                double v[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const double *pv = part[2 * warp + k];
                    v[k] = (pv[lane] + pv[lane + 64]) + (pv[lane + 32] + pv[lane + 96]);
                }
#pragma unroll
                for (int o2 = 16; o2 > 0; o2 >>= 1) {
                    v[0] += __shfl_down_sync(0xffffffffu, v[0], o2);
                    v[1] += __shfl_down_sync(0xffffffffu, v[1], o2);
                }
                if (lane == 0) {
                    size[mine] = sn;
                    if (sn > 0) {
                        cx[mine] = (float)(v[0] / (double)sn);
                        cy[mine] = (float)(v[1] / (double)sn);
                    }
                }
            }
            if (t == 0) dirty_sh = 0;
            __syncthreads();
        }
    }
    /* per-cluster mean and standard deviation of X, Y, I, two clusters a round */
    for (int c0 = 0; c0 < K; c0 += 2) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            double a[3] = {0, 0, 0}, a2[3] = {0, 0, 0};
            int j = t / K, s = t - j * K;
            for (int p = t; p < npts; p += THREADS) {
                if (asg[p] == c0 + k) {
                    const double v[3] = {PX[p], PY[p], rp[(int64_t)recs[j] * REC + 5 + 2 * S + s]};
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        a[q] += v[q];
                        a2[q] += v[q] * v[q];
                    }
                }
                j += dj;
                s += ds;
                if (s >= K) {
                    s -= K;
                    ++j;
                }
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                part[6 * k + q][t] = a[q];
                part[6 * k + 3 + q][t] = a2[q];
            }
        }
        __syncthreads();
        tree_sums(part, min(2, K - c0) * 6, res);
        __syncthreads();
        if (t < 6 && c0 + t / 3 < K) {
            const int c = c0 + t / 3, q = t % 3;
            mean_std((double)size[c], res[t / 3 * 6 + q], res[t / 3 * 6 + 3 + q], o + 6 + q * S + c,
                     o + 6 + (3 + q) * S + c);
        }
    }
}

/* mcmc.m:142-169: per-slot mean and std over the second half of a
 * fixed-count chain (the count is taken from the first record in range).
 * Thread t owns the records t, t + 128, ...; two slots a round of sums. */
__global__ void __launch_bounds__(THREADS) refine_stats_kernel(const float *__restrict__ pos, int pos_len,
                                                               int pos_thin, const int32_t *__restrict__ n_entries,
                                                               int n, float *__restrict__ out)
{
    __shared__ double part[TREES][THREADS], res[TREES];
    const int roi = blockIdx.x, t = threadIdx.x;
    if (roi >= n) return;
    float *o = out + (int64_t)roi * BAMF_MAP_RECORD;
    const float *rp = pos + (int64_t)roi * pos_len * REC;
    const Range rg = second_half(n_entries[roi]);
    const int nw = min(pos_len, (n_entries[roi] + pos_thin - 1) / pos_thin);
    /* records r in range: rg.lo <= r * pos_thin <= rg.hi */
    const int r0 = max(0, (rg.lo + pos_thin - 1) / pos_thin);
    const int r1 = min(nw - 1, rg.hi >= 0 ? rg.hi / pos_thin : -1);
    const int nrec = max(0, r1 - r0 + 1);
    const int kf = nrec > 0 ? min((int)rp[(int64_t)r0 * REC + 1], S) : 0;
    if (t == 0) {
        o[0] = (float)kf;
        o[1] = (float)nrec;
        o[2] = o[3] = o[4] = o[5] = nanf_();
    }
    for (int s = t; s < 6 * S; s += THREADS) o[6 + s] = nanf_();
    for (int s0 = 0; s0 < kf; s0 += 2) {
        double a[6] = {0, 0, 0, 0, 0, 0}, a2[6] = {0, 0, 0, 0, 0, 0}; /* [slot][X, Y, I] */
        for (int r = r0 + t; r <= r1; r += THREADS) {
            const float *rec = rp + (int64_t)r * REC + 5 + s0;
            const bool two = s0 + 1 < kf;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double v = rec[k * S];
                a[k] += v;
                a2[k] += v * v;
                if (two) {
                    const double w = rec[k * S + 1];
                    a[3 + k] += w;
                    a2[3 + k] += w * w;
                }
            }
        }
        __syncthreads(); /* the last round's sums are read; the NaNs are written */
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            part[2 * k][t] = a[k];
            part[2 * k + 1][t] = a2[k];
        }
        __syncthreads();
        tree_sums(part, min(2, kf - s0) * 6, res);
        __syncthreads();
        if (t < 6 && s0 + t / 3 < kf) {
            const int sl = s0 + t / 3, k = t % 3;
            mean_std((double)nrec, res[2 * t], res[2 * t + 1], o + 6 + k * S + sl, o + 6 + (3 + k) * S + sl);
        }
    }
}

}  // namespace

extern "C" bamf_status bamf_map_kmeans_device(const float *pos_trace, int pos_len, int pos_thin,
                                              const int32_t *n_entries, const int32_t *map_n, int n, int max_iter,
                                              float *out, void *stream)
{
    if (n < 0 || pos_len < 1 || pos_len > MAX_POS_LEN || pos_thin < 1 || max_iter < 1) return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    if (!pos_trace || !n_entries || !map_n || !out) return BAMF_ERR_INVALID_ARG;
    const size_t smem = kmeans_smem(pos_len);
    if (allow_smem(map_kmeans_kernel, kmeans_smem(MAX_POS_LEN)) != cudaSuccess) return clear_cuda_error();
    map_kmeans_kernel<<<n, THREADS, smem, (cudaStream_t)stream>>>(pos_trace, pos_len, pos_thin, n_entries, map_n,
                                                                  n, max_iter, out);
    return cudaGetLastError() == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

extern "C" bamf_status bamf_refine_stats_device(const float *pos_trace, int pos_len, int pos_thin,
                                                const int32_t *n_entries, int n, float *out, void *stream)
{
    if (n < 0 || pos_len < 1 || pos_thin < 1) return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    if (!pos_trace || !n_entries || !out) return BAMF_ERR_INVALID_ARG;
    refine_stats_kernel<<<n, THREADS, 0, (cudaStream_t)stream>>>(pos_trace, pos_len, pos_thin, n_entries, n, out);
    return cudaGetLastError() == cudaSuccess ? BAMF_OK : BAMF_ERR_CUDA;
}

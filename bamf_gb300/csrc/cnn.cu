/*
 * cnn.cu - the learned birth proposal (include/bamf_cnn.h): synthetic ROI
 * generator, the network's forward (net_kernel, for training and for
 * inference into the sampler's LEARNED birth tables) and backward kernels,
 * Adam, and a CUDA-graph training step.
 *
 * Layouts.  Activations are channels-last BF16, [roi][p][32] with pixel
 * p = y + 16 x.  The three 32 -> 32 convolutions run on the 5th-generation
 * tensor cores (tcgen05.mma from shared-memory descriptors into TMEM): the
 * forward pass in net_kernel, the input and weight gradients in
 * conv_bwd_kernel, per ROI implicit GEMMs over its 256 pixels whose operands
 * are the channels-last rows as they lie, without a transpose.
 */
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "bamf.h"
#include "bamf_cnn.h"
#include "bamf_philox.h"
#include "tc_ptx.cuh"

namespace {

constexpr int S = BAMF_CNN_SIDE;  /* 16 */
constexpr int NPX = S * S;        /* 256 */
constexpr int CH = BAMF_CNN_CH;   /* 32 */
constexpr int PS = S + 2;         /* padded side */
constexpr int NC = BAMF_CNN_COUNTS;
constexpr int NSUB = 16;
constexpr int MAX_BATCH = 4096;

/* parameter offsets */
constexpr int O_W1 = 0, O_B1 = 288, O_W2 = 320, O_B2 = 9536, O_W3 = 9568, O_B3 = 18784, O_W4 = 18816,
              O_B4 = 28032, O_WL = 28064, O_BL = 28576, O_WC = 28592, O_BC = 28944, NPARAM = 28955;
static_assert(NPARAM == BAMF_CNN_NPARAM, "parameter count");
static_assert(O_B1 == O_W1 + 288 && O_BC + NC == NPARAM, "conv1 block and head layout");
constexpr int HEAD_NPARAM = NPARAM - O_WL; /* WL, BL, WC, BC: the heads' parameters, contiguous */
static_assert(O_BL == O_WL + NSUB * CH && O_WC == O_BL + NSUB && O_BC == O_WC + NC * CH, "head layout");
constexpr int C1_NPARAM = O_W2;            /* W1, B1 */
/* the WC part of ROI r's head-gradient row */
__device__ __forceinline__ float *row_wc(float *rows, int r) { return rows + (size_t)r * HEAD_NPARAM + (O_WC - O_WL); }
constexpr int PKT = 9 * CH * CH; /* tensor-core operand weights of one layer */

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float u01(uint32_t w)
{
    return ((float)(w >> 8) + 0.5f) * (1.0f / 16777216.0f); /* (0, 1) */
}

/* ------------------------------------------------------------- generator */
/* Poisson(lam): multiplication method below 10, else the PTRS transformed
 * rejection of W. Hoermann, "The transformed rejection method for generating
 * Poisson random variables", Insurance: Mathematics and Economics 12 (1993).
 * Uniforms come from the Philox blocks (c0, c1, c2, j) of key (k0, k1). */
__device__ int poisson_draw(float lam, uint32_t c0, uint32_t c1, uint32_t c2, uint32_t k0, uint32_t k1)
{
    if (!(lam > 0.0f)) return 0;
    if (lam < 10.0f) {
        float L = expf(-lam), prod = 1.0f;
        int n = 0;
        for (uint32_t j = 0; j < 16; ++j) {
            bamf_philox_block b = bamf_philox4x32_10(c0, c1, c2, j, k0, k1);
            for (int w = 0; w < 4; ++w) {
                prod *= u01(b.v[w]);
                if (prod <= L) return n;
                ++n;
            }
        }
        return n;
    }
    const float slam = sqrtf(lam), loglam = logf(lam);
    const float b = 0.931f + 2.53f * slam;
    const float a = -0.059f + 0.02483f * b;
    const float invalpha = 1.1239f + 1.1328f / (b - 3.4f);
    const float vr = 0.9277f - 3.6224f / (b - 2.0f);
    for (uint32_t j = 0; j < 32; ++j) {
        bamf_philox_block blk = bamf_philox4x32_10(c0, c1, c2, j, k0, k1);
        for (int h = 0; h < 2; ++h) {
            float U = u01(blk.v[2 * h]) - 0.5f;
            float V = u01(blk.v[2 * h + 1]);
            float us = 0.5f - fabsf(U);
            float k = floorf((2.0f * a / us + b) * U + lam + 0.43f);
            if (us >= 0.07f && V <= vr) return (int)k;
            if (k < 0.0f || (us < 0.013f && V > us)) continue;
            if (logf(V) + logf(invalpha) - logf(a / (us * us) + b) <= -lam + k * loglam - lgammaf(k + 1.0f))
                return (int)k;
        }
    }
    return (int)floorf(lam + 0.5f); /* not reached in practice (acceptance > 0.9 per round) */
}

__global__ void synth_kernel(bamf_synth_params sp, uint32_t seed, uint64_t first, const int *step_dev,
                             int batch, int n, float *__restrict__ data, int32_t *__restrict__ n_em,
                             float *__restrict__ xyi)
{
    __shared__ float ex[BAMF_SYNTH_NMAX], ey[BAMF_SYNTH_NMAX], ei[BAMF_SYNTH_NMAX];
    __shared__ int ne;
    int r = blockIdx.x;
    if (r >= n) return;
    uint64_t k = (step_dev ? (uint64_t)(*step_dev) * (uint64_t)batch : first) + (uint64_t)r;
    uint32_t klo = (uint32_t)k, khi = (uint32_t)(k >> 32);
    const uint32_t K1 = 0x6a09e667u ^ khi;
    int t = threadIdx.x;
    if (t == 0) {
        float L = expf(-sp.mean_n), prod = 1.0f;
        int cnt = 0;
        bool done = false;
        for (uint32_t j = 0; j < 16 && !done; ++j) {
            bamf_philox_block b = bamf_philox4x32_10(klo, 0u, j, 0u, seed, K1);
            for (int w = 0; w < 4; ++w) {
                prod *= u01(b.v[w]);
                if (prod <= L) {
                    done = true;
                    break;
                }
                ++cnt;
            }
        }
        ne = min(cnt, BAMF_SYNTH_NMAX);
    }
    if (t < BAMF_SYNTH_NMAX) {
        bamf_philox_block b = bamf_philox4x32_10(klo, 1u, (uint32_t)t, 0u, seed, K1);
        ex[t] = (float)S * u01(b.v[0]);
        ey[t] = (float)S * u01(b.v[1]);
        float z = sqrtf(-2.0f * logf(u01(b.v[2]))) * cospif(2.0f * u01(b.v[3]));
        ei[t] = expf(logf(sp.i_median) + sp.i_logsd * z);
    }
    __syncthreads();
    const int nn = ne;
    if (t < BAMF_SYNTH_NMAX) {
        float *o = xyi + ((size_t)r * BAMF_SYNTH_NMAX + t) * 3;
        bool on = t < nn;
        o[0] = on ? ex[t] : 0.0f;
        o[1] = on ? ey[t] : 0.0f;
        o[2] = on ? ei[t] : 0.0f;
    }
    if (t == 0) n_em[r] = nn;
    int x = t / S, y = t - (t / S) * S;
    const float c = 1.0f / (sqrtf(2.0f) * sp.sigma);
    float bgv = sp.bg;
    if (sp.bg_max > sp.bg) {
        bamf_philox_block bb = bamf_philox4x32_10(klo, 3u, 0u, 0u, seed, K1);
        bgv = sp.bg + (sp.bg_max - sp.bg) * u01(bb.v[0]);
    }
    float lam = bgv;
    for (int e = 0; e < nn; ++e) {
        float sx = 0.5f * (erff(((float)x - ex[e] + 1.0f) * c) - erff(((float)x - ex[e]) * c));
        float sy = 0.5f * (erff(((float)y - ey[e] + 1.0f) * c) - erff(((float)y - ey[e]) * c));
        lam += ei[e] * sx * sy;
    }
    data[(size_t)r * NPX + t] = (float)poisson_draw(lam, klo, 2u, (uint32_t)t, seed, K1);
}

/* -------------------------------------------------------- weight packing */
/* The B operands of the 32 -> 32 convolutions for the tensor cores, per
 * layer [tap][ci group g][n][8] BF16 (K-major core matrices: 8 n x 8 k):
 * forward Wf: B[n = co][k = ci] = W_l[co][ci][tap]; input gradient Wb:
 * B[n = ci][k = co] = W_l[co][ci][8 - tap]. */
__global__ void pack_kernel(const float *__restrict__ P, bf16 *__restrict__ Wf, bf16 *__restrict__ Wb)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * PKT) return;
    int l = i / PKT, rem = i - l * PKT;
    int tap = rem / (CH * CH), nk = rem - tap * CH * CH;
    int nn = nk / CH, kk = nk - nn * CH;
    const float *W = P + (l == 0 ? O_W2 : (l == 1 ? O_W3 : O_W4));
    const int o = l * PKT + tap * CH * CH + (kk >> 3) * (CH * 8) + nn * 8 + (kk & 7);
    Wf[o] = __float2bfloat16_rn(W[(nn * CH + kk) * 9 + tap]);
    Wb[o] = __float2bfloat16_rn(W[(kk * CH + nn) * 9 + (8 - tap)]);
}

/* --------------------------------------------------------------- conv1 */
/* dW1, db1 from dz1 (= dL/d pre-activation of conv1) and x0: each CTA's
 * sums over its ROIs into row blockIdx.x of `rows` (C1_NPARAM floats).  Warp w
 * owns output channels 4w .. 4w + 3 (all 9 taps and the bias), lane l the
 * pixels l + 32 i: per pixel 9 neighbours and 4 dz values from shared
 * memory feed 40 register accumulators, kept over all the CTA's ROIs and
 * reduced over the warp once at the end. */
__global__ void __launch_bounds__(256) conv1_bwd_kernel(const float *__restrict__ x0, const bf16 *__restrict__ dz1,
                                                        int n, float *__restrict__ rows)
{
    __shared__ float xp[PS * PS];
    __shared__ float dz[NPX * (CH + 1)];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float acc[4][9], accb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        accb[j] = 0.0f;
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[j][k] = 0.0f;
    }
    for (int i = t; i < PS * PS; i += blockDim.x) xp[i] = 0.0f;
    for (int r = blockIdx.x; r < n; r += gridDim.x) {
        __syncthreads();
        {
            const int x = t / S, y = t - (t / S) * S;
            xp[(x + 1) * PS + (y + 1)] = x0[(size_t)r * NPX + t];
            const uint4 *src = (const uint4 *)(dz1 + ((size_t)r * NPX + t) * CH);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 u = src[q];
                const __nv_bfloat162 *b = (const __nv_bfloat162 *)&u;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(b[e]);
                    dz[t * (CH + 1) + 8 * q + 2 * e] = f.x;
                    dz[t * (CH + 1) + 8 * q + 2 * e + 1] = f.y;
                }
            }
        }
        __syncthreads();
#pragma unroll 2
        for (int i = 0; i < NPX / 32; ++i) {
            const int p = lane + 32 * i, x = p >> 4, y = p & 15;
            float nb[9];
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) nb[kx * 3 + ky] = xp[(x + kx) * PS + (y + ky)];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float d = dz[p * (CH + 1) + 4 * warp + j];
                accb[j] += d;
#pragma unroll
                for (int k = 0; k < 9; ++k) acc[j][k] += d * nb[k];
            }
        }
    }
    float *row = rows + (size_t)blockIdx.x * C1_NPARAM;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            float v = acc[j][k];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) row[(4 * warp + j) * 9 + k] = v;
        }
        float v = accb[j];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) row[288 + 4 * warp + j] = v;
    }
}

/* ------------------------------------ backward of the 32 -> 32 convolutions */
/* Per layer, last one first: from act (the layer's input) and dz (dL/d pre-activation of its
 * output), the input gradient masked by the input's ReLU,
 *   out[p][ci] = (act[p][ci] > 0) * sum over taps and co of
 *                dz[p + tap][co] Wb_tap[ci][co],
 * (Wb: taps flipped, pack_kernel), and the weight and bias gradients
 *   dW[co][ci][tap] = sum over ROIs and pixels p of act[p + tap][ci] dz[p][co],
 * tap = 3 kx + ky the shift (kx - 1, ky - 1) in (x, y).
 *
 * As a layer needs nothing of other ROIs, a persistent CTA runs its ROIs through
 * all three layers, one ROI per iteration, dz going back and forth between two
 * buffers of which it reads only what it wrote itself.  It stages dz once, [padded x][co
 * group g][padded y][8 co], and act as three copies shifted along y, [x][ky][ci
 * group g][y][8 ci], copy ky holding act[y + ky - 1] at y.  A 16-byte chunk of the
 * channels-last tensors (8 channels of one pixel) is a row of a core matrix in
 * both products, K-major in the first, MN-major in the second:
 *   input gradient: D[pixel][ci], 18 MMAs of 128 x 32 x 16 for each half y in [8
 *     h, 8 h + 8) of the ROI: a core matrix is 8 y of one x and g, the next 8 rows
 *     are the next x, tap (kx, ky) starts kx columns and ky rows in.
 *   weight gradient: D[(ky, ci)][(j, co)] += sum over y of act[x][y + ky - 1][ci]
 *     dz[x - 1 + j][y][co], j = 2 - kx, one MMA of 128 x 96 x 16 for each x: the
 *     columns of dz lie 4 groups apart, so the rows 32 j + co of B are one stride
 *     and the shift in x costs nothing; rows 96..127 of A are the column after
 *     (in bounds, ignored).  It stays in TMEM over all ROIs of the CTA.
 * The next ROI's chunks are loaded into registers while the MMAs run; the input
 * gradient's epilogue and the bias gradient's sums run during the weight
 * gradient's MMAs.  Each CTA writes its partial sums (D, then the 32 bias sums) to
 * its own slice of `part`; reduce_kernel adds the slices in a fixed order (no
 * atomics, the same bits every run).
 *
 * Bound by shared memory: 36 MMAs of 40 cycles and 16 of 56 a ROI, 2340 cycles
 * and layer (two CTAs per SM: 26 us for 1024 ROIs).  1024 ROIs are three or four a
 * CTA, so what a launch costs before its first MMA (2.6 to 4 us of allocation, first
 * loads and cold instructions) stands out: two kernels per layer, each with its own
 * staging, took 115 us, one per layer 72, this one 64, and 58 with the weights as
 * one bulk copy under the rest of the prologue.
 *
 * The mbarrier waits are bounded; a timeout is recorded in *status, and the CTA
 * starts no further copy or MMA, writes zeros, waits once more for what it has
 * started, frees its TMEM and returns. */
constexpr int BW_AG = S * 16;                    /* bytes of a group of act: 16 y of 8 channels */
constexpr int BW_ACOL = 12 * BW_AG;              /* an x column of the three copies of act */
constexpr int BW_DG = PS * 16;                   /* a group of dz */
constexpr int BW_DCOL = 4 * BW_DG;               /* an x column of dz */
constexpr int BW_ACT = PKT * 2;                  /* offsets: weights, act, dz, barriers */
constexpr int BW_DZ = BW_ACT + S * BW_ACOL + 4 * BW_AG;
constexpr int BW_BAR = BW_DZ + PS * BW_DCOL;
constexpr size_t SMEM_BW = BW_BAR + 3 * sizeof(uint64_t);
constexpr int BW_THREADS = 256;
constexpr int BW_TMEM = 256;                     /* columns: 96 of dW, 2 x 32 of the input gradient */
constexpr int DW_PART = 96 * 96 + CH;            /* floats of one CTA's partial sums */
constexpr uint32_t TC_IDESC = bamf::tc::idesc_bf16_f32(128, 32);
constexpr uint32_t DW_IDESC = bamf::tc::idesc_bf16_f32_mn(128, 96);
static_assert(BW_ACT % 16 == 0 && BW_DZ % 16 == 0 && BW_BAR % 16 == 0, "shared-memory alignment");

struct Backward {
    const bf16 *act[3]; /* the layers' inputs */
    bf16 *dz[2];        /* dL/dz of the last layer in dz[0]; layers 2, 1, 0 leave theirs in dz[1], [0], [1] */
    const bf16 *Wb;     /* packed weights, three layers */
    float *part;        /* layer l's slices at l * pitch */
    size_t pitch;
};

__global__ void __launch_bounds__(BW_THREADS, 2) conv_bwd_kernel(const Backward bw, int n, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *const As = smem_raw + BW_ACT, *const Ds = smem_raw + BW_DZ;
    uint64_t *const bar_in = (uint64_t *)(smem_raw + BW_BAR), *const bar_w = bar_in + 1, *const bar_wt = bar_in + 2;
    __shared__ uint32_t tslot;
    __shared__ float bred[4][CH];
    const int t = threadIdx.x, lane = t & 31;
    const int warp = __shfl_sync(0xffffffffu, t >> 5, 0); /* warp-uniform, and known to be */
    if (warp == 0) bamf::tc::tmem_alloc(&tslot, BW_TMEM);
    /* chunk k of this thread: pixel p0 + 64 k, channel group g; the 8 lanes of a
     * 16-byte store phase write 8 consecutive y of one group */
    constexpr int CPT = NPX * 4 / BW_THREADS;
    const int g = (t >> 3) & 3, p0 = (t & 7) + 8 * warp;
    uint4 pa[CPT], pd[CPT];
    float bsum[8];
    const auto load = [&](int l, int r) {
        const bf16 *act = l == 2 ? bw.act[2] : l == 1 ? bw.act[1] : bw.act[0], *dz = l == 1 ? bw.dz[1] : bw.dz[0];
        const uint4 *sa = (const uint4 *)(act + (size_t)r * NPX * CH) + p0 * 4 + g;
        const uint4 *sd = (const uint4 *)(dz + (size_t)r * NPX * CH) + p0 * 4 + g;
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            pa[k] = sa[64 * 4 * k];
            pd[k] = __ldcg(sd + 64 * 4 * k); /* written by this kernel: not through the read-only path */
        }
    };

    const auto stage = [&]() {
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int p = p0 + 64 * k, x = p >> 4, y = p & 15;
            *(uint4 *)(Ds + (x + 1) * BW_DCOL + g * BW_DG + (y + 1) * 16) = pd[k];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                const int yo = y - ky + 1;
                if (yo >= 0 && yo < S) *(uint4 *)(As + x * BW_ACOL + (4 * ky + g) * BW_AG + yo * 16) = pa[k];
            }
        }
    };
    /* warps 4..7: a group's 8 channels over the pixels (t & 7) + 8 (warp - 4) + 32 k */
    const auto bias_sums = [&]() {
        const int pb = p0 - 32;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int p = pb + 32 * k;
            const uint4 u = *(const uint4 *)(Ds + ((p >> 4) + 1) * BW_DCOL + g * BW_DG + ((p & 15) + 1) * 16);
            const __nv_bfloat162 *h = (const __nv_bfloat162 *)&u;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 f = __bfloat1622float2(h[c]);
                bsum[2 * c] += f.x;
                bsum[2 * c + 1] += f.y;
            }
        }
    };
    const int r0 = blockIdx.x;
    load(2, r0);
    if (t == 0) {
        bamf::tc::mbar_init(bar_in, 1);
        bamf::tc::mbar_init(bar_w, 1);
        bamf::tc::mbar_init(bar_wt, 1);
        bamf::tc::bulk_load(smem_raw, bw.Wb + 2 * PKT, PKT * 2, bar_wt);
    }
    {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int i = t; i < (BW_BAR - BW_ACT) / 16; i += BW_THREADS) ((uint4 *)As)[i] = z;
    }
    bamf::tc::fence_before_sync();
    __syncthreads();
    bamf::tc::fence_after_sync();
    const uint32_t tw = __shfl_sync(0xffffffffu, tslot, 0), tin = tw + 96;
    const uint64_t wd = bamf::tc::smem_desc(bamf::tc::smem_addr(smem_raw), CH * 16, 128);
    const uint64_t dk = bamf::tc::smem_desc(bamf::tc::smem_addr(Ds), BW_DG, BW_DCOL);
    const uint64_t am = bamf::tc::smem_desc(bamf::tc::smem_addr(As), 128, BW_AG);
    const uint64_t dm = bamf::tc::smem_desc(bamf::tc::smem_addr(Ds) + 16, 128, BW_DG);
    /* this thread's pixel of the input gradient: row m of half h */
    const int h = warp >> 2, m = 32 * (warp & 3) + lane, ex = m >> 3, ey = 8 * h + (m & 7);
    const uint32_t tlane = (uint32_t)((warp & 3) * 32) << 16;
    bool alive = true;
    uint32_t phase = 0;
    int loaded = 2; /* the last layer whose weights were asked for */
#pragma unroll 1
    for (int l = 2; l >= 0; --l) {
        bool first = true;
#pragma unroll
        for (int c = 0; c < 8; ++c) bsum[c] = 0.0f;
        bf16 *const out = l == 1 ? bw.dz[0] : bw.dz[1];
        stage();
        if (alive && !bamf::tc::mbar_wait(bar_wt, l & 1, 1u << 24)) { /* the layer's weights */
            atomicExch(status, 1);
            alive = false;
        }
        alive = __syncthreads_and(alive);
        for (int r = r0; r < n && alive; r += gridDim.x) {
            bamf::tc::fence_proxy_async();
            bamf::tc::fence_before_sync();
            __syncthreads();
            bamf::tc::fence_after_sync();
            if (warp == 0) {
                /* descriptors by adding to the address field (no carry out of it:
                 * shared memory is below 2^18 bytes) */
                const uint32_t one = bamf::tc::elect_one();
#pragma unroll
                for (int hh = 0; hh < 2; ++hh)
#pragma unroll
                    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
                        for (int cb = 0; cb < 2; ++cb)
                            bamf::tc::mma_bf16_warp(
                                tin + 32 * hh,
                                dk + (tap / 3 * BW_DCOL + 2 * cb * BW_DG + tap % 3 * 16 + 128 * hh) / 16,
                                wd + (tap * (CH * CH * 2) + 2 * cb * (CH * 16)) / 16, TC_IDESC, tap + cb > 0 ? 1u : 0u,
                                one);
                if (one) bamf::tc::commit(bar_in);
#pragma unroll
                for (int x = 0; x < S; ++x)
                    bamf::tc::mma_bf16_warp(tw, am + x * BW_ACOL / 16, dm + x * BW_DCOL / 16, DW_IDESC,
                                            first && x == 0 ? 0u : 1u, one);
                if (one) bamf::tc::commit(bar_w);
            }
            first = false;
            const int rn = r + gridDim.x;
            if (rn < n) load(l, rn);
            if (warp >= 4) bias_sums();
            bool ok = bamf::tc::mbar_wait(bar_in, phase, 1u << 24);
            bamf::tc::fence_after_sync();
            if (ok) {
                float v[32];
                bamf::tc::tmem_ld32(tin + 32 * h + tlane, v);
                uint4 *dst = (uint4 *)(out + ((size_t)r * NPX + 16 * ex + ey) * CH);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 mk = *(const uint4 *)(As + ex * BW_ACOL + (4 + q) * BW_AG + ey * 16);
                    const __nv_bfloat162 *m2 = (const __nv_bfloat162 *)&mk;
                    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        o[c] = __floats2bfloat162_rn(__bfloat162float(m2[c].x) > 0.0f ? v[8 * q + 2 * c] : 0.0f,
                                                     __bfloat162float(m2[c].y) > 0.0f ? v[8 * q + 2 * c + 1] : 0.0f);
                    dst[q] = *(const uint4 *)o;
                }
            }
            ok = bamf::tc::mbar_wait(bar_w, phase, 1u << 24) && ok;
            phase ^= 1u;
            bamf::tc::fence_after_sync();
            if (!ok) {
                atomicExch(status, 1);
                alive = false;
            }
            bamf::tc::fence_before_sync();
            /* the MMAs and the epilogue have read the tiles before they are restaged */
            alive = __syncthreads_and(alive);
            bamf::tc::fence_after_sync();
            if (alive && rn < n) stage();
        }
        /* every MMA of the layer is done and every row of dz written: the next layer's
         * first ROI and weights, and this one's sums */
        if (l > 0) {
            load(l - 1, r0);
            if (alive) loaded = l - 1;
            if (alive && t == 0) bamf::tc::bulk_load(smem_raw, bw.Wb + (l - 1) * PKT, PKT * 2, bar_wt);
        }
        {
            float *mine = bw.part + l * bw.pitch + (size_t)blockIdx.x * DW_PART;
            if ((warp & 3) < 3) {
                /* lane 32 ky + ci, column 32 j + co, stored at (32 j + co) * 96 + 32 ky + ci */
#pragma unroll 1
                for (int j = h; j < 3; j += 2) {
                    float v[32];
                    if (alive) {
                        bamf::tc::tmem_ld32(tw + 32 * j + tlane, v);
                    } else {
#pragma unroll
                        for (int co = 0; co < CH; ++co) v[co] = 0.0f;
                    }
#pragma unroll
                    for (int co = 0; co < CH; ++co) mine[(32 * j + co) * 96 + m] = v[co];
                }
            }
            /* bias: lanes with equal (lane >> 3) hold the same 8 channels */
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                float v = bsum[c];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                v += __shfl_xor_sync(0xffffffffu, v, 4);
                bsum[c] = v;
            }
            if (warp >= 4 && (t & 7) == 0)
#pragma unroll
                for (int c = 0; c < 8; ++c) bred[warp - 4][8 * g + c] = bsum[c];
            __syncthreads();
            if (t < CH) mine[96 * 96 + t] = alive ? (bred[0][t] + bred[1][t]) + (bred[2][t] + bred[3][t]) : 0.0f;
        }
    }
    if (!alive) {
        bamf::tc::mbar_wait(bar_wt, loaded & 1, 1u << 24);
        bamf::tc::mbar_wait(bar_in, phase ^ 1u, 1u << 24);
        bamf::tc::mbar_wait(bar_w, phase ^ 1u, 1u << 24);
    }
    bamf::tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) bamf::tc::tmem_dealloc(tw, BW_TMEM);
}

/* Column sums of a row-major [nrows][width] array of partial sums, in a
 * fixed order (no atomics: the same bits every run).  A CTA of 8 warps owns 32
 * consecutive columns (lane = column, coalesced) and adds 32 strands of rows, w,
 * w + 32, ... into four interleaved accumulators each, four strands per warp (so
 * that 16 loads are in flight and every CTA of a step is resident at once); then
 * warp 0 adds the 32 sums in order.  The result is valid in warp 0. */
constexpr int RED_THREADS = 256;
__device__ __forceinline__ float column_sum(const float *__restrict__ part, int nrows, int width, int j,
                                            float (*red)[33])
{
    constexpr int RW = RED_THREADS / 32, SV = 32 / RW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float a[SV][4];
#pragma unroll
    for (int v = 0; v < SV; ++v)
#pragma unroll
        for (int k = 0; k < 4; ++k) a[v][k] = 0.0f;
    if (j < width) {
        const float *p = part + j;
        int base = 0;
        for (; base + 128 <= nrows; base += 128)
#pragma unroll
            for (int v = 0; v < SV; ++v)
#pragma unroll
                for (int k = 0; k < 4; ++k) a[v][k] += p[(size_t)(base + warp + RW * v + 32 * k) * width];
        if (base < nrows) {
            float f[SV][4];
#pragma unroll
            for (int v = 0; v < SV; ++v)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int c = base + warp + RW * v + 32 * k;
                    f[v][k] = c < nrows ? p[(size_t)c * width] : 0.0f;
                }
#pragma unroll
            for (int v = 0; v < SV; ++v) {
                const bool whole = base + warp + RW * v + 96 < nrows;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    a[v][k] += whole || k == 0 ? f[v][k] : 0.0f;
                    if (k > 0) a[v][0] += whole ? 0.0f : f[v][k];
                }
            }
        }
    }
#pragma unroll
    for (int v = 0; v < SV; ++v) red[warp + RW * v][lane] = (a[v][0] + a[v][1]) + (a[v][2] + a[v][3]);
    __syncthreads();
    float sum = 0.0f;
    if (warp == 0)
#pragma unroll
        for (int k = 0; k < 32; ++k) sum += red[k][lane];
    return sum;
}

/* The backward kernels' partial sums, and what a training step does with them. */
struct Partials {
    const float *head; /* [nhead][HEAD_NPARAM] */
    const float *c1;   /* [nc1][C1_NPARAM] */
    const float *dw;   /* three layers of [ndw][DW_PART], layer l at l * dw_pitch */
    size_t dw_pitch;
    int nhead, nc1, ndw;
};
struct Optimiser {
    float *P, *m, *v;
    bf16 *Wf, *Wb;
    int *step;      /* the step being taken; incremented by the last CTA */
    unsigned *done; /* CTAs that have finished; left at zero */
    int steps_total;
    float lr0;
};
/* CTAs of 32 columns: the head's first (their rows, one per ROI, take longest) */
constexpr int RB_HEAD = (HEAD_NPARAM + 31) / 32, RB_C1 = (C1_NPARAM + 31) / 32, RB_DW = (DW_PART + 31) / 32;
constexpr int RB_ALL = RB_HEAD + RB_C1 + 3 * RB_DW;

/* Every parameter's gradient from the partial sums, in one launch.  ADAM: the
 * parameter's Adam update and its BF16 copies for the tensor cores at once;
 * else grad[j] = the sum.  Bound by latency: of the 34 MB of partial sums (in
 * L2) the longest chain is a warp's n / 32 rows.  A step of 1024 ROIs ran five
 * reductions, Adam, the packing and the step count as eight launches, 50 us;
 * this one takes 13 (28 with a strand per warp of 1024 threads, 19 with two). */
template <bool ADAM>
__global__ void __launch_bounds__(RED_THREADS) reduce_kernel(Partials pt, float *__restrict__ grad, Optimiser opt)
{
    __shared__ float red[32][33];
    const int lane = threadIdx.x & 31;
    int b = blockIdx.x, l = 0, nrows, width;
    const float *part;
    if (b < RB_HEAD) {
        part = pt.head, nrows = pt.nhead, width = HEAD_NPARAM;
    } else if (b < RB_HEAD + RB_C1) {
        b -= RB_HEAD;
        part = pt.c1, nrows = pt.nc1, width = C1_NPARAM;
    } else {
        b -= RB_HEAD + RB_C1;
        l = b / RB_DW;
        b -= l * RB_DW;
        part = pt.dw + l * pt.dw_pitch, nrows = pt.ndw, width = DW_PART;
    }
    const int j = b * 32 + lane;
    const bool mine = threadIdx.x < 32 && j < width;
    /* the parameter, and a convolution weight's place in the packed operands */
    int i, of = -1, ob = -1;
    if (width == HEAD_NPARAM) {
        i = O_WL + j;
    } else if (width == C1_NPARAM) {
        i = O_W1 + j;
    } else if (j < 96 * 96) {
        /* column 32 (2 - kx) + co, row 32 ky + ci of conv_bwd_kernel's D */
        const int col = j / 96, row = j - col * 96;
        const int kx = 2 - (col >> 5), co = col & 31, ky = row >> 5, ci = row & 31, tap = 3 * kx + ky;
        i = (l == 0 ? O_W2 : l == 1 ? O_W3 : O_W4) + (co * CH + ci) * 9 + tap;
        of = l * PKT + tap * (CH * CH) + (ci >> 3) * (CH * 8) + co * 8 + (ci & 7);
        ob = l * PKT + (8 - tap) * (CH * CH) + (co >> 3) * (CH * 8) + ci * 8 + (co & 7);
    } else {
        i = (l == 0 ? O_B2 : l == 1 ? O_B3 : O_B4) + j - 96 * 96;
    }
    /* Adam's inputs, loaded while the sums run */
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float p = 0.0f, m = 0.0f, v = 0.0f, lr = 0.0f, c1 = 0.0f, c2 = 0.0f;
    int step = 0;
    if (ADAM) {
        step = *opt.step;
        if (mine) {
            p = opt.P[i];
            m = opt.m[i];
            v = opt.v[i];
            const float frac = opt.steps_total > 1 ? (float)step / (float)(opt.steps_total - 1) : 0.0f;
            lr = opt.lr0 * (1.0f - 0.9f * fminf(frac, 1.0f));
            const float t = (float)(step + 1);
            c1 = 1.0f - powf(b1, t);
            c2 = 1.0f - powf(b2, t);
        }
    }
    const float g = column_sum(part, nrows, width, j, red);
    if (mine) {
        if (ADAM) {
            const float mi = b1 * m + (1.0f - b1) * g;
            const float vi = b2 * v + (1.0f - b2) * g * g;
            opt.m[i] = mi;
            opt.v[i] = vi;
            const float mh = mi / c1, vh = vi / c2;
            p -= lr * mh / (sqrtf(vh) + eps);
            opt.P[i] = p;
            if (of >= 0) {
                opt.Wf[of] = __float2bfloat16_rn(p);
                opt.Wb[ob] = __float2bfloat16_rn(p);
            }
        } else {
            grad[i] = g;
        }
    }
    if (ADAM && threadIdx.x == 0) {
        /* every CTA has read *step before it counts itself */
        __threadfence();
        if (atomicAdd(opt.done, 1u) == gridDim.x - 1) {
            *opt.done = 0;
            *opt.step = step + 1;
        }
    }
}

/* ----------------------------------------------------------------- heads */
/* Training: one CTA of 128 threads per ROI: loss, head gradients (row r of
 * `hrows`, HEAD_NPARAM floats per ROI: WL, BL, WC, BC), dz4 = dL/d(pre-activation of
 * conv4).  Three products of 131072 FP32 multiply-adds a ROI; as a 16-byte
 * shared-memory load takes 4 cycles of the SM whether or not its lanes share
 * addresses, their tiles are 4 pixels x 8 sub-cells (loc), 4 pixels x 16 channels
 * (dz4) and, a quarter of the pixels per warp, 4 sub-cells x 4 channels (dWL) per
 * thread, with a4 kept in BF16.  Bound by
 * issue (27,000 warp instructions a ROI, 12,300 of them multiply-adds): 1024 ROIs
 * took 53 us with a pixel per thread, 42 with these tiles. */
constexpr int HD_THREADS = 128;
constexpr int HD_H = CH + 8;    /* bf16 per pixel row of H, floats per pixel row of D: */
constexpr int HD_D = NSUB + 4;  /* 80 bytes, 8 rows in distinct banks */
__device__ __forceinline__ float bf_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf_hi(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }

__global__ void __launch_bounds__(HD_THREADS, 5) head_kernel(const bf16 *__restrict__ a4, int n,
                                                             const float *__restrict__ P,
                                                             const int32_t *__restrict__ n_em,
                                                             const float *__restrict__ xyi, float inv_batch,
                                                             float *__restrict__ hrows, bf16 *__restrict__ dz4,
                                                             float *__restrict__ loss_buf,
                                                             const int *__restrict__ step_dev)
{
    __shared__ __align__(16) bf16 H[NPX * HD_H];
    __shared__ __align__(16) float D[NPX * HD_D]; /* loc, then dL/dloc */
    __shared__ __align__(16) float Wl[NSUB * CH];
    __shared__ __align__(16) float dg[CH];
    __shared__ float bl[NSUB], Wc[NC * CH], bc[NC];
    __shared__ float part[8][CH], gmean[CH], dzc[NC], red[8], wmax[4];
    __shared__ float ex[BAMF_SYNTH_NMAX], ey[BAMF_SYNTH_NMAX];
    __shared__ float lcnt_sh, lsum[4];
    const int r = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < NPX * 4; i += HD_THREADS)
        *(uint4 *)(H + (i >> 2) * HD_H + (i & 3) * 8) = ((const uint4 *)(a4 + (size_t)r * NPX * CH))[i];
    ((float4 *)Wl)[t] = make_float4(P[O_WL + 4 * t], P[O_WL + 4 * t + 1], P[O_WL + 4 * t + 2], P[O_WL + 4 * t + 3]);
    for (int i = t; i < NC * CH; i += HD_THREADS) Wc[i] = P[O_WC + i];
    if (t < NSUB) bl[t] = P[O_BL + t];
    if (t < NC) bc[t] = P[O_BC + t];
    if (t < BAMF_SYNTH_NMAX) {
        ex[t] = xyi[((size_t)r * BAMF_SYNTH_NMAX + t) * 3 + 0];
        ey[t] = xyi[((size_t)r * BAMF_SYNTH_NMAX + t) * 3 + 1];
    }
    const int ntrue = n_em[r];
    __syncthreads();
    { /* loc = Wl a4 + bl */
        const int s0 = 8 * (lane >> 4), q0 = 64 * warp + (lane & 15); /* pixels q0 + 16 j */
        float z[4][8];
#pragma unroll
        for (int s = 0; s < 8; ++s)
#pragma unroll
            for (int j = 0; j < 4; ++j) z[j][s] = bl[s0 + s];
#pragma unroll 1
        for (int c8 = 0; c8 < CH; c8 += 8) {
            uint4 u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = *(const uint4 *)(H + (q0 + 16 * j) * HD_H + c8);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float hv[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t a = hf ? u[j].z : u[j].x, b = hf ? u[j].w : u[j].y;
                    hv[j][0] = bf_lo(a);
                    hv[j][1] = bf_hi(a);
                    hv[j][2] = bf_lo(b);
                    hv[j][3] = bf_hi(b);
                }
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const float4 w = *(const float4 *)(Wl + (s0 + s) * CH + c8 + 4 * hf);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        z[j][s] += w.x * hv[j][0];
                        z[j][s] += w.y * hv[j][1];
                        z[j][s] += w.z * hv[j][2];
                        z[j][s] += w.w * hv[j][3];
                    }
                }
            }
        }
        float mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float4 *row = (float4 *)(D + (q0 + 16 * j) * HD_D + s0);
            row[0] = make_float4(z[j][0], z[j][1], z[j][2], z[j][3]);
            row[1] = make_float4(z[j][4], z[j][5], z[j][6], z[j][7]);
#pragma unroll
            for (int s = 0; s < 8; ++s) mx = fmaxf(mx, z[j][s]);
        }
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) wmax[warp] = mx;
    }
    /* count head: mean of a4 over pixels (channel lane, pixels k, k + 8, ...) */
#pragma unroll
    for (int k = warp; k < 8; k += 4) {
        float sacc = 0.0f;
#pragma unroll 8
        for (int p = k; p < NPX; p += 8) sacc += __bfloat162float(H[p * HD_H + lane]);
        part[k][lane] = sacc;
    }
    __syncthreads();
    const float mx = fmaxf(fmaxf(wmax[0], wmax[1]), fmaxf(wmax[2], wmax[3]));
    /* softmax over all sub-cells: thread = pixels t and t + 128 */
    float e[2][NSUB];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float se = 0.0f;
#pragma unroll
        for (int q = 0; q < NSUB / 4; ++q) {
            const float4 z = *(const float4 *)(D + (t + 128 * j) * HD_D + 4 * q);
            e[j][4 * q] = expf(z.x - mx);
            e[j][4 * q + 1] = expf(z.y - mx);
            e[j][4 * q + 2] = expf(z.z - mx);
            e[j][4 * q + 3] = expf(z.w - mx);
#pragma unroll
            for (int k = 0; k < 4; ++k) se += e[j][4 * q + k];
        }
        for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
        if (lane == 0) red[warp + 4 * j] = se;
    }
    if (warp == 3) { /* count head: logits, loss, gradients */
        float g = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) g += part[k][lane];
        gmean[lane] = g * (1.0f / NPX);
        __syncwarp();
        float zc = -INFINITY;
        if (lane < NC) {
            zc = bc[lane];
            for (int c = 0; c < CH; ++c) zc += Wc[lane * CH + c] * gmean[c];
        }
        float m = zc;
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const float ec = lane < NC ? expf(zc - m) : 0.0f;
        float sacc = 0.0f;
#pragma unroll
        for (int c = 0; c < NC; ++c) sacc += __shfl_sync(0xffffffffu, ec, c);
        const int cls = min(ntrue, NC - 1);
        if (lane == cls) lcnt_sh = -(zc - m - logf(sacc));
        if (lane < NC) dzc[lane] = (ec / sacc - (lane == cls ? 1.0f : 0.0f)) * inv_batch;
        __syncwarp();
        float v = 0.0f;
        for (int c = 0; c < NC; ++c) v += Wc[c * CH + lane] * dzc[c];
        dg[lane] = v * (1.0f / NPX);
    }
    __syncthreads();
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += red[k];
    const float inv_sum = 1.0f / sum, logS = logf(sum) + mx;
    /* targets, loss, dL/dloc */
    int nin = 0;
    uint64_t tg[2][2] = {{0, 0}, {0, 0}}; /* emitters per sub-cell of the two pixels, 8 bits each */
    for (int k = 0; k < ntrue; ++k) {
        const float X = ex[k], Y = ey[k];
        if (!(X >= 0.0f && X < (float)S && Y >= 0.0f && Y < (float)S)) continue;
        nin++;
        const int cx = min((int)X, S - 1), cy = min((int)Y, S - 1), p = cx * S + cy;
        const int s = min((int)((Y - (float)cy) * 4.0f), 3) + 4 * min((int)((X - (float)cx) * 4.0f), 3);
        const uint64_t one = 1ull << (8 * (s & 7));
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (p == t + 128 * j) {
                tg[j][0] += s < 8 ? one : 0;
                tg[j][1] += s < 8 ? 0 : one;
            }
    }
    const float wloc = nin > 0 ? 1.0f / (float)nin : 0.0f, scale = nin > 0 ? inv_batch : 0.0f;
    float lloc[2] = {0.0f, 0.0f};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        float *row = D + (t + 128 * j) * HD_D;
        if (tg[j][0] | tg[j][1]) {
#pragma unroll
            for (int s = 0; s < NSUB; ++s) {
                const float tgt = (float)(uint32_t)(tg[j][s >> 3] >> (8 * (s & 7)) & 255u);
                if (tgt > 0.0f) lloc[j] -= tgt * wloc * (row[s] - logS);
                e[j][s] = (e[j][s] * inv_sum - tgt * wloc) * scale;
            }
        } else {
#pragma unroll
            for (int s = 0; s < NSUB; ++s) e[j][s] = e[j][s] * inv_sum * scale;
        }
#pragma unroll
        for (int q = 0; q < NSUB / 4; ++q)
            *(float4 *)(row + 4 * q) = make_float4(e[j][4 * q], e[j][4 * q + 1], e[j][4 * q + 2], e[j][4 * q + 3]);
    }
    {
        float l = lloc[0] + lloc[1];
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) lsum[warp] = l;
    }
    __syncthreads();
    if (t == 0)
        atomicAdd(&loss_buf[*step_dev], (((lsum[0] + lsum[1]) + (lsum[2] + lsum[3])) + lcnt_sh) * inv_batch);
    { /* dz4: pixels q0 + 16 j, channels c0 .. c0 + 15 */
        const int c0 = 16 * (lane & 1), q0 = 64 * warp + (lane >> 1);
        float v[4][16];
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
            const float4 b = *(const float4 *)(dg + c0 + c);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j][c] = b.x;
                v[j][c + 1] = b.y;
                v[j][c + 2] = b.z;
                v[j][c + 3] = b.w;
            }
        }
#pragma unroll 1
        for (int k4 = 0; k4 < NSUB; k4 += 4) {
            float d[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) *(float4 *)d[j] = *(const float4 *)(D + (q0 + 16 * j) * HD_D + k4);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int c = 0; c < 16; c += 4) {
                    const float4 w = *(const float4 *)(Wl + (k4 + k) * CH + c0 + c);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        v[j][c] += d[j][k] * w.x;
                        v[j][c + 1] += d[j][k] * w.y;
                        v[j][c + 2] += d[j][k] * w.z;
                        v[j][c + 3] += d[j][k] * w.w;
                    }
                }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int p = q0 + 16 * j;
            uint4 *dst = (uint4 *)(dz4 + ((size_t)r * NPX + p) * CH + c0);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const uint4 u = *(const uint4 *)(H + p * HD_H + c0 + 8 * hf);
                const uint32_t hw[4] = {u.x, u.y, u.z, u.w};
                __align__(16) __nv_bfloat162 o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    o[k] = __floats2bfloat162_rn(bf_lo(hw[k]) > 0.0f ? v[j][8 * hf + 2 * k] : 0.0f,
                                                 bf_hi(hw[k]) > 0.0f ? v[j][8 * hf + 2 * k + 1] : 0.0f);
                dst[hf] = *(const uint4 *)o;
            }
        }
    }
    /* dWL[s][c] = sum over pixels of D[p][s] H[p][c] and dBL[s] = sum of D[p][s]: warp
     * w adds the pixels 64 w .. 64 w + 63, lane the 4 x 4 block (s0, c0); the four
     * warps' sums are added through shared memory (over D, once it has been read) */
    {
        const int s0 = 4 * (lane >> 3), c0 = 4 * (lane & 7);
        float g[4][4] = {}, gb[4] = {};
#pragma unroll 4
        for (int p = 64 * warp; p < 64 * warp + 64; ++p) {
            const uint2 u = *(const uint2 *)(H + p * HD_H + c0);
            const float4 d4 = *(const float4 *)(D + p * HD_D + s0);
            const float hv[4] = {bf_lo(u.x), bf_hi(u.x), bf_lo(u.y), bf_hi(u.y)}, d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                gb[a] += d[a];
#pragma unroll
                for (int k = 0; k < 4; ++k) g[a][k] += d[a] * hv[k];
            }
        }
        __syncthreads();
        constexpr int QW = NSUB * CH + NSUB; /* one warp's WL and BL sums */
        float *q = D + warp * QW;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            *(float4 *)(q + (s0 + a) * CH + c0) = make_float4(g[a][0], g[a][1], g[a][2], g[a][3]);
            if ((lane & 7) == 0) q[NSUB * CH + s0 + a] = gb[a];
        }
        __syncthreads();
        float *row = hrows + (size_t)r * HEAD_NPARAM;
        for (int o = t; o < QW; o += HD_THREADS) row[o] = (D[o] + D[QW + o]) + (D[2 * QW + o] + D[3 * QW + o]);
    }
    for (int o = t; o < NC * CH; o += HD_THREADS) row_wc(hrows, r)[o] = dzc[o / CH] * gmean[o - (o / CH) * CH];
    if (t < NC) row_wc(hrows, r)[NC * CH + t] = dzc[t];
}
static_assert(4 * (NSUB * CH + NSUB) <= NPX * HD_D && NSUB * CH == 4 * HD_THREADS && BAMF_SYNTH_NMAX <= HD_THREADS,
              "head_kernel's shared memory and loads");

/* ------------------------------------------------------ fused forward */
/* The whole network on a ROI without leaving the SM (NET_TRAIN: up to a4, the
 * activations also written out for the backward kernels, 1024 ROIs in 37 us
 * for 72 us of four kernels).  A persistent CTA keeps
 * the packed weights of the three convolutions resident and runs GROUPS groups
 * of 256 threads; a group takes one ROI per iteration: conv1 (FP32), three 32 ->
 * 32 convolutions and the 1x1 head on tcgen05, the birth tables written out.
 *
 * One activation buffer per group, [ci group g][padded x 0..17][padded y
 * 0..17][8 ci] BF16 with zero borders, serves every tap without shifted copies:
 * M tile `mt` is the ROI's half y in [8 mt, 8 mt + 8), its row m the pixel x = m
 * / 8, y = 8 mt + m mod 8, so a core matrix is 8 consecutive y of one x (128
 * contiguous bytes), the next one is one padded column away (SBO = 288), and
 * tap (kx, ky) starts (18 kx + ky) 16-byte rows in.  The epilogue of a layer
 * (bias, ReLU, BF16) writes the next layer's input over it once the layer's
 * MMAs completed.
 *
 * The 1x1 head keeps FP32 weights: each is the exact sum of three BF16 parts
 * (8 significant bits each), a4 is BF16, so loc = a4 Wl^T is three exact-product
 * GEMMs with FP32 accumulation, one MMA of N = 48 per 16 channels, whose
 * results are added smallest first.  On 50,000 ROIs the tables' error against
 * 64 bits (3.2e-3, from the BF16 activations) is the same as with FP32 FMAs.
 *
 * Bound: shared memory.  Each of the 108 convolution MMAs reads a 4 KB A tile
 * and 1 KB of weights for 32 columns, 40 cycles of the SM's 128 bytes/cycle;
 * a 16-byte broadcast load takes 4 of them, so conv1 gives a thread 4 pixels x
 * 8 channels (18 weight loads instead of 72 for one pixel x 32).  Four groups
 * on an SM (two CTAs of two) overlap one's MMAs with the others' epilogues.
 * 50,000 ROIs: 3.78 ms as five launches per 4096 ROIs, 1.93 ms with the heads in
 * FP32 FMAs and one thread building every descriptor, 1.53 with this conv1 and
 * head, 1.32 with the warp-uniform issue, 1.26 with GROUPS = 2 instead of 1, 1.24
 * with the weights as one bulk copy (304 CTAs reading the same lines with plain loads
 * waited some 6000 cycles);
 * 0.74 ms is 108 x 40 + 4 x 44 cycles per ROI and SM. */
constexpr int IB_G = PS * PS * 16;                 /* bytes of one ci group of the buffer */
constexpr int IB_BYTES = 4 * IB_G;
constexpr int INF_GROUPS = 2;
constexpr int IH_N = 3 * NSUB;                     /* head columns: three parts of 16 sub-cells */
constexpr int IH_BYTES = 4 * IH_N * 16;            /* [ci group][48][8 ci] */
/* byte offsets: convolution weights, head weights, conv1 weights [tap][co],
 * biases of conv1 .. conv4, then per group buffer, conv1 input, reductions */
constexpr int INF_WH = 3 * PKT * 2;
constexpr int INF_W1 = INF_WH + IH_BYTES;
constexpr int INF_BIAS = INF_W1 + 9 * CH * 4;
constexpr int INF_GRP = INF_BIAS + 4 * CH * 4;
struct alignas(16) InferGroup {
    unsigned char buf[IB_BYTES];
    float xp[PS * PS];
    float se[NPX];
    float part[8][CH];
    float gmean[CH], red[8], red2[8], red3[8];
    uint64_t mbar;
    int dead;
};
constexpr size_t SMEM_INFER = INF_GRP + INF_GROUPS * sizeof(InferGroup);
constexpr int INF_TMEM = 128; /* columns per group: 64 of a convolution, then 96 of the head over them */
constexpr uint32_t IH_IDESC = bamf::tc::idesc_bf16_f32(128, IH_N);
static_assert(INF_W1 % 16 == 0 && INF_GRP % 16 == 0, "shared-memory alignment");

/* two FP32 fused multiply-adds, each rounded as fmaf rounds it */
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

/* 32 bytes of one thread in one store: a whole L2 sector */
__device__ __forceinline__ void store8(float *p, const float *v)
{
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

__device__ __forceinline__ uint4 relu_bf16(const float (&v)[8])
{
    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = __floats2bfloat162_rn(fmaxf(v[2 * q], 0.0f), fmaxf(v[2 * q + 1], 0.0f));
    return *(const uint4 *)o;
}

/* what training keeps of a forward pass: x0 [roi][p], a1..a4 [roi][p][32] */
struct Kept {
    float *x0;
    bf16 *a[4];
};
enum NetMode { NET_INFER, NET_INFER_WIDE, NET_TRAIN }; /* WIDE: `sub` at a 32-byte boundary */

template <int MODE>
__global__ void __launch_bounds__(256 * INF_GROUPS, 2) net_kernel(
    const float *__restrict__ data, int n, const float *__restrict__ P, const bf16 *__restrict__ Wt,
    float *__restrict__ cdf, float *__restrict__ sub, float *__restrict__ cnt_out, Kept kept,
    int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *w1 = (float *)(smem_raw + INF_W1), *bias = (float *)(smem_raw + INF_BIAS);
    __shared__ uint32_t tslot;
    __shared__ uint64_t wbar; /* the packed weights' arrival */
    __shared__ float Wc[NC * CH], bc[NC], bl[NSUB];
    const int t = threadIdx.x % 256, lane = t & 31;
    /* warp-uniform, and known to be */
    const int wid = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), grp = wid >> 3, warp = wid & 7;
    InferGroup &G = ((InferGroup *)(smem_raw + INF_GRP))[grp];
    unsigned char *const buf = G.buf;
    if (threadIdx.x < 32) bamf::tc::tmem_alloc(&tslot, INF_TMEM * INF_GROUPS);
    if (threadIdx.x == 0) {
        bamf::tc::mbar_init(&wbar, 1);
        bamf::tc::bulk_load(smem_raw, Wt, 3 * PKT * 2, &wbar);
    }
    {
        const int nt = 256 * INF_GROUPS, i0 = threadIdx.x;
        for (int i = i0; i < (MODE == NET_TRAIN ? 0 : CH * NSUB); i += nt) {
            const int s = i / CH, c = i - s * CH;
            bf16 *w = (bf16 *)(smem_raw + INF_WH) + (c >> 3) * (IH_N * 8) + s * 8 + (c & 7);
            float v = P[O_WL + i];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const bf16 h = __float2bfloat16_rn(v);
                w[k * NSUB * 8] = h;
                v -= __bfloat162float(h); /* exact */
            }
        }
        for (int i = i0; i < 9 * CH; i += nt) w1[i] = P[O_W1 + (i % CH) * 9 + i / CH];
        for (int i = i0; i < 4 * CH; i += nt) {
            const int l = i / CH;
            bias[i] = P[(l == 0 ? O_B1 : l == 1 ? O_B2 : l == 2 ? O_B3 : O_B4) + i % CH];
        }
        if (MODE != NET_TRAIN) {
            for (int i = i0; i < NC * CH; i += nt) Wc[i] = P[O_WC + (i % NC) * CH + i / NC];
            if (i0 < NSUB) bl[i0] = P[O_BL + i0];
            if (i0 < NC) bc[i0] = P[O_BC + i0];
        }
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int i = t; i < IB_BYTES / 16; i += 256) ((uint4 *)buf)[i] = z;
        for (int i = t; i < PS * PS; i += 256) G.xp[i] = 0.0f;
    }
    if (t == 0) {
        bamf::tc::mbar_init(&G.mbar, 1);
        G.dead = 0;
    }
    bamf::tc::fence_before_sync();
    __syncthreads();
    bamf::tc::fence_after_sync();
    const auto group_sync = [&]() { asm volatile("barrier.sync %0, 256;" ::"r"(1 + grp) : "memory"); };
    const uint32_t tbase = __shfl_sync(0xffffffffu, tslot, 0) + INF_TMEM * grp;
    const uint64_t ad0 = bamf::tc::smem_desc(bamf::tc::smem_addr(buf), IB_G, PS * 16);
    const uint64_t bd0 = bamf::tc::smem_desc(bamf::tc::smem_addr(smem_raw), CH * 16, 128);
    const uint64_t hd0 = bamf::tc::smem_desc(bamf::tc::smem_addr(smem_raw) + INF_WH, IH_N * 16, 128);
    /* this thread's pixel in the convolutions' epilogues and the head (its TMEM
     * lane's), and that pixel's 16-byte row of a ci group */
    const int mt = warp >> 2, m = 32 * (warp & 3) + lane;
    const int pe = 16 * (m >> 3) + 8 * mt + (m & 7);
    const int epi = ((pe >> 4) + 1) * PS + (pe & 15) + 1;
    const uint32_t tlane = tbase + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t phase = 0;
    /* a last round that not every group has is spread over the CTAs */
    const int stride = gridDim.x * INF_GROUPS, r0 = blockIdx.x + gridDim.x * grp;
    float next = r0 < n ? data[(size_t)r0 * NPX + t] : 0.0f;
    /* every thread of the group waits for the group's MMAs; false (for all)
     * when the wait ran out */
    const auto mma_done = [&]() {
        if (!bamf::tc::mbar_wait(&G.mbar, phase, 1u << 24)) {
            G.dead = 1;
            atomicExch(status, 1);
        }
        phase ^= 1u;
        bamf::tc::fence_after_sync();
    };
    const auto mma_ready = [&]() {
        bamf::tc::fence_proxy_async();
        bamf::tc::fence_before_sync();
        group_sync();
        bamf::tc::fence_after_sync();
    };
    for (int r = r0; r < n; r += stride) {
        /* conv1: the normalisation, thread = pixel */
        const float v = sqrtf(fmaxf(next, 0.0f) + 0.375f);
        if (r + stride < n) next = data[(size_t)(r + stride) * NPX + t];
        float s = v;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) G.red[warp] = s;
        group_sync();
        if (MODE == NET_TRAIN && G.dead) break; /* set before this barrier, seen by the whole group */
        float mean = 0.0f;
        for (int k = 0; k < 8; ++k) mean += G.red[k];
        mean *= (1.0f / NPX);
        const float xv = (v - mean) * 0.25f;
        G.xp[((t >> 4) + 1) * PS + (t & 15) + 1] = xv;
        if (MODE == NET_TRAIN) kept.x0[(size_t)r * NPX + t] = xv;
        group_sync();
        {
            /* this thread: channels 8 g .. 8 g + 7 of the pixels y = lane & 15,
             * x = x0 + 2 j */
            const int g = warp & 3, y = lane & 15, x0 = 8 * (warp >> 2) + (lane >> 4);
            float2 z[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 b = ((const float2 *)bias)[4 * g + q];
#pragma unroll
                for (int j = 0; j < 4; ++j) z[j][q] = b;
            }
            float in[9][3]; /* padded rows x0 .. x0 + 8 of columns y .. y + 2 */
#pragma unroll
            for (int k = 0; k < 9; ++k)
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) in[k][ky] = G.xp[(x0 + k) * PS + y + ky];
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {
                const float4 wa = ((const float4 *)w1)[tap * (CH / 4) + 2 * g];
                const float4 wb = ((const float4 *)w1)[tap * (CH / 4) + 2 * g + 1];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 x2 = make_float2(in[2 * j + tap / 3][tap % 3], in[2 * j + tap / 3][tap % 3]);
                    z[j][0] = fma2(make_float2(wa.x, wa.y), x2, z[j][0]);
                    z[j][1] = fma2(make_float2(wa.z, wa.w), x2, z[j][1]);
                    z[j][2] = fma2(make_float2(wb.x, wb.y), x2, z[j][2]);
                    z[j][3] = fma2(make_float2(wb.z, wb.w), x2, z[j][3]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float o[8] = {z[j][0].x, z[j][0].y, z[j][1].x, z[j][1].y,
                                    z[j][2].x, z[j][2].y, z[j][3].x, z[j][3].y};
                const uint4 u = relu_bf16(o);
                *(uint4 *)(buf + g * IB_G + ((x0 + 2 * j + 1) * PS + y + 1) * 16) = u;
                if (MODE == NET_TRAIN)
                    ((uint4 *)kept.a[0])[((size_t)r * NPX + (x0 + 2 * j) * S + y) * 4 + g] = u;
            }
        }
        if (r == r0 && !bamf::tc::mbar_wait(&wbar, 0, 1u << 24)) {
            G.dead = 1;
            atomicExch(status, 1);
        }
#pragma unroll 1
        for (int l = 0; l < 3; ++l) {
            mma_ready();
            if (warp == 0) {
                /* descriptors by adding to the first one's address field (no
                 * carry out of it: shared memory is below 2^18 bytes) */
                const uint64_t bd = bd0 + (uint32_t)l * (PKT * 2 / 16);
                const uint32_t one = bamf::tc::elect_one();
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
                        for (int cb = 0; cb < 2; ++cb)
                            bamf::tc::mma_bf16_warp(
                                tbase + 32 * h, ad0 + (2 * cb * IB_G + (tap / 3 * PS + tap % 3 + 8 * h) * 16) / 16,
                                bd + (tap * (CH * CH * 2) + 2 * cb * (CH * 16)) / 16, TC_IDESC, tap + cb > 0 ? 1u : 0u,
                                one);
                if (one) bamf::tc::commit(&G.mbar);
            }
            mma_done();
            float d[32];
            bamf::tc::tmem_ld32(tlane + 32 * mt, d);
            uint4 *keep = MODE == NET_TRAIN
                              ? (uint4 *)(l == 0 ? kept.a[1] : l == 1 ? kept.a[2] : kept.a[3]) + ((size_t)r * NPX + pe) * 4
                              : nullptr;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float4 ba = ((const float4 *)bias)[(l + 1) * (CH / 4) + 2 * g];
                const float4 bb = ((const float4 *)bias)[(l + 1) * (CH / 4) + 2 * g + 1];
                const float o[8] = {d[8 * g] + ba.x,     d[8 * g + 1] + ba.y, d[8 * g + 2] + ba.z, d[8 * g + 3] + ba.w,
                                    d[8 * g + 4] + bb.x, d[8 * g + 5] + bb.y, d[8 * g + 6] + bb.z, d[8 * g + 7] + bb.w};
                const uint4 u = relu_bf16(o);
                if (MODE != NET_TRAIN || l < 2) *(uint4 *)(buf + g * IB_G + epi * 16) = u;
                if (MODE == NET_TRAIN) keep[g] = u;
            }
        }
        if (MODE == NET_TRAIN) continue;
        mma_ready();
        if (warp == 0) {
            const uint32_t one = bamf::tc::elect_one();
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int cb = 0; cb < 2; ++cb)
                    bamf::tc::mma_bf16_warp(tbase + IH_N * h, ad0 + (2 * cb * IB_G + (PS + 1 + 8 * h) * 16) / 16,
                                            hd0 + 2 * cb * IH_N, IH_IDESC, (uint32_t)cb, one);
            if (one) bamf::tc::commit(&G.mbar);
        }
        if (cnt_out) { /* mean of a4 over pixels: channel lane, pixels warp, warp + 8, ... */
            const bf16 *hc = (const bf16 *)(buf + (lane >> 3) * IB_G) + (lane & 7);
            float sacc = 0.0f;
#pragma unroll
            for (int p = warp; p < NPX; p += 8) sacc += __bfloat162float(hc[(((p >> 4) + 1) * PS + (p & 15) + 1) * 8]);
            G.part[warp][lane] = sacc;
        }
        mma_done();
        float e[NSUB];
        {
            float d[32], d3[16];
            bamf::tc::tmem_ld32(tlane + IH_N * mt, d);
            bamf::tc::tmem_ld16(tlane + IH_N * mt + 32, d3);
#pragma unroll
            for (int k = 0; k < NSUB; ++k) e[k] = ((d3[k] + d[16 + k]) + d[k]) + bl[k];
        }
        float mx = -INFINITY;
#pragma unroll
        for (int k = 0; k < NSUB; ++k) mx = fmaxf(mx, e[k]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) G.red[warp] = mx;
        group_sync();
        if (G.dead) break; /* set before this barrier, seen by the whole group */
        mx = G.red[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) mx = fmaxf(mx, G.red[k]);
        if (cnt_out && t < CH) {
            float sacc = 0.0f;
            for (int k = 0; k < 8; ++k) sacc += G.part[k][t];
            G.gmean[t] = sacc * (1.0f / NPX);
        }
        float se = 0.0f;
#pragma unroll
        for (int k = 0; k < NSUB; ++k) {
            e[k] = expf(e[k] - mx);
            se += e[k];
        }
        G.se[pe] = se;
        const float inv_se = 1.0f / se;
#pragma unroll
        for (int k = 0; k < NSUB; ++k) e[k] *= inv_se;
        float *dst = sub + ((size_t)r * NPX + pe) * NSUB;
        if (MODE == NET_INFER_WIDE) {
            store8(dst, e);
            store8(dst + 8, e + 8);
        } else {
#pragma unroll
            for (int k = 0; k < NSUB; ++k) dst[k] = e[k];
        }
        group_sync();
        /* the running sum over pixels, thread = pixel */
        se = G.se[t];
        float tot = se;
        for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (lane == 0) G.red2[warp] = tot;
        group_sync();
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; ++k) sum += G.red2[k];
        float incl = se * (1.0f / sum);
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) G.red3[warp] = incl;
        group_sync();
        float base = 0.0f;
        for (int k = 0; k < warp; ++k) base += G.red3[k];
        cdf[(size_t)r * NPX + t] = base + incl;
        if (cnt_out && warp == 7 && lane < NC) {
            float c = bc[lane];
#pragma unroll
            for (int k = 0; k < CH; ++k) c += Wc[k * NC + lane] * G.gmean[k];
            cnt_out[(size_t)r * NC + lane] = c;
        }
    }
    if (G.dead) { /* a wait ran out: once more for what the group has started */
        bamf::tc::mbar_wait(&wbar, 0, 1u << 24);
        bamf::tc::mbar_wait(&G.mbar, phase ^ 1u, 1u << 24);
    }
    bamf::tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) bamf::tc::tmem_dealloc(tslot, INF_TMEM * INF_GROUPS);
}

/* --------------------------------------------------------- start states */
/* A chain start per ROI from the network: n0 = argmax of the count logits
 * (at most max_n), positions = the n0 most probable sub-cells, greedily,
 * each suppressing the cells within 1 px of it; intensity `intensity`.
 * One CTA (256 threads, thread = pixel) per ROI. */
__global__ void __launch_bounds__(256) init_kernel(const float *__restrict__ cdf, const float *__restrict__ sub,
                                                   const float *__restrict__ cnt, int n, float intensity,
                                                   int max_n, int32_t *__restrict__ init_n,
                                                   float *__restrict__ init_ixy)
{
    __shared__ float bv[8];
    __shared__ int bi[8];
    __shared__ int win;
    const int r = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (r >= n) return;
    int n0 = 0;
    {
        const float *c = cnt + (size_t)r * NC;
        float m = c[0];
        for (int k = 1; k < NC; ++k)
            if (c[k] > m) {
                m = c[k];
                n0 = k;
            }
        n0 = min(n0, max_n);
    }
    const float pp = cdf[(size_t)r * NPX + t] - (t > 0 ? cdf[(size_t)r * NPX + t - 1] : 0.0f);
    float pr[NSUB];
    for (int s = 0; s < NSUB; ++s) pr[s] = pp * sub[((size_t)r * NPX + t) * NSUB + s];
    const int px = t / S, py = t - (t / S) * S;
    float *ixy = init_ixy + (size_t)r * 3 * BAMF_NMAX;
    for (int k = 0; k < n0; ++k) {
        float v = -1.0f;
        int idx = 0;
        for (int s = 0; s < NSUB; ++s)
            if (pr[s] > v) {
                v = pr[s];
                idx = t * NSUB + s;
            }
        for (int o = 16; o > 0; o >>= 1) {
            float ov = __shfl_xor_sync(0xffffffffu, v, o);
            int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) {
                v = ov;
                idx = oi;
            }
        }
        if (lane == 0) {
            bv[warp] = v;
            bi[warp] = idx;
        }
        __syncthreads();
        if (t == 0) {
            float m = bv[0];
            int w = bi[0];
            for (int q = 1; q < 8; ++q)
                if (bv[q] > m || (bv[q] == m && bi[q] < w)) {
                    m = bv[q];
                    w = bi[q];
                }
            win = w;
        }
        __syncthreads();
        const int wp = win / NSUB, ws = win - (win / NSUB) * NSUB;
        const float wx = (float)(wp / S) + ((float)(ws >> 2) + 0.5f) * 0.25f;
        const float wy = (float)(wp - (wp / S) * S) + ((float)(ws & 3) + 0.5f) * 0.25f;
        if (t == 0) {
            ixy[k] = intensity;
            ixy[BAMF_NMAX + k] = wx;
            ixy[2 * BAMF_NMAX + k] = wy;
        }
        for (int s = 0; s < NSUB; ++s) {
            float cx = (float)px + ((float)(s >> 2) + 0.5f) * 0.25f, cy = (float)py + ((float)(s & 3) + 0.5f) * 0.25f;
            if ((cx - wx) * (cx - wx) + (cy - wy) * (cy - wy) < 1.0f) pr[s] = 0.0f;
        }
        __syncthreads();
    }
    if (t == 0) init_n[r] = n0;
}

/* ---------------------------------------------------- training examples */
/* Training batch `step` from caller-provided examples: ROI b of the batch is
 * example (step * batch + b) mod n_examples; counts clipped to the target
 * capacity.  One CTA of NPX threads per ROI. */
__global__ void gather_examples_kernel(const float *__restrict__ data, const int32_t *__restrict__ n_em,
                                       const float *__restrict__ xyi, int n_examples, const int *step_dev,
                                       int batch, float *__restrict__ gdata, int32_t *__restrict__ gn,
                                       float *__restrict__ gxyi)
{
    const int b = blockIdx.x, t = threadIdx.x;
    const int64_t k = ((int64_t)(*step_dev) * batch + b) % n_examples;
    gdata[(size_t)b * NPX + t] = data[(size_t)k * NPX + t];
    if (t == 0) gn[b] = min(max(n_em[k], 0), BAMF_SYNTH_NMAX);
    if (t < BAMF_SYNTH_NMAX * 3) gxyi[(size_t)b * BAMF_SYNTH_NMAX * 3 + t] = xyi[(size_t)k * BAMF_SYNTH_NMAX * 3 + t];
}

}  // namespace

/* ================================================================ host */
struct bamf_cnn {
    float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;
    bf16 *Wf = nullptr, *Wb = nullptr;
    /* batch buffers (MAX_BATCH) */
    float *x0 = nullptr;
    bf16 *a[4] = {nullptr, nullptr, nullptr, nullptr};
    bf16 *dzA = nullptr, *dzB = nullptr;
    float *gdata = nullptr, *gxyi = nullptr;
    int32_t *gn = nullptr;
    int *step = nullptr;
    unsigned *done = nullptr; /* reduce_kernel's count of finished CTAs */
    int *tc_status = nullptr; /* set by a convolution whose tensor-core wait timed out */
    float *dwpart = nullptr;  /* per-CTA partial weight gradients, three layers, 2 CTAs per SM */
    float *hpart = nullptr;   /* per-ROI head gradients (MAX_BATCH rows) */
    float *c1part = nullptr;  /* per-CTA conv1 gradients, 4 CTAs per SM */
    float *loss = nullptr;
    int loss_cap = 0;
    int sms = 1;
    bool packed = false;
};

namespace {

std::mutex g_attr_mutex;
bool g_attr_done = false;

cudaError_t set_attrs()
{
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    if (g_attr_done) return cudaSuccess;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(conv_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BW)))
        return e;
    for (const auto kernel : {net_kernel<NET_INFER>, net_kernel<NET_INFER_WIDE>, net_kernel<NET_TRAIN>})
        if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_INFER))) return e;
    g_attr_done = true;
    return cudaSuccess;
}

#define CK(x)                                                                                                    \
    do {                                                                                                         \
        cudaError_t e_ = (x);                                                                                    \
        if (e_ != cudaSuccess) {                                                                                 \
            cudaGetLastError();                                                                                  \
            return BAMF_ERR_CUDA;                                                                                \
        }                                                                                                        \
    } while (0)

int grid_for(int n, int per_sm, int sms) { return std::max(1, std::min(n, per_sm * sms)); }

/* CTAs of net_kernel: a ROI per group, two CTAs per SM */
int net_grid(int n, int sms) { return grid_for((n + INF_GROUPS - 1) / INF_GROUPS, 2, sms); }

/* forward of a batch of n <= capacity ROIs from data, activations kept */
bamf_status forward(bamf_cnn *net, const float *data, int n, cudaStream_t s)
{
    const Kept kept = {net->x0, {net->a[0], net->a[1], net->a[2], net->a[3]}};
    net_kernel<NET_TRAIN><<<net_grid(n, net->sms), 256 * INF_GROUPS, SMEM_INFER, s>>>(
        data, n, net->P, net->Wf, nullptr, nullptr, nullptr, kept, net->tc_status);
    CK(cudaGetLastError());
    return BAMF_OK;
}

/* loss and gradients' partial sums of the batch whose forward ran */
Partials backward(bamf_cnn *net, const int32_t *n_em, const float *xyi, int n, float inv_batch, cudaStream_t s)
{
    const Partials pt = {net->hpart, net->c1part, net->dwpart, (size_t)2 * net->sms * DW_PART,
                         n, grid_for(n, 4, net->sms), grid_for(n, 2, net->sms)};
    head_kernel<<<n, HD_THREADS, 0, s>>>(net->a[3], n, net->P, n_em, xyi, inv_batch, net->hpart, net->dzA, net->loss,
                                         net->step);
    const Backward bw = {{net->a[0], net->a[1], net->a[2]}, {net->dzA, net->dzB}, net->Wb, net->dwpart, pt.dw_pitch};
    conv_bwd_kernel<<<pt.ndw, BW_THREADS, SMEM_BW, s>>>(bw, n, net->tc_status);
    conv1_bwd_kernel<<<pt.nc1, 256, 0, s>>>(net->x0, net->dzB, n, net->c1part);
    return pt;
}

bamf_status pack(bamf_cnn *net, cudaStream_t s)
{
    pack_kernel<<<(3 * 9 * CH * CH + 255) / 256, 256, 0, s>>>(net->P, net->Wf, net->Wb);
    CK(cudaGetLastError());
    return BAMF_OK;
}

}  // namespace

extern "C" bamf_status bamf_synth_generate(const bamf_synth_params *sp, uint32_t seed, uint64_t first, int n,
                                           float *data, int32_t *n_em, float *xyi, void *stream)
{
    if (!sp || n < 0 || (n > 0 && (!data || !n_em || !xyi))) return BAMF_ERR_INVALID_ARG;
    if (!(sp->sigma > 0.0f) || !(sp->mean_n >= 0.0f) || !(sp->i_median > 0.0f) || !(sp->bg >= 0.0f))
        return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    synth_kernel<<<n, 256, 0, (cudaStream_t)stream>>>(*sp, seed, first, nullptr, 0, n, data, n_em, xyi);
    CK(cudaGetLastError());
    return BAMF_OK;
}

extern "C" void bamf_cnn_destroy(bamf_cnn *net)
{
    if (!net) return;
    void *ps[] = {net->P, net->G, net->M, net->V, net->Wf, net->Wb, net->x0, net->a[0], net->a[1], net->a[2],
                  net->a[3], net->dzA, net->dzB, net->gdata, net->gxyi, net->gn, net->step, net->loss,
                  net->tc_status, net->dwpart, net->hpart, net->c1part, net->done};
    for (void *p : ps)
        if (p) cudaFree(p);
    delete net;
}

extern "C" bamf_status bamf_cnn_create(bamf_cnn **out, uint32_t seed)
{
    if (!out) return BAMF_ERR_INVALID_ARG;
    *out = nullptr;
    if (bamf_device_count() < 1) return BAMF_ERR_NO_DEVICE;
    if (set_attrs() != cudaSuccess) return BAMF_ERR_CUDA;
    bamf_cnn *net = new bamf_cnn();
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&net->sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t B = MAX_BATCH;
    bool ok = cudaMalloc(&net->P, NPARAM * 4) == cudaSuccess && cudaMalloc(&net->G, NPARAM * 4) == cudaSuccess &&
              cudaMalloc(&net->M, NPARAM * 4) == cudaSuccess && cudaMalloc(&net->V, NPARAM * 4) == cudaSuccess &&
              cudaMalloc(&net->Wf, 3 * PKT * 2) == cudaSuccess && cudaMalloc(&net->Wb, 3 * PKT * 2) == cudaSuccess &&
              cudaMalloc(&net->tc_status, sizeof(int)) == cudaSuccess &&
              cudaMalloc(&net->dwpart, (size_t)3 * 2 * net->sms * DW_PART * 4) == cudaSuccess &&
              cudaMalloc(&net->hpart, B * HEAD_NPARAM * 4) == cudaSuccess &&
              cudaMalloc(&net->c1part, (size_t)4 * net->sms * C1_NPARAM * 4) == cudaSuccess &&
              cudaMalloc(&net->x0, B * NPX * 4) == cudaSuccess && cudaMalloc(&net->dzA, B * NPX * CH * 2) == cudaSuccess &&
              cudaMalloc(&net->dzB, B * NPX * CH * 2) == cudaSuccess &&
              cudaMalloc(&net->gdata, B * NPX * 4) == cudaSuccess &&
              cudaMalloc(&net->gxyi, B * BAMF_SYNTH_NMAX * 3 * 4) == cudaSuccess &&
              cudaMalloc(&net->gn, B * 4) == cudaSuccess && cudaMalloc(&net->step, sizeof(int)) == cudaSuccess &&
              cudaMalloc(&net->done, sizeof(unsigned)) == cudaSuccess;
    for (int l = 0; l < 4 && ok; ++l) ok = cudaMalloc(&net->a[l], B * NPX * CH * 2) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        bamf_cnn_destroy(net);
        return BAMF_ERR_CUDA;
    }
    /* He initialisation from a Philox stream (Box-Muller), zero biases */
    std::vector<float> h(NPARAM, 0.0f);
    uint32_t ctr = 0;
    auto normal = [&]() {
        bamf_philox_block b = bamf_philox4x32_10(ctr++, 0u, 0u, 0u, seed, 0x2545F491u);
        double u1 = ((double)(b.v[0] >> 8) + 0.5) / 16777216.0, u2 = ((double)(b.v[1] >> 8) + 0.5) / 16777216.0;
        return (float)(std::sqrt(-2.0 * std::log(u1)) * std::cos(2.0 * M_PI * u2));
    };
    auto fill = [&](int off, int count, int fan_in) {
        float sd = std::sqrt(2.0f / (float)fan_in);
        for (int i = 0; i < count; ++i) h[off + i] = sd * normal();
    };
    fill(O_W1, 288, 9);
    fill(O_W2, 9216, 288);
    fill(O_W3, 9216, 288);
    fill(O_W4, 9216, 288);
    fill(O_WL, 512, 32);
    fill(O_WC, 352, 32);
    bool ok2 = cudaMemcpy(net->P, h.data(), NPARAM * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
               cudaMemset(net->G, 0, NPARAM * 4) == cudaSuccess && cudaMemset(net->M, 0, NPARAM * 4) == cudaSuccess &&
               cudaMemset(net->V, 0, NPARAM * 4) == cudaSuccess && cudaMemset(net->step, 0, sizeof(int)) == cudaSuccess &&
               cudaMemset(net->done, 0, sizeof(unsigned)) == cudaSuccess &&
               cudaMemset(net->tc_status, 0, sizeof(int)) == cudaSuccess;
    if (!ok2 || pack(net, nullptr) != BAMF_OK || cudaDeviceSynchronize() != cudaSuccess) {
        cudaGetLastError();
        bamf_cnn_destroy(net);
        return BAMF_ERR_CUDA;
    }
    *out = net;
    return BAMF_OK;
}

extern "C" bamf_status bamf_cnn_get_params(bamf_cnn *net, float *params)
{
    if (!net || !params) return BAMF_ERR_INVALID_ARG;
    CK(cudaMemcpy(params, net->P, NPARAM * 4, cudaMemcpyDeviceToHost));
    return BAMF_OK;
}

extern "C" bamf_status bamf_cnn_set_params(bamf_cnn *net, const float *params)
{
    if (!net || !params) return BAMF_ERR_INVALID_ARG;
    CK(cudaMemcpy(net->P, params, NPARAM * 4, cudaMemcpyHostToDevice));
    bamf_status r = pack(net, nullptr);
    if (r) return r;
    CK(cudaDeviceSynchronize());
    return BAMF_OK;
}

/* after a synchronisation: a convolution whose tensor-core completion wait
 * ran out left garbage outputs; report it */
static bamf_status check_tc(bamf_cnn *net)
{
    int st = 0;
    CK(cudaMemcpy(&st, net->tc_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st) {
        cudaMemset(net->tc_status, 0, sizeof(int));
        return BAMF_ERR_CUDA;
    }
    return BAMF_OK;
}

static bamf_status ensure_loss(bamf_cnn *net, int cap)
{
    if (net->loss_cap >= cap) return BAMF_OK;
    if (net->loss) cudaFree(net->loss);
    net->loss = nullptr;
    net->loss_cap = 0;
    CK(cudaMalloc(&net->loss, (size_t)cap * sizeof(float)));
    net->loss_cap = cap;
    return BAMF_OK;
}

extern "C" bamf_status bamf_cnn_loss_grad(bamf_cnn *net, const float *data, const int32_t *n_em, const float *xyi,
                                          int n, float *loss, float *grad)
{
    if (!net || !data || !n_em || !xyi || n < 1 || n > MAX_BATCH) return BAMF_ERR_INVALID_ARG;
    bamf_status r;
    if ((r = ensure_loss(net, 1))) return r;
    int saved = 0;
    CK(cudaMemcpy(&saved, net->step, sizeof(int), cudaMemcpyDeviceToHost));
    CK(cudaMemset(net->step, 0, sizeof(int)));
    CK(cudaMemset(net->loss, 0, sizeof(float)));
    if ((r = forward(net, data, n, nullptr))) return r;
    const Partials pt = backward(net, n_em, xyi, n, 1.0f / (float)n, nullptr);
    reduce_kernel<false><<<RB_ALL, RED_THREADS>>>(pt, net->G, Optimiser{});
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
    if ((r = check_tc(net))) return r;
    if (loss) CK(cudaMemcpy(loss, net->loss, sizeof(float), cudaMemcpyDeviceToHost));
    if (grad) CK(cudaMemcpy(grad, net->G, NPARAM * 4, cudaMemcpyDeviceToHost));
    CK(cudaMemcpy(net->step, &saved, sizeof(int), cudaMemcpyHostToDevice));
    return BAMF_OK;
}

/* `steps` Adam steps, each one replay of a CUDA graph of: produce(s) (the
 * step's batch into gdata / gn / gxyi), forward, backward, Adam, weight
 * packing, step counter.  Optimiser state starts from zero. */
template <typename Produce>
static bamf_status train_graph(bamf_cnn *net, int steps, int batch, float lr, float *loss_trace, Produce produce)
{
    bamf_status r;
    if ((r = ensure_loss(net, steps))) return r;
    cudaStream_t s;
    CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    bamf_status res = BAMF_OK;
    do {
        if (cudaMemsetAsync(net->step, 0, sizeof(int), s) != cudaSuccess ||
            cudaMemsetAsync(net->loss, 0, (size_t)steps * sizeof(float), s) != cudaSuccess ||
            cudaMemsetAsync(net->M, 0, NPARAM * 4, s) != cudaSuccess ||
            cudaMemsetAsync(net->V, 0, NPARAM * 4, s) != cudaSuccess) {
            res = BAMF_ERR_CUDA;
            break;
        }
        if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
            res = BAMF_ERR_CUDA;
            break;
        }
        produce(s);
        bamf_status r1 = forward(net, net->gdata, batch, s);
        const Partials pt = backward(net, net->gn, net->gxyi, batch, 1.0f / (float)batch, s);
        const Optimiser opt = {net->P, net->M, net->V, net->Wf, net->Wb, net->step, net->done, steps, lr};
        reduce_kernel<true><<<RB_ALL, RED_THREADS, 0, s>>>(pt, nullptr, opt);
        const cudaError_t el = cudaGetLastError(), ec = cudaStreamEndCapture(s, &graph);
        if (r1 || el != cudaSuccess || ec != cudaSuccess) {
            res = r1 ? r1 : BAMF_ERR_CUDA;
            break;
        }
        if (cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) {
            res = BAMF_ERR_CUDA;
            break;
        }
        for (int i = 0; i < steps; ++i)
            if (cudaGraphLaunch(exec, s) != cudaSuccess) {
                res = BAMF_ERR_CUDA;
                break;
            }
        if (res) break;
        if (cudaStreamSynchronize(s) != cudaSuccess) {
            res = BAMF_ERR_CUDA;
            break;
        }
        if ((res = check_tc(net))) break;
        if (loss_trace &&
            cudaMemcpy(loss_trace, net->loss, (size_t)steps * sizeof(float), cudaMemcpyDeviceToHost) != cudaSuccess)
            res = BAMF_ERR_CUDA;
    } while (0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaStreamDestroy(s);
    if (res) cudaGetLastError();
    return res;
}

extern "C" bamf_status bamf_cnn_train(bamf_cnn *net, const bamf_synth_params *sp, int steps, int batch, float lr,
                                      uint32_t data_seed, float *loss_trace)
{
    if (!net || !sp || steps < 0 || batch < 1 || batch > MAX_BATCH || !(lr > 0.0f)) return BAMF_ERR_INVALID_ARG;
    if (steps == 0) return BAMF_OK;
    const bamf_synth_params spv = *sp;
    return train_graph(net, steps, batch, lr, loss_trace, [&](cudaStream_t s) {
        synth_kernel<<<batch, 256, 0, s>>>(spv, data_seed, 0, net->step, batch, batch, net->gdata, net->gn,
                                           net->gxyi);
    });
}

extern "C" bamf_status bamf_cnn_train_examples(bamf_cnn *net, const float *data, const int32_t *n_em,
                                               const float *xyi, int n_examples, int steps, int batch, float lr,
                                               float *loss_trace)
{
    if (!net || !data || !n_em || !xyi || n_examples < 1 || steps < 0 || batch < 1 || batch > MAX_BATCH ||
        !(lr > 0.0f))
        return BAMF_ERR_INVALID_ARG;
    if (steps == 0) return BAMF_OK;
    return train_graph(net, steps, batch, lr, loss_trace, [&](cudaStream_t s) {
        gather_examples_kernel<<<batch, NPX, 0, s>>>(data, n_em, xyi, n_examples, net->step, batch, net->gdata,
                                                     net->gn, net->gxyi);
    });
}

extern "C" bamf_status bamf_cnn_init_states(const float *cdf, const float *sub, const float *count_logits, int n,
                                            float intensity, int max_n, int32_t *init_n, float *init_ixy,
                                            void *stream)
{
    if (n < 0 || max_n < 0 || max_n > BAMF_NMAX) return BAMF_ERR_INVALID_ARG;
    if (n > 0 && (!cdf || !sub || !count_logits || !init_n || !init_ixy)) return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    init_kernel<<<n, 256, 0, (cudaStream_t)stream>>>(cdf, sub, count_logits, n, intensity, max_n, init_n, init_ixy);
    CK(cudaGetLastError());
    return BAMF_OK;
}

extern "C" bamf_status bamf_cnn_infer(bamf_cnn *net, const float *data, int n, float *cdf, float *sub,
                                      float *count_logits, void *stream)
{
    if (!net || n < 0 || (n > 0 && (!data || !cdf || !sub))) return BAMF_ERR_INVALID_ARG;
    if (n == 0) return BAMF_OK;
    /* 32-byte stores need the table at a 32-byte boundary */
    const auto kernel = ((uintptr_t)sub & 31) == 0 ? net_kernel<NET_INFER_WIDE> : net_kernel<NET_INFER>;
    kernel<<<net_grid(n, net->sms), 256 * INF_GROUPS, SMEM_INFER, (cudaStream_t)stream>>>(
        data, n, net->P, net->Wf, cdf, sub, count_logits, Kept{}, net->tc_status);
    CK(cudaGetLastError());
    return BAMF_OK;
}

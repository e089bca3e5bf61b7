/*
 * sampler_kernel.cuh - the batched RJMCMC sampler (cRJMCMC's algorithm,
 * source/c/LibRJMCMC.cpp) as a persistent CUDA kernel for sm_103a.
 *
 * Layout of the work:
 *   - one warp runs one ROI chain from burn-in to the last trial, then pulls
 *     the next ROI id from a device work queue (atomic counter);
 *   - lane j holds emitter slot j (I, X, Y, Signal) of the current state A
 *     and of the proposed state T in registers (BAMF_NMAX = 32 slots), so
 *     emitter edits are register moves and neighbour searches are ballots;
 *   - the ROI pixels D, the current model M, the proposed model Mt and the
 *     per-pixel work buffer live in shared memory; pixel p = y + x*Ysize is
 *     handled by lane p mod 32;
 *   - the scalar move logic (proposal, priors, Hastings ratio, accept) runs
 *     warp-uniformly: every lane evaluates it on the same values, so no
 *     broadcasts are needed and the warp never diverges there;
 *   - uniforms come from the chain's Philox stream (include/bamf_philox.h):
 *     each lane generates one 4-word block, 32 blocks = 128 uniforms per
 *     refill, kept as floats in shared memory; a draw is one broadcast load.
 *   - what is the same on every lane anyway is done for two or three arguments
 *     at once, one per part of the warp: Irwin-Hall draws, prior lookups.
 *
 * Two instantiations (template parameter EXACT):
 *   EXACT = true  (sampler_exact.cu, built with -fmad=false): the reference's
 *     float operation order, parity erf/log/exp, full model rebuild per
 *     proposal and serial pixel sums, so the chain is the reference chain
 *     bit for bit given the same uniforms.
 *   EXACT = false (sampler_fast.cu): hardware math, incremental model
 *     updates (only changed emitters' stencils are evaluated), cached
 *     log-model and warp-tree reductions; same moves and acceptance rule.
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bamf.h"
#include "bamf_parity_math.h"
#include "parity_quick.cuh"
#include "bamf_philox.h"
#include "sampler_common.h"

namespace bamf {

#define BAMF_FULL 0xffffffffu

/* counter slots, in bamf_counters order */
enum {
    C_N_jump, C_N_split, C_N_merge, C_N_birth, C_N_death,
    C_A_jump, C_A_split, C_A_merge, C_A_birth, C_A_death,
    C_N_jumpFg, C_N_splitFg, C_N_mergeFg, C_N_birthFg, C_N_deathFg,
    C_A_jumpFg, C_A_splitFg, C_A_mergeFg, C_A_birthFg, C_A_deathFg,
    C_N_jumpBg, C_N_splitBg, C_N_mergeBg, C_N_birthBg, C_N_deathBg,
    C_A_jumpBg, C_A_splitBg, C_A_mergeBg, C_A_birthBg, C_A_deathBg,
    C_COUNT
};

template <bool EXACT>
struct SMath;

template <>
struct SMath<true> {
    static __device__ __forceinline__ float erf_(float x) { return pq::erf_q(x); }
    static __device__ __forceinline__ float log_(float x) { return pq::log_q(x); }
    static __device__ __forceinline__ float exp_(float x) { return pq::exp_q(x); }
    static __device__ __forceinline__ float powf_(float x, float y) { return bamf_pm_powf(x, y); }
};

template <>
struct SMath<false> {
    static __device__ __forceinline__ float erf_(float x) { return erff(x); }
    static __device__ __forceinline__ float log_(float x) { return __logf(x); }
    static __device__ __forceinline__ float exp_(float x) { return __expf(x); }
    static __device__ __forceinline__ float powf_(float x, float y) { return powf(x, y); }
};

/* Per-warp shared-memory carve-out, in floats.  Exact: data D, model M,
 * proposal model Mt, per-pixel work E, sCMOS (each rounded up to 16 bytes,
 * for the vector loads of the serial sums), a pool of 2 x 32 stencil rows
 * NX/NY shared by A and T, 128 buffered uniforms.
 * Fast: D, M, Mt, the compact stencil rows SX/SY (old ones, of A, then new ones,
 * of T), the buffered uniforms and the shared draws of the next jumps; log2 M is recomputed in each likelihood pass (the
 * SFU has room; the smaller carve-out keeps 3 CTAs of 8 chains resident
 * up to 24x24 ROIs); sCMOS is read from global memory at model rebuilds
 * only.  Both: the neighbour pick list. */
/* Fast mode keeps stencil rows only for the emitters a proposal changes:
 * up to FAST_ROWS old rows (A) and FAST_ROWS new rows (T); larger proposals
 * (rare: a jump of a cluster of more than 4 emitters) and periodic rebuilds
 * stream the model one emitter at a time. */
#define FAST_ROWS 4
#define EXACT_ROWS (2 * BAMF_NMAX) /* stencil rows of the exact sampler's pool */
#define UBUF 128      /* buffered uniforms */
#define MOVE_AHEAD 32 /* jumps whose shared move draws are formed together (fast) */
__host__ __device__ inline int exact_npix(int side_max) { return (side_max * side_max + 3) & ~3; }
__host__ __device__ inline int warp_smem_floats(int side_max, bool exact)
{
    int npix = side_max * side_max, nxs = BAMF_NMAX * side_max;
    return exact ? 5 * exact_npix(side_max) + 4 * nxs + UBUF + BAMF_NMAX + 2 + 2
                 : (3 * npix + 4 * FAST_ROWS * side_max + 3 & ~3) + UBUF + 2 * MOVE_AHEAD + BAMF_NMAX;
}

/* double helpers that nvcc may not contract */
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }

/* Out-of-line helpers.  They are called from many places of the chain loop
 * but run rarely per jump; keeping one copy of each keeps the loop's code
 * small enough for the instruction cache (a fully inlined loop spent most
 * of its cycles waiting on instruction fetch). */

/* One Philox4x32-10 block of a chain's stream (include/bamf_philox.h). */
static __device__ __noinline__ uint4 philox_block(uint32_t ctr, uint32_t seed, uint32_t chain)
{
    bamf_philox_block b = bamf_philox4x32_10(ctr, 0u, 0u, 0u, seed, chain);
    return make_uint4(b.v[0], b.v[1], b.v[2], b.v[3]);
}

/* Stat::findPDF (source/c/LibRJMCMC.cpp:219-246): linear interpolation of
 * the pdf at I, 0 outside (0, x[L-1]).  The grid is x[i] = x[i-1] + DX, so
 * the first node strictly above I (what the reference's linear scan finds)
 * is reached from the guess I / DX in a step or two. */
static __device__ __noinline__ float stat_pdf(const float *__restrict__ x, const float *__restrict__ pdf, int L,
                                       float I)
{
    float xl = __ldg(&x[L - 1]);
    if (I >= xl || I <= 0.0f || I != I) return 0.0f;
    float x1 = __ldg(&x[1]);
    int j = min(max((int)(I / x1) + 1, 1), L - 1);
    float xj = __ldg(&x[j]), xj1 = __ldg(&x[j - 1]);
    while (j > 1 && xj1 > I) {
        --j;
        xj = xj1;
        xj1 = __ldg(&x[j - 1]);
    }
    while (j < L - 1 && !(xj > I)) {
        ++j;
        xj1 = xj;
        xj = __ldg(&x[j]);
    }
    return (__ldg(&pdf[j]) * (I - xj1) + __ldg(&pdf[j - 1]) * (xj - I)) / (x1 - __ldg(&x[0]));
}

/* Fast-arithmetic findPDF: the grid is uniform (x[i] = i DX up to float
 * rounding), so the interval of I is found by one multiply and its two
 * nodes are loaded together with the grid's end - one memory round trip
 * instead of a dependent walk.  Same linear interpolation, 0 outside
 * (0, x[L-1]). */
static __device__ __noinline__ float stat_pdf_fast(const float *__restrict__ x, const float *__restrict__ pdf, int L,
                                                   float inv_dx, float I)
{
    if (L < 2) return 0.0f;
    float u = fminf(fmaxf(I * inv_dx, 0.0f), (float)(L - 1)); /* NaN -> 0 */
    int j = min((int)u + 1, L - 1);
    float xl = __ldg(&x[L - 1]);
    float p1 = __ldg(&pdf[j]), p0 = __ldg(&pdf[j - 1]);
    float w = u - (float)(j - 1);
    float v = p1 * w + p0 * (1.0f - w);
    return (I >= xl || I <= 0.0f || I != I) ? 0.0f : v;
}

/* Fast-arithmetic genRand: the same first unique-CDF node above R, found by
 * a 32-way search (each lane tests one candidate, a ballot keeps the
 * bracket: two or three rounds of loads instead of a dependent binary
 * search), then the same interpolation.  Call with the whole warp. */
static __device__ __noinline__ float stat_rand_warp(const float *__restrict__ ux, const float *__restrict__ uc,
                                                    int nu, float R, int lane)
{
    if (R <= 0.0f) return 0.0f;
    if (R >= 1.0f) return __ldg(&ux[nu - 1]);
    if (nu < 2) return 0.0f;
    int lo = 0, hi = nu - 1; /* uc[lo] <= R < uc[hi] */
    while (hi - lo > 1) {
        int step = (hi - lo + 31) >> 5;
        int k = lo + (lane + 1) * step;
        bool above = k >= hi || __ldg(&uc[k]) > R;
        uint32_t m = __ballot_sync(0xffffffffu, above);
        int f = __ffs(m) - 1;
        int nlo = f == 0 ? lo : lo + f * step;
        hi = min(lo + (f + 1) * step, hi);
        lo = nlo;
    }
    float uc1 = __ldg(&uc[hi]), uc0 = __ldg(&uc[hi - 1]);
    return (__ldg(&ux[hi - 1]) * (uc1 - R) + __ldg(&ux[hi]) * (R - uc0)) / (uc1 - uc0);
}

/* Stat::genRand (:248-282) given its uniform R: first unique-CDF node above R
 * by binary search (the CDF is strictly increasing), then interpolation. */
static __device__ __noinline__ float stat_rand(const float *__restrict__ ux, const float *__restrict__ uc, int nu,
                                        float R)
{
    if (R <= 0.0f) return 0.0f;
    if (R >= 1.0f) return __ldg(&ux[nu - 1]);
    if (nu < 2) return 0.0f;
    int lo = 0, hi = nu - 1;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (__ldg(&uc[mid]) > R) hi = mid; else lo = mid;
    }
    float uc1 = __ldg(&uc[hi]), uc0 = __ldg(&uc[hi - 1]);
    return (__ldg(&ux[hi - 1]) * (uc1 - R) + __ldg(&ux[hi]) * (R - uc0)) / (uc1 - uc0);
}

/* Fast-mode Irwin-Hall draws: the 12 uniforms from u (the warp's buffer) on
 * lanes 0..11 of each half of the warp, added in a butterfly; STEP = 12 gives
 * the upper half the next twelve, so that a warp makes two draws at once.  Call
 * with the whole warp. */
template <int STEP>
static __device__ __noinline__ float irwin_hall12(const float *u, int lane)
{
    float v = (lane & 15) < 12 ? u[(lane & 15) + STEP * (lane >> 4)] : 0.0f;
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    return v - 6.0f;
}

/* Uniform in [0, 1) shared by the warps of a CTA in move-synchronous mode:
 * a 32-bit integer hash (the "lowbias32" xorshift-multiply finaliser,
 * applied twice) of (seed, group, step, which). */
__device__ __forceinline__ float shared_uniform(uint32_t seed, uint32_t grp, uint32_t step, uint32_t which)
{
    uint32_t x = seed * 0x9E3779B1u ^ grp * 0x85EBCA77u ^ (step * 2u + which) * 0xC2B2AE3Du;
    for (int r = 0; r < 2; ++r) {
        x ^= x >> 16;
        x *= 0x7feb352du;
        x ^= x >> 15;
        x *= 0x846ca68bu;
        x ^= x >> 16;
    }
    return (float)(x >> 8) * 5.9604644775390625e-08f;
}

/* (1 / A) / q(x, y) for the LEARNED birth proposal q = (learned + uniform)/2
 * on a box of area A; the learned part is the ROI's pixel running sum cdf
 * times the pixel's 16 sub-cell probabilities sub (16 cells per px^2). */
/* The learned position density at (x, y) per px^2 (pixel probability from
 * the running sum, sub-cell probability, 16 sub-cells per px^2); 0 outside
 * the ROI.  Call with the whole warp on the same arguments: lanes 0..15 load
 * the pixel's sub-cell probabilities and a butterfly sums them. */
static __device__ __noinline__ float learned_density(float x, float y, int X, int Y, int npix,
                                                     const float *__restrict__ cdf,
                                                     const float *__restrict__ sub)
{
    if (!(x >= 0.0f && y >= 0.0f && x < (float)X && y < (float)Y)) return 0.0f;
    const int lane = threadIdx.x & 31;
    int px = min((int)x, X - 1), py = min((int)y, Y - 1);
    int pix = py + px * Y;
    int sc = min((int)((y - (float)py) * 4.0f), 3) + 4 * min((int)((x - (float)px) * 4.0f), 3);
    float pp = __ldg(&cdf[pix]) - (pix > 0 ? __ldg(&cdf[pix - 1]) : 0.0f);
    const float *sp = sub + 16 * pix;
    const float v = lane < 16 ? __ldg(&sp[lane]) : 0.0f;
    float ps = v;
    for (int o = 1; o < 32; o <<= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
    const float vs = __shfl_sync(0xffffffffu, v, sc);
    return (pp / __ldg(&cdf[npix - 1])) * (vs / ps) * 16.0f;
}

/* (1 / A) / q(x, y) for the birth mixture q = 1/2 learned + 1/2 uniform on
 * the extended box of area A. */
static __device__ __noinline__ float learned_q_ratio(float x, float y, int X, int Y, int npix, float A,
                                                     const float *__restrict__ cdf,
                                                     const float *__restrict__ sub)
{
    const float qa = learned_density(x, y, X, Y, npix, cdf, sub) * A; /* learned density times box area */
    return 1.0f / (0.5f * qa + 0.5f);
}

/* normpdf (LibRJMCMCreturn.hpp:19-21) with (float)sqrt(2.0f*pi), pi = 3.141592. */
template <bool EXACT>
static __device__ __noinline__ float normpdf_f(float x, float u, float s)
{
    const float sq2pi = (float)sqrt(2.0 * 3.141592);
    float d = x - u;
    return 1.0f / (sq2pi * s) * SMath<EXACT>::exp_(-d * d / (2.0f * s * s));
}

/* Exact mode, a chain run by a team of TEAM warps: what its first warp asks
 * the others to do with their share of the pixels (TeamCmd::ASK_*), and the
 * state they need for it. */
struct TeamCmd {
    enum { ASK_END, ASK_MODEL, ASK_SCORE };
    int ask, X, Y, n;
    float BG, ABG, BBG;
    const float *D, *M, *NX, *NY, *scm;
    float *E, *out, *sink;
    int row[BAMF_NMAX];
};

template <bool EXACT, bool NUM, int TEAM = 1>
struct ChainWarp {
    typedef SMath<EXACT> MT;
    const SamplerConsts *K;
    const SamplerBatch *B;
    int lane;
    int roi;
    /* geometry */
    int X, Y, npix;
    static constexpr int STEP = 32 * TEAM; /* pixels of a pass */
    int px_dx, px_dy; /* pixel p -> p + STEP moves x by px_dx and y by px_dy (then wraps) */
    TeamCmd *cmd;     /* TEAM > 1: shared memory */
    float sigma, Cst, MeanN;
    /* shared memory */
    float *D, *M, *Mt, *E, *NX, *NY;
    /* exact mode: row r of the pool is NX[r X ..], NY[r Y ..]; arow / trow is
     * the row of this lane's emitter of A / of T (an emitter T left unchanged
     * keeps A's row; -1: changed or new, not evaluated yet) */
    int arow, trow;
    float *ubuf; /* uniforms base * 4 .. base * 4 + 127 of the stream */
    float *ahead; /* fast mode: the shared draws of MOVE_AHEAD jumps: move, then sub-branch */
    float *SX, *SY; /* fast mode: compact stencil rows */
    const float *scm; /* sCMOS: shared memory (exact) or global/null (fast) */
    /* sampled PSF (OptModel 1): [P0 y][P1 x][P2 y-sub][P3 x-sub], y fastest;
     * null for the Gaussian model */
    const float *psf;
    int pn0, pn01, pn012, ptot, pos;
    int cnt; /* lane k: counter k */
    int *cl;
    int rec_n[2];
    /* current state A (lane j = slot j) */
    int an;
    float aI, aX, aY;
    int aS;
    float aBG, aABG, aBBG;
    /* proposed state T */
    int tn;
    float tI, tX, tY;
    int tS;
    float tBG, tABG, tBBG;
    bool t_overflow;
    /* uniform stream */
    uint32_t seed, chain, base;
    uint32_t idx; /* next uniform of ubuf */
    /* phase */
    int is_burnin;
    float P[8];
    int entries;
    int overflow;
    int n_llr;
    /* incremental-model bookkeeping (fast mode) */
    uint32_t a_dirty, t_dirty;
    int llr_box; /* pixels the last likelihood pass changed: x0 | x1 << 8 | y0 << 16 | y1 << 24 */
    float pdf_aBG; /* offset-prior density of aBG */
    /* move-synchronous mode: the jump sub-branch uniform comes from the CTA */
    bool use_shared_ub;
    float shared_ub;

    /* ---------------------------------------------------------- RNG */
    __device__ __forceinline__ void refill()
    {
        /* block numbers wrap where a 32-bit stream index wraps */
        const uint4 b = philox_block((base + (uint32_t)lane) & 0x3fffffffu, seed, chain);
        __syncwarp();
        reinterpret_cast<float4 *>(ubuf)[lane] =
            make_float4(bamf_u31_to_float(b.x >> 1), bamf_u31_to_float(b.y >> 1), bamf_u31_to_float(b.z >> 1),
                        bamf_u31_to_float(b.w >> 1));
        __syncwarp();
    }
    /* the next n uniforms into the buffer (n <= 36): it then starts at the block
     * of the next one */
    __device__ __forceinline__ void ensure(uint32_t n)
    {
        if (idx + n > (uint32_t)UBUF) {
            base += idx >> 2;
            idx &= 3u;
            refill();
        }
    }
    __device__ __forceinline__ float urand()
    {
        ensure(1u);
        return ubuf[idx++];
    }
    /* Irwin-Hall sum of 12 uniforms (LibRJMCMCreturn.hpp:23-26).  Exact
     * mode adds them in draw order; fast mode in a butterfly over 12 lanes
     * (same distribution, other rounding). */
    __device__ __forceinline__ float randn()
    {
        ensure(12u);
        float t = 0;
        if (EXACT) {
            const float *u = ubuf + idx;
#pragma unroll
            for (int k = 0; k < 12; ++k) t = t + u[k];
            t = t - 6.0f;
        } else {
            t = irwin_hall12<0>(ubuf + idx, lane);
        }
        idx += 12u;
        return t;
    }

    /* Three consecutive randn().  Exact mode: lane k adds the k-th draw's twelve
     * uniforms, in draw order.  Fast mode: two at once in the warp's halves. */
    __device__ __forceinline__ void randn3(float &a, float &b, float &c)
    {
        ensure(36u);
        if (EXACT) {
            const float *u = ubuf + idx + 12 * min(lane, 2);
            float t = 0;
#pragma unroll
            for (int k = 0; k < 12; ++k) t = t + u[k];
            t = t - 6.0f;
            a = __shfl_sync(BAMF_FULL, t, 0);
            b = __shfl_sync(BAMF_FULL, t, 1);
            c = __shfl_sync(BAMF_FULL, t, 2);
        } else {
            const float t = irwin_hall12<12>(ubuf + idx, lane);
            a = __shfl_sync(BAMF_FULL, t, 0);
            b = __shfl_sync(BAMF_FULL, t, 16);
            c = irwin_hall12<0>(ubuf + idx + 24, lane);
        }
        idx += 36u;
    }

    /* ------------------------------------------------------ lane access */
    __device__ __forceinline__ float A_I(int k) const { return __shfl_sync(BAMF_FULL, aI, k); }
    __device__ __forceinline__ float A_X(int k) const { return __shfl_sync(BAMF_FULL, aX, k); }
    __device__ __forceinline__ float A_Y(int k) const { return __shfl_sync(BAMF_FULL, aY, k); }
    __device__ __forceinline__ int A_S(int k) const { return __shfl_sync(BAMF_FULL, aS, k); }
    __device__ __forceinline__ float T_I(int k) const { return __shfl_sync(BAMF_FULL, tI, k); }
    __device__ __forceinline__ int T_S(int k) const { return __shfl_sync(BAMF_FULL, tS, k); }

    __device__ __forceinline__ void setT(int k, float I, float x, float y)
    {
        if (lane == k) {
            tI = I;
            tX = x;
            tY = y;
            if (EXACT) trow = -1;
        }
        if (!EXACT) t_dirty |= 1u << k;
    }
    __device__ __forceinline__ void addT(float I, float x, float y, int s)
    {
        if (tn >= BAMF_NMAX) {
            t_overflow = true;
            return;
        }
        if (lane == tn) {
            tI = I;
            tX = x;
            tY = y;
            tS = s;
            if (EXACT) trow = -1;
        }
        if (!EXACT) t_dirty |= 1u << tn;
        tn++;
    }
    /* Emitters::remove (LibRJMCMC.cpp:478-490) */
    __device__ __forceinline__ void removeT(int id)
    {
        float vI = __shfl_down_sync(BAMF_FULL, tI, 1);
        float vX = __shfl_down_sync(BAMF_FULL, tX, 1);
        float vY = __shfl_down_sync(BAMF_FULL, tY, 1);
        int vS = __shfl_down_sync(BAMF_FULL, tS, 1);
        int vrow = EXACT ? __shfl_down_sync(BAMF_FULL, trow, 1) : 0;
        if (lane >= id) {
            tI = vI; tX = vX; tY = vY; tS = vS;
            if (EXACT) trow = vrow;
        }
        if (!EXACT) {
            uint32_t lo = t_dirty & ((1u << id) - 1u);
            uint32_t hi = id < 31 ? (t_dirty >> (id + 1)) << id : 0u;
            t_dirty = lo | hi;
        }
        tn--;
    }
    __device__ __forceinline__ void copyA2T()
    {
        tn = an; tI = aI; tX = aX; tY = aY; tS = aS;
        tBG = aBG; tABG = aABG; tBBG = aBBG;
        t_overflow = false;
        if (EXACT) trow = arow;
        if (!EXACT) {
            a_dirty = 0u;
            t_dirty = 0u;
        }
    }
    __device__ __forceinline__ void cinc(int k)
    {
        if (lane == k) cnt++;
    }

    /* Emitters::test (:492-514) with Bnd_out cast to int. */
    __device__ __forceinline__ bool testT() const
    {
        int bnd = (int)K->p.Bnd_out;
        bool bad = false;
        if (lane < tn)
            bad = (tI < 0.0f) || (tX < (float)(-bnd)) || (tY < (float)(-bnd)) ||
                  (tX > (float)(X + bnd)) || (tY > (float)(Y + bnd));
        return !__any_sync(BAMF_FULL, bad);
    }

    __device__ __forceinline__ float nsignalA() const
    {
        return (float)__popc(__ballot_sync(BAMF_FULL, lane < an && aS == 1));
    }

    /* ---------------------------------------------------- prior tables */
    __device__ __forceinline__ float findPDF(const DevStat &s, float I) const
    {
        if (EXACT) return stat_pdf(s.x, s.pdf, s.L, I);
        return stat_pdf_fast(s.x, s.pdf, s.L, s.inv_dx, I);
    }
    /* findPDF of two intensities at once: one in each half of the warp */
    __device__ __forceinline__ void findPDF2(const DevStat &s, float I0, float I1, float &p0, float &p1) const
    {
        const float v = findPDF(s, lane < 16 ? I0 : I1);
        p0 = __shfl_sync(BAMF_FULL, v, 0);
        p1 = __shfl_sync(BAMF_FULL, v, 16);
    }
    __device__ __forceinline__ float genRand(const DevStat &s)
    {
        float R = urand();
        if (EXACT) return stat_rand(s.ux, s.uc, s.nu, R);
        return stat_rand_warp(s.ux, s.uc, s.nu, R, lane);
    }
    __device__ __forceinline__ float sob(int signal, float I) const
    {
        const DevStat &s = signal == 1 ? K->sig : K->back;
        return findPDF(s, I);
    }
    __device__ __forceinline__ float normpdf(float x, float u, float s) const
    {
        return normpdf_f<EXACT>(x, u, s);
    }

    /* a / b for 0 <= a < 2^10, 1 <= b <= 64 (fast mode): (a + 1/2) / b is at least
     * 1/128 from an integer, far more than the reciprocal's error (2e-4) */
    static __device__ __forceinline__ int small_div(int a, float rb) { return (int)(((float)a + 0.5f) * rb); }

    /* ------------------------------------------------ neighbour search */
    __device__ __forceinline__ uint32_t near_mask(int jj, float dmin) const
    {
        float xj = A_X(jj), yj = A_Y(jj);
        bool in = false;
        if (lane < an && lane != jj) {
            float dx = aX - xj, dy = aY - yj;
            if (EXACT) {
                /* the reference compares (float)sqrt of the double sum; where
                 * the float sum of squares (three roundings, 1.8e-7) is more
                 * than 1e-6 from dmin^2 the answer is the same, and only the
                 * rest, NaN included, pays for FP64; a negative dmin has no
                 * neighbours, whatever its square */
                const float s = dx * dx + dy * dy, q = dmin * dmin;
                in = dmin > 0.0f && q > 1e-30f && s < q * 0.999999f;
                if (!in && !(q > 1e-30f && s > q * 1.000001f))
                    in = (float)sqrt(dadd(dmul((double)dx, (double)dx), dmul((double)dy, (double)dy))) < dmin;
            } else {
                const float d = sqrtf(dx * dx + dy * dy);
                in = d < dmin;
            }
        }
        return __ballot_sync(BAMF_FULL, in);
    }
    static __device__ __forceinline__ int nth_bit(uint32_t m, int q)
    {
        for (int t = 0; t < q; ++t) m &= m - 1u;
        return __ffs(m) - 1;
    }
    /* Emitters::closest (:525-558). */
    __device__ __forceinline__ int closest(int jj, float dmin)
    {
        uint32_t m = near_mask(jj, dmin);
        int num = __popc(m);
        if (num > 0) {
            float Ua = urand();
            int mm = min((int)(Ua * (float)num), num - 1);
            return nth_bit(m, mm);
        }
        uint32_t others = (an >= 32 ? BAMF_FULL : ((1u << an) - 1u)) & ~(1u << jj);
        float Ua = urand();
        int mm = min((int)(Ua * (float)(an - 1)), an - 2);
        return nth_bit(others, mm);
    }
    /* Emitters::closestMulti (:615-650); picks go to cl[] in pick order. */
    __device__ __forceinline__ int closestMulti(int jj, float dmin)
    {
        uint32_t m = near_mask(jj, dmin);
        int num = __popc(m);
        int np = 0;
        if (num > 0) {
            float Ua = urand();
            int Np;
            if (Ua < 1.0f / (float)num) Np = num;
            else Np = min((int)(Ua * (float)num), num - 1);
            for (int n = 0; n < Np; ++n) {
                Ua = urand();
                int q = min((int)(Ua * (float)(num - n)), num - n - 1);
                int b = nth_bit(m, q);
                m &= ~(1u << b);
                if (lane == 0) cl[np] = b;
                np++;
            }
        }
        __syncwarp();
        return np;
    }

    /* ------------------------------------------------------------ model */
    /* Exact mode, Stencil (:15-37): rows of the pool for the emitters in
     * `todo` (lane k's emitter for bit k) of the state (I, Xv, Yv, row); `keep`
     * is the row of this lane that must survive, or -1.  Unchanged emitters
     * keep their rows: the same function of the same inputs, so the same
     * bits.  One emitter's X + Y entries go over the lanes together; the kept
     * rows are at most BAMF_NMAX of A's, so BAMF_NMAX are free. */
    __device__ __forceinline__ void exact_rows(uint32_t todo, int keep, float I, float Xv, float Yv, int &row)
    {
        if (todo == 0u) return;
        uint32_t f0 = ~__reduce_or_sync(BAMF_FULL, keep >= 0 && keep < 32 ? 1u << keep : 0u);
        uint32_t f1 = ~__reduce_or_sync(BAMF_FULL, keep >= 32 ? 1u << (keep - 32) : 0u);
        const int XY = X + Y;
#pragma unroll 1
        for (; todo; todo &= todo - 1u) {
            const int k = __ffs(todo) - 1;
            int r;
            if (f0) {
                r = __ffs(f0) - 1;
                f0 &= f0 - 1u;
            } else {
                r = 31 + __ffs(f1);
                f1 &= f1 - 1u;
            }
            if (lane == k) row = r;
            const float Ik = __shfl_sync(BAMF_FULL, I, k), Xk = __shfl_sync(BAMF_FULL, Xv, k);
            const float Yk = __shfl_sync(BAMF_FULL, Yv, k);
#pragma unroll 1
            for (int c = lane; c < XY; c += 32) {
                const bool isx = c < X;
                const int cc = isx ? c : c - X;
                const float mu = isx ? Xk : Yk;
                const float x1 = ((float)cc - mu + 1.0f) * Cst, x0 = ((float)cc - mu) * Cst;
                float e1 = pq::erf_try(x1), e0 = pq::erf_try(x0); /* both in flight */
                if (e1 != e1) e1 = pq::erf_rest(x1);
                if (e0 != e0) e0 = pq::erf_rest(x0);
                if (isx) NX[r * X + cc] = Ik * 0.5f * (e1 - e0);
                else NY[r * Y + cc] = 0.5f * (e1 - e0);
            }
        }
        __syncwarp();
    }
    /* Exact mode, Model (:39-59) of pixels p + STEP j, j < J: the background
     * plane and sCMOS, then the emitters in slot order, into out; SCORE: the
     * likelihood-ratio term of each pixel into E.  J independent pixels per
     * lane keep the row loads and the logarithms in flight (one at a time: 7.2k
     * cycles per 16x16 proposal, four: 5.4k, eight: 5.0k, but with 16 chains on
     * an SM, where instruction fetch binds, 24k, 32k and 35k); lanes past the
     * last pixel store to `sink`, so there is no branch.  (x, y) is this
     * lane's pixel p, moved on to p + STEP J. */
    template <int J, bool SCORE>
    __device__ __forceinline__ void exact_pixels(int p, int &x, int &y, int n, int row, float BG, float ABG, float BBG,
                                                 float *out, float *sink)
    {
        int xs[J], ys[J];
        float m[J];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int q = p + STEP * j;
            const bool in = q < npix;
            xs[j] = in ? x : 0;
            ys[j] = in ? y : 0;
            m[j] = BG + ABG * (float)xs[j] + BBG * (float)ys[j] + scm[in ? q : 0];
            x += px_dx;
            y += px_dy;
            if (y >= Y) {
                y -= Y;
                x++;
            }
        }
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            const int r = __shfl_sync(BAMF_FULL, row, k);
            const float *nx = NX + r * X, *ny = NY + r * Y;
#pragma unroll
            for (int j = 0; j < J; ++j) m[j] += nx[xs[j]] * ny[ys[j]];
        }
        uint32_t open = 0u; /* pixels whose quotient or logarithm the quick forms leave open */
        if (SCORE) {
            /* all loads before the first store (which may alias them) */
            float ma[J], d[J], lg[J];
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int q = p + STEP * j < npix ? p + STEP * j : 0;
                ma[j] = M[q];
                d[j] = D[q];
            }
#pragma unroll
            for (int j = 0; j < J; ++j) lg[j] = pq::log_try(pq::div_try(m[j], ma[j]));
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const bool in = p + STEP * j < npix;
                *(in ? E + p + STEP * j : sink) = ma[j] - m[j] + d[j] * lg[j];
                if (in && lg[j] != lg[j]) open |= 1u << j;
            }
        }
#pragma unroll
        for (int j = 0; j < J; ++j) *(p + STEP * j < npix ? out + p + STEP * j : sink) = m[j];
        if (SCORE) {
#pragma unroll 1
            for (; open; open &= open - 1u) {
                const int q = p + STEP * (__ffs(open) - 1);
                const float mt = out[q];
                E[q] = M[q] - mt + D[q] * pq::log_slow(mt / M[q]);
            }
        }
    }
    /* This warp's share (warp `part` of TEAM) of the model of a state. */
    template <bool SCORE>
    __device__ __forceinline__ void exact_share(int part, int n, int row, float BG, float ABG, float BBG, float *out,
                                                float *sink)
    {
        int p = 32 * part + lane, x = p / Y, y = p - x * Y;
        if (TEAM == 1) {
#pragma unroll 1
            for (; p - lane + 64 < npix; p += 4 * STEP) exact_pixels<4, SCORE>(p, x, y, n, row, BG, ABG, BBG, out, sink);
        }
#pragma unroll 1
        for (; p - lane < npix; p += 2 * STEP) exact_pixels<2, SCORE>(p, x, y, n, row, BG, ABG, BBG, out, sink);
    }
    /* the team's barrier (CTA barrier 1, all its warps); a CTA is one team */
    static __device__ __forceinline__ void team_sync()
    {
        asm volatile("barrier.sync 1, %0;" ::"n"(STEP) : "memory");
    }
    template <bool SCORE>
    __device__ __forceinline__ void exact_model(int n, int row, float BG, float ABG, float BBG, float *out)
    {
        float *sink = (float *)(cl + BAMF_NMAX);
        if (TEAM > 1) {
            cmd->row[lane] = row;
            if (lane == 0) {
                cmd->ask = SCORE ? TeamCmd::ASK_SCORE : TeamCmd::ASK_MODEL;
                cmd->X = X;
                cmd->Y = Y;
                cmd->n = n;
                cmd->BG = BG;
                cmd->ABG = ABG;
                cmd->BBG = BBG;
                cmd->D = D;
                cmd->M = M;
                cmd->NX = NX;
                cmd->NY = NY;
                cmd->scm = scm;
                cmd->E = E;
                cmd->out = out;
                cmd->sink = sink;
            }
            team_sync();
        }
        exact_share<SCORE>(0, n, row, BG, ABG, BBG, out, sink);
        if (TEAM > 1) team_sync();
        else __syncwarp();
    }
    /* warps 1 .. TEAM - 1 of a team: serve until its first warp ends */
    __device__ __forceinline__ void team_serve(int part)
    {
        for (;;) {
            team_sync();
            const int ask = cmd->ask;
            if (ask == TeamCmd::ASK_END) return;
            X = cmd->X;
            Y = cmd->Y;
            npix = X * Y;
            px_dx = STEP / Y;
            px_dy = STEP - px_dx * Y;
            D = const_cast<float *>(cmd->D);
            M = const_cast<float *>(cmd->M);
            NX = const_cast<float *>(cmd->NX);
            NY = const_cast<float *>(cmd->NY);
            scm = cmd->scm;
            E = cmd->E;
            if (ask == TeamCmd::ASK_SCORE)
                exact_share<true>(part, cmd->n, cmd->row[lane], cmd->BG, cmd->ABG, cmd->BBG, cmd->out, cmd->sink);
            else
                exact_share<false>(part, cmd->n, cmd->row[lane], cmd->BG, cmd->ABG, cmd->BBG, cmd->out, cmd->sink);
            team_sync();
        }
    }
    /* Exact mode: the sum of E in pixel order, on every lane.  The additions
     * are one dependent chain; 16-byte loads one step ahead keep it at the
     * adder's latency. */
    __device__ __forceinline__ float exact_sum() const
    {
        const float4 *E4 = reinterpret_cast<const float4 *>(E);
        const int nq = npix >> 2;
        float t = 0.0f;
        int q = 0;
        float4 v[4];
        if (nq >= 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = E4[j];
        }
#pragma unroll 1
        for (; q + 4 <= nq; q += 4) {
            float4 w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = E4[min(q + 4 + j, nq - 1)];
#pragma unroll
            for (int j = 0; j < 4; ++j) t = t + v[j].x + v[j].y + v[j].z + v[j].w;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = w[j];
        }
#pragma unroll 1
        for (int p = 4 * q; p < npix; ++p) t += E[p];
        return t;
    }
    /* Exact mode: E becomes its running sum, in place (every lane adds the
     * same chain, lane 0 stores). */
    __device__ __forceinline__ void exact_scan()
    {
        float4 *E4 = reinterpret_cast<float4 *>(E);
        const int nq = npix >> 2;
        float t = 0.0f;
        int q = 0;
#pragma unroll 1
        for (; q + 8 <= nq; q += 8) {
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = E4[q + j];
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                t = q + j == 0 ? v[j].x : v[j].x + t;
                v[j].x = t;
                v[j].y = t = v[j].y + t;
                v[j].z = t = v[j].z + t;
                v[j].w = t = v[j].w + t;
            }
            if (lane == 0) {
#pragma unroll
                for (int j = 0; j < 8; ++j) E4[q + j] = v[j];
            }
        }
        __syncwarp();
        if (lane == 0) {
#pragma unroll 1
            for (int p = 4 * q; p < npix; ++p) {
                if (p > 0) E[p] += E[p - 1];
            }
        }
        __syncwarp();
    }

    /* Fast mode: stencil rows of the emitters a proposal changes, compact:
     * row q of SX/SY is the old stencil of the q-th slot of a_dirty (from
     * A), row na + q the new stencil of the q-th slot of t_dirty (from
     * T).  mx, my: the columns and rows where any of them is not zero. */
    __device__ __forceinline__ void stencil_rows(int na, int nt, uint32_t &mx, uint32_t &my)
    {
        const int XY = X + Y, nr = na + nt;
        /* the rows' entries one after the other, 32 a pass: as few passes as
         * there can be for rows that do not fill 32 lanes */
        const int total = nr * XY;
        const float rXY = __frcp_rn((float)XY);
        uint32_t ux = 0u, uy = 0u;
#pragma unroll 1
        for (int e0 = 0; e0 < total; e0 += 32) {
            const int e = min(e0 + lane, total - 1);
            const int r = small_div(e, rXY), c = e - r * XY;
            const bool isnew = r >= na;
            const int q = isnew ? r - na : r;
            const int k = nth_bit(isnew ? t_dirty : a_dirty, q);
            /* a shuffle returns the source lane's value, so fetch both
             * states and select here (lanes of one pass may read rows of
             * different states) */
            const float Ia = __shfl_sync(BAMF_FULL, aI, k), It = __shfl_sync(BAMF_FULL, tI, k);
            const float Xa = __shfl_sync(BAMF_FULL, aX, k), Xt = __shfl_sync(BAMF_FULL, tX, k);
            const float Ya = __shfl_sync(BAMF_FULL, aY, k), Yt = __shfl_sync(BAMF_FULL, tY, k);
            const bool isx = c < X;
            const int cc = isx ? c : c - X;
            const float mu = isx ? (isnew ? Xt : Xa) : (isnew ? Yt : Ya);
            const float v = 0.5f * (MT::erf_(((float)cc - mu + 1.0f) * Cst) - MT::erf_(((float)cc - mu) * Cst));
            const float sv = isx ? (isnew ? It : Ia) * v : v;
            if (e0 + lane < total) (isx ? SX + r * X : SY + r * Y)[cc] = sv;
            const uint32_t bit = sv != 0.0f ? 1u << cc : 0u;
            ux |= isx ? bit : 0u;
            uy |= isx ? 0u : bit;
        }
        mx = __reduce_or_sync(BAMF_FULL, ux);
        my = __reduce_or_sync(BAMF_FULL, uy);
        __syncwarp();
    }

    /* Fast mode: out = background plane + sCMOS + sum of the state's emitter
     * stencils, one emitter at a time (its rows go through SX/SY row 0). */
    __device__ __forceinline__ void model_stream(int n, float I, float Xv, float Yv, float BG, float ABG,
                                                 float BBG, float *out)
    {
        int x = lane / Y, y = lane - (lane / Y) * Y;
#pragma unroll 1
        for (int p = lane; p < npix; p += 32) {
            out[p] = BG + ABG * (float)x + BBG * (float)y + (scm ? scm[p] : 0.0f);
            x += px_dx;
            y += px_dy;
            if (y >= Y) {
                y -= Y;
                x++;
            }
        }
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
            float Ik = __shfl_sync(BAMF_FULL, I, k), Xk = __shfl_sync(BAMF_FULL, Xv, k);
            float Yk = __shfl_sync(BAMF_FULL, Yv, k);
            __syncwarp();
#pragma unroll 1
            for (int c = lane; c < X + Y; c += 32) {
                bool isx = c < X;
                int cc = isx ? c : c - X;
                float mu = isx ? Xk : Yk;
                float v = 0.5f * (MT::erf_(((float)cc - mu + 1.0f) * Cst) - MT::erf_(((float)cc - mu) * Cst));
                if (isx) SX[cc] = Ik * v;
                else SY[cc] = v;
            }
            __syncwarp();
            x = lane / Y;
            y = lane - (lane / Y) * Y;
#pragma unroll 1
            for (int p = lane; p < npix; p += 32) {
                out[p] += SX[x] * SY[y];
                x += px_dx;
                y += px_dy;
                if (y >= Y) {
                    y -= Y;
                    x++;
                }
            }
        }
        __syncwarp();
    }

    /* ------------------------------------------ sampled-PSF model */
    /* NumModel (:67-170) places emitter (x, y) on four planes of the sampled
     * PSF: pixel (xx, yy) of the ROI reads flat index b_i + yy + xx P0 of
     * plane i and blends them bilinearly with weights wx (x) and wy (y).
     * Exact mode repeats the reference's double arithmetic; fast mode takes
     * the same steps in float. */
    struct NumPlace {
        int b1, b2, b3, b4;
        float wx, wy;
    };
    __device__ __forceinline__ NumPlace num_place(float xf, float yf) const
    {
        const int c0 = pn0 / 2;
        int sx, sy, ix, iy;
        NumPlace q;
        if (EXACT) {
            const double xd = (double)xf, yd = (double)yf, os = (double)pos;
            const double fx = dadd(xd, -floor(xd)), fy = dadd(yd, -floor(yd));
            sx = (int)ceil(dadd((double)c0, -xd));
            ix = (int)floor(dmul(os, fx));
            sy = (int)ceil(dadd((double)c0, -yd));
            iy = (int)floor(dmul(os, fy));
            q.wy = (float)dadd(1.0, -dmul(dadd(fy, -__ddiv_rn((double)iy, os)), os));
            q.wx = (float)dadd(1.0, -dmul(dadd(fx, -__ddiv_rn((double)ix, os)), os));
        } else {
            const float os = (float)pos;
            const float fx = xf - floorf(xf), fy = yf - floorf(yf);
            sx = (int)ceilf((float)c0 - xf);
            ix = (int)floorf(os * fx);
            sy = (int)ceilf((float)c0 - yf);
            iy = (int)floorf(os * fy);
            q.wy = 1.0f - (fy * os - (float)iy);
            q.wx = 1.0f - (fx * os - (float)ix);
        }
        int sx2 = sx, ix2 = ix + 1, sy2 = sy, iy2 = iy + 1;
        if (ix == pos - 1) {
            sx2 = sx - 1;
            ix2 = 0;
        }
        if (iy == pos - 1) {
            sy2 = sy - 1;
            iy2 = 0;
        }
        q.b1 = sy + sx * pn0 + iy * pn01 + ix * pn012;
        q.b2 = sy + sx2 * pn0 + iy * pn01 + ix2 * pn012;
        q.b3 = sy2 + sx * pn0 + iy2 * pn01 + ix * pn012;
        q.b4 = sy2 + sx2 * pn0 + iy2 * pn01 + ix2 * pn012;
        return q;
    }
    /* a flat index outside the array reads its last element (:131-157) */
    __device__ __forceinline__ float psf_at(int i) const
    {
        return psf[(i >= ptot || i < 0) ? ptot - 1 : i];
    }
    /* the blended PSF value of pixel offset o = yy + xx P0 */
    __device__ __forceinline__ float num_value(const NumPlace &q, int o) const
    {
        float a = q.wx * psf_at(q.b1 + o) + (1.0f - q.wx) * psf_at(q.b2 + o);
        float b = q.wx * psf_at(q.b3 + o) + (1.0f - q.wx) * psf_at(q.b4 + o);
        return q.wy * a + (1.0f - q.wy) * b;
    }
    __device__ __forceinline__ static NumPlace shfl_place(const NumPlace &q, int k)
    {
        NumPlace r;
        r.b1 = __shfl_sync(BAMF_FULL, q.b1, k);
        r.b2 = __shfl_sync(BAMF_FULL, q.b2, k);
        r.b3 = __shfl_sync(BAMF_FULL, q.b3, k);
        r.b4 = __shfl_sync(BAMF_FULL, q.b4, k);
        r.wx = __shfl_sync(BAMF_FULL, q.wx, k);
        r.wy = __shfl_sync(BAMF_FULL, q.wy, k);
        return r;
    }

    /* NumModel of a lane-distributed state into out[] (both modes: the
     * background plane, then the emitters in slot order, per pixel). */
    __device__ __forceinline__ void model_num(int n, float I, float Xv, float Yv, float BG, float ABG, float BBG,
                                              float *out)
    {
        NumPlace q = num_place(lane < n ? Xv : 0.0f, lane < n ? Yv : 0.0f);
#pragma unroll 1
        for (int b0 = 0; b0 < npix; b0 += 32) {
            const int p = b0 + lane;
            const bool v = p < npix;
            const int x = p / Y, y = p - x * Y;
            float m = v ? BG + ABG * (float)x + BBG * (float)y + (scm ? scm[p] : 0.0f) : 0.0f;
            const int o = y + x * pn0;
#pragma unroll 1
            for (int k = 0; k < n; ++k) {
                NumPlace r = shfl_place(q, k);
                float Ik = __shfl_sync(BAMF_FULL, I, k);
                if (v) m = m + Ik * num_value(r, o);
            }
            if (v) out[p] = m;
        }
        __syncwarp();
    }

    /* Fast mode, sampled PSF: Mt = M + the background change - the changed
     * emitters of A + the changed emitters of T (lane q < na + nt holds
     * changed slot q, intensity negated for A's); returns the pixel sum of
     * D (ln Mt - ln M) - (Mt - M). */
    __device__ __forceinline__ float llr_num_fast(int na, int nt)
    {
        const float LN2 = 0.69314718f;
        const int nr = na + nt;
        const bool isnew = lane >= na;
        const int qq = isnew ? lane - na : lane;
        int k = lane < nr ? nth_bit(isnew ? t_dirty : a_dirty, qq) : 0;
        float Ia = __shfl_sync(BAMF_FULL, aI, k), It = __shfl_sync(BAMF_FULL, tI, k);
        float Xa = __shfl_sync(BAMF_FULL, aX, k), Xt = __shfl_sync(BAMF_FULL, tX, k);
        float Ya = __shfl_sync(BAMF_FULL, aY, k), Yt = __shfl_sync(BAMF_FULL, tY, k);
        const float Iq = lane < nr ? (isnew ? It : -Ia) : 0.0f;
        NumPlace q = num_place(isnew ? Xt : Xa, isnew ? Yt : Ya);
        const float dBG = tBG - aBG, dABG = tABG - aABG, dBBG = tBBG - aBBG;
        float acc = 0.0f;
#pragma unroll 1
        for (int b0 = 0; b0 < npix; b0 += 32) {
            const int p = b0 + lane;
            const bool v = p < npix;
            const int x = p / Y, y = p - x * Y;
            float d = dBG + dABG * (float)x + dBBG * (float)y;
            const int o = y + x * pn0;
#pragma unroll 1
            for (int r = 0; r < nr; ++r) {
                NumPlace g = shfl_place(q, r);
                float Ir = __shfl_sync(BAMF_FULL, Iq, r);
                if (v) d += Ir * num_value(g, o);
            }
            if (v) {
                float mt = M[p] + d;
                Mt[p] = mt;
                acc += D[p] * (__log2f(mt) - __log2f(M[p])) * LN2 - d;
            }
        }
        return acc;
    }

    /* likelihood_ratio (:1650-1686).  M always holds Model(A). */
    __device__ __forceinline__ float llr()
    {
        n_llr++;
        if (EXACT) {
            if constexpr (NUM) {
                model_num(tn, tI, tX, tY, tBG, tABG, tBBG, Mt);
                for (int p = lane; p < npix; p += 32)
                    E[p] = M[p] - Mt[p] + D[p] * MT::log_(Mt[p] / M[p]);
                __syncwarp();
            } else {
                exact_rows(__ballot_sync(BAMF_FULL, lane < tn && trow < 0), lane < an ? arow : -1, tI, tX, tY, trow);
                exact_model<true>(tn, trow, tBG, tABG, tBBG, Mt);
            }
            return MT::exp_(exact_sum());
        } else {
            /* Mt = M + background delta - old stencils of A's changed slots
             *        + new stencils of T's changed slots;
             * sum over pixels of (M - Mt) + D (ln Mt - ln M) */
            const float LN2 = 0.69314718f;
            int na = __popc(a_dirty), nt = __popc(t_dirty);
            float acc = 0.0f;
            if constexpr (NUM) {
                llr_box = full_box();
                if (na <= FAST_ROWS && nt <= FAST_ROWS) {
                    acc = llr_num_fast(na, nt);
                } else {
                    model_num(tn, tI, tX, tY, tBG, tABG, tBBG, Mt);
#pragma unroll 1
                    for (int p = lane; p < npix; p += 32) {
                        float mt = Mt[p];
                        acc += D[p] * (__log2f(mt) - __log2f(M[p])) * LN2 - (mt - M[p]);
                    }
                }
            } else {
                if (na <= FAST_ROWS && nt <= FAST_ROWS) {
                    uint32_t mx = 0u, my = 0u;
                    stencil_rows(na, nt, mx, my);
                    const int nr = na + nt;
                    /* Support box: unless the background changes, a pixel
                     * outside the union of the changed rows' nonzero x- and
                     * y-stencil entries has d = 0 exactly (Mt = M, a zero
                     * term), so the pass covers only the box.  Stencils of
                     * sigma ~1.3 vanish in float ~7 px from the emitter. */
                    int x0 = 0, x1 = X - 1, y0 = 0, y1 = Y - 1;
                    if (tBG == aBG && tABG == aABG && tBBG == aBBG) {
                        if (mx == 0u || my == 0u) {
                            llr_box = 1; /* empty: Mt = M everywhere, LLR = 1 */
                            return 1.0f;
                        }
                        x0 = __ffs(mx) - 1;
                        x1 = 31 - __clz(mx);
                        y0 = __ffs(my) - 1;
                        y1 = 31 - __clz(my);
                    }
                    llr_box = x0 | (x1 << 8) | (y0 << 16) | (y1 << 24);
                    /* lane -> row y = y0 + lane mod h of column x0 + lane / h
                     * (h the box height); a pass covers 32 / h columns.  The
                     * model change of a pixel is bg delta + sum_q w_q(y)
                     * SX_q[x] over the changed rows q (old rows with weight
                     * -SY, new with +SY); each lane holds its first four
                     * weights in registers. */
                    const int h = y1 - y0 + 1;
                    const float rh = __frcp_rn((float)h);
                    const int xo = small_div(lane, rh), yl = y0 + lane - xo * h, R = small_div(32, rh);
                    float w[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float sy = q < nr ? SY[q * Y + yl] : 0.0f;
                        w[q] = q < na ? -sy : sy;
                    }
                    const float base = (tBG - aBG) + (tBBG - aBBG) * (float)yl, dABG = tABG - aABG;
                    if (xo < R) {
                        /* two columns at a time: one column's loads and
                         * logarithms hide the other's; added in order */
#pragma unroll 1
                        for (int xx = x0 + xo; xx <= x1; xx += 2 * R) {
                            const bool two = xx + R <= x1;
                            const int xb = two ? xx + R : xx, p0 = yl + Y * xx, p1 = yl + Y * xb;
                            const float m0 = M[p0], m1 = M[p1], v0 = D[p0], v1 = D[p1];
                            float d0 = base + dABG * (float)xx, d1 = base + dABG * (float)xb;
                            if (nr > 0) {
                                d0 += w[0] * SX[xx];
                                d1 += w[0] * SX[xb];
                            }
                            if (nr > 1) {
                                d0 += w[1] * SX[X + xx];
                                d1 += w[1] * SX[X + xb];
                            }
                            if (nr > 2) {
                                d0 += w[2] * SX[2 * X + xx];
                                d1 += w[2] * SX[2 * X + xb];
                            }
                            if (nr > 3) {
                                d0 += w[3] * SX[3 * X + xx];
                                d1 += w[3] * SX[3 * X + xb];
                            }
                            for (int q = 4; q < nr; ++q) {
                                const bool old = q < na;
                                const float *sr = SX + q * X;
                                const float sy = SY[q * Y + yl];
                                d0 = __fadd_rn(d0, __fmul_rn(old ? -sr[xx] : sr[xx], sy));
                                d1 = __fadd_rn(d1, __fmul_rn(old ? -sr[xb] : sr[xb], sy));
                            }
                            const float t0 = m0 + d0, t1 = m1 + d1;
                            Mt[p0] = t0;
                            acc += v0 * (__log2f(t0) - __log2f(m0)) * LN2 - d0;
                            if (two) {
                                Mt[p1] = t1;
                                acc += v1 * (__log2f(t1) - __log2f(m1)) * LN2 - d1;
                            }
                        }
                    }
                } else {
                    model_stream(tn, tI, tX, tY, tBG, tABG, tBBG, Mt);
                    llr_box = full_box();
#pragma unroll 1
                    for (int p = lane; p < npix; p += 32) {
                        float mt = Mt[p];
                        acc += D[p] * (__log2f(mt) - __log2f(M[p])) * LN2 - (mt - M[p]);
                    }
                }
            }
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(BAMF_FULL, acc, o);
            return MT::exp_(acc);
        }
    }

    /* fast mode: fold the accepted proposal into M (Mt differs from M only
     * inside the box of the last likelihood pass) */
    __device__ __forceinline__ int full_box() const { return (X - 1) << 8 | (Y - 1) << 24; }
    __device__ __forceinline__ void commit_fast()
    {
        const int x0 = llr_box & 255, x1 = (llr_box >> 8) & 255, y0 = (llr_box >> 16) & 255, y1 = llr_box >> 24;
        if (x0 <= x1) {
            const int h = y1 - y0 + 1;
            const float rh = __frcp_rn((float)h);
            const int xo = small_div(lane, rh), yy = y0 + lane - xo * h, R = small_div(32, rh);
            if (xo < R) {
#pragma unroll 1
                for (int xx = x0 + xo; xx <= x1; xx += R) M[yy + Y * xx] = Mt[yy + Y * xx];
            }
        }
        __syncwarp();
    }

    __device__ __forceinline__ void accept_T()
    {
        if (!EXACT) commit_fast();
        if (tBG != aBG) pdf_aBG = findPDF(K->off, tBG);
        an = tn; aI = tI; aX = tX; aY = tY; aS = tS;
        aBG = tBG; aABG = tABG; aBBG = tBBG;
        if (EXACT) {
            float *t = M;
            M = Mt;
            Mt = t;
            arow = trow;
        }
    }

    /* Full rebuild of M. */
    __device__ __forceinline__ void rebuild_model()
    {
        if (EXACT) {
            if constexpr (NUM) model_num(an, aI, aX, aY, aBG, aABG, aBBG, M);
            else {
                exact_rows(__ballot_sync(BAMF_FULL, lane < an), -1, aI, aX, aY, arow);
                exact_model<false>(an, arow, aBG, aABG, aBBG, M);
            }
        } else {
            /* with a drift output, a periodic rebuild goes to Mt (free
             * between proposals) first, to measure how far the incrementally
             * updated M has moved from the model of its state */
            const bool chk = B->model_drift != nullptr && entries > 0;
            float *dst = chk ? Mt : M;
            if constexpr (NUM) model_num(an, aI, aX, aY, aBG, aABG, aBBG, dst);
            else model_stream(an, aI, aX, aY, aBG, aABG, aBBG, dst);
            __syncwarp();
            if (chk) {
                float d = 0.0f;
                for (int p = lane; p < npix; p += 32) {
                    const float m = Mt[p];
                    d = fmaxf(d, fabsf(M[p] - m) / m);
                    M[p] = m;
                }
                for (int o = 16; o > 0; o >>= 1) d = fmaxf(d, __shfl_xor_sync(BAMF_FULL, d, o));
                /* non-negative floats order like their bit patterns */
                if (lane == 0) atomicMax((int *)&B->model_drift[roi], __float_as_int(d));
                __syncwarp();
            }
        }
    }

    /* ------------------------------------------------------- recording */
    __device__ __forceinline__ void record_one(int w, int n, float I, float x, float y, int s, float BG, float ABG,
                               float BBG, float LLR, float PR, int type, int acc)
    {
        bamf_chain *ch = &B->chains[2 * roi + w];
        int e = entries;
        if (e >= ch->capacity_entries) return;
        /* the entry's eight fields are consecutive pointers of bamf_chain: lane
         * k loads the k-th and stores the k-th value */
        if (lane < 8) {
            uint32_t v = lane == 0 ? (uint32_t)n : lane == 1 ? __float_as_uint(LLR) : __float_as_uint(PR);
            v = lane == 3 ? (uint32_t)type : lane == 4 ? (uint32_t)acc : v;
            v = lane == 5 ? __float_as_uint(BG) : lane == 6 ? __float_as_uint(ABG) : lane == 7 ? __float_as_uint(BBG) : v;
            reinterpret_cast<uint32_t *const *>(&ch->N)[lane][e] = v;
        }
        int rc = rec_n[w];
        int nrec = n < 1 ? 1 : n;
        if (rc + nrec <= ch->capacity_records) {
            /* all pointers before the first store (which may alias them) */
            int32_t *pi = ch->Index + rc + lane, *ps = ch->Signal + rc + lane;
            float *pp = ch->Photons + rc + lane, *px = ch->X + rc + lane, *py = ch->Y + rc + lane;
            if (lane < nrec) {
                *pi = e + 1;
                *pp = n < 1 ? 0.0f : I;
                *px = n < 1 ? -100.0f : x + K->p.DriftX;
                *py = n < 1 ? -100.0f : y + K->p.DriftY;
                *ps = n < 1 ? -1 : s;
            }
        }
        rec_n[w] = rc + nrec;
    }

    /* mean X of the Signal==1 emitters of A (NaN when none) into x_trace */
    __device__ __forceinline__ void record_x()
    {
        bool on = lane < an && aS == 1;
        float sx = on ? aX : 0.0f;
        for (int o = 16; o > 0; o >>= 1) sx += __shfl_xor_sync(BAMF_FULL, sx, o);
        int ns = __popc(__ballot_sync(BAMF_FULL, on));
        if (lane == 0)
            B->x_trace[(int64_t)roi * B->x_cap + entries] = ns > 0 ? sx / (float)ns : __int_as_float(0x7fc00000);
    }

    /* thinned state record: entry, Signal==1 count, BG, ABG, BBG, then X, Y,
     * I of the Signal==1 emitters in slot order (NaN past the count) */
    __device__ __forceinline__ void record_pos()
    {
        float *rec = B->pos_trace + ((int64_t)roi * B->pos_len + entries / B->pos_thin) * BAMF_POS_RECORD;
        bool on = lane < an && aS == 1;
        uint32_t m = __ballot_sync(BAMF_FULL, on);
        int rank = __popc(m & ((1u << lane) - 1u));
        int ns = __popc(m);
        if (lane == 0) {
            rec[0] = (float)entries;
            rec[1] = (float)ns;
            rec[2] = aBG;
            rec[3] = aABG;
            rec[4] = aBBG;
        }
        if (lane < BAMF_POS_SLOTS) {
            const float nan = __int_as_float(0x7fc00000);
            rec[5 + lane] = nan;
            rec[5 + BAMF_POS_SLOTS + lane] = nan;
            rec[5 + 2 * BAMF_POS_SLOTS + lane] = nan;
        }
        __syncwarp();
        if (on && rank < BAMF_POS_SLOTS) {
            rec[5 + rank] = aX;
            rec[5 + BAMF_POS_SLOTS + rank] = aY;
            rec[5 + 2 * BAMF_POS_SLOTS + rank] = aI;
        }
    }

    /* RJMCMCChain::addEmitters on Chain (A) and Chain_Test (T). */
    __device__ __forceinline__ void record2(float LLR, float PR, int type, int acc)
    {
        if (B->nsig_trace && entries < B->trace_cap) {
            int ns = __popc(__ballot_sync(BAMF_FULL, lane < an && aS == 1));
            if (lane == 0) B->nsig_trace[(int64_t)roi * B->trace_cap + entries] = (uint8_t)(an < 1 ? 0 : ns);
        }
        if (B->x_trace && entries < B->x_cap) record_x();
        if (B->pos_trace) {
            /* every pos_thin-th entry, pos_len at most; the product with 1 / pos_thin is
             * off by at most one below 2^22 entries and settles all others without
             * a division */
            const int rem = entries - (int)((float)entries * B->pos_rthin) * B->pos_thin;
            if ((rem == 0 || rem == B->pos_thin || rem == -B->pos_thin || entries >= (1 << 22)) &&
                entries % B->pos_thin == 0 && entries / B->pos_thin < B->pos_len)
                record_pos();
        }
        if (B->chains) {
            record_one(0, an, aI, aX, aY, aS, aBG, aABG, aBBG, LLR, PR, type, acc);
            record_one(1, tn, tI, tX, tY, tS, tBG, tABG, tBBG, LLR, PR, type, acc);
        }
        entries++;
    }

    /* floor(g + 0.5) as the reference forms it, in double.  Below 2^22 the
     * fraction g - floor(g) is exact in float, or rounds within [1/2, 1] (g in
     * (-1/2, 0)), so its comparison with 1/2 gives the same integer. */
    static __device__ __forceinline__ int kround(float g)
    {
        if (fabsf(g) < 4194304.0f) {
            const float f = floorf(g);
            return (int)f + (g - f >= 0.5f ? 1 : 0);
        }
        return (int)floor(dadd((double)g, 0.5));
    }

    /* RJMCMC::update_grids (:1629-1648). */
    __device__ __forceinline__ void update_grids()
    {
        if (is_burnin || !B->pgrid) return;
        int Z = K->p.Grid_Zoom;
        if (lane < an) {
            /* the float sum with 0.5 is exact for |coordinate| < 2^22: fast
             * mode rounds as the reference's double sum does */
            const float gx = (float)Z * (aX + K->p.DriftX), gy = (float)Z * (aY + K->p.DriftY);
            int x = EXACT ? kround(gx) : (int)floorf(gx + 0.5f);
            int y = EXACT ? kround(gy) : (int)floorf(gy + 0.5f);
            float *gb = aS == 1 ? B->pgrid : B->pback;
            if (gb && x >= 0 && x < X * Z && y >= 0 && y < Y * Z && aI > K->p.Icutoff) {
                /* grid slot (ROIs sharing one accumulate) and column stride */
                int64_t slot = B->grid_slot ? (int64_t)B->grid_slot[roi] : (int64_t)roi;
                int64_t ld = B->grid_ld > 0 ? (int64_t)B->grid_ld : (int64_t)Y * Z;
                atomicAdd(&gb[slot * B->grid_stride + (int64_t)x * ld + y], 1.0f);
            }
        }
    }


    /* ------------------------------------------------------------ moves */
    /* Every move is split in two: propose_*() consumes the move's uniforms,
     * builds T and returns what happens next; finish_*() turns the
     * likelihood ratio into the move's posterior ratio (no uniforms).  The
     * likelihood ratio, the accept draw, the commit and the chain record are
     * then one shared code path in step(), in the reference's order
     * (proposal draws, test, likelihood_ratio, priors, accept draw). */
    enum { ACT_SKIP = 0, ACT_GRIDS = 1, ACT_REJECT = 2, ACT_EVAL = 3 };
    enum { MV_JUMP, MV_SPLIT, MV_MERGE, MV_BIRTH, MV_DEATH, MV_GSPLIT, MV_GMERGE };
    /* pending proposal between propose and finish */
    int pk_move, pk_type, pk_c1, pk_c2, pk_i0, pk_i1, pk_i2;
    float pk_f0, pk_f1, pk_f2, pk_f3, pk_f4, pk_f5;

    /* RJMCMC::jump (:752-970) up to the likelihood ratio. */
    __device__ __forceinline__ int propose_jump()
    {
        cinc(C_N_jump);
        int type = 1;
        float PrI = 1.0f, IPDF, IPDFtest;
        copyA2T();
        if (an < 1) return ACT_SKIP;
        float Ua = urand();
        int nn = min((int)(Ua * (float)tn), tn - 1);
        float Ub = use_shared_ub ? shared_ub : urand();
        const bamf_mcmc_params &p = K->p;
        if (Ub < 0.25f) {
            type = 2;
            float g0, g1, g2;
            randn3(g0, g1, g2);
            tBG = tBG + p.BG_std * g0;
            tABG = tABG + p.ABBG_std * g1;
            tBBG = tBBG + p.ABBG_std * g2;
        } else if (Ub < 0.50f && Ub >= 0.25f) {
            if (an < 2) return ACT_SKIP;
            type = 10;
            int Np = closestMulti(nn, 2 * sigma);
            if (Np == 0) return ACT_SKIP;
            float I0 = A_I(nn);
            for (int i = 0; i < Np; ++i) I0 = I0 + A_I(cl[i]);
            float II0 = 0, XI0 = 0, YI0 = 0, XII0 = 0, YII0 = 0;
            for (int i = 0; i < Np; ++i) {
                int c = cl[i];
                float aIc = A_I(c), aXc = A_X(c), aYc = A_Y(c);
                int aSc = A_S(c);
                float nX, nY, nI;
                if (aSc == 1) {
                    float g0, g1, g2;
                    randn3(g0, g1, g2);
                    nX = aXc + p.X_stdFg * g0;
                    nY = aYc + p.X_stdFg * g1;
                    nI = (I0 / (float)(Np + 1)) * (0.15f * g2 + 1.0f);
                    findPDF2(K->sig, nI, aIc, IPDFtest, IPDF);
                } else {
                    float g0, g1, g2;
                    randn3(g0, g1, g2);
                    nX = aXc + p.X_stdBg * g0;
                    nY = aYc + p.X_stdBg * g1;
                    nI = (I0 / (float)(Np + 1)) * (0.15f * g2 + 1.0f);
                    findPDF2(K->back, nI, aIc, IPDFtest, IPDF);
                }
                PrI = PrI * IPDFtest / IPDF;
                setT(c, nI, nX, nY);
                if (!EXACT) a_dirty |= 1u << c;
                XI0 = XI0 + aIc * aXc;
                YI0 = YI0 + aIc * aYc;
                XII0 = XII0 + nI * nX;
                YII0 = YII0 + nI * nY;
                II0 = II0 + nI;
            }
            float aIn = A_I(nn), aXn = A_X(nn), aYn = A_Y(nn);
            int aSn = A_S(nn);
            float tIn = I0 - II0;
            float tXn = (XI0 + aIn * aXn - XII0) / tIn;
            float tYn = (YI0 + aIn * aYn - YII0) / tIn;
            setT(nn, tIn, tXn, tYn);
            if (!EXACT) a_dirty |= 1u << nn;
            IPDFtest = sob(aSn, tIn);
            IPDF = sob(aSn, aIn);
            PrI = PrI * IPDFtest / IPDF;
        } else if (Ub >= 0.5f && Ub < 0.75f) {
            type = 3;
            int NN = closestMulti(nn, 2 * sigma);
            if (lane == 0) cl[NN] = nn;
            __syncwarp();
            NN++;
            for (int i = 0; i < NN; ++i) {
                int c = cl[i];
                float aIc = A_I(c);
                int aSc = A_S(c);
                float cI = T_I(c);
                float cX = __shfl_sync(BAMF_FULL, tX, c), cY = __shfl_sync(BAMF_FULL, tY, c);
                float nI, nX, nY;
                if (aSc == 1) {
                    cinc(C_N_jumpFg);
                    float g0, g1, g2;
                    randn3(g0, g1, g2);
                    nI = cI + p.I_stdFg * g0;
                    nX = cX + p.X_stdFg * g1;
                    nY = cY + p.X_stdFg * g2;
                    findPDF2(K->sig, nI, aIc, IPDFtest, IPDF);
                } else {
                    cinc(C_N_jumpBg);
                    float g0, g1, g2;
                    randn3(g0, g1, g2);
                    nI = cI + p.I_stdBg * g0;
                    nX = cX + p.X_stdBg * g1;
                    nY = cY + p.X_stdBg * g2;
                    findPDF2(K->back, nI, aIc, IPDFtest, IPDF);
                }
                PrI = PrI * IPDFtest / IPDF;
                setT(c, nI, nX, nY);
                if (!EXACT) a_dirty |= 1u << c;
            }
        } else {
            float aIn = A_I(nn), aXn = A_X(nn), aYn = A_Y(nn);
            int aSn = A_S(nn);
            float nI, nX, nY;
            if (!EXACT && K->proposal == BAMF_PROPOSAL_LEARNED && urand() < 0.25f) {
                /* LEARNED relocation (no reference counterpart): an
                 * independence proposal of the emitter's position from the
                 * birth mixture q = 1/2 learned + 1/2 uniform on the extended
                 * box, intensity kept; Hastings factor q(old) / q(new) =
                 * birth_q_ratio(new) / birth_q_ratio(old), position prior
                 * uniform on the box, so the target is unchanged for any q */
                cinc(aSn == 1 ? C_N_jumpFg : C_N_jumpBg);
                birth_position(&nX, &nY);
                setT(nn, aIn, nX, nY);
                if (!EXACT) a_dirty |= 1u << nn;
                pk_move = MV_JUMP;
                pk_type = type;
                pk_f0 = birth_q_ratio(nX, nY) / birth_q_ratio(aXn, aYn);
                pk_c1 = C_A_jump;
                pk_c2 = aSn == 1 ? C_A_jumpFg : C_A_jumpBg;
                return testT() ? ACT_EVAL : ACT_REJECT;
            }
            if (aSn == 1) {
                cinc(C_N_jumpFg);
                float g0, g1, g2;
                randn3(g0, g1, g2);
                nI = aIn + p.I_stdFg * g0;
                nX = aXn + p.X_stdFg * g1;
                nY = aYn + p.X_stdFg * g2;
                findPDF2(K->sig, nI, aIn, IPDFtest, IPDF);
            } else {
                cinc(C_N_jumpBg);
                float g0, g1, g2;
                randn3(g0, g1, g2);
                nI = aIn + p.I_stdBg * g0;
                nX = aXn + p.X_stdBg * g1;
                nY = aYn + p.X_stdBg * g2;
                findPDF2(K->back, nI, aIn, IPDFtest, IPDF);
            }
            PrI = IPDFtest / IPDF;
            setT(nn, nI, nX, nY);
            if (!EXACT) a_dirty |= 1u << nn;
        }
        pk_move = MV_JUMP;
        pk_type = type;
        pk_f0 = PrI;
        pk_c1 = C_A_jump;
        pk_c2 = A_S(nn) == 1 ? C_A_jumpFg : C_A_jumpBg;
        return testT() ? ACT_EVAL : ACT_REJECT;
    }
    __device__ __forceinline__ float finish_jump(float LLR)
    {
        if (!EXACT) {
            /* fast: the offset prior of the current BG is cached, and the
             * factors of an unchanged BG / slope are 1 (x / x, exp(0)) */
            float BgPDFtest = tBG == aBG ? pdf_aBG : findPDF(K->off, tBG);
            float PrBg = BgPDFtest / pdf_aBG;
            if (tBBG != aBBG) PrBg *= MT::exp_(-(tBBG * tBBG - aBBG * aBBG) / 2.0f);
            if (tABG != aABG) PrBg *= MT::exp_(-(tABG * tABG - aABG * aABG) / 2.0f);
            return LLR * pk_f0 * PrBg;
        }
        float BgPDF = pdf_aBG;
        float BgPDFtest = tBG == aBG ? pdf_aBG : findPDF(K->off, tBG);
        /* unchanged slopes: exp(-0) = 1, and the product with 1 is exact */
        float PrBg = BgPDFtest / BgPDF;
        const float db = -(tBBG * tBBG - aBBG * aBBG) / 2.0f, da = -(tABG * tABG - aABG * aABG) / 2.0f;
        if (db != 0.0f) PrBg = PrBg * MT::exp_(db);
        if (da != 0.0f) PrBg = PrBg * MT::exp_(da);
        return LLR * pk_f0 * PrBg;
    }

    /* RJMCMC::split (:972-1109). */
    __device__ __forceinline__ int propose_split()
    {
        cinc(C_N_split);
        copyA2T();
        if (an < 1) return ACT_SKIP;
        const bamf_mcmc_params &p = K->p;
        float Ua = urand();
        int jj = min((int)floorf((float)an * Ua), an - 1);
        float Ijp = A_I(jj), mux = A_X(jj), muy = A_Y(jj);
        int BF = A_S(jj);
        cinc(BF == 1 ? C_N_splitFg : C_N_splitBg);
        float u1 = urand();
        float u2, u3;
        if (!EXACT && K->proposal == BAMF_PROPOSAL_LEARNED && urand() < 0.5f) {
            /* learned split: the first emitter's position from the learned
             * density and the intensity fraction from a triangular density on
             * [0.3, 0.7] (the mixture density of (u1, offset) enters
             * finish_split) */
            float lx, ly;
            learned_position(&lx, &ly);
            u1 = 0.3f + 0.2f * (urand() + urand());
            u2 = lx - mux;
            u3 = ly - muy;
        } else {
            u2 = p.Split_std * randn();
            u3 = p.Split_std * randn();
        }
        setT(jj, u1 * Ijp, mux + u2, muy + u3);
        if (!EXACT) a_dirty |= 1u << jj;
        addT((1.0f - u1) * Ijp, mux - u1 * u2 / (1.0f - u1), muy - u1 * u3 / (1.0f - u1), BF);
        pk_move = MV_SPLIT;
        pk_type = 4;
        pk_i0 = jj;
        pk_f0 = u1;
        pk_f1 = u2;
        pk_f2 = u3;
        pk_f3 = Ijp;
        pk_c1 = C_A_split;
        pk_c2 = BF == 1 ? C_A_splitFg : C_A_splitBg;
        if (t_overflow) {
            overflow++;
            return ACT_REJECT;
        }
        return testT() ? ACT_EVAL : ACT_REJECT;
    }
    __device__ __forceinline__ float finish_split(float LLR)
    {
        const bamf_mcmc_params &p = K->p;
        int jj = pk_i0;
        float u1 = pk_f0, u2 = pk_f1, u3 = pk_f2, Ijp = pk_f3;
        float tmp1 = 1.0f, tmp2 = 1.0f;
        tmp1 = tmp1 * sob(A_S(jj), A_I(jj));
        tmp2 = tmp2 * sob(T_S(jj), T_I(jj));
        tmp2 = tmp2 * sob(T_S(tn - 1), T_I(tn - 1));
        float Norm1 = normpdf(u2, 0.0f, p.Split_std);
        float Norm2 = normpdf(u3, 0.0f, p.Split_std);
        float NEm = nsignalA();
        float PrM = MeanN / (NEm + 1.0f);
        float PrI = tmp2 / tmp1;
        float Area = (float)(((float)X + p.Bnd_out) * ((float)Y + p.Bnd_out));
        float PrX = 1.0f / Area;
        float Us = 1.0f / (Norm1 * Norm2);
        float om = 1.0f - u1;
        float Jacob = EXACT ? (float)(__ddiv_rn((double)Ijp, dmul((double)om, (double)om))) : Ijp / (om * om);
        if (!EXACT && K->proposal != BAMF_PROPOSAL_REFERENCE) {
            /* exact split/merge pair accounting: the merge proposes this pair
             * with probability (1/k_a + 1/k_b) / (n + 1) (a random partner
             * within 3 sigma of a random emitter; k = such partners), the
             * split draws it from either emitter as the first:
             * (1/n) (q_a / J_a + q_b / J_b) */
            const float xa = __shfl_sync(BAMF_FULL, tX, jj), ya = __shfl_sync(BAMF_FULL, tY, jj);
            const float xb = __shfl_sync(BAMF_FULL, tX, tn - 1), yb = __shfl_sync(BAMF_FULL, tY, tn - 1);
            const float dmax = 3.0f * sigma;
            const float dx = xa - xb, dy = ya - yb;
            if (!(sqrtf(dx * dx + dy * dy) < dmax)) return 0.0f; /* no merge undoes it */
            const float ka = (float)near_count_T(jj, dmax), kb = (float)near_count_T(tn - 1, dmax);
            const float mux = A_X(jj), muy = A_Y(jj);
            const float qa = pair_density(u1, xa - mux, ya - muy, xa, ya, Ijp);
            const float qb = pair_density(1.0f - u1, xb - mux, yb - muy, xb, yb, Ijp);
            return LLR * PrI * (1.0f / box_area()) * (P[2] / P[1]) * PrM * (float)an * (1.0f / ka + 1.0f / kb) /
                   (qa + qb);
        }
        return LLR * PrI * PrX * Us * Jacob * (P[1] / P[2]) * PrM;
    }

    /* RJMCMC::merge (:1111-1255). */
    __device__ __forceinline__ int propose_merge()
    {
        cinc(C_N_merge);
        copyA2T();
        if (an < 2) return ACT_GRIDS;
        float Ua = urand();
        int jj = min((int)floorf((float)an * Ua), an - 1);
        int ii = closest(jj, 3 * sigma);
        int aSj = A_S(jj);
        cinc(aSj == 1 ? C_N_mergeFg : C_N_mergeBg);
        float aIj = A_I(jj), aXj = A_X(jj), aYj = A_Y(jj);
        float aIi = A_I(ii), aXi = A_X(ii), aYi = A_Y(ii);
        {
            float dx = aXj - aXi, dy = aYj - aYi;
            float d2 = EXACT ? (float)dadd(dmul((double)dx, (double)dx), dmul((double)dy, (double)dy))
                             : dx * dx + dy * dy;
            if (sqrtf(d2) > 3 * sigma) return ACT_GRIDS;
        }
        float Ijp = aIj + aIi;
        float muxjp = (aIj * aXj + aIi * aXi) / Ijp;
        float muyjp = (aIj * aYj + aIi * aYi) / Ijp;
        float u1 = aIj / Ijp;
        float u2 = aXj - muxjp;
        float u3 = aYj - muyjp;
        setT(jj, Ijp, muxjp, muyjp);
        float PDFfg = findPDF(K->sig, Ijp);
        float PDFbg = findPDF(K->back, Ijp);
        if (lane == jj) tS = (PDFbg > PDFfg) ? 0 : 1;
        if (!EXACT) a_dirty |= (1u << jj) | (1u << ii);
        removeT(ii);
        pk_move = MV_MERGE;
        pk_type = 5;
        pk_i0 = jj;
        pk_i1 = ii;
        pk_i2 = aSj;
        pk_f0 = u1;
        pk_f1 = u2;
        pk_f2 = u3;
        pk_f3 = Ijp;
        pk_f4 = aIj;
        pk_f5 = aIi;
        pk_c1 = aSj == 1 ? C_A_mergeFg : C_A_mergeBg;
        pk_c2 = C_A_merge;
        return testT() ? ACT_EVAL : ACT_REJECT;
    }
    __device__ __forceinline__ float finish_merge(float LLR)
    {
        const bamf_mcmc_params &p = K->p;
        int jj = pk_i0, ii = pk_i1, aSj = pk_i2;
        float u1 = pk_f0, u2 = pk_f1, u3 = pk_f2, Ijp = pk_f3, aIj = pk_f4, aIi = pk_f5;
        float tmp1 = 1.0f, tmp2 = 1.0f;
        tmp1 = tmp1 * sob(aSj, aIj);
        tmp1 = tmp1 * sob(A_S(ii), aIi);
        int jt = ii > jj ? jj : jj - 1;
        tmp2 = tmp2 * sob(T_S(jt), T_I(jt));
        float Norm1 = normpdf(u2, 0.0f, p.Split_std);
        float Norm2 = normpdf(u3, 0.0f, p.Split_std);
        float NEm = nsignalA();
        float PrI = tmp1 / tmp2;
        float Area = (float)(((float)X + p.Bnd_out) * ((float)Y + p.Bnd_out));
        float PrX = 1.0f / Area;
        float Us = 1.0f / (Norm1 * Norm2);
        float om = 1.0f - u1;
        float Jacob = EXACT ? (float)(__ddiv_rn((double)Ijp, dmul((double)om, (double)om))) : Ijp / (om * om);
        float PrM = MeanN / NEm;
        if (!EXACT && K->proposal != BAMF_PROPOSAL_REFERENCE) {
            /* the inverse of the split ratio that would undo this merge
             * (pair accounting as in finish_split) */
            const float dmax = 3.0f * sigma;
            const float kj = (float)__popc(near_mask(jj, dmax)), ki = (float)__popc(near_mask(ii, dmax));
            const float muxjp = __shfl_sync(BAMF_FULL, tX, jj > ii ? jj - 1 : jj);
            const float muyjp = __shfl_sync(BAMF_FULL, tY, jj > ii ? jj - 1 : jj);
            const float xa = A_X(jj), ya = A_Y(jj), xb = A_X(ii), yb = A_Y(ii);
            const float qa = pair_density(u1, xa - muxjp, ya - muyjp, xa, ya, Ijp);
            const float qb = pair_density(1.0f - u1, xb - muxjp, yb - muyjp, xb, yb, Ijp);
            return LLR / (PrI * (1.0f / box_area()) * (P[2] / P[1]) * PrM * (float)(an - 1) *
                          (1.0f / kj + 1.0f / ki) / (qa + qb));
        }
        return LLR / (PrI * PrX * Jacob * Us * PrM * P[1] / P[2]);
    }

    /* Density of a split that makes (x1, y1) the first emitter, over the
     * Jacobian: q(u1, u) (1 - u1)^2 / I for intensity fraction u1 and offset
     * u = (first emitter) - (split emitter).  q: UNIFORM, U(0, 1) x
     * N(0, Split_std^2)^2; LEARNED, half of that and half the triangular
     * density on [0.3, 0.7] x the learned density at (x1, y1). */
    __device__ __forceinline__ float pair_density(float u1, float u2, float u3, float x1, float y1, float I) const
    {
        const float s = K->p.Split_std;
        float q = normpdf(u2, 0.0f, s) * normpdf(u3, 0.0f, s);
        if (K->proposal == BAMF_PROPOSAL_LEARNED) {
            const int64_t off = B->offsets[roi];
            const float ql = learned_density(x1, y1, X, Y, npix, B->birth_cdf + off, B->birth_sub + 16 * off);
            const float tri = fmaxf(0.0f, 1.0f - fabsf(u1 - 0.5f) * 5.0f) * 5.0f;
            q = 0.5f * q + 0.5f * tri * ql;
        }
        const float om = 1.0f - u1;
        return q * om * om / I;
    }
    /* emitters of T within dmin of T's emitter k (k excluded) */
    __device__ __forceinline__ int near_count_T(int k, float dmin) const
    {
        const float xk = __shfl_sync(BAMF_FULL, tX, k), yk = __shfl_sync(BAMF_FULL, tY, k);
        const float dx = tX - xk, dy = tY - yk;
        return __popc(__ballot_sync(BAMF_FULL, lane < tn && lane != k && sqrtf(dx * dx + dy * dy) < dmin));
    }

    /* Area of the extended box [-Bnd, X+Bnd] x [-Bnd, Y+Bnd] that test()
     * admits (Bnd = (int)Bnd_out): the support of the position prior. */
    __device__ __forceinline__ float box_area() const
    {
        int bnd = (int)K->p.Bnd_out;
        return (float)(X + 2 * bnd) * (float)(Y + 2 * bnd);
    }

    /* Birth position of the UNIFORM and LEARNED proposals: uniform on the
     * extended box, or (LEARNED, with probability 1/2) a pixel drawn from
     * the ROI's running sum birth_cdf, a sub-cell drawn from birth_sub and a
     * uniform point inside that sub-cell. */
    __device__ __forceinline__ void birth_position(float *bx, float *by)
    {
        const int bnd = (int)K->p.Bnd_out;
        bool learned = K->proposal == BAMF_PROPOSAL_LEARNED && urand() < 0.5f;
        if (!learned) {
            *bx = (float)(-bnd) + (float)(X + 2 * bnd) * urand();
            *by = (float)(-bnd) + (float)(Y + 2 * bnd) * urand();
            return;
        }
        learned_position(bx, by);
    }

    /* A position drawn from the learned density: a pixel from the ROI's
     * running sum birth_cdf, a sub-cell from birth_sub, a uniform point in
     * the sub-cell.  Call with the whole warp. */
    __device__ __forceinline__ void learned_position(float *bx, float *by)
    {
        const int64_t off = B->offsets[roi];
        const float *cdf = B->birth_cdf + off;
        float rr = urand() * __ldg(&cdf[npix - 1]);
        /* the first pixel whose running sum reaches rr, in two rounds of
         * loads: the first 32-pixel block whose last sum reaches it (npix <=
         * 1024, so one lane per block), then the pixel inside it */
        const int nblk = (npix + 31) >> 5;
        const uint32_t mb =
            __ballot_sync(BAMF_FULL, lane < nblk && rr <= __ldg(&cdf[min(32 * lane + 31, npix - 1)]));
        const int blk = mb ? __ffs(mb) - 1 : nblk - 1;
        const int q = 32 * blk + lane;
        const uint32_t mp = __ballot_sync(BAMF_FULL, q < npix && rr <= __ldg(&cdf[min(q, npix - 1)]));
        const int pix = mp ? 32 * blk + __ffs(mp) - 1 : npix - 1;
        const float *sub = B->birth_sub + 16 * (off + pix);
        float v = lane < 16 ? __ldg(&sub[lane]) : 0.0f;
        for (int o = 1; o < 16; o <<= 1) {
            float t = __shfl_up_sync(BAMF_FULL, v, o);
            if (lane >= o) v += t;
        }
        float tot = __shfl_sync(BAMF_FULL, v, 15);
        float r2 = urand() * tot;
        uint32_t m = __ballot_sync(BAMF_FULL, lane < 16 && r2 <= v);
        int sc = m ? __ffs(m) - 1 : 15;
        int px = pix / Y, py = pix - px * Y;
        *bx = (float)px + ((float)(sc >> 2) + urand()) * 0.25f;
        *by = (float)py + ((float)(sc & 3) + urand()) * 0.25f;
    }

    /* (1 / box area) / q(x, y): the position prior over the birth proposal
     * density at (x, y); 1 for UNIFORM. */
    __device__ __forceinline__ float birth_q_ratio(float x, float y) const
    {
        if (K->proposal != BAMF_PROPOSAL_LEARNED) return 1.0f;
        const int64_t off = B->offsets[roi];
        return learned_q_ratio(x, y, X, Y, npix, box_area(), B->birth_cdf + off, B->birth_sub + 16 * off);
    }

    /* RJMCMC::find_Birth (:1688-1736); PixProb is overwritten with 1. */
    __device__ __forceinline__ void find_birth(float *bx, float *by)
    {
        float total;
        float *Pf = EXACT ? E : Mt; /* prefix buffer; Mt is free before the proposal is scored */
        if (EXACT) {
            for (int p = lane; p < npix; p += 32) {
                float v = D[p] - M[p];
                E[p] = (0.0f > v) ? 0.0f : v;
            }
            __syncwarp();
            exact_scan();
            total = E[npix - 1];
        } else {
            /* Fast: the residual's running sum is never stored.  Lane j sums
             * the contiguous chunk j of ceil(npix/32) pixels, a warp scan
             * gives the chunk ends, a ballot finds the chunk that reaches
             * rr, and that chunk's pixels (one per lane) are scanned again
             * to find the pixel: the same draw (the first pixel whose
             * running sum reaches rr), two passes over the chunk's pixels
             * instead of three over all. */
            const int per = (npix + 31) >> 5;
            const int p0 = min(lane * per, npix), p1 = min(p0 + per, npix);
            float s = 0.0f;
#pragma unroll 1
            for (int p = p0; p < p1; ++p) {
                float v = D[p] - M[p];
                s += v > 0.0f ? v : 0.0f;
            }
            float incl = s;
            for (int o = 1; o < 32; o <<= 1) {
                float t = __shfl_up_sync(BAMF_FULL, incl, o);
                if (lane >= o) incl += t;
            }
            total = __shfl_sync(BAMF_FULL, incl, 31);
            const float rr = total * urand();
            const uint32_t mc = __ballot_sync(BAMF_FULL, p0 < p1 && rr <= incl);
            int ii;
            if (mc) {
                const int cj = __ffs(mc) - 1;
                const float base = __shfl_sync(BAMF_FULL, incl - s, cj);
                const int q0 = cj * per, q = q0 + lane;
                float v = 0.0f;
                if (lane < per && q < npix) {
                    v = D[q] - M[q];
                    v = v > 0.0f ? v : 0.0f;
                }
                for (int o = 1; o < 32; o <<= 1) {
                    float t = __shfl_up_sync(BAMF_FULL, v, o);
                    if (lane >= o) v += t;
                }
                const uint32_t mq = __ballot_sync(BAMF_FULL, lane < per && q < npix && rr <= base + v);
                ii = mq ? q0 + __ffs(mq) - 1 : min(q0 + per, npix) - 1;
            } else {
                ii = npix; /* rr beyond the total (total 0: every pixel zero) */
            }
            *by = (float)(ii - Y * (ii / Y)) + urand() - 0.5f;
            *bx = (float)(int)floorf((float)ii / (float)Y) + urand() - 0.5f;
            return;
        }
        float rr = total * urand();
        int first = npix;
#pragma unroll 1
        for (int p = lane; p < npix; p += 32)
            if (rr <= Pf[p]) {
                first = p;
                break;
            }
        for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(BAMF_FULL, first, o));
        int ii = first;
        *by = (float)(ii - Y * (ii / Y)) + urand() - 0.5f;
        *bx = (float)(int)floorf((float)ii / (float)Y) + urand() - 0.5f;
        __syncwarp();
    }

    /* RJMCMC::birth (:1258-1330). */
    __device__ __forceinline__ int propose_birth()
    {
        cinc(C_N_birth);
        copyA2T();
        const bamf_mcmc_params &p = K->p;
        float bx, by;
        if (!EXACT && K->proposal != BAMF_PROPOSAL_REFERENCE) birth_position(&bx, &by);
        else find_birth(&bx, &by);
        pk_f0 = bx;
        pk_f1 = by;
        int BF;
        if (p.IsBackg == 1) BF = EXACT ? (int)floor(dadd((double)urand(), 0.5)) : (int)floorf(urand() + 0.5f);
        else BF = 1;
        float I_new;
        if (BF == 1) {
            cinc(C_N_birthFg);
            I_new = genRand(K->sig);
        } else {
            cinc(C_N_birthBg);
            I_new = genRand(K->back);
        }
        addT(I_new, bx, by, BF);
        pk_move = MV_BIRTH;
        pk_type = 6;
        pk_c1 = BF == 1 ? C_A_birthFg : C_A_birthBg;
        pk_c2 = C_A_birth;
        if (t_overflow) {
            overflow++;
            return ACT_REJECT;
        }
        return testT() ? ACT_EVAL : ACT_REJECT;
    }
    __device__ __forceinline__ float finish_birth(float LLR)
    {
        const bamf_mcmc_params &p = K->p;
        float NEm = nsignalA();
        float PrM = MeanN / (NEm + 1.0f);
        if (!EXACT && K->proposal != BAMF_PROPOSAL_REFERENCE)
            return LLR * PrM * (P[4] / P[3]) * birth_q_ratio(pk_f0, pk_f1);
        const float PixProb = 1.0f;
        return LLR * P[3] / (P[4] * ((float)X + p.Bnd_out) * ((float)Y + p.Bnd_out) * PixProb) * PrM;
    }

    /* RJMCMC::death (:1332-1387). */
    __device__ __forceinline__ int propose_death()
    {
        cinc(C_N_death);
        copyA2T();
        if (an < 1) return ACT_SKIP;
        float Ua = urand();
        int jj = min((int)floorf((float)an * Ua), an - 1);
        int aSj = A_S(jj);
        cinc(aSj == 1 ? C_N_deathFg : C_N_deathBg);
        if (!EXACT) a_dirty |= 1u << jj;
        removeT(jj);
        pk_move = MV_DEATH;
        pk_type = 7;
        pk_i0 = jj;
        pk_c1 = C_A_death;
        pk_c2 = aSj == 1 ? C_A_deathFg : C_A_deathBg;
        return ACT_EVAL;
    }
    __device__ __forceinline__ float finish_death(float LLR)
    {
        float NEm = nsignalA();
        float PrM = NEm / MeanN;
        if (!EXACT && K->proposal != BAMF_PROPOSAL_REFERENCE)
            return LLR * PrM * (P[3] / P[4]) / birth_q_ratio(A_X(pk_i0), A_Y(pk_i0));
        return LLR * (P[4] / P[3]) * PrM;
    }

    /* RJMCMC::gSplit (:1389-1485).  The reference does not test the
     * proposal's bounds here. */
    __device__ __forceinline__ int propose_gsplit()
    {
        if (an < 2) return ACT_SKIP;
        copyA2T();
        float Ua = urand();
        int jj = min((int)floorf((float)an * Ua), an - 1);
        int Np = closestMulti(jj, 2 * sigma);
        if (lane == 0) cl[Np] = jj;
        __syncwarp();
        Np++;
        if (Np == 1) return ACT_SKIP;
        float I0 = 0.0f, X0 = 0.0f, Y0 = 0.0f;
        for (int n = 0; n < Np; ++n) {
            int c = cl[n];
            I0 = I0 + A_I(c);
            X0 = X0 + A_X(c);
            Y0 = Y0 + A_Y(c);
        }
        float u1 = 0.3f * randn();
        float u2 = 0.3f * randn();
        float u3 = (1.0f / (float)Np) * urand();
        for (int n = 0; n < Np; ++n) {
            int c = cl[n];
            float aXc = A_X(c), aYc = A_Y(c), aIc = A_I(c);
            setT(c, (1.0f - u3) * aIc, (aXc - u3 * (X0 / (float)Np + u1)) / (1.0f - u3),
                 (aYc - u3 * (Y0 / (float)Np + u2)) / (1.0f - u3));
            if (!EXACT) a_dirty |= 1u << c;
        }
        addT(u3 * I0, X0 / (float)Np + u1, Y0 / (float)Np + u2, 1);
        pk_move = MV_GSPLIT;
        pk_type = 8;
        pk_i0 = Np;
        pk_f0 = u1;
        pk_f1 = u2;
        pk_f2 = u3;
        pk_f3 = I0;
        pk_c1 = pk_c2 = -1;
        if (t_overflow) {
            overflow++;
            return ACT_REJECT;
        }
        return ACT_EVAL;
    }
    __device__ __forceinline__ float finish_gsplit(float LLR)
    {
        int Np = pk_i0;
        float u1 = pk_f0, u2 = pk_f1, u3 = pk_f2, I0 = pk_f3;
        float PrI = 1.0f, tmpCurrent, tmpProposed;
        for (int n = 0; n < Np; ++n) {
            int c = cl[n];
            tmpCurrent = sob(A_S(c), A_I(c));
            tmpProposed = sob(T_S(n), T_I(c));
            PrI = PrI * tmpProposed / tmpCurrent;
        }
        tmpProposed = sob(T_S(tn - 1), T_I(tn - 1));
        PrI = PrI * (tmpProposed);
        float PDFu1 = normpdf(u1, 0.0f, 0.4f);
        float PDFu2 = normpdf(u2, 0.0f, 0.4f);
        float PDFu3 = (float)Np;
        float Us = 1.0f / (PDFu1 * PDFu2 * PDFu3);
        float NEm = nsignalA();
        float PrM = MeanN / (NEm + 1.0f);
        const bamf_mcmc_params &p = K->p;
        float Area = (float)(((float)X + p.Bnd_out) * ((float)Y + p.Bnd_out));
        float PrX = 1.0f / Area;
        float Jacob = I0 / MT::powf_(1.0f - u3, (float)(Np + 1));
        return LLR * PrI * PrX * Us * Jacob * PrM * (P[5] / P[6]);
    }

    /* RJMCMC::gMerge (:1487-1584). */
    __device__ __forceinline__ int propose_gmerge()
    {
        if (an < 3) return ACT_SKIP;
        copyA2T();
        float Ua = urand();
        int jj = min((int)floorf((float)an * Ua), an - 1);
        int Np = closestMulti(jj, 3 * sigma);
        if (Np == 0) return ACT_SKIP;
        float aIj = A_I(jj), aXj = A_X(jj), aYj = A_Y(jj);
        float I0 = aIj;
        for (int n = 0; n < Np; ++n) I0 = I0 + A_I(cl[n]);
        float XX0 = 0.0f, YY0 = 0.0f;
        float U3 = aIj / I0;
        for (int n = 0; n < Np; ++n) {
            int c = cl[n];
            float aIc = A_I(c), aXc = A_X(c), aYc = A_Y(c);
            float nX = U3 * aXj + (1.0f - U3) * aXc;
            XX0 = XX0 + U3 * aXj + (1.0f - U3) * aXc;
            float nY = U3 * aYj + (1.0f - U3) * aYc;
            YY0 = YY0 + U3 * aYj + (1.0f - U3) * aYc;
            setT(c, aIc / (1.0f - U3), nX, nY);
            if (!EXACT) a_dirty |= 1u << c;
        }
        float U1 = aXj - XX0 / (float)Np;
        float U2 = aYj - YY0 / (float)Np;
        float PrI = 1.0f, tmpProposed, tmpCurrent;
        for (int n = 0; n < Np; ++n) {
            int c = cl[n];
            tmpProposed = sob(T_S(c), T_I(c));
            tmpCurrent = sob(A_S(c), A_I(c));
            PrI = PrI * (tmpCurrent / tmpProposed);
        }
        tmpCurrent = sob(A_S(jj), aIj);
        PrI = PrI * tmpCurrent;
        if (!EXACT) a_dirty |= 1u << jj;
        removeT(jj);
        pk_move = MV_GMERGE;
        pk_type = 9;
        pk_i0 = Np;
        pk_f0 = U1;
        pk_f1 = U2;
        pk_f2 = U3;
        pk_f3 = I0;
        pk_f4 = PrI;
        pk_c1 = pk_c2 = -1;
        return ACT_EVAL;
    }
    __device__ __forceinline__ float finish_gmerge(float LLR)
    {
        int Np = pk_i0;
        float U1 = pk_f0, U2 = pk_f1, U3 = pk_f2, I0 = pk_f3, PrI = pk_f4;
        float PDFu1 = normpdf(U1, 0.0f, 0.4f);
        float PDFu2 = normpdf(U2, 0.0f, 0.4f);
        float PDFu3 = (float)Np;
        float Us = 1.0f / (PDFu1 * PDFu2 * PDFu3);
        float NEm = nsignalA();
        float PrM = NEm / MeanN;
        const bamf_mcmc_params &p = K->p;
        float Area = (float)(((float)X + p.Bnd_out) * ((float)Y + p.Bnd_out));
        float PrX = 1.0f / Area;
        float Jacob = I0 / MT::powf_(1.0f - U3, (float)(Np + 1));
        float PR = LLR / (PrI * PrX * Us * Jacob * PrM * (P[5] / P[6]));
        if (PDFu1 == 0.0f || PDFu2 == 0.0f) PR = -1.0f;
        return PR;
    }

    /* RJMCMC::backFore (:1586-1627): relabels in place, records nothing. */
    __device__ __forceinline__ void mv_backfore()
    {
        if (an == 0) return;
        if (K->p.IsBackg == 0) return;
        float Ua = urand();
        int nn = min((int)floorf((float)an * Ua), an - 1);
        float In = A_I(nn);
        int Sn = A_S(nn);
        float BackP = findPDF(K->back, In);
        float SignalP = findPDF(K->sig, In);
        int ns = Sn;
        if (Sn == 1) {
            if (SignalP != 0.0f) {
                float PrSig = BackP / SignalP;
                if (PrSig > urand()) ns = 0;
            } else {
                ns = 0;
            }
        } else {
            if (BackP != 0.0f) {
                float PrSig = SignalP / BackP;
                if (PrSig > urand()) ns = 1;
            } else {
                ns = 1;
            }
        }
        if (lane == nn) aS = ns;
    }

    /* One jump of start_Chain (:693-717, :725-748): W = this phase's
     * cumulative probabilities, V = PV_Burnin for the gSplit/gMerge slots. */
    __device__ __forceinline__ void step(const float *V, const float *W, float t)
    {
        int act;
        if (t < W[0]) act = propose_jump();
        else if (t >= W[0] && t < W[1]) act = propose_split();
        else if (t >= W[1] && t < W[2]) act = propose_merge();
        else if (t >= W[2] && t < W[3]) act = propose_birth();
        else if (t >= W[3] && t < W[4]) act = propose_death();
        else if (t >= V[4] && t < V[5]) act = propose_gsplit();
        else if (t >= V[5] && t < V[6]) act = propose_gmerge();
        else {
            mv_backfore();
            act = ACT_SKIP;
        }
        float LLR = 0.0f, PR = 0.0f;
        int accept = 0;
        if (act == ACT_EVAL) {
            LLR = llr();
            switch (pk_move) {
            case MV_JUMP: PR = finish_jump(LLR); break;
            case MV_SPLIT: PR = finish_split(LLR); break;
            case MV_MERGE: PR = finish_merge(LLR); break;
            case MV_BIRTH: PR = finish_birth(LLR); break;
            case MV_DEATH: PR = finish_death(LLR); break;
            case MV_GSPLIT: PR = finish_gsplit(LLR); break;
            default: PR = finish_gmerge(LLR); break;
            }
            accept = (urand() < PR);
            if (accept) {
                if (pk_c1 >= 0) cinc(pk_c1);
                if (pk_c2 >= 0) cinc(pk_c2);
                accept_T();
            }
        }
        if (act >= ACT_REJECT) record2(LLR, PR, pk_type, accept);
        if (act >= ACT_GRIDS) update_grids();
    }

    /* RJMCMC::start_Chain (:685-750). */
    /* Move-synchronous chain (fast mode): every warp of the CTA takes the
     * same move type and jump sub-branch at each jump, drawn from a stream
     * shared by the CTA, and the warps meet at a barrier before each jump,
     * so the warps of an SM run the same code.  For each chain the move
     * choice is still i.i.d. with the configured probabilities and
     * independent of its state, so its transition kernel is unchanged.
     * Warps without a ROI (the tail of the queue) only take the barriers. */
    __device__ __forceinline__ void run_chain_sync(bool active, uint32_t grp)
    {
        const bamf_mcmc_params &p = K->p;
        use_shared_ub = true;
        int since_rebuild = 0;
        const int total = p.N_Burnin + p.N_Trials;
        for (int n = 0; n < total; ++n) {
            __syncthreads();
            if (n == 0 || n == p.N_Burnin) {
                is_burnin = n < p.N_Burnin;
                /* the reference's ratios see the cumulative trial vector
                 * (LibRJMCMC.cpp:721-722); the other proposals use the raw one */
                const float *Pt = K->proposal == BAMF_PROPOSAL_REFERENCE ? K->PVT : p.P_Trials;
                for (int k = 0; k < 8; ++k) P[k] = is_burnin ? p.P_Burnin[k] : Pt[k];
            }
            if (!active) continue;
            /* the next jumps' shared draws, a lane each */
            if ((n & (MOVE_AHEAD - 1)) == 0) {
                __syncwarp();
                ahead[lane] = shared_uniform(K->seed, grp, (uint32_t)(n + lane), 0u);
                ahead[MOVE_AHEAD + lane] = shared_uniform(K->seed, grp, (uint32_t)(n + lane), 1u);
                __syncwarp();
            }
            const float t = ahead[n & (MOVE_AHEAD - 1)];
            shared_ub = ahead[MOVE_AHEAD + (n & (MOVE_AHEAD - 1))];
            step(K->PVB, is_burnin ? K->PVB : K->PVT, t);
            if (++since_rebuild == 512) {
                rebuild_model();
                since_rebuild = 0;
            }
        }
    }

    __device__ __forceinline__ void run_chain()
    {
        const bamf_mcmc_params &p = K->p;
        is_burnin = 1;
        for (int k = 0; k < 8; ++k) P[k] = p.P_Burnin[k];
        int since_rebuild = 0;
        for (int n = 0; n < p.N_Burnin; ++n) {
            float t = urand();
            step(K->PVB, K->PVB, t);
            if (!EXACT && ++since_rebuild == 512) {
                rebuild_model();
                since_rebuild = 0;
            }
        }
        is_burnin = 0;
        for (int k = 0; k < 8; ++k) P[k] = K->PVT[k];
        for (int n = 0; n < p.N_Trials; ++n) {
            float t = urand();
            step(K->PVB, K->PVT, t);
            if (!EXACT && ++since_rebuild == 512) {
                rebuild_model();
                since_rebuild = 0;
            }
        }
    }
};

/* Loads ROI `roi` into a warp's carve-out and sets up its chain (the
 * set-up of cRJMCMC.cpp:103-148).  Returns false, with the ROI's status set,
 * when the ROI does not fit the launch. */
template <bool EXACT, bool NUM, int TEAM>
__device__ __forceinline__ bool begin_roi(ChainWarp<EXACT, NUM, TEAM> &w, const SamplerConsts *Kp, const SamplerBatch &Bt,
                                          float *sw, int roi)
{
    const int lane = w.lane;
    w.roi = roi;
    int X = Bt.xsize[roi], Y = Bt.ysize[roi];
    w.X = X;
    w.Y = Y;
    w.npix = X * Y;
    w.px_dx = w.STEP / Y;
    w.px_dy = w.STEP - (w.STEP / Y) * Y;
    int npix_max = EXACT ? exact_npix(Bt.side_max) : Bt.side_max * Bt.side_max;
    w.D = sw;
    w.M = sw + npix_max;
    w.Mt = sw + 2 * npix_max;
    float *scm_smem = nullptr;
    if (EXACT) {
        w.E = sw + 3 * npix_max;
        scm_smem = sw + 4 * npix_max;
        w.NX = sw + 5 * npix_max;
        w.NY = w.NX + EXACT_ROWS * Bt.side_max;
        w.ubuf = w.NY + EXACT_ROWS * Bt.side_max;
        w.SX = w.SY = nullptr;
        w.cl = (int *)(w.ubuf + UBUF);
        w.ahead = nullptr;
        w.arow = w.trow = -1;
    } else {
        const int rs = 2 * FAST_ROWS * Bt.side_max;
        w.E = nullptr;
        w.NX = w.NY = nullptr;
        w.SX = sw + 3 * npix_max;
        w.SY = w.SX + rs;
        w.ubuf = sw + ((3 * npix_max + 2 * rs + 3) & ~3);
        w.ahead = w.ubuf + UBUF;
        w.cl = (int *)(w.ahead + 2 * MOVE_AHEAD);
    }
    int n0 = Bt.init_n ? Bt.init_n[roi] : 0;
    bool ok = X >= 1 && Y >= 1 && X <= Bt.side_max && Y <= Bt.side_max && n0 <= BAMF_NMAX;
    if (!ok) {
        if (lane == 0 && Bt.status) Bt.status[roi] = BAMF_ERR_TOO_LARGE;
        return false;
    }
    const float *src = Bt.data + Bt.offsets[roi];
    const float *scm_src = Bt.scmos ? Bt.scmos + Bt.offsets[roi] : nullptr;
    for (int p = lane; p < w.npix; p += 32) {
        w.D[p] = src[p];
        if (EXACT) scm_smem[p] = scm_src ? scm_src[p] : 0.0f;
    }
    w.scm = EXACT ? scm_smem : scm_src;
    {
        const int k = lane;
        const bool isN = (k <= C_N_death) || (k >= C_N_jumpFg && k <= C_N_deathFg) ||
                         (k >= C_N_jumpBg && k <= C_N_deathBg);
        w.cnt = isN ? 1 : 0;
    }
    float s = Bt.psf_sigma ? Bt.psf_sigma[roi] : Kp->p.PSFsigma;
    w.sigma = s;
    w.Cst = 1.0f / (s * sqrtf(2.0f));
    if (NUM) {
        const int32_t *P = Kp->p.PSFsize;
        w.pn0 = P[0];
        w.pn01 = P[0] * P[1];
        w.pn012 = w.pn01 * P[2];
        w.ptot = w.pn012 * P[3];
        w.pos = P[3];
        const int slot = Bt.psf_slot ? Bt.psf_slot[roi] : 0;
        if (slot < 0 || slot >= Bt.n_psf) {
            if (lane == 0 && Bt.status) Bt.status[roi] = BAMF_ERR_INVALID_ARG;
            return false;
        }
        w.psf = Bt.sampled_psf + (int64_t)slot * w.ptot;
    } else {
        w.psf = nullptr;
    }
    w.MeanN = Kp->p.Rho * (float)X * (float)Y;
    /* start state (cRJMCMC.cpp:120-133) */
    w.an = n0;
    w.aI = w.aX = w.aY = 0.0f;
    w.aS = 1;
    if (n0 > 0 && lane < n0) {
        const float *ixy = Bt.init_ixy + (size_t)roi * 3 * BAMF_NMAX;
        w.aI = ixy[lane];
        w.aX = ixy[BAMF_NMAX + lane];
        w.aY = ixy[2 * BAMF_NMAX + lane];
    }
    w.aBG = Bt.init_bg ? Bt.init_bg[roi] : Kp->bg0;
    if (w.aBG == 0.0f) w.aBG = 1.0f;
    w.pdf_aBG = w.findPDF(Kp->off, w.aBG);
    w.aABG = 0.0f;
    w.aBBG = 0.0f;
    w.seed = Kp->seed;
    w.chain = Bt.chain_ids ? Bt.chain_ids[roi] : (uint32_t)roi;
    w.idx = Bt.rng_offset ? Bt.rng_offset[roi] : 0u;
    w.base = w.idx >> 2;
    w.idx &= 3u;
    w.refill();
    w.entries = 0;
    w.overflow = 0;
    w.n_llr = 0;
    w.a_dirty = w.t_dirty = 0u;
    w.use_shared_ub = false;
    w.shared_ub = 0.0f;
    w.rec_n[0] = w.rec_n[1] = 0;
    if (!EXACT && Bt.model_drift && lane == 0) Bt.model_drift[roi] = 0.0f;
    __syncwarp();
    w.rebuild_model();
    return true;
}

/* Writes the chain's per-ROI results. */
template <bool EXACT, bool NUM, int TEAM>
__device__ __forceinline__ void end_roi(ChainWarp<EXACT, NUM, TEAM> &w, const SamplerBatch &Bt)
{
    const int lane = w.lane, roi = w.roi;
    if (Bt.final_n && lane == 0) Bt.final_n[roi] = w.an;
    if (Bt.final_state) {
        float *fs = Bt.final_state + (size_t)roi * (4 + 4 * BAMF_NMAX);
        if (lane == 0) {
            fs[0] = w.aBG; fs[1] = w.aABG; fs[2] = w.aBBG; fs[3] = (float)w.an;
        }
        fs[4 + lane] = lane < w.an ? w.aI : 0.0f;
        fs[4 + BAMF_NMAX + lane] = lane < w.an ? w.aX : 0.0f;
        fs[4 + 2 * BAMF_NMAX + lane] = lane < w.an ? w.aY : 0.0f;
        fs[4 + 3 * BAMF_NMAX + lane] = lane < w.an ? (float)w.aS : 0.0f;
    }
    __syncwarp();
    static_assert(C_COUNT <= 32, "a lane per counter");
    if (Bt.counters && lane < C_COUNT) Bt.counters[(size_t)roi * C_COUNT + lane] = w.cnt;
    if (Bt.chains && lane == 0) {
        Bt.chains[2 * roi].n_entries = min(w.entries, Bt.chains[2 * roi].capacity_entries);
        Bt.chains[2 * roi + 1].n_entries = min(w.entries, Bt.chains[2 * roi + 1].capacity_entries);
        Bt.chains[2 * roi].n_records = w.rec_n[0];
        Bt.chains[2 * roi + 1].n_records = w.rec_n[1];
    }
    if (lane == 0) {
        if (Bt.n_entries) Bt.n_entries[roi] = w.entries;
        if (Bt.uniforms_used)
            Bt.uniforms_used[roi] = 4u * w.base + w.idx - (Bt.rng_offset ? Bt.rng_offset[roi] : 0u);
        if (Bt.overflow) Bt.overflow[roi] = w.overflow;
        if (Bt.llr_evals) Bt.llr_evals[roi] = w.n_llr;
        if (Bt.status) Bt.status[roi] = BAMF_OK;
    }
    __syncwarp();
}

/* Persistent sampler: each warp pulls ROI ids from the work queue and runs
 * their chains one after another. */
template <bool EXACT, bool NUM>
__global__ void __launch_bounds__(128, 4) rjmcmc_kernel(const __grid_constant__ SamplerConsts Kc,
                                                     const __grid_constant__ SamplerBatch Bc)
{
    extern __shared__ __align__(16) float smem_raw[];
    const SamplerBatch &Bt = Bc;
    int warp = threadIdx.x >> 5;
    int lane = threadIdx.x & 31;
    float *sw = smem_raw + (size_t)warp * warp_smem_floats(Bt.side_max, EXACT);
    ChainWarp<EXACT, NUM> w;
    w.K = &Kc;
    w.B = &Bc;
    w.lane = lane;
    int q_begin = 0, q_end = Bt.n_rois;
    if (Bt.class_range) {
        q_begin = Bt.class_range[2 * Bt.cls];
        q_end = Bt.class_range[2 * Bt.cls + 1];
    }
    for (;;) {
        int slot = 0;
        if (lane == 0) slot = q_begin + atomicAdd(Bt.queue, 1);
        slot = __shfl_sync(BAMF_FULL, slot, 0);
        if (slot >= q_end) break;
        int roi = Bt.order ? Bt.order[slot] : slot;
        if (!begin_roi(w, &Kc, Bt, sw, roi)) continue;
        w.run_chain();
        end_roi(w, Bt);
    }
}

/* Exact sampler for few ROIs: a CTA of TEAM warps runs one chain at a time.
 * The first warp runs the chain; the others take their share of every
 * proposal's pixels (the model and the likelihood-ratio terms, 40% of a
 * chain's time on one warp).  The terms are then added by the first warp in
 * pixel order, so the chain is the same.  A chain is latency-bound (3,100 warp
 * instructions of the team per jump, issue slots 11% busy).  16x16, 3000+3000
 * jumps, 200 ROIs: 42.1 ms with a warp per chain, 35.6 ms with teams of four; one
 * ROI: 37.7 and 30.1 ms in the same run. */
template <int TEAM>
__global__ void __launch_bounds__(32 * TEAM, 2) rjmcmc_kernel_team(const __grid_constant__ SamplerConsts Kc,
                                                                const __grid_constant__ SamplerBatch Bc)
{
    extern __shared__ __align__(16) float smem_raw[];
    __shared__ TeamCmd cmd;
    const SamplerBatch &Bt = Bc;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ChainWarp<true, false, TEAM> w;
    w.K = &Kc;
    w.B = &Bc;
    w.lane = lane;
    w.cmd = &cmd;
    if (warp > 0) {
        w.team_serve(warp);
        return;
    }
    int q_begin = 0, q_end = Bt.n_rois;
    if (Bt.class_range) {
        q_begin = Bt.class_range[2 * Bt.cls];
        q_end = Bt.class_range[2 * Bt.cls + 1];
    }
    for (;;) {
        int slot = 0;
        if (lane == 0) slot = q_begin + atomicAdd(Bt.queue, 1);
        slot = __shfl_sync(BAMF_FULL, slot, 0);
        if (slot >= q_end) break;
        int roi = Bt.order ? Bt.order[slot] : slot;
        if (!begin_roi(w, &Kc, Bt, smem_raw, roi)) continue;
        w.run_chain();
        end_roi(w, Bt);
    }
    if (lane == 0) cmd.ask = TeamCmd::ASK_END;
    w.team_sync();
}

/* Move-synchronous persistent sampler (fast arithmetic): the CTA pulls one
 * ROI per warp at a time and its warps run their chains in lockstep, one
 * barrier per jump, with the move type and jump sub-branch shared across the
 * CTA (run_chain_sync). */
template <bool NUM, int MIN_CTAS>
__global__ void __launch_bounds__(MIN_CTAS == 1 ? 32 * BAMF_SYNC_GROUP : 256, MIN_CTAS) rjmcmc_kernel_sync(const __grid_constant__ SamplerConsts Kc,
                                                          const __grid_constant__ SamplerBatch Bc)
{
    extern __shared__ __align__(16) float smem_raw[];
    __shared__ int grp_base;
    const SamplerBatch &Bt = Bc;
    const int nwarps = blockDim.x >> 5;
    int warp = threadIdx.x >> 5;
    int lane = threadIdx.x & 31;
    float *sw = smem_raw + (size_t)warp * warp_smem_floats(Bt.side_max, false);
    ChainWarp<false, NUM> w;
    w.K = &Kc;
    w.B = &Bc;
    w.lane = lane;
    int q_begin = 0, q_end = Bt.n_rois;
    if (Bt.class_range) {
        q_begin = Bt.class_range[2 * Bt.cls];
        q_end = Bt.class_range[2 * Bt.cls + 1];
        const int count = q_end - q_begin;
        if (Bt.count_max > 0 && (count <= Bt.count_min || count > Bt.count_max)) return;
    }
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) grp_base = q_begin + atomicAdd(Bt.queue, nwarps);
        __syncthreads();
        int base = grp_base;
        if (base >= q_end) break;
        int slot = base + warp;
        bool active = slot < q_end;
        if (active) {
            int roi = Bt.order ? Bt.order[slot] : slot;
            active = begin_roi(w, &Kc, Bt, sw, roi);
        }
        /* the shared move stream is keyed by the slot group of BAMF_SYNC_GROUP
         * ROIs, not by the CTA, so a chain's moves (and its result) do not
         * depend on the launch's warps per block (any divisor of the group) */
        w.run_chain_sync(active, (uint32_t)(q_begin + (base - q_begin) / BAMF_SYNC_GROUP * BAMF_SYNC_GROUP));
        if (active) end_roi(w, Bt);
    }
}

}  // namespace bamf

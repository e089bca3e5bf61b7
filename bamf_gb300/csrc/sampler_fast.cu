/*
 * sampler_fast.cu - the fast sampler with the Gaussian PSF: hardware SFU
 * math, incremental model updates, warp-tree reductions, and
 * move-synchronous CTAs (the warps of a CTA draw the move type and jump
 * sub-branch from one shared stream and meet at a barrier before each jump,
 * so an SM's warps run the same code and the instruction cache stops
 * thrashing; each chain's move choice stays i.i.d. with the configured
 * probabilities and independent of its state).  Also the fast launchers,
 * which pick the likelihood model's build.
 */
#include <cmath>

#include "sampler_kernel.cuh"
#include "sampler_launch.h"

namespace bamf {

cudaError_t launch_fast_gauss(const SamplerConsts &K, const SamplerBatch &B, size_t smem, int blocks, int threads,
                              int min_ctas, cudaStream_t stream)
{
    if (min_ctas == 1) return launch_kernel(rjmcmc_kernel_sync<false, 1>, K, B, smem, blocks, threads, stream);
    return min_ctas == 3 ? launch_kernel(rjmcmc_kernel_sync<false, 3>, K, B, smem, blocks, threads, stream)
                         : launch_kernel(rjmcmc_kernel_sync<false, 2>, K, B, smem, blocks, threads, stream);
}

int occupancy_fast_gauss(size_t smem, int threads, int min_ctas)
{
    if (min_ctas == 1) return resident_ctas(rjmcmc_kernel_sync<false, 1>, smem, threads);
    return min_ctas == 3 ? resident_ctas(rjmcmc_kernel_sync<false, 3>, smem, threads)
                         : resident_ctas(rjmcmc_kernel_sync<false, 2>, smem, threads);
}

cudaError_t launch_rjmcmc_fast(const SamplerConsts &K, const SamplerBatch &B, int side_max, int blocks,
                               int warps_per_block, int min_ctas, cudaStream_t stream)
{
    if (warps_per_block < 1 || BAMF_SYNC_GROUP % warps_per_block != 0) return cudaErrorInvalidValue;
    if (min_ctas < 1 || min_ctas > 3) return cudaErrorInvalidValue;
    size_t smem = (size_t)warp_smem_floats(side_max, false) * sizeof(float) * warps_per_block;
    (void)K.sync_moves; /* always move-synchronous in fast arithmetic */
    return K.opt_model == 1 ? launch_fast_num(K, B, smem, blocks, 32 * warps_per_block, min_ctas, stream)
                            : launch_fast_gauss(K, B, smem, blocks, 32 * warps_per_block, min_ctas, stream);
}

int blocks_per_sm_fast(int side_max, int warps_per_block, int min_ctas, int opt_model)
{
    size_t smem = (size_t)warp_smem_floats(side_max, false) * sizeof(float) * warps_per_block;
    return opt_model == 1 ? occupancy_fast_num(smem, 32 * warps_per_block, min_ctas)
                          : occupancy_fast_gauss(smem, 32 * warps_per_block, min_ctas);
}

/* A batch of n ROIs with w chains resident per SM, in units of a round of 16:
 * the first round costs `a` (it holds the brightest ROIs), later ones 0.77 a, a
 * last one that is not full 0.25 a more; less than one round costs between 0.68
 * and 1 of it.  Fitted to batches of 2,400 to 10,000 ROIs of 8, 16 and 24 px:
 * within 8%.
 * `whole`: the w chains are one CTA, so that less than a round leaves SMs without
 * any instead of giving every SM fewer. */
static float batch_cost(int n, int sms, int w, float a, bool whole)
{
    const float x = (float)n / (float)(w * sms);
    if (x <= 1.0f) return whole ? a : a * (0.68f + 0.32f * x);
    const float frac = x - floorf(x);
    return a * (1.0f + 0.77f * (x - 1.0f) + (frac > 0.02f ? 0.25f : 0.0f));
}

int best_fast_shape(int side_max, int opt_model, int n_rois, int sms, int *warps_per_block, int *min_ctas)
{
    /* A batch that one CTA per SM can hold: the fewest chains per CTA that do,
     * on the register budget without spills.  Chains of a CTA wait for each
     * other at every jump, and an SM's instruction cache serves one or a few
     * move streams either way (500 + 500 jumps of uneven ROIs, us, with 1 / 2 / 4 /
     * 8 chains per CTA against the shapes with the most resident chains: 64
     * ROIs 4759 / 5076 / 5468 / 6000 against 7006, 300 ROIs 5606 / 5347 / 5703 /
     * 6213 against 7753, 1216 ROIs 10827 / 9254 / 7530 / 6716 against 8772). */
    for (int w = 1; w <= 8; w *= 2)
        if (n_rois <= w * sms) {
            const int per = blocks_per_sm_fast(side_max, w, 2, opt_model);
            if (per > 0) {
                *warps_per_block = w;
                *min_ctas = 2;
                return per;
            }
        }
    int best_w = 0, best_wpb = 8, best_mc = 2, best_per = 0;
    const int cand[3] = {8, 4, 2};
    for (int mc = 2; mc <= 3; ++mc)
        for (int i = 0; i < 3; ++i) {
            int per = blocks_per_sm_fast(side_max, cand[i], mc, opt_model);
            if (per * cand[i] > best_w) {
                best_w = per * cand[i];
                best_wpb = cand[i];
                best_mc = mc;
                best_per = per;
            }
        }
    /* Up to side 20, one CTA of a whole move-stream group per SM (all of the SM's
     * warps on one instruction stream) instead of three CTAs of 8 chains, when it
     * keeps as many chains resident and fills its rounds (250 + 250 jumps, us, one /
     * three: 16 px 2600 ROIs 3672 / 3399, 3380 3737 / 3748, 7300 5919 / 6752, 10,000
     * 8551 / 9963, 30,000 27183 / 27373; 20 px 7010 / 7723, 10660 / 11146 at 7300 and
     * 10,000; 24 px 8140 / 7876, 11726 / 11272). */
    const int group_per = side_max <= 20 && opt_model != 1 ? blocks_per_sm_fast(side_max, BAMF_SYNC_GROUP, 1, opt_model) : 0;
    const int group_w = group_per * BAMF_SYNC_GROUP;
    /* Two CTAs of 8 on the larger register budget run a round in 1 / 1.42 of the
     * time of three on the smaller (one CTA of 24: 1 / 1.25 at 8 to 12 px, 1 / 1.33 at
     * 16, 1 / 1.4 at 20), so which is faster depends on how full the last round is (16 px, 250 + 250
     * jumps: 2432 ROIs 2812 us against 3130 with three, 5000: 5568 against 5876, 7300: 6893
     * against 6752). */
    float best = best_w > 0 ? batch_cost(n_rois, sms, best_w, best_mc == 2 ? 1.0f : 1.42f, false) : INFINITY;
    if (group_w > 0 && group_w >= best_w) {
        const float c = batch_cost(n_rois, sms, group_w, side_max <= 12 ? 1.25f : side_max <= 16 ? 1.33f : 1.4f,
                                   group_per == 1);
        if (c < best) {
            best = c;
            best_wpb = BAMF_SYNC_GROUP;
            best_mc = 1;
            best_per = group_per;
        }
    }
    /* The costs are those of CTAs of 8 and 24 chains.  More, smaller CTAs keep a few
     * more chains resident where three of 8 do not fit, but an SM then runs as many
     * move streams (25 px, 3000 ROIs: 6.1 ms in five CTAs of 4, 4.7 in two of 8). */
    const int per2 = blocks_per_sm_fast(side_max, 8, 2, opt_model);
    if (per2 * 8 >= 16 && best_w > per2 * 8 &&
        (best_wpb < 8 || batch_cost(n_rois, sms, per2 * 8, 1.0f, false) < best)) {
        best_wpb = 8;
        best_mc = 2;
        best_per = per2;
    }
    *warps_per_block = best_wpb;
    *min_ctas = best_mc;
    return best_per;
}

}  // namespace bamf

"""The exact sampler's neighbour test at distances of every sign: a negative PSF width has no neighbours
(its distance limits 2 sigma and 3 sigma are negative), so group and merge moves pick as the oracle does."""
import numpy as np
import pytest

from bamf_gb300 import rjstruct, sampler, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [1.3, -1.3, -0.4, 1e-16, -1e-16, 1e3])
def test_neighbour_picks_equal_the_oracle(cuda_lib, oracle_port, sigma):
    rng = np.random.default_rng(17)
    x, y = rng.uniform(2, 12, 6), rng.uniform(2, 12, 6)
    roi = rng.poisson(synth.model_image(14, 14, x, y, [900.0] * 6, 10.0, 1.3)).astype(np.float32)
    rj = rjstruct.c0_rjstruct()
    rj.N_Burnin = rj.N_Trials = 200
    rj.P_Burnin = [0.3, 0.1, 0.1, 0.1, 0.1, 0.1, 0.1, 0.1]
    rj.P_Trials = [0.4, 0.1, 0.1, 0.05, 0.05, 0.1, 0.1, 0.1]
    p = rjstruct.mcmc_params(rj)
    p.PSFsigma = sigma
    args = (p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons)
    kw = dict(e0=([900.0] * 6, list(x), list(y), 10.0), rng=(23, 4, 0))
    got = sampler.crjmcmc_raw(roi, *args, arith="exact", **kw)
    ref = oracle_port.run_chain("port", roi, *args, **kw)
    for w in ("chain", "chain_test"):
        for k, a in got[w].items():
            b = ref[w][k].astype(a.dtype)
            assert a.shape == b.shape, (w, k)
            if a.dtype == np.float32:  # an NaN is an NaN
                assert ((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all(), (w, k)
            else:
                assert np.array_equal(a, b), (w, k)

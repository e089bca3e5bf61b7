"""The gaussMLE kernels at every kind of fit window (the unrolled sizes, one and two rounds of a
group's lanes per axis, the smallest and the largest) and at batch ends inside a block."""
import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 5, 7, 8, 9, 15, 16, 17, 21]


def _rois(sz, n, seed=0, s0=1.3, s1=1.3):
    """(sz, sz, n) Poisson ROIs, one emitter within a pixel of the middle."""
    rng = np.random.default_rng(seed)
    erf = np.vectorize(math.erf)
    i = np.arange(sz)[None, :]

    def prof(c, s):
        c, s = c[:, None], np.broadcast_to(np.asarray(s, float), (n,))[:, None] * math.sqrt(2.0)
        return 0.5 * (erf((i - c + 1) / s) - erf((i - c) / s))
    y, x = rng.uniform(sz / 2 - 1, sz / 2 + 1, (2, n))
    lam = rng.uniform(5, 30, n)[:, None, None] + rng.lognormal(math.log(1500), 0.3, n)[:, None, None] \
        * prof(y, s0)[:, :, None] * prof(x, s1)[:, None, :]
    return np.ascontiguousarray(np.transpose(rng.poisson(lam).astype(np.float32), (1, 2, 0)))


def _device(rois, n, it):
    import torch
    from bamf_gb300 import frontend
    flat = torch.from_numpy(np.ascontiguousarray(rois[:, :, :n].ravel(order="F"))).cuda()
    P, CR, LL = frontend.gauss_mle_device(flat, rois.shape[0], n, 1.3, it)
    torch.cuda.synchronize()
    return P.cpu().numpy().reshape(4, n).T, CR.cpu().numpy().reshape(4, n).T, LL.cpu().numpy()


@pytest.mark.parametrize("sz", SIZES)
def test_basic_fits_of_every_window(cuda_lib, sz):
    n = 17 if sz > 9 else 100
    rois = _rois(sz, n, seed=sz)
    # start values: sums of at most 21 + 21 positive terms, so 45 ulp of the largest value
    P, _, _ = _device(rois, n, 0)
    ref = oracle.gaussmle(rois, 1.3, 0, double=True)["P"]
    scale = np.stack([np.full(n, max(sz, 1)), np.full(n, max(sz, 1)),
                      4 * math.pi * 1.69 * rois.max((0, 1)), rois.max((0, 1))], 1)
    assert (np.abs(P - ref) <= 2e-5 * scale).all()
    if sz >= 5:  # four parameters are determined: the bounds the 7 px fits are held to elsewhere
        P, CR, LL = _device(rois, n, 10)
        ref = oracle.gaussmle(rois, 1.3, 10, double=True)
        rel = np.abs(P - ref["P"]) / np.maximum(np.abs(ref["P"]), 1e-3)
        assert np.median(rel) < 1e-5 and np.percentile(rel, 99) < 1e-3
        np.testing.assert_allclose(LL, ref["LL"], rtol=1e-3, atol=1e-2)
        relc = np.abs(CR - ref["CRLB"]) / np.abs(ref["CRLB"])
        assert np.percentile(relc, 99) < 1e-3
        # a fit does not depend on its place in a block or on the batch's end
        for m in (1, 15, 16):
            Pm, CRm, LLm = _device(rois, m, 10)
            np.testing.assert_array_equal(Pm, P[:m])
            np.testing.assert_array_equal(CRm, CR[:m])
            np.testing.assert_array_equal(LLm, LL[:m])

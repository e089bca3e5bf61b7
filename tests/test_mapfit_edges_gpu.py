"""The chain summaries where their loops end: no record, one, around a warp and a block of records and of
points, the largest count, truncated and short traces."""
import numpy as np
import pytest

from bamf_gb300 import mapfit
from oracle import mapfit_port

pytestmark = pytest.mark.gpu
S = mapfit_port.S


def _trace(rng, n, pos_len, ks, other=0.15):
    """[n][pos_len][record] states: ROI i's emitters scatter about ks[i] points 3 px apart, a few
    records hold another count."""
    t = np.full((n, pos_len, 5 + 3 * S), np.nan, np.float32)
    for i, k in enumerate(ks):
        t[i, :, 0] = 1.0
        t[i, :, 1] = np.where(rng.random(pos_len) < other, k + 1, k)
        t[i, :, 2:5] = rng.normal(10.0, 0.5, (pos_len, 3))
        perm = np.array([rng.permutation(k) for _ in range(pos_len)]).reshape(pos_len, k)
        for j, step in ((0, 3.0), (1, 2.0), (2, 100.0)):
            t[i, :, 5 + j * S:5 + j * S + k] = step * perm + rng.normal(0, 0.1, (pos_len, k)) + 1.0
    return t


@pytest.mark.parametrize("pos_len", [1, 2, 3, 31, 64, 66, 200, 255, 256])
def test_summaries_at_the_ends_of_their_loops(cuda_lib, pos_len):
    import torch
    rng = np.random.default_rng(pos_len)
    ks = np.array([0, 1, 2, 3, 4, 5, 8, 17, 31, 32], np.int32)
    n = len(ks)
    trace = _trace(rng, n, pos_len, ks)
    fixed = _trace(rng, n, pos_len, ks, other=0.0)  # refine_stats takes fixed-count chains
    for thin, entries in ((1, pos_len), (3, 3 * pos_len - 1), (2, 3 * pos_len), (4, 2), (1, 1), (1, 0)):
        ne = np.full(n, entries, np.int32)
        a = [torch.from_numpy(x).cuda() for x in (trace, ne, ks)]
        km = mapfit.map_kmeans(a[0], thin, a[1], a[2]).cpu().numpy()
        rs = mapfit.refine_stats(torch.from_numpy(fixed).cuda(), thin, a[1]).cpu().numpy()
        for i in range(n):
            for rec, ref in ((km, mapfit_port.map_kmeans(trace[i], thin, entries, ks[i])),
                             (rs, mapfit_port.refine_stats(fixed[i], thin, entries))):
                got = mapfit.unpack(rec[i:i + 1])
                assert got["N"][0] == ref["N"] and got["records"][0] == ref["records"]
                for name in ("X", "Y", "I", "X_SE", "Y_SE", "I_SE"):
                    np.testing.assert_allclose(got[name][0], ref[name], rtol=2e-4, atol=2e-5, equal_nan=True,
                                               err_msg=f"{pos_len} {thin} {entries} roi {i} {name}")

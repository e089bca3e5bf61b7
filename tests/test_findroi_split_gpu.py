"""The filter's two forms give the oracle's DoG bit for bit at the sizes where
they begin and end: rows and columns around the 16-row groups and 32-column
chunks, stacks around the number of frames that takes a CTA per frame, and
frames too large for a slot in more than one pass."""
import numpy as np
import pytest

import oracle
from bamf_gb300 import frontend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ys,xs,zs", [(1, 1, 1), (2, 3, 1), (15, 16, 2), (16, 17, 2), (33, 31, 3), (31, 33, 3),
                                      (33, 47, 3), (65, 190, 1), (250, 190, 1), (24, 25, 75), (24, 25, 76),
                                      (24, 28, 77), (40, 36, 151), (34, 32, 310), (400, 300, 110)])
def test_dog_bit_exact_at_the_edges_of_the_dispatch(cuda_lib, ys, xs, zs):
    import torch
    rng = np.random.default_rng(ys * 1000 + xs)
    st = np.asfortranarray(rng.poisson(20.0, (ys, xs, zs)).astype(np.float32))
    st[rng.integers(0, ys, zs), rng.integers(0, xs, zs), np.arange(zs)] = 4000.0
    want = oracle.findroi_dog(st, 1.3, 2.6)
    got = frontend.FindRoiDevice().dog(torch.from_numpy(st.ravel(order="F")).cuda(), ys, xs, zs, 1.3, 2.6)
    bad = np.flatnonzero(got.cpu().numpy().view(np.uint32) != want.view(np.uint32))
    assert bad.size == 0, (bad.size, bad[:5])

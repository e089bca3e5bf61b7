"""Small frames around the line between the filter's two forms: a frame's DoG is the same alone and inside a
stack that takes a CTA per frame."""
import numpy as np
import pytest

from bamf_gb300 import frontend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ys,xs", [(31, 32), (32, 32), (33, 33), (36, 36), (37, 32), (32, 37), (64, 64), (64, 68), (68, 68),
                                   (132, 32), (128, 64), (64, 128), (160, 32), (192, 32), (193, 32), (32, 129), (96, 96)])
def test_a_frame_alone_and_in_a_stack(cuda_lib, ys, xs):
    import torch
    rng = np.random.default_rng(ys * 1000 + xs)
    st = rng.poisson(20.0, (160, xs, ys)).astype(np.float32)
    st[np.arange(160), rng.integers(0, xs, 160), rng.integers(0, ys, 160)] = 4000.0
    a = torch.from_numpy(st).cuda()
    f = frontend.FindRoiDevice()
    whole = f.dog(a, ys, xs, 160).view(160, -1)
    for z0, z in ((0, 1), (7, 3), (100, 50)):
        part = f.dog(a[z0:z0 + z].contiguous(), ys, xs, z).view(z, -1)
        assert torch.equal(part.view(torch.int32), whole[z0:z0 + z].view(torch.int32)), (z0, z)

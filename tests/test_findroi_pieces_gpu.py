"""Frames copied from host memory in pieces: pieces cut to whole waves of the SMs, pieces cut to what
the link hides, several pieces per compaction, and a short last piece give the device call's ROIs and
their fits bit for bit."""
import numpy as np
import pytest

from bamf_gb300 import frontend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ys,xs,zs,chunk,short", [(256, 256, 700, 250, 40), (256, 256, 310, 153, 0),
                                                  (300, 290, 480, 150, 0), (350, 412, 90, 250, 0),
                                                  (64, 96, 1100, 250, 0), (40, 33, 9, 4, 3)])
def test_pieces_give_the_device_calls_rois_and_fits(cuda_lib, ys, xs, zs, chunk, short):
    import torch
    rng = np.random.default_rng(ys + zs)
    g = torch.Generator().manual_seed(ys * zs)
    host = torch.poisson(torch.full((zs, xs, ys), 20.0), generator=g)
    k = torch.arange(7) - 3.0
    spot = 800.0 * torch.exp(-(k[:, None] ** 2 + k[None, :] ** 2) / (2 * 1.3 ** 2))
    for z in range(zs):
        for _ in range(4):
            x, y = rng.integers(0, xs - 7), rng.integers(0, ys - 7)
            host[z, x:x + 7, y:y + 7] += spot.round()
    host = host.reshape(-1).pin_memory()
    fr = frontend.FindRoiDevice()
    a = fr.run(host.cuda(), ys, xs, zs, boxsize=7)
    torch.cuda.synchronize()
    count = int(a["count"].item())
    assert count > zs
    c = count - short  # a capacity below the count: the first ROIs only
    b = fr.run_fit_pinned(host, ys, xs, zs, boxsize=7, psf_sigma=1.3, iterations=10, chunk_frames=chunk, capacity=c)
    torch.cuda.synchronize()
    assert int(b["count"].item()) == count
    for name in ("coords", "corners", "stack"):
        assert torch.equal(a[name][:c], b[name][:c]), name
    P, CR, LL = frontend.gauss_mle_device(a["stack"][:c].contiguous(), 7, c, 1.3, 10)
    torch.cuda.synchronize()
    for want, got in ((P, b["P"]), (CR, b["CR"]), (LL, b["LL"])):
        assert torch.equal(want.view(torch.int32).reshape(-1), got[..., :c].reshape(-1).view(torch.int32))

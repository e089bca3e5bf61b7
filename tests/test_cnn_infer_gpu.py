"""The fused inference kernel: every ROI's tables are independent of the batch
size (fewer ROIs than groups, odd counts, one more than a full wave) and of the
output's alignment, and match the network in plain PyTorch with BF16 rounding
at the points where the kernels store BF16."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(cuda_lib):
    import torch
    from bamf_gb300 import learned
    g = torch.Generator().manual_seed(5)
    net = learned.ProposalNet(3)
    p = net.get_params()
    p = p + 0.05 * torch.randn(p.size, generator=g).numpy().astype(np.float32) * (p == 0)  # biases
    net.set_params(p)
    data = learned.generate(1300, seed=8)["data"]
    return net, p, data, {k: v.cpu() for k, v in net.infer(data).items()}


@pytest.mark.parametrize("n", [1, 2, 3, 607, 609, 1217])
def test_tables_do_not_depend_on_the_batch(net, n):
    m, _, data, full = net
    out = m.infer(data[:n].contiguous())
    for k, per in (("cdf", 256), ("sub", 4096), ("count_logits", None)):
        a, b = out[k].cpu(), full[k][:n * per] if per else full[k][:n]
        assert a.numpy().tobytes() == b.numpy().tobytes(), k


def test_output_that_is_not_32_byte_aligned(net):
    import torch
    from bamf_gb300 import learned
    m, _, data, full = net
    n = 5
    cdf = torch.empty(n * 256 + 1, device="cuda")
    sub = torch.empty(n * 4096 + 1, device="cuda")
    st = learned._lib().bamf_cnn_infer(m._h, data.data_ptr(), n, cdf[1:].data_ptr(), sub[1:].data_ptr(), None, None)
    assert st == 0
    assert sub[1:].cpu().numpy().tobytes() == full["sub"][:n * 4096].numpy().tobytes()
    assert cdf[1:].cpu().numpy().tobytes() == full["cdf"][:n * 256].numpy().tobytes()
    assert learned._lib().bamf_cnn_infer(m._h, None, 0, None, None, None, C.c_void_p(0)) == 0


def test_tables_match_the_torch_network(net):
    import torch
    from oracle import cnn_torch
    _, p, data, full = net
    d = data[:64].cpu()
    with torch.no_grad():
        cdf, sub = cnn_torch.birth_tables(torch.from_numpy(p), d)
        _, cnt, _ = cnn_torch.forward(torch.from_numpy(p), d)
    # a BF16 rounding that falls the other way (2^-9 of one activation) is the
    # largest difference; the tolerances of the layer-by-layer kernels' test
    assert np.abs(full["cdf"][:64 * 256].numpy() - cdf.numpy()).max() < 5e-3
    assert np.abs(full["count_logits"][:64].numpy() - cnt.numpy()).max() < 2e-2
    assert np.abs(full["sub"][:64 * 4096].numpy() - sub.numpy()).max() < 5e-3

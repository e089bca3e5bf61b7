"""The training kernels where their loops end: batches around the persistent grids' sizes, and the
optimiser's step with the operands it packs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 303, 305, 913])
def test_gradients_at_batch_ends(cuda_lib, n):
    import torch

    from bamf_gb300 import learned
    from oracle import cnn_torch
    net = learned.ProposalNet(seed=7)
    b = learned.generate(n, seed=19)
    loss, grad = net.loss_grad(b)
    loss2, grad2 = net.loss_grad(b)
    np.testing.assert_array_equal(grad, grad2)  # fixed summation orders
    host = {k: v.cpu().numpy() for k, v in b.items()}
    theta = torch.tensor(net.get_params()).requires_grad_(True)
    L = cnn_torch.loss(theta, torch.tensor(host["data"]), host["n_em"], host["xyi"], bf16=True)
    (g,) = torch.autograd.grad(L, theta)
    assert loss == pytest.approx(L.item(), rel=2e-3)
    g = g.numpy().astype(np.float64)
    for name, (o, shp) in cnn_torch.OFF.items():
        a, r = grad[o:o + int(np.prod(shp))].astype(np.float64), g[o:o + int(np.prod(shp))]
        # the bounds the gradients are held to elsewhere
        rel = np.linalg.norm(a - r) / max(np.linalg.norm(r), 1e-12)
        assert rel < 5e-2, (name, rel)


@pytest.mark.parametrize("batch", [1, 305])
def test_one_step_is_adams_and_packs_its_operands(cuda_lib, batch):
    from bamf_gb300 import learned
    net = learned.ProposalNet(seed=3)
    p0 = net.get_params()
    _, g = net.loss_grad(learned.generate(batch, seed=5))
    net.train(1, batch=batch, lr=1e-3, data_seed=5)
    p1 = net.get_params()
    g = g.astype(np.float64)
    # from zero moments the first step is lr g / (|g| + eps), exact but for a few roundings
    want = p0 - 1e-3 * g / (np.abs(g) + 1e-8)
    assert (np.abs(p1 - want) <= 1e-7 * np.abs(p0) + 1e-7 + 1e-3 * 1e-5).all()
    # the operands packed with the step are those of a network given the same parameters
    other = learned.ProposalNet(seed=4)
    other.set_params(p1)
    b = learned.generate(40, seed=8)
    np.testing.assert_array_equal(net.loss_grad(b)[1], other.loss_grad(b)[1])

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


Z = {"Ax": 0.05, "Bx": 0.03, "Ay": -0.04, "By": 0.02, "Gamma": 0.2, "D": 0.5}
PI = 3.141592  # the kernels' constant


def _fit64(rois, fit, sigma, it, var=None, corners=None):
    """gaussMLE's Newton iteration in 64 bits: parameters [n][k], CRLB, log-likelihood."""
    from scipy.special import erf
    sz, _, n = rois.shape
    d = np.transpose(rois, (2, 0, 1)).astype(np.float64)  # [fit][axis 0][axis 1]
    q = np.arange(sz, dtype=np.float64)
    tot = d.sum((1, 2))
    s = sigma if fit == "Z" else [float(np.mean(sigma))] * 2
    w = np.exp(-(q[:, None] - q[None, :]) ** 2 / (2.0 * s[0] ** 2))
    f = np.einsum("nij,ik,jl->nkl", d, w, w) / (w.sum(0)[:, None] * w.sum(0)[None, :])
    bg = f.min((1, 2))
    scale = 2 * PI * s[0] * s[1] * math.sqrt(2.0) if fit == "Z" else 4 * PI * s[0] ** 2
    th = [(d.sum(2) * q).sum(1) / tot, (d.sum(1) * q).sum(1) / tot,
          np.maximum(0, (f.max((1, 2)) - bg) * scale), bg]
    if fit == "Z":
        th.append(np.zeros(n))
    elif fit != "Basic":
        th += [np.full(n, s[0])] * (1 if fit == "Sigma" else 2)
    g = np.zeros((n, sz, sz))
    if var is not None:
        r = corners[:, 0].astype(int)[:, None, None] + np.arange(sz)[None, :, None]
        c = corners[:, 1].astype(int)[:, None, None] + np.arange(sz)[None, None, :]
        g = var.astype(np.float64)[r, c]

    def axis(c, S, N):
        u, v = q + 1 - c[:, None], q - c[:, None]
        S, N = np.broadcast_to(S, (n,))[:, None], N[:, None]
        a, b = np.exp(-0.5 * (u / S) ** 2), np.exp(-0.5 * (v / S) ** 2)
        r2 = math.sqrt(2 * PI)
        s1 = -N / r2 / S ** 2 * (a * u - b * v)
        return (0.5 * (erf(u / S / math.sqrt(2)) - erf(v / S / math.sqrt(2))), -N / r2 / S * (a - b),
                -N / r2 / S ** 3 * (u * a - v * b), s1, -2 / S * s1 - N / r2 / S ** 5 * (a * u ** 3 - b * v ** 3))

    def terms():
        s0, s1, z0, z1 = s[0], s[1], None, None
        if fit in ("Sigma", "SigmaYX"):
            s0, s1 = th[4], th[-1]
        if fit == "Z":
            out = []
            for zz, A, B, w0 in ((th[4] - Z["Gamma"], Z["Ax"], Z["Bx"], s[0]), (th[4] + Z["Gamma"], Z["Ay"], Z["By"], s[1])):
                t, D = zz / Z["D"], Z["D"]
                al = 1 + t ** 2 + A * t ** 3 + B * t ** 4
                d1 = (2 * t + 3 * A * t ** 2 + 4 * B * t ** 3) / D
                d2 = (2 + 6 * A * t + 12 * B * t ** 2) / D ** 2
                out.append((w0 * np.sqrt(al), w0 / 2 / np.sqrt(al) * d1,
                            -w0 / 4 / al ** 1.5 * d1 ** 2 + w0 / 2 / np.sqrt(al) * d2))
            (s0, *z0), (s1, *z1) = out
        X, Y = axis(th[0], s0, th[2]), axis(th[1], s1, th[2])
        o = lambda a, b: a[:, :, None] * b[:, None, :]  # noqa: E731
        psf = o(X[0], Y[0])
        du = [o(X[1], Y[0]), o(X[0], Y[1]), psf, np.ones_like(psf)]
        d2 = [o(X[2], Y[0]), o(X[0], Y[2]), 0 * psf, 0 * psf]
        sx, sy, sx2, sy2 = o(X[3], Y[0]), o(X[0], Y[3]), o(X[4], Y[0]), o(X[0], Y[4])
        if fit == "Sigma":
            du, d2 = du + [sx + sy], d2 + [sx2 + sy2]
        if fit == "SigmaYX":
            du, d2 = du + [sx, sy], d2 + [sx2, sy2]
        if fit == "Z":
            e = [np.asarray(k)[:, None, None] for k in (*z0, *z1)]
            du = du + [sx * e[0] + sy * e[2]]
            d2 = d2 + [sx2 * e[0] ** 2 + sx * e[1] + sy2 * e[2] ** 2 + sy * e[3]]
        return th[3][:, None, None] + th[2][:, None, None] * psf, du, d2

    for _ in range(it):
        m, du, d2 = terms()
        ok = m > 10e-3
        cf = np.minimum(np.where(ok, (d - m) / (m + g), 0), 10e4)
        df = np.minimum(np.where(ok, (d + g) / (m + g) ** 2, 0), 10e4)
        step = [(a * cf).sum((1, 2)) / (b * cf - a * a * df).sum((1, 2)) for a, b in zip(du, d2)]
        for k in range(len(th)):
            j = 1.0 if k < 2 else 0.1 if fit == "Z" and k == 4 else th[k]
            th[k] = th[k] - np.minimum(np.maximum(step[k], -j), j)
        th[2], th[3] = np.maximum(th[2], 1.0), np.maximum(th[3], 0.01)
        if fit in ("Sigma", "SigmaYX"):
            th[4:] = [np.clip(t, 0.5, sz / 2.0) for t in th[4:]]
    m, du, _ = terms()
    gl = g[:, -1:, -1:] if it else 0 * g[:, -1:, -1:]
    U = np.stack(du)
    F = np.einsum("anij,bnij->nab", U / (m + gl), U)
    D = d + gl
    LL = ((D * np.log(m + gl) - m - np.where(D > 0, D * np.log(np.where(D > 0, D, 1)), 0) + d) * (D > 0)
          + (-m - gl) * (D <= 0)).sum((1, 2))
    return np.stack(th, 1), np.diagonal(np.linalg.inv(F), axis1=1, axis2=2), LL


@pytest.mark.parametrize("camera", ["CCD", "SCMOS"])
@pytest.mark.parametrize("fit", ["Basic", "Sigma", "SigmaYX", "Z"])
@pytest.mark.parametrize("sz", [7, 8, 9, 16, 17, 21])
def test_fit_types_of_every_window(cuda_lib, fit, camera, sz):
    pytest.importorskip("scipy")
    from bamf_gb300 import frontend
    n = 35 if sz > 9 else 101
    sigma = [1.2, 1.3] if fit == "Z" else 1.3
    if fit == "Z":
        t0, t1 = (0.1 - Z["Gamma"]) / Z["D"], (0.1 + Z["Gamma"]) / Z["D"]
        s0 = 1.2 * math.sqrt(1 + t0 ** 2 + Z["Ax"] * t0 ** 3 + Z["Bx"] * t0 ** 4)
        s1 = 1.3 * math.sqrt(1 + t1 ** 2 + Z["Ay"] * t1 ** 3 + Z["By"] * t1 ** 4)
    else:
        s0 = s1 = 1.3
    rois = _rois(sz, n, seed=100 + sz, s0=s0, s1=s1)
    args, var, corners = [], None, None
    if camera == "SCMOS":
        rng = np.random.default_rng(sz)
        var = rng.uniform(1.0, 20.0, (64, 64)).astype(np.float32)
        corners = rng.integers(0, 64 - sz, size=(n, 2)).astype(np.float32)
        args = [var, corners]
    if fit == "Z":
        args.append(Z)
    names = ["Y", "X", "Photons", "BG"] + frontend.FIT_EXTRA[fit]
    for it in (1, 20):
        res = frontend.gaussMLE(rois, fit, camera, sigma, *args, Iterations=it)
        P = np.stack([res[k] for k in names], 1)
        ref, CR, LL = _fit64(rois, fit, sigma, it, var, corners)
        rel = np.abs(P - ref) / np.maximum(np.abs(ref), 1e-3)
        # the bounds that the 7 px fits are held to elsewhere
        assert (np.median(rel, 0) < 1e-5).all() and (np.quantile(rel, 0.99, axis=0) < 1e-3).all()
        SE = np.stack([res[k + "_SE"] for k in names], 1)
        good = (CR > 0).all(1) & np.isfinite(SE).all(1)
        assert good.mean() > 0.9
        assert np.quantile(np.abs(SE[good] ** 2 / CR[good] - 1), 0.99) < 1e-3
        assert np.quantile(np.abs(res["LogLikelihood"] - LL) / np.maximum(np.abs(LL), 1.0), 0.99) < 1e-3


@pytest.mark.parametrize("sz,n", [(1, 1), (2, 1), (5, 31), (6, 32), (7, 33), (21, 65)])
def test_fits_do_not_depend_on_the_memory_order(cuda_lib, sz, n):
    from bamf_gb300 import frontend
    rois = np.random.default_rng(sz).poisson(20.0, (sz, sz, n)).astype(np.float32)
    a = frontend.gaussMLE(np.asfortranarray(rois), "Sigma", "CCD", 1.3, Iterations=2)
    wide = np.zeros((sz, sz + 1, n + 2), np.float32)
    wide[:, 1:, 1:-1] = rois
    for other in (rois, rois.astype(np.float64), wide[:, 1:, 1:-1]):
        b = frontend.gaussMLE(other, "Sigma", "CCD", 1.3, Iterations=2)
        for k in a:
            np.testing.assert_array_equal(a[k], b[k])

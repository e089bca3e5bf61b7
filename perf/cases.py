"""The work that programs have this framework do, as cases that can be timed.

listed() names them, prepare() makes what a program has in hand before the
call (inputs from the seed alone, and the workspace or network it keeps),
run() makes one call through the public entry points, work() counts the
bytes and operations that no implementation can do without, exact() states
the results in 64 bits where that is possible.

Sizes are those of the benchmark, the tests and the reference's defaults:
16x16 ROIs and 8..24 px ROIs at 3000 + 3000 jumps, 16x16 sub-regions of dense
frames, 256x256 frames with about 50 emitters, 7x7 and 8x8 fits, training
batches of 1024 ROIs.
"""
import math
import types

import numpy as np
import torch

from bamf_gb300 import frontend, learned, mapfit, rjstruct, sampler

NPX = 256
MLE_PI = 3.141592


def listed():
    return [
        # the MEX call of a MATLAB program: one ROI, both chains, the grids
        dict(name="rjmcmc_call", kind="call", side=16, burnin=3000, trials=3000),
        # the parity workload: 200 ROIs in the reference's own arithmetic
        dict(name="rjmcmc_exact_200", kind="exact", n=200, side=16, burnin=3000, trials=3000),
        # a first look at a few ROIs, shorter chains
        dict(name="rjmcmc_fast_64", kind="fast", n=64, smin=8, smax=24, step=4, burnin=1000, trials=1000),
        # the headline workload (batched uneven ROIs) at a frame series' size
        dict(name="rjmcmc_fast_30k", kind="fast", n=30000, smin=8, smax=24, step=4, burnin=3000, trials=3000),
        # the tile analysis of RJ.analyzeData: sampler with learned births and
        # state trace, MAP k-means, fixed-count refinement (5 frames' tiles)
        dict(name="analyze_tiles", kind="analyze", n=3380, burnin=3000, trials=2000, mean_n=5.0),
        # one camera frame of an odd size as it arrives
        dict(name="findroi_frame", kind="findroi", y=250, x=190, z=1, box=7, density=36.0),
        # a whole acquisition already on the GPU
        dict(name="findroi_2000", kind="findroi", y=256, x=256, z=2000, box=7, density=50.0),
        # an acquisition in host memory: maxima and fits in one pipelined call
        dict(name="find_fit_1000", kind="findfit", y=256, x=256, z=1000, box=7, density=50.0),
        # the fits of a whole acquisition
        dict(name="gaussmle_80k", kind="mle", n=79787, size=7, iterations=10),
        # findPSF's width fits through the MATLAB-style call on host arrays
        dict(name="gaussmle_sigma_20k", kind="fit", n=20000, size=8, fit="Sigma", camera="CCD", iterations=20),
        # the learned proposal: tables for a frame series' tiles, and training
        dict(name="cnn_infer_50k", kind="infer", n=50000),
        dict(name="cnn_train_1024", kind="train", batch=1024, steps=100),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choice(["call", "exact", "fast", "fast", "analyze", "findroi", "findroi", "findfit", "mle", "fit", "infer",
                       "train"])
    if kind == "call":
        return dict(kind=kind, side=rng.randint(7, 16), burnin=_log(rng, 300, 3000), trials=_log(rng, 300, 3000))
    if kind == "exact":
        return dict(kind=kind, n=_log(rng, 2, 200), side=rng.randint(7, 16), burnin=_log(rng, 300, 3000),
                    trials=_log(rng, 300, 3000))
    if kind == "fast":
        jumps = _log(rng, 200, 3000)
        smin = rng.randint(6, 16)
        return dict(kind=kind, n=_log(rng, 16, 25000), smin=smin, smax=rng.randint(smin, 24), step=rng.choice([1, 2, 4]),
                    burnin=jumps, trials=jumps)
    if kind == "analyze":
        return dict(kind=kind, n=_log(rng, 40, 3300), burnin=_log(rng, 300, 3000), trials=_log(rng, 300, 2000),
                    mean_n=round(rng.uniform(1.0, 6.0), 2))
    if kind in ("findroi", "findfit"):
        y, x = rng.choice([(256, 256), (rng.randint(24, 400), rng.randint(24, 400)),
                           (32 * rng.randint(2, 12), 4 * rng.randint(8, 100))])
        most = (2000 if kind == "findroi" else 1000) * 65536 // (x * y)
        return dict(kind=kind, y=y, x=x, z=_log(rng, 1 if kind == "findroi" else 8, min(most, 3000)),
                    box=rng.randint(5, 13) if kind == "findroi" else rng.randint(7, 10),
                    density=round(x * y * rng.uniform(2e-4, 1e-3), 2))
    if kind == "mle":
        return dict(kind=kind, n=_log(rng, 8, 79000), size=rng.randint(6, 12), iterations=rng.choice([10, 20]))
    if kind == "fit":
        return dict(kind=kind, n=_log(rng, 8, 19000), size=rng.randint(7, 12),
                    fit=rng.choice(["Basic", "Sigma", "SigmaYX", "Z"]), camera=rng.choice(["CCD", "SCMOS"]),
                    iterations=rng.choice([10, 20]))
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 8, 49000))
    return dict(kind=kind, batch=_log(rng, 64, 1000), steps=rng.randint(20, 100))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _profile(side, centre, sigma):
    """[..., side] integrated Gaussian profile of emitters at `centre`."""
    c = (1.0 / (sigma * math.sqrt(2.0)))[..., None] if torch.is_tensor(sigma) else 1.0 / (sigma * math.sqrt(2.0))
    p = torch.arange(side, device=centre.device, dtype=torch.float64)
    u = p - centre.double()[..., None]
    return (0.5 * (torch.erf((u + 1.0) * c) - torch.erf(u * c))).float()


def _images(g, xs, ys, I, bg, sx, sy, sigma):
    """Poisson images [n][sx][sy] (y fastest) of emitters xs, ys, I [n][E]
    (I = 0: none) on a background bg [n]."""
    px, py = _profile(sx, xs, sigma) * I[..., None], _profile(sy, ys, sigma)
    img = bg[:, None, None].expand(-1, sx, sy).contiguous()
    for e in range(xs.shape[1]):
        img.addcmul_(px[:, e, :, None], py[:, e, None, :])
    return torch.poisson(img, generator=g)


def _emitters(g, n, most, count, wx, wy, median, spread):
    """Uniform positions on [0, wx) x [0, wy) (per ROI or one number), log-
    normal intensities, zero past each ROI's count."""
    r = lambda: torch.rand((n, most), generator=g, device="cuda")  # noqa: E731
    xs, ys = r() * wx, r() * wy
    I = median * torch.exp(spread * torch.randn((n, most), generator=g, device="cuda"))
    on = torch.arange(most, device="cuda")[None, :] < count[:, None]
    return xs, ys, torch.where(on, I, torch.zeros_like(I))


def _square_rois(seed, n, side, mean_n, median=1000.0, spread=0.3, bg=10.0, most=16):
    """[n][side*side] ROIs of the plain workload, and their emitters."""
    g = _gen(seed)
    count = torch.poisson(torch.full((n,), mean_n, device="cuda"), generator=g).clamp(max=most)
    xs, ys, I = _emitters(g, n, most, count, side, side, median, spread)
    img = _images(g, xs, ys, I, torch.full((n,), bg, device="cuda"), side, side, 1.3)
    return img.reshape(n, side * side), (xs, ys, I)


def _uneven_rois(seed, n, smin, smax, step):
    """The uneven workload: sides smin, smin + step, .. smax, Poisson(U[0,12])
    emitters, sigma U[1.1,1.5], LogN(ln 1000, 0.4), background U[5,50]."""
    g = _gen(seed)
    u = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    sides = torch.arange(smin, smax + 1, step, device="cuda")
    side = sides[torch.randint(0, sides.numel(), (n,), generator=g, device="cuda")]
    count = torch.poisson(u(n) * 12.0, generator=g).clamp(max=24)
    sigma = 1.1 + 0.4 * u(n)
    bg = 5.0 + 45.0 * u(n)
    xs, ys, I = _emitters(g, n, 24, count, side[:, None], side[:, None], 1000.0, 0.4)
    data = []
    for k in range(0, n, 4096):
        q = slice(k, k + 4096)
        img = _images(g, xs[q], ys[q], I[q], bg[q], smax, smax, sigma[q, None])
        p = torch.arange(smax, device="cuda")
        inside = (p[None, :, None] < side[q, None, None]) & (p[None, None, :] < side[q, None, None])
        data.append(img[inside])
    size = side.long() * side.long()
    return dict(data=torch.cat(data), offsets=torch.cumsum(size, 0) - size, xsize=side.int(), ysize=side.int(),
                psf_sigma=sigma)


def _frames(seed, y, x, z, density):
    """[z][x][y] frames (y fastest): Poisson(density) emitters each."""
    g = _gen(seed)
    most = int(density + 6.0 * math.sqrt(density) + 6.0)
    out = torch.empty((z, x, y), device="cuda")
    step = max(1, (1 << 24) // (x * y))
    for k in range(0, z, step):
        m = min(step, z - k)
        count = torch.poisson(torch.full((m,), float(density), device="cuda"), generator=g).clamp(max=most)
        xs, ys, I = _emitters(g, m, most, count, x, y, 1500.0, 0.3)
        out[k:k + m] = _images(g, xs, ys, I, torch.full((m,), 20.0, device="cuda"), x, y, 1.3)
    return out


def _fit_rois(seed, n, size, sigma=1.3):
    """[n][size*size] windows around maxima: the emitter near the middle."""
    g = _gen(seed)
    mid = (size - 1) / 2.0 + 0.5
    xs, ys, I = _emitters(g, n, 1, torch.ones(n, device="cuda"), 1.0, 1.0, 1500.0, 0.3)
    bg = 15.0 + 10.0 * torch.rand(n, generator=g, device="cuda")
    return _images(g, xs + mid - 0.5, ys + mid - 0.5, I, bg, size, size, sigma).reshape(n, size * size)


def _net_params(seed):
    """He-initialised parameters with small biases, in the network's order."""
    r = np.random.default_rng(seed)
    he = lambda count, fan: r.normal(0.0, math.sqrt(2.0 / fan), count)  # noqa: E731
    b = lambda count: r.normal(0.0, 0.05, count)  # noqa: E731
    parts = [he(288, 9), b(32)]
    for _ in range(3):
        parts += [he(9216, 288), b(32)]
    parts += [he(512, 32), b(16), he(352, 32), b(11)]
    return np.concatenate(parts).astype(np.float32)


def _births(em, side):
    """Birth tables like a trained network's: mass around the emitters over a
    floor, as (cdf [n*npx], sub [n*npx*16])."""
    xs, ys, I = em
    n = xs.shape[0]
    c = (torch.arange(4 * side, device="cuda") + 0.5) / 4.0
    cells = torch.full((n, 4 * side, 4 * side), 0.002, device="cuda")
    for e in range(xs.shape[1]):
        gx = torch.exp(-0.5 * ((c[None, :] - xs[:, e, None]) / 0.35) ** 2)
        gy = torch.exp(-0.5 * ((c[None, :] - ys[:, e, None]) / 0.35) ** 2)
        cells.addcmul_((gx * (I[:, e, None] > 0))[:, :, None], gy[:, None, :])
    cells = cells.view(n, side, 4, side, 4).permute(0, 1, 3, 2, 4).reshape(n, side * side, 16).double()
    pix = cells.sum(2)
    cdf = torch.cumsum(pix, 1) / pix.sum(1, keepdim=True)
    return cdf.float().reshape(-1), (cells / pix[..., None]).float().reshape(-1)


def _rj(burnin, trials, **kw):
    rj = rjstruct.c0_rjstruct()
    rj.N_Burnin, rj.N_Trials = burnin, trials
    for k, v in kw.items():
        setattr(rj, k, v)
    return rj


def _sampler_outs(n):
    outs = {k: torch.zeros(n, dtype=torch.int32, device="cuda")
            for k in ("map_n", "final_n", "n_entries", "status", "overflow", "llr_evals")}
    outs["counters"] = torch.zeros((n, 30), dtype=torch.int32, device="cuda")
    outs["final_state"] = torch.zeros((n, sampler.FINAL_STRIDE), dtype=torch.float32, device="cuda")
    return outs


def prepare(case, seed):
    kind = case["kind"]
    st = types.SimpleNamespace(kind=kind, case=case, seed=seed % (1 << 31))
    if kind == "call":
        side = case["side"]
        data, _ = _square_rois(seed, 1, side, 3.0)
        st.roi = data[0].cpu().numpy().reshape(side, side).T.copy()
        st.rj = _rj(case["burnin"], case["trials"], Rho=3.0 / (side * side))
    elif kind == "exact":
        n, side = case["n"], case["side"]
        data, _ = _square_rois(seed, n, side, 3.0)
        st.rj = _rj(case["burnin"], case["trials"], Rho=3.0 / (side * side))
        sz = np.full(n, side, np.int32)
        st.batch = types.SimpleNamespace(n=n, data=data.cpu().numpy().reshape(-1),
                                         offsets=np.arange(n, dtype=np.int64) * side * side, xsize=sz, ysize=sz,
                                         sigma=np.full(n, 1.3, np.float32))
        st.s = sampler.Sampler()
    elif kind == "fast":
        st.rj = rjstruct.uneven_rjstruct()
        st.rj.N_Burnin, st.rj.N_Trials = case["burnin"], case["trials"]
        st.dev = _uneven_rois(seed, case["n"], case["smin"], case["smax"], case["step"])
        st.outs = _sampler_outs(case["n"])
        st.s = sampler.Sampler()
    elif kind == "analyze":
        n = case["n"]
        st.rj = _rj(case["burnin"], case["trials"], Rho=case["mean_n"] / NPX)
        data, em = _square_rois(seed, n, 16, case["mean_n"], 800.0, 0.5, 50.0)
        cdf, sub = _births(em, 16)
        side = torch.full((n,), 16, dtype=torch.int32, device="cuda")
        st.dev = dict(data=data.reshape(-1), offsets=torch.arange(n, dtype=torch.int64, device="cuda") * NPX, xsize=side,
                      ysize=side, side_max=16, birth_cdf=cdf, birth_sub=sub)
        st.s = sampler.Sampler()
    elif kind == "findroi":
        st.frames = _frames(seed, case["y"], case["x"], case["z"], case["density"])
        st.f = frontend.FindRoiDevice()
    elif kind == "findfit":
        d = _frames(seed, case["y"], case["x"], case["z"], case["density"])
        st.frames = torch.empty(d.numel(), dtype=torch.float32, pin_memory=True)
        st.frames.copy_(d.reshape(-1))
        st.dev_frames = torch.empty(d.numel(), dtype=torch.float32, device="cuda")
        st.f = frontend.FindRoiDevice()
    elif kind == "mle":
        st.rois = _fit_rois(seed, case["n"], case["size"])
    elif kind == "fit":
        st.data, st.args = _fit_inputs(case, seed)
    elif kind == "infer":
        st.data, _ = _square_rois(seed, case["n"], 16, 5.0)
        st.net = learned.ProposalNet(0)
        st.net.set_params(_net_params(seed))
    else:
        st.params = _net_params(seed)
        st.net = learned.ProposalNet(0)
    return st


def _fit_inputs(case, seed):
    """Host arrays of a gaussMLE call: windows (size, size, n) and the
    arguments after the camera type."""
    n, size = case["n"], case["size"]
    data = _fit_rois(seed, n, size).cpu().numpy().reshape(n, size, size).transpose(2, 1, 0)
    args = []
    r = np.random.default_rng(seed)
    if case["camera"] == "SCMOS":
        args += [r.gamma(4.0, 1.0, (128, 128)).astype(np.float32),
                 r.integers(0, 128 - size, (n, 2)).astype(np.float32)]
    if case["fit"] == "Z":
        args.append(dict(Ax=0.0, Ay=0.0, Bx=0.0, By=0.0, Gamma=0.25, D=0.5))
    return np.ascontiguousarray(data), args


def _capacity(case):
    """Room for the maxima that a program expects of these frames."""
    return int(1.3 * case["density"] * case["z"]) + 256


def _found(r):
    """findROI's arrays, zero past the count: a program reads the count before
    it takes them."""
    m = int(r["count"].item())
    for k in ("coords", "corners", "stack", "LL"):
        if k in r:
            r[k][m:] = 0
    for k in ("P", "CR"):
        if k in r:
            r[k][:, m:] = 0
    return {k: r[k] for k in ("count", "coords", "corners", "stack", "P", "CR", "LL") if k in r}


def _chains(r, steps):
    """A call's chains as a program stores them: arrays of one size, zero past
    the entries (at most one a jump) and the emitter records."""
    out = {"pgrid": r["pgrid"], "pback": r["pback"], "counters": np.array(list(r["counters"].values()), np.int64)}
    for name in ("chain", "chain_test"):
        for k, a in r[name].items():
            room = np.zeros(16 * steps if k in ("Index", "Photons", "X", "Y", "Signal") else steps + 1, a.dtype)
            room[:a.size] = a
            out[name + "_" + k] = room
    return out


def run(st):
    c, k = st.case, st.kind
    if k == "call":
        p = rjstruct.mcmc_params(st.rj)
        r = sampler.crjmcmc_raw(st.roi, p, st.rj.P_Offset, st.rj.P_EmPhotons, st.rj.P_BgEmPhotons,
                                e0=([], [], [], rjstruct.initial_bg(st.rj)), rng=(st.seed, 0, 0), arith="exact")
        return _chains(r, c["burnin"] + c["trials"])
    if k == "exact":
        p = rjstruct.mcmc_params(st.rj)
        return st.s.run_host(st.batch, p, st.rj.P_Offset, st.rj.P_EmPhotons, st.rj.P_BgEmPhotons, seed=st.seed,
                             arith="exact", bg0=rjstruct.initial_bg(st.rj))
    if k == "fast":
        p = rjstruct.mcmc_params(st.rj)
        st.s.run_device(st.dev, p, st.rj.P_Offset, st.rj.P_EmPhotons, st.rj.P_BgEmPhotons, seed=st.seed, arith="fast",
                        outs=st.outs, bg0=rjstruct.initial_bg(st.rj))
        return st.outs
    if k == "analyze":
        return mapfit.analyze(st.dev, st.rj, seed=st.seed, proposal="learned", pos_len=200, s=st.s)
    if k == "findroi":
        return _found(st.f.run(st.frames, c["y"], c["x"], c["z"], boxsize=c["box"], capacity=_capacity(c)))
    if k == "findfit":
        return _found(st.f.run_fit_pinned(st.frames, c["y"], c["x"], c["z"], boxsize=c["box"], capacity=_capacity(c),
                                          dev_frames=st.dev_frames))
    if k == "mle":
        return frontend.gauss_mle_device(st.rois, c["size"], c["n"], 1.3, c["iterations"])
    if k == "fit":
        return frontend.gaussMLE(st.data, c["fit"], c["camera"], [1.3, 1.3] if c["fit"] == "Z" else 1.3, *st.args,
                                 Iterations=c["iterations"])
    if k == "infer":
        return st.net.infer(st.data)
    st.net.set_params(st.params)
    loss = st.net.train(c["steps"], batch=c["batch"], data_seed=st.seed)
    return {"loss": loss, "params": st.net.get_params()}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs and outputs once.  Operations: the sampler evaluates
    at least one pixel term (a logarithm, a product, four additions) per
    pixel of a 7x7 PSF footprint for nine jumps in ten; the filters a
    recurrence of seven operations in four directions at two widths; the
    fits 20 operations per pixel and iteration; the network its products."""
    k = case["kind"]
    if k in ("call", "exact", "fast", "analyze"):
        n = case.get("n", 1)
        side = case["side"] if "side" in case else 16 if k == "analyze" else (case["smin"] + case["smax"]) / 2.0
        jumps = case["burnin"] + case["trials"] + (2000 if k == "analyze" else 0)
        out = {"call": 2 * (20 * side) ** 2 * 4 + 2 * jumps * (32 + 3 * 20), "exact": 700, "fast": 700,
               "analyze": 13 * 33 * 4 + NPX * 68}[k]
        return {"bytes": n * (side * side * 4 + out), "flops": 0.9 * jumps * n * 49 * 6.0}
    if k in ("findroi", "findfit"):
        px = case["y"] * case["x"] * case["z"]
        found = 0.8 * case["density"] * case["z"]
        w = {"bytes": px * 4 + found * (20 + 4 * case["box"] ** 2), "flops": px * 8 * 7.0}
        if k == "findfit":
            w["bytes"] += found * 36
            w["flops"] += found * case["box"] ** 2 * 10 * 20.0
        return w
    if k in ("mle", "fit"):
        n, px = case["n"], case["size"] ** 2
        return {"bytes": n * (px * 4 + 36), "flops": n * px * case["iterations"] * 20.0}
    conv = 2.0 * NPX * 9 * 32 * 32
    if k == "infer":
        return {"bytes": case["n"] * (NPX * (4 + 4 + 64) + 44), "flops": case["n"] * (3 * conv + 2.0 * NPX * (9 * 32 + 16 * 32))}
    n = case["batch"] * case["steps"]
    return {"bytes": 2 * learned.NPARAM * 4 + case["steps"] * 4, "flops": 3.0 * n * (3 * conv + 2.0 * NPX * (9 * 32 + 16 * 32))}


# ------------------------------------------------------------ 64-bit results
def exact(case, seed):
    """The fits and the network in 64 bits; None for chains of random draws
    and for what is copied or counted."""
    k = case["kind"]
    if k == "mle":
        rois = _fit_rois(seed, case["n"], case["size"])
        P, CR, LL = _mle64(rois, case["size"], "Basic", case["iterations"])
        return P.t().reshape(-1), CR.t().reshape(-1), LL
    if k == "fit" and case["fit"] != "Z" and case["camera"] == "CCD":
        data, _ = _fit_inputs(case, seed)
        n, size = case["n"], case["size"]
        rois = torch.from_numpy(data.transpose(2, 1, 0).reshape(n, size * size).copy()).cuda()
        P, CR, LL = _mle64(rois, size, case["fit"], case["iterations"])
        SE = torch.sqrt(CR)
        names = ["Y", "X", "Photons", "BG"] + frontend.FIT_EXTRA[case["fit"]]
        out = {"LogLikelihood": LL}
        for i, name in enumerate(names):
            out[name], out[name + "_SE"] = P[:, i], SE[:, i]
        return out
    if k == "infer":
        return _net64(_net_params(seed), _square_rois(seed, case["n"], 16, 5.0)[0])
    return None


def _mle64(rois, size, fit, iterations, sigma0=1.3):
    """gaussMLE's Newton iteration (20 or 10 steps, its start and bounds):
    parameters [n][k], CRLB diagonal, log-likelihood."""
    n, dev = rois.shape[0], rois.device
    d = rois.double().view(n, size, size)  # [fit][axis 1][axis 0]
    q = torch.arange(size, device=dev, dtype=torch.float64)
    tot = d.sum((1, 2))
    t0 = (d.sum(1) * q).sum(1) / tot
    t1 = (d.sum(2) * q).sum(1) / tot
    w = torch.exp(-(q[:, None] - q[None, :]) ** 2 / (2.0 * sigma0 * sigma0))
    f = torch.einsum("nji,jl,ik->nlk", d, w, w) / (w.sum(0)[:, None] * w.sum(0)[None, :])
    bg = f.amin((1, 2))
    I = torch.clamp((f.amax((1, 2)) - bg) * 4.0 * MLE_PI * sigma0 * sigma0, min=0.0)
    s = [torch.full((n,), sigma0, device=dev, dtype=torch.float64) for _ in range(2)]

    def axis(c, sg, I):
        u, v = q + 1.0 - c[:, None], q - c[:, None]
        S, N = sg[:, None], I[:, None]
        a, b = torch.exp(-0.5 * (u / S) ** 2), torch.exp(-0.5 * (v / S) ** 2)
        psf = 0.5 * (torch.erf(u / (S * math.sqrt(2.0))) - torch.erf(v / (S * math.sqrt(2.0))))
        r2p = math.sqrt(2.0 * MLE_PI)
        g = -N / r2p / S ** 2 * (a * u - b * v)
        return (psf, -N / r2p / S * (a - b), -N / r2p / S ** 3 * (u * a - v * b), g,
                -2.0 / S * g - N / r2p / S ** 5 * (a * u ** 3 - b * v ** 3))

    def terms():
        px, dx, ddx, gx, ggx = (t[:, None, :] for t in axis(t0, s[0], I))
        py, dy, ddy, gy, ggy = (t[:, :, None] for t in axis(t1, s[1], I))
        model = bg[:, None, None] + I[:, None, None] * px * py
        zero, one = torch.zeros_like(model), torch.ones_like(model)
        du, d2 = [dx * py, dy * px, px * py, one], [ddx * py, ddy * px, zero, zero]
        if fit == "Sigma":
            du.append(gx * py + gy * px)
            d2.append(ggx * py + ggy * px)
        if fit == "SigmaYX":
            du += [gx * py, gy * px]
            d2 += [ggx * py, ggy * px]
        return model, du, d2

    for _ in range(iterations):
        model, du, d2 = terms()
        fine = model > 10e-3
        cf = torch.clamp(torch.where(fine, d / model - 1.0, torch.zeros_like(d)), max=10e4)
        df = torch.clamp(torch.where(fine, d / model ** 2, torch.zeros_like(d)), max=10e4)
        step = [(a * cf).sum((1, 2)) / (b * cf - a * a * df).sum((1, 2)) for a, b in zip(du, d2)]
        clip = lambda v, m: torch.minimum(torch.maximum(v, -m), m)  # noqa: E731
        t0 = t0 - clip(step[0], torch.ones_like(t0))
        t1 = t1 - clip(step[1], torch.ones_like(t1))
        I, bg = torch.clamp(I - clip(step[2], I), min=1.0), torch.clamp(bg - clip(step[3], bg), min=0.01)
        for j in range(len(du) - 4):
            s[j] = torch.clamp(s[j] - clip(step[4 + j], s[j]), min=0.5, max=size / 2.0)
        if fit == "Sigma":
            s[1] = s[0]
    model, du, _ = terms()
    du = torch.stack([a.expand_as(model).reshape(n, -1) for a in du], 1)
    F = torch.einsum("nap,nbp->nab", du / model.reshape(n, 1, -1), du)
    CR = torch.diagonal(torch.linalg.inv(F), dim1=1, dim2=2)
    ll = torch.where(d > 0, d * torch.log(model) - model - d * torch.log(torch.clamp(d, min=1e-300)) + d, -model)
    P = torch.stack([t0, t1, I, bg] + s[:du.shape[1] - 4], 1)
    return P, CR, ll.sum((1, 2))


def _net64(params, data):
    """The network's tables (cdf, sub, count logits) without BF16 rounding."""
    t = torch.from_numpy(params).cuda().double()
    at, W = 0, []
    for shape in [(32, 1, 3, 3), (32,)] + [(32, 32, 3, 3), (32,)] * 3 + [(16, 32), (16,), (11, 32), (11,)]:
        m = math.prod(shape)
        W.append(t[at:at + m].view(shape))
        at += m
    cdf, sub, cnt = [], [], []
    for k in range(0, data.shape[0], 2048):
        x = data[k:k + 2048].double()
        n = x.shape[0]
        v = torch.sqrt(torch.clamp(x, min=0.0) + 0.375)
        a = ((v - v.mean(1, keepdim=True)) * 0.25).view(n, 1, 16, 16)
        for l in range(4):
            cols = torch.nn.functional.unfold(a, 3, padding=1)
            a = torch.relu(torch.matmul(W[2 * l].reshape(32, -1), cols) + W[2 * l + 1][:, None]).view(n, 32, 16, 16)
        h = a.view(n, 32, NPX)
        z = torch.matmul(W[8], h).transpose(1, 2) + W[9]
        p = torch.softmax(z.reshape(n, -1), 1).view(n, NPX, 16)
        pix = p.sum(2)
        cdf.append(torch.cumsum(pix, 1))
        sub.append(p / pix[..., None])
        cnt.append(h.mean(2) @ W[10].t() + W[11])
    return {"cdf": torch.cat(cdf).reshape(-1), "sub": torch.cat(sub).reshape(-1), "count_logits": torch.cat(cnt)}

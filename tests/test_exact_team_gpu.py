"""The exact sampler's launch shapes give the same chains: a team of warps per
chain for few ROIs, one chain per warp for many, at ROI sizes around the
32-pixel passes and the 16-byte rows of the serial sums; and the quick erf /
log / exp at the edges of their tables equal the header's series."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xs,ys", [(1, 1), (3, 5), (8, 8), (7, 9), (11, 11), (16, 8), (16, 16), (17, 15), (23, 24),
                                   (32, 32)])
def test_exact_chain_equals_oracle_at_odd_sizes(cuda_lib, oracle_port, xs, ys):
    from bamf_gb300 import rjstruct, sampler, synth
    rng = np.random.default_rng(100 * xs + ys)
    roi = rng.poisson(synth.model_image(ys, xs, [xs / 2, xs / 3], [ys / 2, ys / 4], [900.0, 700.0], 10.0,
                                        1.3)).astype(np.float32)
    rj = rjstruct.c0_rjstruct()
    rj.N_Burnin = rj.N_Trials = 150
    rj.SRZoom = 4
    p = rjstruct.mcmc_params(rj)
    args = (p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons)
    kw = dict(e0=([], [], [], rjstruct.initial_bg(rj)), rng=(7, 1, 3))
    got = sampler.crjmcmc_raw(roi, *args, arith="exact", **kw)
    ref = oracle_port.run_chain("port", roi, *args, **kw)
    for w in ("chain", "chain_test"):
        for k, a in got[w].items():
            b = ref[w][k]
            assert a.shape == b.shape and a.tobytes() == b.astype(a.dtype).tobytes(), (w, k)
    assert np.array_equal(got["pgrid"], ref["pgrid"]) and np.array_equal(got["pback"], ref["pback"])


def test_exact_results_do_not_depend_on_batch_size(cuda_lib):
    from bamf_gb300 import rjstruct, sampler, synth
    b = synth.roi_batch_uneven(640, seed=9, sides=(8, 11, 16))
    rj = rjstruct.uneven_rjstruct()
    rj.N_Burnin = rj.N_Trials = 60
    p = rjstruct.mcmc_params(rj)
    s = sampler.Sampler()

    def run(n):
        q = synth.RoiBatch(**{**b.__dict__, "offsets": b.offsets[:n], "xsize": b.xsize[:n], "ysize": b.ysize[:n],
                              "sigma": b.sigma[:n]})
        return s.run_host(q, p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons, seed=3, arith="exact",
                          bg0=rjstruct.initial_bg(rj))

    many = run(640)
    for n in (1, 304, 400):
        few = run(n)
        for k in ("map_n", "final_n", "final_state", "counters", "n_entries", "llr_evals"):
            assert few[k].tobytes() == many[k][:n].tobytes(), (n, k)


@pytest.mark.parametrize("fn", [0, 1, 2])
def test_quick_parity_math_at_table_edges(cuda_lib, oracle_port, fn):
    from bamf_gb300 import abi
    if fn == 0:    # erf intervals of 1/32 up to 4
        e = np.arange(0, 129) / 32.0
    elif fn == 1:  # log intervals of 1/128 of the significand, sqrt 2, around 1
        e = np.concatenate([(1.0 + np.arange(0, 128) / 128.0) * 2.0 ** k for k in (-126, -2, -1, 0, 1, 127)] +
                           [[np.sqrt(2.0), np.sqrt(0.5)]])
    else:          # exp: multiples of ln2/64 and their midpoints, the ends of the normal range
        e = np.concatenate([np.arange(-8100, 8100) * (np.log(2.0) / 128.0), [-104.0, -103.9, -87.4, -87.0, 87.0, 88.8]])
    u = e.astype(np.float32).view(np.int32)[:, None] + np.arange(-3, 4, dtype=np.int32)[None, :]
    x = np.ascontiguousarray(u.reshape(-1).view(np.float32))
    x = np.concatenate([x, -x]) if fn == 0 else x
    dev, host = np.zeros_like(x), np.zeros_like(x)
    L, O = abi.lib(), oracle_port.load("port")
    for f in (L.bamf_parity_math_device, O.oracle_parity_math):
        f.restype, f.argtypes = C.c_int, [C.c_int, C.c_void_p, C.c_int, C.c_void_p]
    assert L.bamf_parity_math_device(fn, x.ctypes.data, x.size, dev.ctypes.data) == 0
    assert O.oracle_parity_math(fn, x.ctypes.data, x.size, host.ctypes.data) == 0
    same = (dev.view(np.uint32) == host.view(np.uint32)) | (np.isnan(dev) & np.isnan(host))
    assert same.all(), (x[~same][:4], dev[~same][:4], host[~same][:4])

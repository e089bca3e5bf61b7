"""The rule that picks the fast sampler's CTA shape, and that results do not depend on the shape, also where the
size classes run one after another in shapes of their own."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shape(side, n, opt_model=0):
    from bamf_gb300 import abi, sampler
    f = sampler._declare().bamf_fast_shape
    f.restype = C.c_int
    f.argtypes = [C.c_int] * 3 + [C.POINTER(C.c_int32)] * 2
    w, m = C.c_int32(), C.c_int32()
    abi.check(f(side, opt_model, n, C.byref(w), C.byref(m)), "bamf_fast_shape")
    return w.value, m.value


@pytest.mark.parametrize("n,sides", [(200, (8, 24)), (2400, (8, 12, 16, 20, 24)), (4000, (16,)), (5000, (7, 16, 32)),
                                     (2000, (8,) * 9 + (24,))])
def test_classes_one_after_another(cuda_lib, n, sides):
    """Every ROI once, whether its class has an equal share of the batch, more than that or less: the results
    of the entry point whose classes run at once."""
    import torch
    from bamf_gb300 import abi, rjstruct, sampler, synth
    b = synth.roi_batch_uneven(200, seed=n, sides=sides)
    pick = np.arange(n) % 200
    dev = {"data": torch.from_numpy(b.data).cuda(), "offsets": torch.from_numpy(b.offsets[pick]).cuda(),
           "xsize": torch.from_numpy(b.xsize[pick]).cuda(), "ysize": torch.from_numpy(b.ysize[pick]).cuda(),
           "psf_sigma": torch.from_numpy(b.sigma[pick]).cuda(), "side_max": int(max(sides))}
    rj = rjstruct.uneven_rjstruct()
    rj.N_Burnin, rj.N_Trials = 20, 15
    p, bg0 = rjstruct.mcmc_params(rj), rjstruct.initial_bg(rj)
    priors = (rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons)
    s = sampler.Sampler()
    got = []
    for call in ("workspace", "noalloc"):
        o = {k: torch.full((n,), -7, dtype=torch.int32, device="cuda") for k in ("final_n", "status", "llr_evals")}
        o["counters"] = torch.zeros((n, 30), dtype=torch.int32, device="cuda")
        o["final_state"] = torch.zeros((n, sampler.FINAL_STRIDE), device="cuda")
        if call == "workspace":
            s.run_device(dev, p, *priors, seed=5, outs=o, bg0=bg0)
        else:
            f = s._L.bamf_rjmcmc_batch_device_noalloc
            f.restype, f.argtypes = C.c_int, None
            pr, keep, bs, rs = s._structs(dev, p, *priors, o, bg0, "reference")
            abi.check(f(C.byref(bs), C.byref(p), C.byref(pr), C.c_uint32(5), sampler.ARITH["fast"], C.byref(rs), None), call)
        got.append({k: v.cpu().numpy() for k, v in o.items()})
    assert not got[0]["status"].any()
    for k in got[0]:
        assert got[0][k].tobytes() == got[1][k].tobytes(), k


def test_ctas_of_eight_chains_where_two_fit(cuda_lib):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for side in range(1, 32):  # at 32 px two CTAs of 8 do not fit
        for n in (8 * sms + 1, 2500, 2700, 2900, 3000, 20 * sms, 22 * sms, 6000, 100_000):
            assert _shape(side, n)[0] >= 8, (side, n, _shape(side, n))


def test_results_are_those_of_every_shape(cuda_lib):
    """One image under many chain ids: the order is the ids', so a small batch's chains are the first of a
    large one's, in another shape."""
    import torch
    from bamf_gb300 import rjstruct, sampler, synth
    rj = rjstruct.uneven_rjstruct()
    rj.N_Burnin, rj.N_Trials = 40, 35
    p = rjstruct.mcmc_params(rj)
    s = sampler.Sampler()
    seen = set()
    for side in (12, 16, 20, 24):
        b = synth.roi_batch_uneven(1, seed=side, sides=(side,))
        large, outs = 7300, {}
        for n in (1, 23, 25, 152, 300, 600, 1216, 2433, 3400, large):
            seen.add(_shape(side, n))
            i32 = torch.full((n,), side, dtype=torch.int32, device="cuda")
            dev = {"data": torch.from_numpy(b.data).cuda(), "offsets": torch.zeros(n, dtype=torch.int64, device="cuda"),
                   "xsize": i32, "ysize": i32, "psf_sigma": torch.full((n,), 1.3, device="cuda"), "side_max": side}
            o = {k: torch.zeros(n, dtype=torch.int32, device="cuda") for k in ("map_n", "final_n", "status", "llr_evals")}
            o["counters"] = torch.zeros((n, 30), dtype=torch.int32, device="cuda")
            o["final_state"] = torch.zeros((n, sampler.FINAL_STRIDE), device="cuda")
            s.run_device(dev, p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons, seed=5, outs=o,
                         bg0=rjstruct.initial_bg(rj))
            outs[n] = {k: v.cpu().numpy() for k, v in o.items()}
        assert not outs[large]["status"].any() and len(np.unique(outs[large]["llr_evals"])) > 10
        for n, o in outs.items():
            for k, v in o.items():
                assert v.tobytes() == outs[large][k][:n].tobytes(), (side, n, k)
    assert {(1, 2), (2, 2), (4, 2), (8, 2), (8, 3), (24, 1)} <= seen, seen

"""The fast sampler's results do not depend on the CTA shape a batch's size
selects: around the sizes where the rule changes shape, a batch gives the same
results as with the shapes the autotuner picks for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 23, 152, 153, 304, 305, 608, 609, 1217, 2433, 3700])
def test_results_do_not_depend_on_the_shape(cuda_lib, n):
    import torch
    from bamf_gb300 import rjstruct, sampler, synth
    b = synth.roi_batch_uneven(n, seed=n, sides=(7, 8, 12, 16, 24))
    rj = rjstruct.uneven_rjstruct()
    rj.N_Burnin, rj.N_Trials = 40, 35
    p = rjstruct.mcmc_params(rj)
    dev = {"data": torch.from_numpy(b.data).cuda(), "offsets": torch.from_numpy(b.offsets).cuda(),
           "xsize": torch.from_numpy(b.xsize).cuda(), "ysize": torch.from_numpy(b.ysize).cuda(),
           "psf_sigma": torch.from_numpy(b.sigma).cuda()}
    args = (dev, p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons)
    bg0 = rjstruct.initial_bg(rj)
    s = sampler.Sampler()

    def run():
        outs = {k: torch.zeros(n, dtype=torch.int32, device="cuda") for k in ("map_n", "final_n", "status", "llr_evals")}
        outs["counters"] = torch.zeros((n, 30), dtype=torch.int32, device="cuda")
        outs["final_state"] = torch.zeros((n, sampler.FINAL_STRIDE), device="cuda")
        s.run_device(*args, seed=5, outs=outs, bg0=bg0)
        return {k: v.cpu().numpy().tobytes() for k, v in outs.items()}

    want = run()
    assert not np.frombuffer(want["status"], np.int32).any()
    s.autotune(*args, jumps=5, sample=n, bg0=bg0)
    assert run() == want

"""Calls of different sizes from two threads at once, each on its own stream (and workspace, where the call
takes one): a kernel's shared-memory limit is shared by the process, and neither call's size may refuse the
other's launch."""
import ctypes as C
import threading

import numpy as np
import pytest

from bamf_gb300 import abi, frontend, mapfit, rjstruct, sampler, synth

pytestmark = pytest.mark.gpu


def _kmeans(pos_len):
    import torch
    t = torch.rand((4, pos_len, mapfit.POS_RECORD), device="cuda")
    t[:, :, 1] = 2
    ne = torch.full((4,), pos_len, dtype=torch.int32, device="cuda")
    k = torch.full((4,), 2, dtype=torch.int32, device="cuda")
    out = torch.empty((4, mapfit.MAP_RECORD), device="cuda")
    f, a = mapfit._lib().bamf_map_kmeans_device, [x.data_ptr() for x in (t, ne, k, out)]
    return lambda s, keep=(t, ne, k, out): abi.check(f(a[0], pos_len, 1, a[1], a[2], 4, 1, a[3], s), "kmeans")


def _basic(size):
    import torch
    r = torch.rand((16, size * size), device="cuda") + 5.0
    o = [torch.empty(n * 16, device="cuda") for n in (4, 4, 1)]
    f, a = frontend._declare().bamf_gauss_mle_device, [x.data_ptr() for x in (r, *o)]
    return lambda s, keep=(r, o): abi.check(f(a[0], size, 16, 1.3, 1, a[1], a[2], a[3], s), "basic")


def _sigma(size):
    import torch
    L = frontend._declare()
    r = torch.rand((16, size * size), device="cuda") + 5.0
    P, CR, LL = (torch.empty(5 * 16, device="cuda"), torch.empty(5 * 16, device="cuda"),
                 torch.empty(16, device="cuda"))
    f = L.bamf_gauss_mle_fit_device
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_float, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int,
                  C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
    a = [x.data_ptr() for x in (r, P, CR, LL)]
    return lambda s, keep=(r, P, CR, LL): abi.check(f(a[0], size, 16, 1, 1.3, None, None, None, 0, 1, *a[1:], s), "sigma")


def _findroi(box):
    import torch
    fr = frontend.FindRoiDevice()
    a = torch.poisson(torch.full((1, 130, 130), 20.0, device="cuda"))
    return lambda s: fr.run(a, 130, 130, 1, boxsize=box, capacity=256, stream=s)


def _chains(side, arith):
    import torch
    b = synth.roi_batch_uneven(2, seed=side, sides=(side,))
    rj = rjstruct.uneven_rjstruct()
    rj.N_Burnin = rj.N_Trials = 2
    p = rjstruct.mcmc_params(rj)
    dev = {k: torch.from_numpy(v).cuda() for k, v in (("data", b.data), ("offsets", b.offsets), ("xsize", b.xsize),
                                                      ("ysize", b.ysize), ("psf_sigma", b.sigma))}
    outs = {"status": torch.zeros(2, dtype=torch.int32, device="cuda")}
    s = sampler.Sampler()
    return lambda st: s.run_device({**dev, "side_max": side}, p, rj.P_Offset, rj.P_EmPhotons, rj.P_BgEmPhotons, seed=1,
                                   arith=arith, outs=outs, bg0=rjstruct.initial_bg(rj), stream=st)


CASES = {"kmeans": lambda: (_kmeans(256), _kmeans(20)), "basic": lambda: (_basic(21), _basic(16)),
         "sigma": lambda: (_sigma(21), _sigma(16)), "findroi": lambda: (_findroi(100), _findroi(60)),
         "fast": lambda: (_chains(32, "fast"), _chains(8, "fast")),
         "exact": lambda: (_chains(32, "exact"), _chains(8, "exact"))}


@pytest.mark.parametrize("case", sorted(CASES))
def test_sizes_do_not_refuse_each_other(cuda_lib, case):
    import torch
    calls = CASES[case]()
    failed = []

    def work(call):
        stream = torch.cuda.Stream()
        try:
            with torch.cuda.stream(stream):
                for i in range(3000):
                    call(stream.cuda_stream)
                    if i % 64 == 63:
                        stream.synchronize()
            stream.synchronize()
        except Exception as e:  # noqa: BLE001 - the other thread goes on
            failed.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed

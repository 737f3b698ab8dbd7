"""nmc_mcxyz_run_noalloc takes the launch shape of nmc_run for the same nmc_ext (include/nmc_abi.h): the same tallies at
the shapes' edges, and, where the shape matters most (a photon per warp), the same time."""
import ctypes as C

import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu


class Caller:
    def __init__(self, gpu, torch, rp, tp, v, ext):
        self.f = gpu.lib().nmc_mcxyz_run_noalloc
        self.f.restype = C.c_int
        self.f.argtypes = [C.POINTER(abi.RunParams), C.POINTER(abi.TissueParams), C.POINTER(abi.Ext), C.c_void_p, C.c_uint64, C.c_uint64,
                           C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
        self.args, self.stream = (rp, tp, ext), torch.cuda.current_stream()
        self.v = torch.from_numpy(v).to("cuda:0")
        self.F = torch.zeros(v.size, dtype=torch.float32, device="cuda:0")
        self.tot = torch.zeros(8, dtype=torch.float64, device="cuda:0")

    def run(self, first, n):
        assert self.f(*(C.byref(a) for a in self.args), self.v.data_ptr(), first, n, self.F.data_ptr(), None, None, self.tot.data_ptr(),
                      self.stream.cuda_stream) == 0


@pytest.mark.parametrize("n,shape", [(1, {}), (2433, {}), (12_160, {}), (12_161, {}), (130_000, {}), (9_000, dict(block_size=64)),
                                     (9_000, dict(blocks_per_sm=1)), (9_000, dict(photons_per_fetch=4))])
def test_shapes_give_the_same_tallies(gpu, n, shape):
    import torch

    rp, tp, v, ext = cases.skin_vessel_case(N=48)
    for k, q in shape.items():
        setattr(ext, k, q)
    c = Caller(gpu, torch, rp, tp, v, ext)
    c.run(5, n)
    torch.cuda.synchronize()
    with gpu.Engine(abi.SIM_MCXYZ, 0, ext) as e:
        e.prepare_data(rp, tp, v)
        e.run(5, n)
        F, s = e.tally(abi.TALLY_F3D), e.summary()
    np.testing.assert_allclose(c.F.cpu().numpy(), F, rtol=1e-6, atol=1e-12)
    t = c.tot.cpu().numpy()
    assert (t[0], t[1], t[2]) == (n, s["substeps"], s["scatters"])


def test_the_shape_is_nmc_runs(gpu):
    # 1,000 photons in full warps of a full SM take 1.75 times as long as one per warp
    import torch

    rp, tp, v, ext = cases.skin_vessel_case(N=100)
    c = Caller(gpu, torch, rp, tp, v, ext)
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    own = []
    for _ in range(5):
        a.record(c.stream)
        c.run(0, 1000)
        b.record(c.stream)
        b.synchronize()
        own.append(a.elapsed_time(b))
    kernel = []
    with gpu.Engine(abi.SIM_MCXYZ, 0, ext) as e:
        e.prepare_data(rp, tp, v)
        for _ in range(5):
            e.reset()
            before = e.summary()["kernel_ms"]
            e.run(0, 1000)
            e.synchronize()
            kernel.append(e.summary()["kernel_ms"] - before)
    assert min(own) < 1.35 * min(kernel)

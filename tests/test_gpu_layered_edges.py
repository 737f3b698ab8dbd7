"""Layered media at the edges of the kernel's branches, against the oracle on the same streams: deposits of a whole
weight, layers without absorption, scattering or anything, matched indices and total reflection, and A(z) tallies on
both sides of the shared-memory limit."""
import math

import numpy as np
import pytest

from nmc_gb300 import layered

pytestmark = pytest.mark.gpu

STACKS = {
    "whole_weight": ([(3.0, 0.0, 0.0, 1.0, math.inf)], 1.0, 50),              # each photon deposits 1.0 at once
    "pure_absorber_below": ([(0.5, 50.0, 0.9, 1.0, 0.05), (8.0, 0.0, 0.0, 1.0, 0.5)], 1.0, 50),
    "no_absorption": ([(0.0, 60.0, 0.8, 1.4, 0.05), (2.0, 60.0, 0.8, 1.4, 0.1)], 1.0, 50),
    "clear_layer": ([(1.0, 80.0, 0.9, 1.4, 0.03), (0.0, 0.0, 0.0, 1.5, 0.02), (1.0, 80.0, 0.9, 1.3, 0.05)], 1.6, 50),
    "many_thin": ([(1.0 + i % 3, 90.0 + i, 0.85, 1.3 + 0.02 * (i % 5), 0.004) for i in range(40)], 1.0, 50),
    "az_in_shared_memory": ([(1.0, 80.0, 0.9, 1.4, math.inf)], 1.0, 2045),    # 1 + 2046 sums of 8 bytes = 16,376 bytes
    "az_in_global_memory": ([(1.0, 80.0, 0.9, 1.4, math.inf)], 1.0, 2047),
}


@pytest.mark.parametrize("name", STACKS)
@pytest.mark.parametrize("a_rz", [False, True])
def test_layered_edges(gpu, oracle, name, a_rz):
    layers, n_below, nz = STACKS[name]
    n = 20_000
    kw = dict(n_above=1.0, n_below=n_below, nr=20, dr=0.02, nz=nz, dz=0.3 / nz, seed=9)
    g = layered.run(layers, n, a_rz=a_rz, **kw)
    o = oracle.layered(layers, n, **kw)
    assert g["photons"] == n
    # the same photons up to the few that FP32 rounding parts: far inside the statistical error
    for k in ("rd", "tt"):
        assert abs(g[k] - o[k]) <= 0.2 * max(g[k + "_se"], o[k + "_se"]) + 1e-6
    np.testing.assert_allclose(g["a_layer"], o["a_layer"], rtol=5e-3, atol=1e-5 * n)
    np.testing.assert_allclose(g["a_z"].sum(), o["a_z"].sum(), rtol=2e-3, atol=1e-6 * n)
    assert np.abs(g["a_z"] - o["a_z"]).sum() <= 2e-2 * o["a_z"].sum() + 1e-5 * n
    # weight is conserved to the fixed point's rounding, and A(z) and A(r, z) are sums of the same deposits
    assert g["a_z"].sum() == pytest.approx(g["A"], rel=1e-6, abs=1e-6 * n)
    if a_rz:
        np.testing.assert_allclose(g["a_rz"].sum(0), g["a_z"], rtol=1e-9, atol=1e-6)
    if name == "whole_weight":
        assert g["A"] == n

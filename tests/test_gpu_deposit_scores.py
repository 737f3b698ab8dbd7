"""Scores summed from the deposit list against a replay of every photon, from
one photon (part of one chunk) to enough for several chunks a thread, with a
fluence loss that is zero over part of the medium.

A photon's score is a float sum over its deposits (some hundreds): in any
order it lies within their number times 2^-24 of the exact sum, about 1e-4 for
1600 of them, which bounds the difference of the gradients at their largest.
"""
import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 97, 4099, 70001])
def test_list_scores_are_the_replayed_scores(gpu, n):
    rp, tp, v, ext, mua, mus, g, bins, dr = cases.adjoint_case()
    rng = np.random.default_rng(n)
    G = rng.uniform(0.5, 1.5, bins + 1).astype(np.float32)
    GF = rng.uniform(0.5, 1.5, rp.Nx * rp.Ny * rp.Nz).astype(np.float32)
    GF[rng.random(GF.size) < 0.4] = 0.0
    with gpu.Engine(abi.SIM_MCXYZ, 0, ext) as e:
        e.prepare_data(rp, tp, v)
        e.set_radial_tally(bins, dr)
        e.set_voxel_props(mua, mus, g)
        e.adjoint_forward(3, n)
        assert not e.deposit_list_complete
        replay = e.adjoint_backward(G, GF)
        e.adjoint_forward(3, n, deposit_capacity=2000 * n)
        assert e.deposit_list_complete
        listed = e.adjoint_backward(G, GF)
    for a, b in zip(replay, listed):
        assert np.abs(a).max() > 0
        np.testing.assert_allclose(b, a, rtol=0, atol=1e-4 * np.abs(a).max())

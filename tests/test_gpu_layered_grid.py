"""Layered runs whose one launch fills the GPU (more than 622,592 photons on 152 SMs) against the same photons in two
launches of two blocks per SM each: the tallies are integer sums, the scalar sums FP64 in another order."""
import numpy as np
import pytest

from nmc_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, abi.FLAG_LAYERED_REF_STREAMS])
@pytest.mark.parametrize("n", [622_594, 700_000])
def test_two_launches_give_the_sums_of_one(gpu, n, flags):
    from nmc_gb300 import layered

    stack = [(3.0, 200.0, 0.8, 1.4, 0.01), (3.0, 150.0, 0.85, 1.4, 0.2), (1.0, 100.0, 0.9, 1.44, float("inf"))]
    run = lambda m, f: layered.run(stack, m, nr=50, dr=0.02, nz=70, dz=0.01, seed=3, first=f, a_rz=True, flags=flags)  # noqa: E731
    whole, parts = run(n, 11), [run(n // 2, 11), run(n // 2, 11 + n // 2)]
    for k in ("photons", "Rd", "Rd2", "Tt", "A", "interactions", "rd_r", "tt_r", "a_z", "a_rz", "a_layer"):
        np.testing.assert_allclose(whole[k], sum(p[k] for p in parts), rtol=1e-11, atol=1e-9, err_msg=k)

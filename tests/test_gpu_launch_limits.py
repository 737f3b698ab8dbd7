"""Calls at the limits of a block's shared memory: both variants of a kernel take them."""
import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phase", [abi.PHASE_HG, abi.PHASE_TWO_TERM])
@pytest.mark.parametrize("n_sets", [1022, 1023, 1024])
def test_sweep_of_the_most_sets(gpu, phase, n_sets):
    # 1024 sets' sums take 48 KB, before the latency variant's own words; an
    # explicit block size takes the other variant
    sets = [abi.SweepSet(mua=0.5, mus=60.0 + k % 50, g=0.8, gf=0.9, af=0.5, gb=0.3, ab=0.5, cc=0.9, n1=1.37, n2=1.0, pad=0, photons=20)
            for k in range(n_sets)]
    rp, tp, ext = cases.mcsub_case(phase=phase, tt=(0.9, 0.5, 0.3, 0.5, 0.9), seed=5)
    got = []
    for block in (0, 256):
        ext.block_size = block
        with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
            e.prepare_data(rp, tp)
            got.append(e.run_sweep(sets))
    assert np.all(got[0]["photons"] == 20)
    for k in got[0]:
        (np.testing.assert_allclose if k in ("E2", "Rd_se") else np.testing.assert_array_equal)(got[0][k], got[1][k], err_msg=k)

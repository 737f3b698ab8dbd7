"""The latency variant of a kernel (few photons per lane) against the variant that fills the GPU: the same photons, so
the same integer tallies, at the edges of its range: one photon, one per warp, all of a warp's lanes, the last size that
takes it, runs of several photons per fetch, and lanes that leave the queue while others still take from it."""
import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu

SUMS = ("photons", "substeps", "scatters", "S", "A", "E", "rd_sum")


def _same(a, b):
    for k in SUMS:
        assert a[0][k] == b[0][k], k
    assert a[0]["rd_sumsq"] == pytest.approx(b[0]["rd_sumsq"], rel=1e-12)
    for k in a[1]:
        np.testing.assert_array_equal(a[1][k], b[1][k], err_msg=k)


RUNS = [(n, per, 101, 0) for n, per in
        [(1, 0), (33, 0), (2432, 0), (2433, 0), (20_000, 0), (77_825, 0), (311_296, 0), (5_000, 4), (100_003, 8)]]
RUNS += [(20_000, 0, 150, 0), (20_000, 0, 101, abi.FLAG_GLOBAL_TALLIES), (20_000, 0, 101, abi.FLAG_SKIP_FLUENCE)]


@pytest.mark.parametrize("phase", [abi.PHASE_HG, abi.PHASE_ISOTROPIC_REF, abi.PHASE_TWO_TERM])
@pytest.mark.parametrize("n,per,bins,flags", RUNS)
def test_semi_infinite(gpu, phase, n, per, bins, flags):
    rp, tp, ext = cases.mcsub_case(phase=phase, tt=(0.9, 0.5, 0.3, 0.5, 0.9), seed=5, bins=bins)
    ext.flags, ext.photons_per_fetch = flags, per
    got = []
    for block in (0, 512 if bins == 101 else 256):  # an explicit block size takes the other variant
        ext.block_size = block
        with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
            e.prepare_data(rp, tp)
            e.run(7, n)
            got.append((e.summary(), e.get_compute_results()))
    _same(*got)
    assert got[0][0]["photons"] == n

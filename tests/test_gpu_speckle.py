"""Speckle mutual interference: the pair arithmetic at the edges of its ranges, against the oracle's double functions."""
import math

import numpy as np
import pytest

from nmc_gb300 import abi, efield

pytestmark = pytest.mark.gpu

PI = np.float32(math.pi)
EDGES = np.array([0.0, -0.0, 1e-30, PI, -PI, np.nextafter(PI, np.float32(0)), np.nextafter(PI, np.float32(4)), 2 * PI, -3 * PI, 4095.9,
                  4096.5, -1e5, np.nan, np.inf, -np.inf], np.float32)


@pytest.mark.parametrize("nx,ny,k,lc", [(1, 1, 0, 0.05), (1, 1, 1, 0.05), (5, 13, 3, 1e-7), (9, 7, 9, 2e-5), (65, 63, 7, 0.05)])
def test_speckle_edges(gpu, oracle, nx, ny, k, lc):
    r = np.random.default_rng(nx + k)
    maps = np.zeros((len(abi.EF_MAPS), nx, ny), np.float32)
    det = r.integers(0, 4, (nx, ny)).astype(np.float32)  # pixels that no photon reached among them
    maps[abi.EF_MAPS.index("Det")] = det
    for q in ("XX", "XY", "Rd"):
        maps[abi.EF_MAPS.index(q)] = r.choice(np.float32([0, 1e-20, 0.3, 1]), (nx, ny)) * det
    for q in ("Phase0", "Phase1", "Phase2", "Phase3"):
        maps[abi.EF_MAPS.index(q)] = r.choice(EDGES[:9], (nx, ny)) * det
    rec = np.zeros((k, nx, ny), abi.SPECKLE_DTYPE)
    for f in ("Phase", "Path", "Scatt", "Total"):
        rec[f] = r.choice(EDGES, rec.shape)
    for f in ("XX", "XY", "Ryx"):
        rec[f] = r.choice(np.float32([0, 1e-20, 0.2, -0.1, 1e16, np.nan, np.inf]), rec.shape)
    counts = r.integers(0, k + 3, (nx, ny)).astype(np.int32)
    lam = 633e-6 if lc > 0.01 else 633e-9
    with np.errstate(all="ignore"):
        got = efield.speckle_mutual(maps, rec, counts, lam, lc)
        want = oracle.speckle_mutual(maps, rec, counts, lam, lc, np.zeros((len(abi.EF_MAPS), nx * ny), np.float32))
    # each of the k terms and of the k sums is off by at most a float's last place
    tol = 2.0 ** -23 * 2 * (k + 1)
    np.testing.assert_allclose(got.reshape(want.shape), want, rtol=tol, atol=tol * 4, equal_nan=True)

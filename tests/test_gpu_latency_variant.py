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


@pytest.mark.parametrize("phase", [abi.PHASE_HG, abi.PHASE_TWO_TERM])
@pytest.mark.parametrize("n_sets,photons", [(1, 1), (3, 700), (40, 5_000), (1000, 100)])
def test_semi_infinite_sweep(gpu, phase, n_sets, photons):
    sets = [abi.SweepSet(mua=0.05 * (1 + k % 7), mus=60.0 + k % 50, g=0.8, gf=0.9, af=0.5, gb=0.3, ab=0.5, cc=0.9, n1=1.37, n2=1.0, pad=0,
                         photons=photons if k % 5 else 0 if n_sets > 1 else photons) for k in range(n_sets)]
    rp, tp, ext = cases.mcsub_case(phase=phase, tt=(0.9, 0.5, 0.3, 0.5, 0.9), seed=5)
    got = []
    for block in (0, 256):
        ext.block_size = block
        with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
            e.prepare_data(rp, tp)
            got.append(e.run_sweep(sets, with_J=True))
    for k in got[0]:
        (np.testing.assert_allclose if k in ("E2", "Rd_se") else np.testing.assert_array_equal)(got[0][k], got[1][k], err_msg=k)


@pytest.mark.parametrize("adjoint", [False, True])
def test_layered(gpu, adjoint):
    # 330,000 photons in one call take the other variant than in three; the
    # tallies are integer sums, the gradients and sums FP64 in another order
    from nmc_gb300 import layered

    stack, n = [(3.0, 200.0, 0.8, 1.4, 0.01), (0.3, 150.0, 0.85, 1.4, 0.2), (0.1, 100.0, 0.9, 1.44, float("inf"))], 330_000
    up = np.linspace(-1.0, 1.0, 51).astype(np.float32)
    run = (lambda m, f: layered.adjoint(stack, m, grad_rd_r=up, nr=50, dr=0.02, seed=3, first=f)) if adjoint else \
          (lambda m, f: layered.run(stack, m, nr=50, dr=0.02, nz=70, dz=0.01, seed=3, first=f, a_rz=True))
    whole, parts = run(n, 11), [run(n // 3, 11 + k * (n // 3)) for k in range(3)]
    for k in ("photons", "Rd", "Rd2", "Tt", "A", "interactions", "rd_r", "tt_r") + (
            ("grad_mua", "grad_mus", "grad_g") if adjoint else ("a_z", "a_rz", "a_layer")):
        np.testing.assert_allclose(whole[k], sum(p[k] for p in parts), rtol=1e-11, atol=1e-9, err_msg=k)


@pytest.mark.parametrize("photons", [1, 300, 330_000])
def test_field(gpu, oracle, photons):
    # 8 settings: one photon of a few warps, thin warps with Raman conversions
    # between their records, and (2.64e6 photons) the variant that fills the
    # GPU; short paths, which the FP32 oracle follows photon for photon
    from nmc_gb300 import efield

    cfg, s633, s700, st = cases.cbs_case(n_settings=8, photons=photons, mu_raman=2.0, sep_half_width=0.05)
    cfg.mua = cfg.raman_mua = 30.0
    cfg.flags = abi.FLAG_PRECISE_MATH
    g = efield.run(cfg, s633, st, S_raman=s700, cone=False, pol_vs_scatt=False, maps=False, raman_depth=False)
    o = oracle.efield(cfg, s633, st, S_raman=s700, cone=False, real_bits=32)
    np.testing.assert_array_equal(g["photons"], o["photons"])
    for k in ("specular", "Rd", "co", "cross", "multi_co", "raman_Rd", "raman_co", "raman_cross"):
        assert np.all(np.abs(g[k] - o[k]) <= 1e-3 * (o["Rd"] + o["raman_Rd"]) + 1e-3), k
    for k in ("raman_n", "scatters"):
        assert np.all(np.abs(g[k] - o[k]) <= 2e-3 * o[k] + 2), k


@pytest.mark.parametrize("n", [1, 2432, 2433, 4865, 9729, 12_160, 12_161, 116_737, 389_121])
@pytest.mark.parametrize("sim,boundary,rng", [(abi.SIM_MCXYZ, 2, abi.RNG_PHILOX), (abi.SIM_MCXYZ, 1, abi.RNG_TAUS_REF),
                                              (abi.SIM_MCXYZ_TT, 0, abi.RNG_PHILOX)])
def test_voxel_launch_shapes(gpu, sim, boundary, rng, n):
    # one photon per warp, a few (blocks of 1 to 5 threads), 2, 3 and 4 blocks
    # per SM: the same tallies as blocks of 256 that fill the GPU
    rp, tp, v = cases.modes_medium(boundaryflag=boundary, mckernelflag=sim)
    if sim == abi.SIM_MCXYZ_TT:
        tp = abi.tissue_params(mua=[0.0001, 1.0, 5.0], mus=[1.0, 80.0, 120.0], g=[1.0, 0.85, 0.9], gf=[0.9] * 3, af=[0.5] * 3,
                               gb=[0.3] * 3, ab=[0.5] * 3, cc=[0.9] * 3)
    got = []
    for block in (0, 256):
        with gpu.Engine(sim, 0, abi.ext_defaults(seed=5, rng=rng, block_size=block)) as e:
            e.prepare_data(rp, tp, v)
            e.run(7, n)
            one = (e.summary(), e.get_compute_results())
            sweep = e.run_sweep_tissues([tp, tp], [n, n // 3]) if rng == abi.RNG_PHILOX else {}
        got.append((one, sweep))
    _same(got[0][0], got[1][0])
    for k in got[0][1]:
        np.testing.assert_allclose(got[0][1][k], got[1][1][k], rtol=1e-12 if k in ("E2", "Rd_se") else 0, err_msg=k)

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


@pytest.mark.parametrize("flags", [0, abi.FLAG_PRECISE_MATH])
@pytest.mark.parametrize("n_angles", [4090, 4091, 4094, 27_002, 27_003, 27_006])
def test_field_of_the_most_angles(gpu, n_angles, flags):
    # 4,094 angles are what fits 48 KB beside the static arrays of the kernel
    # that fills the GPU, 27,006 what fits a block at all
    from nmc_gb300 import efield

    cfg, _, _, st = cases.cbs_case(n_settings=2, photons=500, mu_raman=0.0)
    cfg.mua, cfg.n_angles, cfg.flags = 5.0, n_angles, flags
    g = efield.run(cfg, cases.hg_amplitude_table(0.8, n_angles), st, cone=False, pol_vs_scatt=False, maps=False, raman_depth=False)
    assert list(g["photons"]) == [500, 500]
    assert np.all(g["Rd"] > 0) and np.all(g["Rd"] < 500)


@pytest.mark.parametrize("n", [1, 1217, 10_000, 60_000])
@pytest.mark.parametrize("rng", [abi.RNG_PHILOX, abi.RNG_TAUS_REF])
def test_semi_infinite_with_one_block_per_sm(gpu, rng, n):
    # 128 bins: the private F(r,z) leaves room for one block, whose 8 warps per
    # SM take all the photons
    rp, tp, ext = cases.mcsub_case(bins=128, rng=rng, seed=5)
    got = []
    for block in (0, 512):
        ext.block_size = block
        with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
            e.prepare_data(rp, tp)
            e.run(0, n)
            got.append((e.summary(), e.get_compute_results()))
    assert got[0][0]["photons"] == n
    for k in ("photons", "substeps", "scatters", "S", "A", "E"):
        assert got[0][0][k] == got[1][0][k], k
    for k in got[0][1]:
        np.testing.assert_array_equal(got[0][1][k], got[1][1][k], err_msg=k)


@pytest.mark.parametrize("phase", [abi.PHASE_HG, abi.PHASE_ISOTROPIC_REF])
def test_sweep_that_fills_the_gpu_gives_the_parts(gpu, phase):
    # 8 short-lived sets of 120,000 photons take four blocks per SM, a 24th of them the latency variant
    # and a sixth the kernel of three blocks: the same photons, the same integer sums
    def sets(n, first):
        return [abi.SweepSet(mua=10.0 + k, mus=60.0 + k, g=0.8, gf=0.9, af=0.5, gb=0.3, ab=0.5, cc=0.9, n1=1.37, n2=1.0, pad=0, photons=n,
                             first_photon=first) for k in range(8)]
    rp, tp, ext = cases.mcsub_case(phase=phase, seed=5)
    n = 120_000
    with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
        e.prepare_data(rp, tp)
        whole = e.run_sweep(sets(n, 3), with_J=True)
        for parts in (6, 24):
            got = [e.run_sweep(sets(n // parts, 3 + k * (n // parts)), with_J=True) for k in range(parts)]
            for q in ("photons", "hops", "J"):
                np.testing.assert_array_equal(whole[q], sum(g[q] for g in got), err_msg=q)
            for q in ("S", "A", "E", "E2"):
                np.testing.assert_allclose(whole[q], sum(g[q] for g in got), rtol=1e-12, err_msg=q)


@pytest.mark.parametrize("adjoint", [False, True])
def test_layered_variants_follow_the_same_photons(gpu, adjoint):
    # 8 photons per warp are the latency variant's last size, three times as many the other kernel's
    from nmc_gb300 import layered

    stack, n = [(3.0, 200.0, 0.8, 1.4, 0.01), (0.0, 0.0, 0.0, 1.5, 0.02), (0.3, 150.0, 0.85, 1.4, 0.2), (0.1, 100.0, 0.9, 1.44, float("inf"))], 19_456
    up = np.linspace(-1.0, 1.0, 51).astype(np.float32)
    run = (lambda m, f: layered.adjoint(stack, m, grad_rd_r=up, nr=50, dr=0.02, seed=3, first=f)) if adjoint else \
          (lambda m, f: layered.run(stack, m, nr=50, dr=0.02, nz=70, dz=0.01, seed=3, first=f, a_rz=True))
    whole, parts = run(3 * n, 11), [run(n, 11 + k * n) for k in range(3)]
    for k in ("photons", "Rd", "Rd2", "Tt", "A", "interactions", "rd_r", "tt_r") + (
            ("grad_mua", "grad_mus", "grad_g") if adjoint else ("a_z", "a_rz", "a_layer")):
        np.testing.assert_allclose(whole[k], sum(p[k] for p in parts), rtol=1e-11, atol=1e-9, err_msg=k)

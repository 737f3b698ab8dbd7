"""The two variants of a kernel on the same photons, where no other test compares them: long E-field paths with every tally,
and the semi-infinite kernel on the reference's streams."""
import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, abi.FLAG_PRECISE_MATH])
@pytest.mark.parametrize("photons", [300, 20_000])
def test_field_variants_follow_the_same_photons(gpu, photons, flags):
    # about 1,500 scatterings per photon and up to 9,000; a setting's photons depend on its number alone, so a ninth
    # setting of 1.2e6 photons takes the first eight's from the latency variant to the one that fills the GPU
    from nmc_gb300 import efield

    cfg, s633, s700, st = cases.cbs_case(n_settings=9, photons=photons, mu_raman=0.02, sep_n=256, sep_half_width=0.5, cone_n=32)
    cfg.mua = cfg.raman_mua = 0.1
    cfg.flags, cfg.speckle_max = flags, 8
    a = efield.run(cfg, s633, st[:8], S_raman=s700)
    st[8].photons = 1_200_000
    b = efield.run(cfg, s633, st, S_raman=s700)
    for k in ("photons", "scatters", "raman_n"):
        np.testing.assert_array_equal(a[k], b[k][:8], err_msg=k)
    np.testing.assert_array_equal(a["maps"]["Det"], b["maps"]["Det"][:8])
    np.testing.assert_array_equal(a["speckle_counts"], b["speckle_counts"][:8])
    for k in ("specular", "Rd", "Rd2", "raman_Rd"):  # weights: the same floats, added in FP64 in another order
        np.testing.assert_allclose(a[k], b[k][:8], rtol=1e-12, err_msg=k)
    np.testing.assert_allclose(a["raman_depth"], b["raman_depth"][:8], rtol=1e-12)
    # a pixel's records, where all arrivals were kept (the counts stop at the records' number), in any order
    whole = (a["maps"]["Det"] <= 8)[:, None]
    np.testing.assert_array_equal(*(np.sort(np.where(whole, g["speckles"]["Ryx"][:8], 0), axis=1) for g in (a, b)))
    # intensities: some 30 float roundings per detected photon, which the variants may fuse differently
    for k in ("co", "cross", "multi_co", "multi_cross", "interf_co", "interf_cross", "raman_co", "raman_cross"):
        assert np.all(np.abs(a[k] - b[k][:8]) <= 2e-6 * (a["Rd"] + a["raman_Rd"])), k
    assert np.all(np.abs(a["pol_vs_scatt"] - b["pol_vs_scatt"][:8]) <= 2e-6 * a["pol_vs_scatt"].sum(1, keepdims=True) + 1e-12)
    for k in ("XX", "XY", "YX", "YY", "Rd"):
        assert np.all(np.abs(a["maps"][k] - b["maps"][k][:8]) <= 4e-6 * a["maps"]["Rd"] + 1e-12), k
    assert np.all(np.abs(a["cone"] - b["cone"][:8]).max((2, 3)) <= 1e-5 * np.abs(a["cone"]).max((2, 3)))


@pytest.mark.parametrize("phase", [abi.PHASE_HG, abi.PHASE_ISOTROPIC_REF, abi.PHASE_TWO_TERM])
@pytest.mark.parametrize("n,per,flags", [(1, 0, 0), (2432, 0, 0), (2433, 0, 0), (20_000, 0, 0), (77_825, 0, 0), (100_003, 8, 0),
                                         (20_000, 0, abi.FLAG_GLOBAL_TALLIES), (20_000, 0, abi.FLAG_SKIP_FLUENCE)])
def test_semi_infinite_on_the_reference_streams(gpu, phase, n, per, flags):
    rp, tp, ext = cases.mcsub_case(phase=phase, tt=(0.9, 0.5, 0.3, 0.5, 0.9), seed=5, rng=abi.RNG_TAUS_REF)
    ext.flags, ext.photons_per_fetch = flags, per
    got = []
    for block in (0, 512):
        ext.block_size = block
        with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
            e.prepare_data(rp, tp)
            e.run(0, n)
            got.append((e.summary(), e.get_compute_results()))
    for k in ("photons", "substeps", "scatters", "S", "A", "E"):
        assert got[0][0][k] == got[1][0][k], k
    assert got[0][0]["rd_sumsq"] == pytest.approx(got[1][0]["rd_sumsq"], rel=1e-12)
    for k in got[0][1]:
        np.testing.assert_array_equal(got[0][1][k], got[1][1][k], err_msg=k)

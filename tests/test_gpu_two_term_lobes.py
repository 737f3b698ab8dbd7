"""Two-term lobes at the edges of their form: isotropic lobes, and a weight that always or never takes the forward one.

The lobe's constants are selected before one power is taken; the kernels that read them from the parameters, from a
shared table and from a global table have to sample the same angles as the oracle, photon for photon.
"""
import numpy as np
import pytest

from nmc_gb300 import abi
import nmc_cases as cases

pytestmark = pytest.mark.gpu

LOBES = [(0.0, 0.5, 0.3, 0.5, 0.9), (0.9, 0.5, 0.0, 0.5, 0.9), (0.0, 0.5, 0.0, 0.5, 0.5), (0.9, 0.5, 0.3, 0.5, 0.0), (0.9, 0.5, 0.3, 0.5, 1.0)]


@pytest.mark.parametrize("lobes", LOBES)
def test_two_term_lobes(gpu, oracle, lobes):
    gf, af, gb, ab, cc = lobes
    n = 3000
    rp, tp, ext = cases.mcsub_case(phase=abi.PHASE_TWO_TERM, tt=lobes, seed=3)
    with gpu.Engine(abi.SIM_MCSUB, 0, ext) as e:
        e.prepare_data(rp, tp)
        recs, _ = e.run_traced(0, n)
        e.reset()
        e.run(0, n)
        sm = e.summary()
        sets = [abi.SweepSet(mua=1.0, mus=100.0, g=0.9, gf=gf, af=af, gb=gb, ab=ab, cc=cc, n1=rp.n1, n2=rp.n2, pad=0, photons=n)]
        sw = e.run_sweep(sets)
    o = oracle.run(abi.SIM_MCSUB, rp, tp, ext=ext, n=n, trace=True)
    frac, _ = cases.match_fraction(recs, o["recs"])
    assert frac >= 0.99  # FP32 against FP64 walks; another angle would part every photon at its first scattering
    assert sw["hops"][0] == sm["substeps"]
    assert sw["A"][0] == pytest.approx(sm["A"], rel=1e-6)

    rp, tp, v = cases.modes_medium(mckernelflag=abi.SIM_MCXYZ_TT)
    tp = abi.tissue_params(mua=[0.0001, 1.0, 5.0], mus=[1.0, 80.0, 120.0], g=[1.0, 0.85, 0.9], gf=[gf] * 3, af=[af] * 3, gb=[gb] * 3,
                           ab=[ab] * 3, cc=[cc] * 3)
    with gpu.Engine(abi.SIM_MCXYZ_TT, 0, abi.ext_defaults(seed=3)) as e:
        e.prepare_data(rp, tp, v)
        recs, _ = e.run_traced(0, n)
        e.reset()
        e.run(0, n)
        sm = e.summary()
        sw = e.run_sweep_tissues([tp], [n])
    o = oracle.run(abi.SIM_MCXYZ_TT, rp, tp, v, ext=abi.ext_defaults(seed=3), n=n, trace=True)
    frac, _ = cases.match_fraction(recs, o["recs"])
    assert frac >= 0.97
    assert sw["hops"][0] == sm["substeps"] and sw["A"][0] == pytest.approx(sm["A"], rel=1e-6)

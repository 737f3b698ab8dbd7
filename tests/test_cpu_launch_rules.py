"""The launch rules (nmc_gb300/csrc/launch_rules.h) at media and sizes where both variants were timed on a GB300: the
rule takes the faster one wherever they differ by more than a tenth."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "launch_rules.h"
using namespace nmc;
static WorkTail one(double n, double mua, double mus) { WorkTail w; w.add(n, mua, mus); return w; }
extern "C" {
int sub_lat(double n, double mua, double mus, int blocks) { return sub_latency_pays(one(n, mua, mus), blocks); }
int sweep_lat(int sets, double per, double lo, double hi) {
  WorkTail w;
  for (int k = 0; k < sets; ++k) sweep_add(w, per, lo + (hi - lo) * k / (sets - 1), 100.0);
  return sweep_latency_pays(w);
}
int sweep_full(int sets, double per, double lo, double hi) {
  WorkTail w;
  for (int k = 0; k < sets; ++k) sweep_add(w, per, lo + (hi - lo) * k / (sets - 1), 100.0);
  return sweep_fills_sm(w);
}
int spectrum_lat(int n, const double* photons, const double* mua, const double* mus) {
  WorkTail w;
  for (int k = 0; k < n; ++k) sweep_add(w, photons[k], mua[k], mus[k]);
  return sweep_latency_pays(w);
}
int field_lat(double n, double mua) { return field_latency_pays(one(n, mua, 100.0), (uint64_t)n, 2432); }
int layered(unsigned long long n, int nl, const double* q, int ref) {  // 0: the latency variant, else blocks per SM
  WorkTail w;
  layered_add(w, (double)n, reinterpret_cast<const PlaneLayer*>(q), nl);
  const LayeredShape s = layered_shape(w, n, 2432, ref);
  return s.latency ? 0 : s.blocks ? s.blocks : 4;
}
unsigned lanes(unsigned long long items, unsigned long long warps) { return lat_lanes(items, warps); }
}
"""


@pytest.fixture(scope="session")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "nmc_gb300", "csrc"), str(d / "rules.cpp"),
                    "-o", str(d / "rules.so")], check=True)
    lib = C.CDLL(str(d / "rules.so"))
    lib.sub_lat.argtypes = [C.c_double] * 3 + [C.c_int]
    lib.sweep_full.argtypes = lib.sweep_lat.argtypes = [C.c_int] + [C.c_double] * 3
    lib.spectrum_lat.argtypes = [C.c_int] + [C.c_void_p] * 3
    lib.field_lat.argtypes = [C.c_double] * 2
    lib.layered.argtypes = [C.c_ulonglong, C.c_int, C.c_void_p, C.c_int]
    lib.lanes.argtypes, lib.lanes.restype = [C.c_ulonglong] * 2, C.c_uint
    return lib


@pytest.mark.parametrize("mua,mus,pays,loses", [(1, 100, 70_000, 150_000), (10, 100, 20_000, 70_000), (1, 20, 20_000, 70_000),
                                                (0.2, 300, 200_000, 400_000), (0.05, 100, 300_000, 400_000)])
def test_semi_infinite_with_one_block_per_sm(rules, mua, mus, pays, loses):
    assert rules.sub_lat(pays, mua, mus, 1) and not rules.sub_lat(loses, mua, mus, 1)
    assert rules.sub_lat(pays, mua, mus, 2)  # two blocks pay at least as long


@pytest.mark.parametrize("items,warps,want", [(1, 1216, 1), (1216, 1216, 1), (1217, 1216, 2), (10_000, 1216, 9), (10_000, 2432, 5),
                                              (38_912, 1216, 32), (1 << 40, 1216, 32), (0, 1216, 1)])
def test_every_photon_of_a_small_run_has_a_lane(rules, items, warps, want):
    assert rules.lanes(items, warps) == want
    assert items > 32 * warps or want * warps >= items


@pytest.mark.parametrize("mua,mus,pays,loses", [(1, 100, 200_000, 600_000), (10, 100, 100_000, 150_000), (1, 20, 100_000, 150_000),
                                                (0.2, 300, 600_000, 10_000_000), (0.05, 100, 600_000, 10_000_000)])
def test_semi_infinite_with_two_blocks_per_sm(rules, mua, mus, pays, loses):
    assert rules.sub_lat(pays, mua, mus, 2) and not rules.sub_lat(loses, mua, mus, 2)


def test_semi_infinite_at_the_crossing(rules):
    # 1.90 against 1.75 ms
    assert not rules.sub_lat(300_000, 1.0, 100.0, 2)


@pytest.mark.parametrize("lo,hi,pays,loses", [(0.05, 2.0, 4_000, 20_000), (0.5, 5.0, 500, 3_000), (3.0, 30.0, 0, 2_000),
                                              (0.05, 0.2, 3_000, 10_000)])
def test_semi_infinite_sweep(rules, lo, hi, pays, loses):
    assert (pays == 0 or rules.sweep_lat(351, pays, lo, hi)) and not rules.sweep_lat(351, loses, lo, hi)


# spectra of 351 wavelengths, 3.51e6 photons, by seed: timed with the latency variant and without it (ms, two-term)
@pytest.mark.parametrize("seed,variant,other", [(23, 26.3, 35.8), (16, 29.5, 39.3), (28, 17.6, 23.2), (3, 28.0, 36.9), (29, 23.5, 30.5),
                                                (0, 24.2, 31.8), (26, 11.7, 10.2), (2, 11.3, 9.0), (18, 15.9, 13.4), (12, 14.1, 12.2),
                                                (20, 14.7, 11.3), (27, 12.9, 9.9), (13, 8.6, 6.4), (17, 7.0, 5.1), (1, 9.5, 7.0)])
def test_semi_infinite_sweep_of_spectra(rules, seed, variant, other):
    from perf import cases

    r = np.random.default_rng(seed)
    w = np.exp(r.uniform(0.0, np.log(10.0), 351))
    photons = np.maximum(1, (w / w.sum() * 3_510_000).astype(np.int64)).astype(np.float64)
    mua, mus = (np.ascontiguousarray(q, np.float64) for q in cases._spectrum(r, 351, 0.05, 2.0, 0.05))
    assert bool(rules.spectrum_lat(351, *(q.ctypes.data for q in (photons, mua, mus)))) == (variant < other)


@pytest.mark.parametrize("lo,hi,three,four", [(3.0, 30.0, 1_000, 10_000), (0.5, 5.0, 3_000, 30_000), (0.05, 2.0, 10_000, 100_000),
                                              (0.05, 0.2, 10_000, 100_000)])
def test_one_term_sweep_fills_the_sm(rules, lo, hi, three, four):
    assert not rules.sweep_full(351, three, lo, hi) and rules.sweep_full(351, four, lo, hi)


@pytest.mark.parametrize("mua,pays,loses", [(0.01, 8 * 100_000, 8 * 2_000_000), (0.1, 8 * 50_000, 8 * 310_000), (1.0, 8 * 20_000, 8 * 100_000),
                                            (10.0, 8 * 5_000, 8 * 100_000), (100.0, 8 * 2_000, 8 * 100_000)])
def test_field(rules, mua, pays, loses):
    assert rules.field_lat(pays, mua) and not rules.field_lat(loses, mua)


INF = float("inf")
STACKS = {  # (mua, mus, g, thickness), the last size at which two blocks were not slower, the first at which four were faster by 5%
    "skin": ([(3.0, 200.0, 0.8, 0.01), (0.3, 150.0, 0.85, 0.2), (0.1, 100.0, 0.9, INF)], 600_000, 1_000_000),
    "epidermis": ([(3.0, 200.0, 0.8, INF)], 100_000, 300_000),
    "mua_1": ([(1.0, 100.0, 0.9, INF)], 200_000, 450_000),
    "absorbing": ([(10.0, 100.0, 0.9, 0.05), (20.0, 100.0, 0.9, INF)], 60_000, 200_000),
    "no_absorption": ([(0.0, 100.0, 0.9, 0.3)], 200_000, 300_000),
    "no_absorption_thick": ([(0.0, 100.0, 0.9, 2.0)], 600_000, INF),
    "no_absorption_over": ([(0.0, 100.0, 0.9, 0.3), (1.0, 100.0, 0.9, INF)], 200_000, 450_000),
    "clear_gap": ([(1.0, 80.0, 0.9, 0.03), (0.0, 0.0, 0.0, 0.02), (1.0, 80.0, 0.9, 0.05)], 60_000, 200_000),
    "out_of_reach": ([(20.0, 100.0, 0.8, 0.5), (0.05, 100.0, 0.9, INF)], 60_000, 200_000),
}


@pytest.mark.parametrize("name", STACKS)
def test_layered(rules, name):
    q, two, four = STACKS[name]
    a = np.array(q, np.float64)
    for ref in (0, 1):
        assert rules.layered(two, len(q), a.ctypes.data, ref) == 2
        assert four == INF or rules.layered(four, len(q), a.ctypes.data, ref) == 4
    for n in (1, 1000, 19_456):
        assert rules.layered(n, len(q), a.ctypes.data, 0) == 0
        assert rules.layered(n, len(q), a.ctypes.data, 1) != 0
    assert rules.layered(40_000, len(q), a.ctypes.data, 0) != 0

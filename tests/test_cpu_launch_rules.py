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
#include <cstring>
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
int voxel(unsigned long long n, double mua, double mus, int faces) {  // a map of air and this tissue, 2 cm
  nmc_tissue_params tp;
  std::memset(&tp, 0, sizeof tp);
  tp.muav[1] = 1e-4f; tp.musv[1] = 1.f; tp.gv[1] = 1.f;
  tp.muav[2] = (float)mua; tp.musv[2] = (float)mus; tp.gv[2] = 0.9f;
  tp.muav[3] = 1e-3f; tp.musv[3] = 100.f; tp.gv[3] = 0.9f;  // not in the map
  WorkTail w;
  voxel_add(w, (double)n, tp, false, 6u, 2.0);
  const VoxelShape s = voxel_shape(w, n, 152, faces, false);
  return s.block == 256 ? s.per_sm : -s.block;
}
int voxel_sweep(int n_sets, double per, const double* mua, const double* mus) {
  WorkTail w;
  for (int k = 0; k < n_sets; ++k) w.add(per, mua[k], mus[k]);
  return voxel_shape(w, (uint64_t)(n_sets * per), 152, false, true).per_sm;
}
unsigned lanes(unsigned long long items, unsigned long long warps) { return lat_lanes(items, warps); }
}
"""


@pytest.fixture(scope="session")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "nmc_gb300", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), str(d / "rules.cpp"),
                    "-o", str(d / "rules.so")], check=True)
    lib = C.CDLL(str(d / "rules.so"))
    lib.sub_lat.argtypes = [C.c_double] * 3 + [C.c_int]
    lib.sweep_full.argtypes = lib.sweep_lat.argtypes = [C.c_int] + [C.c_double] * 3
    lib.spectrum_lat.argtypes = [C.c_int] + [C.c_void_p] * 3
    lib.field_lat.argtypes = [C.c_double] * 2
    lib.layered.argtypes = [C.c_ulonglong, C.c_int, C.c_void_p, C.c_int]
    lib.voxel.argtypes = [C.c_ulonglong, C.c_double, C.c_double, C.c_int]
    lib.voxel_sweep.argtypes = [C.c_int, C.c_double, C.c_void_p, C.c_void_p]
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


VOXEL = [  # mua, mus, photons, ms at 2, 3, 4 blocks per SM: a cube of one tissue
    (50, 50, 100_000, (0.109, 0.090, 0.090)), (50, 50, 200_000, (0.191, 0.150, 0.139)), (50, 50, 300_000, (0.278, 0.217, 0.195)),
    (20, 100, 100_000, (0.258, 0.209, 0.214)), (20, 100, 200_000, (0.425, 0.351, 0.338)), (20, 100, 400_000, (0.804, 0.645, 0.610)),
    (5, 100, 100_000, (0.758, 0.689, 0.673)), (5, 100, 200_000, (1.177, 1.044, 1.094)), (5, 100, 600_000, (3.082, 2.591, 2.500)),
    (1, 100, 100_000, (2.997, 3.174, 3.104)), (1, 100, 200_000, (4.663, 4.464, 4.626)), (1, 100, 300_000, (6.356, 5.777, 5.912)),
    (0.5, 200, 100_000, (13.93, 15.68, 15.52)), (0.5, 200, 300_000, (21.40, 20.37, 23.32)), (0.5, 200, 1_000_000, (48.19, 42.93, 43.50)),
    (0.2, 100, 100_000, (15.12, 16.07, 15.54)), (0.2, 100, 300_000, (26.18, 24.22, 25.06)),
]


@pytest.mark.parametrize("mua,mus,n,ms", VOXEL)
def test_voxel(rules, mua, mus, n, ms):
    assert ms[rules.voxel(n, mua, mus, 0) - 2] <= 1.05 * min(ms)
    assert rules.voxel(n, mua, mus, 1) == 4


@pytest.mark.parametrize("n,block", [(1, 1), (2432, 1), (2433, 2), (12_160, 5)])
def test_voxel_few_photons(rules, n, block):
    assert rules.voxel(n, 50.0, 50.0, 0) == rules.voxel(n, 0.5, 200.0, 1) == -block


SPECTRA = [  # absorption against the seeded tables', photons, ms at 2, 3, 4 blocks per SM, one-term
    (1, 300_000, (55.7, 60.8, 59.3)), (1, 1_400_000, (69.2, 76.9, 93.9)), (1, 2_500_000, (120.1, 99.3, 112.7)),
    (1, 3_500_000, (167.3, 135.5, 140.3)), (1, 7_000_000, (333.4, 269.4, 251.8)), (20, 1_400_000, (7.59, 6.97, 7.16)),
    (20, 2_500_000, (12.36, 10.48, 10.47)), (20, 5_000_000, (24.7, 19.7, 19.1)), (20, 7_000_000, (34.6, 27.7, 25.5)),
]


@pytest.mark.parametrize("scale,n,ms", SPECTRA)
def test_voxel_sweep(rules, scale, n, ms):
    import nmc_cases as cases

    _, tables, _ = cases.skin_vessel_spectral_tables(seed=2024)
    best = [max(((t.muav[i] * scale + t.musv[i]) / (t.muav[i] * scale), t.muav[i] * scale, t.musv[i]) for i in (2, 3, 4)) for t in tables]
    mua, mus = (np.array([b[k] for b in best]) for k in (1, 2))
    assert ms[rules.voxel_sweep(351, n // 351, mua.ctypes.data, mus.ctypes.data) - 2] <= 1.03 * min(ms)

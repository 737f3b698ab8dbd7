"""The launch rules (nmc_gb300/csrc/launch_rules.h) at media and sizes where both variants were timed on a GB300: the
rule takes the faster one wherever they differ by more than a tenth."""
import ctypes as C
import os
import subprocess

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
int bands_lat(double clear, double per) {  // a share of the sets long-lived, the others not
  WorkTail w;
  for (int k = 0; k < 351; ++k) sweep_add(w, per, k < 351 * clear ? 0.05 : 2.0, 100.0);
  return sweep_latency_pays(w);
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
    lib.sweep_lat.argtypes = [C.c_int] + [C.c_double] * 3
    lib.bands_lat.argtypes = [C.c_double] * 2
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


def test_semi_infinite_sweep_of_bands(rules):
    # the longest photons are a few sets': the work of the others is small beside that tail up to 1e4 photons each
    assert rules.bands_lat(0.25, 8_000) and not rules.bands_lat(0.25, 30_000)

// launch_rules.h - which variant and launch shape a run takes, from its size
// and its media.  Host arithmetic only: no CUDA header, no state.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "nmc_abi.h"

namespace nmc {

// The latency variant of a kernel runs few photons per lane: kLatBlocks blocks
// of kLatBlock threads per SM (4 warps per scheduler, up to 128 registers)
// instead of a full SM, and, when the queue is empty, warps that "go on thin":
// once at most kThinPhotons of a warp's lanes have a photon, the others
// compute the random part of the coming hops, which depends on the photon and
// the hop's number alone.  A photon looks for that every kThinLook scatterings.
constexpr int kLatBlock = 256, kLatBlocks = 2;
constexpr int kThinPhotons = 8;
constexpr unsigned int kThinLook = 16;

// A run's work, in scatterings, and its tail, the scatterings of its longest
// photon.  Few resident photons finish the tail sooner, many do more work per
// second, so each kernel has a ratio of the two up to which fewer pay.
struct WorkTail {
  double work = 0.0, tail = 0.0;
  // n photons in a medium of these coefficients: about 31 (mu_t / mu_a)^0.56
  // scatterings each (measured from 100 to 10,000: 407, 1,490 and 5,330 at 101,
  // 1e3 and 1e4), the longest until its weight reaches the roulette's 1e-4
  void add(double n, double mua, double mus) {
    const double r = std::min((mua + mus) / std::max(mua, 1e-6), 1e6);
    work += n * 31.0 * std::pow(r, 0.56);
    if (n > 0.0) tail = std::max(tail, 9.2 * r);
  }
  bool below(double ratio) const { return work < ratio * tail; }
};

// Lanes of each of `warps` warps that take photons, so that below one item
// per lane they are spread over all the warps that are really resident.
inline unsigned int lat_lanes(uint64_t items, uint64_t warps) {
  return (unsigned int)std::max<uint64_t>(1, std::min<uint64_t>(32, (items + warps - 1) / warps));
}

// The semi-infinite kernel's latency variant.  Its private F(r,z) can leave
// room for one block per SM only (bins 119 to 158): the variant then has 8
// warps per SM where the other kernel has 16, and pays up to a smaller ratio.
// 128 bins, variant against the other, at photons of (mua, mus): (1, 100) 1e4
// 0.59 / 0.96 ms, 7e4 0.89 / 0.98, 1e5 1.10 / 1.00, 3e5 2.54 / 1.94; (10, 100)
// 4e4 0.13 / 0.15, 1e5 0.26 / 0.18; (0.2, 300) 2.5e5 13.0 / 13.2, 1e6 33 / 25;
// the reference's streams cross at the same ratios.  With two blocks (101 bins):
// (1, 100) 2e5 1.29 / 1.48, 2.5e5 1.76 / 1.69, 3e5 1.90 / 1.75; (10, 100) 1e5
// 0.175 / 0.196, 1.5e5 0.24 / 0.20; (0.05, 100) 1e6 30.1 / 31.3: between 1.0e5
// and 1.3e5 in each medium.
inline bool sub_latency_pays(const WorkTail& w, int resident_blocks) {
  return w.below(resident_blocks >= kLatBlocks ? 1.2e5 : 3.7e4);
}

// The semi-infinite sweep: finding a photon's set and loading its constants
// costs about as much as 60 scatterings, which counts for short-lived sets.
inline void sweep_add(WorkTail& w, double n, double mua, double mus) {
  w.add(n, mua, mus);
  w.work += 60.0 * n;
}
// Its latency variant (two blocks are always resident).  351 sets of mua in the
// range given, variant against the other: 0.05-2, 4e3 photons each 9.2 / 11.8
// ms, 1e4 14.4 / 14.2; 0.5-5, 1e3 1.37 / 1.40, 3e3 2.32 / 2.00, two-term 2e3
// 1.89 / 1.96, 4e3 3.20 / 2.53; 3-30, 500 0.29 / 0.27, 1e3 0.43 / 0.38.  Spectra
// with absorption bands, whose few long-lived sets are the tail, 3.5e6 photons
// two-term: 24.2 / 31.8, 28.0 / 36.9 where the ratio is 1.0e5, 19.5 / 22.2 and
// 19.6 / 18.3 at 1.25e5, 11.7 / 10.2 at 1.6e5.
inline bool sweep_latency_pays(const WorkTail& w) { return w.below(1.1e5); }
// Without it, the one-term sweep runs 4 blocks of 64 registers per SM from this
// ratio on, 3 of 74-78 below (two-term keeps 3: it spills at 4).  3 blocks
// against 4: mua 3-30, 3e4 photons each 7.90 / 7.27 ms; 0.5-5, 1e4 5.55 / 5.47,
// 3e4 16.5 / 15.7; 0.05-2, 3e4 26.6 / 28.9, 1e5 88.2 / 85.3; 0.05-0.2, 1e4
// 24.4 / 28.9, 3e4 63.8 / 66.8, 1e5 208 / 205: they cross at 5e5 to 1e6.
inline bool sweep_fills_sm(const WorkTail& w) { return !w.below(7e5); }

// The E-field kernel's latency variant, up to 32 photons per lane.  8 settings,
// variant against the other, photons each: mua 0.01, 1e5 191 / 289 ms, 3.1e5 345
// / 381, 6e5 575 / 563; mua 0.1, 1e5 34.6 / 37.2, 2e5 60.4 / 56.7; mua 1, 2e4
// 2.6 / 3.4, 5e4 4.9 / 4.8, 1e5 8.2 / 7.4; mua 10, 1e4 0.59 / 0.61, 5e4 1.26 /
// 1.15, 3.1e5 5.8 / 4.2: they cross at 1.1e5 to 2.5e5.
inline bool field_latency_pays(const WorkTail& w, uint64_t photons, uint64_t warps) {
  return photons <= warps * 32 * 32 && w.below(1.6e5);
}

// A plane layer as the rule sees it.
struct PlaneLayer {
  double mua, mus, g, thickness;
};

// n photons in a stack: the longest live in the layer with the most scatterings
// per absorption, where leaving the layer counts as absorption at the rate of
// its slowest diffusion mode, D (pi / L)^2, L the thickness and 6 D beyond each
// face (a refractive step of 1.4).  Layers below nine effective attenuation
// lengths are out of reach, layers that do not scatter hold no walk.
inline void layered_add(WorkTail& w, double n, const PlaneLayer* layers, int n_layers) {
  double best = 1.0, depth = 0.0;
  for (int l = 0; l < n_layers && depth < 9.2; ++l) {
    const PlaneLayer& q = layers[l];
    const double tr = q.mua + q.mus * (1.0 - q.g);  // transport coefficient
    if (q.mus > 0.0 && tr > 0.0) {
      const double D = 1.0 / (3.0 * tr);
      double loss = q.mua;
      if (std::isfinite(q.thickness)) loss += D * std::pow(3.14159265358979 / (q.thickness + 12.0 * D), 2);
      best = std::max(best, (loss + q.mus) / std::max(loss, 1e-6));
    }
    depth += std::sqrt(3.0 * q.mua * tr) * q.thickness;
  }
  w.add(n, 1.0, best - 1.0);
}

// The layered kernel's variant and blocks per SM (0: as many as fit, four).
// * Up to kThinPhotons per warp, where every photon has helper lanes from the
//   start, the latency variant: three-layer skin 1e3 photons 5.1 against 5.8 ms,
//   1e4 7.1 / 7.4, 2e4 7.5 / 7.7, 4e4 8.3 / 7.7; mua 10-20 1e4 0.34 / 0.38.
// * Up to eight photons per lane, while the tail outweighs the work, two blocks
//   of the other one.  2 against 4 blocks: skin 3e5 11.0 / 14.2 ms, 6e5 14.9 /
//   15.6, 1e6 21.4 / 19.7; mua 1, mus 100 2e5 1.68 / 1.78, 3e5 2.20 / 2.02; mua
//   10-20 6e4 0.41 / 0.40, 1e5 0.45 / 0.43, 6e5 1.09 / 0.84; 0.3 cm without
//   absorption 2e5 1.12 / 1.14, 3e5 1.40 / 1.31; gradients and the reference's
//   streams cross at the same sizes: at 0.7e5 to 1.2e5.
struct LayeredShape {
  bool latency;
  int blocks;
};
inline LayeredShape layered_shape(const WorkTail& w, uint64_t photons, uint64_t warps, bool sequential) {
  if (!sequential && photons <= warps * kThinPhotons) return {true, kLatBlocks};
  return {false, photons <= warps * 256 && w.below(1.0e5) ? kLatBlocks : 0};
}

// The longest side of a run's voxel grid.
inline double grid_extent(const nmc_run_params& rp) {
  return std::max({(double)rp.Nx * rp.dx, (double)rp.Ny * rp.dy, (double)rp.Nz * rp.dz});
}

// n photons in a voxel grid whose longest side is `extent` and whose map holds
// the tissues of `present` (bit t: tissue t): the longest live in the tissue with
// the most scatterings per absorption.  A tissue too clear to turn a photon within
// the grid (air) holds no walk.
inline void voxel_add(WorkTail& w, double n, const nmc_tissue_params& tp, bool two_term, uint32_t present, double extent) {
  double best = 1.0;
  for (int t = 0; t < NMC_NTISS; ++t) {
    if (!(present >> t & 1u)) continue;
    const double g = two_term ? tp.CC[t] * tp.gf[t] - (1.0 - tp.CC[t]) * tp.gb[t] : (double)tp.gv[t];
    const double mua = tp.muav[t], mus = tp.musv[t];
    if (mus * (1.0 - g) * extent >= 1.0) best = std::max(best, (mua + mus) / std::max(mua, 1e-6));
  }
  w.add(n, 1.0, best - 1.0);
}

// The launch shape of a voxel run whose caller left it to the library, from
// its queue items (photons, or runs of photons) and work against tail.  A voxel
// sub-step takes a lone photon 0.49 us, a photon in a full warp 1.4 us (its 31
// neighbours walk other branches) and one of eight full warps on a scheduler 2
// us, and 4, 6, 8 warps per scheduler give 77, 94, 100% of the throughput:
//  * up to 5 items per warp of two blocks per SM, each warp takes as few items
//    as fill them all (blocks of that many threads): 1e3 photons through the
//    skin-vessel map take 5.9 instead of 10.1 ms, 1e4 8.7 / 10.2;
//  * 2 or 3 blocks per SM while the tail outweighs the work and photons per lane
//    are few (where the estimate from the table may miss a tissue that few photons
//    reach).  2 / 3 / 4 blocks: skin vessel 1e5 13.9 / 15.7 / 15.5 ms, 2e5 16.8 /
//    17.4 / 20.8, 3e5 21.4 / 20.4 / 23.3, 1e6 48.2 / 42.9 / 43.5; a cube of mua 1
//    1e5 3.00 / 3.17 / 3.10, 2e5 4.66 / 4.46 / 4.63; mua 20 1e5 0.26 / 0.21 /
//    0.21, 4e5 0.80 / 0.65 / 0.61; mua 50 2e5 0.19 / 0.15 / 0.14;
//  * a sweep's sets differ and its tail is longer.  351 sets of the skin vessel,
//    one-term 1.4e6 69 / 77 / 94, 2.5e6 120 / 99 / 113, 5e6 239 / 193 / 186; two-
//    term 1.4e6 57 / 66 / 80, 3.5e6 70 / 78 / 96, 7e6 136 / 110 / 120, other
//    spectra at 3.5e6 64 / 57 / 62 and 92 / 100 / 120; with 20 times the
//    absorption one-term 1.4e6 7.6 / 7.0 / 7.2, 3.5e6 17.3 / 14.0 / 13.5;
//  * photons that end at the grid's faces (boundaryflag 1) run on all blocks that
//    fit: how long they live is the grid's size rather than the table's.  Grids
//    that hold them do have the tail (a 2 cm cube of mua 1, 1e5 photons 2.50 /
//    2.66 / 2.68 ms, 3e5 5.14 / 4.72 / 4.83), small ones do not.
struct VoxelShape {
  int block, per_sm;
};
inline VoxelShape voxel_shape(const WorkTail& w, uint64_t items, int nsm, bool ends_at_faces, bool sweep) {
  const uint64_t warps = (uint64_t)nsm * kLatBlocks * (kLatBlock / 32), lanes = warps * 32;
  if (items <= 5 * warps) return {(int)std::max<uint64_t>(1, (items + warps - 1) / warps), 16};
  if (ends_at_faces) return {256, 4};
  if ((sweep ? items <= 26 * lanes : 2 * items <= 3 * lanes) && w.below(sweep ? 1.0e5 : 5e4)) return {256, 2};
  if (items <= (sweep ? 64 : 5) * lanes && w.below(2.7e5)) return {256, 3};
  return {256, 4};
}

}  // namespace nmc

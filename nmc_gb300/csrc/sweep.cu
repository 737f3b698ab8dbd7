// sweep.cu - many parameter sets of the semi-infinite medium (MCSubKernel,
// kernels.metal:59-319) in one persistent launch.
//
// The reference sweeps wavelengths by rewriting its input files and starting
// one process (one pipeline, ten blocking dispatches) per wavelength
// (NMC-samples/example3.ipynb cell 5).  Here every set's photon budget is a
// slice of one global photon index space: threads take photon indices from
// a warp-aggregated counter (work stealing across sets), find the photon's
// set by binary search over the budgets' prefix sums, and load that set's
// optical constants.  The host lays the sets out in decreasing order of
// estimated cost per photon, so the photons that live longest start first.
// Uneven budgets therefore cost nothing extra: the GPU stays full until the
// last photon of the last set, and there is one tail for the whole sweep
// instead of one per set.
// Per-set totals are u64 fixed point in shared memory, folded into global
// memory once per block; the escaping flux J(r) of each set goes straight to
// global u64 atomics (one deposit per escaping photon).
//
// A photon keeps its set's constants in registers.  Read from the table at
// every hop, the lanes of a warp (in different sets) took up to 32 L1 lines
// per load and waited 3.4 cycles per instruction for them.  The kernel needs
// 74-79 registers for it and runs 3 blocks of 256 per SM: 351 two-term sets
// of 1.4e7 photons in 71.0 ms, against 92.3 ms with the table reads at 4
// blocks (and 85.6 ms with the constants in registers squeezed to 4 blocks);
// 3.5e6 photons, where fewer resident photons also shorten the tail, 37.6
// against 53.8 ms.  Sweeps whose tail outweighs their work take the latency
// variant (99 registers, thin warps): the 3.5e6 photons 28.6 ms.  Large one-term
// sweeps run 4 blocks (64 registers, no spills): launch_rules.h.
#include <cuda_runtime.h>

#include "engine.h"

namespace nmc {
namespace {

// LAT: the latency variant; FULL: four blocks per SM (launch_rules.h).
template <int PHASE, bool FAST, bool LAT, bool FULL = false>
__global__ void __launch_bounds__(kLatBlock, LAT ? kLatBlocks : FULL ? 4 : 3) sweep_kernel(const SweepParams P) {
  using M = Math<FAST>;
  constexpr bool TT = PHASE == kPhaseTT;
  extern __shared__ unsigned long long s_sum[];  // nsets x 5: photons, hops, S, A, E
  double* s_e2 = reinterpret_cast<double*>(s_sum + 5 * P.nsets);
  __shared__ int s_idle[LAT ? kLatBlock / 32 : 1];  // lanes of each warp that found the queue empty
  for (int k = threadIdx.x; k < 6 * P.nsets; k += blockDim.x) s_sum[k] = 0ull;
  if (LAT && threadIdx.x < kLatBlock / 32) s_idle[threadIdx.x] = 0;
  __syncthreads();
  const int BINS = P.bins;
  const uint32_t k0 = P.k0;

  PhiloxRng<TT> rng;
  float x = 0.f, y = 0.f, z = 0.f, ux = 0.f, uy = 0.f, uz = 1.f, W = 0.f, step_u = 1.f;
  float rsp = 0.f, Atot = 0.f, E = 0.f;
  // the set's mu_t, 1 - albedo and phase constants, kept over the photon's life
  float mut = 1.f, oma = 0.f;
  PhaseConst ph;
  uint32_t nsc = 0, nsub = 0, k1 = P.k1;
  int set = 0, slot = 0;
  bool alive = false, have = false;

  auto retire = [&]() {
    unsigned long long* b = s_sum + 5 * set;
    atomicAdd(b + 0, 1ull);
    atomicAdd(b + 1, (unsigned long long)nsub);
    atomicAdd(b + 2, to_fix(rsp));
    atomicAdd(b + 3, to_fix(Atot));
    atomicAdd(b + 4, to_fix(E));
    if (E > 0.f) atomicAdd(s_e2 + set, (double)E * (double)E);
  };
  // HOP (:183-187) by s and ESCAPE (:190-214): true when the photon left
  auto hop = [&](float s) {
    x = fmaf(s, ux, x);
    y = fmaf(s, uy, y);
    z = fmaf(s, uz, z);
    ++nsub;
    if (P.boundaryflag == 1 && z <= P.zs) {
      float uz1;
      const SweepSetDev* S = P.sets + slot;
      if (rng.fres_u(k0, k1) > rfresnel(__ldg(&S->n1), __ldg(&S->n2), -uz, &uz1)) {
        x = fmaf(-s, ux, x);
        y = fmaf(-s, uy, y);
        z = fmaf(-s, uz, z);
        const float s2 = fabsf(z / uz);
        x = fmaf(s2, ux, x);
        y = fmaf(s2, uy, y);
        const float r = sqrtf(x * x + y * y);
        int ir = (int)fminf(r * P.idr, (float)BINS) + 1;
        if (ir > BINS) ir = BINS;
        if (P.J) atomicAdd(P.J + (size_t)set * (BINS + 1) + ir, to_fix(W));
        E += W;
        return true;
      }
      z = -z;
      uz = -uz;
    }
    return false;
  };
  auto drop = [&]() {  // DROP (:224-234): absorbed weight only (no F(r,z) in sweeps)
    const float absorb = W * oma;
    W -= absorb;
    Atot += absorb;
  };
  auto phase = [](const PhaseConst& q, float a, float b) {  // cos(theta)
    if (PHASE == kPhaseTT) return tt_sample_param<FAST>(q, a, b);
    if (PHASE == kPhaseIsoRef) return 2.f * a - 1.f;
    return hg_sample<FAST>(q, a);
  };

  const bool idle = LAT && (threadIdx.x & 31) >= P.lanes;
  while (!idle) {
    if (!alive) {
      if (have) retire();
      have = false;
      const unsigned long long g = next_photon(P.work);
      if (g >= P.total) {
        if (LAT) atomicAdd(&s_idle[threadIdx.x >> 5], 1);
        break;
      }
      have = true;
      // queue slot of global photon g: prefix[k] <= g < prefix[k + 1]
      int lo = 0, hi = P.nsets;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(P.prefix + mid) <= g) lo = mid; else hi = mid;
      }
      slot = lo;
      const SweepSetDev* S = P.sets + lo;
      set = (int)__ldg(&S->id);
      k1 = P.k1 + (uint32_t)set;
      rng.init(__ldg(&S->first) + (g - __ldg(P.prefix + lo)));
      // ---- LAUNCH (kernels.metal:106-168) with this set's indices
      const float n1 = __ldg(&S->n1), n2 = __ldg(&S->n2);
      x = y = z = 0.f;
      ux = uy = uz = 0.f;
      rsp = 0.f;
      LaunchDraws d{rng.block(0xFFFFFFFFu, k0, k1), 0};
      if (P.mcflag == 0) {
        x = P.radius * sqrtf(d.next());
        z = P.zs;
        uz = 1.f;
        rsp = __ldg(&S->rsp);
      } else if (P.mcflag == 1) {
        x = P.radius * sqrtf(-logf(d.next()));
        z = P.zs;
        const float xf = P.waist * sqrtf(-logf(d.next()));
        const float temp = sqrtf((x - xf) * (x - xf) + P.zfocus * P.zfocus);
        const float costheta = P.zfocus / temp;
        float uzn = costheta;
        rsp = rfresnel(n2, n1, costheta, &uzn);
        uz = uzn;
        ux = sqrtf(fmaxf(1.f - uz * uz, 0.f));
      } else if (P.mcflag == 2) {
        x = P.xs;
        y = P.ys;
        z = P.zs;
        const float costheta = 1.f - 2.f * d.next();
        const float sintheta = sqrtf(fmaxf(1.f - costheta * costheta, 0.f));
        float sp, cp;
        M::sincos2pi(d.next(), &sp, &cp);
        ux = sintheta * cp;
        uy = sintheta * sp;
        uz = costheta;
      }
      step_u = rng.first_step(k0, k1);
      mut = __ldg(&S->mut);
      oma = 1.f - __ldg(&S->albedo);
      ph = S->ph;
      W = 1.f - rsp;
      Atot = E = 0.f;
      nsc = nsub = 0;
      alive = true;
    }

    if (hop(M::div(M::neglog(step_u), mut))) {
      alive = false;
      continue;
    }
    drop();
    // ---- SPIN (:243-279), ROULETTE (:289-294), next HOP's draw
    const bool need_roul = W < kTHRESHOLD;
    const SpinDraws dr = rng.spin_draws(need_roul, k0, k1);
    const float costheta = phase(ph, dr.a, dr.b);
    const SpinTrig trig = spin_trig<FAST>(costheta, TT ? dr.c : dr.b);
    float nx, ny, nz;
    const bool vertical = spin_try(costheta, trig, ux, uy, uz, nx, ny, nz);
    ++nsc;
    bool leave = false;
    if (__builtin_expect(vertical | need_roul | (LAT && nsc % kThinLook == 0), 0)) {
      if (vertical) spin_vertical(costheta, trig, ux, uy, uz, nx, ny, nz);
      if (need_roul) {
        if (dr.roul <= kCHANCE)
          W /= kCHANCE;
        else
          alive = false;
      }
      if (LAT) {  // go on thin: the queue is empty and few lanes have a photon
        const int none = *(volatile int*)&s_idle[threadIdx.x >> 5];
        leave = (int)P.lanes - none <= kThinPhotons && (none > 0 || *(volatile unsigned long long*)P.work >= P.total);
      }
    }
    ux = nx;
    uy = ny;
    uz = nz;
    step_u = dr.step;
    if (alive && nsub >= P.step_cap) {
      alive = false;
      atomicOr(P.flags, (unsigned int)NMC_DEVFLAG_STEPCAP);
    }
    if (LAT && leave && alive) break;
  }

  if constexpr (LAT) {
    // the lanes without a photon compute the random part of the coming hops
    const unsigned int lane = threadIdx.x & 31, all = 0xFFFFFFFFu;
    float s = alive ? M::div(M::neglog(step_u), mut) : 0.f;
    unsigned int mask;
    while ((mask = __ballot_sync(all, alive)) != 0) {
      const int n = __popc(mask), per = 32 / n;  // photons, and hops of each in this pass
      const int first = __popc(mask & ((1u << lane) - 1u)) * per;  // my photon's first record
      const int q = (int)lane / per, src = (int)__fns(mask, 0, min(q, n - 1) + 1);
      const uint32_t plo = __shfl_sync(all, rng.plo, src), phi = __shfl_sync(all, rng.phi, src);
      const uint32_t h = __shfl_sync(all, nsc, src) + 1u + (lane - q * per), key = __shfl_sync(all, k1, src);
      const SweepSetDev* S = P.sets + __shfl_sync(all, slot, src);
      const uint4 b = philox4x32_10(make_uint4(plo, phi, h, kPhiloxTag), k0, key);
      const float r_cos = phase(S->ph, u01(b.x), u01(b.y));
      const SpinTrig r_trig = spin_trig<FAST>(r_cos, TT ? u01(b.z) : u01(b.y));
      const float r_s = M::div(M::neglog(u01(b.w)), __ldg(&S->mut));
      for (int o = 0; o < per; ++o) {
        const int k = first + o;
        const float costheta = __shfl_sync(all, r_cos, k);
        SpinTrig trig;
        trig.sintheta = __shfl_sync(all, r_trig.sintheta, k);
        trig.sinpsi = __shfl_sync(all, r_trig.sinpsi, k);
        trig.cospsi = __shfl_sync(all, r_trig.cospsi, k);
        const float s_next = __shfl_sync(all, r_s, k);
        const float roul = TT ? 0.f : u01(__shfl_sync(all, b.z, k));
        if (!alive) continue;
        rng.hop = nsc;
        if (hop(s)) {
          alive = false;
          continue;
        }
        drop();
        float nx, ny, nz;
        const bool vertical = spin_try(costheta, trig, ux, uy, uz, nx, ny, nz);
        ++nsc;
        const bool need_roul = W < kTHRESHOLD;
        if (__builtin_expect(vertical | need_roul, 0)) {
          if (vertical) spin_vertical(costheta, trig, ux, uy, uz, nx, ny, nz);
          if (need_roul) {
            const float u = TT ? u01(rng.block(nsc | 0x40000000u, k0, k1).x) : roul;
            if (u <= kCHANCE)
              W /= kCHANCE;
            else
              alive = false;
          }
        }
        ux = nx;
        uy = ny;
        uz = nz;
        s = s_next;
        if (alive && nsub >= P.step_cap) {
          alive = false;
          atomicOr(P.flags, (unsigned int)NMC_DEVFLAG_STEPCAP);
        }
      }
      if (have && !alive) {
        retire();
        have = false;
      }
    }
  }

  __syncthreads();
  for (int k = threadIdx.x; k < 5 * P.nsets; k += blockDim.x)
    if (s_sum[k]) atomicAdd(P.sums + k, s_sum[k]);
  for (int k = threadIdx.x; k < P.nsets; k += blockDim.x)
    if (s_e2[k] != 0.0) atomicAdd(P.e2 + k, s_e2[k]);
}

template <bool FAST, bool LAT>
const void* pick(int phase, bool full) {
  if (!LAT && full && phase == kPhaseHG) return (const void*)sweep_kernel<kPhaseHG, FAST, false, true>;
  if (!LAT && full && phase == kPhaseIsoRef) return (const void*)sweep_kernel<kPhaseIsoRef, FAST, false, true>;
  if (phase == kPhaseTT) return (const void*)sweep_kernel<kPhaseTT, FAST, LAT>;
  if (phase == kPhaseIsoRef) return (const void*)sweep_kernel<kPhaseIsoRef, FAST, LAT>;
  return (const void*)sweep_kernel<kPhaseHG, FAST, LAT>;
}

}  // namespace

size_t sweep_smem_bytes(int nsets) { return (size_t)nsets * 6 * 8; }

cudaError_t sweep_prepare(const SweepParams& p, const void** f, size_t* sh) {
  if (p.lanes > 0)
    *f = p.fast ? pick<true, true>(p.phase_kind, false) : pick<false, true>(p.phase_kind, false);
  else
    *f = p.fast ? pick<true, false>(p.phase_kind, p.full) : pick<false, false>(p.phase_kind, p.full);
  *sh = sweep_smem_bytes(p.nsets);
  // a block's static shared memory counts against the 48 KB it has without
  // this; 1024 sets alone take all of it
  if (*sh > 32 * 1024) return cudaFuncSetAttribute(*f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*sh);
  return cudaSuccess;
}

cudaError_t launch_sweep(const SweepParams& p, int grid, int block, cudaStream_t stream) {
  const void* f;
  size_t sh;
  cudaError_t e = sweep_prepare(p, &f, &sh);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&p};
  return cudaLaunchKernel(f, dim3(grid), dim3(block), args, sh, stream);
}

cudaError_t sweep_occupancy(const SweepParams& p, int block, int* blocks_per_sm) {
  const void* f;
  size_t sh;
  cudaError_t e = sweep_prepare(p, &f, &sh);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, f, block, sh);
}

}  // namespace nmc

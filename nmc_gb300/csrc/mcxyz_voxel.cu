// mcxyz_voxel.cu - the voxel transport kernel for media with per-voxel
// optical properties (no reference counterpart: the reference indexes at most
// 18 tissue types through a uint8 map, definitions.h:57), forward and
// perturbation Monte Carlo adjoint.  The kernel itself is in mcxyz_kernel.cuh.
#include "mcxyz_kernel.cuh"

namespace nmc {
namespace {

const void* pick_voxel(int mode, bool trace, bool fast) {
  if (mode == kAdjoint)
    return fast ? (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, true, kAdjoint>
                : (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, false, kAdjoint>;
  if (mode == kRecord)
    return fast ? (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, true, kRecord>
                : (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, false, kRecord>;
  if (mode == kScore)
    return fast ? (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, true, kScore>
                : (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, false, kScore>;
  if (trace)
    return fast ? (const void*)mcxyz_kernel<false, PhiloxRng<false>, true, true, kVoxel>
                : (const void*)mcxyz_kernel<false, PhiloxRng<false>, true, false, kVoxel>;
  return fast ? (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, true, kVoxel>
              : (const void*)mcxyz_kernel<false, PhiloxRng<false>, false, false, kVoxel>;
}

__global__ void adjoint_scores_kernel(const AdjEvent* __restrict__ ev, unsigned int n, const float* __restrict__ G,
                                      float* __restrict__ D) {
  for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const AdjEvent e = ev[k];
    const float v = G[e.bin] * e.w;
    if (v != 0.f) atomicAdd(D + e.photon, v);
  }
}

// One warp per chunk of the deposit list: each photon's run of records (from
// its header to the next header or the chunk's end) adds its
// sum GF[voxel] * deposit to D[photon] with one atomic.  The kernel is bound by
// reading the list: a warp reads 64 records (512 bytes) at a time.  (One thread
// per 2 KB chunk left 16 of every 128 bytes fetched unused until they had
// fallen out of the L1: 1.33 ms for the 1e6-photon list of a 64^3 medium,
// against 0.66 now.)
__global__ void __launch_bounds__(256) deposit_scores_kernel(const uint2* __restrict__ pool,
                                                             const unsigned int* __restrict__ fill, unsigned int n_chunks,
                                                             const float* __restrict__ GF, float* __restrict__ D,
                                                             unsigned long long n_photons) {
  static_assert(kDepChunk % 64 == 0, "a warp reads 64 records at a time");
  constexpr unsigned int all = 0xFFFFFFFFu, kHeader = 0xFFFFFFFFu;
  const unsigned int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x / 32);
  for (unsigned int c = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; c < n_chunks; c += warps) {
    const uint4* r = reinterpret_cast<const uint4*>(pool + (size_t)c * kDepChunk);
    const int n = (int)min(fill[c], kDepChunk);
    unsigned int p = kHeader;  // the photon of the records at hand; none before the first header
    float sum = 0.f;           // this lane's part of its score
    auto flush = [&]() {
      for (int k = 16; k > 0; k >>= 1) sum += __shfl_xor_sync(all, sum, k);
      if (lane == 0 && p < n_photons && sum != 0.f) atomicAdd(D + p, sum);
      sum = 0.f;
    };
    for (int at = 0; at < n; at += 64) {
      const int i0 = at + 2 * (int)lane;  // this lane's records i0 and i0 + 1
      const uint4 x = i0 < n ? __ldg(r + i0 / 2) : make_uint4(0u, 0u, 0u, 0u);
      const bool has0 = i0 < n, has1 = i0 + 1 < n, h0 = has0 && x.x == kHeader, h1 = has1 && x.z == kHeader;
      const float v0 = has0 && !h0 ? __ldg(GF + x.x) * __uint_as_float(x.y) : 0.f;
      const float v1 = has1 && !h1 ? __ldg(GF + x.z) * __uint_as_float(x.w) : 0.f;
      unsigned int m0 = __ballot_sync(all, h0), m1 = __ballot_sync(all, h1);
      int from = at;  // records before it are in the sums
      while (m0 | m1) {  // the next header, at record `to`
        const int l0 = m0 ? __ffs(m0) - 1 : 32, l1 = m1 ? __ffs(m1) - 1 : 32;
        const bool first = l0 <= l1;
        const int l = first ? l0 : l1, to = at + 2 * l + (first ? 0 : 1);
        if (i0 >= from && i0 < to) sum += v0;
        if (i0 + 1 >= from && i0 + 1 < to) sum += v1;
        flush();
        p = __shfl_sync(all, first ? x.y : x.w, l);
        from = to + 1;
        if (first) m0 &= m0 - 1; else m1 &= m1 - 1;
      }
      if (i0 >= from) sum += v0;
      if (i0 + 1 >= from) sum += v1;
    }
    flush();
  }
}

}  // namespace

cudaError_t launch_deposit_scores(const uint2* pool, const unsigned int* fill, unsigned int n_chunks,
                                  const float* GF, float* D, unsigned long long n_photons, cudaStream_t stream) {
  if (n_chunks == 0) return cudaSuccess;
  const int block = 256;
  const unsigned int blocks = (n_chunks + block / 32 - 1) / (block / 32), grid = blocks < 8192u ? blocks : 8192u;
  deposit_scores_kernel<<<grid, block, 0, stream>>>(pool, fill, n_chunks, GF, D, n_photons);
  return cudaGetLastError();
}

cudaError_t launch_mcxyz_voxel(const XyzParams& p, int mode, bool trace, int grid, int block,
                               cudaStream_t stream) {
  const void* f = pick_voxel(mode, trace, p.fast_math != 0);
  void* args[] = {(void*)&p};
  return cudaLaunchKernel(f, dim3(grid), dim3(block), args, 0, stream);
}

cudaError_t mcxyz_voxel_occupancy(int mode, bool trace, int block, int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, pick_voxel(mode, trace, true), block, 0);
}

cudaError_t launch_adjoint_scores(const AdjEvent* ev, unsigned int n_ev, const float* G, float* D,
                                  cudaStream_t stream) {
  if (n_ev == 0) return cudaSuccess;
  const int block = 256;
  const unsigned int grid = (n_ev + block - 1) / block < 4096u ? (n_ev + block - 1) / block : 4096u;
  adjoint_scores_kernel<<<grid, block, 0, stream>>>(ev, n_ev, G, D);
  return cudaGetLastError();
}

}  // namespace nmc

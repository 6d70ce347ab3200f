// Residual-augmented energy sums in one launch: block partials, and the last
// block to finish adds them in block order (shared by gbcc_energy, the host
// loop and the whole-solve graph, whose decision follows in the same block).
#pragma once

#include "kernels.h"

namespace gbcc {
namespace {

constexpr int kEnergyThreads = 256;

// sums of N values over the block (256 threads), fixed order; valid in thread 0
template <int N>
__device__ __forceinline__ void block_sums(double (&x)[N], double (*sh)[N]) {
#pragma unroll
  for (int q = 0; q < N; ++q)
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) x[q] += __shfl_down_sync(0xffffffffu, x[q], d);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q) sh[warp][q] = x[q];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      double s = sh[0][q];
      for (int w = 1; w < kEnergyThreads / 32; ++w) s += sh[w][q];
      x[q] = s;
    }
  }
  __syncthreads();
}

// g.out[0..3] (kernels.h, launch_energy_terms).  Returns true in thread 0 of the
// last block, after it has written them.  With g.tau null, tau is formed from t1
// and t2 (the same FMA as make_tau_kernel).
__device__ __forceinline__ bool energy_terms(const EnergyTermsArgs& g) {
  __shared__ double sh[kEnergyThreads / 32][4];
  __shared__ bool last;
  const int o = static_cast<int>(g.o), v = static_cast<int>(g.v), o2 = o * o;
  const unsigned vv = static_cast<unsigned>(v) * static_cast<unsigned>(v);
  double s[4] = {0.0, 0.0, 0.0, 0.0};  // r1^2, r2^2, (f + r1) t1, (g + r2)(2 tau - tau')
  for (unsigned p = blockIdx.x; p < vv; p += gridDim.x) {
    const int a = static_cast<int>(p / static_cast<unsigned>(v)), b = static_cast<int>(p - static_cast<unsigned>(a) * v);
    const int64_t po = static_cast<int64_t>(p) * o2, qo = (static_cast<int64_t>(b) * v + a) * o2;
    for (int ij = threadIdx.x; ij < o2; ij += kEnergyThreads) {
      const double r = g.r2[po + ij];
      double tp, tq;
      if (g.tau) {
        tp = g.tau[po + ij];
        tq = g.tau[qo + ij];
      } else {
        const int i = static_cast<int>(static_cast<unsigned>(ij) / static_cast<unsigned>(o)), j = ij - i * o;
        tp = fma(g.t1[a * o + i], g.t1[b * o + j], g.t2[po + ij]);
        tq = fma(g.t1[b * o + i], g.t1[a * o + j], g.t2[qo + ij]);
      }
      s[1] = fma(r, r, s[1]);
      s[3] = fma(g.g_abij[po + ij] + r, 2.0 * tp - tq, s[3]);
    }
  }
  for (int e = blockIdx.x * kEnergyThreads + threadIdx.x; e < v * o; e += gridDim.x * kEnergyThreads) {
    const double r = g.r1[e];
    s[0] = fma(r, r, s[0]);
    s[2] = fma(g.f_ai[e] + r, g.t1[e], s[2]);
  }
  block_sums(s, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) __stcg(g.partial + blockIdx.x * 4 + q, s[q]);
    __threadfence();
    last = atomicAdd(g.count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
#pragma unroll
  for (int q = 0; q < 4; ++q) s[q] = 0.0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += kEnergyThreads) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] += __ldcg(g.partial + b * 4 + q);
  }
  block_sums(s, sh);
  if (threadIdx.x != 0) return false;
  *g.count = 0u;  // ready for the next launch
#pragma unroll
  for (int q = 0; q < 4; ++q) g.out[q] = s[q];
  return true;
}

// blocks: one per pair (a, b), at most kReduceBlocks
inline unsigned energy_blocks(int64_t v) {
  return static_cast<unsigned>(v * v < kReduceBlocks ? v * v : kReduceBlocks);
}

}  // namespace
}  // namespace gbcc

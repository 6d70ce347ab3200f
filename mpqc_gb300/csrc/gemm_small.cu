// Small FP64 contractions, operands read in place:
//
//   C[cm[m] + cn[n]] = beta C[...] + alpha sum_k A(m, k) B(n, k)
//
// where an operand element is the sum of its gather terms (kernels.h) read
// through their offset tables.  One launch replaces two operand packs, a GEMM
// and a K-split reduction.
//
// What bounds it: an SM runs two FP64 FMAs a clock, so a product this small is
// bound by launches and by FP64 work on padding -- a 64 x 64 tile of the panel
// GEMM costs 1 us for every K element whatever part of it is used (57 x 13 x 13
// took 25 us there).  So the tile is cut to the output: tm x tn <= 256 outputs,
// one per thread, tn the even share of N that is at most 16 wide and tm what
// then fits; tiles of fewer than 128 outputs spread K over the warps left
// over.  An FMA per thread needs no register tile: two shared-memory reads a
// warp against the 16 clocks its FMA holds the pipe.  Small outputs with a
// long K are split over blocks; the last block of a tile to finish adds the
// partial tiles in a fixed order, so the result does not depend on which block
// that is.
//
// FP64 water / cc-pVDZ (o = 5, v = 19): a whole solve 17.7 -> 5.6 ms.
#include <algorithm>

#include "kernels.h"

namespace gbcc {
namespace {

constexpr int kThreads = 256;
constexpr int kStep = 32;           // K elements staged at a time
constexpr int kLd = kStep + 1;      // odd: the rows of a warp's reads fall on different banks
constexpr int kMaxRows = 80;        // A rows + B rows of a tile (tm <= 64, tn <= 16)

__device__ __forceinline__ double small_value(const GatherTerm* t, int nterms, bool plain, int64_t r, int64_t c) {
  if (plain) return t[0].a[t[0].ra[r] + t[0].ca[c]];
  double val = 0.0;
  for (int q = 0; q < nterms; ++q) {
    double x = t[q].a[t[q].ra[r] + t[q].ca[c]];
    if (t[q].b) x *= t[q].b[t[q].rb[r] + t[q].cb[c]];
    val = fma(t[q].coef, x, val);
  }
  return val;
}

// rows [r0, r0 + nr) x columns [c0, c0 + kStep) of an operand into S[row][col], zeros outside R x C
__device__ __forceinline__ void stage(const GatherArgs& g, int64_t r0, int nr, int64_t R, int64_t c0, int64_t cend,
                                      double* S) {
  const bool plain = g.plain != 0, along_rows = g.transpose != 0;
#pragma unroll 4
  for (int e = threadIdx.x; e < nr * kStep; e += kThreads) {
    const int r = along_rows ? e % nr : e / kStep;
    const int c = along_rows ? e / nr : e % kStep;
    S[r * kLd + c] =
        (r0 + r < R && c0 + c < cend) ? small_value(g.t, g.nterms, plain, r0 + r, c0 + c) : 0.0;
  }
}

__global__ void __launch_bounds__(kThreads) gemm_small_kernel(const __grid_constant__ GemmSmallArgs g) {
  __shared__ double S[kMaxRows * kLd];
  __shared__ int last;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int tile = blockIdx.x, split = blockIdx.y;
  const int64_t m0 = static_cast<int64_t>(tile / g.ntn) * g.tm, n0 = static_cast<int64_t>(tile % g.ntn) * g.tn;
  const int P = g.tm * g.tn;
  const int W = (P + 31) / 32;         // warps that cover the outputs
  const int KL = kThreads / 32 / W;    // K lanes: every KL-th K element
  const int out = (warp % W) * 32 + lane, kl = warp / W;
  const bool active = out < P && kl < KL;
  const int ar = out / g.tn, bc = out % g.tn;
  const int64_t kbeg = static_cast<int64_t>(split) * g.kps, kend = min(g.K, kbeg + g.kps);
  double* SB = S + g.tm * kLd;
  double acc = 0.0;
  for (int64_t k0 = kbeg; k0 < kend; k0 += kStep) {
    if (k0 != kbeg) __syncthreads();
    stage(g.a, m0, g.tm, g.M, k0, kend, S);
    stage(g.b, n0, g.tn, g.N, k0, kend, SB);
    __syncthreads();
    if (active) {
      const double *pa = S + ar * kLd, *pb = SB + bc * kLd;
      const int kc = static_cast<int>(min(static_cast<int64_t>(kStep), kend - k0));
      for (int k = kl; k < kc; k += KL) acc = fma(pa[k], pb[k], acc);
    }
  }
  // the K lanes of an output, in lane order (kept in S: P KL <= 256 values)
  auto add_lanes = [&]() {
    if (KL == 1) return;
    __syncthreads();
    if (active) S[kl * P + out] = acc;
    __syncthreads();
    if (active && kl == 0)
      for (int q = 1; q < KL; ++q) acc += S[q * P + out];
  };
  add_lanes();
  if (g.ksplit > 1) {
    const int64_t tiles = gridDim.x;
    if (active && kl == 0) __stcg(g.partial + (split * tiles + tile) * kThreads + out, acc);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(g.count + tile, 1u) == static_cast<unsigned>(g.ksplit - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x == 0) g.count[tile] = 0u;  // ready for the next launch
    acc = 0.0;
    if (active) {
      const double* p = g.partial + tile * static_cast<int64_t>(kThreads) + out;
#pragma unroll 8
      for (int s = kl; s < g.ksplit; s += KL) acc += __ldcg(p + s * tiles * kThreads);
    }
    add_lanes();
  }
  const int64_t m = m0 + ar, n = n0 + bc;
  if (active && kl == 0 && m < g.M && n < g.N) {
    double* c = g.C + g.cm[m] + g.cn[n];
    const double x = g.alpha * acc;
    *c = g.beta == 0.0 ? x : fma(g.beta, *c, x);
  }
}

}  // namespace

// The tile and the K split from the time they should take: an FMA holds an
// SM's FP64 pipe for 16 clocks a warp; a staged step of K costs its two
// dependent loads (about 1.6 us) unless the FMAs of the SM's blocks hide it; a
// K split costs the counter and the partial tiles read back (3 us, and 0.1 us
// for every one a thread adds).  Smaller tiles leave warps for K lanes and
// give a product with few outputs more blocks: 13 x 13 x 42237 took 145 us in
// one tile of 169 outputs split 300 ways.
double plan_gemm_small(GemmSmallArgs& g) {
  auto share = [](int64_t n, int64_t most) {  // the even share of n that is at most `most`
    const int64_t parts = (n + most - 1) / most;
    return static_cast<int>((n + parts - 1) / parts);
  };
  const int64_t sms = num_sms();
  double best = 0.0;
  for (const int outputs : {256, 128, 64, 32}) {
    const int tn = share(g.N, 16);
    const int tm = share(g.M, std::max(1, std::min(64, outputs / tn)));
    const int64_t ntn = (g.N + tn - 1) / tn, tiles = ntn * ((g.M + tm - 1) / tm);
    const int W = (tm * tn + 31) / 32, KL = kThreads / 32 / W;
    for (const int64_t want : {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128}) {
      if (want > 1 && want * kStep > g.K) break;
      const int64_t kps = ((g.K + want - 1) / want + 7) / 8 * 8, ks = (g.K + kps - 1) / kps;
      const double fma_us = static_cast<double>((tiles * ks + sms - 1) / sms) * kps * 16 * W / 2000.0;
      const double step_us = 1.6 * static_cast<double>((kps + kStep - 1) / kStep);
      // (a smaller tile stages more for every FMA: 741^3 takes 711 us in tiles
      // of 256 outputs and 957 us in tiles of 128, whose last wave is fuller)
      const double us = std::max(outputs < 256 ? 1.25 * fma_us : fma_us, step_us) + (ks > 1 ? 3.0 + 0.1 * static_cast<double>(ks) / KL : 0.0);
      if (best != 0.0 && us >= best) continue;
      best = us;
      g.tm = tm;
      g.tn = tn;
      g.ntn = static_cast<int>(ntn);
      g.tiles = tiles;
      g.ksplit = static_cast<int>(ks);
      g.kps = static_cast<int>(kps);
    }
  }
  g.partial_elems = g.ksplit > 1 ? static_cast<size_t>(g.ksplit) * g.tiles * kThreads : 0;
  return best;
}

void launch_gemm_small(const GemmSmallArgs& g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0) return;
  const dim3 grid(static_cast<unsigned>(g.tiles), static_cast<unsigned>(g.ksplit));
  gemm_small_kernel<<<grid, kThreads, 0, st>>>(g);
}

}  // namespace gbcc

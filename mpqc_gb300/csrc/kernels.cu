// Elementwise, gather/pack, reduction and DIIS kernels of the CCSD engine.
//
// The amplitude-sized arrays (o^2 v^2 doubles) are streamed once per kernel
// with coalesced accesses, so HBM bandwidth is the bound these kernels aim at.
// GB300 executes FP64 arithmetic and FP64 conversions at ~2 per clock per SM
// (1/64 of FP32), so per-element FP64 work is kept to a few operations: the
// BF16 split works on bit patterns and FP32 remainders, and single-term packs
// are plain copies (their coefficient scales the GEMM instead).
#include "fp_bits.cuh"
#include "energy_terms.cuh"
#include "gather.cuh"
#include "kernels.h"

#include <algorithm>

namespace gbcc {

namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(int64_t n, int threads, int64_t cap = 152 * 32) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return static_cast<unsigned>(b);
}

__global__ void __launch_bounds__(kThreads, 4) gather_kernel(GatherArgs g) {
  const bool rmw = g.out && g.beta != 0.0;
#define GBCC_ROWS(N, P) (rmw ? gather_rows<N, P, true, 0>(g) : gather_rows<N, P, false, 0>(g))
  GBCC_GATHER_DISPATCH(g, GBCC_ROWS);
#undef GBCC_ROWS
}

// 4 K elements per thread into BF16 slices
__global__ void __launch_bounds__(kThreads, 4) gather_split4_kernel(GatherArgs g) {
#define GBCC_SPLIT4(N, P) split4_rows<N, P, 0>(g)
  GBCC_GATHER_DISPATCH(g, GBCC_SPLIT4);
#undef GBCC_SPLIT4
}


// 4 columns per thread into 16-byte aligned FP64 rows (assignments, FP64 panels)
__global__ void __launch_bounds__(kThreads, 3) gather4_f64_kernel(GatherArgs g) {
  const bool rmw = g.beta != 0.0;
#define GBCC_F64X4(N, P) (rmw ? split4_rows<N, P, 2>(g) : split4_rows<N, P, 1>(g))
  GBCC_GATHER_DISPATCH(g, GBCC_F64X4);
#undef GBCC_F64X4
}

__global__ void __launch_bounds__(256) gather_t_kernel(GatherArgs g) {
  __shared__ double tile[32][33];
  const bool rmw = g.out && g.beta != 0.0;
#define GBCC_TILES(N, P) (rmw ? gather_tiles<N, P, true, 0>(g, tile) : gather_tiles<N, P, false, 0>(g, tile))
  GBCC_GATHER_DISPATCH(g, GBCC_TILES);
#undef GBCC_TILES
}

// ---------------------------------------------------------------------------

__device__ __forceinline__ double block_sum(double v, double* sh) {
  // fixed-order tree reduction over the block (deterministic)
  const int tid = threadIdx.x;
  sh[tid] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (tid < s) sh[tid] += sh[tid + s];
    __syncthreads();
  }
  double r = sh[0];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kEnergyThreads) energy_terms_kernel(EnergyTermsArgs g) { (void)energy_terms(g); }

__global__ void __launch_bounds__(kThreads) make_tau_kernel(int64_t o, int64_t v,
                                                            const double* __restrict__ t1,
                                                            const double* __restrict__ t2,
                                                            double* __restrict__ tau) {
  const int64_t o2 = o * o;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t a, b;
    divmod32(p, v, a, b);
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      tau[p * o2 + ij] = fma(t1[a * o + i], t1[b * o + j], t2[p * o2 + ij]);
    }
  }
}

// ---------------------------------------------------------------------------
// Particle-particle ladder over pair-(anti)symmetric combinations.
//
// B(a,b,i,j) = sum_cd G(a,b,c,d) tau(c,d,i,j) splits, with G+ = G_abcd + G_abdc
// (G_abcc on the diagonal), G- = G_abcd - G_abdc, tau+ = (tau_cdij + tau_dcij)/2
// (tau_ccij on the diagonal), tau- = (tau_cdij - tau_dcij)/2, into
//   B = sum_{c<=d} G+ tau+ + sum_{c<d} G- tau-.
// <ab|cd> = <ba|dc> makes G+ symmetric and G- antisymmetric under a<->b, and
// pair-symmetric amplitudes (tau(c,d,i,j) = tau(d,c,j,i)) make tau+ symmetric,
// tau- antisymmetric under i<->j, so the two products are needed for a <= b,
// i <= j (a < b, i < j) only: a quarter of the FLOPs of the plain contraction.
// Pair indices, row-major over the upper triangle:
//   sym(a,b)  = a n - a(a-1)/2 + (b - a)      a <= b < n
//   anti(a,b) = a (n-1) - a(a-1)/2 + (b-a-1)  a < b < n

__device__ __forceinline__ int64_t pair_sym(int64_t a, int64_t b, int64_t n) {
  return a * n - a * (a - 1) / 2 + (b - a);
}
__device__ __forceinline__ int64_t pair_anti(int64_t a, int64_t b, int64_t n) {
  return a * (n - 1) - a * (a - 1) / 2 + (b - a - 1);
}

// One block per (a, b): Gp[sym(a,b)][sym(c,d)], Gm[anti(a,b)][anti(c,d)].  Also
// used for o v^3 blocks (rows = any leading index pair, cols = c <= d) when
// ab_pairs is false: then row r = a*v + b of G maps to row r of the outputs.
__global__ void __launch_bounds__(kThreads) build_gpm_kernel(int64_t rows_v, int64_t v, bool ab_pairs,
                                                             const double* __restrict__ G, double* __restrict__ Gp,
                                                             double* __restrict__ Gm) {
  const int64_t np = v * (v + 1) / 2, nm = v * (v - 1) / 2;
  for (int64_t row = blockIdx.x; row < rows_v * v; row += gridDim.x) {
    int64_t a, b;
    divmod32(row, v, a, b);
    int64_t rp = row, rm = row;
    if (ab_pairs) {
      if (a > b) continue;
      rp = pair_sym(a, b, v);
      rm = a < b ? pair_anti(a, b, v) : -1;
    }
    const double* g = G + row * v * v;
    double* gp = Gp + rp * np;
    double* gm = rm >= 0 ? Gm + rm * nm : nullptr;
    for (int64_t c = 0; c < v; ++c) {
      for (int64_t d = c + threadIdx.x; d < v; d += blockDim.x) {
        const double x = g[c * v + d], y = g[d * v + c];
        gp[pair_sym(c, d, v)] = c < d ? x + y : x;
        if (gm && c < d) gm[pair_anti(c, d, v)] = x - y;
      }
    }
  }
}

// The rows a in [a0, a1) of G+ / G- (pairs a <= b / a < b), from the block
// Gblk[a - a0][b - a0][c][d] = <ab|cd> (b >= a0 only); output rows counted
// from the block's first pair: sym(a,b) - sym(a0,a0) and anti(a,b) - anti(a0,a0+1).
// Bound by memory (the block's rows a <= b read once, G+ and G- written once).  Both
// <ab|cd> and <ab|dc> of a pair of 32 x 32 tiles (C, D), (D, C), C <= D, come from
// shared memory, so every element is read once, along d: reading <ab|dc> down a
// column fetched each 32-byte sector several times (v = 131, one block: 0.84 ->
// 0.80 ms, 3 TB/s; the packed rows start at any multiple of 8 bytes).
__global__ void __launch_bounds__(kThreads) build_gpm_rows_kernel(int64_t a0, int64_t a1, int64_t v,
                                                                  const double* __restrict__ Gblk,
                                                                  double* __restrict__ Gp, double* __restrict__ Gm) {
  __shared__ double sx[32][33];  // [c][d] of tile (C, D)
  __shared__ double sy[32][33];  // [d][c] of tile (D, C)
  const int64_t np = v * (v + 1) / 2, nm = v * (v - 1) / 2, w = v - a0;
  const int64_t p0 = pair_sym(a0, a0, v), m0 = a0 * (v - 1) - a0 * (a0 - 1) / 2;
  const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
  for (int64_t row = blockIdx.x; row < (a1 - a0) * w; row += gridDim.x) {
    int64_t al, bl;
    divmod32(row, w, al, bl);
    const int64_t a = a0 + al, b = a0 + bl;
    if (a > b) continue;
    double* gp = Gp + (pair_sym(a, b, v) - p0) * np;
    double* gm = a < b ? Gm + (pair_anti(a, b, v) - m0) * nm : nullptr;
    const double* g = Gblk + row * v * v;
    for (int64_t C = 0; C < v; C += 32) {
      for (int64_t D = C; D < v; D += 32) {
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
          const int64_t c = C + ty + k, d = D + tx;
          if (c < v && d < v) sx[ty + k][tx] = g[c * v + d];
          const int64_t d2 = D + ty + k, c2 = C + tx;
          if (c2 < v && d2 < v) sy[ty + k][tx] = g[d2 * v + c2];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; k += 8) {
          const int64_t c = C + ty + k, d = D + tx;
          if (d < v && c <= d) {
            const double x = sx[ty + k][tx], y = sy[tx][ty + k];
            gp[pair_sym(c, d, v)] = c < d ? x + y : x;
            if (gm && c < d) gm[pair_anti(c, d, v)] = x - y;
          }
        }
        __syncthreads();
      }
    }
  }
}

// G+ / G- over atomic-orbital pairs from (pq|rs) in chemists' order:
// <pr|qs> = G[p][q][r][s], so Gp[sym(p,r)][sym(q,s)] = (pq|rs) + (ps|rq) and
// Gm[anti(p,r)][anti(q,s)] = (pq|rs) - (ps|rq) (one block per p <= r).
__global__ void __launch_bounds__(kThreads) build_gpm_chem_kernel(int64_t n, const double* __restrict__ G,
                                                                  double* __restrict__ Gp, double* __restrict__ Gm) {
  const int64_t np = n * (n + 1) / 2, nm = n * (n - 1) / 2;
  for (int64_t row = blockIdx.x; row < n * n; row += gridDim.x) {
    int64_t p, r;
    divmod32(row, n, p, r);
    if (p > r) continue;
    double* gp = Gp + pair_sym(p, r, n) * np;
    double* gm = p < r ? Gm + pair_anti(p, r, n) * nm : nullptr;
    for (int64_t q = 0; q < n; ++q) {
      const double* gq = G + ((p * n + q) * n + r) * n;  // (pq|r .)
      for (int64_t s = q + threadIdx.x; s < n; s += blockDim.x) {
        const double x = gq[s];                            // <pr|qs> = (pq|rs)
        const double y = G[((p * n + s) * n + r) * n + q];  // <pr|sq> = (ps|rq)
        gp[pair_sym(q, s, n)] = q < s ? x + y : x;
        if (gm && q < s) gm[pair_anti(q, s, n)] = x - y;
      }
    }
  }
}

// Hole-hole ladder over pair combinations.  With W(k,l,i,j) = W(l,k,j,i) and
// pair-symmetric tau, sum_kl tau(a,b,k,l) W(k,l,i,j) splits like the
// particle-particle ladder: over k <= l into tau+(ab,kl) W+(kl,ij) and over
// k < l into tau-(ab,kl) W-(kl,ij), where tau+- are the ladder's taup / taum
// (tau(a,b,l,k) = tau(b,a,k,l)) and W+ = W(kl,ij) + W(lk,ij) (W(kk,ij) on the
// diagonal), W- = W(kl,ij) - W(lk,ij); the products are symmetric /
// antisymmetric in a <-> b and in i <-> j, so they add to the ladder's Bp / Bm.
// The part sum_cd Gijab(k,l,c,d) tau(c,d,i,j) of W+- is itself a pair
// product: <lk|cd> = <kl|dc> gives W+ = c_kl G+(kl,cd) tau+(cd,ij) and
// W- = 2 G-(kl,cd) tau-(cd,ij), with G+- = G(kl,cd) +- G(kl,dc) (G(kl,cc) on
// the diagonal) and c_kl = 2 (k < l) or 1 (k = l).
//
// Gtp[sym(k,l)][sym(c,d)] = c_kl G+, Gtm[anti(k,l)][anti(c,d)] = 2 G- from
// Gijab[k][l][c][d]; one block per k <= l.
__global__ void __launch_bounds__(kThreads) build_gpm_oo_kernel(int64_t o, int64_t v, const double* __restrict__ G,
                                                                double* __restrict__ Gtp,
                                                                double* __restrict__ Gtm) {
  const int64_t np = v * (v + 1) / 2, nm = v * (v - 1) / 2;
  for (int64_t row = blockIdx.x; row < o * o; row += gridDim.x) {
    int64_t k, l;
    divmod32(row, o, k, l);
    if (k > l) continue;
    const double* g = G + row * v * v;
    double* gp = Gtp + pair_sym(k, l, o) * np;
    double* gm = (Gtm && k < l) ? Gtm + pair_anti(k, l, o) * nm : nullptr;
    const int sk = k < l ? 1 : 0;  // c_kl = 2^sk
    for (int64_t c = 0; c < v; ++c) {
      for (int64_t d = c + threadIdx.x; d < v; d += blockDim.x) {
        const double x = g[c * v + d], y = g[d * v + c];
        gp[pair_sym(c, d, v)] = scale_pow2(c < d ? x + y : x, sk);
        if (gm && c < d) gm[pair_anti(c, d, v)] = scale_pow2(x - y, 1);
      }
    }
  }
}

// Wt[sym(k,l)][sym(i,j)] = W(k,l,i,j) + W(l,k,i,j) (W(k,k,i,j) for k = l) and
// Wm[anti(k,l)][anti(i,j)] = W(k,l,i,j) - W(l,k,i,j), from W[o][o][o][o];
// one block per k <= l.
__global__ void __launch_bounds__(kThreads) pair_combine_oo_kernel(int64_t o, const double* __restrict__ W,
                                                                   double* __restrict__ Wt,
                                                                   double* __restrict__ Wm) {
  const int64_t o2 = o * o, sp = o * (o + 1) / 2, sm = o * (o - 1) / 2;
  for (int64_t row = blockIdx.x; row < o2; row += gridDim.x) {
    int64_t k, l;
    divmod32(row, o, k, l);
    if (k > l) continue;
    const double* x = W + (k * o + l) * o2;
    const double* y = W + (l * o + k) * o2;
    double* wt = Wt + pair_sym(k, l, o) * sp;
    double* wm = (Wm && k < l) ? Wm + pair_anti(k, l, o) * sm : nullptr;
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      if (i > j) continue;
      wt[pair_sym(i, j, o)] = k < l ? x[ij] + y[ij] : x[ij];
      if (wm && i < j) wm[pair_anti(i, j, o)] = x[ij] - y[ij];
    }
  }
}

// One block per (c <= d): taup[sym(c,d)][sym(i,j)], taum[anti(c,d)][anti(i,j)].
__global__ void __launch_bounds__(kThreads) tau_pm_kernel(int64_t o, int64_t v, const double* __restrict__ tau,
                                                          double* __restrict__ taup, double* __restrict__ taum) {
  const int64_t o2 = o * o, sp = o * (o + 1) / 2, sm = o * (o - 1) / 2;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t c, d;
    divmod32(p, v, c, d);
    if (c > d) continue;
    const double* x = tau + (c * v + d) * o2;
    const double* y = tau + (d * v + c) * o2;
    double* tp = taup + pair_sym(c, d, v) * sp;
    double* tm = c < d ? taum + pair_anti(c, d, v) * sm : nullptr;
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      if (i > j) continue;
      if (c == d) {
        tp[pair_sym(i, j, o)] = x[ij];
      } else {
        tp[pair_sym(i, j, o)] = scale_pow2(x[ij] + y[ij], -1);
        if (i < j) tm[pair_anti(i, j, o)] = scale_pow2(x[ij] - y[ij], -1);
      }
    }
  }
}

// out(a,b,i,j) (+)= Bp[sym(ab)][sym(ij)] + s_ab s_ij Bm[anti(ab)][anti(ij)], s = +1 for an
// ordered pair, -1 for a swapped one, 0 on the diagonal.  With ab_pairs false the
// row index r = a*v + b addresses Bp / Bm directly (no symmetry in the row pair).
// ACC: add to out (beta = 1) rather than overwrite it.
template <bool ACC>
__global__ void __launch_bounds__(kThreads) pair_unpack_kernel(int64_t rows_v, int64_t v, int64_t o, bool ab_pairs,
                                                               const double* __restrict__ Bp,
                                                               const double* __restrict__ Bm,
                                                               double* __restrict__ out) {
  const int64_t o2 = o * o, sp = o * (o + 1) / 2, sm = o * (o - 1) / 2;
  for (int64_t row = blockIdx.x; row < rows_v * v; row += gridDim.x) {
    int64_t a, b;
    divmod32(row, v, a, b);
    int64_t rp = row, rm = row;
    bool sab_pos = true;  // s_ab = +1
    if (ab_pairs) {
      const int64_t lo = a < b ? a : b, hi = a < b ? b : a;
      rp = pair_sym(lo, hi, v);
      rm = lo < hi ? pair_anti(lo, hi, v) : -1;
      sab_pos = a < b;
    }
    const double* bp = Bp + rp * sp;
    const double* bm = (Bm && rm >= 0) ? Bm + rm * sm : nullptr;
    double* op = out + row * o2;
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      const int64_t li = i < j ? i : j, hj = i < j ? j : i;
      double val = bp[pair_sym(li, hj, o)];
      if (bm && li < hj) val += flip_sign(bm[pair_anti(li, hj, o)], (i < j) != sab_pos);
      if constexpr (ACC) op[ij] += val;
      else op[ij] = val;
    }
  }
}

// The last pass of r2 (ccsd_r1_r2.h:254-262 and the ladder's unpack):
//   r2(a,b,i,j) (+)= Q(a,b,i,j) + g_abij(a,b,i,j) + P(a,b,i,j),
//   Q(a,b,i,j) = q(a,b,i,j) + q(b,a,j,i),  q = r2u - 0.5 tmp - tmp(b,a,i,j),
// i.e. the symmetrisation r2u(a,b,i,j) + r2u(b,a,j,i) after r2u -= 0.5
// tmp(a,b,i,j) + tmp(b,a,i,j), with P the unpack of pair_unpack_kernel (Bp
// null: none).
//
// Every r2u, tmp and g element is read once, r2 read (if accumulated to) and
// written once; beside that memory traffic (0.5 ms at o = 50, v = 190) the FP64
// pipe, 2 results a clock per SM, bounds it: so Q + P, the same for (a,b,i,j) and
// (b,a,j,i), is formed once (9 operations for two outputs), and pairs are decoded
// in FP32.  One block per pair a <= b holds q(a,b,.,.), q(b,a,.,.) and the pair's
// rows of Bp and Bm in shared memory, loaded as they lie (o^2 consecutive
// elements), and writes r2(a,b,.,.) and r2(b,a,.,.) as they lie; the transposed
// reads are of shared memory, at an odd row length.  Against the tiled kernel
// below: o = 50, v = 190 1.85 -> 0.91 ms, o = 30, v = 120 0.22 -> 0.15.
constexpr int kAssembleSmem = 113 * 1024;

struct AssembleArgs {
  int o, v;
  const double* r2u;
  const double* tmp;
  const double* g;
  const double* Bp;
  const double* Bm;
  double* r2;
};

template <bool ACC>
__global__ void __launch_bounds__(512) r2_assemble_pair_kernel(AssembleArgs A) {
  extern __shared__ double asm_smem[];
  const int o = A.o, v = A.v, o2 = o * o, ld = o | 1, sp = o * (o + 1) / 2, sm = o * (o - 1) / 2;
  double* qa = asm_smem;        // [i][j] of q(a,b,.,.)
  double* qb = qa + o * ld;     // [i][j] of q(b,a,.,.)
  double* sbp = qb + o * ld;
  double* sbm = sbp + sp;
  const int T = blockDim.x, tid = threadIdx.x;
  const int di = T / o, dj = T - di * o, i0 = tid / o, j0 = tid - i0 * o;  // e += T
  for (int64_t p = blockIdx.x; p < static_cast<int64_t>(v) * (v + 1) / 2; p += gridDim.x) {
    // pair (a, b) = p - b (b + 1) / 2, a <= b
    int b = static_cast<int>((sqrtf(8.0f * static_cast<float>(p) + 1.0f) - 1.0f) * 0.5f);
    while (static_cast<int64_t>(b) * (b + 1) / 2 > p) --b;
    while (static_cast<int64_t>(b + 1) * (b + 2) / 2 <= p) ++b;
    const int a = static_cast<int>(p - static_cast<int64_t>(b) * (b + 1) / 2);
    const int64_t ab = (static_cast<int64_t>(a) * v + b) * o2, ba = (static_cast<int64_t>(b) * v + a) * o2;
    const double* bp = A.Bp ? A.Bp + pair_sym(a, b, v) * sp : nullptr;
    const double* bm = (A.Bp && A.Bm && a < b) ? A.Bm + pair_anti(a, b, v) * sm : nullptr;
    {
      const double* __restrict__ ua = A.r2u + ab;
      const double* __restrict__ ub = A.r2u + ba;
      const double* __restrict__ ta = A.tmp + ab;
      const double* __restrict__ tb = A.tmp + ba;
      int i = i0, j = j0;
#pragma unroll 2
      for (int e = tid; e < o2; e += T) {
        const double x = ta[e], y = tb[e];
        qa[i * ld + j] = fma(-0.5, x, ua[e]) - y;
        qb[i * ld + j] = fma(-0.5, y, ub[e]) - x;
        i += di;
        j += dj;
        if (j >= o) {
          j -= o;
          ++i;
        }
      }
      if (bp)
        for (int e = tid; e < sp; e += T) sbp[e] = bp[e];
      if (bm)
        for (int e = tid; e < sm; e += T) sbm[e] = bm[e];
    }
    __syncthreads();
    {
      int i = i0, j = j0;
      for (int e = tid; e < o2; e += T) {
        double x = qa[i * ld + j] + qb[j * ld + i];
        if (bp) {
          // P(a,b,i,j) = P(b,a,j,i): the B- term changes sign with i > j (a < b)
          const int li = min(i, j), hj = max(i, j);
          const int s = li * o - li * (li - 1) / 2 + (hj - li);
          double y = sbp[s];
          if (bm && i != j) y += flip_sign(sbm[s - li - 1], i > j);  // pair_anti
          x += y;
        }
        qa[i * ld + j] = x;  // read by no other thread before the barrier
        i += di;
        j += dj;
        if (j >= o) {
          j -= o;
          ++i;
        }
      }
    }
    __syncthreads();
    {
      const double* __restrict__ ga = A.g + ab;
      const double* __restrict__ gb = A.g + ba;
      double* __restrict__ ra = A.r2 + ab;
      double* __restrict__ rb = A.r2 + ba;
      int i = i0, j = j0;
#pragma unroll 2
      for (int e = tid; e < o2; e += T) {
        const double va = qa[i * ld + j] + ga[e], vb = qa[j * ld + i] + gb[e];
        ra[e] = ACC ? ra[e] + va : va;
        if (a != b) rb[e] = ACC ? rb[e] + vb : vb;
        i += di;
        j += dj;
        if (j >= o) {
          j -= o;
          ++i;
        }
      }
    }
    __syncthreads();
  }
}

// The same for o whose pair does not fit the shared memory above.  Q(b,a,j,i) =
// Q(a,b,i,j) operand for operand, so one block per pair a <= b and 32 x 32 tile
// (I, J) of (i, j) stages q of the tile [a][b][I][J] and of [b][a][J][I] in shared
// memory (coalesced along j and along i) and adds the same Q to r2[a][b][I][J] and
// to r2[b][a][J][I].  On the diagonal a = b only tiles I <= J are taken, and a
// tile I = J once.
__global__ void __launch_bounds__(256) r2_assemble_kernel(int64_t o, int64_t v, const double* __restrict__ r2u,
                                                          const double* __restrict__ tmp,
                                                          const double* __restrict__ g,
                                                          const double* __restrict__ Bp,
                                                          const double* __restrict__ Bm, bool accumulate,
                                                          double* __restrict__ r2) {
  __shared__ double sq[32][33];  // [i][j] of q(a,b,.,.)
  __shared__ double sr[32][33];  // [j][i] of q(b,a,.,.)
  const int64_t o2 = o * o, nt = (o + 31) / 32, nt2 = nt * nt;
  const int64_t sp = o * (o + 1) / 2, sm = o * (o - 1) / 2;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int64_t x = blockIdx.x; x < v * v * nt2; x += gridDim.x) {
    int64_t p, t, a, b, I, J;
    divmod32(x, nt2, p, t);
    divmod32(p, v, a, b);
    if (a > b) continue;
    divmod32(t, nt, I, J);
    if (a == b && I > J) continue;
    const int64_t i0 = I * 32, j0 = J * 32;
    const int64_t ab = (a * v + b) * o2, ba = (b * v + a) * o2;
    for (int k = ty; k < 32; k += 8) {
      const int64_t i = i0 + k, j = j0 + tx;
      if (i < o && j < o) {
        const int64_t e = i * o + j;
        sq[k][tx] = fma(-0.5, tmp[ab + e], r2u[ab + e]) - tmp[ba + e];
      }
      const int64_t jj = j0 + k, ii = i0 + tx;
      if (jj < o && ii < o) {
        const int64_t e = jj * o + ii;
        sr[k][tx] = fma(-0.5, tmp[ba + e], r2u[ba + e]) - tmp[ab + e];
      }
    }
    __syncthreads();
    const double* bp = Bp ? Bp + pair_sym(a, b, v) * sp : nullptr;
    const double* bm = (Bp && Bm && a < b) ? Bm + pair_anti(a, b, v) * sm : nullptr;
    // P(a,b,i,j) = P(b,a,j,i): the B- term changes sign with i > j (a < b)
    auto unpack = [&](int64_t i, int64_t j) {
      const int64_t li = i < j ? i : j, hj = i < j ? j : i;
      double val = bp[pair_sym(li, hj, o)];
      if (bm && li < hj) val += flip_sign(bm[pair_anti(li, hj, o)], i > j);
      return val;
    };
    // r2[a][b][I][J], lanes along j
    for (int k = ty; k < 32; k += 8) {
      const int64_t i = i0 + k, j = j0 + tx;
      if (i < o && j < o) {
        double val = (sq[k][tx] + sr[tx][k]) + g[ab + i * o + j];
        if (bp) val += unpack(i, j);
        double* out = r2 + ab + i * o + j;
        *out = accumulate ? *out + val : val;
      }
    }
    // r2[b][a][J][I], lanes along i
    if (a != b || I != J) {
      for (int k = ty; k < 32; k += 8) {
        const int64_t j = j0 + k, i = i0 + tx;
        if (i < o && j < o) {
          double val = (sq[tx][k] + sr[k][tx]) + g[ba + j * o + i];
          if (bp) val += unpack(i, j);
          double* out = r2 + ba + j * o + i;
          *out = accumulate ? *out + val : val;
        }
      }
    }
    __syncthreads();
  }
}

// g_ac's Giabc term (ccsd_intermediates.h F_VV) read off the diagonals i = k
// of two contractions the residual performs anyway: with
//   Z(k,a,c,i) = sum_d Giabc(k,a,d,c) t1(d,i)   (added to K(k,a,i,c))
//   Q(k,a,c,i) = sum_d (2 Giabc(k,a,c,d) - Giabc(k,a,d,c)) t1(d,i)   (added to P(a,k,i,c))
// sum_kd (2 Giabc(k,a,d,c) - Giabc(k,a,c,d)) t1(d,k) = sum_k 1.5 Z(k,a,c,k) - 0.5 Q(k,a,c,k).
// The increments are the differences of the diagonals after and before
// those contractions: diag_snapshot stores K(k,a,k,c) (which = 0) or
// P(a,k,k,c) (which = 1) as d[k][a][c]; gac_from_diagonals adds the sum.
__global__ void __launch_bounds__(kThreads) diag_snapshot_kernel(int64_t o, int64_t v, int which,
                                                                 const double* __restrict__ X,
                                                                 double* __restrict__ d) {
  const int64_t n = o * v * v;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t ka, c, k, a;
    divmod32(e, v, ka, c);
    divmod32(ka, v, k, a);
    d[e] = which == 0 ? X[((k * v + a) * o + k) * v + c] : X[((a * o + k) * o + k) * v + c];
  }
}

__global__ void __launch_bounds__(kThreads) gac_from_diagonals_kernel(int64_t o, int64_t v,
                                                                      const double* __restrict__ K,
                                                                      const double* __restrict__ P,
                                                                      const double* __restrict__ dK,
                                                                      const double* __restrict__ dP,
                                                                      double* __restrict__ gac) {
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < v * v;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t a, c;
    divmod32(e, v, a, c);
    double s = 0.0;
    for (int64_t k = 0; k < o; ++k) {
      const int64_t kac = (k * v + a) * v + c;
      const double z = K[((k * v + a) * o + k) * v + c] - dK[kac];
      const double q = P[((a * o + k) * o + k) * v + c] - dP[kac];
      s = fma(1.5, z, fma(-0.5, q, s));
    }
    gac[e] += s;
  }
}

// r1(a,i) += sum_k 2 tmp2(k,a,k,i) - tmp2(k,a,i,k) with tmp2[o][v][o][o]: the
// (2 Giabc(k,a,c,d) - Giabc(k,a,d,c)) tau(c,d,k,i) term of r1 read off the
// ladder's tmp2(k,a,i,j) = Giabc(k,a,c,d) tau(c,d,i,j), using
// tau(c,d,k,i) = tau(d,c,i,k)
__global__ void __launch_bounds__(kThreads) r1_from_tmp2_kernel(int64_t o, int64_t v,
                                                                const double* __restrict__ tmp2,
                                                                double* __restrict__ r1) {
  const int64_t n = v * o;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t a, i;
    divmod32(e, o, a, i);
    double s = 0.0;
    for (int64_t k = 0; k < o; ++k) {
      const double* p = tmp2 + (k * v + a) * o * o;
      s = fma(2.0, p[k * o + i], s);
      s -= p[i * o + k];
    }
    r1[e] += s;
  }
}

// t += r / D in place (the Jacobi step of lcao/cc/solvers.h:165-258 without
// DIIS), used to build probe amplitudes for the slice calibration
__global__ void __launch_bounds__(kThreads) jacobi_inplace_kernel(int64_t o, int64_t v, const double* eps_o,
                                                                  const double* eps_v, const double* r1,
                                                                  const double* r2, double* t1, double* t2) {
  const int64_t o2 = o * o;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t a, b;
    divmod32(p, v, a, b);
    const double eab = eps_v[a] + eps_v[b];
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      t2[p * o2 + ij] += r2[p * o2 + ij] / (eps_o[i] + eps_o[j] - eab);
    }
  }
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < v * o;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t a, i;
    divmod32(e, o, a, i);
    t1[e] += r1[e] / (eps_o[i] - eps_v[a]);
  }
}

// dinv2[a][b][i][j] = 1 / (eps_o[i] + eps_o[j] - eps_v[a] - eps_v[b]),
// dinv1[a][i] = 1 / (eps_o[i] - eps_v[a])
__global__ void __launch_bounds__(kThreads) denominators_kernel(int64_t o, int64_t v, const double* eps_o,
                                                                const double* eps_v, double* dinv1,
                                                                double* dinv2) {
  const int64_t o2 = o * o;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t a, b;
    divmod32(p, v, a, b);
    const double eab = eps_v[a] + eps_v[b];
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      dinv2[p * o2 + ij] = 1.0 / (eps_o[i] + eps_o[j] - eab);
    }
  }
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < v * o;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    int64_t a, i;
    divmod32(e, o, a, i);
    dinv1[e] = 1.0 / (eps_o[i] - eps_v[a]);
  }
}

// |x| as its bit pattern: for non-negative doubles the unsigned order of the
// bits is the order of the values (NaN above infinity), so maxima of |x| are
// integer maxima and take no FP64 instruction
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7FFFFFFFFFFFFFFFull;
}

// block maxima of two bit patterns, combined into out[0..1] with atomicMax
__device__ __forceinline__ void block_max2_bits(unsigned long long md, unsigned long long mb,
                                                unsigned long long* out) {
  __shared__ unsigned long long sd[kThreads], sb[kThreads];
  sd[threadIdx.x] = md;
  sb[threadIdx.x] = mb;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      sd[threadIdx.x] = max(sd[threadIdx.x], sd[threadIdx.x + w]);
      sb[threadIdx.x] = max(sb[threadIdx.x], sb[threadIdx.x + w]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicMax(out, sd[0]);
    atomicMax(out + 1, sb[0]);
  }
}

// out[0] = bits of max |t2(a,b,i,j) - t2(b,a,j,i)|, out[1] = bits of max |t2|
// (out zeroed by the caller); a NaN anywhere makes the maximum a NaN
__global__ void __launch_bounds__(kThreads) pair_asym_kernel(int64_t o, int64_t v, const double* t2,
                                                             unsigned long long* out) {
  const int64_t o2 = o * o;
  unsigned long long md = 0ull, mb = 0ull;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t a, b;
    divmod32(p, v, a, b);
    const double* x = t2 + p * o2;
    const double* y = t2 + (b * v + a) * o2;
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      const double xv = x[ij];
      md = max(md, abs_bits(xv - y[j * o + i]));
      mb = max(mb, abs_bits(xv));
    }
  }
  block_max2_bits(md, mb, out);
}

// out[0] = bits of max |a - b|, out[1] = bits of max |b| (out zeroed by the caller): block
// maxima combined with atomicMax on the bit patterns, which order like the
// values for non-negative doubles
__global__ void __launch_bounds__(kThreads) maxabs_diff_kernel(int64_t n, const double* a, const double* b,
                                                               unsigned long long* out) {
  unsigned long long md = 0ull, mb = 0ull;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double bv = b[e];
    md = max(md, abs_bits(a[e] - bv));
    mb = max(mb, abs_bits(bv));
  }
  block_max2_bits(md, mb, out);
}

// ---------------------------------------------------------------------------
// DIIS

constexpr int kDiisMax = 16;

// slot, nvec, slots and the extrapolation flag of this DIIS step, from the
// launch arguments or (graph solve) from device memory, into shared memory
struct DiisMeta {
  int slot, nvec, extrapolate;
  int slots[kDiisMax];
};

__device__ __forceinline__ void load_diis_meta(const DiisArgs& d, DiisMeta* m) {
  const DiisDyn* y = d.dyn;
  if (threadIdx.x < kDiisMax) m->slots[threadIdx.x] = y ? y->slots[threadIdx.x] : d.slots[threadIdx.x];
  if (threadIdx.x == 0) {
    m->slot = y ? y->slot : d.slot;
    m->nvec = y ? y->nvec : d.nvec;
    m->extrapolate = y ? y->extrapolate : d.extrapolate;
  }
  __syncthreads();
}

// |det| of the normalised bordered DIIS matrix below which the oldest stored
// vector is dropped (TiledArray's TA::DIIS test, threshold fixed by the water
// 6-31G iteration trace MPQC records in its validation outputs).
constexpr double kDiisDetMin = 1.0e-15;

// The bordered system of a DIIS step, in shared memory for one warp.
struct DiisSystem {
  double A[(kDiisMax + 1) * (kDiisMax + 1)];
  double rhs[kDiisMax + 1], sol[kDiisMax + 1], f[kDiisMax + 1];
};

// Gaussian elimination with partial pivoting on the row-major n x n system, by
// one warp (every element sees the operations of the serial algorithm in its
// order); returns |det A| (product of the pivots), 0 with sol unset if a pivot
// is zero.  (One thread on arrays in local memory took most of a small solve's
// time outside its residuals.)
__device__ double gepp(DiisSystem& S, int n) {
  const int lane = threadIdx.x % 32;
  double* A = S.A;
  double det = 1.0;
  for (int col = 0; col < n; ++col) {
    // the first row of the largest |A[r][col]|
    double best = (lane >= col && lane < n) ? fabs(A[lane * n + col]) : -1.0;
    int p = lane;
    for (int d = 16; d > 0; d >>= 1) {
      const double ob = __shfl_down_sync(0xffffffffu, best, d);
      const int op = __shfl_down_sync(0xffffffffu, p, d);
      if (ob > best || (ob == best && op < p)) {
        best = ob;
        p = op;
      }
    }
    best = __shfl_sync(0xffffffffu, best, 0);
    p = __shfl_sync(0xffffffffu, p, 0);
    if (!(best > 0.0)) return best == 0.0 ? 0.0 : best;
    det *= best;
    if (p != col) {
      if (lane < n) {
        const double t = A[col * n + lane];
        A[col * n + lane] = A[p * n + lane];
        A[p * n + lane] = t;
      }
      if (lane == 0) {
        const double t = S.rhs[col];
        S.rhs[col] = S.rhs[p];
        S.rhs[p] = t;
      }
      __syncwarp();
    }
    if (lane > col && lane < n) {
      const double f = A[lane * n + col] / A[col * n + col];
      S.f[lane] = f;
      S.rhs[lane] -= f * S.rhs[col];
    }
    __syncwarp();
    const int w = n - col;
    for (int e = lane; e < (w - 1) * w; e += 32) {
      const int r = col + 1 + e / w, c = col + e % w;
      A[r * n + c] -= S.f[r] * A[col * n + c];
    }
    __syncwarp();
  }
  if (lane == 0) {
    for (int r = n - 1; r >= 0; --r) {
      double s = S.rhs[r];
      for (int c = r + 1; c < n; ++c) s -= A[r * n + c] * S.sol[c];
      S.sol[r] = s / A[r * n + r];
    }
  }
  __syncwarp();
  return det;
}

// DIIS coefficients (TiledArray's TA::DIIS extrapolation, cc/solvers.h:112-121)
// from the B matrix of the n stored vectors (slots, oldest first, B by slot
// with leading dimension nd): the bordered system [[0, -1], [-1, B]] on the
// newest n - nskip vectors, normalised by the oldest kept <e, e>, damped on
// the diagonal; the oldest vectors are dropped while |det| < kDiisDetMin (a
// singular or near-singular B), the newest alone as the last resort.  coef
// (by slot, nd entries) is written; returns nskip.  Called by one warp.
__device__ int diis_coefficients(DiisSystem& S, const double* Bmat, int nd, const int* slots, int n, double damping,
                                 double* coef) {
  const int lane = threadIdx.x % 32;
  if (lane < nd) coef[lane] = 0.0;
  for (int nskip = 0; nskip < n; ++nskip) {
    const int m = n - nskip;
    const int w = m + 1;
    // normalise by the oldest kept vector's <e, e>
    const double b0 = fabs(Bmat[slots[nskip] * nd + slots[nskip]]);
    const double norm = b0 > 0.0 ? 1.0 / b0 : 1.0;
    __syncwarp();
    if (lane < w) S.rhs[lane] = (lane == 0) ? -1.0 : 0.0;
    for (int e = lane; e < w * w; e += 32) {
      const int r = e / w, c = e % w;
      double val;
      if (r == 0 && c == 0) val = 0.0;
      else if (r == 0 || c == 0) val = -1.0;
      else val = Bmat[slots[nskip + r - 1] * nd + slots[nskip + c - 1]] * norm;
      if (r > 0 && r == c) val *= 1.0 + damping;
      S.A[e] = val;
    }
    __syncwarp();
    const double det = gepp(S, w);
    if (det > 0.0 && (det >= kDiisDetMin || nskip == n - 1)) {
      if (lane < m) coef[slots[nskip + lane]] = S.sol[lane + 1];
      return nskip;
    }
  }
  __syncwarp();
  if (lane == 0) coef[slots[n - 1]] = 1.0;
  return n - 1;
}

// test hook: diis_coefficients on a given B (slots 0..n-1 in order)
__global__ void diis_coefficients_test_kernel(const double* Bmat, int n, double damping, double* coef,
                                              int* nskip) {
  __shared__ DiisSystem S;
  int slots[kDiisMax];
  for (int q = 0; q < n; ++q) slots[q] = q;
  const int k = diis_coefficients(S, Bmat, n, slots, n, damping, coef);
  if (threadIdx.x == 0) *nskip = k;
}

// Sums of the block partials into the new row and column of B, and the
// coefficients: the last block of diis_jacobi_dots_kernel.
__device__ void diis_solve(const DiisArgs& d, const DiisMeta& meta, unsigned nblocks) {
  __shared__ double dots[kDiisMax];
  __shared__ DiisSystem S;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int slot = meta.slot;
  for (int q = warp; q < meta.nvec; q += kThreads / 32) {
    double s = 0.0;
    for (unsigned b = lane; b < nblocks; b += 32) s += __ldcg(d.partial + b * kDiisMax + q);
    for (int m = 16; m > 0; m >>= 1) s += __shfl_down_sync(0xffffffffu, s, m);
    if (lane == 0) dots[q] = s;
  }
  __syncthreads();
  if (warp != 0) return;
  const int nd = d.ndiis;
  const int* slots = meta.slots;
  if (lane < meta.nvec) {
    d.Bmat[slot * nd + slots[lane]] = dots[lane];
    d.Bmat[slots[lane] * nd + slot] = dots[lane];
  }
  __syncwarp();
  if (!meta.extrapolate) {
    if (lane < nd) d.coef[lane] = lane == slot ? 1.0 : 0.0;
    if (lane == 0) *d.nskip_out = -1;
    return;
  }
  const int k = diis_coefficients(S, d.Bmat, nd, slots, meta.nvec, d.damping, d.coef);
  if (lane == 0) *d.nskip_out = k;
}

__global__ void __launch_bounds__(kThreads) diis_jacobi_dots_kernel(DiisArgs d) {
  __shared__ double sh[kThreads];
  __shared__ DiisMeta meta;
  __shared__ bool last;
  load_diis_meta(d, &meta);
  const int slot = meta.slot, nvec = meta.nvec;
  const int64_t o = d.o, v = d.v, o2 = o * o, n2 = v * v * o2, n1 = v * o;
  double acc[kDiisMax];
#pragma unroll
  for (int q = 0; q < kDiisMax; ++q) acc[q] = 0.0;
  double* x2n = d.x2 + static_cast<int64_t>(slot) * n2;
  double* e2n = d.e2 + static_cast<int64_t>(slot) * n2;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      const int64_t e = p * o2 + ij;
      const double r = d.r2[e];
      x2n[e] = fma(r, d.dinv2[e], d.t2[e]);
      e2n[e] = r;
#pragma unroll
      for (int q = 0; q < kDiisMax; ++q) {
        if (q < nvec) {
          const int sq = meta.slots[q];
          const double eq = (sq == slot) ? r : d.e2[static_cast<int64_t>(sq) * n2 + e];
          acc[q] = fma(r, eq, acc[q]);
        }
      }
    }
  }
  double* x1n = d.x1 + static_cast<int64_t>(slot) * n1;
  double* e1n = d.e1 + static_cast<int64_t>(slot) * n1;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n1;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double r = d.r1[e];
    x1n[e] = fma(r, d.dinv1[e], d.t1[e]);
    e1n[e] = r;
#pragma unroll
    for (int q = 0; q < kDiisMax; ++q) {
      if (q < nvec) {
        const int sq = meta.slots[q];
        const double eq = (sq == slot) ? r : d.e1[static_cast<int64_t>(sq) * n1 + e];
        acc[q] = fma(r, eq, acc[q]);
      }
    }
  }
  for (int q = 0; q < nvec; ++q) {
    const double s = block_sum(acc[q], sh);
    if (threadIdx.x == 0) __stcg(d.partial + blockIdx.x * kDiisMax + q, s);
  }
  // the last block to finish solves for the coefficients
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(d.count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) *d.count = 0u;  // ready for the next launch
  diis_solve(d, meta, gridDim.x);
}

struct ExtrapArgs {
  int64_t o, v;
  const double* x1;
  const double* x2;
  const double* coef;
  int nvec;
  int slots[kDiisMax];
  double* t1;
  double* t2;
  double* tau;
  const DiisDyn* dyn;  // non-NULL: nvec and slots from device memory
};

__device__ __forceinline__ void load_extrap_meta(const ExtrapArgs& x, int* s_slots, int* s_nvec) {
  if (threadIdx.x < kDiisMax) s_slots[threadIdx.x] = x.dyn ? x.dyn->slots[threadIdx.x] : x.slots[threadIdx.x];
  if (threadIdx.x == 0) *s_nvec = x.dyn ? x.dyn->nvec : x.nvec;
  __syncthreads();
}

// t1, t2 and tau of the extrapolated amplitudes.  FUSED: a block forms the rows
// a and b of t1 that its tau needs (2 o FMA chains beside o^2 of them) and blocks
// (a, 0) store them; otherwise (rows beyond shared memory) t1 is there already.
constexpr int kExtrapRows = 1024;  // o of the fused form

__global__ void __launch_bounds__(kThreads) extrapolate_t1_kernel(ExtrapArgs x) {
  __shared__ int slots[kDiisMax];
  __shared__ int nvec;
  load_extrap_meta(x, slots, &nvec);
  const int64_t n1 = x.v * x.o;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n1;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double acc = 0.0;
    for (int q = 0; q < nvec; ++q) acc = fma(x.coef[slots[q]], x.x1[slots[q] * n1 + e], acc);
    x.t1[e] = acc;
  }
}

template <bool FUSED>
__global__ void __launch_bounds__(kThreads) extrapolate_t2_tau_kernel(ExtrapArgs x) {
  __shared__ int slots[kDiisMax];
  __shared__ int s_nvec;
  __shared__ double rows[FUSED ? 2 * kExtrapRows : 1];
  load_extrap_meta(x, slots, &s_nvec);
  const int nvec = s_nvec;
  const int64_t o = x.o, v = x.v, o2 = o * o, n2 = v * v * o2, n1 = v * o;
  double c[kDiisMax];
  for (int q = 0; q < kDiisMax; ++q) c[q] = (q < nvec) ? x.coef[slots[q]] : 0.0;
  for (int64_t p = blockIdx.x; p < v * v; p += gridDim.x) {
    int64_t a, b;
    divmod32(p, v, a, b);
    const double *ta = x.t1 + a * o, *tb = x.t1 + b * o;
    if constexpr (FUSED) {
      __syncthreads();
      for (int e = threadIdx.x; e < 2 * o; e += blockDim.x) {
        const bool second = e >= o;
        const int64_t at = second ? b * o + e - o : a * o + e;
        double acc = 0.0;
        for (int q = 0; q < nvec; ++q) acc = fma(c[q], x.x1[slots[q] * n1 + at], acc);
        rows[second ? kExtrapRows + e - o : e] = acc;
        if (!second && b == 0) x.t1[at] = acc;
      }
      __syncthreads();
      ta = rows;
      tb = rows + kExtrapRows;
    }
    for (int64_t ij = threadIdx.x; ij < o2; ij += blockDim.x) {
      int64_t i, j;
      divmod32(ij, o, i, j);
      const int64_t e = p * o2 + ij;
      double acc = 0.0;
      for (int q = 0; q < nvec; ++q) acc = fma(c[q], x.x2[slots[q] * n2 + e], acc);
      x.t2[e] = acc;
      x.tau[e] = fma(ta[i], tb[j], acc);
    }
  }
}

__global__ void __launch_bounds__(kThreads) splitk_reduce_kernel(int64_t M, int64_t N, int ksplit,
                                                                 const double* __restrict__ partial,
                                                                 int64_t rows, int64_t ldp, double* C,
                                                                 const int64_t* __restrict__ cm,
                                                                 const int64_t* __restrict__ cn,
                                                                 double alpha, double beta) {
  const int64_t total = M * N;
  const int64_t split_stride = rows * ldp;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = e / N, n = e - m * N;
    const double* p = partial + m * ldp + n;
    double acc = 0.0;
    for (int s = 0; s < ksplit; ++s) acc += p[s * split_stride];
    double* c = C + cm[m] + cn[n];
    *c = (beta == 0.0) ? alpha * acc : fma(beta, *c, alpha * acc);
  }
}

__global__ void split_test_kernel(const double* x, int64_t n, int nslices, unsigned short* out) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    unsigned short b[3];
    split_bits(x[i], b, nslices);
    for (int s = 0; s < nslices; ++s) out[s * n + i] = b[s];
  }
}

__global__ void scale_test_kernel(const double* x, int64_t n, GatherTerm T, double* out) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = T.pow2 ? term_scale(T, x[i]) : x[i] * T.coef;  // as the gathers dispatch
}

}  // namespace

void launch_scale_test(const double* x, int64_t n, double coef, double* out, cudaStream_t st) {
  if (n <= 0) return;
  GatherTerm T{};
  gather_set_coef(T, coef);
  scale_test_kernel<<<static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 4096)), 256, 0, st>>>(x, n, T, out);
}

void launch_split_test(const double* x, int64_t n, int nslices, unsigned short* out, cudaStream_t st) {
  if (n <= 0) return;
  split_test_kernel<<<static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, 4096)), 256, 0, st>>>(
      x, n, nslices, out);
}

int num_sms() {
  static const int sms = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  }();
  return sms;
}

void launch_splitk_reduce(int64_t M, int64_t N, int ksplit, const double* partial, int64_t rows,
                          int64_t ldp, double* C, const int64_t* cm, const int64_t* cn, double alpha,
                          double beta, cudaStream_t st) {
  if (M <= 0 || N <= 0) return;
  splitk_reduce_kernel<<<grid_for(M * N, kThreads), kThreads, 0, st>>>(M, N, ksplit, partial, rows, ldp, C,
                                                                      cm, cn, alpha, beta);
}

// ---------------------------------------------------------------------------
// launchers

void launch_gather(const GatherArgs& g, cudaStream_t st) {
  if (g.Rpad <= 0 || g.Cpad <= 0) return;
  if (g.outs && g.fixed) {
    launch_gather_fixed(g, st);
    return;
  }
  const GatherShape sh = gather_shape(g);
  if (sh.kind == GatherShape::kTiles) gather_t_kernel<<<sh.grid, sh.block, 0, st>>>(g);
  else if (sh.kind == GatherShape::kFour && g.outs) gather_split4_kernel<<<sh.grid, sh.block, 0, st>>>(g);
  else if (sh.kind == GatherShape::kFour) gather4_f64_kernel<<<sh.grid, sh.block, 0, st>>>(g);
  else gather_kernel<<<sh.grid, sh.block, 0, st>>>(g);
}

void launch_energy_terms(const EnergyTermsArgs& g, cudaStream_t st) {
  energy_terms_kernel<<<energy_blocks(g.v), kEnergyThreads, 0, st>>>(g);
}

void launch_make_tau(int64_t o, int64_t v, const double* t1, const double* t2, double* tau,
                     cudaStream_t st) {
  make_tau_kernel<<<grid_for(v * v, 1), kThreads, 0, st>>>(o, v, t1, t2, tau);
}

void launch_build_gpm(int64_t rows_v, int64_t v, bool ab_pairs, const double* G, double* Gp, double* Gm,
                      cudaStream_t st) {
  build_gpm_kernel<<<grid_for(rows_v * v, 1), kThreads, 0, st>>>(rows_v, v, ab_pairs, G, Gp, Gm);
}

void launch_build_gpm_oo(int64_t o, int64_t v, const double* Gijab, double* Gtp, double* Gtm, cudaStream_t st) {
  build_gpm_oo_kernel<<<grid_for(o * o, 1), kThreads, 0, st>>>(o, v, Gijab, Gtp, Gtm);
}

void launch_pair_combine_oo(int64_t o, const double* W, double* Wt, double* Wm, cudaStream_t st) {
  pair_combine_oo_kernel<<<grid_for(o * o, 1), kThreads, 0, st>>>(o, W, Wt, Wm);
}

void launch_build_gpm_chem(int64_t n, const double* G, double* Gp, double* Gm, cudaStream_t st) {
  build_gpm_chem_kernel<<<grid_for(n * n, 1), kThreads, 0, st>>>(n, G, Gp, Gm);
}

void launch_build_gpm_rows(int64_t a0, int64_t a1, int64_t v, const double* Gblk, double* Gp, double* Gm,
                           cudaStream_t st) {
  if (a1 <= a0) return;
  build_gpm_rows_kernel<<<grid_for((a1 - a0) * (v - a0), 1), kThreads, 0, st>>>(a0, a1, v, Gblk, Gp, Gm);
}

void launch_tau_pm(int64_t o, int64_t v, const double* tau, double* taup, double* taum, cudaStream_t st) {
  tau_pm_kernel<<<grid_for(v * v, 1), kThreads, 0, st>>>(o, v, tau, taup, taum);
}

void launch_pair_unpack(int64_t rows_v, int64_t v, int64_t o, bool ab_pairs, const double* Bp, const double* Bm,
                        double beta, double* out, cudaStream_t st) {
  if (beta == 0.0)
    pair_unpack_kernel<false><<<grid_for(rows_v * v, 1), kThreads, 0, st>>>(rows_v, v, o, ab_pairs, Bp, Bm, out);
  else
    pair_unpack_kernel<true><<<grid_for(rows_v * v, 1), kThreads, 0, st>>>(rows_v, v, o, ab_pairs, Bp, Bm, out);
}

// A pair's q and, with the ladders' products, its rows of Bp and Bm, in half the
// shared memory of an SM: two blocks an SM.  That is o <= 69, without the products o <=
// 85.  Both sides of the line, v = 100: o = 69 0.57 ms, o = 70 (tiled) 0.99; without
// products o = 85 0.77, o = 86 (tiled) 0.87.
static int64_t r2_assemble_pair_bytes(int64_t o, bool pairs) { return (2 * o * (o | 1) + (pairs ? o * o : 0)) * 8; }

int64_t r2_assemble_pair_max(bool pairs) {
  int64_t o = 1;
  while (r2_assemble_pair_bytes(o + 1, pairs) <= kAssembleSmem) ++o;
  return o;
}

void launch_r2_assemble(int64_t o, int64_t v, const double* r2u, const double* tmp, const double* g,
                        const double* Bp, const double* Bm, bool accumulate, double* r2, cudaStream_t st) {
  static const bool attr =
      cudaFuncSetAttribute(r2_assemble_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAssembleSmem) ==
          cudaSuccess &&
      cudaFuncSetAttribute(r2_assemble_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAssembleSmem) ==
          cudaSuccess;
  const int64_t bytes = r2_assemble_pair_bytes(o, Bp != nullptr);
  if (attr && bytes <= kAssembleSmem) {
    const AssembleArgs A{static_cast<int>(o), static_cast<int>(v), r2u, tmp, g, Bp, Bm, r2};
    const int64_t want = (o * o / 4 + 31) / 32 * 32;  // about four elements a thread
    const unsigned threads = static_cast<unsigned>(std::min<int64_t>(512, std::max<int64_t>(64, want)));
    const unsigned grid = static_cast<unsigned>(std::min<int64_t>(v * (v + 1) / 2, 152LL * 32));
    if (accumulate) r2_assemble_pair_kernel<true><<<grid, threads, bytes, st>>>(A);
    else r2_assemble_pair_kernel<false><<<grid, threads, bytes, st>>>(A);
    return;
  }
  const int64_t nt = (o + 31) / 32;
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(v * v * nt * nt, 152LL * 16));
  r2_assemble_kernel<<<grid, dim3(32, 8), 0, st>>>(o, v, r2u, tmp, g, Bp, Bm, accumulate, r2);
}

void launch_diag_snapshot(int64_t o, int64_t v, int which, const double* X, double* d, cudaStream_t st) {
  diag_snapshot_kernel<<<grid_for(o * v * v, kThreads), kThreads, 0, st>>>(o, v, which, X, d);
}

void launch_gac_from_diagonals(int64_t o, int64_t v, const double* K, const double* P, const double* dK,
                               const double* dP, double* gac, cudaStream_t st) {
  gac_from_diagonals_kernel<<<grid_for(v * v, kThreads), kThreads, 0, st>>>(o, v, K, P, dK, dP, gac);
}

void launch_r1_from_tmp2(int64_t o, int64_t v, const double* tmp2, double* r1, cudaStream_t st) {
  r1_from_tmp2_kernel<<<grid_for(v * o, kThreads), kThreads, 0, st>>>(o, v, tmp2, r1);
}

void launch_denominators(int64_t o, int64_t v, const double* eps_o, const double* eps_v, double* dinv1,
                         double* dinv2, cudaStream_t st) {
  denominators_kernel<<<grid_for(v * v, 1), kThreads, 0, st>>>(o, v, eps_o, eps_v, dinv1, dinv2);
}

void launch_jacobi_inplace(int64_t o, int64_t v, const double* eps_o, const double* eps_v, const double* r1,
                           const double* r2, double* t1, double* t2, cudaStream_t st) {
  jacobi_inplace_kernel<<<grid_for(v * v, 1), kThreads, 0, st>>>(o, v, eps_o, eps_v, r1, r2, t1, t2);
}

void launch_pair_asym(int64_t o, int64_t v, const double* t2, unsigned long long* out, cudaStream_t st) {
  pair_asym_kernel<<<grid_for(v * v, 1), kThreads, 0, st>>>(o, v, t2, out);
}

void launch_maxabs_diff(int64_t n, const double* a, const double* b, unsigned long long* out, cudaStream_t st) {
  if (n <= 0) return;
  maxabs_diff_kernel<<<grid_for(n, kThreads, 1216), kThreads, 0, st>>>(n, a, b, out);
}

void launch_diis_step(const DiisArgs& d, cudaStream_t st) {
  diis_jacobi_dots_kernel<<<energy_blocks(d.v), kThreads, 0, st>>>(d);
}

void launch_diis_coefficients_test(const double* Bmat, int n, double damping, double* coef, int* nskip,
                                   cudaStream_t st) {
  diis_coefficients_test_kernel<<<1, 32, 0, st>>>(Bmat, n, damping, coef, nskip);
}

void launch_diis_extrapolate(int64_t o, int64_t v, const double* x1, const double* x2,
                             const double* coef, int ndiis, const int* slots, int nvec,
                             double* t1, double* t2, double* tau, cudaStream_t st, const DiisDyn* dyn) {
  (void)ndiis;
  ExtrapArgs x;
  x.o = o;
  x.v = v;
  x.x1 = x1;
  x.x2 = x2;
  x.coef = coef;
  x.nvec = nvec;
  for (int q = 0; q < kDiisMax; ++q) x.slots[q] = (slots && q < nvec) ? slots[q] : 0;
  x.t1 = t1;
  x.t2 = t2;
  x.tau = tau;
  x.dyn = dyn;
  if (o <= kExtrapRows) {
    extrapolate_t2_tau_kernel<true><<<grid_for(v * v, 1), kThreads, 0, st>>>(x);
    return;
  }
  extrapolate_t1_kernel<<<grid_for(v * o, kThreads), kThreads, 0, st>>>(x);
  extrapolate_t2_tau_kernel<false><<<grid_for(v * v, 1), kThreads, 0, st>>>(x);
}

}  // namespace gbcc

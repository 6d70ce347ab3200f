// Perturbative triples correction (T) of closed-shell CCSD on the GPU.
//
// The reference's "straight" (T) (src/mpqc/chemistry/qc/lcao/cc/ccsd_t.h:
// 1127-1167, denominators by CCSD_T_Reduce, :2274-2333) forms the connected
// triples of all occupied triplets at once (o^3 v^3 elements).  Here the
// triplets i <= j <= k run in batches (a triplet's abc sum is the same for
// every ordering of i, j, k, so it counts once per distinct ordering):
//   W[a][b][c] = t3(a,b,c,i,j,k) = sum over the six simultaneous
//   permutations of (a,i),(b,j),(c,k) of
//     X(a,b,c,i,j,k) = sum_d <id|ab> t2(d,c,j,k) - sum_l <jk|lc> t2(a,b,i,l),
// each a product over K = v + o (the d and l sums concatenated along K) of the
// panels (rows x K, columns d < v, then l)
//   A  [(x,p,q)] = ( <xd|pq> = Giabc[x][d][p][q] , -t2(p,q,x,l) )
//   At [(x,q,p)] = the same rows with p fastest
//   B  [(y,z,c)] = ( t2(d,c,y,z) , <yz|lc> = Gijka[y][z][l][c] )
//
// Tensor cores (MIXED: three BF16 slices, FP64_TC: six fixed-point ones).  The
// six terms pair up by the output index that runs along B: with A for one and
// At for the other, (i,j,k) and (j,i,k) share rows (a,b) and columns c, (i,k,j)
// and (k,i,j) rows (a,c) and columns b, (j,k,i) and (k,j,i) rows (b,c) and
// columns a.  Each pair is one product over 2 K (gemm_multi.cu), written once
// to its own array, in its own order; the energy kernel adds the three as it
// reads them.  (Six read-modify-write passes of W through scattered offsets, one
// per term and pair i, j, took 113 ms at o = 20, v = 76; this takes 17.5 ms.)  A
// batch is as many triplets as keep the three arrays in about 96 MB, most of
// L2.  The energy kernel takes 8 x 8 x 8 blocks of a <= b <= c: all six
// orderings of a set {a, b, c} are read once and give all six permuted W
// (t3(abc,kij) = W[b][c][a], ...) that each of its terms needs, the disconnected
// v3 from <ij|ab> and t1, and one denominator.
//
// FP64 runs the six terms as GEMMs over batches (i, j; k >= j), each keeping
// one operand fixed over the batch, stacking the other over k and scattering
// into W through its offset tables; its B2 [(y,z,b)] = B [(z,y,b)].
#include <algorithm>
#include <deque>
#include <vector>

#include "../../include/gbcc.h"
#include "engine.h"
#include "gather.cuh"
#include "kernels.h"
#include "triples.h"

namespace gbcc {

// test hook: triplets per batch (0: the default)
int64_t g_triples_chunk = 0;

namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ double block_sum_det(double v, double* sh) {
  // fixed-order tree reduction (deterministic)
  const int tid = threadIdx.x;
  sh[tid] = v;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (tid < s) sh[tid] += sh[tid + s];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

// One FP64 batch (i, j; k = k0 + kk): block (a, kk) sums over (b, c) and writes
// the weighted partial to partial[kk * v + a].
__global__ void __launch_bounds__(kThreads) triples_energy_kernel(
    const double* __restrict__ W, int64_t o, int64_t v, int i, int j, int k0, int nk, const double* __restrict__ Gijab,
    const double* __restrict__ t1, const double* __restrict__ eps_o, const double* __restrict__ eps_v,
    double* __restrict__ partial) {
  __shared__ double sh[kThreads];
  const int64_t a = blockIdx.x;
  const int kk = blockIdx.y;
  const int k = k0 + kk;
  if (kk >= nk) return;
  const double mult = (i < j && j < k) ? 6.0 : ((i == j && j == k) ? 1.0 : 3.0);
  const int64_t v2 = v * v;
  const double* __restrict__ Wk = W + static_cast<int64_t>(kk) * v2 * v;
  const double base = eps_o[i] + eps_o[j] + eps_o[k] - eps_v[a];
  const double t1ai = t1[a * o + i];
  const double* __restrict__ g_ij = Gijab + (static_cast<int64_t>(i) * o + j) * v2;  // <ij|..>
  const double* __restrict__ g_jk = Gijab + (static_cast<int64_t>(j) * o + k) * v2;
  const double* __restrict__ g_ik = Gijab + (static_cast<int64_t>(i) * o + k) * v2;
  double acc = 0.0;
  for (int64_t e = threadIdx.x; e < v2; e += blockDim.x) {
    const int64_t b = e / v, c = e - b * v;
    const double w = Wk[a * v2 + b * v + c];
    const double y = 4.0 * w + Wk[b * v2 + c * v + a] + Wk[c * v2 + a * v + b] -
                     2.0 * (Wk[c * v2 + b * v + a] + Wk[a * v2 + c * v + b] + Wk[b * v2 + a * v + c]);
    const double vv = g_ij[a * v + b] * t1[c * o + k] + g_jk[b * v + c] * t1ai + g_ik[a * v + c] * t1[b * o + j];
    acc += (w + vv) * y / (base - eps_v[b] - eps_v[c]);
  }
  const double s = block_sum_det(acc, sh);
  if (threadIdx.x == 0) partial[static_cast<int64_t>(kk) * v + a] = mult * s;
}

__global__ void __launch_bounds__(kThreads) sum_kernel(const double* __restrict__ x, int64_t n, double scale,
                                                      double* __restrict__ out) {
  __shared__ double sh[kThreads];
  double acc = 0.0;
  for (int64_t e = threadIdx.x; e < n; e += blockDim.x) acc += x[e];
  const double s = block_sum_det(acc, sh);
  if (threadIdx.x == 0) *out = scale * s;
}

// A packed operand of the FP64 path: rows x K.
struct Panel {
  int64_t rows = 0, K = 0;
  double* f64 = nullptr;
};

class Triples {
 public:
  Triples(const TriplesInputs& in, cudaStream_t st) : in_(in), st_(st) {}
  ~Triples() {
    for (void* p : owned_) dev_free(p);
  }

  double run();

 private:
  void* alloc(size_t bytes) {
    void* p = dev_alloc(bytes);
    owned_.push_back(p);
    return p;
  }
  const int64_t* table(const std::vector<int64_t>& h) {
    auto* d = static_cast<int64_t*>(alloc(std::max<size_t>(h.size(), 1) * sizeof(int64_t)));
    tables_.push_back(h);  // the copy's source lives until run() returns
    const std::vector<int64_t>& src = tables_.back();
    if (!src.empty())
      GBCC_CK(cudaMemcpyAsync(d, src.data(), src.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st_));
    return d;
  }
  Panel pack(const double* src1, int64_t n1, const std::vector<int64_t>& ra1, const std::vector<int64_t>& ca1,
             double coef1, const double* src2, int64_t n2, const std::vector<int64_t>& ra2,
             const std::vector<int64_t>& ca2, double coef2, int64_t split);
  void gemm(const Panel& A, int64_t a0, int64_t M, const Panel& B, int64_t b0, int64_t N, const int64_t* cm,
            const int64_t* cn, bool m_major, double beta);

  TriplesInputs in_;
  cudaStream_t st_;
  std::vector<void*> owned_;
  std::deque<std::vector<int64_t>> tables_;  // stable addresses
  double* W_ = nullptr;      // t3 of one batch, [k - j][a][b][c]
  double* mask_ = nullptr;   // {0.0, 1.0}
};

// A panel whose columns c < v come from src1 and the rest from src2 (the d
// and l sums side by side): two gather terms, each multiplied by a 0/1 mask
// over the columns (a 2-element table), so every column takes one source.
// The offsets of both terms are checked against their sources on the host.
Panel Triples::pack(const double* src1, int64_t n1, const std::vector<int64_t>& ra1, const std::vector<int64_t>& ca1,
                    double coef1, const double* src2, int64_t n2, const std::vector<int64_t>& ra2,
                    const std::vector<int64_t>& ca2, double coef2, int64_t split) {
  const int64_t rows = static_cast<int64_t>(ra1.size()), K = static_cast<int64_t>(ca1.size());
  auto inside = [](const std::vector<int64_t>& r, const std::vector<int64_t>& c, int64_t n) {
    const int64_t lo = *std::min_element(r.begin(), r.end()) + *std::min_element(c.begin(), c.end());
    const int64_t hi = *std::max_element(r.begin(), r.end()) + *std::max_element(c.begin(), c.end());
    return lo >= 0 && hi < n;
  };
  if (static_cast<int64_t>(ra2.size()) != rows || static_cast<int64_t>(ca2.size()) != K || !inside(ra1, ca1, n1) ||
      !inside(ra2, ca2, n2) || split < 0 || split > K)
    throw Error(GBCC_ERR_STATE, "(T): operand offsets outside the source");
  Panel p;
  p.rows = rows;
  p.K = K;
  std::vector<int64_t> zero(static_cast<size_t>(rows), 0), m1(static_cast<size_t>(K)), m2(static_cast<size_t>(K));
  for (int64_t c = 0; c < K; ++c) {
    m1[c] = c < split ? 1 : 0;  // index into mask_ = {0.0, 1.0}
    m2[c] = c < split ? 0 : 1;
  }
  const int64_t* rz = table(zero);
  GatherArgs g{};
  g.nterms = 2;
  g.products = 1;
  gather_set_coef(g.t[0], coef1);
  g.t[0].a = src1;
  g.t[0].ra = table(ra1);
  g.t[0].ca = table(ca1);
  g.t[0].b = mask_;
  g.t[0].rb = rz;
  g.t[0].cb = table(m1);
  gather_set_coef(g.t[1], coef2);
  g.t[1].a = src2;
  g.t[1].ra = table(ra2);
  g.t[1].ca = table(ca2);
  g.t[1].b = mask_;
  g.t[1].rb = rz;
  g.t[1].cb = table(m2);
  gather_finish(g);
  g.R = rows;
  g.C = K;
  p.f64 = static_cast<double*>(alloc(static_cast<size_t>(rows) * K * sizeof(double)));
  g.Rpad = rows;
  g.Cpad = K;
  g.ldo = K;
  g.out = p.f64;
  launch_gather(g, st_);
  return p;
}

// C[cm[m] + cn[n]] = beta C + sum_k A[a0 + m][k] B[b0 + n][k], m < M, n < N
void Triples::gemm(const Panel& A, int64_t a0, int64_t M, const Panel& B, int64_t b0, int64_t N, const int64_t* cm,
                   const int64_t* cn, bool m_major, double beta) {
  if (M <= 0 || N <= 0) return;
  // the operand windows lie inside their panels (checked on the host)
  if (a0 < 0 || a0 + M > A.rows || b0 < 0 || b0 + N > B.rows || A.K != B.K)
    throw Error(GBCC_ERR_STATE, "(T): GEMM window outside its operand panel");
  GemmF64Args f{};
  f.M = M;
  f.N = N;
  f.K = A.K;
  f.A = A.f64 + a0 * A.K;
  f.lda = A.K;
  f.B = B.f64 + b0 * B.K;
  f.ldb = B.K;
  f.C = W_;
  f.cm = cm;
  f.cn = cn;
  f.alpha = 1.0;
  f.beta = beta;
  f.m_major = m_major ? 1 : 0;
  launch_gemm_f64(f, st_);
}

double Triples::run() {
  const int64_t o = in_.o, v = in_.v, v2 = v * v, v3 = v2 * v, o2 = o * o, K = v + o;
  const int64_t nG = o * v3, nT = v2 * o2, nR = o2 * o * v;
  mask_ = static_cast<double*>(alloc(2 * sizeof(double)));
  {
    static const double m[2] = {0.0, 1.0};
    GBCC_CK(cudaMemcpyAsync(mask_, m, sizeof(m), cudaMemcpyHostToDevice, st_));
  }
  // ---- operand panels, columns (d < v | l)
  std::vector<int64_t> ra1, ra2, ca1(static_cast<size_t>(K)), ca2(static_cast<size_t>(K));
  auto cols = [&](int64_t sd, int64_t sl) {  // column offsets of the two sources (0 where masked)
    for (int64_t c = 0; c < K; ++c) {
      ca1[c] = c < v ? c * sd : 0;
      ca2[c] = c < v ? 0 : (c - v) * sl;
    }
  };
  // A[(x,p,q)] = (Giabc[x][d][p][q], -t2[p][q][x][l]); At: rows (x,q,p)
  ra1.assign(static_cast<size_t>(o * v2), 0);
  ra2.assign(static_cast<size_t>(o * v2), 0);
  for (int64_t x = 0; x < o; ++x)
    for (int64_t p = 0; p < v; ++p)
      for (int64_t q = 0; q < v; ++q) {
        ra1[(x * v + p) * v + q] = x * v3 + p * v + q;
        ra2[(x * v + p) * v + q] = p * v * o2 + q * o2 + x * o;
      }
  cols(v2, 1);
  const Panel A = pack(in_.Giabc, nG, ra1, ca1, 1.0, in_.t2, nT, ra2, ca2, -1.0, v);
  for (int64_t x = 0; x < o; ++x)
    for (int64_t q = 0; q < v; ++q)
      for (int64_t p = 0; p < v; ++p) {
        ra1[(x * v + q) * v + p] = x * v3 + p * v + q;
        ra2[(x * v + q) * v + p] = p * v * o2 + q * o2 + x * o;
      }
  const Panel At = pack(in_.Giabc, nG, ra1, ca1, 1.0, in_.t2, nT, ra2, ca2, -1.0, v);
  // B[(y,z,c)] = (t2[d][c][y][z], Gijka[y][z][l][c]); B2[(y,z,b)] = (t2[b][d][y][z], Gijka[z][y][l][b])
  ra1.assign(static_cast<size_t>(o2 * v), 0);
  ra2.assign(static_cast<size_t>(o2 * v), 0);
  for (int64_t y = 0; y < o; ++y)
    for (int64_t z = 0; z < o; ++z)
      for (int64_t c = 0; c < v; ++c) {
        ra1[(y * o + z) * v + c] = c * o2 + y * o + z;
        ra2[(y * o + z) * v + c] = (y * o + z) * o * v + c;
      }
  cols(v * o2, v);
  const Panel B = pack(in_.t2, nT, ra1, ca1, 1.0, in_.Gijka, nR, ra2, ca2, 1.0, v);
  for (int64_t y = 0; y < o; ++y)
    for (int64_t z = 0; z < o; ++z)
      for (int64_t b = 0; b < v; ++b) {
        ra1[(y * o + z) * v + b] = b * v * o2 + y * o + z;
        ra2[(y * o + z) * v + b] = (z * o + y) * o * v + b;
      }
  cols(o2, v);
  const Panel B2 = pack(in_.t2, nT, ra1, ca1, 1.0, in_.Gijka, nR, ra2, ca2, 1.0, v);

  // ---- output offset tables of the six permutation terms into W[kk][a][b][c]
  std::vector<int64_t> h;
  auto pq_table = [&](int64_t sp, int64_t sq) {  // rows (p, q): p sp + q sq
    h.assign(static_cast<size_t>(v2), 0);
    for (int64_t p = 0; p < v; ++p)
      for (int64_t q = 0; q < v; ++q) h[p * v + q] = p * sp + q * sq;
    return table(h);
  };
  auto kr_table = [&](int64_t sr) {  // rows (kk, r): kk v^3 + r sr
    h.assign(static_cast<size_t>(o * v), 0);
    for (int64_t kk = 0; kk < o; ++kk)
      for (int64_t r = 0; r < v; ++r) h[kk * v + r] = kk * v3 + r * sr;
    return table(h);
  };
  auto kqp_table = [&](int64_t sq, int64_t sp) {  // rows (kk, q, p): kk v^3 + q sq + p sp
    h.assign(static_cast<size_t>(o * v2), 0);
    for (int64_t kk = 0; kk < o; ++kk)
      for (int64_t q = 0; q < v; ++q)
        for (int64_t p = 0; p < v; ++p) h[(kk * v + q) * v + p] = kk * v3 + q * sq + p * sp;
    return table(h);
  };
  auto r_table = [&](int64_t sr) {
    h.assign(static_cast<size_t>(v), 0);
    for (int64_t r = 0; r < v; ++r) h[r] = r * sr;
    return table(h);
  };
  // term 1 (a,b,c,i,j,k): rows (a,b) x (kk,c), lanes along N (c)
  // term 2 (a,c,b,i,k,j): rows (a,c) x (kk,b), lanes along M (c)
  // term 3 (b,a,c,j,i,k): rows (b,a) x (kk,c), lanes along N
  // term 4 (b,c,a,j,k,i): rows (b,c) x (kk,a), lanes along M
  // term 5 (c,a,b,k,i,j): rows (kk,a,c) of At x b, lanes along M
  // term 6 (c,b,a,k,j,i): rows (kk,b,c) of At x a, lanes along M
  const int64_t* cm1 = pq_table(v2, v);
  const int64_t* cm2 = pq_table(v2, 1);
  const int64_t* cm3 = pq_table(v, v2);
  const int64_t* cm4 = pq_table(v, 1);
  const int64_t* cn13 = kr_table(1);
  const int64_t* cn2 = kr_table(v);
  const int64_t* cn4 = kr_table(v2);
  const int64_t* cm5 = kqp_table(v2, 1);
  const int64_t* cm6 = kqp_table(v, 1);
  const int64_t* cn5 = r_table(v);
  const int64_t* cn6 = r_table(v2);

  // triplets per batch: all k >= j, unless their slice of t3 would pass
  // 8 GB (then chunks of k).  Chunks small enough to keep the slice in L2
  // measured slower (the batches' GEMMs shrink and multiply), so chunking only
  // bounds memory.
  int64_t kc = std::max<int64_t>(1, std::min<int64_t>(o, (static_cast<int64_t>(8) << 30) / (v3 * 8)));
  if (g_triples_chunk > 0) kc = std::min<int64_t>(o, g_triples_chunk);
  {
    // largest offset each term writes, for the largest batch (kk < kc)
    const int64_t last = v - 1, kmax = kc - 1;
    const int64_t worst[] = {last * (v2 + v) + kmax * v3 + last,       // 1, 3
                             last * (v2 + 1) + kmax * v3 + last * v,   // 2
                             last * (v + 1) + kmax * v3 + last * v2,   // 4
                             kmax * v3 + last * (v2 + 1) + last * v,   // 5
                             kmax * v3 + last * (v + 1) + last * v2};  // 6
    for (int64_t w : worst)
      if (w >= kc * v3) throw Error(GBCC_ERR_STATE, "(T): output offsets outside W");
  }
  W_ = static_cast<double*>(alloc(static_cast<size_t>(kc) * v3 * sizeof(double)));
  const int64_t npair = o * (o + 1) / 2;
  double* partial = static_cast<double*>(alloc(static_cast<size_t>(npair) * o * v * sizeof(double)));
  GBCC_CK(cudaMemsetAsync(partial, 0, static_cast<size_t>(npair) * o * v * sizeof(double), st_));
  double* d_e = static_cast<double*>(alloc(sizeof(double)));

  int64_t slot = 0;
  for (int i = 0; i < o; ++i) {
    for (int j = i; j < o; ++j, ++slot) {
      const int64_t pij = (static_cast<int64_t>(i) * o + j) * v;  // rows (i, j, r)
      for (int k0 = j; k0 < o; k0 += static_cast<int>(kc)) {
        const int nk = static_cast<int>(std::min<int64_t>(kc, o - k0));
        const int64_t rj = (static_cast<int64_t>(j) * o + k0) * v;  // rows (j, k = k0.., r)
        const int64_t ri = (static_cast<int64_t>(i) * o + k0) * v;  // rows (i, k = k0.., r)
        const int64_t nkv = static_cast<int64_t>(nk) * v;
        gemm(A, i * v2, v2, B, rj, nkv, cm1, cn13, false, 0.0);
        gemm(A, i * v2, v2, B2, rj, nkv, cm2, cn2, true, 1.0);
        gemm(A, j * v2, v2, B, ri, nkv, cm3, cn13, false, 1.0);
        gemm(A, j * v2, v2, B2, ri, nkv, cm4, cn4, true, 1.0);
        gemm(At, static_cast<int64_t>(k0) * v2, nk * v2, B, pij, v, cm5, cn5, true, 1.0);
        gemm(At, static_cast<int64_t>(k0) * v2, nk * v2, B2, pij, v, cm6, cn6, true, 1.0);
        const dim3 grid(static_cast<unsigned>(v), static_cast<unsigned>(nk));
        double* part = partial + slot * o * v + static_cast<int64_t>(k0 - j) * v;
        triples_energy_kernel<<<grid, kThreads, 0, st_>>>(W_, o, v, i, j, k0, nk, in_.Gijab, in_.t1, in_.eps_o,
                                                          in_.eps_v, part);
      }
    }
  }
  sum_kernel<<<1, kThreads, 0, st_>>>(partial, npair * o * v, 1.0 / 3.0, d_e);
  double e = 0.0;
  GBCC_CK(cudaMemcpyAsync(&e, d_e, sizeof(double), cudaMemcpyDeviceToHost, st_));
  GBCC_CK(cudaStreamSynchronize(st_));
  GBCC_CK(cudaGetLastError());
  return e;
}

// ---------------------------------------------------------------------------
// tensor cores

struct PackArgs {
  int kind;                 // 0: A rows (x,p,q), 1: At rows (x,q,p), 2: B rows (y,z,c)
  int64_t o, v, rows, K, kblocks;
  const double* Giabc;
  const double* Gijka;
  const double* t2;
  __nv_bfloat16* out;       // [slices][kblocks][rows][64]
};

// A block packs 32 rows: a thread takes 8 K elements of a row at a time, warp w
// those at 8 w of each k-block, and stores 16 bytes a slice (the 8 warps fill
// whole 128-byte lines).  Six slices need the row's largest exponent first.
template <int SL>
__global__ void __launch_bounds__(kThreads) triples_pack_kernel(PackArgs g) {
  __shared__ unsigned ex[8][32];
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const int64_t r = static_cast<int64_t>(blockIdx.x) * 32 + lane, v = g.v, o = g.o;
  const double *s1 = nullptr, *s2 = nullptr;
  int64_t st1 = 0, st2 = 0;
  double coef = 1.0;
  const bool in = r < g.rows;
  if (in && g.kind < 2) {
    const int64_t x = r / (v * v), rem = r - x * v * v, hi = rem / v, lo = rem - hi * v;
    const int64_t pq = g.kind == 0 ? rem : lo * v + hi;
    s1 = g.Giabc + x * v * v * v + pq;
    st1 = v * v;
    s2 = g.t2 + pq * o * o + x * o;
    st2 = 1;
    coef = -1.0;
  } else if (in) {
    const int64_t yz = r / v, c = r - yz * v;
    s1 = g.t2 + c * o * o + yz;
    st1 = v * o * o;
    s2 = g.Gijka + yz * o * v + c;
    st2 = v;
  }
  auto load8 = [&](int64_t k0, double x[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t k = k0 + j;
      x[j] = !in || k >= g.K ? 0.0 : (k < v ? s1[k * st1] : flip_sign(s2[(k - v) * st2], coef < 0.0));
    }
  };
  unsigned eb = 0;
  if constexpr (SL != 3) {
    for (int64_t kb = 0; kb < g.kblocks; ++kb) {
      double x[8];
      load8(kb * 64 + w * 8, x);
#pragma unroll
      for (int j = 0; j < 8; ++j) eb = max(eb, exp_field(x[j]));
    }
    ex[w][lane] = eb;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) eb = max(eb, ex[q][lane]);
  }
  if (!in) return;
  const int64_t slice = g.kblocks * g.rows * 64;
  for (int64_t kb = 0; kb < g.kblocks; ++kb) {
    double x[8];
    load8(kb * 64 + w * 8, x);
    unsigned short b[8][SL == 3 ? 3 : kFixedSlices];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if constexpr (SL == 3) split_bits(x[j], b[j], 3);
      else fixed_split(x[j], eb, kFixedSlices, b[j]);
    }
    __nv_bfloat16* out = g.out + (kb * g.rows + r) * 64 + w * 8;
#pragma unroll
    for (int s = 0; s < SL; ++s) {
      uint4 u;
      u.x = b[0][s] | (static_cast<unsigned>(b[1][s]) << 16);
      u.y = b[2][s] | (static_cast<unsigned>(b[3][s]) << 16);
      u.z = b[4][s] | (static_cast<unsigned>(b[5][s]) << 16);
      u.w = b[6][s] | (static_cast<unsigned>(b[7][s]) << 16);
      *reinterpret_cast<uint4*>(out + s * slice) = u;
    }
  }
}

// orderings of three things (the even ones first), and for ordering m = (x,y,z)
// the ordering (x,z,y) and the ordering (y,z,x)
__device__ constexpr int kPerm[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}, {0, 2, 1}, {1, 0, 2}};
__device__ constexpr int kSwap[6] = {4, 5, 3, 2, 0, 1};
__device__ constexpr int kCycle[6] = {1, 2, 0, 5, 3, 4};
// ordered pairs of different things
__device__ constexpr int kPair[6][2] = {{0, 1}, {0, 2}, {1, 0}, {1, 2}, {2, 0}, {2, 1}};
__device__ constexpr int pair_id(int s, int f) { return 2 * s + f - (f > s ? 1 : 0); }

constexpr int kB = 8;              // virtual block
constexpr int kCube = kB * kB * kB;
constexpr int kEnergyThreads = kCube;
constexpr int kEnergyGrid = 152;   // one block an SM

template <typename R>
struct EnergyStage {
  double W[3][6][kCube];           // float2 (three slices) or double words
  R G[3][6][kB * kB];              // <ij|, <jk|, <ik| over ordered block pairs
  R t1[3][3][kB];                  // t1 of i, j, k over the blocks
  double ev[3][kB];
  double eo;                       // eps_i + eps_j + eps_k
};

struct EnergyArgs {
  int o, v;
  int n;                      // triplets of this batch
  const int4* triples;        // theirs
  const unsigned* blocks;     // block triples A <= B <= C, 10 bits each
  int nblocks;
  const double* W;            // [triplet][3][v][v][v]
  const void* Gijab;          // of type R, as t1
  const void* t1;
  const double* eps_v;
  const double* eo;           // per triplet of this batch
  double* partial;            // [gridDim.x]
};

// x to y as the energy's type
template <typename R>
__global__ void __launch_bounds__(kThreads) convert_kernel(const double* __restrict__ x, int64_t n, R* __restrict__ y) {
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * kThreads)
    y[e] = static_cast<R>(x[e]);
}

__global__ void __launch_bounds__(kThreads) triplet_energies_kernel(const int4* __restrict__ tr, int64_t n,
                                                                    const double* __restrict__ eps_o,
                                                                    double* __restrict__ eo) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (t < n) eo[t] = eps_o[tr[t].x] + eps_o[tr[t].y] + eps_o[tr[t].z];
}

// hi + lo += x (TwoSum), for sums of many FP32 terms
__device__ __forceinline__ void add_ff(float& hi, float& lo, float x) {
  const float s = __fadd_rn(hi, x), b = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
  hi = s;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src, bool in) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst)), n = in ? BYTES : 0u;  // 0 source bytes: zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
}

// Where element (x, y, z) of a cube lies: a linear bijection of the nine index bits
// whose low four bits (the 16 banks of 8 bytes) differ over 8 values of any one
// index times 2 neighbouring values of any other, i.e. over the half warp of a
// copy (z, y) and of a read along any two of the three indices.
__device__ __forceinline__ int cube_at(int x, int y, int z) {
  const int x0 = x & 1, x1 = (x >> 1) & 1, x2 = x >> 2, y0 = y & 1, y1 = (y >> 1) & 1, y2 = y >> 2, z0 = z & 1,
            z1 = (z >> 1) & 1, z2 = z >> 2;
  return (z0 ^ y2 ^ x2) | ((y0 ^ z2 ^ x2) << 1) | ((x0 ^ z2 ^ y2) << 2) | ((z1 ^ y1 ^ x1) << 3) | (z2 << 4) |
         (y1 << 5) | (y2 << 6) | (x1 << 7) | (x2 << 8);
}
// and (x, y) of an 8 x 8 tile: a warp's 8 values of one index times 4 of the other
// lie in different banks
__device__ __forceinline__ int tile_at(int x, int y) { return x * kB + (x ^ y); }

// A persistent block takes the batch's pairs (triplet, block triple) w = blockIdx.x,
// blockIdx.x + gridDim.x, ...  R: the arithmetic of the terms (double for
// FP64_TC; float for MIXED, whose products carry ~1e-6: FP32 rounds W, a term and
// its weight, and nothing that is summed -- the arrays of W, the six orderings of a
// set and the running sum are float-float sums, the denominators FP64.  With plain
// FP32 sums of the orderings and denominators (T) at o = 20, v = 76 took 16.97 ms,
// so 17.33, with the running sum in FP64 17.66).
//
// A pair is 18 cubes of W (74 KB) and a few hundred operations per element: one
// thread an element (a, b, c), and two stages, so that the copies of the next
// pair, all asynchronous, run under the terms of this one.  Every cube of
// ordering m is read at F[m], the same six offsets for all three arrays and all
// pairs.  Nine triplets at v = 76: 58 -> 44 us against blocks of one pair each with
// one stage ((T) at o = 20, v = 76: 20.4 -> 17.1 ms, before the sums above).
template <typename R>
__global__ void __launch_bounds__(kEnergyThreads, 1) triples_blocks_kernel(EnergyArgs g) {
  extern __shared__ double smem_d[];
  EnergyStage<R>* stages = reinterpret_cast<EnergyStage<R>*>(smem_d);
  constexpr bool kPairs = sizeof(R) == 4;
  const int tid = threadIdx.x;
  const int v = g.v, o = g.o, v2 = v * v;
  const int64_t v3 = static_cast<int64_t>(v2) * v;
  const R* Gijab = static_cast<const R*>(g.Gijab);
  const R* t1 = static_cast<const R*>(g.t1);
  const int l2 = tid & 7, l1 = (tid >> 3) & 7, l0 = tid >> 6;  // copies: element (l0, l1, l2)
  const int la = l1, lb = l2, lc = l0;                         // terms
  const int put = cube_at(l0, l1, l2), put2 = tile_at(l1, l2);
  int F[6], Q[6];
  {
    auto l = [&](int q) { return q == 0 ? la : (q == 1 ? lb : lc); };
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      F[m] = cube_at(l(kPerm[m][0]), l(kPerm[m][1]), l(kPerm[m][2]));
      Q[m] = tile_at(l(kPair[m][0]), l(kPair[m][1]));
    }
  }

  struct Item {
    int t;
    unsigned code;
    int4 ijk;
  };
  const int64_t items = static_cast<int64_t>(g.n) * g.nblocks;
  auto item = [&](int64_t w) {
    Item x;
    x.t = static_cast<int>(static_cast<uint32_t>(w) / static_cast<uint32_t>(g.nblocks));
    x.code = g.blocks[static_cast<uint32_t>(w) - static_cast<uint32_t>(x.t) * static_cast<uint32_t>(g.nblocks)];
    x.ijk = g.triples[x.t];
    return x;
  };
  auto load = [&](const Item& x, EnergyStage<R>& S) {
    const int A = static_cast<int>(x.code & 1023u) * kB, B = static_cast<int>((x.code >> 10) & 1023u) * kB,
              C = static_cast<int>(x.code >> 20) * kB;
    auto start = [&](int q) { return q == 0 ? A : (q == 1 ? B : C); };
    const double* W = g.W + static_cast<int64_t>(x.t) * 3 * v3;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int gs = start(kPerm[m][0]) + l0, gf = start(kPerm[m][1]) + l1, gr = start(kPerm[m][2]) + l2;
      const bool in = gs < v && gf < v && gr < v;  // zeros past v
      const double* src = W + (in ? static_cast<int64_t>(gs * v + gf) * v + gr : 0);
#pragma unroll
      for (int p = 0; p < 3; ++p) copy_async<8>(&S.W[p][m][put], src + p * v3, in);
    }
    // <ij|, <jk|, <ik| over the six ordered block pairs: 64 elements by 64 threads each
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const int q = l0 + kB * u;
      if (q < 18) {
        const int p = q / 6, m = q - 6 * p;
        const int bs = m >> 1, bf = (m & 1) ? (bs == 2 ? 1 : 2) : (bs == 0 ? 1 : 0);
        const int gs = start(bs) + l1, gf = start(bf) + l2;
        const int x1 = p == 1 ? x.ijk.y : x.ijk.x, x2 = p == 0 ? x.ijk.y : x.ijk.z;
        const bool in = gs < v && gf < v;
        copy_async<sizeof(R)>(&S.G[p][m][put2],
                              Gijab + (static_cast<int64_t>(x1) * o + x2) * v2 + (in ? gs * v + gf : 0), in);
      }
    }
    if (tid < 72) {
      const int e = tid & 7, blk = (tid >> 3) % 3, p = (tid >> 3) / 3;
      const int gx = start(blk) + e, occ = p == 0 ? x.ijk.x : (p == 1 ? x.ijk.y : x.ijk.z);
      copy_async<sizeof(R)>(&S.t1[p][blk][e], t1 + (gx < v ? gx * o + occ : 0), gx < v);
    } else if (tid < 96) {
      const int blk = (tid - 72) >> 3, gx = start(blk) + (tid & 7);
      copy_async<8>(&S.ev[blk][tid & 7], g.eps_v + (gx < v ? gx : 0), gx < v);
    } else if (tid == 96) {
      copy_async<8>(&S.eo, g.eo + x.t, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  double acc = 0.0;
  float ahi = 0.f, alo = 0.f;
  Item cur{}, next{};
  int64_t w = blockIdx.x;
  if (w < items) {
    cur = item(w);
    load(cur, stages[0]);
    if (w + gridDim.x < items) next = item(w + gridDim.x);
  }
  for (int st = 0; w < items; w += gridDim.x, st ^= 1) {
    const bool more = w + gridDim.x < items;
    const Item soon = next;
    if (more) {
      load(next, stages[st ^ 1]);
      if (w + 2 * static_cast<int64_t>(gridDim.x) < items) next = item(w + 2 * static_cast<int64_t>(gridDim.x));
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const EnergyStage<R>& S = stages[st];
    const int a = static_cast<int>(cur.code & 1023u) * kB + la, b = static_cast<int>((cur.code >> 10) & 1023u) * kB + lb,
              c = static_cast<int>(cur.code >> 20) * kB + lc;
    if (a <= b && b <= c && c < v) {
      R ww[6], u[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        const double w0 = S.W[0][m][F[m]], w1 = S.W[1][kSwap[m]][F[kSwap[m]]], w2 = S.W[2][kCycle[m]][F[kCycle[m]]];
        if constexpr (kPairs) {
          // words of (hi, lo) floats
          const float2 f0 = *reinterpret_cast<const float2*>(&w0), f1 = *reinterpret_cast<const float2*>(&w1),
                       f2 = *reinterpret_cast<const float2*>(&w2);
          float hi = f0.x, lo = f0.y;
          add_ff(hi, lo, f1.x);
          add_ff(hi, lo, f2.x);
          ww[m] = hi + (lo + (f1.y + f2.y));
        } else {
          ww[m] = w0 + w1 + w2;
        }
        auto l = [&](int q) { return q == 0 ? la : (q == 1 ? lb : lc); };
        const int px = kPerm[m][0], py = kPerm[m][1], pz = kPerm[m][2];
        const int xy = pair_id(px, py), yz = pair_id(py, pz), xz = pair_id(px, pz);
        u[m] = S.G[0][xy][Q[xy]] * S.t1[2][pz][l(pz)] + S.G[1][yz][Q[yz]] * S.t1[0][px][l(px)] +
               S.G[2][xz][Q[xz]] * S.t1[1][py][l(py)];
      }
      const R even = ww[0] + ww[1] + ww[2], odd = ww[3] + ww[4] + ww[5];
      // 4 t3(abc) + the two cyclic orderings - 2 the three others
      const R ee = even - R(2) * odd, oo = odd - R(2) * even;
      R sum[6];
#pragma unroll
      for (int m = 0; m < 6; ++m) sum[m] = (ww[m] + u[m]) * (R(3) * ww[m] + (m < 3 ? ee : oo));
      // a set with equal members has its orderings counted that many times
      const int i = cur.ijk.x, j = cur.ijk.y, k = cur.ijk.z;
      const R mult = (i < j && j < k) ? R(6) : ((i == j && j == k) ? R(1) : R(3));
      const R share = a == b ? (b == c ? R(1) / R(6) : R(0.5)) : (b == c ? R(0.5) : R(1));
      const double d = S.eo - S.ev[0][la] - S.ev[1][lb] - S.ev[2][lc];
      const R f = (mult * share) / static_cast<R>(d);
      if constexpr (kPairs) {
        float hi[3] = {sum[0], sum[2], sum[4]}, lo[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int q = 0; q < 3; ++q) add_ff(hi[q], lo[q], sum[2 * q + 1]);
        add_ff(hi[0], lo[0], hi[1]);
        add_ff(hi[0], lo[0], hi[2]);
        const float p = hi[0] * f;
        add_ff(ahi, alo, p);
        alo += fmaf(hi[0], f, -p) + (lo[0] + (lo[1] + lo[2])) * f;
      } else {
        acc += (((sum[0] + sum[1]) + sum[2]) + ((sum[3] + sum[4]) + sum[5])) * f;
      }
    }
    cur = soon;
    __syncthreads();  // the stage is free
  }
  const double s = block_sum_det(acc + static_cast<double>(ahi) + static_cast<double>(alo), smem_d);
  if (tid == 0) g.partial[blockIdx.x] = s;
}

// out[blockIdx.x] = sum of its share of x (strided; fixed order)
__global__ void __launch_bounds__(kThreads) sum_blocks_kernel(const double* __restrict__ x, int64_t n,
                                                             double* __restrict__ out) {
  __shared__ double sh[kThreads];
  double acc = 0.0;
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x)
    acc += x[e];
  const double s = block_sum_det(acc, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = s;
}

template <typename R>
void launch_blocks(const EnergyArgs& g, cudaStream_t st) {
  constexpr int bytes = 2 * sizeof(EnergyStage<R>);
  static const bool attr = cudaFuncSetAttribute(triples_blocks_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                bytes) == cudaSuccess;
  if (!attr) throw Error(GBCC_ERR_CUDA, "(T): energy kernel shared memory");
  triples_blocks_kernel<R><<<kEnergyGrid, kEnergyThreads, bytes, st>>>(g);
}

// the energy's inputs: Gijab and t1 as its type (double: where they lie), eps_v and
// the triplets' sums of eps_o
template <typename R>
void prepare_energy(const TriplesInputs& in, const int4* tr, int64_t ntr, char* ws, EnergyArgs& e, cudaStream_t st) {
  const int64_t ng = in.o * in.o * in.v * in.v, nt = in.o * in.v;
  double* eo = reinterpret_cast<double*>(ws);
  triplet_energies_kernel<<<static_cast<unsigned>((ntr + kThreads - 1) / kThreads), kThreads, 0, st>>>(tr, ntr, in.eps_o, eo);
  e.eo = eo;
  e.eps_v = in.eps_v;
  if constexpr (sizeof(R) == 8) {
    e.Gijab = in.Gijab;
    e.t1 = in.t1;
  } else {
    R *G = reinterpret_cast<R*>(eo + ntr), *t1 = G + ng;
    auto convert = [&](const double* x, int64_t n, R* y) {
      convert_kernel<R><<<static_cast<unsigned>(std::min<int64_t>((n + kThreads - 1) / kThreads, 1216)), kThreads, 0, st>>>(x, n, y);
    };
    convert(in.Gijab, ng, G);
    convert(in.t1, nt, t1);
    e.Gijab = G;
    e.t1 = t1;
  }
}

double triples_tc(const TriplesInputs& in, int precision, cudaStream_t st, int* err) {
  const int64_t o = in.o, v = in.v, v3 = v * v * v, K = v + o, kblocks = (K + 63) / 64;
  const int slices = precision == GBCC_PREC_MIXED ? 3 : kFixedSlices;
  const int64_t rowsA = o * v * v, rowsB = o * o * v;
  const int64_t nvb = (v + kB - 1) / kB;
  if (nvb > 1023) throw Error(GBCC_ERR_STATE, "(T): too many virtual orbitals");
  std::vector<int4> tr;
  for (int i = 0; i < o; ++i)
    for (int j = i; j < o; ++j)
      for (int k = j; k < o; ++k) tr.push_back(make_int4(i, j, k, 0));
  std::vector<unsigned> bl;
  for (unsigned a = 0; a < nvb; ++a)
    for (unsigned b = a; b < nvb; ++b)
      for (unsigned c = b; c < nvb; ++c) bl.push_back(a | (b << 10) | (c << 20));
  const int64_t ntr = static_cast<int64_t>(tr.size()), nbl = static_cast<int64_t>(bl.size());
  int64_t batch = std::max<int64_t>(1, std::min<int64_t>(ntr, (int64_t{96} << 20) / (3 * v3 * 8)));
  batch = std::min<int64_t>(batch, (int64_t{1} << 31) / nbl);  // 32-bit counts of (triplet, block triple)
  if (g_triples_chunk > 0) batch = std::min(batch, g_triples_chunk);
  const int64_t nbatch = (ntr + batch - 1) / batch;
  constexpr int kSums = 152;
  size_t total = 0;
  auto part = [&](size_t bytes) {
    const size_t at = total;
    total += (bytes + 1023) / 1024 * 1024;
    return at;
  };
  const size_t elems_a = static_cast<size_t>(slices) * kblocks * rowsA * 64, elems_b = static_cast<size_t>(slices) * kblocks * rowsB * 64;
  const size_t oA = part(elems_a * 2), oA2 = part(elems_a * 2), oB = part(elems_b * 2), oW = part(static_cast<size_t>(batch) * 3 * v3 * 8),
               oT = part(ntr * sizeof(int4)), oBl = part(nbl * sizeof(unsigned)), oP = part(static_cast<size_t>(nbatch) * kEnergyGrid * 8),
               oE = part(ntr * sizeof(double) + (slices == 3 ? (o * o * v * v + o * v) * sizeof(float) : 0)),
               oS = part((kSums + 1) * 8);
  struct Owned {
    char* p;
    ~Owned() { dev_free(p); }
  } ws{static_cast<char*>(dev_alloc(total))};
  auto* A = reinterpret_cast<__nv_bfloat16*>(ws.p + oA);
  auto* A2 = reinterpret_cast<__nv_bfloat16*>(ws.p + oA2);
  auto* B = reinterpret_cast<__nv_bfloat16*>(ws.p + oB);
  auto* W = reinterpret_cast<double*>(ws.p + oW);
  auto* d_tr = reinterpret_cast<int4*>(ws.p + oT);
  auto* d_bl = reinterpret_cast<unsigned*>(ws.p + oBl);
  auto* partial = reinterpret_cast<double*>(ws.p + oP);
  auto* sums = reinterpret_cast<double*>(ws.p + oS);
  GBCC_CK(cudaMemcpyAsync(d_tr, tr.data(), ntr * sizeof(int4), cudaMemcpyHostToDevice, st));
  GBCC_CK(cudaMemcpyAsync(d_bl, bl.data(), nbl * sizeof(unsigned), cudaMemcpyHostToDevice, st));
  for (int kind = 0; kind < 3; ++kind) {
    PackArgs p{kind, o, v, kind == 2 ? rowsB : rowsA, K, kblocks, in.Giabc, in.Gijka, in.t2,
               kind == 0 ? A : (kind == 1 ? A2 : B)};
    const unsigned grid = static_cast<unsigned>((p.rows + 31) / 32);
    if (slices == 3) triples_pack_kernel<3><<<grid, kThreads, 0, st>>>(p);
    else triples_pack_kernel<kFixedSlices><<<grid, kThreads, 0, st>>>(p);
  }
  GemmMultiArgs g{};
  g.K = K;
  g.kblocks = kblocks;
  g.A = A;
  g.A2 = A2;
  g.B = B;
  g.a_rows = rowsA;
  g.o = static_cast<int>(o);
  g.v = static_cast<int>(v);
  g.W = W;
  g.err = err;
  EnergyArgs e{};
  e.o = static_cast<int>(o);
  e.v = static_cast<int>(v);
  e.blocks = d_bl;
  e.nblocks = static_cast<int>(nbl);
  e.W = W;
  if (slices == 3) prepare_energy<float>(in, d_tr, ntr, ws.p + oE, e, st);
  else prepare_energy<double>(in, d_tr, ntr, ws.p + oE, e, st);
  const double* eo = e.eo;
  for (int64_t t0 = 0, k = 0; t0 < ntr; t0 += batch, ++k) {
    const int n = static_cast<int>(std::min(batch, ntr - t0));
    g.triples = d_tr + t0;
    if (!launch_gemm_triples(g, slices, n, st)) throw Error(GBCC_ERR_CUDA, "(T): tcgen05 launch rejected");
    e.n = n;
    e.triples = d_tr + t0;
    e.eo = eo + t0;
    e.partial = partial + k * kEnergyGrid;
    if (slices == 3) launch_blocks<float>(e, st);
    else launch_blocks<double>(e, st);
  }
  sum_blocks_kernel<<<kSums, kThreads, 0, st>>>(partial, nbatch * kEnergyGrid, sums);
  sum_kernel<<<1, kThreads, 0, st>>>(sums, kSums, 1.0 / 3.0, sums + kSums);
  double out = 0.0;
  GBCC_CK(cudaMemcpyAsync(&out, sums + kSums, sizeof(double), cudaMemcpyDeviceToHost, st));
  GBCC_CK(cudaStreamSynchronize(st));
  GBCC_CK(cudaGetLastError());
  return out;
}

}  // namespace

double triples_energy(const TriplesInputs& in, int precision, cudaStream_t st, int* err) {
  if (precision != GBCC_PREC_FP64) return triples_tc(in, precision, st, err);
  Triples t(in, st);
  return t.run();
}

}  // namespace gbcc

extern "C" int gbcc_testing_triples_chunk(int64_t k) {
  if (k < 0) return GBCC_ERR_INVALID_ARG;
  gbcc::g_triples_chunk = k;
  return GBCC_OK;
}

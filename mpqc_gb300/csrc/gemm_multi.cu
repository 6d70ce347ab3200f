// Tensor-core products that load every slice of a K block once (tcgen05 + TMEM
// + TMA, sm_103a): the FP64-grade contractions and the (T) triples terms.
//
// gemm_tc_kernel stages one (A slice, B slice) pair at a time, so a product of
// S slices loads each operand tile (S + 1) / 2 times and, with 128 x 128 tiles,
// asks L2 for 128 bytes a clock per SM while it issues 64 clocks of MMAs per K
// step: with six slices the tensor pipe was 25 % busy, and every weight class
// was a launch of its own with a read-modify-write of C.  Here a pipeline stage
// holds all slices of A and of B for 32 elements of K and the MMA thread runs
// all pairs p + q < S from it (six for three slices, 21 for six): 36 bytes a
// clock at six slices, and C is written once.  19456 x 64 x 4096 at six slices:
// 340 -> 870 TFLOP/s of slice products, now bound by shared memory (6 KB read per
// 128 x 64 x 16 MMA); 1743^3: 0.86 -> 0.32 ms.
//
// Six slices (fixed point, kernels.h): every weight class w = p + q has its own
// TMEM accumulator, whose sum stays exact while it covers at most 1024
// products of its unit; class 5 has 6 pairs, so a chunk is five stages of 32
// (960 products).  The classes of successive chunks rotate through eight
// accumulators of BN <= 64 columns, two more than a chunk needs: the MMAs of
// the next chunk start while the epilogue still drains this one.  The epilogue
// adds the finished sums to two float-float pairs per output, classes 0-2 and
// 3-5, and the pairs meet in FP64.  A pair is exact while its low word holds every
// rounding error of its high one.  In units of class 2 the sum of classes 0-2 over
// K elements is at most 2^14 (2^16 + 2 2^8 + 3) K, below 2^45 for K <= 32000, so an
// addition to the high word errs by at most 2^20 units.  The pair is renormalised
// every four chunks, and a low word of 2^20 with twelve more errors is within the
// 2^24 units that FP32 holds: exact.  Of classes 3-5, sixteen bits further down,
// an addition then loses two units of class 5 at most, 2^-53 of a largest product,
// 10^-4 of what the classes left out (6 on) may hold.  K beyond that runs in
// windows of 32000 elements, a launch each, added to C (or to the partial tiles)
// in FP64.  (Never renormalised and in one window, sums of one sign were off by
// 1.5e-12 at K = 65536 and 3.6e-12 at 262144.  Renormalising every chunk instead
// cost 5 %, windows of 8000 12 % of 4096 x 528 x 51360.)
//
// Three slices (the BF16 split; (T) only): one accumulator per stage (12 MMAs,
// no longer than the 16 of gemm_tc_kernel), summed per segment in FP32
// registers as there; the two segments of a tile meet in a float-float pair.
//
// (T): a tile is 128 rows (8 x 16 virtual pairs) x BN columns of one of the
// three sums of two permutation terms that share their output order (triples.cu);
// its two segments name different operand panels and rows.
//
// Persistent: warp 0 TMA, 1 MMA (and TMEM allocation), 8 or 16 (three
// slices, wide tiles) epilogue warps from 2 on (warp w reads TMEM lanes 32 (w % 4)..), with the bounded waits and teardown of
// gemm_tc.cu.
#include <algorithm>

#include "fp_bits.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace gbcc {
namespace {

constexpr int BM = 128;
constexpr int HB = 32;          // K elements per stage: 64 bytes, one 64-byte swizzle row
constexpr int kEpiWarp0 = 2;     // no idle warps: 200 registers a thread (four sums per output, six slices)

// Shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512
// bytes apart.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(16u >> 4) << 16;   // leading byte offset (unused for swizzled K-major)
  d |= static_cast<uint64_t>(512u >> 4) << 32;  // stride byte offset
  d |= static_cast<uint64_t>(1) << 46;          // descriptor version
  d |= static_cast<uint64_t>(4) << 61;          // 64-byte swizzle
  return d;
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr));
}

template <int SL, int BN>
struct MultiCfg {
  static constexpr uint32_t kASlice = BM * HB * 2;
  static constexpr uint32_t kBSlice = BN * HB * 2;
  static constexpr uint32_t kAStage = SL * kASlice;
  static constexpr uint32_t kStage = SL * (kASlice + kBSlice);
  // three slices: a tile's MMAs are short and its epilogue is a chain of TMEM reads
  // and stores, so four warps a scheduler share it where the tile is wide (v = 120
  // 242 -> 227 ms, v = 97 16.8 -> 16.2; below, equal or 2 % slower: the staging
  // takes a pipeline stage)
  static constexpr int kEpiWarps = SL == 3 && BN > 80 ? 16 : 8;
  static constexpr int kThreads = 32 * (kEpiWarp0 + kEpiWarps);
  // epilogue staging per warp: 32 rows x kStgCols words of 8 bytes
  static constexpr int kStgCols = SL == 3 ? 8 : 4;
  static constexpr int kStgLd = SL == 3 ? 9 : 4;
  static constexpr uint32_t kStg = kEpiWarps * 32 * kStgLd * 8;
  static constexpr int kFit = static_cast<int>((232448u - 1024u - 512u - kStg) / kStage);
  static constexpr int kStages = kFit > 6 ? 6 : kFit;
  static_assert(kStages >= 2, "at least two pipeline stages");
  static constexpr uint32_t kSmem = 1024 + kStages * kStage + kStg + 512;
  static constexpr int kClasses = SL == 3 ? 1 : SL;  // accumulators a chunk fills
  static constexpr int kBufs = SL == 3 ? 4 : 8;      // accumulators they rotate through
  static constexpr int kChunk = SL == 3 ? 1 : 5;     // stages a chunk covers
  static constexpr uint32_t kCols = kBufs * BN <= 64 ? 64 : (kBufs * BN <= 128 ? 128 : (kBufs * BN <= 256 ? 256 : 512));
  static_assert(kBufs * BN <= 512, "tensor memory");
  static_assert(BN % 16 == 0, "MMA width");
  static constexpr int kOut = BN / (kEpiWarps / 4);  // columns per epilogue thread
};

constexpr int kWindow = 1000;  // stages of a tile in one launch (six slices): 200 chunks
constexpr int kRenorm = 4;     // chunks between renormalisations

// one output tile: where its operand segments and its output lie
struct Tile {
  int nseg;
  int a_x[2], b_row[2];  // (T): first index of the A rows, first B row; GEMM: unused, first B row
  int row0, fast0;       // GEMM: first row; (T): slow and fast virtual block starts
  int n0;
  int hb0, hb1;          // stages of K
  int split;
  int64_t out;           // (T): first element of the tile's sum array
};

template <bool TRIPLES>
__device__ __forceinline__ Tile decode(const GemmMultiArgs& g, int t, int BN) {
  Tile T;
  T.hb0 = 0;
  T.hb1 = g.hbs;
  T.split = 0;
  if constexpr (TRIPLES) {
    T.nseg = 2;
    const int nt = t % g.ntn;
    t /= g.ntn;
    const int fast = t % g.ntf;
    t /= g.ntf;
    const int slow = t % g.nts;
    t /= g.nts;
    const int grp = t % 3, tr = t / 3;
    const int4 ijk = g.triples[tr];
    const int i = ijk.x, j = ijk.y, k = ijk.z;
    T.row0 = slow * 8;
    T.fast0 = fast * 16;
    T.n0 = nt * BN;
    // sums of the terms (i,j,k) + (j,i,k); (i,k,j) + (k,i,j); (j,k,i) + (k,j,i)
    const int x1 = grp == 2 ? j : i, y1 = grp == 0 ? j : k, z1 = grp == 0 ? k : (grp == 1 ? j : i);
    const int x2 = grp == 0 ? j : k, y2 = grp == 2 ? j : i, z2 = grp == 0 ? k : (grp == 1 ? j : i);
    T.a_x[0] = x1;
    T.a_x[1] = x2;
    T.b_row[0] = (y1 * g.o + z1) * g.v + T.n0;
    T.b_row[1] = (y2 * g.o + z2) * g.v + T.n0;
    T.out = (static_cast<int64_t>(tr) * 3 + grp) * g.v * g.v * g.v;
  } else {
    T.nseg = 1;
    const int mn = g.ntm * g.ntn;
    T.split = t / mn;
    t -= T.split * mn;
    const int mt = t / g.ntn, nt = t - mt * g.ntn;
    T.row0 = mt * BM;
    T.n0 = nt * BN;
    T.b_row[0] = T.n0;
    const int end = min(g.hbs, (T.split + 1) * g.hb_per_split);
    T.hb0 = min(end, T.split * g.hb_per_split + g.hb_first);
    T.hb1 = min(end, T.hb0 + kWindow);
  }
  return T;
}

template <int SL, int BN, bool TRIPLES>
__global__ void __launch_bounds__(MultiCfg<SL, BN>::kThreads, 1)
    gemm_multi_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA2,
                      const __grid_constant__ CUtensorMap tmB, const __grid_constant__ GemmMultiArgs g) {
  using Cfg = MultiCfg<SL, BN>;
  constexpr int S = Cfg::kStages, NC = Cfg::kClasses, NBUF = Cfg::kBufs, OUT = Cfg::kOut;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* stg_all = smem + S * Cfg::kStage;
  uint64_t* full = reinterpret_cast<uint64_t*>(stg_all + Cfg::kStg);
  uint64_t* empty = full + S;
  uint64_t* acc_full = empty + S;         // [NBUF]
  uint64_t* acc_empty = acc_full + NBUF;  // [NBUF]
  uint64_t* done = acc_empty + NBUF;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < NBUF; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], Cfg::kEpiWarps);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::kCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int kblocks = g.kblocks;
  const uint32_t lead = elect_lead();  // (every warp: only 0 and 1 use it)

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmA);
      if (TRIPLES) prefetch_tmap(&tmA2);
      prefetch_tmap(&tmB);
    }
    __syncwarp();
    const uint32_t smem0 = smem_u32(smem);
    uint32_t gi = 0;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
      const Tile T = decode<TRIPLES>(g, t, BN);
#pragma unroll
      for (int seg = 0; seg < (TRIPLES ? 2 : 1); ++seg) {
        for (int hb = T.hb0; hb < T.hb1 && ok; ++hb, ++gi) {
          ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ph ^ 1, g.err));
          if (!ok) {
            record_error(g.err, kDevTimeout);
            break;
          }
          const uint32_t st = smem0 + s * Cfg::kStage;
          mbar_expect_tx(lead, &full[s], Cfg::kStage);
          const int c0 = HB * (hb & 1), kb = hb >> 1;
#pragma unroll
          for (int p = 0; p < SL; ++p) {
            if constexpr (TRIPLES)
              tma_load_5d(lead, seg ? &tmA2 : &tmA, &full[s], st + p * Cfg::kASlice, c0, T.fast0, T.row0, T.a_x[seg],
                                  p * kblocks + kb);
            else
              tma_load_3d(lead, &tmA, &full[s], st + p * Cfg::kASlice, c0, T.row0, p * kblocks + kb);
            tma_load_3d(lead, &tmB, &full[s], st + Cfg::kAStage + p * Cfg::kBSlice, c0, T.b_row[seg],
                                p * kblocks + kb);
          }
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
        }
      }
    }
    // every copy issued here has landed before the CTA can exit
    const uint32_t first = gi > static_cast<uint32_t>(S) ? gi - S : 0;
    for (uint32_t u = first; u < gi; ++u) mbar_wait_teardown(&full[u % S], (u / S) & 1);
  } else if (warp == 1) {
    constexpr uint32_t idesc = idesc_bf16(BM, BN);
    const uint64_t desc0 = sdesc_sw64(smem_u32(smem));
    uint32_t q = 0;  // accumulators filled
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
      const Tile T = decode<TRIPLES>(g, t, BN);
      for (int seg = 0; seg < T.nseg && ok; ++seg) {
        int pos = 0;
        for (int hb = T.hb0; hb < T.hb1 && ok; ++hb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full[s], ph, g.err));
          if (!ok) break;
          tc_fence_after();
          const bool first = pos == 0, last = pos == Cfg::kChunk - 1 || hb == T.hb1 - 1;
          // the last 32 elements of K may hold 16 or fewer
          const bool two = hb != g.hbs - 1 || g.last_k16 == 2;
          const uint64_t ad0 = desc0 + static_cast<uint64_t>(s * (Cfg::kStage >> 4));
          const uint64_t bd0 = ad0 + (Cfg::kAStage >> 4);
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const uint32_t b = (q + c) % NBUF;
            if (first) {
              ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[b], (((q + c) / NBUF) & 1) ^ 1, g.err));
              if (!ok) break;
              tc_fence_after();
            }
            const uint32_t d = tmem + b * BN;
            // SL 3: pairs p + q < 3, all in one accumulator; SL 6: those of class SL - 1 - c
#pragma unroll
            for (int w = SL == 3 ? 0 : SL - 1 - c; w <= (SL == 3 ? SL - 1 : SL - 1 - c); ++w) {
#pragma unroll
              for (int p = 0; p <= w; ++p) {
                const uint64_t ad = ad0 + ((p * Cfg::kASlice) >> 4), bd = bd0 + (((w - p) * Cfg::kBSlice) >> 4);
                const uint32_t acc = SL == 3 ? (w + p > 0 ? 1u : 0u) : ((!first || p > 0) ? 1u : 0u);
                mma_bf16(lead, d, ad, bd, idesc, acc);
                if (two) mma_bf16(lead, d, ad + 2, bd + 2, idesc, 1u);
              }
            }
            if (last) mma_commit(lead, &acc_full[b]);
          }
          if (!ok) break;
          mma_commit(lead, &empty[s]);
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
          if (last) {
            q += NC;
            pos = 0;
          } else {
            ++pos;
          }
        }
      }
    }
    if (!ok) record_error(g.err, kDevTimeout);
    mma_commit(lead, done);
    mbar_wait_teardown(done, 0);
  } else if (warp >= kEpiWarp0) {
    const int qd = warp & 3, h = (warp - kEpiWarp0) >> 2;
    const int row = qd * 32 + lane, col0 = h * OUT;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    uint8_t* stg = stg_all + (warp - kEpiWarp0) * 32 * Cfg::kStgLd * 8;
    uint32_t q = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < g.tiles && ok; t += gridDim.x) {
      const Tile T = decode<TRIPLES>(g, t, BN);
      // SL 3: x0 the running segment's FP32 sum, x1 the first segment's;
      // SL 6: (x0, x1) and (x2, x3) float-float sums of classes 0-2 and 3-5
      float x0[OUT], x1[OUT], x2[SL == 3 ? 1 : OUT], x3[SL == 3 ? 1 : OUT];
#pragma unroll
      for (int j = 0; j < OUT; ++j) {
        x0[j] = x1[j] = 0.f;
        x2[SL == 3 ? 0 : j] = x3[SL == 3 ? 0 : j] = 0.f;
      }
      const int nchunks = (T.hb1 - T.hb0 + Cfg::kChunk - 1) / Cfg::kChunk;
      int unnorm = 0;  // chunks since the pairs were renormalised
      for (int seg = 0; seg < T.nseg && ok; ++seg) {
        if constexpr (SL == 3) {
          if (seg == 1) {
#pragma unroll
            for (int j = 0; j < OUT; ++j) {
              x1[j] = x0[j];
              x0[j] = 0.f;
            }
          }
        }
        // adds accumulator q + c to float-float sums (hi, lo), or to hi alone
        auto drain = [&](int c, auto& hi, auto& lo) {
          const uint32_t b = (q + c) % NBUF;
          if (!mbar_wait(&acc_full[b], ((q + c) / NBUF) & 1, g.err)) {
            record_error(g.err, kDevTimeout);
            ok = false;
            return;
          }
          tc_fence_after();
          const uint32_t base = tmem + lane_addr + b * BN + col0;
          if constexpr (SL == 3) {
            uint32_t r[OUT];
#pragma unroll
            for (int j0 = 0; j0 < OUT; j0 += 4) tmem_ld4(base + j0, r + j0);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < OUT; ++j) hi[j] = __fadd_rn(hi[j], __uint_as_float(r[j]));
          } else {
#pragma unroll
            for (int j0 = 0; j0 < OUT; j0 += 16) {
              uint32_t r0[8], r1[8];
              tmem_ld8(base + j0, r0);
              if (j0 + 8 < OUT) tmem_ld8(base + j0 + 8, r1);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                if (j0 + j >= OUT) continue;
                two_sum_acc(hi[j0 + j], lo[j0 + j], __uint_as_float(j < 8 ? r0[j & 7] : r1[j & 7]));
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&acc_empty[b]);
        };
        auto renormalise = [&](auto& hi, auto& lo) {
#pragma unroll
          for (int j = 0; j < OUT; ++j) {
            const float h = hi[j];
            hi[j] = __fadd_rn(h, lo[j]);
            // the rounding error of that sum (TwoSum)
            const float v = __fsub_rn(hi[j], h);
            lo[j] = __fadd_rn(__fsub_rn(h, __fsub_rn(hi[j], v)), __fsub_rn(lo[j], v));
          }
        };
        for (int ch = 0; ch < nchunks && ok; ++ch, q += NC) {
          if constexpr (SL == 3) {
            drain(0, x0, x1);
          } else {
#pragma unroll 1
            for (int c = 0; c < SL / 2 && ok; ++c) drain(c, x2, x3);  // classes 5, 4, 3
#pragma unroll 1
            for (int c = SL / 2; c < SL && ok; ++c) drain(c, x0, x1);  // classes 2, 1, 0
            if (++unnorm == kRenorm) {
              unnorm = 0;
              renormalise(x2, x3);
              renormalise(x0, x1);
            }
          }
        }
      }
      if (!ok) break;
      if (*reinterpret_cast<const volatile int*>(g.err) != kDevOk) continue;
      // the value of output column j of this thread's row, FP64 (SL 6)
      auto value = [&](int j) {
        const int k = SL == 3 ? 0 : j;
        return (f2d_exact(x2[k]) + f2d_exact(x3[k])) + (f2d_exact(x0[j]) + f2d_exact(x1[j]));
      };
      if constexpr (!TRIPLES) {
        if (g.ksplit == 1 && g.m_major) {
          const int64_t m = static_cast<int64_t>(T.row0) + row;
          if (m < g.M) {
            double* crow = g.C + g.cm[m];
#pragma unroll
            for (int j0 = 0; j0 < OUT; j0 += 8) {
              double cv[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int64_t n = T.n0 + col0 + j0 + j;
                cv[j] = (g.beta != 0.0 && n < g.N) ? crow[g.cn[n]] : 0.0;
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const int64_t n = T.n0 + col0 + j0 + j;
                if (n >= g.N) continue;
                const double x = value(j0 + j);
                crow[g.cn[n]] = g.beta == 0.0 ? g.alpha * x : fma(g.alpha, x, g.beta == 1.0 ? cv[j] : g.beta * cv[j]);
              }
            }
          }
          continue;
        }
      }
      // through shared memory, a few columns of 32 rows at a time, so that
      // neighbouring lanes write neighbouring columns
      constexpr int SC = Cfg::kStgCols, LD = Cfg::kStgLd, RP = 32 / SC;  // RP rows per store
      const int cj = lane % SC, rj = lane / SC;
      int rrow[SC];  // (T): this lane's rows (slow, fast) of the sum array, -1 past v
      if constexpr (TRIPLES) {
#pragma unroll
        for (int r = 0; r < SC; ++r) {
          const int lr = qd * 32 + rj + RP * r, slow = T.row0 + lr / 16, fast = T.fast0 + lr % 16;
          rrow[r] = (slow < g.v && fast < g.v) ? slow * g.v + fast : -1;
        }
      }
#pragma unroll
      for (int j0 = 0; j0 < OUT; j0 += SC) {
        if constexpr (SL == 3) {
          float2* s2 = reinterpret_cast<float2*>(stg);
#pragma unroll
          for (int j = 0; j < SC; ++j) {
            if (j0 + j >= OUT) continue;
            float hi = x0[j0 + j], lo = 0.f;
            two_sum_acc(hi, lo, x1[j0 + j]);
            s2[lane * LD + j] = make_float2(hi, lo);
          }
        } else {
          double* s8 = reinterpret_cast<double*>(stg);
#pragma unroll
          for (int j = 0; j < SC; ++j) s8[lane * LD + j] = value(j0 + j);
        }
        __syncwarp();
        const int64_t n = T.n0 + col0 + j0 + cj;
        if constexpr (TRIPLES) {
          if (n < g.v && (OUT % SC == 0 || j0 + cj < OUT)) {
            double* out = g.W + T.out + n;
#pragma unroll
            for (int r = 0; r < SC; ++r)
              if (rrow[r] >= 0)
                out[static_cast<int64_t>(rrow[r]) * g.v] = reinterpret_cast<const double*>(stg)[(rj + RP * r) * LD + cj];
          }
        } else {
          const double* s8 = reinterpret_cast<const double*>(stg);
          if (g.ksplit > 1) {
            double* P = g.partial + static_cast<int64_t>(T.split) * g.Mpad * g.Npad + n;
#pragma unroll
            for (int r = 0; r < SC; ++r) {
              const int rr = rj + RP * r;
              double* at = P + (static_cast<int64_t>(T.row0) + qd * 32 + rr) * g.Npad;
              *at = g.hb_first ? *at + s8[rr * LD + cj] : s8[rr * LD + cj];
            }
          } else if (n < g.N) {
            const int64_t on = g.cn[n];
            double cv[SC];
            int64_t off[SC];
#pragma unroll
            for (int r = 0; r < SC; ++r) {
              const int64_t m = static_cast<int64_t>(T.row0) + qd * 32 + rj + RP * r;
              off[r] = m < g.M ? g.cm[m] + on : -1;
              cv[r] = (g.beta != 0.0 && off[r] >= 0) ? g.C[off[r]] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < SC; ++r) {
              if (off[r] < 0) continue;
              const double x = s8[(rj + RP * r) * LD + cj];
              g.C[off[r]] = g.beta == 0.0 ? g.alpha * x : fma(g.alpha, x, g.beta == 1.0 ? cv[r] : g.beta * cv[r]);
            }
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::kCols);
  }
}

// Slice panels are k-block major, [slices][Kpad / 64][rows][64] (gemm_tc.cu); a
// box takes half a k-block of `box_rows` rows.
bool panel_map(CUtensorMap* map, const void* base, int64_t slices, int64_t rows, int64_t kblocks, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(slices * kblocks)};
  cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(rows) * 128};
  cuuint32_t box[3] = {HB, static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A panel of rows (x, slow, fast), x < o and slow, fast < v: a box takes half a
// k-block of 8 x 16 rows, zeros past v
bool pair_panel_map(CUtensorMap* map, const void* base, int64_t slices, int64_t o, int64_t v, int64_t kblocks) {
  auto fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t vv = static_cast<cuuint64_t>(v), oo = static_cast<cuuint64_t>(o);
  cuuint64_t dims[5] = {64, vv, vv, oo, static_cast<cuuint64_t>(slices * kblocks)};
  cuuint64_t strides[4] = {128, 128 * vv, 128 * vv * vv, 128 * vv * vv * oo};
  cuuint32_t box[5] = {HB, 16, 8, 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int SL, int BN, bool TRIPLES>
bool launch(const GemmMultiArgs& g, const CUtensorMap& a, const CUtensorMap& a2, cudaStream_t st) {
  using Cfg = MultiCfg<SL, BN>;
  CUtensorMap b;
  if (!panel_map(&b, g.B, SL, g.b_rows, g.kblocks, BN)) return false;
  static const bool attr = cudaFuncSetAttribute(gemm_multi_kernel<SL, BN, TRIPLES>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                Cfg::kSmem) == cudaSuccess;
  if (!attr) return false;
  gemm_multi_kernel<SL, BN, TRIPLES><<<std::min(g.tiles, num_sms()), Cfg::kThreads, Cfg::kSmem, st>>>(a, a2, b, g);
  return true;
}

}  // namespace

int gemm_multi_bn(int64_t N) { return N <= 32 ? 32 : 64; }

int triples_bn(int slices, int64_t v) {
  // the even share of v in steps of 16, at most 128 columns (three slices) or 64 (six)
  const int64_t most = slices == 3 ? 128 : 64;
  const int64_t parts = (v + most - 1) / most;
  const int64_t bn = ((v + parts - 1) / parts + 15) / 16 * 16;
  return static_cast<int>(slices == 3 ? std::max<int64_t>(bn, 32) : (bn <= 32 ? 32 : 64));
}

int launch_gemm_fixed(GemmMultiArgs g, cudaStream_t st) {
  if (g.M < 1 || g.N < 1 || g.K < 1 || (g.bn != 32 && g.bn != 64) || g.kblocks * 64 < g.K || g.a_rows < g.M ||
      g.b_rows < g.N)
    return 0;
  g.hbs = static_cast<int>((g.K + HB - 1) / HB);
  g.last_k16 = (g.K - 1) % HB < 16 ? 1 : 2;
  const int64_t ntm = (g.M + BM - 1) / BM, ntn = (g.N + g.bn - 1) / g.bn;
  if (g.ksplit < 1) g.ksplit = 1;
  if (g.ksplit == 1) g.hb_per_split = g.hbs;
  if (g.ksplit > 1 && (!g.partial || g.hb_per_split < 1 ||
                       static_cast<int64_t>(g.ksplit - 1) * g.hb_per_split >= g.hbs ||
                       static_cast<int64_t>(g.ksplit) * g.hb_per_split < g.hbs))
    return 0;
  const int64_t tiles = ntm * ntn * g.ksplit;
  if (tiles > (1LL << 30) || g.M > (1LL << 30) || g.N > (1LL << 30)) return 0;
  g.ntm = static_cast<int>(ntm);
  g.ntn = static_cast<int>(ntn);
  g.tiles = static_cast<int>(tiles);
  g.Mpad = ntm * BM;
  g.Npad = ntn * g.bn;
  CUtensorMap a;
  if (!panel_map(&a, g.A, kFixedSlices, g.a_rows, g.kblocks, BM)) return 0;
  int n = 0;
  for (g.hb_first = 0; g.hb_first < g.hb_per_split; g.hb_first += kWindow, ++n) {
    if (!(g.bn == 32 ? launch<kFixedSlices, 32, false>(g, a, a, st) : launch<kFixedSlices, 64, false>(g, a, a, st)))
      return 0;
    g.beta = 1.0;
  }
  return n;
}

bool launch_gemm_triples(GemmMultiArgs g, int slices, int ntriples, cudaStream_t st) {
  if (ntriples < 1) return true;
  if (g.o < 1 || g.v < 1 || g.K < 1 || g.kblocks * 64 < g.K || (slices != 3 && slices != kFixedSlices)) return false;
  g.hbs = static_cast<int>((g.K + HB - 1) / HB);
  g.last_k16 = (g.K - 1) % HB < 16 ? 1 : 2;
  g.bn = triples_bn(slices, g.v);
  g.nts = (g.v + 7) / 8;
  g.ntf = (g.v + 15) / 16;
  g.ntn = (g.v + g.bn - 1) / g.bn;
  const int64_t tiles = static_cast<int64_t>(ntriples) * 3 * g.nts * g.ntf * g.ntn;
  // (32-bit rows of B, virtual pairs and tiles; offsets in the sums are 64-bit)
  if (tiles > (1LL << 30) || static_cast<int64_t>(g.o) * g.o * g.v > (1LL << 30) ||
      static_cast<int64_t>(g.v) * g.v > (1LL << 30))
    return false;
  g.tiles = static_cast<int>(tiles);
  g.b_rows = static_cast<int64_t>(g.o) * g.o * g.v;
  CUtensorMap a, a2;
  if (!pair_panel_map(&a, g.A, slices, g.o, g.v, g.kblocks) || !pair_panel_map(&a2, g.A2, slices, g.o, g.v, g.kblocks))
    return false;
  if (slices == kFixedSlices)
    return g.bn == 32 ? launch<kFixedSlices, 32, true>(g, a, a2, st) : launch<kFixedSlices, 64, true>(g, a, a2, st);
  switch (g.bn) {
    case 32: return launch<3, 32, true>(g, a, a2, st);
    case 48: return launch<3, 48, true>(g, a, a2, st);
    case 64: return launch<3, 64, true>(g, a, a2, st);
    case 80: return launch<3, 80, true>(g, a, a2, st);
    case 96: return launch<3, 96, true>(g, a, a2, st);
    case 112: return launch<3, 112, true>(g, a, a2, st);
    case 128: return launch<3, 128, true>(g, a, a2, st);
    default: return false;
  }
}

}  // namespace gbcc

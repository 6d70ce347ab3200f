// Split-BF16 GEMM on CTA pairs (tcgen05 cta_group::2): 256 x 256 output tiles,
// every slice of a K block staged once.  Same operands and result as
// gemm_tc_kernel (kernels.h); the tuner takes it for large M and N.
//
// What it removes: on one CTA a 128 x 192 tile is bound by shared-memory
// bandwidth, 128 bytes a clock.  An MMA of 128 x 192 x 16 reads 10 KB and runs
// for 96 clocks, and with one slice pair per stage TMA writes another 40 KB
// for every four of them: 160 clocks of traffic per 96 of MMA (1.33 PFLOP/s of
// slice products on 9500^3).  In a pair each CTA holds half of B's rows, so an
// MMA of 256 x 256 x 16 reads 8 KB of each CTA in 128 clocks, and with all
// slices in a stage (32 elements of K: 64-byte swizzled rows) two slices write
// 32 KB for every six MMAs: 107 clocks of traffic per 128.
//
// One CTA per SM, 20 warps: 0 TMA (both CTAs load their halves, counted on the
// leader's barriers), 1 MMA (leader only), 4-19 epilogue -- 64 columns of a row
// a thread, which fits its FP32 sums in registers without spills.  Chunks and
// their FP32 register sums as in gemm_tc.cu's tiles of 192 and 256; bounded
// waits and teardown likewise.
//
// 9500^3, two slices, in bands of 8 tiles: 2.84 ms, 1.81 PFLOP/s of slice products
// (128 x 192 tiles on one CTA: 3.71 ms; 18145 x 1275 x 9000: 0.765 against 0.934 ms).
#include <algorithm>

#include "fp_bits.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace gbcc {
namespace {

constexpr int BM = 128;           // rows per CTA (256 per pair)
constexpr int BN = 256;
constexpr int HB = 32;            // K elements per stage
constexpr int kEpiWarps = 16;
constexpr int kEpiWarp0 = 4;
constexpr int kThreads = 32 * (kEpiWarp0 + kEpiWarps);
constexpr int kOut = BN / (kEpiWarps / 4);  // columns per epilogue thread
constexpr int kSC = 8, kLd = 9;   // epilogue staging: 32 rows x 8 floats a warp

// K-major, 64-byte swizzle, 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(16u >> 4) << 16;
  d |= static_cast<uint64_t>(512u >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;
  return d;
}

template <int SL>
struct PairCfg {
  static constexpr uint32_t kSlice = BM * HB * 2;   // one slice tile of A, and of a CTA's half of B
  static constexpr uint32_t kStage = 2 * SL * kSlice;
  static constexpr uint32_t kStg = kEpiWarps * 32 * kLd * 4;
  static constexpr int kStages = static_cast<int>((232448u - 1024u - 512u - kStg) / kStage);
  static constexpr uint32_t kSmem = 1024 + kStages * kStage + kStg + 512;
  static_assert(kStages >= 3, "pipeline stages");
};

template <int SL>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ GemmTcArgs g) {
  using Cfg = PairCfg<SL>;
  constexpr int S = Cfg::kStages;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const int unit = static_cast<int>(blockIdx.x / 2), nunits = static_cast<int>(gridDim.x / 2);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  float* stg_all = reinterpret_cast<float*>(smem + S * Cfg::kStage);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * Cfg::kStage + Cfg::kStg);
  uint64_t* empty = full + S;
  uint64_t* acc_full = empty + S;      // [2]
  uint64_t* acc_empty = acc_full + 2;  // [2]
  uint64_t* done = acc_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int ntm = static_cast<int>((g.M + 2 * BM - 1) / (2 * BM)), ntn = static_cast<int>((g.N + BN - 1) / BN);
  const int ksplit = g.ksplit > 1 ? g.ksplit : 1;
  const int ntiles_mn = ntm * ntn, ntiles = ntiles_mn * ksplit;
  const int kblocks = static_cast<int>(g.Kpad / kTcBK);
  const int kb_per_split = ksplit > 1 ? g.kb_per_split : kblocks;
  // stages per TMEM accumulation: g.chunk counts (64-element k-block, pair) steps
  constexpr int kPairs = SL * (SL + 1) / 2;
  const int chunk = max(1, 2 * g.chunk / kPairs);
  const int group = g.group > 1 ? g.group : 1;
  auto decode = [&](int tile, int& m0, int& n0, int& hb0, int& nhb, int& split) {
    split = tile / ntiles_mn;
    const int mn = tile - split * ntiles_mn;
    const int band = mn / (group * ntn);
    const int rows = min(ntm - band * group, group);
    const int idx = mn - band * group * ntn;
    m0 = (band * group + idx % rows) * 2 * BM + static_cast<int>(rank) * BM;
    n0 = idx / rows * BN;
    hb0 = 2 * split * kb_per_split;
    nhb = 2 * min(kblocks - split * kb_per_split, kb_per_split);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * kEpiWarps);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc2(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // both CTAs' barriers exist before any remote arrive
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lead = elect_lead();

  if (warp == 0) {
    if (lane == 0) {
      prefetch_tmap(&tmA);
      prefetch_tmap(&tmB);
    }
    __syncwarp();
    const uint32_t smem0 = smem_u32(smem), full0 = map_to_rank(&full[0], 0);
    uint32_t gi = 0;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = unit; tile < ntiles && ok; tile += nunits) {
      int m0, n0, hb0, nhb, split;
      decode(tile, m0, n0, hb0, nhb, split);
      const int nb0 = n0 + static_cast<int>(rank) * BM;
      for (int hb = hb0; hb < hb0 + nhb; ++hb, ++gi) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ph ^ 1, g.err));
        if (!ok) {
          record_error(g.err, kDevTimeout);
          break;
        }
        // the leader's full barrier counts the bytes of both CTAs
        const uint32_t bar = full0 + static_cast<uint32_t>(s) * 8u, st = smem0 + s * Cfg::kStage;
        if (leader) mbar_expect_tx(lead, &full[s], 2 * Cfg::kStage);
        const int c0 = HB * (hb & 1), kb = hb >> 1;
#pragma unroll
        for (int p = 0; p < SL; ++p) {
          tma_load_3d_pair(lead, &tmA, bar, st + p * Cfg::kSlice, c0, m0, p * kblocks + kb);
          tma_load_3d_pair(lead, &tmB, bar, st + (SL + p) * Cfg::kSlice, c0, nb0, p * kblocks + kb);
        }
        if (++s == S) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    // every copy issued here has landed before the CTA can exit: the leader's
    // full barriers count them; the partner sees them consumed
    const uint32_t first = gi > static_cast<uint32_t>(S) ? gi - S : 0;
    for (uint32_t u = first; u < gi; ++u) {
      if (leader) mbar_wait_teardown(&full[u % S], (u / S) & 1);
      else mbar_wait_teardown(&empty[u % S], (u / S) & 1);
    }
  } else if (warp == 1) {
    if (leader) {
      constexpr uint32_t idesc = idesc_bf16(2 * BM, BN);
      const uint64_t desc0 = sdesc_sw64(smem_u32(smem));
      uint32_t c = 0;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int tile = unit; tile < ntiles && ok; tile += nunits) {
        int m0, n0, hb0, nhb, split;
        decode(tile, m0, n0, hb0, nhb, split);
        int pos = 0;
        for (int it = 0; it < nhb; ++it) {
          const uint32_t b = c & 1;
          if (pos == 0) ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[b], ((c >> 1) & 1) ^ 1, g.err));
          if (ok) ok = __all_sync(0xffffffffu, mbar_wait(&full[s], ph, g.err));
          if (!ok) {
            record_error(g.err, kDevTimeout);
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + b * BN;
          const uint64_t ad0 = desc0 + static_cast<uint64_t>(s * (Cfg::kStage >> 4));
          const uint64_t bd0 = ad0 + ((SL * Cfg::kSlice) >> 4);
          // pairs p + q < SL
#pragma unroll
          for (int p = 0; p < SL; ++p)
#pragma unroll
            for (int q = 0; q < SL - p; ++q)
#pragma unroll
              for (int k = 0; k < HB / 16; ++k)
                mma_bf16_pair(lead, d, ad0 + ((p * Cfg::kSlice) >> 4) + 2 * k, bd0 + ((q * Cfg::kSlice) >> 4) + 2 * k,
                              idesc, (pos > 0 || p + q + k > 0) ? 1u : 0u);
          mma_commit_pair(lead, &empty[s], 0x3);
          if (++s == S) {
            s = 0;
            ph ^= 1;
          }
          if (++pos == chunk || it == nhb - 1) {
            mma_commit_pair(lead, &acc_full[b], 0x3);
            ++c;
            pos = 0;
          }
        }
      }
      mma_commit_pair(lead, done, 0x1);
      mbar_wait_teardown(done, 0);
    }
  } else if (warp >= kEpiWarp0) {
    const int qd = warp & 3, h = (warp - kEpiWarp0) >> 2;
    const int row = qd * 32 + lane, col0 = h * kOut;
    const uint32_t lane_addr = static_cast<uint32_t>(qd * 32) << 16;
    float* stg = stg_all + (warp - kEpiWarp0) * 32 * kLd;
    const uint32_t ae0 = map_to_rank(&acc_empty[0], 0), ae1 = map_to_rank(&acc_empty[1], 0);
    uint32_t c = 0;
    bool ok = true;
    for (int tile = unit; tile < ntiles && ok; tile += nunits) {
      int m0, n0, hb0, nhb, split;
      decode(tile, m0, n0, hb0, nhb, split);
      const int nchunks = (nhb + chunk - 1) / chunk;
      float p[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) p[j] = 0.f;
      for (int cc = 0; cc < nchunks; ++cc, ++c) {
        const uint32_t b = c & 1;
        if (!mbar_wait(&acc_full[b], (c >> 1) & 1, g.err)) {
          record_error(g.err, kDevTimeout);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t base = tmem + lane_addr + b * BN + col0;
#pragma unroll
        for (int j0 = 0; j0 < kOut; j0 += 16) {
          uint32_t r[16];
          tmem_ld16(base + j0, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) p[j0 + j] = __fadd_rn(p[j0 + j], __uint_as_float(r[j]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(b ? ae1 : ae0);
      }
      if (!ok) break;
      if (*reinterpret_cast<const volatile int*>(g.err) != kDevOk) continue;
      const double alpha = g.alpha, beta = g.beta;
      if (ksplit == 1 && g.m_major) {
        // C contiguous in M: every lane owns a row, the lanes of a warp write
        // 32 consecutive rows of one column
        const int64_t m = static_cast<int64_t>(m0) + row;
        if (m < g.M) {
          double* crow = g.C + g.cm[m];
#pragma unroll
          for (int j0 = 0; j0 < kOut; j0 += 4) {
            double cv[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int64_t n = static_cast<int64_t>(n0) + col0 + j0 + j;
              cv[j] = (beta != 0.0 && n < g.N) ? crow[g.cn[n]] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int64_t n = static_cast<int64_t>(n0) + col0 + j0 + j;
              if (n >= g.N) continue;
              const double x = f2d_exact(p[j0 + j]);
              crow[g.cn[n]] = beta == 0.0 ? alpha * x : fma(alpha, x, beta == 1.0 ? cv[j] : beta * cv[j]);
            }
          }
        }
        continue;
      }
      // 32 rows x 8 columns at a time through shared memory: 8 lanes write 64
      // contiguous bytes where C is contiguous in N
      const int cj = lane % kSC, rj = lane / kSC;
#pragma unroll
      for (int j0 = 0; j0 < kOut; j0 += kSC) {
#pragma unroll
        for (int j = 0; j < kSC; ++j) stg[lane * kLd + j] = p[j0 + j];
        __syncwarp();
        const int64_t n = static_cast<int64_t>(n0) + col0 + j0 + cj;
        if (ksplit > 1) {
          if (n < g.Npad) {
            double* P = g.partial + static_cast<int64_t>(split) * g.Mpad * g.Npad + n;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int rr = rj + 4 * r;
              const int64_t m = static_cast<int64_t>(m0) + qd * 32 + rr;
              if (m < g.Mpad) P[m * g.Npad] = f2d_exact(stg[rr * kLd + cj]);
            }
          }
        } else if (n < g.N) {
          const int64_t on = g.cn[n];
#pragma unroll
          for (int r0 = 0; r0 < 8; r0 += 4) {
            int64_t off[4];
            double cv[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const int64_t m = static_cast<int64_t>(m0) + qd * 32 + rj + 4 * (r0 + r);
              off[r] = m < g.M ? g.cm[m] + on : -1;
              cv[r] = (beta != 0.0 && off[r] >= 0) ? g.C[off[r]] : 0.0;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              if (off[r] < 0) continue;
              const double x = f2d_exact(stg[(rj + 4 * (r0 + r)) * kLd + cj]);
              g.C[off[r]] = beta == 0.0 ? alpha * x : fma(alpha, x, beta == 1.0 ? cv[r] : beta * cv[r]);
            }
          }
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  cluster_sync();  // no remote arrive or MMA into this CTA is pending
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc2(tmem, 512);
  }
}

bool panel_map(CUtensorMap* map, const void* base, int64_t slices, int64_t rows, int64_t kblocks) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(slices * kblocks)};
  cuuint64_t strides[2] = {128, static_cast<cuuint64_t>(rows) * 128};
  cuuint32_t box[3] = {HB, BM, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int SL>
bool launch(const GemmTcArgs& g, cudaStream_t st) {
  using Cfg = PairCfg<SL>;
  CUtensorMap a, b;
  const int64_t kblocks = g.Kpad / kTcBK;
  if (!panel_map(&a, g.A, SL, g.a_rows ? g.a_rows : g.Mpad, kblocks) ||
      !panel_map(&b, g.B, SL, g.b_rows ? g.b_rows : g.Npad, kblocks))
    return false;
  static const bool attr = cudaFuncSetAttribute(gemm_pair_kernel<SL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                Cfg::kSmem) == cudaSuccess;
  if (!attr) return false;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Cfg::kSmem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  static const int max_pairs = [&cfg] {
    cfg.gridDim = dim3(2 * (num_sms() / 2));
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<SL>, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = num_sms() / 2;
    }
    return n;
  }();
  const int64_t tiles = ((g.M + 2 * BM - 1) / (2 * BM)) * ((g.N + BN - 1) / BN) * (g.ksplit > 1 ? g.ksplit : 1);
  cfg.gridDim = dim3(static_cast<unsigned>(2 * std::min<int64_t>(tiles, max_pairs)));
  return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<SL>, a, b, g) == cudaSuccess;
}

}  // namespace

bool launch_gemm_pair(const GemmTcArgs& g, cudaStream_t st) {
  // whole panels of two or three slices, every pair p + q below the slice count
  const int sl = g.a_slices;
  if ((sl != 2 && sl != 3) || g.b_slices != sl || g.npairs != sl * (sl + 1) / 2 ||
      g.chunk < 1 || g.skip_stage1)
    return false;
  for (int q = 0; q < g.npairs; ++q)
    if (g.pa[q] < 0 || g.pb[q] < 0 || g.pa[q] + g.pb[q] >= sl) return false;
  return sl == 2 ? launch<2>(g, st) : launch<3>(g, st);
}

}  // namespace gbcc

// linear_sm100.cu — the projections on either side of the attention op for B200 (sm_100a):
//   out_j[M, N] = X[M, K] W_j[N, K]^T + b_j[N]  (+ residual[M, N])      j = 0 .. n_mats-1
// as ONE persistent tcgen05 kernel. It replaces, per layer of the reference's static GPT-2 graph,
//   * the three Q/K/V projections, each a cublasSgemm plus a bias pass
//     (darkforest-core/src/engine/static_gpt2.rs:1324-1326 -> darkforest-cuda/src/lib.rs:1138-1201,
//      darkforest-cuda/kernels/elementwise.cu:230-249): one launch writes Q, K and V straight into the
//     [S, H*D] slices the attention kernels read;
//   * the output projection, its bias pass and the first residual add (static_gpt2.rs:1339-1341).
// The CPU engine's definition is cpu_linear (static_gpt2.rs:2717-2733): acc = b[o] + sum_i x[i] w[o, i].
//
// Arithmetic: X and W are rounded to TF32 (nearest even) by the TFLOAT32 tensor maps in flight, products
// accumulate in fp32 in tensor memory, bias and residual are added in fp32 in the epilogue: the same
// arithmetic width as the attention op of the fp32 API.
//
// Structure (one CTA per SM at most, 320 threads):
//   warp 0      TMA producer: a ring of stages, each a 128 x 32 tile of X (16 KB) and this CTA's share of a TN x 32 tile of W_j,
//               128-byte swizzle, K-major - both operands are already K-major in global memory (rows of X and rows of W
//               are contiguous along the contraction);
//   warp 1      MMA issuer: kind::tf32 SS MMAs (four per stage) into one of two TN-column accumulators in tensor memory, so
//               that the epilogue of tile i overlaps the products of i+1;
//   warps 2-9   epilogue: tensor memory -> registers -> turned over in shared memory (+ bias, + residual, GELU) -> whole lines.
// What bounds it is moving operands: per 32 of K a CTA with a 128 x 256 tile brings in 48 KB for 512 cycles of MMA and reads
// them once more, 192 bytes a cycle where shared memory has 128 and L2 delivers about 52 per SM. In the pair form (PAIR, a
// cluster of two CTAs, cta_group::2) the two SMs share W: 32 KB each for the same 512 cycles. The tile width TN is chosen
// per call from a small cost model (see choose_form): wide where there are tiles enough, narrower to fill the last wave or, for
// few rows, the chip; where even narrow tiles leave SMs idle, a cluster of two to eight CTAs splits the contraction.
// Measured on B200, width 768, against one CTA per 128 x 256 tile and stores through the copy engine: 8192 rows Q/K/V 51 -> 46
// us, output projection with residual 43 -> 25, MLP up with GELU 89 -> 80, MLP down 95 -> 66; 100 rows 17.7 -> 8.9, 23 -> 7.6,
// 23 -> 9.6, 42 -> 12.3; 32768 rows Q/K/V 186 -> 164 (707 TFLOP/s, at the chip's power limit like cuBLAS).
// Tiles are numbered with the output-feature tile fastest, so CTAs working at the same time share the
// same rows of X through L2 while the W_j (a few MB) stay resident there. Rows beyond M, features beyond N
// and a ragged end of K are zero-filled by the copy engine on loads.
// Every mbarrier wait is bounded (sm100_ptx.cuh); there is no named-barrier or spin wait without a limit.
#include <math.h>
#include <stdio.h>

#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {
namespace {

using namespace ptx;

constexpr int TM = 128, TK = 32;
constexpr int kEpiWarps = 8, kLinThreads = (2 + kEpiWarps) * 32;
constexpr uint32_t kABytes = TM * TK * 4;
constexpr uint32_t kSlabBytes = 32 * 32 * 4;                      // a warp's staging slab: 32 rows x 32 floats
constexpr uint32_t kSmemLimit = 227 * 1024;

template <int TN_, bool PAIR_, int KS_>
struct LinCfg {
  static constexpr int TN = TN_;
  static constexpr bool PAIR = PAIR_;
  static constexpr int KS = KS_;                                  // CTAs (a cluster) that share a tile's contraction
  static constexpr int kBRows = TN / (PAIR ? 2 : 1);              // rows of W in this CTA's shared memory
  static constexpr uint32_t kBBytes = kBRows * TK * 4, kStageBytes = kABytes + kBBytes;
  static constexpr int kFit = (int)((kSmemLimit - 1024 - 320 - kEpiWarps * kSlabBytes) / kStageBytes);
  static constexpr int kStages = kFit > 8 ? 8 : kFit;
  static constexpr uint32_t kSmemStaging = kStages * kStageBytes;
  static constexpr uint32_t kSmemBars = kSmemStaging + kEpiWarps * kSlabBytes;
  static constexpr uint32_t kSmemTotal = kSmemBars + 320 + 1024;
  static constexpr uint32_t kTmemCols = 2 * TN <= 128 ? 128 : (2 * TN <= 256 ? 256 : 512);
  static constexpr int FULL = 0, EMPTY = FULL + kStages, ACC_FULL = EMPTY + kStages, ACC_EMPTY = ACC_FULL + 2, DRAIN = ACC_EMPTY + 2,
                       NUM_BARS = DRAIN + 1;
  static_assert(NUM_BARS * 8 <= 192, "barriers overlap the abort flag");
  // split contraction: partial sums meet as [KS][128][kPartLd] over the operand stages of the CTA that owns their columns
  static constexpr int kOwned = TN / KS, kPartLd = kOwned + 4;
  static_assert(KS == 1 || (!PAIR && (uint32_t)KS * TM * kPartLd * 4 <= kSmemStaging), "partial sums do not fit");
};

struct LinParams {
  const float *bias[3];
  const float *residual;
  float *out[3];
  float *gelu_out;  // one matrix: a second output that receives gelu(x W^T + b)
  int store_pre;    // with gelu_out: also write the pre-activation (the backward needs it)
  uint32_t M, N, K;
  int n_mats, n_tiles_per_mat, n_tiles_total;  // output-feature tiles per matrix / over all matrices
  long long tiles;
  unsigned int *status;
};

template <class C>
__global__ void __launch_bounds__(kLinThreads, 1)
k_linear_tf32(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW0,
              const __grid_constant__ CUtensorMap tmW1, const __grid_constant__ CUtensorMap tmW2, const LinParams p) {
  constexpr int TN = C::TN, kStages = C::kStages, KS = C::KS;
  constexpr bool PAIR = C::PAIR;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t a0 = smem_u32(smem);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::kSmemBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + C::kSmemBars + 192);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + C::kSmemBars + 196);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = PAIR ? cluster_rank() : 0, part = KS > 1 ? cluster_rank() : 0;
  auto bar = [&](int id) { return smem_u32(&bars[id]); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NUM_BARS; ++i)
      mbar_init(bar(i), i == C::ACC_EMPTY || i == C::ACC_EMPTY + 1 ? (PAIR ? 2 : 1) * kEpiWarps : 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(tmem_holder), C::kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(tmem_holder), C::kTmemCols);
      tmem_relinquish();
    }
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW0);
  }
  tc_fence_before_sync();
  if (PAIR) cluster_sync();  // the other CTA's barriers are initialised, too
  else __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  pdl_wait();  // everything above touched only this CTA's shared and tensor memory
  const int all_kb = (int)((p.K + TK - 1) / TK), kb_first = (int)part * all_kb / KS, n_kb = ((int)part + 1) * all_kb / KS - kb_first;
  constexpr int kCtas = PAIR ? 2 : KS;  // CTAs per tile
  const long long first_tile = blockIdx.x / kCtas, tile_step = gridDim.x / kCtas;

  // tile number -> (this CTA's 128-row block, matrix, feature tile); the feature tile runs fastest
  auto decode = [&](long long id, int *m_tile, int *mat, int *n_tile) {
    *m_tile = (int)(id / p.n_tiles_total) * (PAIR ? 2 : 1) + (int)rank;
    const int nn = (int)(id % p.n_tiles_total);
    *mat = nn / p.n_tiles_per_mat;
    *n_tile = nn % p.n_tiles_per_mat;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (in a pair: each CTA its own tiles)
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (long long id = first_tile; ok && id < p.tiles; id += tile_step) {
        int m_tile, mat, n_tile;
        decode(id, &m_tile, &mat, &n_tile);
        const CUtensorMap *tw = mat == 0 ? &tmW0 : (mat == 1 ? &tmW1 : &tmW2);
        for (int kb = 0; kb < n_kb; ++kb, ++it) {
          const uint32_t s = it % kStages, use = it / kStages;
          if (use > 0 && !mbar_wait(bar(C::EMPTY + s), (use - 1) & 1, abort_flag)) { ok = false; break; }
          const uint32_t sa = a0 + s * C::kStageBytes;
          if (PAIR) {
            // both CTAs' copies count on the even CTA's barrier, which expects the bytes of both
            const uint32_t full = map_to_rank(bar(C::FULL + s), 0);
            if (rank == 0) mbar_arrive_expect_tx(bar(C::FULL + s), 2 * C::kStageBytes);
            tma_load_2d_pair(sa, &tmX, full, kb * TK, m_tile * TM);
            tma_load_2d_pair(sa + kABytes, tw, full, kb * TK, n_tile * TN + (int)rank * C::kBRows);
          } else {
            mbar_arrive_expect_tx(bar(C::FULL + s), C::kStageBytes);
            tma_load_2d(sa, &tmX, bar(C::FULL + s), (kb_first + kb) * TK, m_tile * TM);
            tma_load_2d(sa + kABytes, tw, bar(C::FULL + s), (kb_first + kb) * TK, n_tile * TN);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (in a pair: the even CTA)
    // The whole warp runs this role, warp-uniformly; one elected lane issues the MMA and commit instructions and
    // every wait returns the same answer in all lanes (see elect_one).
    if (rank == 0) {
      const uint32_t idesc = make_idesc(kFmtTF32, PAIR ? 2 * TM : TM, TN, 0, 0);
      uint32_t it = 0, j = 0;
      bool ok = true;
      for (long long id = first_tile; ok && id < p.tiles; id += tile_step, ++j) {
        const uint32_t acc = j & 1;
        if (j >= 2 && !mbar_wait_warp(bar(C::ACC_EMPTY + acc), ((j >> 1) - 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        for (int kb = 0; kb < n_kb; ++kb, ++it) {
          const uint32_t s = it % kStages;
          if (!mbar_wait_warp(bar(C::FULL + s), (it / kStages) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = a0 + s * C::kStageBytes, sb = sa + kABytes;
          const uint64_t da = make_smem_desc(sa, 16, 1024, kSwz128), db = make_smem_desc(sb, 16, 1024, kSwz128);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < TK / 8; ++k) {
              const uint64_t off = (uint64_t)((k * 32) >> 4);
              if (PAIR) mma_tf32_ss_pair(tmem + acc * TN, da + off, db + off, idesc, (kb > 0 || k > 0) ? 1u : 0u);
              else mma_tf32_ss(tmem + acc * TN, da + off, db + off, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            }
            if (PAIR) mma_commit_pair(bar(C::EMPTY + s));
            else mma_commit(bar(C::EMPTY + s));
            if (kb + 1 == n_kb) {
              if (PAIR) mma_commit_pair(bar(C::ACC_FULL + acc));
              else mma_commit(bar(C::ACC_FULL + acc));
            }
          }
          __syncwarp();
        }
      }
    }
  } else if (KS == 1) {
    // ------------------------------------------------------------ epilogue
    // A warp has the 32 accumulator rows of its quarter of tensor memory (a row per lane) and half of the tile's columns,
    // 32 at a time. It turns each 32 x 32 block over in a slab of shared memory of its own, so that bias, residual and
    // results move as whole 128-byte lines (four rows per instruction), and waits for no other warp. The residual of the
    // next block is on its way while the current one is worked on, the tile's first while its products still run.
    // (Tensor stores from the slab instead, with their proxy fence and the wait for the slab, took 1.2 us per block.)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    constexpr int kGroups = TN / 64;  // 32-column blocks of this warp
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    float4 *slab = reinterpret_cast<float4 *>(smem + C::kSmemStaging + (warp - 2) * kSlabBytes);
    const int lrow = lane >> 3, chunk = lane & 7;  // turned over: this lane has 16-byte chunk `chunk` of rows lrow, lrow + 4, ..
    uint32_t j = 0;
    for (long long id = first_tile; id < p.tiles; id += tile_step, ++j) {
      int m_tile, mat, n_tile;
      decode(id, &m_tile, &mat, &n_tile);
      const float *bias = mat == 0 ? p.bias[0] : (mat == 1 ? p.bias[1] : p.bias[2]);
      float *out = mat == 0 ? p.out[0] : (mat == 1 ? p.out[1] : p.out[2]);
      const uint32_t acc = j & 1;
      const int first_col = n_tile * TN + half * (TN / 2) + 4 * chunk;
      const long long row0 = (long long)m_tile * TM + quarter * 32 + lrow;
      const int n_rows = (long long)p.M - row0 <= 0 ? 0 : ((long long)p.M - row0 >= 32 ? 8 : (int)((p.M - row0 + 3) >> 2));  // of this lane's 8
      const size_t at0 = (size_t)row0 * p.N + first_col;
      float4 res[8], b4 = make_float4(0.f, 0.f, 0.f, 0.f);
      auto fetch = [&](int cg) {
        if (first_col + cg * 32 < (int)p.N) {
          if (bias) b4 = __ldg(reinterpret_cast<const float4 *>(bias + first_col + cg * 32));
          if (p.residual) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (i < n_rows) res[i] = __ldg(reinterpret_cast<const float4 *>(p.residual + at0 + cg * 32 + (size_t)(4 * i) * p.N));
          }
        }
      };
      fetch(0);
      if (!mbar_wait_warp(bar(C::ACC_FULL + acc), (j >> 1) & 1, abort_flag)) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int cg = 0; cg < kGroups; ++cg) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + acc * TN + half * (TN / 2) + cg * 32, r);
        tmem_wait_ld();
        if (cg == kGroups - 1) {
          // this warp's share of the accumulator has been read: the MMA warp may start the tile after next in it
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            if (PAIR) mbar_arrive_cluster(map_to_rank(bar(C::ACC_EMPTY + acc), 0));
            else mbar_arrive(bar(C::ACC_EMPTY + acc));
          }
        }
        __syncwarp();  // the block before has been read
#pragma unroll
        for (int x = 0; x < 8; ++x)
          slab[lane * 8 + (x ^ (lane & 7))] = make_float4(__uint_as_float(r[4 * x]), __uint_as_float(r[4 * x + 1]), __uint_as_float(r[4 * x + 2]),
                                                          __uint_as_float(r[4 * x + 3]));
        __syncwarp();
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[i] = slab[(4 * i + lrow) * 8 + (chunk ^ ((4 * i + lrow) & 7))];
          v[i].x += b4.x; v[i].y += b4.y; v[i].z += b4.z; v[i].w += b4.w;
          if (p.residual) {
            v[i].x += res[i].x; v[i].y += res[i].y; v[i].z += res[i].z; v[i].w += res[i].w;
          }
        }
        const bool in = first_col + cg * 32 < (int)p.N;  // N is a multiple of 4
        if (cg + 1 < kGroups) fetch(cg + 1);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (!in || i >= n_rows) continue;
          const size_t at = at0 + cg * 32 + (size_t)(4 * i) * p.N;
          if (!p.gelu_out || p.store_pre) *reinterpret_cast<float4 *>(out + at) = v[i];
          // the activated output; the pre-activation above is what the backward reads
          if (p.gelu_out)
            *reinterpret_cast<float4 *>(p.gelu_out + at) = make_float4(gelu_value(v[i].x), gelu_value(v[i].y), gelu_value(v[i].z), gelu_value(v[i].w));
        }
      }
    }
  }

  if constexpr (KS > 1) {
    // ------------------------------------------------------------ split contraction (one tile per cluster)
    // Every CTA holds the partial sums of its slice of K. When all of them are done with their operands, each sends
    // every other its columns, and each adds up its own in the order of the slices (the same bits every time).
    constexpr int OW = C::kOwned, LD = C::kPartLd;
    bool ok = true;
    if (warp >= 2) {
      ok = mbar_wait_warp(bar(C::ACC_FULL), 0, abort_flag);
      tc_fence_after_sync();
    }
    __syncthreads();
    cluster_sync();
    const int quarter = warp & 3, half = (warp - 2) >> 2, row = quarter * 32 + lane;
    if (warp >= 2 && ok) {
#pragma unroll 1
      for (int cg = 0; cg < TN / 64; ++cg) {
        const int c0 = half * (TN / 2) + cg * 32;
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + c0, r);
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          const int c = c0 + x, owner = c / OW;
          const uint32_t dst = map_to_rank(a0 + (uint32_t)(((int)part * TM + row) * LD + c - owner * OW) * 4u, (uint32_t)owner);
          asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(r[x]), "r"(r[x + 1]), "r"(r[x + 2]), "r"(r[x + 3])
                       : "memory");
        }
      }
      tc_fence_before_sync();
    }
    cluster_sync();
    int m_tile, mat, n_tile;
    decode(first_tile, &m_tile, &mat, &n_tile);
    const long long grow = (long long)m_tile * TM + row;
    if (warp >= 2 && ok && grow < (long long)p.M) {
      const float *bias = mat == 0 ? p.bias[0] : (mat == 1 ? p.bias[1] : p.bias[2]);
      float *out = mat == 0 ? p.out[0] : (mat == 1 ? p.out[1] : p.out[2]);
      const float *mine = reinterpret_cast<const float *>(smem);
#pragma unroll
      for (int x = 0; x < OW / 2; x += 4) {
        const int lc = half * (OW / 2) + x, col = n_tile * TN + (int)part * OW + lc;
        if (col >= (int)p.N) break;
        float4 v = *reinterpret_cast<const float4 *>(mine + row * LD + lc);
#pragma unroll
        for (int k = 1; k < KS; ++k) {
          const float4 a = *reinterpret_cast<const float4 *>(mine + (k * TM + row) * LD + lc);
          v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        if (bias) {
          const float4 a = __ldg(reinterpret_cast<const float4 *>(bias + col));
          v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        const size_t at = (size_t)grow * p.N + col;
        if (p.residual) {
          const float4 a = __ldg(reinterpret_cast<const float4 *>(p.residual + at));
          v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        if (!p.gelu_out || p.store_pre) *reinterpret_cast<float4 *>(out + at) = v;
        if (p.gelu_out) *reinterpret_cast<float4 *>(p.gelu_out + at) = make_float4(gelu_value(v.x), gelu_value(v.y), gelu_value(v.z), gelu_value(v.w));
      }
    }
  }

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (warp == 1 && rank == 0) {
      if (elect_one()) {  // the lane that issued the MMAs: the election is deterministic
        if (PAIR) mma_commit_pair(bar(C::DRAIN));
        else mma_commit(bar(C::DRAIN));
      }
      __syncwarp();
      for (int n = 0; n < (1 << 16) && !mbar_try_wait(bar(C::DRAIN), 0); ++n) {
      }
    }
    if (warp == 0 && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (PAIR) cluster_sync();  // neither CTA leaves while the other may still signal its barriers or use its shared memory
  if (warp == 1) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem, C::kTmemCols);
    else tmem_dealloc(tmem, C::kTmemCols);
  }
}

using LinKernel = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const LinParams);
struct LinForm {
  LinKernel kernel;
  uint32_t smem;
  int tn;
  bool pair;
  int b_rows, ks;
  float ends;  // cycles of a launch that are not products, see choose_form
};
template <int TN, bool PAIR, int KS = 1>
constexpr LinForm form(float ends) {
  using C = LinCfg<TN, PAIR, KS>;
  return {k_linear_tf32<C>, C::kSmemTotal, TN, PAIR, C::kBRows, KS, ends};
}
const LinForm kForms[] = {form<256, true>(13900.f),     form<192, true>(12700.f),     form<128, true>(10600.f),
                          form<256, false>(9700.f),     form<128, false>(8500.f),     form<64, false>(6100.f),
                          form<64, false, 2>(10000.f),  form<64, false, 4>(11200.f),  form<128, false, 4>(14600.f),
                          form<128, false, 8>(17000.f)};
constexpr int kNumForms = (int)(sizeof(kForms) / sizeof(kForms[0]));

struct DeviceInfo {
  std::once_flag once;
  int n_sm = 0;
  int slots[kNumForms] = {0};  // tiles of each form that the device works on at the same time
  bool ok = false;
};
DeviceInfo g_dev[64];

// The form with the least estimated time: waves of tiles times the cycles of one tile, and the cycles at its ends. Per 32 of K a
// tile takes its MMA cycles (2 TN) or the time its bytes take to arrive, whichever is more: 64 a cycle for one SM, about 52
// when most of them ask at once. The ends (launch, first operands, last epilogue; sending and adding the partial sums of a split
// contraction) are measured: one wave of 200 rows by 768 features at K = 768 and 3072, extrapolated to K = 0.
int choose_form(const DeviceInfo &di, uint32_t M, uint32_t K, uint32_t N, int n_mats) {
  int best = 0;
  double best_cost = 1e300;
  const uint32_t n_kb = (K + TK - 1) / TK;
  for (int i = 0; i < kNumForms; ++i) {
    const LinForm &f = kForms[i];
    const uint64_t tiles = (uint64_t)((M + (f.pair ? 2 * TM : TM) - 1) / (f.pair ? 2 * TM : TM)) * ((N + f.tn - 1) / f.tn) * n_mats;
    const uint64_t slots = di.slots[i], waves = (tiles + slots - 1) / slots;
    if (f.ks > 1 && (waves > 1 || n_kb < 4u * f.ks)) continue;
    const double bytes = kABytes + f.b_rows * TK * 4, mma = 2.0 * f.tn;
    const bool crowded = tiles * (f.pair ? 2 : f.ks) > (uint64_t)di.n_sm / 2;
    const double arrive = bytes / (crowded ? 52.0 : 64.0);
    const double cost = (double)waves * (((n_kb + f.ks - 1) / f.ks) * (arrive > mma ? arrive : mma) + 1000.0) + f.ends;
    if (cost < best_cost) {
      best_cost = cost;
      best = i;
    }
  }
  return best;
}

}  // namespace

bool tensor_linear_supported(const float *x, const float *const *w, const float *const *bias, float *const *out,
                             const float *residual, int n_mats, uint32_t M, uint32_t K, uint32_t N) {
  if (n_mats < 1 || n_mats > 3 || M == 0 || K == 0 || N == 0) return false;
  if ((K & 3u) || (N & 3u)) return false;  // row pitches must be multiples of 16 bytes
  uintptr_t bits = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual);
  for (int j = 0; j < n_mats; ++j)
    bits |= reinterpret_cast<uintptr_t>(w[j]) | reinterpret_cast<uintptr_t>(out[j]) | reinterpret_cast<uintptr_t>(bias ? bias[j] : nullptr);
  if (bits & 15u) return false;
  if ((uint64_t)M * K >= (1ull << 38) || (uint64_t)M * N >= (1ull << 38)) return false;
  return true;
}

int tensor_linear(const float *x, const float *const *w, const float *const *bias, float *const *out, const float *residual,
                  float *gelu_out, int n_mats, uint32_t M, uint32_t K, uint32_t N, cudaStream_t s) {
  if (gelu_out && (n_mats != 1 || residual || (reinterpret_cast<uintptr_t>(gelu_out) & 15u))) return DF_ERR_UNSUPPORTED;
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK || dev < 0 || dev >= 64) return DF_ERR_CUDA;
  DeviceInfo &di = g_dev[dev];
  std::call_once(di.once, [&]() {
    bool ok = cudaDeviceGetAttribute(&di.n_sm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && di.n_sm > 1;
    for (int i = 0; ok && i < kNumForms; ++i) {
      const LinForm &f = kForms[i];
      const int ctas = f.pair ? 2 : f.ks;
      ok = cudaFuncSetAttribute(f.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem) == cudaSuccess;
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = ctas;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(64 * ctas);
      cfg.blockDim = dim3(kLinThreads);
      cfg.dynamicSmemBytes = f.smem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      ok = ok && cudaOccupancyMaxActiveClusters(&di.slots[i], f.kernel, &cfg) == cudaSuccess && di.slots[i] > 0;
    }
    di.ok = ok;
  });
  if (!di.ok) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  // Reading W once is all there is to do for a few rows: up to 8 the warp-per-feature kernel is 5 to 12 times faster.
  if (M <= kLinearRowsMax && (uint64_t)N * n_mats < (1u << 28)) return rows_linear(x, w, bias, out, residual, gelu_out, n_mats, M, K, N, di.n_sm, s);
  const int form_index = choose_form(di, M, K, N, n_mats);
  const LinForm &f = kForms[form_index];
  CUtensorMap tmX, tmW[3];
  bool ok = encode_matrix_map(&tmX, x, M, K, TM, false);
  for (int j = 0; j < 3; ++j) {
    if (j < n_mats) ok = ok && encode_matrix_map(&tmW[j], w[j], N, K, f.b_rows, false);
    else tmW[j] = tmW[0];  // never loaded through
  }
  if (!ok) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  LinParams p;
  p.store_pre = (gelu_out && out[0] != gelu_out) ? 1 : 0;
  for (int j = 0; j < 3; ++j) p.bias[j] = (bias && j < n_mats) ? bias[j] : nullptr;
  p.residual = residual;
  p.M = M; p.N = N; p.K = K;
  p.n_mats = n_mats;
  p.n_tiles_per_mat = (int)((N + f.tn - 1) / f.tn);
  p.n_tiles_total = p.n_tiles_per_mat * n_mats;
  const uint32_t rows = f.pair ? 2 * TM : TM;
  p.tiles = (long long)((M + rows - 1) / rows) * p.n_tiles_total;
  p.status = device_status_ptr();
  for (int j = 0; j < 3; ++j) p.out[j] = out[j < n_mats ? j : 0];
  p.gelu_out = gelu_out;
  const int ctas = f.pair ? 2 : f.ks;
  const long long slots = di.slots[form_index], grid = (p.tiles < slots ? p.tiles : slots) * ctas;
  launch_clusters(f.kernel, ctas > 1 ? ctas : 0, dim3((unsigned)grid), dim3(kLinThreads), f.smem, s, tmX, tmW[0], tmW[1], tmW[2], p);
  note_launch();
  return check_cuda(cudaGetLastError());
}

}  // namespace df

// attn_bwd_sm100.cu — fused causal attention backward for B200 (sm_100a), fp32 API, TF32 MMA.
//
// Replaces the arithmetic of kernel_mha_bwd_all_heads
// (darkforest-cuda/kernels/attention_fused.cu:390-516) from saved logsumexp and delta:
//   P = exp(scale*QK^T - lse)   dP = dO V^T   dS = P o (dP - delta)
//   dV = P^T dO                 dK = scale * dS^T Q        dQ = scale * dS K
// with no S x S scratch, no atomics (bit-reproducible) and no memsets: two kernels (a whole-sequence call runs
// dQ first, which also forms delta, then dK/dV), each recomputing P tile by tile on the tensor cores.
//
// dK/dV kernel: a CTA owns 128 keys (TMEM lanes = keys) and walks the 128-query tiles that can see them.  K and V lie in tensor memory from an item's
//   second step on: S^T = K Q^T and dP^T = V dO^T are TS MMAs over K-major tiles of Q and dO in rings of two (SS in the first step, so that nothing waits
//   for the move); dV += P^T dO and dK += dS^T Q are TS MMAs whose B operand (dO, Q as [query, d]) is MN-major.  A 32-bit MN-major operand needs a
//   different shared-memory swizzle (32-byte atoms) than a K-major one, so Q and dO tiles are fetched twice by TMA, once per layout.  The queries'
//   statistics come in as one more K-step of the first two products: S^T - lse / scale, dP^T - delta.  A step's queries are two halves with barriers of
//   their own: warps 0-3 turn one half's S^T into P^T and dP^T into dS^T in place in TMEM, warps 4-7 the other's, and neither group waits for the other.
//   What bounds it: the tensor pipe, with 2.18 K of the 2.50 K cycles that a step takes at 1 x 12 x 16384 (87 % busy); in short sequences the ends of items
//   (8 x 12 x 1024: 54 %). When the compute warps read the statistics from shared memory (a quarter of their time) and went in step it was 3.4 K.
//   Backward on B200, us, before / now: 8 x 12 x 1024 causal 115 / 109, 1 x 12 x 8192 669 / 577, 2 x 16 x 2000 all keys 228 / 203, 1 x 12 x 512 18.0 / 17.4.
// dQ kernel: a CTA owns 128 queries (lanes = queries) and walks the key tiles they can see:
//   S = Q K^T, dP = dO V^T (SS), dS in TMEM, dQ += dS K (TS, K tile MN-major: K is fetched twice).
//   2.55 K cycles a step at 1 x 12 x 4096 (2.24 K at 16384) where the tensor pipe needs 1.54 K: the latency of the issuing and the compute warps' loops
//   (at 4096 tensor pipe 58 %, exponentials 39 %, issue slots 33 % busy). The dK/dV kernel's halves and operands in tensor memory gave it 2 % at 8192 rows and cost 1-2 % at 8 x 1024 and 512.
// One-tile kernel (at the end): up to 128 queries and keys, both halves in one launch.
// MMA issue: tcgen05 MMAs of one thread execute in issue order, which is what lets single shared-memory stages
// suffice. The dQ kernel has one MMA warp that interleaves the phases of consecutive tiles (.., S_{j+1}, dP_{j+1},
// dQ_j, ..: dP has two buffers in tensor memory and runs a step ahead of dQ); the dK/dV kernel has one MMA warp per
// product chain (dV_i, S_{i+1} and dK_i, dP_{i+1}, each half by half: they share nothing).
// An MMA role is run by all 32 lanes of its warp, warp-uniformly, with elect.sync around the tensor instructions.
// Both kernels run a CTA's tiles as one uninterrupted pipeline, heaviest tiles first, and hand finished tiles to the copy engine
// through shared memory. The dQ kernel deals its tiles out in advance; dK/dV CTAs take over tiles whose CTA has not started, and in a
// whole-sequence call they start on SMs that the dQ kernel has left, as soon as every row sum is written (pdl_trigger). Measured on
// B200 against two static kernels in turn, us, H = 12: 1 x 1024 37.3 -> 34.4, 1 x 4096 174 -> 167,
// 1 x 8192 709 -> 690, 8 x 1024 117.1 -> 116.3 (causal; all keys: -2..+2 %). Tiles that become free at different times land on barriers of their own (K and V in the dK/dV
// kernel, Q and dO/O in the dQ kernel), so that an item's last accumulating product never queues behind the wait for
// a tile of the next item that it does not need.
//
// Inputs are rounded to TF32 by the TFLOAT32 tensor maps (nearest even); P and dS are rounded
// with cvt.rna before they are written back to TMEM. Every wait is bounded (see mbar_wait) and,
// in roles of whole warps, decided by the warp together.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {
namespace {

using namespace ptx;

constexpr int BT = 128;  // tile edge: keys per CTA / queries per step (and vice versa)
constexpr int HD = 64;
constexpr int kBwdThreads = 352;  // dQ kernel: warps 0-7 compute, 8-9 TMA producers, 10 MMA issuer
// dK/dV kernel: warps 0-7 compute (two groups of four, each with half of a step's queries), 8-9 TMA producers, 10-11 MMA issuers. With sixteen compute
// warps (96 registers each, some spilled) it took 362 us where eight take 348 (1 x 12 x 8192, causal).
constexpr int kKvThreads = 384;
constexpr uint32_t kSlab = 128 * 128;
constexpr uint32_t kTile = 2 * kSlab;
constexpr uint32_t kTmemCols = 512;

// Optional phase trace (build with -DDF_ATTN_TRACE): (event id, SM clock) pairs recorded by lane 0 of compute warp 0
// (slot 1) of CTA 0 of the dK/dV kernel, or with -DDF_ATTN_TRACE_DQ of the dQ kernel, there by its MMA warp as well
// (slot 0; in the dK/dV kernel that slot has the kernel's start alone); the launcher prints them when
// DF_ATTN_TRACE_DUMP is set. Compiled out by default.
#ifdef DF_ATTN_TRACE
__device__ unsigned long long g_bwd_trace[2 * 1024];
#define DF_BTRACE(slot, id)                                           \
  do {                                                                \
    if (trace_on && tr_n < 511) {                                     \
      g_bwd_trace[(slot)*1024 + 2 * tr_n] = (id);                     \
      g_bwd_trace[(slot)*1024 + 2 * tr_n + 1] = clock64();            \
      ++tr_n;                                                         \
    }                                                                 \
  } while (0)
#else
#define DF_BTRACE(slot, id) do { } while (0)
#endif

struct BwdParams {
  const float *lse;
  const float *delta;
  float *delta_out;  // dQ kernel with fused row sums: delta = rowsum(dO o O) is computed there and written here
  float *dq, *dk, *dv;
  uint32_t B, H, Sq, Sk;
  float scale, scale_log2;
  float inv_scale, kv_scale_log2;  // dK/dV: one over the scale, and log2 e times the number that inv_scale is one over
  int causal;
  long long shift;
  uint32_t zero_tiles;  // dK/dV: key tiles (times heads) beyond the items, which no query sees
  int early;            // dQ lets the dependent launch begin once its row sums are written; dK/dV then waits for dQ at its end
  unsigned int *status;
};

// MMA batches. The descriptor words of every K-step of a tile are computed once per kernel (TileK / TileMN); a batch
// is then issued by ONE elected lane as nothing but tcgen05.mma instructions (and the commits that follow it): the
// issuing warp shares its scheduler with busy compute warps, and every other instruction between two MMAs costs the
// tensor pipe time (see mma_tf32_ts_lohi). Shared memory ends below 256 KB, so the 14-bit address field never carries.
struct TileK {   // K-major 128 x 64 fp32 tile of two 128-byte slabs: 8 K-steps
  uint32_t lo[HD / 8], hi;
};
struct TileMN {  // MN-major [128 rows (K), 64 dims (N)] tile: 16 K-steps
  uint32_t lo[BT / 8], hi;
};
__device__ __forceinline__ TileK tile_k(uint32_t tile_smem) {
  TileK t;
  const uint64_t d = make_smem_desc(tile_smem, 16, 1024, kSwz128);
  t.hi = (uint32_t)(d >> 32);
#pragma unroll
  for (int kk = 0; kk < HD / 8; ++kk) t.lo[kk] = (uint32_t)d + (((kk >> 2) * kSlab + (kk & 3) * 32) >> 4);
  return t;
}
__device__ __forceinline__ TileMN tile_mn(uint32_t tile_smem) {
  TileMN t;
  const uint64_t d = make_smem_desc(tile_smem, kSlab, 512, kSwz128B32);
  t.hi = (uint32_t)(d >> 32);
#pragma unroll
  for (int kk = 0; kk < BT / 8; ++kk) t.lo[kk] = (uint32_t)d + ((kk * 1024) >> 4);
  return t;
}
// To be called by the elected lane only.
// 128x64x64 TS MMA, 8 K-steps: A = 64 TMEM columns, B = 64 rows of a K-major tile of a ring (off: their descriptor offset).
__device__ __forceinline__ void batch_ts_scores(uint32_t d_tmem, uint32_t a_tmem, const TileK &b, uint32_t off, uint32_t idesc) {
#pragma unroll
  for (int kk = 0; kk < HD / 8; ++kk) mma_tf32_ts_lohi(d_tmem, a_tmem + kk * 8, b.lo[kk] + off, b.hi, idesc, kk > 0 ? 1u : 0u);
}
// The same with A, a whole tile, in shared memory too: what an item's first step takes, before its K (V) is in tensor memory.
__device__ __forceinline__ void batch_ss_scores(uint32_t d_tmem, const TileK &t, uint32_t a_off, uint32_t b_off, uint32_t idesc) {
#pragma unroll
  for (int kk = 0; kk < HD / 8; ++kk) mma_tf32_ss_lohi(d_tmem, t.lo[kk] + a_off, t.hi, t.lo[kk] + b_off, t.hi, idesc, kk > 0 ? 1u : 0u);
}
// 8 K-steps from FROM on (half) of a 128x64x128 TS MMA: A = 128 TMEM columns, B = MN-major tile.
template <int FROM>
__device__ __forceinline__ void batch_ts_128x64(uint32_t d_tmem, uint32_t a_tmem, const TileMN &b, uint32_t idesc, bool accumulate) {
  mma_tf32_ts_lohi(d_tmem, a_tmem + FROM * 8, b.lo[FROM], b.hi, idesc, accumulate ? 1u : 0u);
#pragma unroll
  for (int kk = FROM + 1; kk < FROM + BT / 16; ++kk) mma_tf32_ts_lohi_acc(d_tmem, a_tmem + kk * 8, b.lo[kk], b.hi, idesc);
}
// The dQ kernel keeps the other form - all lanes call these, one lane is elected per MMA, the descriptor is base +
// constant: with pure-MMA batches it measured 1.5 % faster at S = 1024 but 4 % slower at S = 16384 (the dK/dV kernel
// gained 1-3 % at both).
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t tile_smem) { return make_smem_desc(tile_smem, 16, 1024, kSwz128); }
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t tile_smem) { return make_smem_desc(tile_smem, kSlab, 512, kSwz128B32); }
__device__ __forceinline__ void issue_ss_128x128(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc) {
#pragma unroll
  for (int kk = 0; kk < HD / 8; ++kk) {
    const uint64_t off = (uint64_t)(((kk >> 2) * kSlab + (kk & 3) * 32) >> 4);
    if (elect_one()) mma_tf32_ss(d_tmem, a_desc + off, b_desc + off, idesc, kk > 0);
  }
}
__device__ __forceinline__ void issue_ts_128x64(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                                bool accumulate) {
#pragma unroll
  for (int kk = 0; kk < BT / 8; ++kk)
    if (elect_one()) mma_tf32_ts(d_tmem, a_tmem + kk * 8, b_desc + (uint64_t)((kk * 1024) >> 4), idesc, (accumulate || kk > 0) ? 1u : 0u);
}
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap *m, uint32_t bar, int h, int row0, int b) {
  mbar_arrive_expect_tx(bar, kTile);
  tma_load_4d(dst, m, bar, 0, h, row0, b);
  tma_load_4d(dst + kSlab, m, bar, 32, h, row0, b);
}

__device__ __forceinline__ void store_cluster(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// SPLIT kernels: 16 accumulator columns of a thread's row (dims d0 .. d0 + 15) into the other CTA's staging tile, which has the layout of the store's
// tensor map (slabs of 32 dims, 16-byte chunk c of row r at c ^ (r % 8)), and there, in place, the sum with the finishing CTA's own columns.
__device__ __forceinline__ void send_cols(uint32_t peer_tile, int row, int d0, uint32_t taddr) {
  uint32_t rr[16];
  tmem_ld16(taddr + d0, rr);
  tmem_wait_ld();
#pragma unroll
  for (int x = 0; x < 4; ++x)
    store_cluster(peer_tile + (uint32_t)(d0 >> 5) * kSlab + row * 128 + (uint32_t)((((d0 & 31) >> 2) + x) ^ (row & 7)) * 16,
                  make_float4(__uint_as_float(rr[4 * x]), __uint_as_float(rr[4 * x + 1]), __uint_as_float(rr[4 * x + 2]), __uint_as_float(rr[4 * x + 3])));
}
__device__ __forceinline__ void finish_cols(uint8_t *tile, int row, int d0, uint32_t taddr, bool own, bool other, float mul) {
  uint32_t rr[16];
  tmem_ld16(taddr + d0, rr);
  tmem_wait_ld();
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    float4 *at = reinterpret_cast<float4 *>(tile + (d0 >> 5) * kSlab + row * 128 + ((((d0 & 31) >> 2) + x) ^ (row & 7)) * 16);
    float4 a = make_float4(__uint_as_float(rr[4 * x]), __uint_as_float(rr[4 * x + 1]), __uint_as_float(rr[4 * x + 2]), __uint_as_float(rr[4 * x + 3]));
    if (!own) a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (other) {
      const float4 b = *at;
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    *at = make_float4(a.x * mul, a.y * mul, a.z * mul, a.w * mul);
  }
}

// =========================================================================================
// Work distribution shared by both kernels
// =========================================================================================
// A work item is one 128-row tile of one head; items are numbered heaviest first ((batch, head) fastest). The dQ kernel's grid has at
// most one CTA per SM and deals them out in rounds, odd rounds in reverse CTA order, which balances the causal triangle as well as a
// greedy longest-first assignment; the dK/dV kernel has a CTA per item and claims further ones. A CTA runs its items
// as ONE pipeline: barrier phases are counted over all steps of all items, so the copies and the
// first two MMAs of the next item are in flight while the last products of the current item
// finish and its result tile is stored.
__device__ __forceinline__ int item_of_round(int r, int n_items) {
  return (int)snake_item(r, (int)gridDim.x, (int)blockIdx.x, n_items);
}

// =========================================================================================
// dK / dV
// =========================================================================================
constexpr int kClaims = 8;  // answers to item claims kept in shared memory (the roles are at most three items apart)

namespace kv {
// *_FULL / *_EMPTY of the Q and dO rings: + slot; of the MN-major tiles: + half of the rows; S_FULL .. DS_FULL: + half of the step's queries
enum Bar { QK_FULL = 0, QK_EMPTY = 2, GK_FULL = 4, GK_EMPTY = 6, QM_FULL = 8, QM_EMPTY = 10, GM_FULL = 12, GM_EMPTY = 14,
           S_FULL = 16, P_FULL = 18, DP_FULL = 20, DS_FULL = 22, K_READY = 24, V_READY, K_FREE, V_FREE, FIRST, ACC_FULL, EPI_FULL, DRAIN,
           CLAIM, NUM = CLAIM + kClaims };  // CLAIM + answer
constexpr uint32_t kOnes = 6 * kTile;              // A of the statistics' K-step: 128 rows of (1, 1, 1, 0, 0, 0, 0, 0)
constexpr uint32_t kStats = kOnes + BT * 32;       // B: [lse, delta][half of the queries][64 rows of 8]
constexpr uint32_t kStatTile = BT / 2 * 32;
constexpr uint32_t kAnswers = kStats + 4 * kStatTile;
constexpr uint32_t kBars = kAnswers + kClaims * 16;
constexpr uint32_t kSmemTotal = kBars + 336 + 1024;
static_assert(NUM * 8 <= 320, "barriers");

// One work item: 128 keys of one head and the query tiles that can see them.
struct Item {
  uint32_t idx, b, h;
  long long k0;       // first key row
  long long i_begin;  // first query tile
  int n_it;           // number of query tiles (at least 1 for an item)
};
__device__ __forceinline__ Item decode(const BwdParams &p, int idx) {
  Item it;
  const uint32_t n_bh = p.B * p.H, bh = (uint32_t)idx % n_bh;
  it.idx = (uint32_t)idx;
  it.b = bh / p.H;
  it.h = bh % p.H;
  it.k0 = (long long)((uint32_t)idx / n_bh) * BT;  // key tile 0 sees the most queries: heaviest first
  long long q_first = p.causal ? it.k0 - p.shift : 0;
  if (q_first < 0) q_first = 0;
  it.i_begin = q_first / BT;
  const long long n_qt = ((long long)p.Sq + BT - 1) / BT;
  it.n_it = (int)(n_qt - it.i_begin);
  return it;
}
}  // namespace kv

// SPLIT: a cluster of two CTAs shares an item. Each takes every other query tile; at the end rank 0 finishes dV and rank 1 dK, each
// from its own accumulator and the other's, which comes through distributed shared memory. For problems whose items leave SMs
// without work or are long against an SM's share (split_backward).
template <bool SPLIT>
__global__ void __launch_bounds__(kKvThreads, 1)
k_attn_bwd_dkdv_tf32_d64(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                         const __grid_constant__ CUtensorMap tmQk, const __grid_constant__ CUtensorMap tmGk,
                         const __grid_constant__ CUtensorMap tmQm, const __grid_constant__ CUtensorMap tmGm,
                         const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV,
                         const BwdParams p) {
  using namespace kv;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t aQk = smem_u32(smem), aGk = aQk + 2 * kTile, aQm = aQk + 4 * kTile, aGm = aQk + 5 * kTile;  // rings of two; MN-major tiles
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + kBars + 320);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + kBars + 324);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kCW = 8;               // compute warps
  constexpr int kArrivals = kCW * 32;  // every compute thread arrives (one arrival per warp measured the same)
  constexpr int CPT = BT / 2;          // query columns per compute thread
  constexpr int NCH = CPT / 32;        // 32-column chunks per compute thread
  constexpr int kWarpLoadK = kCW, kWarpLoadM = kCW + 1, kWarpMma = kCW + 2, kWarpMma2 = kCW + 3, kWarpCompute0 = 0;
  const size_t dm = (size_t)p.H * HD;
  constexpr int ST = SPLIT ? 2 : 1;  // query tiles from one step to the next
  const uint32_t rank = SPLIT ? cluster_rank() : 0u;
#ifdef DF_ATTN_TRACE
#ifdef DF_ATTN_TRACE_DQ
  const bool trace_on = false;
#else
  const bool trace_on = blockIdx.x == 0 && lane == 0 && (warp == kWarpMma || warp == kWarpCompute0);
#endif
  int tr_n = 0;
#endif
  DF_BTRACE(warp == kWarpMma ? 0 : 1, 1);

  auto bar = [&](int id) { return smem_u32(&bars[id]); };
  // Items: blockIdx.x first, then those of CTAs that have not started (claimed by the first producer). take(k) is item k of this
  // CTA; false when there is none (or a wait gave up).
  auto take = [&](uint32_t k, Item *out) -> bool {
    uint32_t idx = blockIdx.x / ST;
    if (SPLIT && k > 0) return false;
    if (!SPLIT && k > 0) {
      const int c = (int)((k - 1) % kClaims);
      if (!mbar_wait(bar(CLAIM + c), ((k - 1) / kClaims) & 1, abort_flag)) return false;
      idx = claim_result(smem_u32(smem) + kAnswers + 16 * c);
      if (idx == ~0u) return false;
    }
    *out = decode(p, (int)idx);
    if (SPLIT) {
      out->i_begin += rank;
      out->n_it = (out->n_it + 1 - (int)rank) / 2;
    }
    return !SPLIT || out->n_it > 0;
  };
  if (warp == kWarpLoadK) {
    for (int i = lane; i < NUM; i += 32)
      mbar_init(bar(i), (i == K_READY || i == V_READY || i == FIRST || i == EPI_FULL) ? kArrivals : (i == P_FULL || i == P_FULL + 1 || i == DS_FULL || i == DS_FULL + 1) ? kArrivals / 2 : ((i == ACC_FULL || i == DRAIN) ? 2 : 1));
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    Item first;
    if (lane == 0 && take(0, &first)) {  // the first tiles are under way while the others set up
      if (!p.early) pdl_wait();
      load_tile(aQk, &tmK, bar(QK_FULL), (int)first.h, (int)first.k0, (int)first.b);
      load_tile(aQk + kTile, &tmQk, bar(QK_FULL + 1), (int)first.h, (int)(first.i_begin * BT), (int)first.b);
      load_tile(aGk, &tmV, bar(GK_FULL), (int)first.h, (int)first.k0, (int)first.b);
      load_tile(aGk + kTile, &tmGk, bar(GK_FULL + 1), (int)first.h, (int)(first.i_begin * BT), (int)first.b);
    }
  }
  if (warp == kWarpMma) {
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  // 16-byte units of the statistics' operands, unswizzled: chunk c (of two) of row r at (r / 8) * 256 + c * 128 + (r % 8) * 16
  if (warp < kCW) {
    for (uint32_t u = threadIdx.x; u < (BT * 32 + 4 * kStatTile) / 16; u += kCW * 32)
      *reinterpret_cast<float4 *>(smem + kOnes + u * 16) = u < BT * 2 && !(u & 8) ? make_float4(1.0f, 1.0f, 1.0f, 0.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    fence_proxy_async_smem();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  const uint32_t tK = tmem, tV = tmem + 64, tS = tmem + 128, tDP = tmem + 256, tDV = tmem + 384, tDK = tmem + 448;
  if (!p.early) pdl_wait();  // everything above touched only this CTA's shared and tensor memory

  auto take_warp = [&](uint32_t k, Item *out) -> bool { return __all_sync(0xffffffffu, take(k, out)) != 0; };

  // Counters every role keeps for itself: g = steps (query tiles) done over all items, n = items
  // done. A barrier used once per step is in phase g & 1, one used once per item in phase n & 1.
  if (warp == kWarpLoadK) {
    // ---------------------------------------------- producer: rings of K-major tiles: an item's K (V), then Q (dO) of every step
    if (lane == 0) {
      Item cur;
      uint32_t n = 0, r = 0;  // r: tiles of either ring so far
      bool ok = true;
      auto ring = [&](const CUtensorMap *mq, const CUtensorMap *mg, int row) {  // the next tile of both
        const uint32_t slot = r & 1;
        if (r > 1 && !mbar_wait(bar(QK_EMPTY + slot), ((r >> 1) - 1) & 1, abort_flag)) return false;
        if (r > 1) load_tile(aQk + slot * kTile, mq, bar(QK_FULL + slot), (int)cur.h, row, (int)cur.b);  // the first two: during set-up
        if (r > 1 && !mbar_wait(bar(GK_EMPTY + slot), ((r >> 1) - 1) & 1, abort_flag)) return false;
        if (r > 1) load_tile(aGk + slot * kTile, mg, bar(GK_FULL + slot), (int)cur.h, row, (int)cur.b);
        ++r;
        return true;
      };
      for (; ok && take(n, &cur); ++n) {
        ok = ring(&tmK, &tmV, (int)cur.k0);
        for (int it = 0; ok && it < cur.n_it; ++it) {
          if (!SPLIT && it == (cur.n_it > 1 ? cur.n_it - 2 : 0)) {  // ask for the next item: its K and V follow this item's last tiles
            const int c = (int)(n % kClaims);
            fence_proxy_async_smem();
            mbar_arrive_expect_tx(bar(CLAIM + c), 16);
            claim_request(smem_u32(smem) + kAnswers + 16 * c, bar(CLAIM + c));
          }
          ok = ring(&tmQk, &tmGk, (int)((cur.i_begin + it * ST) * BT));
        }
      }
    }
  } else if (warp == kWarpLoadM) {
    // ---------------------------------------------- producer: MN-major dO and Q tiles per step in halves, result stores per item
    if (lane == 0) {
      Item cur;
      uint32_t g = 0, n = 0;
      for (; take(n, &cur); ++n) {
        bool ok = true;
        for (int it = 0; ok && it < cur.n_it; ++it, ++g) {
          const int q0 = (int)((cur.i_begin + it * ST) * BT);
          // A tile has one buffer. Its halves are released by commits of their own in the middle and at the end of the product that reads them, so
          // the next step's first half is on its way while this step's second one is still read.
          auto half = [&](int full, int empty, uint32_t dst, const CUtensorMap *m, int x) {
            if (g > 0 && !mbar_wait(bar(empty + x), (g - 1) & 1, abort_flag)) return false;
            mbar_arrive_expect_tx(bar(full + x), kTile / 2);
            for (int sl = 0; sl < 2; ++sl) tma_load_4d(dst + sl * kSlab + x * (kSlab / 2), m, bar(full + x), 32 * sl, (int)cur.h, q0 + x * (BT / 2), (int)cur.b);
            return true;
          };
          ok = half(GM_FULL, GM_EMPTY, aGm, &tmGm, 0) && half(GM_FULL, GM_EMPTY, aGm, &tmGm, 1) && half(QM_FULL, QM_EMPTY, aQm, &tmQm, 0) &&
               half(QM_FULL, QM_EMPTY, aQm, &tmQm, 1);
        }
        if (SPLIT) break;
        // The compute warps stage the item's dV and dK tiles in these two buffers; this thread
        // hands them to the copy engine (key rows beyond Sk are dropped) and may refill the
        // buffers for the next item once the store has read them.
        if (!ok || !mbar_wait(bar(EPI_FULL), n & 1, abort_flag)) break;
        tma_store_4d(&tmDV, aGm, 0, (int)cur.h, (int)cur.k0, (int)cur.b);
        tma_store_4d(&tmDV, aGm + kSlab, 32, (int)cur.h, (int)cur.k0, (int)cur.b);
        tma_store_4d(&tmDK, aQm, 0, (int)cur.h, (int)cur.k0, (int)cur.b);
        tma_store_4d(&tmDK, aQm + kSlab, 32, (int)cur.h, (int)cur.k0, (int)cur.b);
        tma_store_commit();
        tma_store_wait_read_all();
      }
    }
  } else if (warp == kWarpMma || warp == kWarpMma2) {
    // ---------------------------------------------- MMA issuers
    // The step's four products form two chains that share neither tensor memory nor operand buffers nor barriers:
    //   warp kWarpMma :  .., dV_g (needs P_g), S_{g+1} (overwrites P^T_g after dV_g has read it), ..
    //   warp kWarpMma2:  .., dK_g (needs dS_g), dP_{g+1} (overwrites dS^T_g after dK_g has read it), ..
    // Each chain has its own warp: MMAs of one thread execute in issue order, which is all a chain needs, and while one warp sits between two batches
    // (poll, fence, the first MMA's start-up) the other's MMAs keep the tensor pipe busy.
    // The whole warp runs its role; only the MMA and commit instructions are issued by one elected lane.
    const bool s_chain = warp == kWarpMma;
    const uint32_t idesc_st = make_idesc(kFmtTF32, BT, BT / 2, 0, 0), idesc_ts = make_idesc(kFmtTF32, BT, HD, 0, 1);
    const uint32_t tA = s_chain ? tK : tV, tX = s_chain ? tS : tDP, tR = s_chain ? tDV : tDK;
    const int full = s_chain ? QK_FULL : GK_FULL, empty = s_chain ? QK_EMPTY : GK_EMPTY, ready = s_chain ? P_FULL : DS_FULL;
    const int m_full = s_chain ? GM_FULL : QM_FULL, m_empty = s_chain ? GM_EMPTY : QM_EMPTY;
    const TileK dB = tile_k(s_chain ? aQk : aGk);
    const uint64_t dOnes = make_smem_desc(aQk + kOnes, 128, 256, kSwzNone), dStat = make_smem_desc(aQk + kStats + (s_chain ? 0 : 2 * kStatTile), 128, 256, kSwzNone);
    const TileMN dM = tile_mn(s_chain ? aGm : aQm);
    Item cur;
    uint32_t g = 0, r = 0;
    bool ok = true, staged = false;
    // S^T - lse / scale = K Q^T + 1 (-lse / scale), or dP^T - delta, for half h of the queries of the ring's next tile: the queries' statistics, cut in
    // three TF32 parts, come in as one more K-step, so that the compute warps do not read them (they took a quarter of the warps' time). It is the last
    // one: the accumulator truncates, so with the statistics first eight sums lose bits of a number as large as lse / scale, with them last only the
    // difference is rounded. 2 x 12 x 1000, |lse| 291, mean relative error of dV against float64: first 6.5e-6, last 5e-7, subtracted in fp32 5e-7.
    // `frees`: the item's last, from tensor memory.
    auto issue_first = [&](int h, bool from_smem, bool frees) -> bool {
      const uint32_t slot = r & 1, b_off = slot * (kTile >> 4) + h * (kSlab / 2 >> 4);
      if (h == 0) {
        if (!mbar_wait_warp(bar(full + slot), (r >> 1) & 1, abort_flag)) return false;
        tc_fence_after_sync();
      }
      if (from_smem) {
        if (elect_one()) batch_ss_scores(tX + h * (BT / 2), dB, (slot ^ 1) * (kTile >> 4), b_off, idesc_st);
        __syncwarp();
        if (!staged) {  // the CTA's first statistics come out of global memory while its first tiles do
          if (!mbar_wait_warp(bar(FIRST), 0, abort_flag)) return false;
          tc_fence_after_sync();
          staged = true;
        }
      }
      if (elect_one()) {
        if (!from_smem) batch_ts_scores(tX + h * (BT / 2), tA, dB, b_off, idesc_st);
        mma_tf32_ss(tX + h * (BT / 2), dOnes, dStat + h * (kStatTile >> 4), idesc_st, 1u);
        mma_commit(bar((s_chain ? S_FULL : DP_FULL) + h));
        if (h == 1) mma_commit(bar(empty + slot));
        if (h == 1 && frees) mma_commit(bar(s_chain ? K_FREE : V_FREE));
      }
      __syncwarp();
      if (h == 1) ++r;
      return true;
    };
    uint32_t moved = 0;  // items whose K (V) went to tensor memory
    for (uint32_t n = 0; ok && take_warp(n, &cur); ++n) {
      const uint32_t slot = r & 1;  // K's, or V's
      if (!mbar_wait_warp(bar(full + slot), (r >> 1) & 1, abort_flag)) break;
      ++r;
      ok = issue_first(0, true, false) && issue_first(1, true, false);
      if (ok && cur.n_it > 1) {  // from the second step on K (V) is read from tensor memory
        ok = mbar_wait_warp(bar(s_chain ? K_READY : V_READY), moved & 1, abort_flag);
        ++moved;
      }
      commit_elected(bar(empty + slot));  // its ring slot is free once the first step's products are done
      for (int it = 0; ok && it < cur.n_it; ++it, ++g) {
        const bool last = it + 1 == cur.n_it;
        const uint32_t ph = g & 1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t m = mbar_test3_warp(bar(ready + h), ph, bar(m_full + h), ph, bar(m_full + h), ph);
          if ((!(m & 1u) && !mbar_wait_warp(bar(ready + h), ph, abort_flag)) || (!(m & 2u) && !mbar_wait_warp(bar(m_full + h), ph, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          if (elect_one()) {  // dV += P^T dO, or dK += dS^T Q, over this half of the queries
            if (h == 0) batch_ts_128x64<0>(tR, tX, dM, idesc_ts, it > 0);
            else batch_ts_128x64<BT / 16>(tR, tX, dM, idesc_ts, true);
            mma_commit(bar(m_empty + h));
            if (last && h == 1) mma_commit(bar(ACC_FULL));  // the second of its two arrivals completes the item's accumulators
          }
          __syncwarp();
          if (!last && !issue_first(h, false, it + 2 == cur.n_it)) {
            ok = false;
            break;
          }
        }
      }
    }
  } else {
    // ---------------------------------------------- compute warps: lanes = keys, columns = queries
    const int quarter = warp & 3, sub = (warp - kWarpCompute0) >> 2;
    const int row = quarter * 32 + lane;
    const int stat_q = sub * 64 + (row & 63);  // of the group's 64 queries: half of the threads fetch lse, the others delta
    const bool stat_lse = row < 64;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int col0 = sub * CPT;
    // result tiles: the first half of the column groups hands over dV, the second half scale * dK, each thread
    // kOutCols dims of its key row starting at out0
    constexpr int kOutCols = HD, out0 = 0;
    const bool is_dk = sub != 0;
    // keys that no query sees (only with a causal shift or more keys than queries): dK = dV = 0. Item idx writes those tiles
    // beyond the items whose number is idx modulo the number of items.
    auto zero_unseen = [&](const Item &im) {
      const uint32_t items = gridDim.x;
      for (uint32_t z_idx = im.idx; z_idx < p.zero_tiles; z_idx += items) {
        const Item z = decode(p, (int)(items + z_idx));
        const long long kj = z.k0 + row;
        if (kj < (long long)p.Sk) {
          float4 *dst = reinterpret_cast<float4 *>((is_dk ? p.dk : p.dv) + ((size_t)z.b * p.Sk + (size_t)kj) * dm + z.h * HD + out0);
#pragma unroll
          for (int x = 0; x < kOutCols / 4; ++x) dst[x] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    };
    // row statistics of a query tile: threads 0-127 fetch lse, 128-255 fetch delta (the others none)
    // The value comes back RAW: nothing is computed from it here, so the thread does not stall on the load; it is
    // turned into what the products use (`stage`) only when it is written to shared memory, a phase or two later.
    auto fetch_stat = [&](const Item &im, int it) -> float {
      const long long q = (im.i_begin + it * ST) * BT + stat_q;
      if (q >= (long long)p.Sq) return stat_lse ? -INFINITY : 0.0f;
      const size_t s_base = ((size_t)im.b * p.H + im.h) * p.Sq;
      return __ldcg((stat_lse ? p.lse : p.delta) + s_base + q);  // delta may still be being written when this kernel starts: not cached
    };
    // What the statistics' K-step adds, -lse / scale (-inf for a row without visible keys: P = 0) or -delta, in three TF32 parts
    auto stage = [&](float raw) {
      const float x = stat_lse ? -raw * p.inv_scale : -raw;
      const float hi = stat_lse && fabsf(raw) == INFINITY ? -INFINITY : __uint_as_float(cvt_rna_tf32(x));
      const float rest = fabsf(hi) == INFINITY ? 0.0f : x - hi, mid = __uint_as_float(cvt_rna_tf32(rest));
      const uint32_t q = (uint32_t)row & 63;
      *reinterpret_cast<float4 *>(smem + kStats + ((stat_lse ? 0 : 2) + sub) * kStatTile + (q >> 3) * 256 + (q & 7) * 16) = make_float4(hi, mid, rest - mid, 0.0f);
      fence_proxy_async_smem();
    };
    // Hands the finished accumulators of the CTA's item number `nd` to the second producer thread: half of the column
    // groups hand over dV, the other half scale * dK. Every MMA of the item has finished by then, so
    // the MN-major dO buffer stages dV and the MN-major Q buffer dK, in the 128-byte-swizzled
    // slab layout of the store's tensor map (16-byte chunk c of row r at c ^ (r % 8)).
    auto hand_over = [&](uint32_t nd) -> bool {
      if (!mbar_wait_warp(bar(ACC_FULL), nd & 1, abort_flag)) return false;
      DF_BTRACE(1, 60);
      tc_fence_after_sync();
      const float mul = is_dk ? p.scale : 1.0f;
      uint8_t *stage = smem + (is_dk ? 4 : 5) * kTile + row * 128;
#pragma unroll 1
      for (int c = out0 / 32; c < (out0 + kOutCols) / 32; ++c) {
        uint32_t rr[32];
        tmem_ld32((is_dk ? tDK : tDV) + lane_base + c * 32, rr);
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < 8; ++x)
          *reinterpret_cast<float4 *>(stage + c * kSlab + ((x ^ (row & 7)) << 4)) =
              make_float4(__uint_as_float(rr[4 * x]) * mul, __uint_as_float(rr[4 * x + 1]) * mul,
                          __uint_as_float(rr[4 * x + 2]) * mul, __uint_as_float(rr[4 * x + 3]) * mul);
      }
      tc_fence_before_sync();  // the next item's first dV/dK overwrite the accumulators just read
      fence_proxy_async_smem();
      mbar_arrive(bar(EPI_FULL));
      DF_BTRACE(1, 61);
      return true;
    };
    // K (or V) of the CTA's next item from its ring (tile number r there) into tensor memory: as operand A from there it costs the shared-memory port
    // nothing, and the 64 KB of the two hold a second tile of Q and dO. Items of one step go without. `moved`: items before it that did not.
    auto load_resident = [&](bool v, uint32_t r, uint32_t moved) -> bool {
      if (moved > 0 && !mbar_wait_warp(bar(v ? V_FREE : K_FREE), (moved - 1) & 1, abort_flag)) return false;
      const uint32_t slot = r & 1;
      if (!mbar_wait_warp(bar((v ? GK_FULL : QK_FULL) + slot), (r >> 1) & 1, abort_flag)) return false;
      tc_fence_after_sync();
      const uint8_t *src = smem + ((v ? 2 : 0) + slot) * kTile + sub * kSlab + row * 128;
#pragma unroll 1
      for (int c = 0; c < 8; c += 4) {
        uint32_t rr[16];
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const uint4 t = *reinterpret_cast<const uint4 *>(src + (((c + x) ^ (row & 7)) << 4));
          rr[4 * x] = t.x; rr[4 * x + 1] = t.y; rr[4 * x + 2] = t.z; rr[4 * x + 3] = t.w;
        }
        tmem_st16((v ? tV : tK) + lane_base + sub * 32 + c * 4, rr);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(bar(v ? V_READY : K_READY));
      return true;
    };
    Item cur, nxt;
    uint32_t g = 0, n = 0, r = 0, moved = 0;  // r: the item's first tile in the rings; moved: items so far whose K and V went to tensor memory
    bool more = take_warp(0, &cur), ok = true;
    // Row statistics of a step are staged one step ahead, in the one place there is: the score (dP) product of this step, which read it, is complete
    // when the compute warps are at its result, and the next one follows their arrival on P_FULL (DS_FULL).
    if (more) {
      stage(fetch_stat(cur, 0));
      mbar_arrive(bar(FIRST));
      if (cur.n_it > 1) ok = load_resident(false, 0, 0);
    }
    while (more && ok) {
      if (p.zero_tiles > 0) zero_unseen(cur);
      for (int it = 0; it < cur.n_it; ++it, ++g) {
        const uint32_t ph = g & 1;
        const long long q0 = (cur.i_begin + it * ST) * BT;
        const long long kj = cur.k0 + row;
        // next step's statistics: loaded now, staged after the phases below
        const bool last = it + 1 == cur.n_it;
        if (last) more = take_warp(n + 1, &nxt);
        const bool has_next_step = !last || more;
        float stat_next = 0.0f;
        if (has_next_step) stat_next = last ? fetch_stat(nxt, 0) : fetch_stat(cur, it + 1);
        // visible iff key <= query + shift  <=>  column >= kj - shift - q0
        const bool need_mask = p.causal && (q0 + p.shift < cur.k0 + (BT - 1));
        long long cmin_ll = kj - p.shift - q0;
        const int cmin = !need_mask ? 0 : (cmin_ll > BT ? BT : (cmin_ll < 0 ? 0 : (int)cmin_ll));
        DF_BTRACE(1, 50);
        if (!mbar_wait_warp(bar(S_FULL + sub), ph, abort_flag)) { ok = false; break; }
        DF_BTRACE(1, 51);
        tc_fence_after_sync();
        float pr[CPT];
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          uint32_t rr[32];
          tmem_ld32(tS + lane_base + col0 + c * 32, rr);
          tmem_wait_ld();
          // only a tile on the diagonal has hidden scores: they become -inf here (and 0 below), so that the
          // exponentials of every other tile carry no compare and select
          if (need_mask) {
#pragma unroll
            for (int x = 0; x < 32; ++x)
              if (col0 + c * 32 + x < cmin) rr[x] = 0xff800000u;
          }
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = mul2(as_float2(rr[x], rr[x + 1]), make_float2(p.kv_scale_log2, p.kv_scale_log2));
            // rounded with the low bits cleared, so that one register serves as the P^T operand of dV and as P for dS
            // (keeping the unrounded value as well measured slower: 64 more live registers)
            rr[x] = cvt_rna_tf32(ex2_approx(t.x));
            rr[x + 1] = cvt_rna_tf32(ex2_approx(t.y));
            pr[c * 32 + x] = __uint_as_float(rr[x]);
            pr[c * 32 + x + 1] = __uint_as_float(rr[x + 1]);
          }
          tmem_st32(tS + lane_base + col0 + c * 32, rr);
        }
        if (stat_lse && has_next_step) stage(stat_next);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(P_FULL + sub));
        DF_BTRACE(1, 52);
        // the next item's K: its second step's scores follow soon after; and the very first item's V, which nobody waits for before this
        if (last) r += cur.n_it + 1;
        const bool first_v = g == 0 && cur.n_it > 1;
        if (first_v || (!SPLIT && last && more && nxt.n_it > 1)) {
          if (!load_resident(first_v, first_v ? 0 : r, moved)) { ok = false; break; }
          if (first_v) ++moved;
        }
        if (!mbar_wait_warp(bar(DP_FULL + sub), ph, abort_flag)) { ok = false; break; }
        DF_BTRACE(1, 53);
        tc_fence_after_sync();
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          uint32_t rr[32];
          tmem_ld32(tDP + lane_base + col0 + c * 32, rr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = mul2(make_float2(pr[c * 32 + x], pr[c * 32 + x + 1]), as_float2(rr[x], rr[x + 1]));
            rr[x] = tf32_rna_operand(t.x);
            rr[x + 1] = tf32_rna_operand(t.y);
          }
          tmem_st32(tDP + lane_base + col0 + c * 32, rr);
        }
        if (!stat_lse && has_next_step) stage(stat_next);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(DS_FULL + sub));
        DF_BTRACE(1, 54);
      }
      if (SPLIT) {
        if (ok) ok = mbar_wait_warp(bar(ACC_FULL), n & 1, abort_flag);
        break;
      }
      if (ok && more && nxt.n_it > 1) ok = load_resident(true, r, moved++);
      if (!ok || !hand_over(n)) { ok = false; break; }
      cur = nxt;
      ++n;
    }
  }
  if constexpr (SPLIT) {
    tc_fence_before_sync();
    cluster_sync();  // both CTAs' products are done and their operand buffers free
    tc_fence_after_sync();
    const Item it = decode(p, (int)(blockIdx.x / 2));
    const bool own = it.n_it + 1 - (int)rank >= 2, other = it.n_it + (int)rank >= 2;
    // rank 0 finishes dV and rank 1 dK, in the buffer of the MN-major dO tile; the threads of a row have half of its columns each
    const int row = (warp & 3) * 32 + lane, d0 = (warp >> 2) * 32;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16, t_own = (rank ? tDK : tDV) + lanes, t_send = (rank ? tDV : tDK) + lanes;
    if (warp < kCW && own) {
      send_cols(map_to_rank(aGm, rank ^ 1), row, d0, t_send);
      send_cols(map_to_rank(aGm, rank ^ 1), row, d0 + 16, t_send);
    }
    cluster_sync();
    if (warp < kCW) {
      finish_cols(smem + 5 * kTile, row, d0, t_own, own, other, rank ? p.scale : 1.0f);
      finish_cols(smem + 5 * kTile, row, d0 + 16, t_own, own, other, rank ? p.scale : 1.0f);
      fence_proxy_async_smem();
      mbar_arrive(bar(EPI_FULL));
    } else if (warp == kWarpLoadM && lane == 0 && mbar_wait(bar(EPI_FULL), 0, abort_flag)) {
      for (int sl = 0; sl < 2; ++sl) tma_store_4d(rank ? &tmDK : &tmDV, aGm + sl * kSlab, 32 * sl, (int)it.h, (int)it.k0, (int)it.b);
      tma_store_commit();
      tma_store_wait_read_all();
    }
    __syncwarp();
    tc_fence_before_sync();
  }
  if (p.early) pdl_wait();  // whoever waits for this kernel waits for the dQ kernel too

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (warp == kWarpMma || warp == kWarpMma2) {
      commit_elected(bar(DRAIN));  // by the lane that issued the MMAs: the election is deterministic; two arrivals
      for (int t = 0; t < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++t) {
      }
    }
    if ((warp == kWarpLoadK || warp == kWarpLoadM) && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == kWarpMma) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// =========================================================================================
// dQ
// =========================================================================================
namespace dq {
enum Bar { Q_FULL = 0, GO_FULL, Q_EMPTY, G_EMPTY, KK_FULL, VK_FULL, KM_FULL, KM_EMPTY, S_FULL, S_FREE, DP_FULL0, DP_FULL1,
           DS_FULL0, DS_FULL1, ACC_FULL, EPI_FULL, O_FREE, DX_FULL, DELTA_DONE, DRAIN, NUM };
constexpr uint32_t kBars = 6 * kTile;              // Q, dO, K (K-major), V, K (MN-major), O (only with fused row sums)
constexpr uint32_t kXch = kBars + 256;             // partial row sums of two items in turn, [2][2][128]
constexpr uint32_t kXchItem = 2 * 128 * 4;
constexpr uint32_t kSmemTotal = kXch + 2 * kXchItem + 1024;  // 1024: the tiles begin on the next 1024-byte boundary

// One work item: 128 queries of one head and the key tiles they can see.
struct Item {
  uint32_t b, h;
  long long q0;  // first query row
  int n_kv;      // number of key tiles (0: the rows see no key)
};
__device__ __forceinline__ Item decode(const BwdParams &p, int idx, int n_qt) {
  Item it;
  const uint32_t n_bh = p.B * p.H, bh = (uint32_t)idx % n_bh;
  it.b = bh / p.H;
  it.h = bh % p.H;
  it.q0 = (long long)(n_qt - 1 - (int)((uint32_t)idx / n_bh)) * BT;  // the latest query tile sees the most keys
  long long kv_end = p.causal ? it.q0 + (BT - 1) + p.shift + 1 : (long long)p.Sk;
  if (kv_end > (long long)p.Sk) kv_end = p.Sk;
  if (kv_end < 0) kv_end = 0;
  it.n_kv = (int)((kv_end + BT - 1) / BT);
  return it;
}
__device__ __forceinline__ int next_round(const BwdParams &p, int r, int n_items, int n_qt, Item *out) {
  for (;; ++r) {
    const int idx = item_of_round(r, n_items);
    if (idx < 0) return -1;
    *out = decode(p, idx, n_qt);
    if (out->n_kv > 0) return r;
  }
}
}  // namespace dq

// FUSE_DELTA: the kernel also fetches the O tile of its queries, computes delta = rowsum(dO o O)
// itself (dO as rounded to TF32 by its tensor map, the same values the dP product sees) and
// writes it to p.delta_out for the dK/dV kernel, which then has to run after this one.
// SPLIT (with FUSE_DELTA): as in the dK/dV kernel, two CTAs take every other key tile of an item; rank r finishes dims 32 r...
template <bool FUSE_DELTA, bool SPLIT>
__global__ void __launch_bounds__(kBwdThreads, 1)
k_attn_bwd_dq_tf32_d64(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                       const __grid_constant__ CUtensorMap tmKk, const __grid_constant__ CUtensorMap tmVk,
                       const __grid_constant__ CUtensorMap tmKm, const __grid_constant__ CUtensorMap tmDQ,
                       const __grid_constant__ CUtensorMap tmO, const BwdParams p, const int n_items) {
  using namespace dq;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t aQ = smem_u32(smem), aG = aQ + kTile, aKk = aQ + 2 * kTile, aVk = aQ + 3 * kTile, aKm = aQ + 4 * kTile,
                 aO = aQ + 5 * kTile;
  float *sXch = reinterpret_cast<float *>(smem + kXch);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + kBars + 192);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + kBars + 196);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t dm = (size_t)p.H * HD;
  constexpr int ST = SPLIT ? 2 : 1;  // key tiles from one step to the next
  const int rank = SPLIT ? (int)cluster_rank() : 0;
  const int n_qt = (int)(((long long)p.Sq + BT - 1) / BT);

  auto bar = [&](int id) { return smem_u32(&bars[id]); };
  // item of the first round >= r that has work for this CTA
  auto pick = [&](int r, Item *out) -> int {
    if (!SPLIT) return next_round(p, r, n_items, n_qt, out);
    if (r > 0) return -1;
    *out = decode(p, (int)(blockIdx.x / 2), n_qt);
    out->n_kv = (out->n_kv + 1 - rank) / 2;
    return out->n_kv > 0 ? 0 : -1;
  };
  if (warp == 8) {
    if (lane < NUM) mbar_init(bar(lane), (lane == S_FREE || lane == DS_FULL0 || lane == DS_FULL1 || lane == EPI_FULL || lane == O_FREE || lane == DX_FULL || lane == DELTA_DONE) ? 256 : 1);
    static_assert(NUM <= 32, "a lane per barrier");
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    Item first;
    if (lane == 0 && pick(0, &first) >= 0) {  // the first tiles are under way while the others set up
      pdl_wait();
      load_tile(aQ, &tmQ, bar(Q_FULL), (int)first.h, (int)first.q0, (int)first.b);
      load_tile(aKk, &tmKk, bar(KK_FULL), (int)first.h, rank * BT, (int)first.b);
    }
  }
  if (warp == 10) {
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  // dP / dS is double-buffered (steps alternate): dP of step g+1 is issued ahead of dQ of step g, so the compute warps
  // never wait for it and the item's last dP - whose completion frees dO for the next item - runs a step early
  const uint32_t tS = tmem, tDP0 = tmem + 128, tDQ = tmem + 256, tDP1 = tmem + 320;
#ifdef DF_ATTN_TRACE
  // with -DDF_ATTN_TRACE_DQ the trace follows this kernel instead of the dK/dV kernel (same two slots)
#ifdef DF_ATTN_TRACE_DQ
  const bool trace_on = blockIdx.x == 0 && lane == 0 && (warp == 10 || warp == 0);
#else
  const bool trace_on = false;
#endif
  int tr_n = 0;
#endif
  pdl_wait();  // everything above touched only this CTA's shared and tensor memory

  // g = steps (key tiles) done over all items, n = items done (see the dK/dV kernel)
  if (warp == 8) {
    // ---------------------------------------------- producer: Q, dO per item; K-major K and V tiles per step
    if (lane == 0) {
      Item cur;
      uint32_t g = 0, n = 0;
      for (int r = pick(0, &cur); r >= 0; r = pick(r + 1, &cur), ++n) {
        bool ok = true;
        if (n > 0 && !mbar_wait(bar(Q_EMPTY), (n - 1) & 1, abort_flag)) break;
        // Q lands on a barrier of its own, dO (and O) on another: the next item's first S needs only Q, whose buffer
        // is free a step before dO's. On one barrier the MMA warp stood waiting for all three tiles at the end of every
        // item with the item's last dQ queued behind that wait, and the compute warps behind it.
        if (n > 0) load_tile(aQ, &tmQ, bar(Q_FULL), (int)cur.h, (int)cur.q0, (int)cur.b);  // the first: during set-up
        for (int j = 0; j < cur.n_kv; ++j, ++g) {
          // a K-major K (V) buffer is free once the S (dP) product that read it has completed
          if (g > 0 && !mbar_wait(bar(S_FULL), (g - 1) & 1, abort_flag)) { ok = false; break; }
          if (g > 0) load_tile(aKk, &tmKk, bar(KK_FULL), (int)cur.h, (j * ST + rank) * BT, (int)cur.b);
          if (j == 0) {  // dO (and O) follow the item's first K tile, which does not have to wait for their buffers
            if (n > 0 && !mbar_wait(bar(G_EMPTY), (n - 1) & 1, abort_flag)) { ok = false; break; }
            // with fused row sums the compute warps read the dO and O tiles too: both are replaced
            // only after they are done with them
            if (FUSE_DELTA && n > 0 && !mbar_wait(bar(O_FREE), (n - 1) & 1, abort_flag)) { ok = false; break; }
            mbar_arrive_expect_tx(bar(GO_FULL), (FUSE_DELTA ? 2 : 1) * kTile);
            tma_load_4d(aG, &tmG, bar(GO_FULL), 0, (int)cur.h, (int)cur.q0, (int)cur.b);
            tma_load_4d(aG + kSlab, &tmG, bar(GO_FULL), 32, (int)cur.h, (int)cur.q0, (int)cur.b);
            if (FUSE_DELTA) {
              tma_load_4d(aO, &tmO, bar(GO_FULL), 0, (int)cur.h, (int)cur.q0, (int)cur.b);
              tma_load_4d(aO + kSlab, &tmO, bar(GO_FULL), 32, (int)cur.h, (int)cur.q0, (int)cur.b);
            }
          }
          if (g > 0 && !mbar_wait(bar(DP_FULL0 + ((g - 1) & 1)), ((g - 1) >> 1) & 1, abort_flag)) { ok = false; break; }
          load_tile(aVk, &tmVk, bar(VK_FULL), (int)cur.h, (j * ST + rank) * BT, (int)cur.b);
        }
        if (!ok) break;
      }
    }
  } else if (warp == 9) {
    // ---------------------------------------------- producer: MN-major K tiles per step, result store per item
    if (lane == 0) {
      Item cur;
      uint32_t g = 0, n = 0;
      for (int r = pick(0, &cur); r >= 0; r = pick(r + 1, &cur), ++n) {
        bool ok = true;
        for (int j = 0; j < cur.n_kv; ++j, ++g) {
          // the buffer is released by a commit of its own right after dQ of the step before
          if (g > 0 && !mbar_wait(bar(KM_EMPTY), (g - 1) & 1, abort_flag)) { ok = false; break; }
          load_tile(aKm, &tmKm, bar(KM_FULL), (int)cur.h, (j * ST + rank) * BT, (int)cur.b);
        }
        if (SPLIT) break;
        // the compute warps stage the item's dQ tile in this buffer; hand it to the copy engine
        // (rows beyond Sq are dropped) and refill the buffer once the store has read it
        if (!ok || !mbar_wait(bar(EPI_FULL), n & 1, abort_flag)) break;
        tma_store_4d(&tmDQ, aKm, 0, (int)cur.h, (int)cur.q0, (int)cur.b);
        tma_store_4d(&tmDQ, aKm + kSlab, 32, (int)cur.h, (int)cur.q0, (int)cur.b);
        tma_store_commit();
        tma_store_wait_read_all();
      }
    }
  } else if (warp == 10) {
    // ---------------------------------------------- MMA issuer: .., S_{g+1}, dP_{g+1}, dQ_g, .. over all items
    // (at the last step of an item: S of the next item, dQ_g, then the next item's first dP)
    // (the whole warp runs this role; only the MMA and commit instructions are issued by one elected lane)
    {
      const uint32_t idesc_ss = make_idesc(kFmtTF32, BT, BT, 0, 0);
      const uint32_t idesc_ts = make_idesc(kFmtTF32, BT, HD, 0, 1);
      const uint64_t dQ_ = kmajor_desc(aQ), dG_ = kmajor_desc(aG), dKk = kmajor_desc(aKk), dVk = kmajor_desc(aVk), dKm = mnmajor_desc(aKm);
      Item cur, nxt;
      uint32_t g = 0, n = 0;
      int r = pick(0, &cur);
      bool ok = r >= 0;
      // `last` = last step of its item: Q (for S) or dO (for dP) may then be replaced
      // `landed`: the caller has already seen the operand tile's barrier complete
      auto issue_s = [&](uint32_t gs, bool last, bool landed) -> bool {
        if (!landed) {
          if (!mbar_wait_warp(bar(KK_FULL), gs & 1, abort_flag)) return false;
          tc_fence_after_sync();
        }
        issue_ss_128x128(tS, dQ_, dKk, idesc_ss);  // S = Q K^T
        commit_elected(bar(S_FULL));
        if (last) commit_elected(bar(Q_EMPTY));
        return true;
      };
      auto issue_dp = [&](uint32_t gs, bool last) -> bool {
        if (!mbar_wait_warp(bar(VK_FULL), gs & 1, abort_flag)) return false;
        tc_fence_after_sync();
        issue_ss_128x128((gs & 1) ? tDP1 : tDP0, dG_, dVk, idesc_ss);  // dP = dO V^T
        commit_elected(bar(DP_FULL0 + (gs & 1)));
        if (last) commit_elected(bar(G_EMPTY));
        return true;
      };
      if (ok) ok = mbar_wait_warp(bar(Q_FULL), 0, abort_flag);
      if (ok) ok = issue_s(0, cur.n_kv == 1, false);
      if (ok) ok = mbar_wait_warp(bar(GO_FULL), 0, abort_flag);
      if (ok) ok = issue_dp(0, cur.n_kv == 1);
      while (ok) {
        const int rn = pick(r + 1, &nxt);
        for (int j = 0; ok && j < cur.n_kv; ++j, ++g) {
          const bool last = j + 1 == cur.n_kv;
          const bool has_next = !last || rn >= 0;
          const bool next_last = last ? (nxt.n_kv == 1) : (j + 2 == cur.n_kv);
          const uint32_t ph = g & 1, phn = ph ^ 1;
          if (has_next) {
            // S_{g+1} may overwrite S_g once the compute warps hold P_g in registers; one poll covers that and
            // the operand tile, only a barrier that is still open is then waited for on its own
            const uint32_t m = mbar_test3_warp(bar(S_FREE), ph, bar(KK_FULL), phn, bar(KK_FULL), phn);
            if (!(m & 1u) && !mbar_wait_warp(bar(S_FREE), ph, abort_flag)) { ok = false; break; }
            DF_BTRACE(0, 10);
            if (last && !mbar_wait_warp(bar(Q_FULL), (n + 1) & 1, abort_flag)) { ok = false; break; }
            DF_BTRACE(0, 11);
            tc_fence_after_sync();
            if (!issue_s(g + 1, next_last, (m & 2u) != 0u)) { ok = false; break; }
            DF_BTRACE(0, 12);
            // dP_{g+1} of the same item goes out now, into the buffer dQ_{g-1} (issued a step ago by this thread) read
            if (!last && !issue_dp(g + 1, next_last)) { ok = false; break; }
          }
          // dS has a barrier per dP buffer: dP_{g+1} is out already, so dS_{g+1} may be complete before this warp has looked for
          // dS_g, and on one barrier it would then wait for a phase that has come round again
          const uint32_t ph2 = (g >> 1) & 1;
          const uint32_t m = mbar_test3_warp(bar(DS_FULL0 + ph), ph2, bar(KM_FULL), ph, bar(KM_FULL), ph);
          if ((!(m & 1u) && !mbar_wait_warp(bar(DS_FULL0 + ph), ph2, abort_flag)) || (!(m & 2u) && !mbar_wait_warp(bar(KM_FULL), ph, abort_flag))) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
          DF_BTRACE(0, 31);
          issue_ts_128x64(tDQ, ph ? tDP1 : tDP0, dKm, idesc_ts, j > 0);  // dQ += dS K
          DF_BTRACE(0, 32);
          commit_elected(bar(KM_EMPTY));
          if (last) commit_elected(bar(ACC_FULL));
          if (has_next && last) {
            // the first dP of the next item needs its dO tile, which can only be loaded once this item's last dP is
            // done: it follows the item's last dQ, so that the finished accumulator never waits behind that tile
            if (!mbar_wait_warp(bar(GO_FULL), (n + 1) & 1, abort_flag)) { ok = false; break; }
            if (!issue_dp(g + 1, next_last)) { ok = false; break; }
          }
          DF_BTRACE(0, 33);
        }
        if (rn < 0) break;
        r = rn;
        cur = nxt;
        ++n;
      }
    }
  } else {
    // ---------------------------------------------- compute warps: lanes = queries, columns = keys
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int col0 = half * 64;
    // query rows that see no key: dQ = 0
    for (int r0 = 0; !SPLIT; ++r0) {
      const int idx = item_of_round(r0, n_items);
      if (idx < 0) break;
      const Item z = decode(p, idx, n_qt);
      if (z.n_kv > 0) continue;
      const long long i = z.q0 + row;
      if (i < (long long)p.Sq) {
        float4 *dst = reinterpret_cast<float4 *>(p.dq + ((size_t)z.b * p.Sq + (size_t)i) * dm + z.h * HD + half * 32);
#pragma unroll
        for (int x = 0; x < 8; ++x) dst[x] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    // logsumexp (in log2 units) and delta of this thread's query row in item `im`
    // The logsumexp comes back RAW (-inf for a row beyond the sequence): nothing is computed from it here, so the
    // thread does not stall on the load; lse2_of() turns it into log2 units when the item starts.
    auto fetch_stats = [&](const Item &im, float *lse_raw, float *dlt) {
      const long long i = im.q0 + row;
      *lse_raw = -INFINITY;
      *dlt = 0.0f;
      if (i < (long long)p.Sq) {
        const size_t s_idx = ((size_t)im.b * p.H + im.h) * p.Sq + (size_t)i;
        *lse_raw = __ldg(p.lse + s_idx);
        if (!FUSE_DELTA) *dlt = __ldg(p.delta + s_idx);
      }
    };
    auto lse2_of = [](float raw) -> float { return (raw == -INFINITY) ? INFINITY : raw * kLog2e; };
    // Fused row sums: delta of this thread's row of item `im` (the nn-th item of this CTA) from the
    // dO and O tiles in shared memory. Each of the row's two threads sums its 32 dims (one
    // 128-byte slab row, 16-byte chunk c at c ^ (row % 8)); the halves meet in shared memory.
    auto fused_delta = [&](const Item &im, uint32_t nn, float *out) -> bool {
      if (!mbar_wait_warp(bar(GO_FULL), nn & 1, abort_flag)) return false;
      const uint8_t *g_row = smem + kTile + half * kSlab + row * 128;
      const uint8_t *o_row = smem + 5 * kTile + half * kSlab + row * 128;
      float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t off = (uint32_t)((x ^ (row & 7)) << 4);
        const float4 gv = *reinterpret_cast<const float4 *>(g_row + off);
        const float4 ov = *reinterpret_cast<const float4 *>(o_row + off);
        acc0 = fmaf(gv.x, ov.x, acc0); acc1 = fmaf(gv.y, ov.y, acc1);
        acc0 = fmaf(gv.z, ov.z, acc0); acc1 = fmaf(gv.w, ov.w, acc1);
      }
      float *xs = sXch + (nn & 1) * (kXchItem / 4);
      xs[half * 128 + row] = acc0 + acc1;
      mbar_arrive(bar(O_FREE));
      mbar_arrive(bar(DX_FULL));
      if (!mbar_wait_warp(bar(DX_FULL), nn & 1, abort_flag)) return false;
      *out = xs[row] + xs[128 + row];
      const long long i = im.q0 + row;
      if (half == 0 && rank == 0 && i < (long long)p.Sq) p.delta_out[((size_t)im.b * p.H + im.h) * p.Sq + (size_t)i] = *out;
      return true;
    };
    Item cur, nxt;
    uint32_t g = 0, n = 0;
    int r = pick(0, &cur);
    bool ok = true;
    if (SPLIT && r < 0 && p.early && warp == 0) pdl_trigger();  // no step for this CTA
    float lse_raw = -INFINITY, dlt = 0.0f, lse_raw_next = -INFINITY, dlt_next = 0.0f;
    if (r >= 0) fetch_stats(cur, &lse_raw, &dlt);
    if (FUSE_DELTA && r >= 0) ok = fused_delta(cur, 0, &dlt);
    while (r >= 0 && ok) {
      const int rn = pick(r + 1, &nxt);
      if (FUSE_DELTA && p.early && rn < 0) {
        // All row sums of this CTA are written: the dK/dV kernel may start on SMs that have run out of items.
        // (Decided by a whole warp: the tensor-memory instructions that follow need their warps converged.)
        __threadfence();
        mbar_arrive(bar(DELTA_DONE));
        if (warp == 0 && mbar_wait_warp(bar(DELTA_DONE), 0, abort_flag)) pdl_trigger();
        __syncwarp();
      }
      if (rn >= 0) fetch_stats(nxt, &lse_raw_next, &dlt_next);  // in flight while this item computes
      const float lse2 = lse2_of(lse_raw);
      const long long i = cur.q0 + row;
      long long kmax_ll = p.causal ? i + p.shift + 1 : (long long)p.Sk;
      if (kmax_ll > (long long)p.Sk) kmax_ll = p.Sk;
      if (kmax_ll < 0) kmax_ll = 0;
      const int kmax = (int)kmax_ll;
      for (int j = 0; j < cur.n_kv; ++j, ++g) {
        const uint32_t ph = g & 1;
        const int key0 = (j * ST + rank) * BT;
        const bool need_mask = key0 + BT > kmax;
        DF_BTRACE(1, 50);
        if (!mbar_wait_warp(bar(S_FULL), ph, abort_flag)) { ok = false; break; }
        DF_BTRACE(1, 51);
        tc_fence_after_sync();
        float pr[64];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t rr[32];
          tmem_ld32(tS + lane_base + col0 + c * 32, rr);
          tmem_wait_ld();
          // only the last key tiles of a row have hidden scores: they become -inf here (and 0 below), so that the
          // exponentials of every other tile carry no compare and select
          if (need_mask) {
#pragma unroll
            for (int x = 0; x < 32; ++x)
              if (!(key0 + col0 + c * 32 + x < kmax)) rr[x] = 0xff800000u;
          }
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = fma2(as_float2(rr[x], rr[x + 1]), make_float2(p.scale_log2, p.scale_log2), make_float2(-lse2, -lse2));
            pr[c * 32 + x] = ex2_approx(t.x);
            pr[c * 32 + x + 1] = ex2_approx(t.y);
          }
        }
        tc_fence_before_sync();
        mbar_arrive(bar(S_FREE));
        DF_BTRACE(1, 52);
        if (!mbar_wait_warp(bar(DP_FULL0 + ph), (g >> 1) & 1, abort_flag)) { ok = false; break; }
        DF_BTRACE(1, 53);
        tc_fence_after_sync();
        const uint32_t tDP = ph ? tDP1 : tDP0;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t rr[32];
          tmem_ld32(tDP + lane_base + col0 + c * 32, rr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const float2 t = mul2(make_float2(pr[c * 32 + x], pr[c * 32 + x + 1]), add2(as_float2(rr[x], rr[x + 1]), make_float2(-dlt, -dlt)));
            rr[x] = tf32_rna_operand(t.x);
            rr[x + 1] = tf32_rna_operand(t.y);
          }
          tmem_st32(tDP + lane_base + col0 + c * 32, rr);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(DS_FULL0 + ph));
        DF_BTRACE(1, 54);
      }
      // the next item's dO and O tiles are on their way or already here: its row sums are
      // computed while the last dQ product of this item is still running (handing the finished dQ over first,
      // and the row sums after it, measured the same)
      if (FUSE_DELTA && ok && rn >= 0) ok = fused_delta(nxt, n + 1, &dlt_next);
      DF_BTRACE(1, 59);
      if (!ok || !mbar_wait_warp(bar(ACC_FULL), n & 1, abort_flag)) { ok = false; break; }
      DF_BTRACE(1, 60);
      tc_fence_after_sync();
      if (SPLIT) break;
      {
        uint32_t rr[32];
        tmem_ld32(tDQ + lane_base + half * 32, rr);  // each half handles 32 of the 64 dims = one 128-byte slab
        tmem_wait_ld();
        // staged over the MN-major K buffer (free: every MMA of the item has finished) in the
        // swizzled slab layout of the store's tensor map; the second producer thread stores it
        uint8_t *stage = smem + 4 * kTile + half * kSlab + row * 128;
#pragma unroll
        for (int x = 0; x < 8; ++x)
          *reinterpret_cast<float4 *>(stage + ((x ^ (row & 7)) << 4)) =
              make_float4(__uint_as_float(rr[4 * x]) * p.scale, __uint_as_float(rr[4 * x + 1]) * p.scale,
                          __uint_as_float(rr[4 * x + 2]) * p.scale, __uint_as_float(rr[4 * x + 3]) * p.scale);
        tc_fence_before_sync();
        fence_proxy_async_smem();
        mbar_arrive(bar(EPI_FULL));
        DF_BTRACE(1, 61);
      }
      r = rn;
      cur = nxt;
      lse_raw = lse_raw_next;
      dlt = dlt_next;
      ++n;
    }
  }

  if constexpr (SPLIT) {
    tc_fence_before_sync();
    cluster_sync();  // both CTAs' products are done and their operand buffers free
    tc_fence_after_sync();
    const Item it = decode(p, (int)(blockIdx.x / 2), n_qt);
    const bool own = it.n_kv + 1 - rank >= 2, other = it.n_kv + rank >= 2;
    // rank r finishes dims 32 r .. 32 r + 31, in a slab of the buffer of the MN-major K tile; the threads of a row have half of them each
    const int row = (warp & 3) * 32 + lane, d_own = rank * 32 + (warp >> 2) * 16, d_send = (rank ^ 1) * 32 + (warp >> 2) * 16;
    const uint32_t taddr = tDQ + ((uint32_t)((warp & 3) * 32) << 16);
    if (warp < 8 && own) send_cols(map_to_rank(aKm, (uint32_t)(rank ^ 1)), row, d_send, taddr);
    cluster_sync();
    if (warp < 8) {
      finish_cols(smem + 4 * kTile, row, d_own, taddr, own, other, p.scale);
      fence_proxy_async_smem();
      mbar_arrive(bar(EPI_FULL));
    } else if (warp == 9 && lane == 0 && mbar_wait(bar(EPI_FULL), 0, abort_flag)) {
      tma_store_4d(&tmDQ, aKm + rank * kSlab, 32 * rank, (int)it.h, (int)it.q0, (int)it.b);
      tma_store_commit();
      tma_store_wait_read_all();
    }
    __syncwarp();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (warp == 10) {
      commit_elected(bar(DRAIN));  // by the lane that issued the MMAs: the election is deterministic
      for (int t = 0; t < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++t) {
      }
    }
    if ((warp == 8 || warp == 9) && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == 10) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// =========================================================================================
// One tile: at most 128 queries and 128 keys
// =========================================================================================
namespace one {
// QK_FULL, GV_FULL: two tiles each. The scores and dP exist twice, as [queries, keys] for dQ and as [keys, queries] (.._T) for dK and dV.
enum Bar { QK_FULL = 0, GV_FULL, O_FULL, GM_FULL, QM_FULL, KM_FULL, LSE_FULL, DELTA_FULL, S_FULL, ST_FULL, DP_FULL, DPT_FULL, PT_FULL, DST_FULL, DS_FULL,
           DQ_FULL, DV_FULL, DK_FULL, DRAIN, NUM };
// Sixteen warps that all compute (a seventeenth would leave 96 registers a thread): warp 0 also loads and issues S, dP and dQ, warp 8 the other products.
constexpr int kThreads = 512;
constexpr uint32_t kLse = 7 * kTile;             // Q, K, dO, V (K-major), dO, Q, K (MN-major); logsumexp of the queries in log2 units
constexpr uint32_t kDelta = kLse + BT * 4;       // their row sums in two halves
constexpr uint32_t kBars = kDelta + 2 * BT * 4;
constexpr uint32_t kSmemTotal = kBars + 192 + 1024;
static_assert(NUM * 8 <= 184 && kSmemTotal <= 227 * 1024, "");
}  // namespace one

// The whole backward of a head whose queries and keys are one tile each. What such a call costs is latency: the chain of two kernels (launch,
// set-up, first loads, scores, results, twice, the second behind the first's row sums) where one step's products take 1.5 us. Here both sides run at the
// same time, on tiles that are all loaded at once (224 KB): the score products come out in both orientations (sharing one would mean turning P over
// through shared memory), for dQ with lanes = queries, for dK and dV with lanes = keys. SPLIT: a CTA for either side, while there are SMs for it; else one
// CTA has both, eight warps each, and its result accumulators lie over scores that have been read. Every instruction runs once or a few times, so that
// fetching them is what the phases wait for: short loops instead of straight code. Columns that a warp's rows do not see are skipped (16 at a time).
// B200, fp32, S = 128, causal, H = 12, us against the two kernels: batch 1 11.6 -> 7.3, 4 12.1 -> 7.3, 8 16.4 -> 8.8, 12 17.6 -> 9.0, 20 23.6 -> 17.0. The
// parts at batch 1: one kernel 11.0, straight code into loops and no spills 9.2, O through the copy engine and plain stores 8.7, a CTA per side 7.3.
template <bool SPLIT>
__global__ void __launch_bounds__(one::kThreads, 1)
k_attn_bwd_tile_tf32_d64(const __grid_constant__ CUtensorMap tmQk, const __grid_constant__ CUtensorMap tmGk,
                         const __grid_constant__ CUtensorMap tmKk, const __grid_constant__ CUtensorMap tmVk,
                         const __grid_constant__ CUtensorMap tmQm, const __grid_constant__ CUtensorMap tmGm,
                         const __grid_constant__ CUtensorMap tmKm, const __grid_constant__ CUtensorMap tmO, const BwdParams p) {
  using namespace one;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t aQ = smem_u32(smem), aK = aQ + kTile, aG = aQ + 2 * kTile, aV = aQ + 3 * kTile, aGm = aQ + 4 * kTile, aQm = aQ + 5 * kTile, aKm = aQ + 6 * kTile;
  float *sLse = reinterpret_cast<float *>(smem + kLse), *sDelta = reinterpret_cast<float *>(smem + kDelta);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + kBars + 184);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + kBars + 188);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t bh = SPLIT ? blockIdx.x >> 1 : blockIdx.x, h = bh % p.H, b = bh / p.H;
  const bool keys = SPLIT ? (blockIdx.x & 1) != 0 : warp >= 8;  // lanes = keys: dV and dK; else lanes = queries: dQ
  auto bar = [&](int id) { return smem_u32(&bars[id]); };
  auto load_mn = [&](uint32_t dst, const CUtensorMap *m, int id, int box) {
    mbar_arrive_expect_tx(bar(id), kTile);
    for (int row = 0; row < BT; row += box)
      for (int sl = 0; sl < 2; ++sl) tma_load_4d(dst + sl * kSlab + row * 128, m, bar(id), 32 * sl, (int)h, row, (int)b);
  };
  if (warp == 0) {
    static_assert(NUM <= 32, "a lane per barrier");
    if (lane < NUM) {
      const bool two = lane == QK_FULL || lane == GV_FULL || lane == DRAIN;
      const bool all = (lane >= PT_FULL && lane <= DS_FULL) || lane == DELTA_FULL;
      mbar_init(bar(lane), two ? 2 : all ? (SPLIT && lane != DELTA_FULL ? 512 : 256) : lane == LSE_FULL ? 128 : 1);
    }
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    if (lane == 0) {  // the tiles are under way while the others set up
      pdl_wait();
      load_tile(aQ, &tmQk, bar(QK_FULL), (int)h, 0, (int)b);
      load_tile(aK, &tmKk, bar(QK_FULL), (int)h, 0, (int)b);
      load_tile(aG, &tmGk, bar(GV_FULL), (int)h, 0, (int)b);
      load_tile(aV, &tmVk, bar(GV_FULL), (int)h, 0, (int)b);
      load_tile(aKm, &tmO, bar(O_FULL), (int)h, 0, (int)b);  // K's place is O's at first
      if (!SPLIT || keys) {
        load_mn(aGm, &tmGm, GM_FULL, BT / 2);
        load_mn(aQm, &tmQm, QM_FULL, BT / 2);
      }
    }
    __syncwarp();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  const uint32_t tS = tmem, tST = tmem + 128, tDP = tmem + 256, tDPT = tmem + 384;
  const uint32_t tDQ = tS, tDV = tS + 64, tDK = tST;  // over scores that have been read, and over P^T after its product
  pdl_wait();  // everything above touched only this CTA's shared and tensor memory

  // Products by the calling warp, one elected lane issues; loops, not straight code: every instruction here runs once, and what costs is fetching it.
  // d = x y^T, of K-major tiles
  auto scores = [&](uint32_t d, uint32_t x, uint32_t y, int done) {
    const uint64_t dx = make_smem_desc(x, 16, 1024, kSwz128), dy = make_smem_desc(y, 16, 1024, kSwz128);
    if (elect_one()) {
#pragma unroll 1
      for (uint32_t sl = 0; sl < 2; ++sl)
#pragma unroll
        for (uint32_t kk = 0; kk < 4; ++kk) {
          const uint32_t off = sl * (kSlab >> 4) + kk * 2;
          mma_tf32_ss_lohi(d, (uint32_t)dx + off, (uint32_t)(dx >> 32), (uint32_t)dy + off, (uint32_t)(dy >> 32), make_idesc(kFmtTF32, BT, BT, 0, 0), sl + kk);
        }
      mma_commit(bar(done));
    }
    __syncwarp();
  };
  // d = x y, x in tensor memory, y an MN-major tile
  auto result = [&](uint32_t d, uint32_t x, uint32_t y, int done) {
    tc_fence_after_sync();
    const uint64_t dy = make_smem_desc(y, kSlab, 512, kSwz128B32);
    if (elect_one()) {
#pragma unroll 1
      for (uint32_t k4 = 0; k4 < BT / 8; k4 += 4)
#pragma unroll
        for (uint32_t kk = k4; kk < k4 + 4; ++kk)
          mma_tf32_ts_lohi(d, x + kk * 8, (uint32_t)dy + kk * (1024 >> 4), (uint32_t)(dy >> 32), make_idesc(kFmtTF32, BT, HD, 0, 1), kk);
      mma_commit(bar(done));
    }
    __syncwarp();
  };
  {
    // a thread has CW columns of its lane's row; half: of the row's dims, where two threads share them
    constexpr int CW = SPLIT ? 32 : 64;
    const int row = (warp & 3) * 32 + lane, half = (warp >> 2) & 1, col0 = SPLIT ? (warp >> 2) * 32 : half * 64;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    auto lse2_of = [](float raw) -> float { return (raw == -INFINITY) ? INFINITY : raw * kLog2e; };
    bool ok = false;
    auto row_sums = [&]() -> bool {  // by warps 0-7
      // row sums of dO o O, dO as rounded by its tensor map: the values that the dP products see
      if (!mbar_wait_warp(bar(GV_FULL), 0, abort_flag) || !mbar_wait_warp(bar(O_FULL), 0, abort_flag)) return false;
      const uint8_t *g_row = smem + 2 * kTile + half * kSlab + row * 128, *o_row = smem + 6 * kTile + half * kSlab + row * 128;
      float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t off = (uint32_t)((x ^ (row & 7)) << 4);
        const float4 gv = *reinterpret_cast<const float4 *>(g_row + off);
        const float4 ov = *reinterpret_cast<const float4 *>(o_row + off);
        acc0 = fmaf(gv.x, ov.x, acc0); acc1 = fmaf(gv.y, ov.y, acc1);
        acc0 = fmaf(gv.z, ov.z, acc0); acc1 = fmaf(gv.w, ov.w, acc1);
      }
      sDelta[half * BT + row] = acc0 + acc1;
      mbar_arrive(bar(DELTA_FULL));
      return true;
    };
    const size_t stat0 = ((size_t)b * p.H + h) * p.Sq;
    // S = Q K^T and dP = dO V^T, by warp 0; S^T = K Q^T and dP^T = V dO^T, by warp 8
    if (warp == (keys ? 8 : 0)) {
#pragma unroll 1
      for (int x = 0; x < 2; ++x) {
        if (!mbar_wait_warp(bar(QK_FULL + x), 0, abort_flag)) break;
        tc_fence_after_sync();
        const uint32_t lhs = aQ + (2 * x + (keys ? 1 : 0)) * kTile, rhs = aQ + (2 * x + (keys ? 0 : 1)) * kTile;
        scores((x ? tDP : tS) + (keys ? 128 : 0), lhs, rhs, (x ? DP_FULL : S_FULL) + (keys ? 1 : 0));
      }
    }
    if (!keys) {
      do {
        if (warp < 8 && !row_sums()) break;
        const float lse_raw = row < (int)p.Sq ? __ldg(p.lse + stat0 + row) : -INFINITY;
        const float lse2 = lse2_of(lse_raw);
        long long kmax_ll = p.causal ? row + p.shift + 1 : (long long)p.Sk;
        if (kmax_ll > (long long)p.Sk) kmax_ll = p.Sk;
        const int kmax = kmax_ll < 0 ? 0 : (int)kmax_ll, k_end = __reduce_max_sync(0xffffffffu, kmax);
        if (!mbar_wait_warp(bar(DELTA_FULL), 0, abort_flag)) break;
        if (warp == 0 && lane == 0) load_mn(aKm, &tmKm, KM_FULL, BT);  // O has been read
        __syncwarp();
        const float dlt = sDelta[row] + sDelta[BT + row];
        if (warp < 4 && row < (int)p.Sq) p.delta_out[stat0 + row] = dlt;
        if (!mbar_wait_warp(bar(S_FULL), 0, abort_flag) || !mbar_wait_warp(bar(DP_FULL), 0, abort_flag)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = col0; c < col0 + CW; c += 16) {
          uint32_t rr[16], pr[16];
          if (c >= k_end) {  // no row of the warp sees these keys
#pragma unroll
            for (int x = 0; x < 16; ++x) rr[x] = 0u;
            tmem_st16(tDP + lane_base + c, rr);
            continue;
          }
          tmem_ld16(tS + lane_base + c, pr);
          tmem_ld16(tDP + lane_base + c, rr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; x += 2) {
            const float2 e = fma2(as_float2(c + x < kmax ? pr[x] : 0xff800000u, c + x + 1 < kmax ? pr[x + 1] : 0xff800000u),
                                  make_float2(p.scale_log2, p.scale_log2), make_float2(-lse2, -lse2));
            const float2 y = mul2(make_float2(ex2_approx(e.x), ex2_approx(e.y)), add2(as_float2(rr[x], rr[x + 1]), make_float2(-dlt, -dlt)));
            rr[x] = tf32_rna_operand(y.x);
            rr[x + 1] = tf32_rna_operand(y.y);
          }
          tmem_st16(tDP + lane_base + c, rr);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(DS_FULL));
        if (warp == 0) {
          if (!mbar_wait_warp(bar(DS_FULL), 0, abort_flag) || !mbar_wait_warp(bar(KM_FULL), 0, abort_flag)) break;
          result(tDQ, tDP, aKm, DQ_FULL);
        }
        ok = true;
      } while (false);
    } else {
      do {
        if ((warp >> 2) == 2) {
          sLse[row] = lse2_of(row < (int)p.Sq ? __ldg(p.lse + stat0 + row) : -INFINITY);
          mbar_arrive(bar(LSE_FULL));
        }
        // key `row` is visible from query row - shift on
        long long qmin_ll = p.causal ? row - p.shift : 0;
        const int qmin = qmin_ll < 0 ? 0 : (qmin_ll > BT ? BT : (int)qmin_ll), q_begin = __reduce_min_sync(0xffffffffu, qmin);
        auto unseen = [&](int c) { return c + 16 <= q_begin || c >= (int)p.Sq; };  // 16 queries that see no key of the warp
        const uint32_t zero[16] = {0u};
        if (!mbar_wait_warp(bar(LSE_FULL), 0, abort_flag) || !mbar_wait_warp(bar(ST_FULL), 0, abort_flag)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = col0; c < col0 + CW; c += 16) {
          uint32_t rr[16];
          if (unseen(c)) {
            tmem_st16(tST + lane_base + c, zero);
            continue;
          }
          tmem_ld16(tST + lane_base + c, rr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; x += 2) {
            const float2 l = *reinterpret_cast<const float2 *>(sLse + c + x);
            const float2 y = fma2(as_float2(c + x >= qmin ? rr[x] : 0xff800000u, c + x + 1 >= qmin ? rr[x + 1] : 0xff800000u),
                                  make_float2(p.scale_log2, p.scale_log2), make_float2(-l.x, -l.y));
            rr[x] = cvt_rna_tf32(ex2_approx(y.x));  // low bits cleared: P of dS, too
            rr[x + 1] = cvt_rna_tf32(ex2_approx(y.y));
          }
          tmem_st16(tST + lane_base + c, rr);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(PT_FULL));
        if (SPLIT && warp == 8) {
          if (!mbar_wait_warp(bar(PT_FULL), 0, abort_flag) || !mbar_wait_warp(bar(GM_FULL), 0, abort_flag)) break;
          result(tDV, tST, aGm, DV_FULL);
        }
        if (SPLIT && warp < 8 && !row_sums()) break;
        if (!mbar_wait_warp(bar(DELTA_FULL), 0, abort_flag) || !mbar_wait_warp(bar(DPT_FULL), 0, abort_flag)) break;
        tc_fence_after_sync();
#pragma unroll 1
        for (int c = col0; c < col0 + CW; c += 16) {
          uint32_t rr[16], pr[16];
          if (unseen(c)) {
            tmem_st16(tDPT + lane_base + c, zero);
            continue;
          }
          tmem_ld16(tST + lane_base + c, pr);
          tmem_ld16(tDPT + lane_base + c, rr);
          tmem_wait_ld();
#pragma unroll
          for (int x = 0; x < 16; x += 2) {
            const float2 d = add2(*reinterpret_cast<const float2 *>(sDelta + c + x), *reinterpret_cast<const float2 *>(sDelta + BT + c + x));
            const float2 y = mul2(as_float2(pr[x], pr[x + 1]), add2(as_float2(rr[x], rr[x + 1]), make_float2(-d.x, -d.y)));
            rr[x] = tf32_rna_operand(y.x);
            rr[x + 1] = tf32_rna_operand(y.y);
          }
          tmem_st16(tDPT + lane_base + c, rr);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(DST_FULL));
        if (warp == 8) {
          if (!SPLIT) {  // dV goes where the scores were, and dK where P^T was
            if (!mbar_wait_warp(bar(PT_FULL), 0, abort_flag) || !mbar_wait_warp(bar(DS_FULL), 0, abort_flag) || !mbar_wait_warp(bar(GM_FULL), 0, abort_flag)) break;
            result(tDV, tST, aGm, DV_FULL);
          }
          if (!mbar_wait_warp(bar(DST_FULL), 0, abort_flag) || !mbar_wait_warp(bar(QM_FULL), 0, abort_flag)) break;
          result(tDK, tDPT, aQm, DK_FULL);
        }
        ok = true;
      } while (false);
    }
    // Results: dQ, dV and dK. A warp turns 32 rows of 32 columns over in an operand tile that no product reads any more, so that whole 128-byte
    // lines leave (tensor stores took 1.4 us more: their barrier, their start, and the wait before the tile may go).
    const int x0 = !keys ? 0 : SPLIT ? 1 + (warp >> 3) : 1, x1 = !keys ? (warp < 8 ? 1 : 0) : SPLIT ? x0 + 1 : 3;
    const int n_rows = (int)(keys ? p.Sk : p.Sq) - (warp & 3) * 32;
#pragma unroll 1
    for (int x = x0; ok && x < x1; ++x) {
      if (!mbar_wait_warp(bar(DQ_FULL + x), 0, abort_flag)) break;
      tc_fence_after_sync();
      const float mul = x == 1 ? 1.0f : p.scale;
      uint32_t rr[32];
      tmem_ld32((x == 0 ? tDQ : x == 1 ? tDV : tDK) + lane_base + half * 32, rr);
      tmem_wait_ld();
      uint8_t *slab = smem + (x == 0 ? 6 : 3 + x) * kTile + half * kSlab + (warp & 3) * 32 * 128;
#pragma unroll
      for (int y = 0; y < 8; ++y)
        *reinterpret_cast<float4 *>(slab + lane * 128 + ((y ^ (lane & 7)) << 4)) = make_float4(
            __uint_as_float(rr[4 * y]) * mul, __uint_as_float(rr[4 * y + 1]) * mul, __uint_as_float(rr[4 * y + 2]) * mul, __uint_as_float(rr[4 * y + 3]) * mul);
      __syncwarp();
      float *dst = (x == 0 ? p.dq : x == 1 ? p.dv : p.dk) + (((size_t)b * (keys ? p.Sk : p.Sq) + (warp & 3) * 32) * p.H + h) * HD + half * 32 + 4 * (lane & 7);
#pragma unroll
      for (int y = 0; y < 32; y += 4) {
        const int r = y + (lane >> 3);
        const float4 v = *reinterpret_cast<const float4 *>(slab + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
        if (r < n_rows) *reinterpret_cast<float4 *>(dst + (size_t)r * p.H * HD) = v;
      }
    }
  }

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (warp == 0 || warp == 8) {
      commit_elected(bar(DRAIN));  // by the lanes that issued the MMAs: the election is deterministic; two arrivals
      for (int t = 0; t < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++t) {
      }
    }
    if (warp == 1 && lane == 0) {  // copies
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == 8) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace

bool tensor_backward_supported(const AttnParams &p) {
  if (option(DF_OPT_DISABLE_TENSOR) != 0) return false;
  if (p.D != HD || p.Sk == 0 || p.Sq == 0 || p.B == 0) return false;
  if (!(p.scale > 0.0f) || !isfinite(p.scale)) return false;
  const uintptr_t bits = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                         reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.d_out) |
                         reinterpret_cast<uintptr_t>(p.d_q) | reinterpret_cast<uintptr_t>(p.d_k) |
                         reinterpret_cast<uintptr_t>(p.d_v);
  if (bits & 15u) return false;
  if ((uint64_t)p.B * p.H * ((uint64_t)(p.Sq > p.Sk ? p.Sq : p.Sk) / BT + 1) > 0x7fffffffull) return false;
  if ((uint64_t)p.Sq * p.H * HD * 4 >= (1ull << 40) || (uint64_t)p.Sk * p.H * HD * 4 >= (1ull << 40)) return false;
  if (p.shift > (1ll << 40) || p.shift < -(1ll << 40)) return false;
  return true;
}

namespace {
// Per device: kernel attributes and SM count, set up once under a lock.
struct DeviceInfo {
  std::once_flag once;
  int n_sm = 0;
  bool ok = false;
};
DeviceInfo g_dev[64];

int device_info(int *n_sm) {
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK || dev < 0 || dev >= 64) return DF_ERR_CUDA;
  DeviceInfo &d = g_dev[dev];
  std::call_once(d.once, [&]() {
    d.ok = cudaFuncSetAttribute(k_attn_bwd_dkdv_tf32_d64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kv::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_dkdv_tf32_d64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kv::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_dq_tf32_d64<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_dq_tf32_d64<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_dq_tf32_d64<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dq::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_tile_tf32_d64<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one::kSmemTotal) == cudaSuccess &&
           cudaFuncSetAttribute(k_attn_bwd_tile_tf32_d64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one::kSmemTotal) == cudaSuccess &&
           cudaDeviceGetAttribute(&d.n_sm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && d.n_sm > 0;
  });
  if (!d.ok) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  *n_sm = d.n_sm;
  return DF_OK;
}

// Side stream of the block backward. The dQ and dK/dV kernels of a block call do not depend on
// each other; with one CTA per SM each, running them on two streams lets the CTAs of one start on
// SMs that the other has already left. The side stream and its fork/join events belong to the
// CALLING THREAD (one set per thread and device), so concurrent callers never record each
// other's events. They are created by df_attn_init or by the thread's first block backward on the
// device (the only place the library creates a CUDA object) and destroyed when the thread exits.
struct SideStreams {
  struct Side { cudaStream_t stream = nullptr; cudaEvent_t fork = nullptr, join = nullptr; bool ok = false, tried = false; };
  Side dev[64];
  ~SideStreams() {
    for (Side &sd : dev)
      if (sd.ok) {  // errors ignored: at process exit the driver may already be gone
        cudaEventDestroy(sd.fork);
        cudaEventDestroy(sd.join);
        cudaStreamDestroy(sd.stream);
      }
  }
  Side *get() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return nullptr;
    Side &sd = dev[d];
    if (!sd.tried) {
      sd.tried = true;
      sd.ok = cudaStreamCreateWithFlags(&sd.stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaEventCreateWithFlags(&sd.fork, cudaEventDisableTiming) == cudaSuccess &&
              cudaEventCreateWithFlags(&sd.join, cudaEventDisableTiming) == cudaSuccess;
    }
    return sd.ok ? &sd : nullptr;
  }
};
thread_local SideStreams t_side;

// Whether an item of the whole-sequence backward goes to a cluster of two CTAs: only where all halves run at once. A CTA costs
// about 5 us beside its steps of 1.8 us, so with a second wave the halves lose (B200, H = 12, causal, both kernels, us, whole /
// halves: S = 256 16.0 / 14.7, 512 22.3 / 18.7, 1024 34.8 / 37.7, 2048 60.8 / 80.3).
bool split_backward(const AttnParams &p, int n_sm) {
  if (p.Sq != p.Sk || p.shift != 0 || p.Sq <= BT) return false;
  return 2ull * ((p.Sq + BT - 1) / BT) * p.B * p.H <= (uint64_t)n_sm;
}

// Events that df_attn_backward_profile asks the launcher to record around the two kernels.
thread_local cudaEvent_t *t_profile_events = nullptr;
}  // namespace

int tensor_backward_init() {
  int n_sm = 0;
  if (device_info(&n_sm) != DF_OK) return DF_ERR_CUDA;
  return t_side.get() ? DF_OK : DF_ERR_CUDA;
}

void tensor_backward_set_profile_events(cudaEvent_t *three_events) { t_profile_events = three_events; }

int tensor_backward(const AttnParams &p, cudaStream_t s) {
  int n_sm = 0;
  if (device_info(&n_sm) != DF_OK) return DF_ERR_CUDA;
  // Row sums fused into the dQ kernel when the caller passes O and a delta buffer to fill instead of
  // ready-made row sums; the dK/dV kernel then runs after the dQ kernel on the same stream.
  const bool fuse = p.delta_in == nullptr && p.o_in != nullptr && p.delta != nullptr;
  if (!fuse && p.delta_in == nullptr) return DF_ERR_INVALID_ARG;
  CUtensorMap tmQk, tmQm, tmGk, tmGm, tmKk, tmKm, tmVk, tmDQ, tmDK, tmDV, tmO;
  if (!encode_head_tile_map(&tmQk, p.q, false, HD, p.B, p.H, p.Sq, BT, false) ||
      !encode_head_tile_map(&tmQm, p.q, false, HD, p.B, p.H, p.Sq, BT / 2, true) ||
      !encode_head_tile_map(&tmGk, p.d_out, false, HD, p.B, p.H, p.Sq, BT, false) ||
      !encode_head_tile_map(&tmGm, p.d_out, false, HD, p.B, p.H, p.Sq, BT / 2, true) ||
      !encode_head_tile_map(&tmKk, p.k, false, HD, p.B, p.H, p.Sk, BT, false) ||
      !encode_head_tile_map(&tmKm, p.k, false, HD, p.B, p.H, p.Sk, BT, true) ||
      !encode_head_tile_map(&tmVk, p.v, false, HD, p.B, p.H, p.Sk, BT, false) ||
      !encode_head_tile_map(&tmDQ, p.d_q, false, HD, p.B, p.H, p.Sq, BT, false, true) ||
      !encode_head_tile_map(&tmDK, p.d_k, false, HD, p.B, p.H, p.Sk, BT, false, true) ||
      !encode_head_tile_map(&tmDV, p.d_v, false, HD, p.B, p.H, p.Sk, BT, false, true) ||
      !encode_head_tile_map(&tmO, fuse ? p.o_in : p.q, false, HD, p.B, p.H, p.Sq, BT, false, true)) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  BwdParams bp;
  bp.lse = p.lse_in;
  bp.delta = fuse ? p.delta : p.delta_in;
  bp.delta_out = fuse ? p.delta : nullptr;
  bp.dq = p.d_q; bp.dk = p.d_k; bp.dv = p.d_v;
  bp.B = p.B; bp.H = p.H; bp.Sq = p.Sq; bp.Sk = p.Sk;
  bp.scale = p.scale;
  bp.scale_log2 = p.scale * kLog2e;
  // The dK/dV kernel subtracts lse / scale before it multiplies by the scale, so both go by one number. It is 1e-37 at least: below, lse / scale may be
  // past fp32, and scale * s is below 1e-37 |s| either way, nothing beside lse unless |s| is 1e30 or more.
  const float kv_scale = fmaxf(p.scale, 1e-37f);
  bp.inv_scale = 1.0f / kv_scale;
  bp.kv_scale_log2 = kv_scale * kLog2e;
  bp.causal = p.causal;
  bp.shift = p.shift;
  bp.status = device_status_ptr();
  // dK/dV: an item per key tile that a query sees (the first ones of a head); dQ: at most one CTA per SM, each walking its share
  const uint32_t key_tiles = (p.Sk + BT - 1) / BT;
  uint32_t seen_tiles = key_tiles;
  if (p.causal) {
    const long long seen_keys = (long long)p.Sq + p.shift;  // keys [0, Sq + shift) have a query
    const long long t = seen_keys <= 0 ? 0 : (seen_keys + BT - 1) / BT;
    if (t < (long long)key_tiles) seen_tiles = (uint32_t)t;
  }
  const uint32_t items_kv = seen_tiles * p.B * p.H;
  bp.zero_tiles = (key_tiles - seen_tiles) * p.B * p.H;
  const int items_q = (int)(((p.Sq + BT - 1) / BT) * p.B * p.H);
  const dim3 grid_q(items_q < n_sm ? items_q : n_sm);
  cudaEvent_t *prof = t_profile_events;
  const bool split = fuse && split_backward(p, n_sm);
  SideStreams::Side *sd = (!fuse && prof == nullptr && option(DF_OPT_BWD_OVERLAP) != 0) ? t_side.get() : nullptr;
  cudaStream_t s_dq = s;
  if (sd) {
    // fork after everything already queued on `s`, join back into `s`: callers see ordinary stream semantics
    if (check_cuda(cudaEventRecord(sd->fork, s)) != DF_OK || check_cuda(cudaStreamWaitEvent(sd->stream, sd->fork, 0)) != DF_OK)
      return DF_ERR_CUDA;
    s_dq = sd->stream;
  }
  if (prof && check_cuda(cudaEventRecord(prof[0], s)) != DF_OK) return DF_ERR_CUDA;
  // A gradient that overwrites what the dQ kernel reads keeps the two kernels apart.
  auto overlap = [](const void *a, uint64_t na, const void *b, uint64_t nb) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + nb && y < x + na;
  };
  const uint64_t q_bytes = (uint64_t)p.B * p.Sq * p.H * HD * 4, k_bytes = (uint64_t)p.B * p.Sk * p.H * HD * 4;
  bool apart = true;
  if (fuse)
    for (const void *g : {(const void *)p.d_k, (const void *)p.d_v})
      for (const void *in : {(const void *)p.q, (const void *)p.k, (const void *)p.v, (const void *)p.d_out, (const void *)p.o_in, (const void *)p.d_q})
        if (overlap(g, k_bytes, in, in == p.k || in == p.v ? k_bytes : q_bytes)) apart = false;
  bp.early = fuse && prof == nullptr && apart && items_kv > 0 && option(DF_OPT_PDL) != 0;
  // One tile of queries and of keys: both kernels' work in one (not when the two are to be timed one by one, or kept apart). It has no pipeline over
  // items, so after some waves of heads the two kernels are faster, sooner where all keys are visible: 25 x 12 heads of 128, 27.0 us (two kernels) against
  // 24.5, all keys 26.4 and 25.7; 36 x 12 33.0 and 32.2, all keys 32.8 and 34.1; 64 x 12 60.4 and 60.1, all keys 60.0 and 63.7.
  if (fuse && prof == nullptr && apart && items_kv > 0 && p.Sq <= BT && p.Sk <= BT && (uint64_t)p.B * p.H <= (p.causal ? 3ull : 2ull) * n_sm) {
    // (d_q may take O's place where one CTA reads O)
    const bool halves = 2 * p.B * p.H <= (uint32_t)n_sm && !overlap(p.d_q, q_bytes, p.o_in, q_bytes);
    const cudaError_t e = launch_kernel(halves ? k_attn_bwd_tile_tf32_d64<true> : k_attn_bwd_tile_tf32_d64<false>, dim3(p.B * p.H * (halves ? 2 : 1)),
                                        dim3(one::kThreads), one::kSmemTotal, s, tmQk, tmGk, tmKk, tmVk, tmQm, tmGm, tmKm, tmO, bp);
    note_launch();
    return check_cuda(e);
  }
  // A profiled call launches each kernel kProfileReps times back to back between its events (the results are the
  // same every time): an event pair around a single launch adds several microseconds to a 70-microsecond kernel.
  const int reps = prof ? kProfileReps : 1;
  for (int rep = 0; (fuse || prof) && rep < reps; ++rep) {
    // (a profiled call with ready-made row sums runs its dQ kernel here too, so that the events split the two kernels)
    const cudaError_t e = split ? launch_clusters(k_attn_bwd_dq_tf32_d64<true, true>, 2, dim3(2 * items_q), dim3(kBwdThreads), dq::kSmemTotal, s,
                                                  tmQk, tmGk, tmKk, tmVk, tmKm, tmDQ, tmO, bp, items_q)
                          : fuse ? launch_kernel(k_attn_bwd_dq_tf32_d64<true, false>, grid_q, dim3(kBwdThreads), dq::kSmemTotal, s,
                                               tmQk, tmGk, tmKk, tmVk, tmKm, tmDQ, tmO, bp, items_q)
                               : launch_kernel(k_attn_bwd_dq_tf32_d64<false, false>, grid_q, dim3(kBwdThreads), dq::kSmemTotal, s,
                                               tmQk, tmGk, tmKk, tmVk, tmKm, tmDQ, tmO, bp, items_q);
    note_launch();
#if defined(DF_ATTN_TRACE) && defined(DF_ATTN_TRACE_DQ)
    if (getenv("DF_ATTN_TRACE_DUMP")) {
      static unsigned long long host[2 * 1024];
      cudaDeviceSynchronize();
      cudaMemcpyFromSymbol(host, g_bwd_trace, sizeof(host));
      for (int slot = 0; slot < 2; ++slot)
        for (int ev = 0; ev < 511; ++ev)
          if (host[slot * 1024 + 2 * ev + 1])
            printf("btrace slot %d ev %llu t %llu\n", slot, host[slot * 1024 + 2 * ev], host[slot * 1024 + 2 * ev + 1] - host[1]);
    }
#endif
    if (check_cuda(e) != DF_OK) return DF_ERR_CUDA;
  }
  if (prof && check_cuda(cudaEventRecord(prof[1], s)) != DF_OK) return DF_ERR_CUDA;
  for (int rep = 0; rep < reps; ++rep) {
    if (items_kv == 0) {  // no key is seen by any query
      if (check_cuda(cudaMemsetAsync(p.d_k, 0, k_bytes, s)) != DF_OK || check_cuda(cudaMemsetAsync(p.d_v, 0, k_bytes, s)) != DF_OK) return DF_ERR_CUDA;
      continue;
    }
    const cudaError_t e = split ? launch_clusters(k_attn_bwd_dkdv_tf32_d64<true>, 2, dim3(2 * items_kv), dim3(kKvThreads), kv::kSmemTotal, s, tmKk,
                                                  tmVk, tmQk, tmGk, tmQm, tmGm, tmDK, tmDV, bp)
                          : launch_kernel(k_attn_bwd_dkdv_tf32_d64<false>, dim3(items_kv), dim3(kKvThreads), kv::kSmemTotal, s, tmKk, tmVk,
                                        tmQk, tmGk, tmQm, tmGm, tmDK, tmDV, bp);
    note_launch();
#if defined(DF_ATTN_TRACE) && !defined(DF_ATTN_TRACE_DQ)
    if (getenv("DF_ATTN_TRACE_DUMP")) {
      static unsigned long long host[2 * 1024];
      cudaDeviceSynchronize();
      cudaMemcpyFromSymbol(host, g_bwd_trace, sizeof(host));
      for (int slot = 0; slot < 2; ++slot)
        for (int ev = 0; ev < 511; ++ev)
          if (host[slot * 1024 + 2 * ev + 1])
            printf("btrace slot %d ev %llu t %llu\n", slot, host[slot * 1024 + 2 * ev], host[slot * 1024 + 2 * ev + 1] - host[1]);
    }
#endif
    if (check_cuda(e) != DF_OK) return DF_ERR_CUDA;
  }
  if (!fuse && !prof) {
    // with ready-made row sums the dQ kernel is independent of the dK/dV kernel
    const cudaError_t e = launch_kernel(k_attn_bwd_dq_tf32_d64<false, false>, grid_q, dim3(kBwdThreads), dq::kSmemTotal, s_dq,
                                        tmQk, tmGk, tmKk, tmVk, tmKm, tmDQ, tmO, bp, items_q);
    note_launch();
    if (check_cuda(e) != DF_OK) return DF_ERR_CUDA;
  }
  if (prof && check_cuda(cudaEventRecord(prof[2], s)) != DF_OK) return DF_ERR_CUDA;
  if (sd) {
    if (check_cuda(cudaEventRecord(sd->join, sd->stream)) != DF_OK || check_cuda(cudaStreamWaitEvent(s, sd->join, 0)) != DF_OK)
      return DF_ERR_CUDA;
  }
  return DF_OK;
}

}  // namespace df

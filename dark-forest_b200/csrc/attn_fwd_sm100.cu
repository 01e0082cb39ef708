// attn_fwd_sm100.cu — fused causal attention forward for B200 (sm_100a): fp32 API (TF32 MMA, head dimension 64) and bf16 (head
// dimension 64, and 128 in split items; attn_fwd_row2_sm100.cu has the rest of bf16).
//
// Replaces the arithmetic of kernel_fused_mha_fwd_tiled (darkforest-cuda/kernels/attention_fused.cu:41-159): O = softmax(scale *
// Q K^T + mask) V per head on [S, H*D] tensors, plus the logsumexp the reference does not save.
//
// One CTA per SM works on items of two slots, A and B, so that the tensor pipe has one slot's products while the other slot is
// in its softmax. A pair item is two query tiles of a head that share every K/V tile; a split item is one query tile whose even
// key tiles go to slot A and odd ones to slot B, the halves combined at the end through shared memory (items half as long, twice
// as many: for few or long items, see split_items). Items are numbered heaviest first, a CTA per item in the grid; a running CTA
// takes over items whose CTA has not started (cluster launch control), so set-up is paid once per SM and SMs of unequal
// speed end together. The pipeline (rings, barrier phases) runs on across items. fp32 sequences of one tile have a kernel of their own, k_attn_fwd_tile.
//   warps 0-3   softmax of slot A, warps 4-7 of slot B: a thread owns a query row. It reads its 128 scores from tensor memory, masks
//               the diagonal tile, keeps a lazily updated running maximum (O and l are rescaled only when the maximum grew by more
//               than 2^8) and writes P = 2^(s * scale * log2e - m) over S, TF32-rounded or packed bf16, handed over in two halves
//   warp 8      TMA: Q and K tiles, and the claims of further items; warp 9 the V tiles. Two-stage rings released by MMA commits.
//               The maps of fp32 tensors are typed TFLOAT32: the copy engine rounds to TF32 in flight (fed raw fp32 the MMA truncates)
//   warp 10     issues S = Q K^T (SS), warp 11 O += P V (TS: P from tensor memory; V is MN-major, in 32-byte atoms for 32-bit
//               elements). With three score buffers the two chains only meet at barriers; with two (head dimension 128) one warp
//               issues both, since the next scores then wait for the PV product that reads the buffer
// Tensor memory: score buffers of 128 columns (three, or two at head dimension 128), then O of slot A and B.
//
// What bounds it: the cycle scores -> softmax -> PV -> scores of a buffer. Per step (128 queries x 128 keys, head dimension 64,
// TF32) 1.85 K cycles of 1.02 K each in the tensor pipe, the exponentials (MUFU) and the shared-memory port. Measured on B200
// against the kernels before (one tile pair per CTA; a persistent form for short sequences; both with two threads per row and
// one issuing warp), H = 12, causal, fp32, us: 1 x 128 8.5 -> 7.1, 1 x 1024 22.1 -> 13.2, 1 x 2048 38.0 -> 20.9, 1 x 4096 72.0 -> 54.2,
// 8 x 1024 41.5 -> 36.4, 1 x 8192 213 -> 178, 1 x 32768 2780 -> 2510-2650; bf16 H = 16, 1 x 8192 228-238 -> 191-217. The parts: issue split
// over two warps 225 -> 175 (8192), bookkeeping between batches cut and P in halves 44.5 -> 37.7 (8 x 1024), split items 34 -> 21
// (2048).
//
// Every mbarrier wait is bounded (sm100_ptx.cuh: mbar_wait) and, in roles of whole warps, decided by the warp together. If one
// gives up, the CTA raises its abort flag, all roles fall through to the common teardown (drain copies and MMAs, free tensor
// memory), and bit 0 of the device status word is set for df_sync_status to report.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include <mutex>
#include <type_traits>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {

PFN_encodeTiled get_encode_tiled() {
  static PFN_encodeTiled fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_encodeTiled>(p);
  }
  return fn;
}

namespace {

using namespace ptx;

constexpr int BM = 128;           // query rows per tile
constexpr int BN = 128;           // keys per K/V tile
constexpr int kStages = 2;        // K and V ring depth
constexpr int kWarpK = 8, kWarpV = 9, kWarpQk = 10, kWarpPv = 11;  // warps 0-3 softmax of slot A, 4-7 of slot B
constexpr int kClaims = 8;        // answers to item claims kept in shared memory (the roles are at most five items apart)
constexpr uint32_t kSlabBytes = 128 * 128;  // 128 rows x 128 B
constexpr uint32_t kTmemCols = 512;
constexpr float kRescaleThreshold = 8.0f;   // log2 units

struct FwdParams {
  void *out;  // fp32 or bf16 elements, see FwdCfg
  float *lse;
  uint32_t B, H, Sq, Sk;
  float scale_log2;
  int causal;
  long long shift;
  uint32_t tiles;    // query tiles per head
  uint32_t n_units;  // per head: pairs of query tiles, or query tiles when `split`
  int claims;        // more items than SMs: CTAs take over items that have not been started
  int wide;          // the output may be stored 32 bytes at a time
  unsigned int *status;
};

// Barrier indices. A parity tells a phase from the one before only, so every waiter sees every phase of its barrier or is known
// to be less than two behind: hence score barriers per slot, and O_LAST for the end of an item.
enum Bar {
  K_FULL = 0, K_EMPTY = 2, V_FULL = 4, V_EMPTY = 6,   // + stage
  Q_FULL = 8, Q_EMPTY = 10,                           // + Q buffer
  O_FULL = 12, O_LAST = 14,                           // + slot: every product, the item's last product
  PV_DONE = 16,                                       // + score buffer (up to 3)
  P_FULL = 19,                                        // + 3 * half of the keys + score buffer
  S_FULL = 25,                                        // + 3 * slot + score buffer: a slot sees every phase of its own three
  X_FULL = 31, X_EMPTY = 32,                          // exchange of the two halves of a split item
  CLAIM = 33,                                         // + answer
  DRAIN = CLAIM + kClaims, NUM_BARS
};

// Compile-time shape of one kernel instance: head dimension, element type of Q/K/V, of O (fp32 partials of bf16 inputs are
// merged by the ring), kind of items. A K-step of an MMA consumes 32 bytes of a row of K, or 8 (TF32) or 16 (bf16) keys.
template <int HD_, bool BF16_, bool OUT_F32_, bool SPLIT_>
struct FwdCfg {
  static constexpr int HD = HD_;
  static constexpr bool SPLIT = SPLIT_;
  static constexpr bool BF16 = BF16_;
  static constexpr bool OUT_F32 = OUT_F32_;
  static constexpr uint32_t kOutElt = OUT_F32_ ? 4 : 2;
  static constexpr uint32_t kElt = BF16_ ? 2 : 4;
  static constexpr uint32_t kSlabs = HD_ * kElt / 128;
  static constexpr uint32_t kBoxElems = 128 / kElt;
  static constexpr uint32_t kTileBytes = kSlabs * kSlabBytes;   // 128 rows x HD
  static constexpr uint32_t kQBufs = SPLIT_ && HD_ == 128 ? 1 : 2;
  static constexpr uint32_t kSmemK = kQBufs * kTileBytes;       // after the Q buffers
  static constexpr uint32_t kSmemV = kSmemK + kStages * kTileBytes;
  static constexpr uint32_t kSmemX = kSmemV + kStages * kTileBytes;             // split items: 2 x 128 rows x HD / 2 floats
  static constexpr uint32_t kSmemMl = kSmemX + (SPLIT_ ? 2 * 128 * (HD_ / 2) * 4 : 0);  // and 2 x 128 (max, sum)
  static constexpr uint32_t kSmemClaims = kSmemMl + (SPLIT_ ? 2 * 128 * 8 : 0);
  static constexpr uint32_t kSmemBars = kSmemClaims + kClaims * 16;
  static constexpr uint32_t kSmemTotal = kSmemBars + NUM_BARS * 8 + 16;  // see the alignment of smem below
  static constexpr uint32_t kFmt = BF16_ ? kFmtBF16 : kFmtTF32;
  static constexpr int kQkSteps = HD_ * kElt / 32;
  static constexpr int kPvSteps = BF16_ ? 8 : 16;
  static constexpr uint32_t kPvStepBytes = BF16_ ? 2048 : 1024;  // 16 or 8 key rows of 128 B
  static constexpr int kBufs = HD_ == 64 ? 3 : 2;                // score buffers in tensor memory
  static constexpr bool kOneIssuer = kBufs == 2;
  static constexpr int kThreads = 32 * (kOneIssuer ? kWarpPv : kWarpPv + 1);
  static constexpr uint32_t kOCols = kBufs * 128;                // TMEM column of O_A; O_B follows at + HD
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// packed fp32 pairs: the pipe's rate is the same, the issue slots are half
__device__ __forceinline__ void fma_pair(float &d0, float &d1, float a0, float a1, float b, float c) {
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void add_pair(float &d0, float &d1, float a0, float a1) {
  asm("{\n\t.reg .b64 ra, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rd, {%0, %1};\n\t"
      "add.rn.f32x2 rd, rd, ra;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1));
}
__device__ __forceinline__ void store_32(void *dst, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
               "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// Number of key tiles visible to the 128-row query tile that starts at q0 (0 if q0 >= Sq).
__host__ __device__ __forceinline__ int visible_kv_tiles(const FwdParams &p, long long q0) {
  if (q0 >= (long long)p.Sq) return 0;
  long long kv_end = p.causal ? q0 + (BM - 1) + p.shift + 1 : (long long)p.Sk;
  if (kv_end > (long long)p.Sk) kv_end = p.Sk;
  if (kv_end < 0) kv_end = 0;
  return (int)((kv_end + BN - 1) / BN);
}

struct Item {
  uint32_t b, h;
  long long qa, qb;  // first query row of slot A and B (negative: nothing of it exists)
  int n0, n1;    // steps of slot A and B
  int kv;        // key tiles that pass through the rings
};
template <bool SPLIT>
__device__ __forceinline__ Item decode_item(const FwdParams &p, uint32_t idx) {
  Item it;
  const uint32_t n_bh = p.B * p.H, bh = idx % n_bh;
  const long long u = (long long)p.n_units - 1 - (long long)(idx / n_bh);  // heaviest first
  it.b = bh / p.H;
  it.h = bh % p.H;
  if (SPLIT) {
    it.qa = it.qb = u * BM;
    it.kv = max(2, visible_kv_tiles(p, u * BM));
    it.n0 = (it.kv + 1) / 2;
    it.n1 = it.kv / 2;
  } else {
    const long long q0 = (2 * u - (long long)(p.tiles & 1)) * BM;  // an odd number of tiles: the first one is alone
    it.qa = q0 < 0 ? 0 : q0;
    it.qb = q0 < 0 ? -BM : q0 + BM;
    it.n0 = max(1, visible_kv_tiles(p, it.qa));
    it.n1 = q0 < 0 ? it.n0 : max(1, visible_kv_tiles(p, it.qb));
    it.kv = max(it.n0, it.n1);
  }
  return it;
}

template <class C>
__global__ void __launch_bounds__(C::kThreads, 1)
k_attn_fwd(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
           const FwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem[];  // tiles first: every one on a 1024-byte boundary, as the swizzle wants
  constexpr int HD = C::HD, NB = C::kBufs;
  constexpr bool SPLIT = C::SPLIT;
  constexpr uint32_t kTileBytes = C::kTileBytes;
  const uint32_t aQ = smem_u32(smem), aK = aQ + C::kSmemK, aV = aQ + C::kSmemV, aClaim = aQ + C::kSmemClaims, aBar = aQ + C::kSmemBars;
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + C::kSmemBars + NUM_BARS * 8);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + C::kSmemBars + NUM_BARS * 8 + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((aQ & 1023u) != 0) {  // not on any driver seen; without this check the tiles would be read wrongly
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    return;
  }

  auto bar = [&](int id) { return aBar + 8 * id; };
  auto load_tile = [&](const CUtensorMap *m, uint32_t dst, int full, const Item &it, long long row) {
    mbar_arrive_expect_tx(bar(full), kTileBytes);
    for (uint32_t sl = 0; sl < C::kSlabs; ++sl)  // rows outside the sequence are zero-filled
      tma_load_4d(dst + sl * kSlabBytes, m, bar(full), (int)(sl * C::kBoxElems), (int)it.h, (int)row, (int)it.b);
  };
  if (warp == kWarpK) {
    for (int i = lane; i < NUM_BARS; i += 32) {
      const uint32_t count = (i >= P_FULL && i < P_FULL + 6) ? 4 : (i == X_FULL || i == X_EMPTY) ? 8 : i == DRAIN ? (C::kOneIssuer ? 1 : 2) : 1;
      mbar_init(bar(i), count);
    }
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    if (lane == 0) {  // the first tiles are under way while the others set up
      const Item it = decode_item<SPLIT>(p, blockIdx.x);
      pdl_wait();
      load_tile(&tmQ, aQ, Q_FULL, it, it.qa);
      load_tile(&tmK, aK, K_FULL, it, 0);
      if (!SPLIT) load_tile(&tmQ, aQ + kTileBytes, Q_FULL + 1, it, it.qb);
      load_tile(&tmV, aV, V_FULL, it, 0);
    }
  }
  if (warp == kWarpQk) {
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  pdl_wait();

  // The item after the k-th: the answer to the k-th claim, or ~0 when there is none (or the wait gave up).
  auto next_item = [&](uint32_t k) -> uint32_t {
    if (!p.claims) return ~0u;
    const int c = (int)(k % kClaims);
    if (!mbar_wait(bar(CLAIM + c), (k / kClaims) & 1, abort_flag)) return ~0u;
    return claim_result(aClaim + 16 * c);
  };

  if (warp == kWarpK) {
    // ------------------------------------------------------------ Q and K copies, claims
    if (lane == 0) {
      uint32_t idx = blockIdx.x, pos = 1;
      bool ok = true;
      for (uint32_t k = 0; idx != ~0u; ++k) {
        const Item it = decode_item<SPLIT>(p, idx);
        auto load_q = [&](uint32_t buf, uint32_t use, long long row) {
          if (use > 0 && !mbar_wait(bar(Q_EMPTY + buf), (use - 1) & 1, abort_flag)) return false;
          load_tile(&tmQ, aQ + buf * kTileBytes, Q_FULL + buf, it, row);
          return true;
        };
        auto load_k = [&](int j) {
          const uint32_t s = pos & 1, use = pos >> 1;
          ++pos;
          if (use > 0 && !mbar_wait(bar(K_EMPTY + s), (use - 1) & 1, abort_flag)) return false;
          load_tile(&tmK, aK + s * kTileBytes, K_FULL + s, it, (long long)j * BN);
          return true;
        };
        if (k > 0) {  // the first item's were requested during set-up
          ok = (SPLIT ? load_q(k % C::kQBufs, k / C::kQBufs, it.qa) : load_q(0, k, it.qa)) && load_k(0);
          if (!SPLIT) ok = ok && load_q(1, k, it.qb);
        }
        for (int j = 1; ok && j < it.kv - 1; ++j) ok = load_k(j);
        if (!ok) break;
        // The next item is asked for when one key tile is left to load: the answer takes about a step, and an item claimed
        // earlier than needed goes to the wrong CTA (at the start of the item: 1 x 4096 62 -> 74 us).
        if (p.claims) {
          const int c = (int)(k % kClaims);
          fence_proxy_async_smem();
          mbar_arrive_expect_tx(bar(CLAIM + c), 16);
          claim_request(aClaim + 16 * c, bar(CLAIM + c));
        }
        if (it.kv > 1 && !load_k(it.kv - 1)) break;
        idx = next_item(k);
      }
    }
  } else if (warp == kWarpV) {
    // ------------------------------------------------------------ V copies
    if (lane == 0) {
      uint32_t idx = blockIdx.x, pos = 1;
      bool ok = true;
      for (uint32_t k = 0; idx != ~0u; ++k) {
        const Item it = decode_item<SPLIT>(p, idx);
        for (int j = k > 0 ? 0 : 1; j < it.kv; ++j, ++pos) {
          const uint32_t s = pos & 1, use = pos >> 1;
          if (use > 0 && !mbar_wait(bar(V_EMPTY + s), (use - 1) & 1, abort_flag)) { ok = false; break; }
          load_tile(&tmV, aV + s * kTileBytes, V_FULL + s, it, (long long)j * BN);
        }
        if (!ok) break;
        idx = next_item(k);
      }
    }
  } else if (warp >= kWarpQk) {
    // ------------------------------------------------------------ MMA issuers
    // A walk over the steps of this CTA's items, in the order that all roles share. In a pair of query tiles step i is key
    // tile i / 2 of tile i % 2 (tile B may have one key tile more: the item's last step); in a split item it is key tile i.
    struct Steps {
      uint32_t k, base, buf, use;  // items begun, ring position of the item's first key tile, score buffer, its uses before
      int i, n, n0, kv;
    };
    auto enter = [&](Steps &w, uint32_t idx) {
      const Item it = decode_item<SPLIT>(p, idx);
      w.n0 = it.n0; w.n = it.n0 + it.n1; w.kv = it.kv;
    };
    auto begin = [&](Steps &w) {
      w.k = w.base = w.use = 0;
      w.i = -1;
      w.buf = NB - 1;
      enter(w, blockIdx.x);
      w.use = ~0u;
    };
    auto advance = [&](Steps &w) -> bool {
      if (++w.buf == NB) { w.buf = 0; ++w.use; }
      if (++w.i < w.n) return true;
      const uint32_t idx = __shfl_sync(0xffffffffu, next_item(w.k), 0);
      if (idx == ~0u) return false;
      w.base += w.kv;
      ++w.k;
      w.i = 0;
      enter(w, idx);
      return true;
    };
    const uint64_t dQ0 = make_smem_desc(aQ, 16, 1024, kSwz128), dK0 = make_smem_desc(aK, 16, 1024, kSwz128);
    const uint64_t dV0 = make_smem_desc(aV, kSlabBytes, C::BF16 ? 1024 : 512, C::BF16 ? kSwz128 : kSwz128B32);
    const uint32_t idesc_qk = make_idesc(C::kFmt, BM, BN, 0, 0), idesc_pv = make_idesc(C::kFmt, BM, HD, 0, 1);
    const uint32_t hiQK = (uint32_t)(dQ0 >> 32), hiV = (uint32_t)(dV0 >> 32);
    // One batch of products (elected lane only): nothing but MMAs, with the operands' buffers known at compile time.
    auto qk_batch = [&](auto tq, auto sk, uint32_t d_tmem) {
      const uint32_t q = (uint32_t)dQ0 + decltype(tq)::value * (kTileBytes >> 4), k = (uint32_t)dK0 + decltype(sk)::value * (kTileBytes >> 4);
#pragma unroll
      for (int kk = 0; kk < C::kQkSteps; ++kk) {
        const uint32_t off = ((kk >> 2) * kSlabBytes + (kk & 3) * 32) >> 4;
        if (C::BF16) mma_f16_ss_lohi(d_tmem, q + off, hiQK, k + off, hiQK, idesc_qk, kk > 0 ? 1u : 0u);
        else mma_tf32_ss_lohi(d_tmem, q + off, hiQK, k + off, hiQK, idesc_qk, kk > 0 ? 1u : 0u);
      }
    };
    auto pv_batch = [&](auto sv, auto half, uint32_t d_tmem, uint32_t a_tmem, uint32_t acc0) {
      const uint32_t v = (uint32_t)dV0 + decltype(sv)::value * (kTileBytes >> 4);
      constexpr int k0 = decltype(half)::value * (C::kPvSteps / 2);
#pragma unroll
      for (int kk = k0; kk < k0 + C::kPvSteps / 2; ++kk) {
        const uint32_t off = (kk * C::kPvStepBytes) >> 4;
        if (C::BF16) mma_f16_ts_lohi(d_tmem, a_tmem + kk * 8, v + off, hiV, idesc_pv, kk > 0 ? 1u : acc0);
        else mma_tf32_ts_lohi(d_tmem, a_tmem + kk * 8, v + off, hiV, idesc_pv, kk > 0 ? 1u : acc0);
      }
    };
    using I0 = std::integral_constant<int, 0>;
    using I1 = std::integral_constant<int, 1>;
    auto last_of_slot = [&](const Steps &w) { return SPLIT ? w.i >= w.n - 2 : (w.i == w.n - 1 || w.i == 2 * (w.n0 - 1)); };
    // S = Q K^T. With one issuer the buffer's last reader, a PV product, was issued before by the same thread.
    auto issue_qk = [&](const Steps &w) -> bool {
      const uint32_t t = SPLIT ? (uint32_t)(w.i & 1) : (uint32_t)((w.i & 1) | (w.i == w.n - 1)), q = SPLIT ? w.k % C::kQBufs : t;
      const uint32_t pos = w.base + (SPLIT ? w.i : w.i >> 1), s = pos & 1;
      if (!C::kOneIssuer && w.use > 0 && !mbar_wait_warp(bar(PV_DONE + w.buf), (w.use - 1) & 1, abort_flag)) return false;
      if ((SPLIT ? w.i == 0 : w.i < 2) && !mbar_wait_warp(bar(Q_FULL + q), (SPLIT ? w.k / C::kQBufs : w.k) & 1, abort_flag)) return false;
      if ((SPLIT || !(w.i & 1)) && !mbar_wait_warp(bar(K_FULL + s), (pos >> 1) & 1, abort_flag)) return false;
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem + w.buf * 128;
      if (elect_one()) {
        if (q == 0) { if (s) qk_batch(I0{}, I1{}, d_tmem); else qk_batch(I0{}, I0{}, d_tmem); }
        else        { if (s) qk_batch(I1{}, I1{}, d_tmem); else qk_batch(I1{}, I0{}, d_tmem); }
        mma_commit(bar(S_FULL + 3 * t + w.buf));
        if (SPLIT || t) mma_commit(bar(K_EMPTY + s));
        if (SPLIT ? w.i == w.n - 1 : last_of_slot(w)) mma_commit(bar(Q_EMPTY + q));
      }
      __syncwarp();
      return true;
    };
    // O += P V, each half of the keys as soon as its probabilities are there
    auto issue_pv = [&](const Steps &w) -> bool {
      const uint32_t t = SPLIT ? (uint32_t)(w.i & 1) : (uint32_t)((w.i & 1) | (w.i == w.n - 1));
      const uint32_t pos = w.base + (SPLIT ? w.i : w.i >> 1), s = pos & 1;
      const uint32_t d_tmem = tmem + C::kOCols + t * HD, a_tmem = tmem + w.buf * 128;
      if ((SPLIT || !(w.i & 1)) && !mbar_wait_warp(bar(V_FULL + s), (pos >> 1) & 1, abort_flag)) return false;
      if (!mbar_wait_warp(bar(P_FULL + w.buf), w.use & 1, abort_flag)) return false;
      tc_fence_after_sync();
      if (elect_one()) {
        if (s) pv_batch(I1{}, I0{}, d_tmem, a_tmem, w.i >= 2 ? 1u : 0u); else pv_batch(I0{}, I0{}, d_tmem, a_tmem, w.i >= 2 ? 1u : 0u);
      }
      __syncwarp();
      if (!mbar_wait_warp(bar(P_FULL + 3 + w.buf), w.use & 1, abort_flag)) return false;
      tc_fence_after_sync();
      if (elect_one()) {
        if (s) pv_batch(I1{}, I1{}, d_tmem, a_tmem, 1u); else pv_batch(I0{}, I1{}, d_tmem, a_tmem, 1u);
        if (!C::kOneIssuer) mma_commit(bar(PV_DONE + w.buf));
        mma_commit(bar(O_FULL + t));
        if (SPLIT || t) mma_commit(bar(V_EMPTY + s));
        if (last_of_slot(w)) mma_commit(bar(O_LAST + t));
      }
      __syncwarp();
      return true;
    };
    Steps w;
    begin(w);
    if (C::kOneIssuer) {
      if (warp == kWarpQk) {
        Steps wq;
        begin(wq);
        bool ok = true, more = true;
        for (int b = 0; ok && more && b < NB; ++b) {
          more = advance(wq);
          if (more) ok = issue_qk(wq);
        }
        while (ok && advance(w)) {
          ok = issue_pv(w);
          if (ok && more) {
            more = advance(wq);
            if (more) ok = issue_qk(wq);
          }
        }
      }
    } else if (warp == kWarpQk) {
      while (advance(w) && issue_qk(w)) {
      }
    } else {
      while (advance(w) && issue_pv(w)) {
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue: a thread owns a query row
    const int t = warp >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tO = tmem + C::kOCols + t * HD + lane_base;
    uint32_t seen = 0, buf0 = 0, o_done = 0;  // phase of each score buffer (one bit), buffer of the item's first step, PVs of this slot before it
    bool ok = true;
    uint32_t idx = blockIdx.x;
    for (uint32_t k = 0; idx != ~0u; ++k) {
      const Item it = decode_item<SPLIT>(p, idx);
      const int nkv = (t ? it.n1 : it.n0);
      const long long i = (t ? it.qb : it.qa) + row;
      const bool row_ok = i >= 0 && i < (long long)p.Sq;
      uint8_t *dst = reinterpret_cast<uint8_t *>(p.out) + (((size_t)it.b * p.Sq + (size_t)(row_ok ? i : 0)) * p.H + it.h) * (HD * C::kOutElt);
      float *lse = p.lse ? p.lse + ((size_t)it.b * p.H + it.h) * p.Sq + (size_t)(row_ok ? i : 0) : nullptr;
      // 32 output columns of this thread's row from c0 on
      auto store_cols = [&](int c0, const float (&v)[32]) {
        uint32_t w[32 * C::kOutElt / 4];
#pragma unroll
        for (int x = 0; x < (int)(32 * C::kOutElt / 4); ++x) w[x] = C::OUT_F32 ? __float_as_uint(v[x]) : pack_bf16x2(v[(2 * x) & 31], v[(2 * x + 1) & 31]);
        uint8_t *d = dst + c0 * C::kOutElt;
#pragma unroll
        for (int x = 0; x < (int)(C::kOutElt); ++x) {
          const uint32_t g[8] = {w[8 * x], w[8 * x + 1], w[8 * x + 2], w[8 * x + 3], w[8 * x + 4], w[8 * x + 5], w[8 * x + 6], w[8 * x + 7]};
          if (p.wide) {
            store_32(d + 32 * x, g);
          } else {
            reinterpret_cast<uint4 *>(d + 32 * x)[0] = make_uint4(g[0], g[1], g[2], g[3]);
            reinterpret_cast<uint4 *>(d + 32 * x)[1] = make_uint4(g[4], g[5], g[6], g[7]);
          }
        }
      };
      long long kmax_ll = p.causal ? i + p.shift + 1 : (long long)p.Sk;
      if (kmax_ll > (long long)p.Sk) kmax_ll = p.Sk;
      if (kmax_ll < 0) kmax_ll = 0;
      const int kmax = (int)kmax_ll;  // keys [0, kmax) are visible to this row
      float m_run = -INFINITY, m_used = -INFINITY;
      float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f, l3 = 0.0f;
      for (int j = 0; j < nkv; ++j) {
        const uint32_t buf = (buf0 + (SPLIT || j < it.n0 ? 2 * j + t : 2 * j)) % NB;
        const uint32_t tS = tmem + buf * 128 + lane_base;
        if (!mbar_wait_warp(bar(S_FULL + 3 * t + buf), (seen >> buf) & 1, abort_flag)) { ok = false; break; }
        seen ^= 1u << buf;
        tc_fence_after_sync();
        const int key0 = (SPLIT ? 2 * j + t : j) * BN;
        uint32_t rs[4][32];
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, rs[c]);
        tmem_wait_ld();
        if (key0 + BN > kmax) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int x = 0; x < 32; ++x)
              if (!(key0 + c * 32 + x < kmax)) rs[c][x] = 0xff800000u;  // -inf: exponentiates to 0
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int x = 0; x < 32; x += 2) mx[c] = fmaxf(mx[c], fmaxf(__uint_as_float(rs[c][x]), __uint_as_float(rs[c][x + 1])));
        m_run = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * p.scale_log2);
        // lazy rescale, decided per warp so that the TMEM accesses stay warp-uniform
        const bool want = (m_run - m_used > kRescaleThreshold) || (m_used == -INFINITY && m_run > -INFINITY);
        if (__any_sync(0xffffffffu, want)) {
          const float alpha = (m_used == -INFINITY) ? 0.0f : ex2_approx(m_used - m_run);
          l0 *= alpha; l1 *= alpha; l2 *= alpha; l3 *= alpha;
          m_used = m_run;
          if (j > 0) {
            if (!mbar_wait_warp(bar(O_FULL + t), (o_done + j - 1) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after_sync();
#pragma unroll 1
            for (int c = 0; c < HD / 16; ++c) {
              uint32_t ro[16];
              asm volatile(
                  "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                  : "=r"(ro[0]), "=r"(ro[1]), "=r"(ro[2]), "=r"(ro[3]), "=r"(ro[4]), "=r"(ro[5]), "=r"(ro[6]), "=r"(ro[7]),
                    "=r"(ro[8]), "=r"(ro[9]), "=r"(ro[10]), "=r"(ro[11]), "=r"(ro[12]), "=r"(ro[13]), "=r"(ro[14]), "=r"(ro[15])
                  : "r"(tO + c * 16)
                  : "memory");
              tmem_wait_ld();
#pragma unroll
              for (int x = 0; x < 16; ++x) ro[x] = __float_as_uint(__uint_as_float(ro[x]) * alpha);
              asm volatile(
                  "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                  ::"r"(tO + c * 16), "r"(ro[0]), "r"(ro[1]), "r"(ro[2]), "r"(ro[3]), "r"(ro[4]), "r"(ro[5]),
                    "r"(ro[6]), "r"(ro[7]), "r"(ro[8]), "r"(ro[9]), "r"(ro[10]), "r"(ro[11]), "r"(ro[12]), "r"(ro[13]), "r"(ro[14]),
                    "r"(ro[15])
                  : "memory");
            }
          }
        }
        const float neg_m = (m_used == -INFINITY) ? 0.0f : -m_used;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
          for (int x = 0; x < 32; x += 4) {
            float e0, e1, e2, e3;
            fma_pair(e0, e1, __uint_as_float(rs[c][x]), __uint_as_float(rs[c][x + 1]), p.scale_log2, neg_m);
            fma_pair(e2, e3, __uint_as_float(rs[c][x + 2]), __uint_as_float(rs[c][x + 3]), p.scale_log2, neg_m);
            e0 = ex2_approx(e0); e1 = ex2_approx(e1); e2 = ex2_approx(e2); e3 = ex2_approx(e3);
            add_pair(l0, l1, e0, e1);
            add_pair(l2, l3, e2, e3);
            if (C::BF16) {
              rs[c >> 1][(c & 1) * 16 + x / 2] = pack_bf16x2(e0, e1);
              rs[c >> 1][(c & 1) * 16 + x / 2 + 1] = pack_bf16x2(e2, e3);
            } else {
              rs[c][x] = tf32_rna_operand(e0); rs[c][x + 1] = tf32_rna_operand(e1);
              rs[c][x + 2] = tf32_rna_operand(e2); rs[c][x + 3] = tf32_rna_operand(e3);
            }
          }
          if (!C::BF16) tmem_st32(tS + c * 32, rs[c]);
          else if (c & 1) tmem_st32(tS + (c >> 1) * 32, rs[c >> 1]);
          if (c & 1) {
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(P_FULL + 3 * (c >> 1) + buf));
          }
        }
      }
      if (!ok) break;
      float l = (l0 + l1) + (l2 + l3);
      if (!mbar_wait_warp(bar(O_LAST + t), k & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      if (SPLIT) {
        // Both slots hold a partial result of the same rows: each hands over the columns that the other one stores.
        float *xo = reinterpret_cast<float *>(smem + C::kSmemX);
        float2 *ml = reinterpret_cast<float2 *>(smem + C::kSmemMl);
        if (k > 0 && !mbar_wait_warp(bar(X_EMPTY), (k - 1) & 1, abort_flag)) { ok = false; break; }
        constexpr int XC = HD / 2;
#pragma unroll 1
        for (int c = 0; c < XC; c += 32) {
          uint32_t ro[32];
          tmem_ld32(tO + (t ^ 1) * XC + c, ro);
          tmem_wait_ld();
          float4 *mine = reinterpret_cast<float4 *>(xo + (t * 128 + row) * XC + c);
#pragma unroll
          for (int x = 0; x < 8; ++x)
            mine[x ^ (row & 7)] = make_float4(__uint_as_float(ro[4 * x]), __uint_as_float(ro[4 * x + 1]), __uint_as_float(ro[4 * x + 2]), __uint_as_float(ro[4 * x + 3]));
        }
        ml[t * 128 + row] = make_float2(m_used, l);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(X_FULL));
        if (!mbar_wait_warp(bar(X_FULL), k & 1, abort_flag)) { ok = false; break; }
        const float2 o = ml[(t ^ 1) * 128 + row];
        const float m = fmaxf(m_used, o.x);
        const float fa = m_used == -INFINITY ? 0.0f : ex2_approx(m_used - m), fb = o.x == -INFINITY ? 0.0f : ex2_approx(o.x - m);
        l = l * fa + o.y * fb;
        const float inv = l > 0.0f ? 1.0f / l : 0.0f, ia = fa * inv, ib = fb * inv;
        // a half without a visible key has factor 0, and its products of zeros with V must not bring in a NaN
        auto mix = [&](float a, float b) { return (ia > 0.0f ? a * ia : 0.0f) + (ib > 0.0f ? b * ib : 0.0f); };
#pragma unroll 1
        for (int c = 0; c < XC; c += 32) {
          uint32_t ro[32];
          tmem_ld32(tO + t * XC + c, ro);
          tmem_wait_ld();
          const float4 *theirs = reinterpret_cast<const float4 *>(xo + ((t ^ 1) * 128 + row) * XC + c);
          float v[32];
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const float4 q = theirs[x ^ (row & 7)];
            v[4 * x] = mix(__uint_as_float(ro[4 * x]), q.x);
            v[4 * x + 1] = mix(__uint_as_float(ro[4 * x + 1]), q.y);
            v[4 * x + 2] = mix(__uint_as_float(ro[4 * x + 2]), q.z);
            v[4 * x + 3] = mix(__uint_as_float(ro[4 * x + 3]), q.w);
          }
          if (row_ok) store_cols(t * XC + c, v);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(X_EMPTY));
        if (row_ok && t == 0 && lse) *lse = l > 0.0f ? (m + lg2_approx(l)) * kLn2 : -INFINITY;
      } else {
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          float v[32];
          uint32_t ro[32];
          tmem_ld32(tO + c * 32, ro);
          tmem_wait_ld();
          // rows that see no key at all: O = 0, lse = -inf (reference guard, attention_fused.cu:104)
#pragma unroll
          for (int x = 0; x < 32; ++x) v[x] = l > 0.0f ? __uint_as_float(ro[x]) * inv : 0.0f;
          if (row_ok) store_cols(c * 32, v);
        }
        if (row_ok && lse) *lse = l > 0.0f ? (m_used + lg2_approx(l)) * kLn2 : -INFINITY;
      }
      tc_fence_before_sync();
      buf0 = (buf0 + it.n0 + it.n1) % NB;
      o_done += nkv;
      idx = __shfl_sync(0xffffffffu, next_item(k), 0);
    }
  }

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    // error path only: give outstanding copies and MMAs a bounded chance to land before the
    // shared and tensor memory of this CTA are released
    if (warp == kWarpQk || (!C::kOneIssuer && warp == kWarpPv)) {
      commit_elected(bar(DRAIN));  // by the lane that issued the MMAs: the election is deterministic
      for (int n = 0; n < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++n) {
      }
    }
    if (warp == kWarpK && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == kWarpQk) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// =========================================================================================
// One tile: at most 128 queries and 128 keys (fp32)
// =========================================================================================
namespace one {
enum Bar { T_QK_FULL = 0, T_V_FULL, T_S_FULL, T_P_FULL, T_O_FULL, T_DRAIN, T_MAX_FULL, T_NUM = T_MAX_FULL + 4 };  // T_MAX_FULL + quarter of the rows
constexpr int kThreads = 512;
constexpr uint32_t kTile = 2 * kSlabBytes;
constexpr uint32_t kMax = 3 * kTile, kSum = kMax + 4 * BM * 4;  // Q, K, V; a row's maximum and sum over each quarter of the keys
constexpr uint32_t kBars = kSum + 4 * BM * 4;
constexpr uint32_t kSmemTotal = kBars + 96 + 1024;
static_assert(T_NUM * 8 <= 80, "barriers overlap the abort flag");
}  // namespace one

// The whole forward of a head whose queries and keys are one tile each: a CTA per head, two to an SM, all sixteen warps compute, a thread a quarter of a
// row; maxima and sums of the rows meet in shared memory. What bounds such a call is latency, and with many heads the ends of items; the kernel
// above has a tile on four warps (the other slot stands idle) in straight code for a whole row per thread, fetched once to run once.
// B200, fp32, S = 128, causal, H = 12, us (above / here): batch 1 6.5 / 6.0, 8 7.1 / 6.3, 12 7.9 / 6.4, 24 12.9 / 8.6, 128 60.8 / 53.2; S = 50, batch 128
// 48.3 / 32.0.
__global__ void __launch_bounds__(one::kThreads, 2)
k_attn_fwd_tile(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                const FwdParams p) {
  using namespace one;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t aQ = smem_u32(smem), aK = aQ + kTile, aV = aQ + 2 * kTile;
  float *sMax = reinterpret_cast<float *>(smem + kMax), *sSum = reinterpret_cast<float *>(smem + kSum);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + kBars + 80);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + kBars + 84);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t h = blockIdx.x % p.H, b = blockIdx.x / p.H;
  auto bar = [&](int id) { return smem_u32(&bars[id]); };
  if (warp == 0) {
    if (lane < T_NUM) mbar_init(bar(lane), lane == T_QK_FULL ? 2 : lane == T_P_FULL ? kThreads : lane >= T_MAX_FULL ? 128 : 1);
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    if (lane == 0) {  // the tiles are under way while the others set up
      pdl_wait();
      auto load = [&](uint32_t dst, const CUtensorMap *m, int id) {
        mbar_arrive_expect_tx(bar(id), kTile);
        for (int sl = 0; sl < 2; ++sl) tma_load_4d(dst + sl * kSlabBytes, m, bar(id), 32 * sl, (int)h, 0, (int)b);
      };
      load(aQ, &tmQ, T_QK_FULL);
      load(aK, &tmK, T_QK_FULL);
      load(aV, &tmV, T_V_FULL);
    }
    __syncwarp();
  }
  if (warp == 8) {
    tmem_alloc(smem_u32(tmem_holder), 256);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tS = *tmem_holder, tO = tS + 128;
  pdl_wait();  // everything above touched only this CTA's shared and tensor memory

  const int row = (warp & 3) * 32 + lane, group = warp >> 2, col0 = group * 32;
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  do {
    if (warp == 0) {  // S = Q K^T
      if (!mbar_wait_warp(bar(T_QK_FULL), 0, abort_flag)) break;
      tc_fence_after_sync();
      const uint64_t dq = make_smem_desc(aQ, 16, 1024, kSwz128), dk = make_smem_desc(aK, 16, 1024, kSwz128);
      if (elect_one()) {
#pragma unroll 1
        for (uint32_t sl = 0; sl < 2; ++sl)
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk) {
            const uint32_t off = sl * (kSlabBytes >> 4) + kk * 2;
            mma_tf32_ss_lohi(tS, (uint32_t)dq + off, (uint32_t)(dq >> 32), (uint32_t)dk + off, (uint32_t)(dk >> 32), make_idesc(kFmtTF32, BM, BN, 0, 0), sl + kk);
          }
        mma_commit(bar(T_S_FULL));
      }
      __syncwarp();
    }
    long long kmax_ll = p.causal ? row + p.shift + 1 : (long long)p.Sk;
    if (kmax_ll > (long long)p.Sk) kmax_ll = p.Sk;
    const int kmax = kmax_ll < 0 ? 0 : (int)kmax_ll, k_end = __reduce_max_sync(0xffffffffu, kmax);  // keys [0, kmax) are visible to this row
    if (!mbar_wait_warp(bar(T_S_FULL), 0, abort_flag)) break;
    tc_fence_after_sync();
    uint32_t r[32];
    float mx = -INFINITY, l0 = 0.0f, l1 = 0.0f;
    if (col0 < k_end) {
      tmem_ld32(tS + lane_base + col0, r);
      tmem_wait_ld();
#pragma unroll
      for (int x = 0; x < 32; ++x) {
        if (!(col0 + x < kmax)) r[x] = 0xff800000u;  // -inf: exponentiates to 0
        mx = fmaxf(mx, __uint_as_float(r[x]));
      }
    }
    sMax[group * BM + row] = mx;
    mbar_arrive(bar(T_MAX_FULL + (warp & 3)));
    if (!mbar_wait_warp(bar(T_MAX_FULL + (warp & 3)), 0, abort_flag)) break;
    const float m = fmaxf(fmaxf(sMax[row], sMax[BM + row]), fmaxf(sMax[2 * BM + row], sMax[3 * BM + row])) * p.scale_log2;
    const float neg_m = m == -INFINITY ? 0.0f : -m;
    if (col0 < k_end) {
#pragma unroll
      for (int x = 0; x < 32; x += 2) {
        const float2 y = fma2(as_float2(r[x], r[x + 1]), make_float2(p.scale_log2, p.scale_log2), make_float2(neg_m, neg_m));
        const float e0 = ex2_approx(y.x), e1 = ex2_approx(y.y);
        l0 += e0;
        l1 += e1;
        r[x] = tf32_rna_operand(e0);
        r[x + 1] = tf32_rna_operand(e1);
      }
    } else {
#pragma unroll
      for (int x = 0; x < 32; ++x) r[x] = 0u;
    }
    tmem_st32(tS + lane_base + col0, r);
    sSum[group * BM + row] = l0 + l1;
    tmem_wait_st();
    tc_fence_before_sync();
    mbar_arrive(bar(T_P_FULL));
    if (!mbar_wait_warp(bar(T_P_FULL), 0, abort_flag)) break;
    if (warp == 0) {  // O = P V
      if (!mbar_wait_warp(bar(T_V_FULL), 0, abort_flag)) break;
      tc_fence_after_sync();
      const uint64_t dv = make_smem_desc(aV, kSlabBytes, 512, kSwz128B32);
      if (elect_one()) {
#pragma unroll 1
        for (uint32_t k4 = 0; k4 < BN / 8; k4 += 4)
#pragma unroll
          for (uint32_t kk = k4; kk < k4 + 4; ++kk)
            mma_tf32_ts_lohi(tO, tS + kk * 8, (uint32_t)dv + kk * (1024 >> 4), (uint32_t)(dv >> 32), make_idesc(kFmtTF32, BM, 64, 0, 1), kk);
        mma_commit(bar(T_O_FULL));
      }
      __syncwarp();
    }
    const float l = (sSum[row] + sSum[BM + row]) + (sSum[2 * BM + row] + sSum[3 * BM + row]);
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    if (group == 0 && p.lse && row < (int)p.Sq) p.lse[((size_t)b * p.H + h) * p.Sq + row] = l > 0.0f ? (m + lg2_approx(l)) * kLn2 : -INFINITY;
    if (!mbar_wait_warp(bar(T_O_FULL), 0, abort_flag)) break;
    tc_fence_after_sync();
    uint32_t ro[16];
    tmem_ld16(tO + lane_base + group * 16, ro);
    tmem_wait_ld();
    // rows that see no key at all: O = 0, lse = -inf (reference guard, attention_fused.cu:104)
#pragma unroll
    for (int x = 0; x < 16; ++x) ro[x] = l > 0.0f ? __float_as_uint(__uint_as_float(ro[x]) * inv) : 0u;
    if (row < (int)p.Sq) {
      float *dst = reinterpret_cast<float *>(p.out) + (((size_t)b * p.Sq + row) * p.H + h) * 64 + group * 16;
#pragma unroll
      for (int x = 0; x < 16; x += 8) {
        const uint32_t g[8] = {ro[x], ro[x + 1], ro[x + 2], ro[x + 3], ro[x + 4], ro[x + 5], ro[x + 6], ro[x + 7]};
        if (p.wide) {
          store_32(dst + x, g);
        } else {
          reinterpret_cast<uint4 *>(dst + x)[0] = make_uint4(g[0], g[1], g[2], g[3]);
          reinterpret_cast<uint4 *>(dst + x)[1] = make_uint4(g[4], g[5], g[6], g[7]);
        }
      }
    }
  } while (false);
  __syncwarp();

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (warp == 0) {
      commit_elected(bar(T_DRAIN));  // by the lane that issued the MMAs: the election is deterministic
      for (int t = 0; t < (1 << 16) && !mbar_try_wait(bar(T_DRAIN), 0); ++t) {
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
    tmem_dealloc(tS, 256);
  }
}

}  // namespace

bool tensor_forward_supported(const AttnParams &p) {
  if (option(DF_OPT_DISABLE_TENSOR) == 1) return false;  // debugging aid: SIMT kernels only
  if (p.Sk == 0 || p.Sq == 0 || p.B == 0) return false;
  if (p.bf16 ? (p.D != 64 && p.D != 128) : (p.D != 64)) return false;
  if (!(p.scale > 0.0f) || !isfinite(p.scale)) return false;
  const uintptr_t bits = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                         reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.out);
  if (bits & 15u) return false;
  if ((uint64_t)p.B * p.H * ((p.Sq + 2 * BM - 1) / (2 * BM)) > 0x7fffffffull) return false;
  if ((uint64_t)p.Sq * p.H * p.D * 4 >= (1ull << 40) || (uint64_t)p.Sk * p.H * p.D * 4 >= (1ull << 40)) return false;
  if (p.shift > (1ll << 40) || p.shift < -(1ll << 40)) return false;
  return true;
}

namespace {
template <class C, bool TILE = false>
int launch_forward(const AttnParams &p, cudaStream_t s) {
  static_assert(!TILE || (!C::BF16 && C::HD == 64), "");
  static std::once_flag once[64];
  static bool ready[64];
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK || dev < 0 || dev >= 64) return DF_ERR_CUDA;
  std::call_once(once[dev], [&]() {
    ready[dev] = TILE ? cudaFuncSetAttribute(k_attn_fwd_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)one::kSmemTotal) == cudaSuccess
                      : cudaFuncSetAttribute(k_attn_fwd<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kSmemTotal) == cudaSuccess;
  });
  CUtensorMap tmQ, tmK, tmV;
  // V is an MN-major operand: 32-bit elements need the 32-byte-atom swizzle, 16-bit ones do not
  if (!ready[dev] || !encode_head_tile_map(&tmQ, p.q, C::BF16, C::HD, p.B, p.H, p.Sq, BM, false) ||
      !encode_head_tile_map(&tmK, p.k, C::BF16, C::HD, p.B, p.H, p.Sk, BN, false) ||
      !encode_head_tile_map(&tmV, p.v, C::BF16, C::HD, p.B, p.H, p.Sk, BN, !C::BF16)) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  FwdParams fp;
  fp.out = p.out;
  fp.lse = p.lse;
  fp.B = p.B; fp.H = p.H; fp.Sq = p.Sq; fp.Sk = p.Sk;
  fp.scale_log2 = p.scale * kLog2e;
  fp.causal = p.causal;
  fp.shift = p.shift;
  fp.wide = ((uintptr_t)p.out & 31u) == 0;
  fp.status = device_status_ptr();
  const uint32_t tiles = (p.Sq + BM - 1) / BM, pairs = (tiles + 1) / 2;
  fp.tiles = tiles;
  fp.n_units = C::SPLIT ? tiles : pairs;
  fp.claims = (uint64_t)fp.n_units * p.B * p.H > (uint64_t)sm_count();
  const cudaError_t err = TILE ? launch_kernel(k_attn_fwd_tile, dim3(p.B * p.H), dim3(one::kThreads), one::kSmemTotal, s, tmQ, tmK, tmV, fp)
                               : launch_kernel(k_attn_fwd<C>, dim3(fp.n_units * p.B * p.H), dim3(C::kThreads), C::kSmemTotal, s, tmQ, tmK, tmV, fp);
  note_launch();
  return check_cuda(err);
}
}  // namespace

namespace {
template <int HD, bool BF16, bool OUT_F32>
int launch_items(const AttnParams &p, bool split, cudaStream_t s) {
  return split ? launch_forward<FwdCfg<HD, BF16, OUT_F32, true>>(p, s) : launch_forward<FwdCfg<HD, BF16, OUT_F32, false>>(p, s);
}

// tensor_forward_supported sees to it that a CTA per pair of query tiles is a valid grid; a CTA per tile can be one too many.
constexpr bool split_grid_fits(uint64_t tiles, uint64_t n_bh) { return tiles * n_bh <= 0x7fffffffull; }
static_assert(split_grid_fits(2, 0x3fffffff) && !split_grid_fits(2, 0x40000000) && split_grid_fits(1, 0x7fffffff), "");

// Pairs of query tiles or split items? Split items are half as long and twice as many: they win where pairs leave SMs without
// work, or a pair of tiles is longer than an SM's share; pairs read K and V half as often. Both times are estimated from
// what an item costs in thousands of cycles (measured slopes over S = 1000..2000 on B200): pairs 8.5 + 1.72 per step,
// split 7 + 1.85; at head dimension 128 8 + 1.8 and 9 + 2. Heaviest items first: the longest item, an SM's share of the sum, and
// the two items of the SM that ends last in the first round. Split has to be 5 % better (10 % at head dimension 128). Measured (pairs / split, us; fp32, causal, H = 12): 1 x 1000 19.3 / 12.9, 1 x 2000 34.0 / 20.8, 1 x 4000 62.8 / 54.0,
// 1 x 6000 96.8 / 102.6, 8 x 1000 37.4 / 45.9.
bool split_items(const AttnParams &p, int n_sm) {
  const int mode = option(DF_OPT_FWD_PERSIST);
  const uint64_t tiles = (p.Sq + BM - 1) / BM, n_bh = (uint64_t)p.B * p.H;
  if (!split_grid_fits(tiles, n_bh)) return false;
  if (mode != 1) return mode == 2;
  if (tiles < 2) return false;
  FwdParams fp;
  fp.Sq = p.Sq; fp.Sk = p.Sk; fp.causal = p.causal; fp.shift = p.shift;
  auto keys = [&](uint64_t tile) { return (double)visible_kv_tiles(fp, (long long)tile * BM); };
  double sum = 0;  // key tiles over all query tiles of a head: their number grows by one per tile between two clipped ends
  for (uint64_t i = 0; i < 8; ++i) sum += keys((2 * i + 1) * tiles / 16) * (double)tiles / 8;
  const bool wide = p.D == 128;
  auto estimate = [&](bool split) {
    const double item0 = split ? (wide ? 9.0 : 7.0) : (wide ? 8.0 : 8.5), step = split ? (wide ? 2.0 : 1.85) : (wide ? 1.8 : 1.72);
    const uint64_t units = split ? tiles : (tiles + 1) / 2, items = units * n_bh;
    auto cost = [&](uint64_t item) {  // items are numbered heaviest first
      const uint64_t above = item / n_bh;  // units ahead of it
      if (split) return item0 + step * keys(tiles - 1 - above);
      const uint64_t last = tiles - 1 - 2 * above;
      return item0 + step * (keys(last) + (last > 0 ? keys(last - 1) : 0.0));
    };
    if (!p.causal) return cost(0) * (double)((items + n_sm - 1) / n_sm);
    double t = (item0 * (double)units + step * sum) * (double)n_bh / n_sm;
    if (cost(0) > t) t = cost(0);
    if (items > (uint64_t)n_sm && cost(n_sm - 1) + cost(n_sm) > t) t = cost(n_sm - 1) + cost(n_sm);
    return t;
  };
  return (wide ? 1.1 : 1.05) * estimate(true) < estimate(false);
}
}  // namespace

int tensor_forward(const AttnParams &p, cudaStream_t s) {
  const int n_sm = sm_count();
  if (n_sm <= 0) return DF_ERR_CUDA;
  const bool split = split_items(p, n_sm);
  // One tile: only a call of many full tiles without a mask has enough steps to a head for the kernel with a pipeline over items (us, that / one tile: 32 x 12
  // heads of 128, all keys, 15.3 / 13.5, 64 x 12 28.2 / 28.3, 128 x 12 55.3 / 57.0; causal 60.8 / 53.2).
  if (!p.bf16 && p.Sq <= BM && p.Sk <= BN && option(DF_OPT_FWD_PERSIST) == 1 && (p.causal || p.Sk <= BN / 2 || (uint64_t)p.B * p.H <= 3ull * n_sm))
    return launch_forward<FwdCfg<64, false, true, false>, true>(p, s);
  if (!p.bf16) return launch_items<64, false, true>(p, split, s);
  if (!split && (p.D == 128 || p.Sq <= BM)) return tensor_forward_row2(p, s);
  if (p.D == 64) return p.out_f32 ? launch_items<64, true, true>(p, split, s) : launch_items<64, true, false>(p, split, s);
  return p.out_f32 ? launch_forward<FwdCfg<128, true, true, true>>(p, s) : launch_forward<FwdCfg<128, true, false, true>>(p, s);
}

}  // namespace df

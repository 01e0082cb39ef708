// attn_fwd_row2_sm100.cu — bf16 attention forward with two threads per query row: head dimension 128 in pairs of query tiles, and
// single-tile sequences of head dimension 64 (attn_fwd_sm100.cu has the other forms and the choice between them).
//
// At head dimension 128 tensor memory holds two score buffers (2 x 128 columns next to two O tiles of 128), so a tile's next
// scores wait for its last PV product and the softmax of a step lies on the critical path; so it does where a sequence is one
// tile. Two threads per query row (sixteen softmax warps) halve that path. One thread per row measured 8-10 % slower at head
// dimension 128 (B200, S = 8192, H = 12: causal 216 against 206 us, all keys 436 against 391 us) and 6.9 against 5.4 us at head
// dimension 64 and S = 96. One CTA per pair of query tiles, heaviest first; that chain bounds it (tensor pipe 57 % of active cycles, S = 16384).
//   warp 16     TMA producer: Q_A, Q_B once, then K_j / V_j tiles (128 keys, 128-byte swizzled slabs) through two-stage rings
//               released by MMA commits
//   warp 17     MMA issuer, order PV_A(j) QK_A(j+1) PV_B(j) QK_B(j+1) ... One election per MMA: batches of nothing but MMAs, which
//               the TF32 kernels use, measured 5-11 % slower here (S = 8192: 224 against 210 us).
//   warps 0-7   softmax of tile A, warps 8-15 of tile B: two threads per query row (64 keys each) read S from tensor memory, mask
//               the diagonal tile, combine their maxima through shared memory, keep a lazily updated running maximum, write P as
//               packed bf16 over S, and finally normalise O and store O and lse.
// Every mbarrier wait is bounded and, in roles of whole warps, decided by the warp together; if one gives up, the CTA raises its abort
// flag, all roles fall through to the common teardown and bit 0 of the device status word is set.
#include <math.h>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {

namespace {

using namespace ptx;

constexpr int BM = 128;        // query rows per tile; a CTA owns two tiles
constexpr int BN = 128;        // keys per K/V tile
constexpr int kStages = 2;     // K and V ring depth
constexpr int kFwdThreads = 576;  // warps 0-15 softmax (8 per tile), 16 TMA, 17 MMA
constexpr uint32_t kSlabBytes = 128 * 128;        // 128 rows x 128 B
constexpr uint32_t kTmemCols = 512;               // S/P: 2 x 128 columns, O: 2 x 64 columns
constexpr float kRescaleThreshold = 8.0f;         // log2 units

struct FwdParams {
  void *out;  // fp32 or bf16 elements, see FwdCfg
  float *lse;
  uint32_t B, H, Sq, Sk;
  float scale_log2;
  int causal;
  long long shift;
  unsigned int *status;
};

// barrier indices; the ones followed by "+ stage" / "+ tile" are pairs
enum Bar {
  Q_FULL = 0,
  K_FULL = 1, K_EMPTY = 3, V_FULL = 5, V_EMPTY = 7,                 // + stage
  S_FULL = 9, P_FULL = 11, O_FULL = 13, X_FULL = 15, L_FULL = 17,   // + tile
  DRAIN = 19, NUM_BARS = 20
};

template <int HD_, bool OUT_F32_>
struct FwdCfg {
  static constexpr int HD = HD_;
  static constexpr bool OUT_F32 = OUT_F32_;                     // O as fp32 (ring partials are merged in fp32) instead of bf16
  static constexpr uint32_t kOutElt = OUT_F32_ ? 4 : 2;
  static constexpr uint32_t kSlabs = HD_ / 64;
  static constexpr uint32_t kBoxElems = 64;                     // elements per 128-byte slab row
  static constexpr uint32_t kTileBytes = kSlabs * kSlabBytes;   // 128 rows x HD
  static constexpr uint32_t kSmemK = 2 * kTileBytes;            // after Q_A, Q_B
  static constexpr uint32_t kSmemV = kSmemK + kStages * kTileBytes;
  static constexpr uint32_t kSmemXch = kSmemV + kStages * kTileBytes;  // per tile: max[2][2][128] + l[2][128] floats
  static constexpr uint32_t kSmemBars = kSmemXch + 2 * 768 * 4;
  static constexpr uint32_t kSmemTotal = kSmemBars + 256 + 1024;
  static constexpr int kQkSteps = HD_ / 16, kPvSteps = 8;       // MMAs of a product: 16 dims or 16 keys each
  static constexpr uint32_t kOCols = 256;                       // TMEM column of O_A; O_B follows at + HD
  // A finished bf16 O tile is staged in the shared memory of its Q tile and written by one tiled bulk store; with fp32 output
  // every thread stores its half row directly.
  static constexpr bool kStoreViaSmem = !OUT_F32_;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Number of key tiles visible to the 128-row query tile that starts at q0 (0 if q0 >= Sq).
__device__ __forceinline__ int visible_kv_tiles(const FwdParams &p, long long q0) {
  if (q0 >= (long long)p.Sq) return 0;
  long long kv_end = p.causal ? q0 + (BM - 1) + p.shift + 1 : (long long)p.Sk;
  if (kv_end > (long long)p.Sk) kv_end = p.Sk;
  if (kv_end < 0) kv_end = 0;
  return (int)((kv_end + BN - 1) / BN);
}

template <class C>
__global__ void __launch_bounds__(kFwdThreads, 1)
k_attn_fwd(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int HD = C::HD;
  constexpr uint32_t kTileBytes = C::kTileBytes;
  const uint32_t aQ = smem_u32(smem), aK = aQ + C::kSmemK, aV = aQ + C::kSmemV;
  float *sXch = reinterpret_cast<float *>(smem + C::kSmemXch);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::kSmemBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + C::kSmemBars + 192);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + C::kSmemBars + 196);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // 1-D grid, (batch, head) fastest: all heads' heaviest (latest) pair of query tiles are
  // dispatched first, then the next lighter one, ... (longest-processing-time-first over the GPU)
  const uint32_t n_bh = p.B * p.H, bh = blockIdx.x % n_bh;
  const int pair = (int)(gridDim.x / n_bh) - 1 - (int)(blockIdx.x / n_bh);
  const uint32_t b = bh / p.H, h = bh % p.H;
  // the HD/2 output elements of query row `row` that the thread of column half `half` stores
  auto out_ptr = [&](long long row, int half) -> uint8_t * {
    return reinterpret_cast<uint8_t *>(p.out) +
           ((((size_t)b * p.Sq + (size_t)row) * p.H + h) * HD + (size_t)half * (HD / 2)) * C::kOutElt;
  };
  const long long q0 = (long long)pair * (2 * BM);         // tile A rows q0.., tile B rows q0+128..
  const int n_kv[2] = {visible_kv_tiles(p, q0), visible_kv_tiles(p, q0 + BM)};
  const int n_max = n_kv[0] > n_kv[1] ? n_kv[0] : n_kv[1];

  pdl_wait();
  // Rows that exist but see no key at all: O = 0, lse = -inf (reference guard, attention_fused.cu:104).
  if (warp < 16) {
    const int t = warp >> 3;
    if (n_kv[t] == 0) {
      const long long i = q0 + t * BM + (warp & 3) * 32 + lane;
      if (i < (long long)p.Sq) {
        const int half = (warp >> 2) & 1;
        float4 *dst = reinterpret_cast<float4 *>(out_ptr(i, half));
#pragma unroll
        for (int x = 0; x < (int)(HD / 2 * C::kOutElt / 16); ++x) dst[x] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (half == 0 && p.lse) p.lse[((size_t)b * p.H + h) * p.Sq + (size_t)i] = -INFINITY;
      }
    }
  }
  if (n_max == 0) return;

  auto bar = [&](int id) { return smem_u32(&bars[id]); };
  // K_j and V_j into ring stage j % kStages
  auto load_kv = [&](int j) {
    const int s = j & 1;
    mbar_arrive_expect_tx(bar(K_FULL + s), kTileBytes);
    for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
      tma_load_4d(aK + s * kTileBytes + sl * kSlabBytes, &tmK, bar(K_FULL + s), (int)(sl * C::kBoxElems), (int)h, j * BN, (int)b);
    mbar_arrive_expect_tx(bar(V_FULL + s), kTileBytes);
    for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
      tma_load_4d(aV + s * kTileBytes + sl * kSlabBytes, &tmV, bar(V_FULL + s), (int)(sl * C::kBoxElems), (int)h, j * BN, (int)b);
  };
  if (warp == 16 && lane == 0) {
    // The producer thread initialises the barriers itself and starts the first copies (Q, then
    // as many K/V tiles as the ring holds) before the CTA-wide set-up barrier, so that their
    // latency overlaps the tensor-memory allocation.
    for (int i = 0; i < NUM_BARS; ++i) {
      const bool wide = (i >= P_FULL && i < P_FULL + 2) || (i >= X_FULL && i < X_FULL + 2) || (i >= L_FULL && i < L_FULL + 2);
      mbar_init(bar(i), wide ? 256 : 1);
    }
    *abort_flag = 0;
    mbar_init_fence();
    mbar_arrive_expect_tx(bar(Q_FULL), 2 * kTileBytes);
    for (int t = 0; t < 2; ++t) {
      // rows beyond Sq are zero-filled by the copy engine
      for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
        tma_load_4d(aQ + t * kTileBytes + sl * kSlabBytes, &tmQ, bar(Q_FULL), (int)(sl * C::kBoxElems), (int)h,
                    (int)(q0 + t * BM), (int)b);
    }
    for (int j = 0; j < n_max && j < kStages; ++j) load_kv(j);
  }
  if (warp == 17) {
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  // TMEM columns: S/P of tile t at [128 t, 128 t + 128), O of tile t at [256 + 64 t, 256 + 64 t + 64)

  if (warp == 16) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      // the first kStages tiles were requested during set-up; every later one waits for its slot
      for (int j = kStages; j < n_max; ++j) {
        const int s = j & 1, use = j >> 1;  // ring stage and how often it has been used before
        if (!mbar_wait(bar(K_EMPTY + s), (use - 1) & 1, abort_flag)) break;
        mbar_arrive_expect_tx(bar(K_FULL + s), kTileBytes);
        for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
          tma_load_4d(aK + s * kTileBytes + sl * kSlabBytes, &tmK, bar(K_FULL + s), (int)(sl * C::kBoxElems), (int)h, j * BN, (int)b);
        if (!mbar_wait(bar(V_EMPTY + s), (use - 1) & 1, abort_flag)) break;
        mbar_arrive_expect_tx(bar(V_FULL + s), kTileBytes);
        for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
          tma_load_4d(aV + s * kTileBytes + sl * kSlabBytes, &tmV, bar(V_FULL + s), (int)(sl * C::kBoxElems), (int)h, j * BN, (int)b);
      }
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp runs this role, warp-uniformly; one elected lane issues the MMA and commit instructions and
    // every wait returns the same answer in all lanes (see elect_one).
    {
      const uint32_t idesc_qk = make_idesc(kFmtBF16, BM, BN, 0, 0), idesc_pv = make_idesc(kFmtBF16, BM, HD, 0, 1);
      bool ok = mbar_wait_warp(bar(Q_FULL), 0, abort_flag);
      const uint64_t dQ = make_smem_desc(aQ, 16, 1024, kSwz128), dK = make_smem_desc(aK, 16, 1024, kSwz128);
      const uint64_t dV = make_smem_desc(aV, kSlabBytes, 1024, kSwz128);
      // S_t = Q_t K_j^T. The last tile to use K_j releases its ring slot.
      auto issue_qk = [&](int t, int j) -> bool {
        const int s = j & 1;
        // tile B reuses the K tile that tile A's product has just waited for (same thread, same phase)
        if ((t == 0 || j >= n_kv[0]) && !mbar_wait_warp(bar(K_FULL + s), (j >> 1) & 1, abort_flag)) return false;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem + t * 128;
        const int last_user = (j < n_kv[1]) ? 1 : 0;
        const uint64_t da = dQ + (uint64_t)(t * (kTileBytes >> 4)), db = dK + (uint64_t)(s * (kTileBytes >> 4));
#pragma unroll
        for (int kk = 0; kk < C::kQkSteps; ++kk) {
          const uint64_t off = (uint64_t)(((kk >> 2) * kSlabBytes + (kk & 3) * 32) >> 4);
          if (elect_one()) mma_f16_ss(d_tmem, da + off, db + off, idesc_qk, kk > 0);
        }
        commit_elected(bar(S_FULL + t));
        if (t == last_user) commit_elected(bar(K_EMPTY + s));
        return true;
      };
      // O_t += P_t V_j
      auto issue_pv = [&](int t, int j) -> bool {
        const int s = j & 1;
        if ((t == 0 || j >= n_kv[0]) && !mbar_wait_warp(bar(V_FULL + s), (j >> 1) & 1, abort_flag)) return false;
        if (!mbar_wait_warp(bar(P_FULL + t), j & 1, abort_flag)) return false;
        tc_fence_after_sync();
        // P occupies 8 TMEM columns per K-step (16 packed bf16 values)
        const uint32_t d_tmem = tmem + C::kOCols + t * HD, a_tmem = tmem + t * 128;
        const int last_user = (j < n_kv[1]) ? 1 : 0;
        const uint64_t db = dV + (uint64_t)(s * (kTileBytes >> 4));
#pragma unroll
        for (int kk = 0; kk < C::kPvSteps; ++kk)
          if (elect_one()) mma_f16_ts(d_tmem, a_tmem + kk * 8, db + (uint64_t)(kk * (2048 >> 4)), idesc_pv, (j > 0 || kk > 0) ? 1u : 0u);
        commit_elected(bar(O_FULL + t));
        if (t == last_user) commit_elected(bar(V_EMPTY + s));
        return true;
      };
      if (ok && n_kv[0] > 0) ok = issue_qk(0, 0);
      if (ok && n_kv[1] > 0) ok = issue_qk(1, 0);
      for (int j = 0; ok && j < n_max; ++j) {
        for (int t = 0; ok && t < 2; ++t) {
          if (j < n_kv[t]) {
            ok = issue_pv(t, j);
            if (ok && j + 1 < n_kv[t]) ok = issue_qk(t, j + 1);  // overwrites P_t(j) after PV_t(j) has read it
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue
    // Warps 0-7 serve tile A, 8-15 tile B. Within a tile two warpgroups share every query row:
    // warps 0-3 own key columns 0-63 of the K/V tile, warps 4-7 columns 64-127 (a warp reads TMEM
    // lanes 32*(w%4)..+31). The row maximum is combined with the partner thread through shared
    // memory, after which both take identical rescale decisions.
    const int t = warp >> 3;
    const int quarter = warp & 3, half = (warp >> 2) & 1;
    const int row = quarter * 32 + lane;
    const long long i = q0 + t * BM + row;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem + t * 128, tO = tmem + C::kOCols + t * HD;
    const int col0 = half * 64;
    const int nkv = n_kv[t];
    float *xch = sXch + t * 768;
    long long kmax_ll = p.causal ? i + p.shift + 1 : (long long)p.Sk;
    if (kmax_ll > (long long)p.Sk) kmax_ll = p.Sk;
    if (kmax_ll < 0) kmax_ll = 0;
    const int kmax = (int)kmax_ll;  // keys [0, kmax) are visible to this row
    float m_run = -INFINITY, m_used = -INFINITY;
    float l0 = 0.0f, l1 = 0.0f, l2 = 0.0f, l3 = 0.0f;
    bool ok = nkv > 0;
    for (int j = 0; j < nkv; ++j) {
      if (!mbar_wait_warp(bar(S_FULL + t), j & 1, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      const int key0 = j * BN + col0;
      const bool need_mask = key0 + 64 > kmax;
      // single pass: the thread's 64 scores stay in registers from the maximum to the exponentials
      uint32_t ra[32], rb[32];
      tmem_ld32(tS + lane_base + col0, ra);
      tmem_ld32(tS + lane_base + col0 + 32, rb);
      tmem_wait_ld();
      if (need_mask) {
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          if (!(key0 + x < kmax)) ra[x] = 0xff800000u;  // -inf: exponentiates to 0
          if (!(key0 + 32 + x < kmax)) rb[x] = 0xff800000u;
        }
      }
      float mx_half;
      {
        float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
          mx0 = fmaxf(mx0, fmaxf(__uint_as_float(ra[x]), __uint_as_float(rb[x])));
          mx1 = fmaxf(mx1, fmaxf(__uint_as_float(ra[x + 1]), __uint_as_float(rb[x + 1])));
          mx2 = fmaxf(mx2, fmaxf(__uint_as_float(ra[x + 2]), __uint_as_float(rb[x + 2])));
          mx3 = fmaxf(mx3, fmaxf(__uint_as_float(ra[x + 3]), __uint_as_float(rb[x + 3])));
        }
        mx_half = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      }
      // exchange the half-row maxima (double-buffered by tile parity)
      float *xmax = xch + (j & 1) * 256;
      xmax[half * 128 + row] = mx_half;
      mbar_arrive(bar(X_FULL + t));
      if (!mbar_wait_warp(bar(X_FULL + t), j & 1, abort_flag)) { ok = false; break; }
      const float mx = fmaxf(mx_half, xmax[(half ^ 1) * 128 + row]);
      m_run = fmaxf(m_run, mx * p.scale_log2);
      // lazy rescale, decided per warp so that the TMEM accesses stay warp-uniform; the partner
      // warp sees the same rows and the same maxima, hence takes the same decision
      const bool want = (m_run - m_used > kRescaleThreshold) || (m_used == -INFINITY && m_run > -INFINITY);
      if (__any_sync(0xffffffffu, want)) {
        const float alpha = (m_used == -INFINITY) ? 0.0f : ex2_approx(m_used - m_run);
        l0 *= alpha; l1 *= alpha; l2 *= alpha; l3 *= alpha;
        m_used = m_run;
        if (j > 0) {
          if (!mbar_wait_warp(bar(O_FULL + t), (j - 1) & 1, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
          // each half rescales HD/2 of the O columns, 16 at a time to stay within the register budget
#pragma unroll 1
          for (int c = 0; c < HD / 32; ++c) {
            uint32_t ro[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(ro[0]), "=r"(ro[1]), "=r"(ro[2]), "=r"(ro[3]), "=r"(ro[4]), "=r"(ro[5]), "=r"(ro[6]), "=r"(ro[7]),
                  "=r"(ro[8]), "=r"(ro[9]), "=r"(ro[10]), "=r"(ro[11]), "=r"(ro[12]), "=r"(ro[13]), "=r"(ro[14]), "=r"(ro[15])
                : "r"(tO + lane_base + half * (HD / 2) + c * 16)
                : "memory");
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < 16; ++x) ro[x] = __float_as_uint(__uint_as_float(ro[x]) * alpha);
            asm volatile(
                "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                ::"r"(tO + lane_base + half * (HD / 2) + c * 16), "r"(ro[0]), "r"(ro[1]), "r"(ro[2]), "r"(ro[3]), "r"(ro[4]), "r"(ro[5]),
                  "r"(ro[6]), "r"(ro[7]), "r"(ro[8]), "r"(ro[9]), "r"(ro[10]), "r"(ro[11]), "r"(ro[12]), "r"(ro[13]), "r"(ro[14]),
                  "r"(ro[15])
                : "memory");
          }
        }
      }
      const float neg_m = (m_used == -INFINITY) ? 0.0f : -m_used;
      // P = 2^(s*scale_log2 - m), written over S as packed bf16 pairs (keys
      // 2c, 2c+1 in TMEM column c; every thread of the row loaded its scores before the exchange
      // barrier above, so overwriting the partner's S columns is safe)
#pragma unroll
      for (int x = 0; x < 32; x += 4) {
        const float e0 = ex2_approx(fmaf(__uint_as_float(ra[x]), p.scale_log2, neg_m));
        const float e1 = ex2_approx(fmaf(__uint_as_float(ra[x + 1]), p.scale_log2, neg_m));
        const float e2 = ex2_approx(fmaf(__uint_as_float(ra[x + 2]), p.scale_log2, neg_m));
        const float e3 = ex2_approx(fmaf(__uint_as_float(ra[x + 3]), p.scale_log2, neg_m));
        ra[x / 2] = pack_bf16x2(e0, e1);
        ra[x / 2 + 1] = pack_bf16x2(e2, e3);
        l0 += e0; l1 += e1; l2 += e2; l3 += e3;
      }
#pragma unroll
      for (int x = 0; x < 32; x += 4) {
        const float e0 = ex2_approx(fmaf(__uint_as_float(rb[x]), p.scale_log2, neg_m));
        const float e1 = ex2_approx(fmaf(__uint_as_float(rb[x + 1]), p.scale_log2, neg_m));
        const float e2 = ex2_approx(fmaf(__uint_as_float(rb[x + 2]), p.scale_log2, neg_m));
        const float e3 = ex2_approx(fmaf(__uint_as_float(rb[x + 3]), p.scale_log2, neg_m));
        ra[16 + x / 2] = pack_bf16x2(e0, e1);   // ra[0..15] hold this thread's first 32 keys
        ra[16 + x / 2 + 1] = pack_bf16x2(e2, e3);
        l0 += e0; l1 += e1; l2 += e2; l3 += e3;
      }
      tmem_st32(tS + lane_base + half * 32, ra);
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(bar(P_FULL + t));
    }
    // combine the two half-row sums, then normalise and store 32 of the 64 output columns each
    float l = (l0 + l1) + (l2 + l3);
    if (ok) {
      float *xl = xch + 512;
      xl[half * 128 + row] = l;
      mbar_arrive(bar(L_FULL + t));
      if (!mbar_wait_warp(bar(L_FULL + t), 0, abort_flag)) ok = false;
      else l += xl[(half ^ 1) * 128 + row];
    }
    if (ok && mbar_wait_warp(bar(O_FULL + t), (nkv - 1) & 1, abort_flag)) {
      tc_fence_after_sync();
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
      const bool row_ok = i < (long long)p.Sq;
      uint8_t *dst = out_ptr(row_ok ? i : 0, half);
      // staging address of this thread's half row inside the (no longer needed) Q tile: the
      // 128-byte swizzle of the store's tensor map puts 16-byte chunk c of row r at c ^ (r % 8)
      constexpr uint32_t kHalfBytes = HD / 2 * C::kOutElt;
      const uint32_t st_off = (uint32_t)half * kHalfBytes;
      uint8_t *stage = smem + t * kTileBytes + (st_off / 128) * kSlabBytes + row * 128;
      const uint32_t chunk0 = (st_off % 128) / 16;
#pragma unroll 1
      for (int c = 0; c < HD / 64; ++c) {   // 32 O columns per step
        uint32_t ro[32];
        tmem_ld32(tO + lane_base + half * (HD / 2) + c * 32, ro);
        tmem_wait_ld();
        if (C::kStoreViaSmem) {
          if (!C::OUT_F32) {
#pragma unroll
            for (int x = 0; x < 4; ++x)
              *reinterpret_cast<uint4 *>(stage + (((chunk0 + c * 4 + x) ^ (row & 7)) << 4)) =
                  make_uint4(pack_bf16x2(__uint_as_float(ro[8 * x]) * inv, __uint_as_float(ro[8 * x + 1]) * inv),
                             pack_bf16x2(__uint_as_float(ro[8 * x + 2]) * inv, __uint_as_float(ro[8 * x + 3]) * inv),
                             pack_bf16x2(__uint_as_float(ro[8 * x + 4]) * inv, __uint_as_float(ro[8 * x + 5]) * inv),
                             pack_bf16x2(__uint_as_float(ro[8 * x + 6]) * inv, __uint_as_float(ro[8 * x + 7]) * inv));
          } else {
#pragma unroll
            for (int x = 0; x < 8; ++x)
              *reinterpret_cast<float4 *>(stage + (((chunk0 + c * 8 + x) ^ (row & 7)) << 4)) =
                  make_float4(__uint_as_float(ro[4 * x]) * inv, __uint_as_float(ro[4 * x + 1]) * inv,
                              __uint_as_float(ro[4 * x + 2]) * inv, __uint_as_float(ro[4 * x + 3]) * inv);
          }
        } else if (row_ok) {
          if (!C::OUT_F32) {
            uint4 *d4 = reinterpret_cast<uint4 *>(dst + c * 64);
#pragma unroll
            for (int x = 0; x < 4; ++x)
              d4[x] = make_uint4(pack_bf16x2(__uint_as_float(ro[8 * x]) * inv, __uint_as_float(ro[8 * x + 1]) * inv),
                                 pack_bf16x2(__uint_as_float(ro[8 * x + 2]) * inv, __uint_as_float(ro[8 * x + 3]) * inv),
                                 pack_bf16x2(__uint_as_float(ro[8 * x + 4]) * inv, __uint_as_float(ro[8 * x + 5]) * inv),
                                 pack_bf16x2(__uint_as_float(ro[8 * x + 6]) * inv, __uint_as_float(ro[8 * x + 7]) * inv));
          } else {
            float4 *d4 = reinterpret_cast<float4 *>(dst + c * 128);
#pragma unroll
            for (int x = 0; x < 8; ++x)
              d4[x] = make_float4(__uint_as_float(ro[4 * x]) * inv, __uint_as_float(ro[4 * x + 1]) * inv,
                                  __uint_as_float(ro[4 * x + 2]) * inv, __uint_as_float(ro[4 * x + 3]) * inv);
          }
        }
      }
      if (row_ok) {
        if (half == 0 && p.lse)
          p.lse[((size_t)b * p.H + h) * p.Sq + (size_t)i] =
              l > 0.0f ? (m_used + lg2_approx(l)) * kLn2 : -INFINITY;
      }
      if (C::kStoreViaSmem) {
        // all 256 threads of the tile have staged their rows (second phase of the tile's
        // row-sum barrier); one thread then hands the tile to the copy engine, which drops rows
        // beyond Sq
        fence_proxy_async_smem();
        mbar_arrive(bar(L_FULL + t));
        if ((warp & 7) == 0 && lane == 0 && mbar_wait(bar(L_FULL + t), 1, abort_flag)) {
          for (uint32_t sl = 0; sl < C::kSlabs; ++sl)
            tma_store_4d(&tmO, aQ + t * kTileBytes + sl * kSlabBytes, (int)(sl * C::kBoxElems), (int)h,
                         (int)(q0 + t * BM), (int)b);
          tma_store_commit();
          tma_store_wait_read_all();
        }
      }
    }
  }

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag != 0u) {
    // error path only: give outstanding copies and MMAs a bounded chance to land before the
    // shared and tensor memory of this CTA are released
    if (warp == 17) {
      commit_elected(bar(DRAIN));  // by the lane that issued the MMAs: the election is deterministic
      for (int n = 0; n < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++n) {
      }
    }
    if (warp == 16 && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (global_timer_ns() - t0 < 2000000ull) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == 17) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace

namespace {
template <class C>
int launch_forward(const AttnParams &p, cudaStream_t s) {
  static bool attr_set[64] = {false};
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK) return DF_ERR_CUDA;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (check_cuda(cudaFuncSetAttribute(k_attn_fwd<C>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)C::kSmemTotal)) != DF_OK)
      return DF_ERR_CUDA;
    attr_set[dev] = true;
  }
  CUtensorMap tmQ, tmK, tmV, tmO;
  // V is an MN-major operand: 32-bit elements need the 32-byte-atom swizzle, 16-bit ones do not
  if (!encode_head_tile_map(&tmQ, p.q, true, C::HD, p.B, p.H, p.Sq, BM, false) ||
      !encode_head_tile_map(&tmK, p.k, true, C::HD, p.B, p.H, p.Sk, BN, false) ||
      !encode_head_tile_map(&tmV, p.v, true, C::HD, p.B, p.H, p.Sk, BN, false) ||
      !encode_head_tile_map(&tmO, C::kStoreViaSmem ? p.out : p.q, true, C::HD, p.B, p.H, p.Sq, BM, false, true)) {
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
  fp.status = device_status_ptr();
  const dim3 grid(((p.Sq + 2 * BM - 1) / (2 * BM)) * p.B * p.H);
  launch_kernel(k_attn_fwd<C>, grid, dim3(kFwdThreads), C::kSmemTotal, s, tmQ, tmK, tmV, tmO, fp);
  note_launch();
  return check_cuda(cudaGetLastError());
}
}  // namespace

int tensor_forward_row2(const AttnParams &p, cudaStream_t s) {
  if (p.D == 64) return p.out_f32 ? launch_forward<FwdCfg<64, true>>(p, s) : launch_forward<FwdCfg<64, false>>(p, s);
  return p.out_f32 ? launch_forward<FwdCfg<128, true>>(p, s) : launch_forward<FwdCfg<128, false>>(p, s);
}

}  // namespace df

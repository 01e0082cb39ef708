// attn_split_sm100.cu - fp32 attention in full fp32 precision on the tensor cores (sm_100a), for head sizes that the TF32 kernels do not take.
//
// Same mathematics as attn_simt.cu (darkforest-cuda/kernels/attention_fused.cu:41-159, 390-516), for sequences of more than kMinSteps - 1 steps.
// Every fp32 operand is cut into three bf16 parts, a = a1 + a2 + a3, each what is left rounded to bf16: |a2| <= 2^-8 |a|, |a3| <= 2^-17 |a|, and nothing
// is left after the third. A product is six of the nine products of parts (a1 b1, a1 b2, a2 b1, a2 b2, a1 b3, a3 b1), the small ones first; what is left
// out, a2 b3 + a3 b2 + a3 b3, is at most 2^-24 of |a| |b| and of either sign. (Parts cut off by truncation would leave out up to 2^-21, always of the sign
// of a b: dQ 10.4e-7 off with operands near 1 + 2^-7, 2.0e-7 rounded.) The tensor cores add into fp32 with truncation, so sums there are kept short: a
// step's 64 rows are contracted in tensor memory and added to fp32 registers, rounded to nearest, and scores have two accumulators, one of which takes
// only half of the largest product. The bounds hold for operands of 2^-101 and more, where all parts are normal numbers; a smaller one loses bits that are
// below 2^-133. An infinity has no parts (inf - inf), so rows with a result that is not finite are formed again in fp32 arithmetic (fp32_row).
// Relative error (2-norm) against 64 bits, normal inputs, this / attn_simt.cu, in 1e-7:
//   B x H x S x D                  O            logsumexp      dQ           dK           dV
//   2 x 8 x 1000 x 128, causal     1.3 / 2.7    0.31 / 0.28    2.7 / 4.1    3.1 / 8.0    2.5 / 7.8
//   2 x 6 x  400 x  32, causal     1.0 / 1.8    0.30 / 0.29    2.2 / 3.1    2.5 / 5.1    2.2 / 5.0
//   1 x 8 x  333 x  80, causal     1.4 / 1.9    0.38 / 0.34    2.7 / 3.2    2.9 / 4.9    2.4 / 4.7
//   1 x 4 x  260 x 112             1.5 / 3.2    0.29 / 0.33    2.7 / 4.4    2.8 / 4.8    2.5 / 4.6
//   1 x 4 x 300 x 128, causal, operands near 1 + 2^-7
//                                  1.0 / 2.3    0.30 / 0.34    2.0 / 3.4    2.3 / 4.9    1.8 / 4.7
// (of the logsumexp 0.22 are its own rounding to fp32)
//
// Four passes from one text, `Pass`:
//               resident rows A1, A2    streamed rows B1, B2    T (per step)                        result R
//   FORWARD     queries  Q              keys     K, V           P = 2^(s - running max)             O   = sum T V, by rows' alpha, over sums
//   DQ          queries  Q, dO          keys     K, V           dS = P (dP - delta)                 dQ  = scale sum T K
//   DK          keys     K, V           queries  Q, dO          dS^T                                dK  = scale sum T Q
//   DV          keys     K              queries  Q, dO          P^T                                 dV  = sum T dO
// with S = A1 B1^T and, in DQ and DK, dP = A2 B2^T. A CTA owns 128 resident rows of one head (the lanes of tensor memory) and walks the other side in
// steps of 64 rows. The three passes of a backward share a launch, heaviest blocks first.
//   warps 0-7   compute: warp w holds rows 32 (w % 4) + 16 (w / 4) .. + 15 whole (16x256b fragments: four lanes per row), so maxima and sums stay in
//               the warp; it turns S (and dP) into T, cut in three, and adds R to its registers
//   warps 8-14  streamed rows: fp32 from global memory, cut, into 128-byte-swizzled tiles that serve as K-major operand (S, dP) and as MN-major one (R)
//   warp 15     issues the products
// Of a resident tile two parts lie in tensor memory and the third, which only one product reads, in shared memory: an operand A read from there
// costs as much of the port as the 64-column product that reads it may take in all. dK and dV are passes of their own, at the price of one more S:
// tensor memory does not hold two results beside K and V.
//
// What bounds it: a step of FORWARD or DV is 12 products of 128 x 64 x DP, 3.1 K cycles of tensor pipe at DP = 128, and takes 4.5 K; of DQ or DK
// 18, 4.9 K, and takes 8.5 K: the issue (50 cycles an MMA of 64 columns, 32 in the pipe), and in DQ and DK the way from dP to T, which the pipe waits
// for since tensor memory is full. Instructions count too (six of sixteen warps' issue slots go into the cuts), hence two fp32 operations per
// instruction wherever they come in pairs.
// Measured on B200, us, this / attn_simt.cu, forward and backward with the row sums, causal, 2 x 8 x 1000 x 128: 39 / 115, 122 / 371; 1 x 4 x 700 x 96:
// 18 / 42, 32 / 72; 2 x 8 x 500 x 96: 18 / 36, 38 / 88; 1 x 8 x 1000 x 16: 15 / 30, 36 / 66; 1 x 6 x 192 x 128: 13.5 / 17.7, 24 / 30.
#include <math.h>

#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {
namespace {

using namespace ptx;

// MMAs that all lanes of the warp come to and that are issued by the lane whose `mine` is set (elect_one). Without a branch around them the descriptors
// are computed for the whole warp at once: an election and a branch around a batch took 63 cycles an MMA of 64 columns, this form 52, of the pipe's 32.
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate, uint32_t mine) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tmov.b64 db, {%2, %3};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(mine)
      : "memory");
}
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate, uint32_t mine) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\tmov.b64 da, {%1, %2};\n\tmov.b64 db, {%3, %4};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(mine)
      : "memory");
}
template <int N> struct ic { static constexpr int value = N; };
enum Pass { FORWARD, DQ, DK, DV };

constexpr int BM = 128;  // resident rows of a CTA
constexpr int BN = 64;   // streamed rows of a step
constexpr int kStreamWarps = 7, kMmaWarp = 8 + kStreamWarps;
// Registers: the launch gives 128 to each thread of four warpgroups; the two of the compute warps take over 40 from each thread of the others.
constexpr int kLaunchRegs = 128, kComputeRegs = 168, kOtherRegs = 88;
static_assert(2 * kComputeRegs + 2 * kOtherRegs <= 4 * kLaunchRegs, "setmaxnreg waits for registers that the block was not launched with");
template <int N> __device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_less() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kComputeThreads = 256, kStreamThreads = 32 * kStreamWarps;
constexpr uint32_t kTmemCols = 512;

// DP: head size rounded up to 32, 64, 96 or 128; the columns beyond the head size are zeros.
template <int DP_, Pass PASS_>
struct Cfg {
  static constexpr int DP = DP_;
  static constexpr Pass PASS = PASS_;
  static constexpr bool TWO = PASS_ == DQ || PASS_ == DK;             // dP is needed
  static constexpr bool ROWS_ARE_KEYS = PASS_ == DK || PASS_ == DV;
  static constexpr int KS = DP_ / 16;                                  // K-steps of a product over the head dimension
  static constexpr uint32_t SLABS = (DP_ + 63) / 64;                   // 128-byte slabs (64 bf16) of a row
  static constexpr uint32_t kSlab = BN * 128, kPart = SLABS * kSlab, kTile = 3 * kPart;  // streamed tile
  static constexpr uint32_t kSlabA = BM * 128, kPartA = SLABS * kSlabA;                  // third part of a resident tile
  static constexpr int ST1 = 2, ST2 = TWO && SLABS == 2 ? 1 : 2;                         // shared memory is full at two slabs
  static constexpr int NSTATS = PASS_ == DK ? 3 : PASS_ == DV ? 2 : 0;                   // values staged per streamed row
  static constexpr uint32_t oB1 = (TWO ? 2 : 1) * kPartA, oB2 = oB1 + ST1 * kTile, oStats = oB2 + ST2 * kTile;
  static constexpr uint32_t oBars = oStats + 3 * NSTATS * BN * 4, kSmem = oBars + 256 + 1024;  // 1024: tiles begin on the next 1024-byte boundary
  // Tensor memory: the first two parts of A1 (and A2), then
  //   one product: two regions of 96 columns that hold S and then T, the scores' second accumulator, R
  //   two:         S and dP side by side, T over them; R, whose columns hold the second accumulators until R is formed
  static constexpr uint32_t kPartCols = DP_ / 2, cA1 = 0, cA2 = 2 * kPartCols, cX0 = (TWO ? 4 : 2) * kPartCols, cX1 = cX0 + (TWO ? 0 : 96);
  static constexpr uint32_t cDP = cX0 + 64, cS2 = TWO ? cX0 + 128 : cX1 + 96, cDP2 = cS2 + 64, cR = TWO ? cS2 : cS2 + 64;
  static_assert(cR + (TWO && DP_ < 128 ? 128 : DP_) <= kTmemCols, "tensor memory");
  static_assert(kSmem <= 227 * 1024, "shared memory");
  // shape of the streaming warps' accesses: G groups of four dims a row, RPW rows per warp and access, RPA rows per access, U accesses per tile
  static constexpr int G = DP_ / 4, RPW = 32 / G, RPA = kStreamWarps * RPW, U = (BN + RPA - 1) / RPA;
};

enum Bar { A_READY = 0, B1_FULL, B1_EMPTY = B1_FULL + 2, B2_FULL = B1_EMPTY + 2, B2_EMPTY = B2_FULL + 2, S_FULL = B2_EMPTY + 2, S_FREE = S_FULL + 2, DP_FULL,
           T_FULL, R_FULL = T_FULL + 2, R_FREE, STAT_FULL, DRAIN, NUM };

// The fragments of 16 rows in tensor memory: lane i holds columns 2 (i % 4), + 1 of every eight of rows i / 4 and i / 4 + 8.
__device__ __forceinline__ void tmem_ld_rows16(uint32_t taddr, uint32_t (&r)[16]) {  // 16 rows x 32 columns
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_rows16(uint32_t taddr, const uint32_t (&r)[8]) {  // 16 rows x 16 columns (32 packed values)
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Loads that a false predicate leaves out. As predicated instructions on the registers themselves: written as a branch, the value is moved into place
// behind it, and the move waits for every load where it stands (12 K cycles a step instead of 3 K).
__device__ __forceinline__ void load4(float4 &x, const float *at, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+f"(x.x), "+f"(x.y), "+f"(x.z), "+f"(x.w)
               : "l"(at), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ float2 load2(const float *at, bool on) {
  float2 x = make_float2(0.f, 0.f);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p ld.global.v2.f32 {%0, %1}, [%2];\n\t}" : "+f"(x.x), "+f"(x.y) : "l"(at), "r"((int)on) : "memory");
  return x;
}

// mbar_wait_warp with its polling loop in place: a kernel that moves registers between its warps (setmaxnreg) cannot be compiled with calls.
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile uint32_t *abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  const uint64_t t0 = global_timer_ns();
  bool done = false, late = false;
#pragma unroll 1
  for (uint32_t polls = 1; !done && !late; ++polls) {
    done = __all_sync(0xffffffffu, mbar_try_wait(bar, parity));
    if ((polls & 255u) == 0u) late = __any_sync(0xffffffffu, *abort_flag != 0u || polls >= kWaitMaxPolls || global_timer_ns() - t0 > kWaitBudgetNs);
  }
  if (!done) *abort_flag = 1u;
  return done;
}

__device__ __forceinline__ void store_cluster(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ float2 f2(uint32_t x, uint32_t y) { return as_float2(x, y); }

// Cuts two values: out[part] = (part of y) << 16 | part of x. An infinity (or what rounds to one) gives one in the second part, and so NaN; a NaN does.
__device__ __forceinline__ void cut(float2 x, uint32_t (&out)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out[i]) : "f"(x.y), "f"(x.x));
    if (i < 2) x = fma2(f2(out[i] << 16, out[i] & 0xffff0000u), make_float2(-1.f, -1.f), x);
  }
}
// 16 rows x 32 values of a warp, as fragments, into the parts of an A operand in tensor memory; what does not go there is left in w[2].
template <int PARTS>
__device__ __forceinline__ void store_parts(uint32_t taddr, uint32_t part_cols, const float2 *v, uint32_t (&w)[3][8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    uint32_t c[3];
    cut(v[i], c);
#pragma unroll
    for (int s = 0; s < 3; ++s) w[s][i] = c[s];
  }
#pragma unroll
  for (int s = 0; s < PARTS; ++s) tmem_st_rows16(taddr + s * part_cols, w[s]);
}

// A product of parts, K-steps [FROM, TO): A in tensor memory, or the third part in shared memory. `accumulate` is for the first of them.
template <int FROM, int TO, class F>
__device__ __forceinline__ void product_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, F b_step, uint32_t idesc, bool accumulate, uint32_t mine) {
#pragma unroll
  for (int kk = FROM; kk < TO; ++kk) mma_ts(d, a + kk * 8, b_lo + (b_step(kk) >> 4), b_hi, idesc, accumulate || kk > FROM ? 1u : 0u, mine);
}
template <int STEPS, class FA, class F>
__device__ __forceinline__ void product_ss(uint32_t d, uint32_t a_lo, uint32_t a_hi, FA a_step, uint32_t b_lo, uint32_t b_hi, F b_step, uint32_t idesc, uint32_t mine) {
#pragma unroll
  for (int kk = 0; kk < STEPS; ++kk) mma_ss(d, a_lo + (a_step(kk) >> 4), a_hi, b_lo + (b_step(kk) >> 4), b_hi, idesc, 1u, mine);
}

// Index i of W elements of a tensor of n, as it is; range-checked in checked builds where the access is `on` (DF_IDX, df_common.cuh).
template <int W>
__device__ __forceinline__ size_t elem(size_t i, size_t n, const AttnParams &p, bool on = true) {
#ifdef DF_BOUNDS_CHECK
  return on && df_checked_index(i + W - 1, n, p.status) == i + W - 1 ? i : 0;
#else
  return i;
#endif
}
// Elements of the tensors of queries, of keys, and of the row statistics.
__device__ __forceinline__ size_t q_elements(const AttnParams &p) { return (size_t)p.B * p.Sq * p.H * p.D; }
__device__ __forceinline__ size_t k_elements(const AttnParams &p) { return (size_t)p.B * p.Sk * p.H * p.D; }
__device__ __forceinline__ size_t stat_elements(const AttnParams &p) { return (size_t)p.B * p.H * p.Sq; }

// logsumexp in log2 units, negated, in two fp32 numbers: rounded to one, ten times 2^-24 of it goes into every P. No visible key: P = 0.
__device__ __forceinline__ float neg_lse2(float raw, float *lo) {
  const float hi = raw * kLog2e;
  *lo = fabsf(hi) < INFINITY ? -fmaf(raw, 1.92596299e-8f, fmaf(raw, kLog2e, -hi)) : 0.f;  // log2 e = kLog2e + 1.926e-8
  return raw == -INFINITY ? -INFINITY : -hi;
}

// One row of a pass in fp32 arithmetic by one warp: the visible streamed rows and no others. An infinity has no parts, and a hidden row's infinity or
// NaN times a P of zero is NaN too, so what is not finite in a block's results says nothing yet about what the row should be. It is no fast path:
// lanes read rows of their own, and when every row needs it a call takes 17 to 42 times as long as attn_simt.cu (B200, ms, forward / backward, 2 x 8 x 1000 x
// 128, V infinite at key 0: 3.6 / 6.5 here, 0.13 / 0.38 there; one NaN in Q: forward 0.21). Loops unrolled eight times made that 3.0 / 5.2 and calls with
// finite operands, which are the ones that matter, up to 5 % slower.
template <Pass PASS>
__device__ __forceinline__ void fp32_row(const AttnParams &p, size_t q_base, size_t k_base, size_t s_base, long long row) {
  constexpr bool KEYS = PASS == DK || PASS == DV, TWO = PASS == DQ || PASS == DK;
  const uint32_t lane = threadIdx.x & 31;
  const size_t dm = (size_t)p.H * p.D, res = (KEYS ? k_base : q_base) + (size_t)row * dm, str = KEYS ? q_base : k_base;
  const size_t n_res = KEYS ? k_elements(p) : q_elements(p), n_str = KEYS ? q_elements(p) : k_elements(p), n_stat = stat_elements(p);
  const float *a1 = KEYS ? p.k : p.q, *a2 = KEYS ? p.v : p.d_out, *b1 = KEYS ? p.q : p.k, *b2 = KEYS ? p.d_out : p.v;
  long long from = 0, to = KEYS ? p.Sq : p.Sk;
  if (p.causal && KEYS && row > p.shift) from = row - p.shift;
  if (p.causal && !KEYS && row + p.shift + 1 < to) to = row + p.shift + 1;
  auto dot = [&](const float *x, const float *y, long long j) {  // of this row and row j of the streamed side
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll 1
    for (uint32_t d = 0; d < p.D; d += 4) {
      const float4 u = *reinterpret_cast<const float4 *>(x + elem<4>(res + d, n_res, p)), w = *reinterpret_cast<const float4 *>(y + elem<4>(str + (size_t)j * dm + d, n_str, p));
      sum = fma2(make_float2(u.z, u.w), make_float2(w.z, w.w), fma2(make_float2(u.x, u.y), make_float2(w.x, w.y), sum));
    }
    return sum.x + sum.y;
  };
  float m = -INFINITY, l = 0.f, neg = 0.f, lo = 0.f, delta = 0.f;
  if (PASS == DQ) {
    neg = neg_lse2(p.lse_in[elem<1>(s_base + row, n_stat, p)], &lo);
    delta = p.delta_in[elem<1>(s_base + row, n_stat, p)];
  }
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);  // dims 4 lane .. + 3
#pragma unroll 1
  for (long long c = from; c < to; c += 32) {
    const long long j = c + lane;
    const bool seen = j < to;
    float t = 0.f;
    const float s = seen ? dot(a1, b1, j) * p.scale_log2 : -INFINITY;
    if (PASS == FORWARD) {
      float top = s;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float mn = fmaxf(m, top), alpha = mn == -INFINITY ? 1.f : ex2_approx(m - mn);
      m = mn;
      t = ex2_approx(s - (m == -INFINITY ? 0.f : m));
      float sum = t;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l = fmaf(l, alpha, sum);
      acc = make_float4(acc.x * alpha, acc.y * alpha, acc.z * alpha, acc.w * alpha);
    } else if (seen) {
      if (KEYS) neg = neg_lse2(p.lse_in[elem<1>(s_base + j, n_stat, p)], &lo);
      if (PASS == DK) delta = p.delta_in[elem<1>(s_base + j, n_stat, p)];
      t = ex2_approx(s + neg + lo);
      if (TWO) t *= dot(a2, b2, j) - delta;
    }
#pragma unroll 1
    for (int x = 0; x < 32 && c + x < to; ++x) {
      const float tx = __shfl_sync(0xffffffffu, t, x);
      if (4 * lane < p.D) {
        const float4 y = *reinterpret_cast<const float4 *>((TWO ? b1 : b2) + elem<4>(str + (size_t)(c + x) * dm + 4 * lane, n_str, p));
        acc = make_float4(fmaf(tx, y.x, acc.x), fmaf(tx, y.y, acc.y), fmaf(tx, y.z, acc.z), fmaf(tx, y.w, acc.w));
      }
    }
  }
  const float f = PASS == FORWARD ? (l > 0.f ? 1.f / l : 0.f) : PASS == DV ? 1.f : p.scale;  // reference guard, attention_fused.cu:104
  float *dst = PASS == FORWARD ? p.out : PASS == DQ ? p.d_q : PASS == DK ? p.d_k : p.d_v;
  if (4 * lane < p.D) *reinterpret_cast<float4 *>(dst + elem<4>(res + 4 * lane, n_res, p)) = make_float4(acc.x * f, acc.y * f, acc.z * f, acc.w * f);
  if (PASS == FORWARD && p.lse && lane == 0) p.lse[elem<1>(s_base + row, n_stat, p)] = l > 0.f ? fmaf(m, kLn2, logf(l)) : -INFINITY;
}

// One block of 128 resident rows. A cluster of CL CTAs shares it: each takes a range of the steps, rank 0 puts the results together.
template <class C, int CL>
__device__ __forceinline__ void split_block(const AttnParams &p, uint32_t tile, uint32_t bh) {
  constexpr Pass PASS = C::PASS;
  constexpr int DP = C::DP;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  float *sStats = reinterpret_cast<float *>(smem + C::oStats);  // [3][NSTATS][64]
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::oBars);
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem + C::oBars + 240);
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(smem + C::oBars + 244);
  uint32_t *again = reinterpret_cast<uint32_t *>(smem + C::oBars + 208);  // of each compute warp: rows to be formed in fp32 arithmetic
  static_assert(NUM * 8 <= 208, "barriers");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto bar = [&](int id) { return smem_u32(&bars[id]); };

  const uint32_t b = bh / p.H, h = bh % p.H;
  const size_t dm = (size_t)p.H * p.D;
  const size_t q_base = (size_t)b * p.Sq * dm + (size_t)h * p.D, k_base = (size_t)b * p.Sk * dm + (size_t)h * p.D, s_base = (size_t)bh * p.Sq;
  const size_t el_res = C::ROWS_ARE_KEYS ? k_elements(p) : q_elements(p), el_str = C::ROWS_ARE_KEYS ? q_elements(p) : k_elements(p), el_stat = stat_elements(p);
  const long long row0 = (long long)tile * BM;
  const long long n_res = C::ROWS_ARE_KEYS ? p.Sk : p.Sq, n_str = C::ROWS_ARE_KEYS ? p.Sq : p.Sk;
  long long begin = 0, end = n_str;  // streamed rows that any resident row sees
  if (p.causal) {
    if (C::ROWS_ARE_KEYS) {
      begin = row0 - p.shift;
      begin = begin < 0 ? 0 : begin / BN * BN;
    } else {
      const long long last = row0 + BM < n_res ? row0 + BM : n_res;
      if (last + p.shift < end) end = last + p.shift;
    }
  }
  const int rank = CL > 1 ? (int)cluster_rank() : 0, n_all = end > begin ? (int)((end - begin + BN - 1) / BN) : 0;
  const int first = (int)((long long)n_all * rank / CL), n = (int)((long long)n_all * (rank + 1) / CL) - first;  // steps
  begin += (long long)first * BN;

  if (warp == kMmaWarp) {
    for (int i = lane; i < NUM; i += 32)
      mbar_init(bar(i), (i == A_READY || i == T_FULL || i == T_FULL + 1 || i == S_FREE || i == R_FREE || i == STAT_FULL) ? kComputeThreads
                        : (i == B1_FULL || i == B1_FULL + 1 || i == B2_FULL || i == B2_FULL + 1) ? kStreamThreads : 1);
    if (lane == 0) *abort_flag = 0;
    mbar_init_fence();
    __syncwarp();
    tmem_alloc(smem_u32(tmem_holder), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_holder;
  pdl_wait();

  if (warp >= 8) {
    regs_less<kOtherRegs>();
  }
  if (warp >= 8 && warp < kMmaWarp) {
    // ---------------------------------------------- streamed rows: fp32 -> three bf16 tiles
    const int sw = warp - 8, sub = lane / C::G, g = lane % C::G;
    const bool on = sub < C::RPW;
    const int first_row = sw * C::RPW + sub;
    const bool dims = on && 4 * g < (int)p.D;  // columns past the head size stay zero
    auto offset = [&](int row) {  // 16-byte chunk c of row r of a 128-byte-swizzled slab lies at c ^ (r % 8)
      return (uint32_t)(g >> 4) * C::kSlab + (uint32_t)row * 128 + ((((uint32_t)(g & 15) >> 1) ^ ((uint32_t)row & 7)) << 4) + (uint32_t)(g & 1) * 8;
    };
    auto put = [&](uint32_t at, const float4 &x) {
      uint32_t lo[3], hi[3];
      cut(make_float2(x.x, x.y), lo);
      cut(make_float2(x.z, x.w), hi);
      if (on) {
#pragma unroll
        for (int s = 0; s < 3; ++s) asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + s * C::kPart), "r"(lo[s]), "r"(hi[s]) : "memory");
      }
    };
    const float *src1 = C::ROWS_ARE_KEYS ? p.q : p.k, *src2 = C::ROWS_ARE_KEYS ? p.d_out : p.v;
    const size_t str_base = C::ROWS_ARE_KEYS ? q_base : k_base;
    float4 buf[C::U];
    // Tile t of the stream: B1 and B2 in turn. What a value held is stored while the next tile's is on its way.
    // Rows past the end repeat the last one: their scores are hidden, and P and dS are zero there.
    uint32_t to[C::U];
#pragma unroll
    for (int u = 0; u < C::U; ++u) {
      buf[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      to[u] = offset(first_row + C::RPA * u);
    }
    auto load_tile = [&](int t, int u) {
      const long long row = begin + (long long)(t >> 1) * BN + first_row + C::RPA * u;
      const bool valid = dims && first_row + C::RPA * u < BN;
      load4(buf[u], ((t & 1) ? src2 : src1) + elem<4>(str_base + (size_t)min(row, n_str - 1) * dm + 4 * g, el_str, p, valid), valid);
    };
    if (n > 0) {
#pragma unroll
      for (int u = 0; u < C::U; ++u) load_tile(0, u);
      for (int t = 0; t < 2 * n; ++t) {
        const int j = t >> 1, b2 = t & 1, stages = b2 ? C::ST2 : C::ST1, st = stages == 2 ? (j & 1) : 0, use = stages == 2 ? (j >> 1) : j;
        if (use > 0 && !wait_warp(bar((b2 ? B2_EMPTY : B1_EMPTY) + st), (use - 1) & 1, abort_flag)) break;
        const uint32_t dst = sbase + (b2 ? C::oB2 : C::oB1) + st * C::kTile;
#pragma unroll
        for (int u = 0; u < C::U; ++u) {
          if (C::RPA * (u + 1) <= BN || first_row + C::RPA * u < BN) put(dst + to[u], buf[u]);
          load_tile(t + 1, u);  // past the last tile: the last row, not used
        }
        fence_proxy_async_smem();
        mbar_arrive(bar((b2 ? B2_FULL : B1_FULL) + st));
      }
    }
  } else if (warp == kMmaWarp) {
    // ---------------------------------------------- MMA issuer (the whole warp runs the role, one elected lane issues)
    const uint32_t idesc_s = make_idesc(kFmtBF16, BM, BN, 0, 0), idesc_r = make_idesc(kFmtBF16, BM, DP, 0, 1);
    const uint32_t mine = elect_one() ? 1u : 0u;
    constexpr bool R_FROM_B1 = C::TWO;  // R's second operand: K or Q; else V or dO
    constexpr int KS = C::KS, KH = KS / 2;
    const uint64_t d1 = make_smem_desc(sbase + C::oB1, 16, 1024, kSwz128), d2 = make_smem_desc(sbase + C::oB2, 16, 1024, kSwz128);
    const uint64_t dr = make_smem_desc(sbase + (R_FROM_B1 ? C::oB1 : C::oB2), C::kSlab, 1024, kSwz128);
    const uint64_t da = make_smem_desc(sbase, 16, 1024, kSwz128);  // third part of A1; A2's is kPartA further
    auto a_step = [](int kk) { return (uint32_t)((kk >> 2) * C::kSlabA + (kk & 3) * 32); };
    auto k_step = [](int kk) { return (uint32_t)((kk >> 2) * C::kSlab + (kk & 3) * 32); };
    auto r_step = [](int kk) { return (uint32_t)(kk * 2048); };
    auto stage1 = [&](int j) { return j & 1; };
    auto stage2 = [&](int j) { return C::ST2 == 2 ? (j & 1) : 0; };
    auto phase1 = [&](int j) { return (uint32_t)(j >> 1) & 1u; };
    auto phase2 = [&](int j) { return (uint32_t)(C::ST2 == 2 ? (j >> 1) : j) & 1u; };
    // A B^T over the head size in two accumulators, the first: everything but the second half of the largest product
    auto scores1 = [&](uint32_t d, uint32_t a, uint32_t a3_lo, uint32_t b_lo, uint32_t b_hi) {
      constexpr uint32_t PA = C::kPartCols, PB = C::kPart >> 4;
      product_ts<0, KS>(d, a, b_lo + 2 * PB, b_hi, k_step, idesc_s, false, mine);
      product_ss<KS>(d, a3_lo, (uint32_t)(da >> 32), a_step, b_lo, b_hi, k_step, idesc_s, mine);
      product_ts<0, KS>(d, a + PA, b_lo + PB, b_hi, k_step, idesc_s, true, mine);
      product_ts<0, KS>(d, a, b_lo + PB, b_hi, k_step, idesc_s, true, mine);
      product_ts<0, KS>(d, a + PA, b_lo, b_hi, k_step, idesc_s, true, mine);
      product_ts<0, KH>(d, a, b_lo, b_hi, k_step, idesc_s, true, mine);
    };
    auto scores2 = [&](uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi) { product_ts<KH, KS>(d, a, b_lo, b_hi, k_step, idesc_s, false, mine); };
    // waits for up to three barriers with one round trip where all are there already
    auto wait3 = [&](int b0, uint32_t p0, int b1, uint32_t p1, int b2, uint32_t p2) -> bool {
      const uint32_t m = mbar_test3_warp(bar(b0), p0, bar(b1), p1, bar(b2), p2);
      return ((m & 1u) || wait_warp(bar(b0), p0, abort_flag)) && ((m & 2u) || wait_warp(bar(b1), p1, abort_flag)) && ((m & 4u) || wait_warp(bar(b2), p2, abort_flag));
    };
    auto issue_s = [&](int j) -> bool {
      const int st = stage1(j), full = B1_FULL + st;
      const uint32_t b_lo = (uint32_t)d1 + ((st * C::kTile) >> 4), b_hi = (uint32_t)(d1 >> 32), ph = phase1(j);
      // the second accumulator is free when the last step's has been read, or where it lies in R's columns, when R has
      const int freed = j > 0 ? (C::TWO ? R_FREE : S_FREE) : full;
      const uint32_t ph_freed = j > 0 ? (uint32_t)(j - 1) & 1u : ph;
      const uint32_t m = mbar_test3_warp(bar(full), ph, bar(freed), ph_freed, bar(freed), ph_freed);
      if (!(m & 1u) && !wait_warp(bar(full), ph, abort_flag)) return false;
      tc_fence_after_sync();
      scores1(tmem + ((j & 1) ? C::cX1 : C::cX0), tmem + C::cA1, (uint32_t)da, b_lo, b_hi);
      if (!(m & 2u)) {
        if (!wait_warp(bar(freed), ph_freed, abort_flag)) return false;
        tc_fence_after_sync();
      }
      scores2(tmem + C::cS2, tmem + C::cA1, b_lo, b_hi);
      commit_elected(bar(S_FULL + (C::TWO ? 0 : (j & 1))));
      if (!R_FROM_B1) commit_elected(bar(B1_EMPTY + st));
      return true;
    };
    auto issue_dp = [&](int j) -> bool {
      const int st = stage2(j);
      const uint32_t b_lo = (uint32_t)d2 + ((st * C::kTile) >> 4), b_hi = (uint32_t)(d2 >> 32);
      if (!wait_warp(bar(B2_FULL + st), phase2(j), abort_flag)) return false;
      tc_fence_after_sync();
      scores1(tmem + C::cDP, tmem + C::cA2, (uint32_t)da + (C::kPartA >> 4), b_lo, b_hi);
      scores2(tmem + C::cDP2, tmem + C::cA2, b_lo, b_hi);
      commit_elected(bar(DP_FULL));
      commit_elected(bar(B2_EMPTY + st));
      return true;
    };
    // R = T B: the five smaller products over K-steps [FROM, TO) of the step's rows, and the largest
    auto products_r = [&](auto from, auto to, uint32_t t, uint32_t b_lo, uint32_t b_hi) {
      constexpr int F = decltype(from)::value, T = decltype(to)::value;
      constexpr uint32_t PB = C::kPart >> 4;
      product_ts<F, T>(tmem + C::cR, t, b_lo + 2 * PB, b_hi, r_step, idesc_r, F > 0, mine);
      product_ts<F, T>(tmem + C::cR, t + 64, b_lo, b_hi, r_step, idesc_r, true, mine);
      product_ts<F, T>(tmem + C::cR, t + 32, b_lo + PB, b_hi, r_step, idesc_r, true, mine);
      product_ts<F, T>(tmem + C::cR, t, b_lo + PB, b_hi, r_step, idesc_r, true, mine);
      product_ts<F, T>(tmem + C::cR, t + 32, b_lo, b_hi, r_step, idesc_r, true, mine);
    };
    auto issue_r = [&](int j) -> bool {
      const int st = R_FROM_B1 ? stage1(j) : stage2(j), x = C::TWO ? 0 : (j & 1);
      const uint32_t ph_t = (uint32_t)(C::TWO ? j : (j >> 1)) & 1u;
      if (C::TWO ? !wait_warp(bar(T_FULL), ph_t, abort_flag)
                 : !wait3(T_FULL + x, ph_t, B2_FULL + st, phase2(j), j > 0 ? (int)R_FREE : T_FULL + x, j > 0 ? (uint32_t)(j - 1) & 1u : ph_t))
        return false;
      tc_fence_after_sync();
      const uint32_t t = tmem + (x ? C::cX1 : C::cX0), b_lo = (uint32_t)dr + ((st * C::kTile) >> 4), b_hi = (uint32_t)(dr >> 32);
      constexpr int H = BN / 32;
      if (C::TWO) {  // T comes in halves: products over the first run while the second is formed
        products_r(ic<0>(), ic<H>(), t, b_lo, b_hi);
        if (!wait_warp(bar(T_FULL + 1), ph_t, abort_flag)) return false;
        tc_fence_after_sync();
        products_r(ic<H>(), ic<2 * H>(), t, b_lo, b_hi);
      } else {
        products_r(ic<0>(), ic<2 * H>(), t, b_lo, b_hi);
      }
      product_ts<0, 2 * H>(tmem + C::cR, t, b_lo, b_hi, r_step, idesc_r, true, mine);
      commit_elected(bar(R_FULL));
      commit_elected(bar((R_FROM_B1 ? B1_EMPTY : B2_EMPTY) + st));
      return true;
    };
    if (n > 0 && wait_warp(bar(A_READY), 0, abort_flag)) {
      tc_fence_after_sync();
      bool ok = issue_s(0);
      if (C::TWO) {
        for (int j = 0; ok && j < n; ++j) ok = issue_dp(j) && issue_r(j) && (j + 1 >= n || issue_s(j + 1));
      } else {
        for (int j = 0; ok && j < n; ++j) ok = (j + 1 >= n || issue_s(j + 1)) && issue_r(j);
      }
    }
  } else {
    // ---------------------------------------------- compute warps
    regs_more<kComputeRegs>();
    const int base16 = (warp & 3) * 32 + (warp >> 2) * 16, t4 = lane & 3;
    const uint32_t lanes = (uint32_t)base16 << 16;
    const long long rowA = row0 + base16 + (lane >> 2), rowB = rowA + 8;  // this lane's two rows
    const size_t res_base = C::ROWS_ARE_KEYS ? k_base : q_base;
    const float scale2 = p.scale_log2;
    // resident tiles: two parts into tensor memory, the third into shared memory
    auto load_resident = [&](const float *src, uint32_t cols, uint32_t third) {
      const uint32_t rA = (uint32_t)(base16 + (lane >> 2)), rB = rA + 8;  // the same modulo 8
      float2 v[DP / 4];
#pragma unroll
      for (int g = 0; g < DP / 8; ++g) {
        const int d = g * 8 + 2 * t4;
        const bool onA = rowA < n_res && d < (int)p.D, onB = rowB < n_res && d < (int)p.D;
        v[2 * g] = load2(src + elem<2>(res_base + (size_t)rowA * dm + d, el_res, p, onA), onA);
        v[2 * g + 1] = load2(src + elem<2>(res_base + (size_t)rowB * dm + d, el_res, p, onB), onB);
      }
#pragma unroll
      for (int c = 0; c < DP / 32; ++c) {
        uint32_t w[3][8];
        store_parts<2>(tmem + lanes + cols + c * 16, C::kPartCols, v + 8 * c, w);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint32_t at = sbase + third + (uint32_t)(c >> 1) * C::kSlabA + ((((uint32_t)((c & 1) * 4 + g)) ^ (rA & 7)) << 4) + 4 * t4;
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + rA * 128), "r"(w[2][2 * g]) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + rB * 128), "r"(w[2][2 * g + 1]) : "memory");
        }
      }
    };
    load_resident(C::ROWS_ARE_KEYS ? p.k : p.q, C::cA1, 0);
    if (C::TWO) load_resident(C::ROWS_ARE_KEYS ? p.v : p.d_out, C::cA2, C::kPartA);
    tmem_wait_st();
    tc_fence_before_sync();
    fence_proxy_async_smem();
    mbar_arrive(bar(A_READY));
    float2 acc[DP / 4];  // fragments of 16 rows x DP: columns 8 i + 2 t4, + 1 of row A at 2 i, of row B at 2 i + 1
#pragma unroll
    for (int i = 0; i < DP / 4; ++i) acc[i] = make_float2(0.f, 0.f);
    // row statistics: of this lane's rows (queries), or staged for a step's queries one step ahead, in one of three buffers (a thread past the wait
    // of step j knows that all others are past step j - 2)
    float mA = -INFINITY, mB = -INFINITY, lA = 0.f, lB = 0.f, dA = 0.f, dB = 0.f;
    float fA = p.scale, fB = p.scale;  // factors of the results
    if (PASS == DQ) {
      if (rowA < n_res) { mA = p.lse_in[elem<1>(s_base + rowA, el_stat, p)]; dA = -p.delta_in[elem<1>(s_base + rowA, el_stat, p)]; }
      if (rowB < n_res) { mB = p.lse_in[elem<1>(s_base + rowB, el_stat, p)]; dB = -p.delta_in[elem<1>(s_base + rowB, el_stat, p)]; }
      float loA, loB;
      mA = neg_lse2(mA, &loA);
      mB = neg_lse2(mB, &loB);
      fA = fmaf(fA, loA * kLn2, fA);  // 2^lo
      fB = fmaf(fB, loB * kLn2, fB);
    }
    auto fetch_stat = [&](int j) -> float {
      const int tid = threadIdx.x;
      const long long q = begin + (long long)j * BN + (tid & (BN - 1));
      if (tid >= 2 * BN) return 0.f;
      if (tid < BN) return q < n_str ? p.lse_in[elem<1>(s_base + q, el_stat, p)] : -INFINITY;
      return PASS == DK && q < n_str ? p.delta_in[elem<1>(s_base + q, el_stat, p)] : 0.f;
    };
    auto put_stat = [&](int j, float raw) {
      float *to = sStats + (j % 3) * C::NSTATS * BN;
      if (threadIdx.x < BN) {
        float lo;
        to[threadIdx.x] = neg_lse2(raw, &lo);
        to[BN + threadIdx.x] = lo;
      } else if (PASS == DK && threadIdx.x < 2 * BN) {
        to[BN + threadIdx.x] = -raw;
      }
      mbar_arrive(bar(STAT_FULL));
    };
    bool ok = true;
    uint32_t odd_rows = 0;
    if (C::ROWS_ARE_KEYS && n > 0) put_stat(0, fetch_stat(0));
    // R of step j into the registers
    auto add_r = [&](int j) -> bool {
      if (!wait_warp(bar(R_FULL), (uint32_t)j & 1u, abort_flag)) return false;
      tc_fence_after_sync();
#pragma unroll
      for (int c = 0; c < DP / 32; ++c) {
        uint32_t r[16];
        tmem_ld_rows16(tmem + lanes + C::cR + c * 32, r);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[c * 8 + i] = add2(acc[c * 8 + i], f2(r[2 * i], r[2 * i + 1]));
      }
      tc_fence_before_sync();
      mbar_arrive(bar(R_FREE));
      return true;
    };
    for (int j = 0; j < n; ++j) {
      const long long c0 = begin + (long long)j * BN;
      if (C::TWO && j > 0 && !add_r(j - 1)) { ok = false; break; }  // this step's scores take R's columns
      float stat_next = 0.f;
      if (C::ROWS_ARE_KEYS) {
        if (j + 1 < n) stat_next = fetch_stat(j + 1);
        if (!wait_warp(bar(STAT_FULL), (uint32_t)j & 1u, abort_flag)) { ok = false; break; }
      }
      const float *stats = sStats + (j % 3) * C::NSTATS * BN;
      const int x = C::TWO ? 0 : (j & 1);
      uint32_t s[32];
      const uint32_t tX = tmem + lanes + (x ? C::cX1 : C::cX0);
      // 32 columns of scores (or dP): the sum of the two accumulators
      auto read2 = [&](uint32_t t1, uint32_t t2, uint32_t *out) {
        uint32_t r1[16], r2[16];
        tmem_ld_rows16(t1, r1);
        tmem_ld_rows16(t2, r2);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float2 y = add2(f2(r1[2 * i], r1[2 * i + 1]), f2(r2[2 * i], r2[2 * i + 1]));
          out[2 * i] = __float_as_uint(y.x);
          out[2 * i + 1] = __float_as_uint(y.y);
        }
      };
      if (!wait_warp(bar(S_FULL + x), (uint32_t)(C::TWO ? j : (j >> 1)) & 1u, abort_flag)) { ok = false; break; }
      tc_fence_after_sync();
      read2(tX, tmem + lanes + C::cS2, s);
      read2(tX + 32, tmem + lanes + C::cS2 + 32, s + 16);
      if (!C::TWO) {
        tc_fence_before_sync();
        mbar_arrive(bar(S_FREE));
      }
      // Which columns a row sees: queries of a key from `low` on, keys of a query up to `high`.
      const long long off = C::ROWS_ARE_KEYS ? (p.causal ? -p.shift - c0 : -(1ll << 40)) : (p.causal ? p.shift + 1 - c0 : 1ll << 40);
      auto clamp = [](long long v) { return v > BN ? BN : (v < 0 ? 0 : (int)v); };
      int limA, limB;
      bool all;
      if (C::ROWS_ARE_KEYS) {
        limA = rowA < n_res ? clamp(rowA + off) : BN;
        limB = rowB < n_res ? clamp(rowB + off) : BN;
        all = row0 + BM - 1 + off <= 0 && row0 + BM <= n_res;  // queries past the end have P = 0 by their statistics
      } else {
        const int left = clamp(n_str - c0);
        limA = min(left, clamp(rowA + off));
        limB = min(left, clamp(rowB + off));
        all = row0 + off >= BN && left == BN;
      }
      if (!all) {
#pragma unroll
        for (int g = 0; g < 8; ++g)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int col = 8 * g + 2 * t4 + (e & 1), lim = e < 2 ? limA : limB;
            if (C::ROWS_ARE_KEYS ? col < lim : col >= lim) s[4 * g + e] = 0xff800000u;
          }
      }
      float2 v[16];
      float alphaA = 1.f, alphaB = 1.f;
      if (PASS == FORWARD) {
        float topA = -INFINITY, topB = -INFINITY;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          topA = fmaxf(topA, fmaxf(__uint_as_float(s[4 * g]), __uint_as_float(s[4 * g + 1])));
          topB = fmaxf(topB, fmaxf(__uint_as_float(s[4 * g + 2]), __uint_as_float(s[4 * g + 3])));
        }
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
          topA = fmaxf(topA, __shfl_xor_sync(0xffffffffu, topA, o));
          topB = fmaxf(topB, __shfl_xor_sync(0xffffffffu, topB, o));
        }
        const float nA = fmaxf(mA, topA * scale2), nB = fmaxf(mB, topB * scale2);  // scale2 > 0
        alphaA = nA == -INFINITY ? 1.f : ex2_approx(mA - nA);  // before the first visible key: 0
        alphaB = nB == -INFINITY ? 1.f : ex2_approx(mB - nB);
        mA = nA;
        mB = nB;
        const float subA = nA == -INFINITY ? 0.f : nA, subB = nB == -INFINITY ? 0.f : nB;
        float2 sumA = make_float2(0.f, 0.f), sumB = sumA;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const float2 xA = fma2(f2(s[4 * g], s[4 * g + 1]), make_float2(scale2, scale2), make_float2(-subA, -subA));
          const float2 xB = fma2(f2(s[4 * g + 2], s[4 * g + 3]), make_float2(scale2, scale2), make_float2(-subB, -subB));
          v[2 * g] = make_float2(ex2_approx(xA.x), ex2_approx(xA.y));
          v[2 * g + 1] = make_float2(ex2_approx(xB.x), ex2_approx(xB.y));
          sumA = add2(sumA, v[2 * g]);
          sumB = add2(sumB, v[2 * g + 1]);
        }
        lA = fmaf(lA, alphaA, sumA.x + sumA.y);
        lB = fmaf(lB, alphaB, sumB.x + sumB.y);
      } else {
#pragma unroll
        for (int g = 0; g < 8; ++g)
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const float2 neg = C::ROWS_ARE_KEYS ? *reinterpret_cast<const float2 *>(stats + 8 * g + 2 * t4) : half ? make_float2(mB, mB) : make_float2(mA, mA);
            float2 x2 = fma2(f2(s[4 * g + 2 * half], s[4 * g + 2 * half + 1]), make_float2(scale2, scale2), neg);
            if (C::ROWS_ARE_KEYS) x2 = add2(x2, *reinterpret_cast<const float2 *>(stats + BN + 8 * g + 2 * t4));
            v[2 * g + half] = make_float2(ex2_approx(x2.x), ex2_approx(x2.y));
          }
      }
      uint32_t w[3][8];
      if (C::TWO) {
        if (!wait_warp(bar(DP_FULL), (uint32_t)j & 1u, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
        // all of dP is read before any of T is handed over: T takes the place of its first columns, R that of its second accumulator
        read2(tmem + lanes + C::cDP, tmem + lanes + C::cDP2, s);
        read2(tmem + lanes + C::cDP + 32, tmem + lanes + C::cDP2 + 32, s + 16);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const float2 neg = C::ROWS_ARE_KEYS ? *reinterpret_cast<const float2 *>(stats + 2 * BN + 32 * c + 8 * g + 2 * t4) : half ? make_float2(dB, dB) : make_float2(dA, dA);
              float2 &y = v[8 * c + 2 * g + half];
              y = mul2(y, add2(f2(s[16 * c + 4 * g + 2 * half], s[16 * c + 4 * g + 2 * half + 1]), neg));
            }
          store_parts<3>(tX + 16 * c, 32, v + 8 * c, w);
          tmem_wait_st();
          tc_fence_before_sync();
          mbar_arrive(bar(T_FULL + c));
        }
      } else {
        store_parts<3>(tX, 32, v, w);
        store_parts<3>(tX + 16, 32, v + 8, w);
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(T_FULL + x));
      }
      if (C::ROWS_ARE_KEYS && j + 1 < n) put_stat(j + 1, stat_next);
      if (!C::TWO && j > 0 && !add_r(j - 1)) { ok = false; break; }
      if (PASS == FORWARD && __any_sync(0xffffffffu, alphaA != 1.f || alphaB != 1.f)) {
#pragma unroll
        for (int g = 0; g < DP / 8; ++g) {
          acc[2 * g] = mul2(acc[2 * g], make_float2(alphaA, alphaA));
          acc[2 * g + 1] = mul2(acc[2 * g + 1], make_float2(alphaB, alphaB));
        }
      }
    }
    if (ok && n > 0) ok = add_r(n - 1);
    if (CL > 1) {
      constexpr uint32_t kSlot = kComputeThreads * 16 * (DP / 8 + 1);  // an accumulator and m, l of every compute thread, 16 bytes of each in turn
      static_assert((CL - 1) * kSlot <= C::oStats, "the others' results fit where the tiles were");
      cluster_sync();  // all products are done and all tiles used up
      if (rank > 0) {
        const uint32_t at = map_to_rank(sbase, 0) + (rank - 1) * kSlot + threadIdx.x * 16;
#pragma unroll
        for (int i = 0; i < DP / 8; ++i) store_cluster(at + i * kComputeThreads * 16, make_float4(acc[2 * i].x, acc[2 * i].y, acc[2 * i + 1].x, acc[2 * i + 1].y));
        if (PASS == FORWARD) store_cluster(at + DP / 8 * kComputeThreads * 16, make_float4(mA, mB, lA, lB));
      }
      cluster_sync();
      if (rank == 0) {
#pragma unroll 1
        for (int r = 1; r < CL; ++r) {
          const uint8_t *from = smem + (r - 1) * kSlot + threadIdx.x * 16;
          float2 wA = make_float2(1.f, 1.f), wB = wA;  // weights of this CTA's sums and of the other's, rows A and B
          if (PASS == FORWARD) {
            const float4 ml = *reinterpret_cast<const float4 *>(from + DP / 8 * kComputeThreads * 16);
            const float nA = fmaxf(mA, ml.x), nB = fmaxf(mB, ml.y), subA = nA == -INFINITY ? 0.f : nA, subB = nB == -INFINITY ? 0.f : nB;
            wA = make_float2(ex2_approx(mA - subA), ex2_approx(ml.x - subA));
            wB = make_float2(ex2_approx(mB - subB), ex2_approx(ml.y - subB));
            mA = nA;
            mB = nB;
            lA = lA * wA.x + ml.z * wA.y;
            lB = lB * wB.x + ml.w * wB.y;
          }
#pragma unroll
          for (int i = 0; i < DP / 8; ++i) {
            const float4 o = *reinterpret_cast<const float4 *>(from + i * kComputeThreads * 16);
            acc[2 * i] = fma2(make_float2(o.x, o.y), make_float2(wA.y, wA.y), mul2(acc[2 * i], make_float2(wA.x, wA.x)));
            acc[2 * i + 1] = fma2(make_float2(o.z, o.w), make_float2(wB.y, wB.y), mul2(acc[2 * i + 1], make_float2(wB.x, wB.x)));
          }
        }
      }
    }
    if (ok && rank == 0) {
      if (PASS == DV) fA = fB = 1.f;
      if (PASS == FORWARD) {
#pragma unroll
        for (int o = 1; o <= 2; o <<= 1) {
          lA += __shfl_xor_sync(0xffffffffu, lA, o);
          lB += __shfl_xor_sync(0xffffffffu, lB, o);
        }
        fA = lA > 0.f ? 1.f / lA : 0.f;  // reference guard, attention_fused.cu:104
        fB = lB > 0.f ? 1.f / lB : 0.f;
      }
      // rows with a result or a sum that is not finite (0 * x is NaN): a bit for each, lane 4 i of rows A and B
      float2 oddA = make_float2(lA * 0.f, 0.f), oddB = make_float2(lB * 0.f, 0.f);
#pragma unroll
      for (int g = 0; g < DP / 8; ++g) {
        oddA = fma2(acc[2 * g], make_float2(0.f, 0.f), oddA);
        oddB = fma2(acc[2 * g + 1], make_float2(0.f, 0.f), oddB);
      }
      auto row_bits = [](bool x) {
        uint32_t bits = __ballot_sync(0xffffffffu, x);
        bits |= bits >> 1;
        return (bits | bits >> 2) & 0x11111111u;
      };
      const uint32_t bitsA = row_bits(rowA < n_res && !(oddA.x + oddA.y == 0.f)), bitsB = row_bits(rowB < n_res && !(oddB.x + oddB.y == 0.f));
      const bool storeA = rowA < n_res && !(bitsA >> (lane & 28) & 1u), storeB = rowB < n_res && !(bitsB >> (lane & 28) & 1u);
      if (PASS == FORWARD && p.lse && t4 == 0) {
        if (storeA) p.lse[elem<1>(s_base + rowA, el_stat, p)] = lA > 0.f ? fmaf(mA, kLn2, logf(lA)) : -INFINITY;
        if (storeB) p.lse[elem<1>(s_base + rowB, el_stat, p)] = lB > 0.f ? fmaf(mB, kLn2, logf(lB)) : -INFINITY;
      }
      float *dst = PASS == FORWARD ? p.out : PASS == DQ ? p.d_q : PASS == DK ? p.d_k : p.d_v;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const long long row = half ? rowB : rowA;
        if (!(half ? storeB : storeA)) continue;
        const float f = half ? fB : fA;
#pragma unroll
        for (int g = 0; g < DP / 8; ++g) {
          const int d = 8 * g + 2 * t4;
          if (d < (int)p.D) *reinterpret_cast<float2 *>(dst + elem<2>(res_base + (size_t)row * dm + d, el_res, p)) = make_float2(acc[2 * g + half].x * f, acc[2 * g + half].y * f);
        }
      }
      odd_rows = bitsA | bitsB << 1;
    }
    if (lane == 0) again[warp] = odd_rows;
  }

  if (CL > 1 && warp >= 8) {  // the compute warps' two meetings
    cluster_sync();
    cluster_sync();
  }

  // ---------------------------------------------------------------- teardown (all roles)
  tc_fence_before_sync();
  __syncthreads();
  // Here, by all warps, and not by the compute warps behind their results: there the loops below cost 2-5 % of every call (registers and instruction
  // fetch; us, without them / there / here: forward and backward 2 x 8 x 1000 x 128 165.0 / 171.0 / 164.4, 1 x 4 x 700 x 96 48.8 / 50.5 / 49.9).
  const uint4 again0 = reinterpret_cast<const uint4 *>(again)[0], again1 = reinterpret_cast<const uint4 *>(again)[1];
  if (__builtin_expect((again0.x | again0.y | again0.z | again0.w | again1.x | again1.y | again1.z | again1.w) != 0u, 0)) {
#pragma unroll 1
    for (int i = warp; i < BM; i += kMmaWarp + 1) {  // row i % 16 of the 16 of compute warp i / 16; bit 4 r of its word is row r, 4 r + 1 row r + 8
      const int w = i >> 4, r = i & 15;
      if (again[w] >> (4 * (r & 7) + (r >> 3)) & 1u) fp32_row<PASS>(p, q_base, k_base, s_base, row0 + (w & 3) * 32 + (w >> 2) * 16 + r);
    }
  }
  if (*abort_flag != 0u) {
    if (warp == kMmaWarp) {
      commit_elected(bar(DRAIN));  // by the lane that issued the MMAs: the election is deterministic
      for (int t = 0; t < (1 << 16) && !mbar_try_wait(bar(DRAIN), 0); ++t) {
      }
    }
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, DEV_STATUS_WAIT_EXPIRED);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

// Heaviest blocks first: the last row block of a causal forward, the first key block.
template <int DP, int CL>
__global__ void __launch_bounds__(kThreads, 1) k_split_fwd(const AttnParams p, const uint32_t tiles) {
  const uint32_t heads = p.B * p.H, block = blockIdx.x / CL, rank = block / heads, bh = block - rank * heads;
  split_block<Cfg<DP, FORWARD>, CL>(p, p.causal ? tiles - 1 - rank : rank, bh);
}
// Rank r of the dK, dQ and dV blocks in turn. dK and dQ blocks take 7/4 of the time of a dV block.
template <int DP, int CL>
__global__ void __launch_bounds__(kThreads, 1) k_split_bwd(const AttnParams p, const uint32_t key_tiles, const uint32_t query_tiles) {
  const uint32_t heads = p.B * p.H, block = blockIdx.x / CL, slot = block / heads, bh = block - slot * heads;
  const uint32_t common = min(key_tiles, query_tiles);
  uint32_t rank, pass;  // pass 0 dK, 1 dQ, 2 dV
  if (slot < 3 * common) {
    rank = slot / 3;
    pass = slot - 3 * rank;
  } else if (key_tiles > query_tiles) {
    rank = common + (slot - 3 * common) / 2;
    pass = ((slot - 3 * common) & 1) * 2;
  } else {
    rank = common + (slot - 3 * common);
    pass = 1;
  }
  if (pass == 0) split_block<Cfg<DP, DK>, CL>(p, rank, bh);
  else if (pass == 1) split_block<Cfg<DP, DQ>, CL>(p, query_tiles - 1 - rank, bh);
  else split_block<Cfg<DP, DV>, CL>(p, rank, bh);
}

// The registers a thread that the kernels are taken to be built with. Another number than kLaunchRegs refuses them all (tests build such a library).
#ifndef DF_SPLIT_BUILT_REGS
#define DF_SPLIT_BUILT_REGS kLaunchRegs
#endif
// DF_OK when the kernel can be launched on the current device. Built for fewer registers it would wait for ever in setmaxnreg: DF_ERR_UNSUPPORTED, and the
// dispatch takes the SIMT kernels.
template <auto K>
int ready(uint32_t bytes) {
  static std::once_flag once[64];
  static int status[64];
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK || dev < 0 || dev >= 64) return DF_ERR_CUDA;
  std::call_once(once[dev], [&]() {
    cudaFuncAttributes attr;
    status[dev] = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess || cudaFuncGetAttributes(&attr, K) != cudaSuccess
                      ? DF_ERR_CUDA
                  : attr.numRegs != DF_SPLIT_BUILT_REGS ? DF_ERR_UNSUPPORTED : DF_OK;
  });
  return status[dev];
}

// What the kernels take from the host beside the caller's parameters. The factor of the scores is rounded once: its error is in every one of them (1 x 4 x
// 260 x 112: O 2.2e-7 off with scale * log2 e from two roundings, 1.5e-7 so). Formed on the device the same number cost 3-6 %
// at some head sizes, by other allocations of registers.
void set_by_host(AttnParams *p) {
  p->scale_log2 = (float)((double)p->scale * 1.4426950408889634);
  p->status = device_status_ptr();
}

template <int DP, int CL>
int forward_form(AttnParams p, cudaStream_t s) {
  constexpr uint32_t smem = Cfg<DP, FORWARD>::kSmem;
  if (const int st = ready<k_split_fwd<DP, CL>>(smem)) return st;
  const uint32_t tiles = (p.Sq + BM - 1) / BM;
  set_by_host(&p);
  launch_clusters(k_split_fwd<DP, CL>, CL > 1 ? CL : 0, dim3(CL * tiles * p.B * p.H), dim3(kThreads), smem, s, p, tiles);
  note_launch();
  return check_cuda(cudaGetLastError());
}
template <int DP, int CL>
int backward_form(AttnParams p, cudaStream_t s) {
  constexpr uint32_t a = Cfg<DP, DK>::kSmem, b = Cfg<DP, DV>::kSmem, smem = a > b ? a : b;
  if (const int st = ready<k_split_bwd<DP, CL>>(smem)) return st;
  const uint32_t kt = (p.Sk + BM - 1) / BM, qt = (p.Sq + BM - 1) / BM;
  set_by_host(&p);
  launch_clusters(k_split_bwd<DP, CL>, CL > 1 ? CL : 0, dim3(CL * (2 * kt + qt) * p.B * p.H), dim3(kThreads), smem, s, p, kt, qt);
  note_launch();
  return check_cuda(cudaGetLastError());
}
template <int DP>
int forward_by_cluster(const AttnParams &p, int cl, cudaStream_t s) {
  return cl == 4 ? forward_form<DP, 4>(p, s) : cl == 2 ? forward_form<DP, 2>(p, s) : forward_form<DP, 1>(p, s);
}
template <int DP>
int backward_by_cluster(const AttnParams &p, int cl, cudaStream_t s) {
  return cl == 4 ? backward_form<DP, 4>(p, s) : cl == 2 ? backward_form<DP, 2>(p, s) : backward_form<DP, 1>(p, s);
}

// From four steps (193 keys) on. Up to two steps attn_simt.cu is as fast (1 x 4 x 100 x 96: forward 9.9 there, 11.1 here; backward 16.8, 14.8); at three it
// takes 1.3 times as long, but its sums are still short and dQ was more exact there when the parts here were cut by truncation (D = 128, S = 130: 3.3e-7
// against 3.8e-7).
constexpr uint64_t kMinSteps = 4;
// The longest block's steps, for queries as resident rows and for keys.
uint64_t query_steps(const AttnParams &p) {
  long long keys = p.Sk;
  if (p.causal && (long long)p.Sq + p.shift < keys) keys = (long long)p.Sq + p.shift;
  return keys > 0 ? (uint64_t)(keys + BN - 1) / BN : 0;
}
uint64_t key_steps(const AttnParams &p) {
  const long long first = p.causal && p.shift < 0 ? -p.shift / BN * BN : 0;
  return first < (long long)p.Sq ? (uint64_t)((long long)p.Sq - first + BN - 1) / BN : 0;
}
uint64_t tiles_of(uint32_t rows) { return ((uint64_t)rows + BM - 1) / BM; }

bool split_supported(const AttnParams &p, std::initializer_list<const float *> ptrs) {
  if (p.D == 0 || p.D > 128 || p.Sq == 0 || p.Sk == 0 || p.B == 0 || p.H == 0) return false;
  if (!(p.scale > 0.0f) || !isfinite(p.scale)) return false;
  if ((uint64_t)p.B * p.H > 65535u || 4 * (2 * tiles_of(p.Sk) + tiles_of(p.Sq)) * p.B * p.H > 0x7fffffffull) return false;
  if (p.shift > (1ll << 32) || p.shift < -(1ll << 32)) return false;
  uintptr_t bits = (uintptr_t)p.D * 4;  // rows are moved 16 bytes at a time
  for (const float *x : ptrs) bits |= reinterpret_cast<uintptr_t>(x);
  return (bits & 15u) == 0;
}

// CTAs that share a block: as many as find an SM each, while they have some steps each (B200, us, one / two / four CTAs, forward: 1 x 4 x 700 x 96 29 / 21 /
// 18, 1 x 6 x 200 x 128 16 / 13.6 / 15.5; backward: 1 x 4 x 700 x 96 45 / 32 / 46, there four do not all run at once). In a causal forward two also
// when they do not, since the longest block is twice the mean (1 x 8 x 1400 x 128 57 / 34, 2 x 8 x 1000 x 128 44 / 39; all keys 46 / 56); the three passes
// of a backward fill the SMs by themselves.
int forward_cluster(const AttnParams &p) {
  const uint64_t blocks = tiles_of(p.Sq) * p.B * p.H, n = query_steps(p), sms = (uint64_t)sm_count();
  if (n >= 8 && 4 * blocks <= sms) return 4;
  return n >= 4 && (2 * blocks <= sms || (p.causal && blocks <= sms)) ? 2 : 1;
}
int backward_cluster(const AttnParams &p) {
  const uint64_t blocks = (2 * tiles_of(p.Sk) + tiles_of(p.Sq)) * p.B * p.H, sms = (uint64_t)sm_count();
  const uint64_t a = query_steps(p), b = key_steps(p), n = a > b ? a : b;
  if (n >= 8 && 4 * blocks <= sms) return 4;
  return n >= 2 && 2 * blocks <= sms ? 2 : 1;
}

}  // namespace

bool split_forward_wanted(const AttnParams &p) {
  return option(DF_OPT_DISABLE_TENSOR) != 1 && p.out != nullptr && p.delta == nullptr && split_supported(p, {p.q, p.k, p.v, p.out}) && query_steps(p) >= kMinSteps;
}
bool split_backward_wanted(const AttnParams &p) {
  return option(DF_OPT_DISABLE_TENSOR) == 0 && split_supported(p, {p.q, p.k, p.v, p.d_out, p.d_q, p.d_k, p.d_v}) && (query_steps(p) >= kMinSteps || key_steps(p) >= kMinSteps);
}
int split_forward(const AttnParams &p, cudaStream_t s) {
  const int cl = forward_cluster(p);
  return p.D <= 32 ? forward_by_cluster<32>(p, cl, s) : p.D <= 64 ? forward_by_cluster<64>(p, cl, s) : p.D <= 96 ? forward_by_cluster<96>(p, cl, s) : forward_by_cluster<128>(p, cl, s);
}
int split_backward(const AttnParams &p, cudaStream_t s) {
  const int cl = backward_cluster(p);
  return p.D <= 32 ? backward_by_cluster<32>(p, cl, s) : p.D <= 64 ? backward_by_cluster<64>(p, cl, s) : p.D <= 96 ? backward_by_cluster<96>(p, cl, s) : backward_by_cluster<128>(p, cl, s);
}

}  // namespace df

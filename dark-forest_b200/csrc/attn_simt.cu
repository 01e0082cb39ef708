// attn_simt.cu - fp32 attention kernels for every shape the tensor-core kernels do not take (any S, 1 <= D <= 128, any
// alignment): short sequences with head sizes other than 64 (longer ones: attn_split_sm100.cu), unaligned slices, tiny problems such as the S=5,D=4 and S=4,D=3 cases that the
// reference's own unit tests use (darkforest-cuda/src/lib.rs:2606-2628, 2753-2769).
//
// Arithmetic follows the reference definition (attention_fused.cu:41-159 forward, :390-516 backward) in full fp32, not
// its structure: the products run as register-tiled matrix products out of shared memory, the forward saves logsumexp, and
// the backward is a dK/dV kernel and a dQ kernel that recompute P from logsumexp, so there is no S x S scratch and no
// atomics: results are bit-reproducible run to run.
//
// What bounds them is the fp32 pipe (128 FMA per clock and SM), then shared-memory reads, so:
//   * what a shared-memory read costs is the bytes it returns to registers (a 16-byte read of a warp takes 4 cycles, 2 when
//     each of its quarters reads at most two addresses), so threads hold tiles of 8 x 4 scores and 8 x 8 outputs: 8 cycles
//     of reads per 8 of FMA in the first products, 12 per 16 in the second; a group of 128 threads covers 64 x 64 scores;
//   * products are accumulated in pairs with fma.rn.f32x2: the pipe's rate is the same, the issue slots are half;
//   * rows lie in shared memory at an odd number of 16-byte units, so that the 8 lanes that read different rows do so
//     without bank conflicts, and arrive by cp.async (16 bytes, or 4 where D or the slice is not 16-byte aligned);
//   * P and dS go through shared memory once, transposed (contraction index first), to be an operand of the second products.
// Blocks own 64 rows, or 32 where 64 would leave SMs without one, heaviest blocks first.
// Measured on B200 against the kernels before (four lanes per row, one score at a time), forward / both halves of the
// backward: B=2, H=8, S=1000, D=128, causal 583 / 1286 us -> 119 / 373; B=1, H=8, S=4096, D=128 3852 / 8507 -> 813 / 2642
// (42 TFLOP/s, the two products alone run at 53 and 65 of the pipe's 72); B=1, H=8, S=1000, D=32 287 / 610 -> 35 / 80.
#include <math.h>

#include <initializer_list>
#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {
namespace {

using ptx::ex2_approx;  // exponentials are taken as 2^x of scores scaled by scale * log2 e; maxima are in the same unit
using ptx::fma2;

constexpr int kCols = 64;      // loop-side rows (keys, or queries in the dK/dV part) per step
constexpr int NT = 128;        // threads of a group; a block is two groups
constexpr int TX = 16, TY = 8; // a group's threads along the loop-side rows (and the head dimension), and along the resident rows
constexpr int C = kCols / TX;

__device__ __forceinline__ int clamp_int(long long x) { return x > 1000 ? 1000 : (x < -1000 ? -1000 : (int)x); }
__device__ __forceinline__ void cp16(uint32_t dst, const float *src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const float *src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One head's slice of a [*, H*D] tensor: rows [0, nrows), `total` elements of the whole tensor (checked builds).
struct Slice {
  const float *src;
  size_t base, dm, total;
  long long nrows;
};

// Starts the copies of rows row0 .. row0 + rows - 1 to dst[row * ld + d]; rows past the end are zero-filled. A warp takes
// every (NTH / 32)-th row; `rows` is a multiple of NTH / 32 or zero.
template <int NTH>
__device__ __forceinline__ void load_rows(float *dst, int ld, const Slice &t, long long row0, int rows, uint32_t D, bool vec, int tid,
                                          unsigned int *status) {
  (void)status;
  constexpr int W = NTH / 32;
  const int warp = tid >> 5, lane = tid & 31;
  const long long left = t.nrows - row0;
  const int n_ok = left < rows ? (left > 0 ? (int)left : 0) : rows;
  size_t at = t.base + (size_t)(row0 + warp) * t.dm;
  uint32_t to = ptx::smem_u32(dst) + (uint32_t)(warp * ld) * 4u;
  if (vec) {
    if (4u * lane < D) {
      at += 4 * lane;
      to += 16 * lane;
#pragma unroll 4
      for (int r = warp; r < rows; r += W, at += W * t.dm, to += (uint32_t)(W * ld) * 4u) {
        const bool ok = r < n_ok;
#ifdef DF_BOUNDS_CHECK
        if (ok) DF_IDX(at + 3, t.total, status);
#endif
        cp16(to, ok ? t.src + DF_IDX(at, t.total, status) : t.src, ok);
      }
    }
  } else {
    for (int r = warp; r < rows; r += W, at += W * t.dm, to += (uint32_t)(W * ld) * 4u) {
      const bool ok = r < n_ok;
      for (uint32_t d = lane; d < D; d += 32) cp4(to + 4 * d, ok ? t.src + DF_IDX(at + d, t.total, status) : t.src, ok);
    }
  }
}

// The columns between D and the next multiple of four are read by the first products: they are zeroed once per tile buffer.
template <int NT>
__device__ __forceinline__ void zero_tail(float *dst, int ld, int rows, uint32_t D, int tid) {
  const uint32_t tail = (4u - (D & 3u)) & 3u;
  for (uint32_t i = tid; i < rows * tail; i += NT) dst[(i / tail) * ld + D + i % tail] = 0.0f;
}

// acc[i][j] = sum_d a[ty + TY * i][d] * b[tx + TX * j][d]: first products (scores, dP). Sums of even and odd d are kept apart.
template <int R>
__device__ __forceinline__ void product_nt(float2 (&acc)[R][C], const float *a, const float *b, int ld, uint32_t nd4, int ty, int tx) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
  const float *pa = a + ty * ld, *pb = b + tx * ld;
#pragma unroll 4
  for (uint32_t d = 0; d < nd4; ++d) {
    float4 bv[C];
#pragma unroll
    for (int j = 0; j < C; ++j) bv[j] = *reinterpret_cast<const float4 *>(pb + j * TX * ld + 4 * d);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 av = *reinterpret_cast<const float4 *>(pa + i * TY * ld + 4 * d);
#pragma unroll
      for (int j = 0; j < C; ++j) acc[i][j] = fma2(make_float2(av.x, av.y), make_float2(bv[j].x, bv[j].y), acc[i][j]);
#pragma unroll
      for (int j = 0; j < C; ++j) acc[i][j] = fma2(make_float2(av.z, av.w), make_float2(bv[j].z, bv[j].w), acc[i][j]);
    }
  }
}

// A thread's share of the head dimension in the second products: CG groups of VW consecutive dims, group g at
// (g * TX + tx) * VW. Pairs of dims lie together.
template <int R, int VW, int CG>
using OutTile = float2[R][CG * VW / 2];

// acc[i][.] += sum_j t[j][ty * R + i] * m[j][dims], j < rows: second products. `t` is a transposed tile of row stride ldt.
template <int R, int VW, int CG>
__device__ __forceinline__ void product_tn(OutTile<R, VW, CG> &acc, const float *t, int ldt, const float *m, int ld, int rows, int ty, int tx) {
  const float *pt = t + ty * R, *pm = m + tx * VW;
#pragma unroll 2
  for (int j = 0; j < rows; ++j) {
    float tv[R];
#pragma unroll
    for (int i = 0; i < R; i += 4) {
      const float4 x = *reinterpret_cast<const float4 *>(pt + j * ldt + i);
      tv[i] = x.x; tv[i + 1] = x.y; tv[i + 2] = x.z; tv[i + 3] = x.w;
    }
    float2 mv[CG * VW / 2];
#pragma unroll
    for (int g = 0; g < CG; ++g) {
      if constexpr (VW == 4) {
        const float4 x = *reinterpret_cast<const float4 *>(pm + j * ld + g * TX * VW);
        mv[2 * g] = make_float2(x.x, x.y);
        mv[2 * g + 1] = make_float2(x.z, x.w);
      } else {
        mv[g] = *reinterpret_cast<const float2 *>(pm + j * ld + g * TX * VW);
      }
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < CG * VW / 2; ++c) acc[i][c] = fma2(make_float2(tv[i], tv[i]), mv[c], acc[i][c]);
  }
}

// t[col][ty * R + i] = v[i]: one column of a thread's tile, transposed.
template <int R>
__device__ __forceinline__ void store_column(float *t, int ldt, int col, int ty, const float (&v)[R]) {
  float *p = t + col * ldt + ty * R;
#pragma unroll
  for (int i = 0; i < R; i += 4) *reinterpret_cast<float4 *>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}

// Writes a thread's output tile, times `f[i]`, to rows row0 + ty + TY * i.
template <int R, int VW, int CG>
__device__ __forceinline__ void write_rows(float *dst, const OutTile<R, VW, CG> &acc, const float (&f)[R], size_t base, size_t dm, size_t total,
                                           long long row0, long long nrows, uint32_t D, int ty, int tx, unsigned int *status) {
  (void)total;
  (void)status;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const long long row = row0 + ty + TY * i;
    if (row >= nrows) continue;
#pragma unroll
    for (int c = 0; c < CG * VW / 2; ++c) {
      const uint32_t d = (uint32_t)(((c * 2) / VW * TX + tx) * VW + (c * 2) % VW);
      const size_t at = base + (size_t)row * dm + d;
      if (d < D) dst[DF_IDX(at, total, status)] = acc[i][c].x * f[i];
      if (d + 1 < D) dst[DF_IDX(at + 1, total, status)] = acc[i][c].y * f[i];
    }
  }
}

// Which block of rows, and which (batch, head), a CTA of the forward works on: heaviest blocks first.
struct Order {
  uint32_t tiles;       // row blocks per (batch, head)
  uint32_t heads;       // B * H
  uint32_t heavy_last;  // 1: the last row block is the heaviest (causal problems)
};
__device__ __forceinline__ void my_block(const Order &o, uint32_t *tile, uint32_t *bh) {
  const uint32_t rank = blockIdx.x / o.heads;
  *bh = blockIdx.x - rank * o.heads;
  *tile = o.heavy_last ? o.tiles - 1 - rank : rank;
}

// ---------------------------------------------------------------------------------------
// Forward: two groups of 128 threads; a thread owns R rows (ty + 8 i) and, of a step's 64 keys, tx + 16 j. The groups take alternate key tiles of the block's rows into running maxima, sums and outputs of their own and merge them
// at the end: the copies and exponentials of one run under the products of the other, and the longest row block of a small
// problem takes half the steps. Optional outputs: out, lse; "stats" output: delta = rowsum(dO * O) without
// materialising O (used by the legacy backward when the caller's scratch cannot hold O). The transposed P tile takes the
// place of the K tile, which is used up by then.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }

template <int R, int VW, int CG>
__global__ void __launch_bounds__(256, 1) k_simt_fwd(const AttnParams p, const Order order, const int ld, const int vec) {
  ptx::pdl_wait();
  constexpr int BM = TY * R, LDT = BM + 4;
  extern __shared__ __align__(16) float smem[];
  const int group = threadIdx.x / NT, tid = threadIdx.x % NT, tx = tid % TX, ty = tid / TX;
  const int kv = kCols * ld, kt = kv > kCols * LDT ? kv : kCols * LDT;
  float *sQ = smem, *sV = sQ + BM * ld + group * (kv + kt), *sK = sV + kv, *sT = sK;
  uint32_t tile, bh;
  my_block(order, &tile, &bh);
  const uint32_t b = bh / p.H, h = bh % p.H, nd4 = (p.D + 3) / 4;
  const size_t dm = (size_t)p.H * p.D;
  const size_t q_base = (size_t)b * p.Sq * dm + (size_t)h * p.D, k_base = (size_t)b * p.Sk * dm + (size_t)h * p.D;
  const size_t n_q = (size_t)p.B * p.Sq * dm, n_k = (size_t)p.B * p.Sk * dm, n_s = (size_t)p.B * p.H * p.Sq;
  (void)n_s;
  const Slice q = {p.q, q_base, dm, n_q, p.Sq}, k = {p.k, k_base, dm, n_k, p.Sk}, v = {p.v, k_base, dm, n_k, p.Sk};
  const long long row0 = (long long)tile * BM;
  const long long last = row0 + BM < (long long)p.Sq ? row0 + BM : (long long)p.Sq;  // rows [row0, last)
  long long kmax = p.causal ? last + p.shift : (long long)p.Sk;
  if (kmax > (long long)p.Sk) kmax = p.Sk;

  zero_tail<256>(sQ, ld, BM, p.D, threadIdx.x);
  load_rows<256>(sQ, ld, q, row0, BM, p.D, vec, threadIdx.x, p.status);
  cp_commit();
  load_rows<NT>(sK, ld, k, group * kCols, kCols, p.D, vec, tid, p.status);
  cp_commit();
  load_rows<NT>(sV, ld, v, group * kCols, kCols, p.D, vec, tid, p.status);
  cp_commit();
  cp_wait<2>();
  __syncthreads();

  const float scale2 = p.scale * kLog2e;
  OutTile<R, VW, CG> acc;
  float m[R], l[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.0f;
#pragma unroll
    for (int c = 0; c < CG * VW / 2; ++c) acc[i][c] = make_float2(0.0f, 0.0f);
  }
  for (long long k0 = group * kCols; k0 < kmax; k0 += 2 * kCols) {
    zero_tail<NT>(sK, ld, kCols, p.D, tid);
    cp_wait<1>();
    group_sync(group);
    float2 s2[R][C];
    product_nt<R>(s2, sQ, sK, ld, nd4, ty, tx);
    group_sync(group);  // the group is done with K: its place takes the transposed P
    // key k0 + c is visible to row row0 + r iff c < min(Sk - k0, r + off), and to every row when the tile is `full`
    const int cols = clamp_int((long long)p.Sk - k0), off = p.causal ? clamp_int(row0 + p.shift + 1 - k0) : 1000;
    const bool full = cols >= kCols && off >= kCols;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int n_vis = full ? kCols : min(cols, ty + TY * i + off);
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < C; ++j) {
        s2[i][j].x = tx + TX * j < n_vis ? (s2[i][j].x + s2[i][j].y) * scale2 : -INFINITY;
        top = fmaxf(top, s2[i][j].x);
      }
#pragma unroll
      for (int o = TX / 2; o >= 1; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (__any_sync(0xffffffffu, top > m[i])) {
        const float mn = fmaxf(m[i], top), alpha = mn == -INFINITY ? 1.0f : ex2_approx(m[i] - mn);  // m = -inf before the first visible key: 0
        m[i] = mn;
        l[i] *= alpha;
#pragma unroll
        for (int c = 0; c < CG * VW / 2; ++c) acc[i][c] = make_float2(acc[i][c].x * alpha, acc[i][c].y * alpha);
      }
      const float ms = m[i] == -INFINITY ? 0.0f : m[i];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        s2[i][j].x = ex2_approx(s2[i][j].x - ms);
        l[i] += s2[i][j].x;
      }
    }
#pragma unroll
    for (int j = 0; j < C; ++j) {
      float pr[R];
#pragma unroll
      for (int i = 0; i < R; ++i) pr[i] = s2[i][j].x;
      store_column<R>(sT, LDT, tx + TX * j, ty, pr);
    }
    cp_wait<0>();
    group_sync(group);
    product_tn<R, VW, CG>(acc, sT, LDT, sV, ld, kCols, ty, tx);
    group_sync(group);
    if (k0 + 2 * kCols < kmax) {
      load_rows<NT>(sK, ld, k, k0 + 2 * kCols, kCols, p.D, vec, tid, p.status);
      cp_commit();
      load_rows<NT>(sV, ld, v, k0 + 2 * kCols, kCols, p.D, vec, tid, p.status);
      cp_commit();
    }
  }
  cp_wait<0>();
  __syncthreads();
  // merge: the second group hands over (m, l, O) through its own tile buffers; both sums are over the lanes of a row first
  float *sO = smem + BM * ld + (kv + kt), *sM = smem + BM * ld;  // O in the second group's buffers, (m, l) in the first's
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int o = TX / 2; o >= 1; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);
  if (group == 1) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      sM[(2 * i) * NT + tid] = m[i];
      sM[(2 * i + 1) * NT + tid] = l[i];
#pragma unroll
      for (int c = 0; c < CG * VW / 2; ++c) *reinterpret_cast<float2 *>(sO + ((size_t)(i * CG * VW / 2 + c) * NT + tid) * 2) = acc[i][c];
    }
  }
  __syncthreads();
  if (group == 1) return;
  float inv[R];
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float mo = sM[(2 * i) * NT + tid], lo = sM[(2 * i + 1) * NT + tid];
    const float mn = fmaxf(m[i], mo), ms = mn == -INFINITY ? 0.0f : mn, wa = ex2_approx(m[i] - ms), wb = ex2_approx(mo - ms);
    m[i] = mn;
    l[i] = l[i] * wa + lo * wb;
#pragma unroll
    for (int c = 0; c < CG * VW / 2; ++c) {
      const float2 o2 = *reinterpret_cast<const float2 *>(sO + ((size_t)(i * CG * VW / 2 + c) * NT + tid) * 2);
      acc[i][c] = make_float2(acc[i][c].x * wa + o2.x * wb, acc[i][c].y * wa + o2.y * wb);
    }
    inv[i] = l[i] > 0.0f ? 1.0f / l[i] : 0.0f;  // reference guard, attention_fused.cu:104
    const long long row = row0 + ty + TY * i;
    if (p.delta) {
      float dp = 0.0f;
      if (row < (long long)p.Sq) {
#pragma unroll
        for (int c = 0; c < CG * VW / 2; ++c) {
          const uint32_t d = (uint32_t)(((c * 2) / VW * TX + tx) * VW + (c * 2) % VW);
          const size_t at = q_base + (size_t)row * dm + d;
          if (d < p.D) dp = fmaf(acc[i][c].x * inv[i], __ldg(p.d_out + DF_IDX(at, n_q, p.status)), dp);
          if (d + 1 < p.D) dp = fmaf(acc[i][c].y * inv[i], __ldg(p.d_out + DF_IDX(at + 1, n_q, p.status)), dp);
        }
      }
#pragma unroll
      for (int o = TX / 2; o >= 1; o >>= 1) dp += __shfl_xor_sync(0xffffffffu, dp, o);
      if (tx == 0 && row < (long long)p.Sq) p.delta[DF_IDX((size_t)bh * p.Sq + (size_t)row, n_s, p.status)] = dp;
    }
    if (p.lse && tx == 0 && row < (long long)p.Sq)
      p.lse[DF_IDX((size_t)bh * p.Sq + (size_t)row, n_s, p.status)] = l[i] > 0.0f ? fmaf(m[i], kLn2, logf(l[i])) : -INFINITY;
  }
  if (p.out) write_rows<R, VW, CG>(p.out, acc, inv, q_base, dm, n_q, row0, p.Sq, p.D, ty, tx, p.status);
}

// ---------------------------------------------------------------------------------------
// Backward, both halves from one text. A thread owns R rows (ty + 8 i) of the resident side and, of a step's 64 rows of the
// loop side, tx + 16 j.
//   DKDV: resident keys (K, V), loop over the queries that see them (Q, dO):  dV += P^T dO,  dK += scale * dS^T Q
//   else: resident queries (Q, dO), loop over their visible keys (K, V):      dQ += scale * dS K
//   P = exp(scale * Q K^T - lse); dP = dO V^T; dS = P * (dP - delta)
// The first group forms the scores and P, the second dP. DKDV: the second group then turns P and its dP into dS and adds to
// dK while the first adds to dV. Otherwise both turn half of the step's keys into dS and add those to a dQ of their own; the
// two meet at the end. The loop side's first operand (Q or K) is double-buffered, its second one is not (shared memory is
// full at D = 128). The halves share a launch, so that the small blocks of one fill the SMs that the other leaves.
// ---------------------------------------------------------------------------------------
template <bool DKDV, int R, int VW, int CG>
__device__ __forceinline__ void backward_block(const AttnParams &p, uint32_t tile, uint32_t bh, const int ld, const int vec, float *smem) {
  constexpr int BM = TY * R, LDT = BM + 4, kAll = 2 * NT;
  float *sA1 = smem, *sA2 = sA1 + BM * ld, *sB1 = sA2 + BM * ld, *sB2 = sB1 + 2 * kCols * ld;
  float *sT1 = sB2 + kCols * ld, *sT2 = sT1 + kCols * LDT, *sStats = sT2 + kCols * LDT;
  const int group = threadIdx.x / NT, tid = threadIdx.x % NT, tx = tid % TX, ty = tid / TX;
  const uint32_t b = bh / p.H, h = bh % p.H, nd4 = (p.D + 3) / 4;
  const size_t dm = (size_t)p.H * p.D;
  const size_t q_base = (size_t)b * p.Sq * dm + (size_t)h * p.D, k_base = (size_t)b * p.Sk * dm + (size_t)h * p.D;
  const size_t n_q = (size_t)p.B * p.Sq * dm, n_k = (size_t)p.B * p.Sk * dm, n_s = (size_t)p.B * p.H * p.Sq, s_base = (size_t)bh * p.Sq;
  (void)n_s;
  const Slice q = {p.q, q_base, dm, n_q, p.Sq}, g = {p.d_out, q_base, dm, n_q, p.Sq}, k = {p.k, k_base, dm, n_k, p.Sk},
              v = {p.v, k_base, dm, n_k, p.Sk};
  const Slice &a1 = DKDV ? k : q, &a2 = DKDV ? v : g, &b1 = DKDV ? q : k, &b2 = DKDV ? g : v;
  const long long row0 = (long long)tile * BM;
  long long begin = 0, end = b1.nrows;  // loop-side rows
  if (p.causal) {
    if (DKDV) {  // first query that sees any key of this block
      begin = row0 - p.shift;
      begin = begin < 0 ? 0 : begin / kCols * kCols;
    } else {
      const long long last = row0 + BM < (long long)p.Sq ? row0 + BM : (long long)p.Sq;
      if (last + p.shift < end) end = last + p.shift;
    }
  }
  // Row statistics of the queries, in the unit of the exponentials: of a step's queries (DKDV; two sets in turn, the second
  // group still reads the last step's when the next ones come), else of the block's own. A row that sees no key has
  // lse = -inf; stored as +inf it gives P = 0.
  auto load_stats = [&](float *stats, long long first, int rows) {
    if ((int)threadIdx.x < rows) {
      const long long i = first + threadIdx.x;
      const float lse = i < (long long)p.Sq ? __ldg(p.lse_in + DF_IDX(s_base + i, n_s, p.status)) : -INFINITY;
      stats[threadIdx.x] = lse == -INFINITY ? INFINITY : lse * kLog2e;
      stats[kCols + threadIdx.x] = i < (long long)p.Sq ? __ldg(p.delta_in + DF_IDX(s_base + i, n_s, p.status)) : 0.0f;
    }
  };
  const float scale2 = p.scale * kLog2e;
  OutTile<R, VW, CG> acc;  // dV of the first group and dK of the second, or a share of dQ
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int c = 0; c < CG * VW / 2; ++c) acc[i][c] = make_float2(0.0f, 0.0f);

  zero_tail<kAll>(sA1, ld, 2 * BM, p.D, threadIdx.x);
  zero_tail<kAll>(sB1, ld, 3 * kCols, p.D, threadIdx.x);
  load_rows<kAll>(sA1, ld, a1, row0, BM, p.D, vec, threadIdx.x, p.status);
  load_rows<kAll>(sA2, ld, a2, row0, BM, p.D, vec, threadIdx.x, p.status);
  load_rows<kAll>(sB1, ld, b1, begin, kCols, p.D, vec, threadIdx.x, p.status);
  load_rows<kAll>(sB2, ld, b2, begin, kCols, p.D, vec, threadIdx.x, p.status);
  cp_commit();
  if (!DKDV) load_stats(sStats, row0, BM);

  int buf = 0;
  for (long long c0 = begin; c0 < end; c0 += kCols, buf ^= 1) {
    const float *sB1c = sB1 + buf * kCols * ld;
    float *stats = DKDV ? sStats + buf * 2 * kCols : sStats;
    const int more = c0 + kCols < end ? kCols : 0;
    if (DKDV) load_stats(stats, c0, kCols);
    cp_wait<0>();
    __syncthreads();
    float2 s2[R][C];
    product_nt<R>(s2, group ? sA2 : sA1, group ? sB2 : sB1c, ld, nd4, ty, tx);
    if (group == 0) {
      // resident row r and loop row c see each other iff c >= r + off (DKDV: queries c of keys r) or c <= r + off
      const int off = p.causal ? (DKDV ? clamp_int(row0 - c0 - p.shift) : clamp_int(row0 + p.shift - c0)) : (DKDV ? -1000 : 1000);
      const int keys_left = clamp_int((long long)p.Sk - (DKDV ? row0 : c0));  // keys of the resident or loop side that exist
      const bool full = (DKDV ? off + BM <= 1 : off >= kCols - 1) && keys_left >= (DKDV ? BM : kCols);
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const int col = tx + TX * j;
        float pr[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const int row = ty + TY * i;
          const bool vis = full || (DKDV ? (col >= row + off && row < keys_left) : (col <= row + off && col < keys_left));
          const float x = (s2[i][j].x + s2[i][j].y) * scale2 - stats[DKDV ? col : row];
          pr[i] = vis ? ex2_approx(x) : 0.0f;
        }
        store_column<R>(sT1, LDT, col, ty, pr);
      }
    } else if (DKDV) {
      load_rows<NT>(sB1 + (buf ^ 1) * kCols * ld, ld, b1, c0 + kCols, more, p.D, vec, tid, p.status);
      cp_commit();
    } else {
#pragma unroll
      for (int j = 0; j < C; ++j) {
        float dp[R];
#pragma unroll
        for (int i = 0; i < R; ++i) dp[i] = (s2[i][j].x + s2[i][j].y) - stats[kCols + ty + TY * i];
        store_column<R>(sT2, LDT, tx + TX * j, ty, dp);
      }
      load_rows<NT>(sB1 + (buf ^ 1) * kCols * ld, ld, b1, c0 + kCols, more, p.D, vec, tid, p.status);
      group_sync(group);  // V is used up
      load_rows<NT>(sB2, ld, b2, c0 + kCols, more, p.D, vec, tid, p.status);
      cp_commit();
    }
    __syncthreads();
    if (DKDV) {
      if (group == 0) {
        product_tn<R, VW, CG>(acc, sT1, LDT, sB2, ld, kCols, ty, tx);
        group_sync(group);  // dO is used up
        load_rows<NT>(sB2, ld, b2, c0 + kCols, more, p.D, vec, tid, p.status);
        cp_commit();
      } else {
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const int col = tx + TX * j;
          float ds[R];
#pragma unroll
          for (int i = 0; i < R; i += 4) {
            const float4 x = *reinterpret_cast<const float4 *>(sT1 + col * LDT + ty * R + i);
            ds[i] = x.x; ds[i + 1] = x.y; ds[i + 2] = x.z; ds[i + 3] = x.w;
          }
#pragma unroll
          for (int i = 0; i < R; ++i) ds[i] *= (s2[i][j].x + s2[i][j].y) - stats[kCols + col];
          store_column<R>(sT2, LDT, col, ty, ds);
        }
        group_sync(group);
        product_tn<R, VW, CG>(acc, sT2, LDT, sB1c, ld, kCols, ty, tx);
      }
    } else {
      float *t1 = sT1 + group * (kCols / 2) * LDT, *t2 = sT2 + group * (kCols / 2) * LDT;  // this group's half of the keys
      for (int e = 4 * tid; e < (kCols / 2) * BM; e += 4 * NT) {
        const int at = e / BM * LDT + e % BM;
        const float4 x = *reinterpret_cast<const float4 *>(t1 + at), y = *reinterpret_cast<const float4 *>(t2 + at);
        *reinterpret_cast<float4 *>(t2 + at) = make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w);
      }
      group_sync(group);
      product_tn<R, VW, CG>(acc, t2, LDT, sB1c + group * (kCols / 2) * ld, ld, kCols / 2, ty, tx);
    }
  }
  cp_wait<0>();
  float scale[R];
#pragma unroll
  for (int i = 0; i < R; ++i) scale[i] = DKDV && group == 0 ? 1.0f : p.scale;
  if (DKDV) {
    write_rows<R, VW, CG>(group ? p.d_k : p.d_v, acc, scale, k_base, dm, n_k, row0, p.Sk, p.D, ty, tx, p.status);
  } else {
    __syncthreads();
    float2 *half = reinterpret_cast<float2 *>(sB1);  // the second group's share of dQ
    if (group == 1) {
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < CG * VW / 2; ++c) half[(i * CG * VW / 2 + c) * NT + tid] = acc[i][c];
    }
    __syncthreads();
    if (group == 1) return;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < CG * VW / 2; ++c) {
        const float2 o = half[(i * CG * VW / 2 + c) * NT + tid];
        acc[i][c] = make_float2(acc[i][c].x + o.x, acc[i][c].y + o.y);
      }
    write_rows<R, VW, CG>(p.d_q, acc, scale, q_base, dm, n_q, row0, p.Sq, p.D, ty, tx, p.status);
  }
}

// Blocks of both halves, heaviest first: rank r of the dK/dV blocks (4 products a step), then rank r of the dQ blocks (3).
template <int R, int VW, int CG>
__global__ void __launch_bounds__(256, 1) k_simt_bwd(const AttnParams p, const uint32_t key_tiles, const uint32_t query_tiles, const int ld,
                                                     const int vec) {
  ptx::pdl_wait();
  extern __shared__ __align__(16) float smem[];
  const uint32_t heads = p.B * p.H, slot = blockIdx.x / heads, bh = blockIdx.x - slot * heads;
  const uint32_t both = 2 * min(key_tiles, query_tiles);
  const bool dkdv = slot < both ? (slot & 1) == 0 : key_tiles > query_tiles;
  const uint32_t rank = slot < both ? slot >> 1 : slot - both / 2;
  if (dkdv) backward_block<true, R, VW, CG>(p, rank, bh, ld, vec, smem);
  else backward_block<false, R, VW, CG>(p, query_tiles - 1 - rank, bh, ld, vec, smem);
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
// Every kernel may use the whole shared memory of an SM (asked once per device and kernel).
template <auto K>
bool allow_smem() {
  static std::once_flag once[64];
  static bool ok[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  std::call_once(once[dev], [&]() { ok[dev] = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess; });
  if (!ok[dev]) note_status(DF_ERR_CUDA);
  return ok[dev];
}

// checked builds hand the kernels the device status word that their index checks report to
AttnParams with_status(const AttnParams &p) {
  AttnParams q = p;
#ifdef DF_BOUNDS_CHECK
  q.status = device_status_ptr();
#endif
  return q;
}

// Row stride in shared memory: an odd number of 16-byte units.
int row_stride(uint32_t D) { return 4 * (int)(((D + 3) / 4) | 1u); }

int aligned_rows(uint32_t D, std::initializer_list<const float *> ptrs) {
  uintptr_t bits = (D & 3u) ? 1 : 0;
  for (const float *x : ptrs) bits |= reinterpret_cast<uintptr_t>(x) & 15u;
  return bits == 0;
}

// 64-row blocks, unless 32-row blocks are needed to give every SM one.
bool wide_blocks(uint64_t rows, const AttnParams &p) { return (rows + 63) / 64 * p.B * p.H >= (uint64_t)sm_count(); }

// The second products cover a multiple of 32 dims. Their last row reads past a narrower tile, hence the slack at the end.
constexpr size_t kSlack = 128;

template <int R, int VW, int CG>
int forward_form(const AttnParams &p, cudaStream_t s) {
  constexpr int BM = TY * R;
  if (!allow_smem<k_simt_fwd<R, VW, CG>>()) return DF_ERR_CUDA;
  const int ld = row_stride(p.D);
  const size_t kv = (size_t)kCols * ld, t = (size_t)kCols * (BM + 4), kt = kv > t ? kv : t;
  const size_t o = (size_t)R * CG * VW * NT, q = (size_t)BM * ld;
  const size_t second = kv + kt > o ? kv + kt : o;  // the second group's buffers also carry its output to the first
  Order order;
  order.tiles = (p.Sq + BM - 1) / BM;
  order.heads = p.B * p.H;
  order.heavy_last = p.causal != 0;
  const uint64_t blocks = (uint64_t)order.tiles * order.heads;
  if (blocks > 0x7fffffffull) return DF_ERR_UNSUPPORTED;
  launch_kernel(k_simt_fwd<R, VW, CG>, dim3((unsigned)blocks), dim3(256), (q + kv + kt + second + kSlack) * sizeof(float), s, with_status(p), order, ld, aligned_rows(p.D, {p.q, p.k, p.v}));
  note_launch();
  return check_cuda(cudaGetLastError());
}

template <int R, int VW, int CG>
int backward_form(const AttnParams &p, cudaStream_t s) {
  constexpr int BM = TY * R;
  if (!allow_smem<k_simt_bwd<R, VW, CG>>()) return DF_ERR_CUDA;
  const int ld = row_stride(p.D);
  const size_t tiles = (size_t)3 * kCols * ld + 2 * (size_t)kCols * (BM + 4) + 4 * kCols, half = (size_t)R * CG * VW * NT;
  const size_t floats = (size_t)2 * BM * ld + (tiles > half ? tiles : half) + kSlack;
  const uint32_t key_tiles = (p.Sk + BM - 1) / BM, query_tiles = (p.Sq + BM - 1) / BM;
  const uint64_t blocks = ((uint64_t)key_tiles + query_tiles) * p.B * p.H;
  if (blocks > 0x7fffffffull) return DF_ERR_UNSUPPORTED;
  launch_kernel(k_simt_bwd<R, VW, CG>, dim3((unsigned)blocks), dim3(256), floats * sizeof(float), s, with_status(p), key_tiles, query_tiles, ld,
                                                                            aligned_rows(p.D, {p.q, p.k, p.v, p.d_out}));
  note_launch();
  return check_cuda(cudaGetLastError());
}

// 16 threads x CG groups of VW dims cover 32, 64, 96 or 128 dims.
#define DF_BY_HEAD_DIM(FORM, R)                                                                       \
  (p.D <= 32 ? FORM<R, 2, 1>(p, s) : p.D <= 64 ? FORM<R, 4, 1>(p, s) : p.D <= 96 ? FORM<R, 2, 3>(p, s) \
                                                                                  : FORM<R, 4, 2>(p, s))

}  // namespace

int generic_forward(const AttnParams &p, cudaStream_t s) {
  if (p.Sq == 0 || p.B == 0 || p.H == 0) return DF_OK;
  if ((uint64_t)p.B * p.H > 65535u) return DF_ERR_UNSUPPORTED;  // refused before any CUDA call, as callers were told
  return wide_blocks(p.Sq, p) ? DF_BY_HEAD_DIM(forward_form, 8) : DF_BY_HEAD_DIM(forward_form, 4);
}

// dQ, dK and dV from lse_in and delta_in; with no keys (or no queries) the other side's gradients are zero.
int generic_backward(const AttnParams &p, cudaStream_t s) {
  if ((p.Sq == 0 && p.Sk == 0) || p.B == 0 || p.H == 0) return DF_OK;
  if ((uint64_t)p.B * p.H > 65535u) return DF_ERR_UNSUPPORTED;  // refused before any CUDA call, as callers were told
  return wide_blocks((uint64_t)p.Sq + p.Sk, p) ? DF_BY_HEAD_DIM(backward_form, 8) : DF_BY_HEAD_DIM(backward_form, 4);
}

}  // namespace df

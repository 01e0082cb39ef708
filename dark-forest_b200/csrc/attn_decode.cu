// attn_decode.cu — one-token (decode) attention over a KV cache for B200 (sm_100a).
//
// Replaces kernel_fused_mha_decode_kv, its split-K form with kernel_fused_mha_decode_kv_reduce,
// and the paged / paged split-K / paged bf16 forms
// (darkforest-cuda/kernels/attention_fused.cu:551-626, 635-788, 796-1090): per head
//   out = softmax(scale * q K^T) V   over the first cur_seq_len tokens of the cache.
// The reference runs one warp per head (grid = n_heads), i.e. a dozen warps on the whole GPU.
// This path is pure HBM streaming (2 * T * H * D elements read once), so the tokens of every head are split over many
// CTAs, and what decides the rate is how many bytes every SM keeps in flight:
//   * k_attn_decode_ring (rows on 16- or 8-byte boundaries): every thread owns a private ring in shared memory that it
//     fills with cp.async two to three stages ahead of the one it works on; a group of 8 or 16 lanes covers one K or V
//     row and keeps an online-softmax state, and the rows of the next stage (block-table entries of a paged cache) are
//     resolved one stage before their loads are issued;
//   * k_attn_decode_any: any head size and alignment, scalar loads straight into registers;
//   * entry points WITHOUT scratch buffers launch one cluster of up to 16 CTAs per head: the partial states meet in the
//     shared memory of the cluster's first CTA;
//   * the split-K entry points write one partial state (m, l, o[D]) per CTA into the caller's partial buffers (never
//     more chunks than the caller's ceil(T / chunk_size)) and a second, tiny kernel merges them - the same max / exp
//     rescale as the reference's reduce kernel.
// Paged caches resolve the physical page of a token through the int32 block table; the bf16 pool
// variant converts on load. Arithmetic is fp32 throughout (exp2 with the scale folded in).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <float.h>
#include <math.h>

#include <initializer_list>
#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace cg = cooperative_groups;

namespace df {
namespace {

using ptx::ex2_approx;
using ptx::fma2;

constexpr int kMaxWarps = 16;
constexpr int kMaxCluster = 16;     // CTAs per head in the scratch-free form (above 8: non-portable, asked of the device once)

struct DecParams {
  const float *q;
  const void *k, *v;              // fp32 or bf16 rows of n_heads * d_head elements
  const int32_t *block_table;     // nullptr: contiguous cache
  float *out;
  float *pm, *pl, *po;            // partial states (split form only)
  uint32_t H, T, D, page_size;
  uint32_t chunk;                 // tokens per CTA
  uint32_t n_chunks;
  float scale_log2;
};

// What a CTA's warps leave behind, and (in the first CTA of a cluster) what the cluster's CTAs send.
struct MergeSmem {
  float m[kMaxWarps], l[kMaxWarps];
  float o[kMaxWarps][128];
  float cm[kMaxCluster], cl[kMaxCluster];
  float co[kMaxCluster][128];
};

// Merges the CTA's warp states (already in sm->m, l, o) and hands the result on: one partial state per CTA to the
// partial buffers (SPLIT), or into the shared memory of the cluster's first CTA, which writes the output.
// A state without tokens has m = -FLT_MAX, l = 0, o = 0. The cluster barrier was entered at kernel start, so by now every
// CTA of the cluster is running and its shared memory may be written.
template <bool SPLIT, int kWarps>
__device__ __forceinline__ void merge_and_write(const DecParams &p, MergeSmem *sm, uint32_t h, uint32_t chunk_idx) {
  __syncthreads();
  const uint32_t d = threadIdx.x;
  float M = -FLT_MAX, L = 0.0f, O = 0.0f;
  if (d < 128) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) M = fmaxf(M, sm->m[w]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float wgt = ex2_approx(sm->m[w] - M);
      L = fmaf(sm->l[w], wgt, L);
      O = fmaf(sm->o[w][d], wgt, O);
    }
  }
  if (SPLIT) {
    const size_t slot = (size_t)h * p.n_chunks + chunk_idx;
    if (d == 0) { p.pm[slot] = M; p.pl[slot] = L; }
    if (d < p.D) p.po[slot * p.D + d] = O;
    return;
  }
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), n = cluster.num_blocks();
  cluster.barrier_wait();  // the arrival at kernel start
  MergeSmem *first = cluster.map_shared_rank(sm, 0);
  if (d == 0) { first->cm[rank] = M; first->cl[rank] = L; }
  if (d < 128) first->co[rank][d] = O;
  cluster.sync();
  if (rank == 0 && d < p.D) {
    float Mg = -FLT_MAX, Lg = 0.0f, Og = 0.0f;
    for (unsigned r = 0; r < n; ++r) Mg = fmaxf(Mg, sm->cm[r]);
    for (unsigned r = 0; r < n; ++r) {
      const float wgt = ex2_approx(sm->cm[r] - Mg);
      Lg = fmaf(sm->cl[r], wgt, Lg);
      Og = fmaf(sm->co[r][d], wgt, Og);
    }
    p.out[(size_t)h * p.D + d] = Lg > 0.0f ? Og / Lg : 0.0f;
  }
}

// cp.async of one granule; bytes beyond `valid` (0 or GB) are zero-filled and not read
template <int GB>
__device__ __forceinline__ void cp_async(uint32_t dst, const void *src, bool valid) {
  const int n = valid ? GB : 0;
  if (GB == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One granule (GB bytes) of a thread's ring slot as pairs of floats.
template <bool BF16, int GB>
__device__ __forceinline__ void read_granule(uint32_t addr, float2 (&f)[GB / (BF16 ? 4 : 8)]) {
  uint32_t w[GB / 4];
  if constexpr (GB == 16) asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr));
  else asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "r"(addr));
#pragma unroll
  for (int i = 0; i < GB / (BF16 ? 4 : 8); ++i) {
    if constexpr (BF16) f[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
    else f[i] = make_float2(__uint_as_float(w[2 * i]), __uint_as_float(w[2 * i + 1]));
  }
}

// One CTA: tokens [chunk_idx * chunk, ...) of head h, walked in stages of kWarps * (32 / LPT) * U tokens. LPT lanes cover a
// row of K or V with SLOTS granules of GB bytes each; lane r of a group owns granules r and r + LPT.
// HBM-bound, so the design is about bytes in flight: a stage is 128 bytes of K and V per thread (64 with 8-byte granules), two
// stages in flight while one is worked on, 512 threads per SM (two CTAs of 256 or one of 512). A thread reads back only
// what it copied itself, so the ring needs no barrier. Measured on B200 against the kernel before it (registers as the
// only buffer, the block-table lookup in series with the row loads): 16 heads of 128 bf16 dims, 65537 tokens in pages of
// 16: 386 -> 85 us (6.3 TB/s); 12 heads of 64 fp32 dims, 131072 contiguous tokens: 186 -> 115 us (7.0 TB/s).
template <bool BF16, int GB, int LPT, int SLOTS, int kThreads, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 512 / kThreads) k_attn_decode_ring(const DecParams p) {
  ptx::pdl_wait();
  constexpr int kWarps = kThreads / 32;
  constexpr int G = 32 / LPT, VE = GB / (BF16 ? 2 : 4), U = SLOTS == 1 ? 4 : 2, STAGES = 3;
  constexpr int kRound = kWarps * G;                  // tokens between a group's consecutive tokens
  constexpr int kGran = U * 2 * SLOTS;                // granules of one thread and stage
  constexpr uint32_t kStageBytes = kThreads * kGran * GB;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ MergeSmem sm;
  if (!SPLIT) cg::this_cluster().barrier_arrive();
  const uint32_t h = blockIdx.y, chunk_idx = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / LPT, r = lane % LPT;
  const uint32_t D = p.D;
  const unsigned long long row_bytes = (unsigned long long)p.H * D * (BF16 ? 2 : 4);
  const uint32_t t_begin = chunk_idx * p.chunk, t_end = min(p.T, t_begin + p.chunk);
  const uint32_t t_mine = t_begin + warp * G + g;     // this group's first token
  const int n_stages = t_begin < t_end ? (int)((t_end - t_begin + kRound * U - 1) / (kRound * U)) : 0;
  const uint32_t slot0 = static_cast<uint32_t>(__cvta_generic_to_shared(ring)) + threadIdx.x * GB;
  const uint8_t *kb = static_cast<const uint8_t *>(p.k) + (size_t)h * D * (BF16 ? 2 : 4) + r * GB;
  const uint8_t *vb = static_cast<const uint8_t *>(p.v) + (size_t)h * D * (BF16 ? 2 : 4) + r * GB;
  bool has_gran[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) has_gran[s] = (uint32_t)(s * LPT + r) * VE < D;

  // Lane r of a group resolves the byte offset of the cache row of the group's token r % U of a stage; ~0: past the end.
  auto resolve = [&](int stage) -> unsigned long long {
    const uint32_t t = t_mine + (uint32_t)(stage * U + (r & (U - 1))) * kRound;
    if (stage >= n_stages || t >= t_end) return ~0ull;
    if (p.block_table == nullptr) return (unsigned long long)t * row_bytes;
    const uint32_t lp = t / p.page_size;
    return ((unsigned long long)__ldg(p.block_table + lp) * p.page_size + (t - lp * p.page_size)) * row_bytes;
  };
  auto issue = [&](int stage, unsigned long long rows) {
    const uint32_t dst = slot0 + (uint32_t)(stage % STAGES) * kStageBytes;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned long long off = __shfl_sync(0xffffffffu, rows, g * LPT + u);
      const bool has = off != ~0ull;
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        const bool in = has && has_gran[s];
        cp_async<GB>(dst + ((u * 2 + 0) * SLOTS + s) * kThreads * GB, in ? kb + off + s * LPT * GB : p.k, in);
        cp_async<GB>(dst + ((u * 2 + 1) * SLOTS + s) * kThreads * GB, in ? vb + off + s * LPT * GB : p.v, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  unsigned long long rows = resolve(0);
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) {
    issue(i, rows);
    rows = resolve(i + 1);
  }
  float2 qv[SLOTS][VE / 2], acc[SLOTS][VE / 2];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s)
#pragma unroll
    for (int x = 0; x < VE; ++x) {
      const uint32_t d = (uint32_t)(s * LPT + r) * VE + x;
      const float qd = d < D ? __ldg(p.q + (size_t)h * D + d) * p.scale_log2 : 0.0f;
      if (x & 1) qv[s][x / 2].y = qd;
      else qv[s][x / 2].x = qd;
      acc[s][x / 2] = make_float2(0.0f, 0.0f);
    }
  // The U scores of a stage are summed over the group's lanes by halving: after log2(U) exchange steps lane r holds the
  // partial sum of token my_u only, so the remaining steps, the mask and the exponential are done once per token, and l
  // collects only this lane's tokens.
  constexpr int kSplit = U == 4 ? 2 : 1;
  const int my_u = U == 4 ? ((r & (LPT / 2)) ? 2 : 0) + ((r & (LPT / 4)) ? 1 : 0) : ((r & (LPT / 2)) ? 1 : 0);
  float m = -FLT_MAX, l = 0.0f;
  for (int i = 0; i < n_stages; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    issue(i + STAGES - 1, rows);
    rows = resolve(i + STAGES);
    const uint32_t src = slot0 + (uint32_t)(i % STAGES) * kStageBytes;
    float sc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float2 dot = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        float2 f[VE / 2];
        read_granule<BF16, GB>(src + ((u * 2 + 0) * SLOTS + s) * kThreads * GB, f);
#pragma unroll
        for (int x = 0; x < VE / 2; ++x) dot = fma2(qv[s][x], f[x], dot);
      }
      sc[u] = dot.x + dot.y;
    }
    if constexpr (U == 4) {
      const bool hi = r & (LPT / 2);
      const float g0 = __shfl_xor_sync(0xffffffffu, hi ? sc[0] : sc[2], LPT / 2), g1 = __shfl_xor_sync(0xffffffffu, hi ? sc[1] : sc[3], LPT / 2);
      sc[0] = (hi ? sc[2] : sc[0]) + g0;
      sc[1] = (hi ? sc[3] : sc[1]) + g1;
    }
    {
      const bool hi = r & (U == 4 ? LPT / 4 : LPT / 2);
      const float g0 = __shfl_xor_sync(0xffffffffu, hi ? sc[0] : sc[1], U == 4 ? LPT / 4 : LPT / 2);
      sc[0] = (hi ? sc[1] : sc[0]) + g0;
    }
#pragma unroll
    for (int o = LPT >> (kSplit + 1); o >= 1; o >>= 1) sc[0] += __shfl_xor_sync(0xffffffffu, sc[0], o);
    if (t_mine + (uint32_t)(i * U + my_u) * kRound >= t_end) sc[0] = -INFINITY;
    float top = sc[0];
#pragma unroll
    for (int o = LPT / 2; o >= (LPT >> kSplit); o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (__any_sync(0xffffffffu, top > m)) {
      const float m_new = fmaxf(m, top), alpha = ex2_approx(m - m_new);
      m = m_new;
      l *= alpha;
#pragma unroll
      for (int s = 0; s < SLOTS; ++s)
#pragma unroll
        for (int x = 0; x < VE / 2; ++x) acc[s][x] = make_float2(acc[s][x].x * alpha, acc[s][x].y * alpha);
    }
    const float my_p = ex2_approx(sc[0] - m);
    l += my_p;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float pe = __shfl_sync(0xffffffffu, my_p, g * LPT + u * (LPT / U));
#pragma unroll
      for (int s = 0; s < SLOTS; ++s) {
        float2 f[VE / 2];
        read_granule<BF16, GB>(src + ((u * 2 + 1) * SLOTS + s) * kThreads * GB, f);
#pragma unroll
        for (int x = 0; x < VE / 2; ++x) acc[s][x] = fma2(make_float2(pe, pe), f[x], acc[s][x]);
      }
    }
  }
#pragma unroll
  for (int o = LPT / 2; o >= (LPT >> kSplit); o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  // the groups of a warp, then one state per warp to shared memory
#pragma unroll
  for (int o = LPT; o < 32; o <<= 1) {
    const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
    const float mn = fmaxf(m, mo), wa = ex2_approx(m - mn), wb = ex2_approx(mo - mn);
    l = l * wa + lo * wb;
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
#pragma unroll
      for (int x = 0; x < VE / 2; ++x) {
        acc[s][x].x = acc[s][x].x * wa + __shfl_xor_sync(0xffffffffu, acc[s][x].x, o) * wb;
        acc[s][x].y = acc[s][x].y * wa + __shfl_xor_sync(0xffffffffu, acc[s][x].y, o) * wb;
      }
    m = mn;
  }
  if (lane == 0) { sm.m[warp] = m; sm.l[warp] = l; }
  if (lane < LPT) {
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
#pragma unroll
      for (int x = 0; x < VE; ++x) {
        const uint32_t d = (uint32_t)(s * LPT + r) * VE + x;
        if (d < 128) sm.o[warp][d] = (x & 1) ? acc[s][x / 2].y : acc[s][x / 2].x;
      }
  }
  merge_and_write<SPLIT, kThreads / 32>(p, &sm, h, chunk_idx);
}

template <bool BF16>
__device__ __forceinline__ float load1(const void *base, size_t e) {
  if (BF16) return __uint_as_float((uint32_t)__ldg(static_cast<const uint16_t *>(base) + e) << 16);
  return __ldg(static_cast<const float *>(base) + e);
}

// Any d_head <= 128 and alignment: a half-warp per token, lane i owns dims i, i + 16, ..., two tokens a round.
template <bool BF16, bool SPLIT>
__global__ void __launch_bounds__(256) k_attn_decode_any(const DecParams p) {
  ptx::pdl_wait();
  constexpr int kThreads = 256, kSlots = 8, TOK = 2, kHalfWarps = kThreads / 16;
  __shared__ MergeSmem sm;
  if (!SPLIT) cg::this_cluster().barrier_arrive();
  const uint32_t h = blockIdx.y, chunk_idx = blockIdx.x;
  const int hw = threadIdx.x >> 4, l16 = threadIdx.x & 15, warp = threadIdx.x >> 5;
  // The two half-warps of a warp walk different tokens and may leave the loop at different times:
  // every shuffle names only the 16 lanes of its own half-warp.
  const unsigned hmask = 0xFFFFu << (threadIdx.x & 16);
  const uint32_t D = p.D;
  const size_t dm = (size_t)p.H * D;
  const uint32_t t_begin = chunk_idx * p.chunk;
  const uint32_t t_end = min(p.T, t_begin + p.chunk);
  float qv[kSlots], acc[kSlots];
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    const uint32_t d = (uint32_t)(s * 16 + l16);
    qv[s] = d < D ? __ldg(p.q + (size_t)h * D + d) : 0.0f;
    acc[s] = 0.0f;
  }
  float m = -FLT_MAX, l = 0.0f;
  auto row_of = [&](uint32_t t) -> size_t {
    if (p.block_table == nullptr) return (size_t)t;
    return (size_t)__ldg(p.block_table + t / p.page_size) * p.page_size + (t % p.page_size);
  };
  for (uint32_t t = t_begin + hw; t < t_end; t += TOK * kHalfWarps) {
    bool has[TOK];
    size_t e[TOK];
#pragma unroll
    for (int u = 0; u < TOK; ++u) {
      const uint32_t tu = t + u * kHalfWarps;
      has[u] = tu < t_end;
      e[u] = row_of(has[u] ? tu : t) * dm + (size_t)h * D;  // a missing token re-reads the first one (unused)
    }
    float kk[TOK][kSlots], vv[TOK][kSlots];
#pragma unroll
    for (int u = 0; u < TOK; ++u) {
#pragma unroll
      for (int s = 0; s < kSlots; ++s) {
        const uint32_t d = (uint32_t)(s * 16 + l16);
        kk[u][s] = d < D ? load1<BF16>(p.k, e[u] + d) : 0.0f;
        vv[u][s] = d < D ? load1<BF16>(p.v, e[u] + d) : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < TOK; ++u) {
      if (!has[u]) break;
      float dot = 0.0f;
#pragma unroll
      for (int i = 0; i < kSlots; ++i) dot = fmaf(qv[i], kk[u][i], dot);
#pragma unroll
      for (int o = 8; o >= 1; o >>= 1) dot += __shfl_xor_sync(hmask, dot, o);
      const float s2 = dot * p.scale_log2;
      const float m_new = fmaxf(m, s2);
      const float alpha = ex2_approx(m - m_new);  // m = -FLT_MAX on the first token: 0
      const float pe = ex2_approx(s2 - m_new);
      l = fmaf(l, alpha, pe);
#pragma unroll
      for (int i = 0; i < kSlots; ++i) acc[i] = fmaf(pe, vv[u][i], acc[i] * alpha);
      m = m_new;
    }
  }
  __syncwarp();
  {  // the two half-warps of a warp
    const float mo = __shfl_xor_sync(0xffffffffu, m, 16), lo = __shfl_xor_sync(0xffffffffu, l, 16);
    const float mn = fmaxf(m, mo), wa = ex2_approx(m - mn), wb = ex2_approx(mo - mn);
    l = l * wa + lo * wb;
#pragma unroll
    for (int i = 0; i < kSlots; ++i) acc[i] = acc[i] * wa + __shfl_xor_sync(0xffffffffu, acc[i], 16) * wb;
    m = mn;
  }
  if ((threadIdx.x & 31) == 0) { sm.m[warp] = m; sm.l[warp] = l; }
  if ((threadIdx.x & 31) < 16) {
#pragma unroll
    for (int s = 0; s < kSlots; ++s) sm.o[warp][s * 16 + l16] = acc[s];
  }
  merge_and_write<SPLIT, kThreads / 32>(p, &sm, h, chunk_idx);
}

// Merges the partial states of one head: grid = n_heads, 128 threads. The chunk maxima and sums
// are staged in shared memory with coalesced loads, then thread d accumulates output dim d over the
// chunks with independent, unrolled loads (a plain loop of dependent loads cost 11 us for 25 chunks).
constexpr int kMaxChunks = 1024;
__global__ void __launch_bounds__(128) k_attn_decode_reduce(const float *__restrict__ pm, const float *__restrict__ pl,
                                                            const float *__restrict__ po, float *__restrict__ out,
                                                            uint32_t n_chunks, uint32_t D) {
  __shared__ float s_w[kMaxChunks];
  __shared__ float s_red[4];
  const uint32_t h = blockIdx.x, d = threadIdx.x;
  ptx::pdl_wait();
  float mx = -INFINITY;
  for (uint32_t c = d; c < n_chunks; c += 128) {
    const float mc = pm[(size_t)h * n_chunks + c];
    s_w[c] = mc;
    mx = fmaxf(mx, mc);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((d & 31) == 0) s_red[d >> 5] = mx;
  __syncthreads();
  const float M = fmaxf(fmaxf(s_red[0], s_red[1]), fmaxf(s_red[2], s_red[3]));
  __syncthreads();
  float lsum = 0.0f;
  for (uint32_t c = d; c < n_chunks; c += 128) {
    const float w = M > -INFINITY ? ex2_approx(s_w[c] - M) : 0.0f;
    s_w[c] = w;
    lsum = fmaf(pl[(size_t)h * n_chunks + c], w, lsum);
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if ((d & 31) == 0) s_red[d >> 5] = lsum;
  __syncthreads();
  const float L = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
  if (d >= D) return;
  float O = 0.0f;
  const float *po_h = po + (size_t)h * n_chunks * D + d;
#pragma unroll 8
  for (uint32_t c = 0; c < n_chunks; ++c) O = fmaf(po_h[(size_t)c * D], s_w[c], O);
  out[(size_t)h * D + d] = L > 0.0f ? O / L : 0.0f;
}

int launch_reduce(const DecParams &p, cudaStream_t s) {
  const int st = check_cuda(launch_kernel(k_attn_decode_reduce, dim3(p.H), dim3(128), 0, s, p.pm, p.pl, p.po, p.out, p.n_chunks, p.D));
  note_launch();
  return st;
}

// What the host needs to know of one kernel pair on one device, asked once: the number of SMs and, for every cluster size
// c, how many clusters of c CTAs the device keeps resident at the same time (its GPCs hold 16 to 20 SMs, so sizes above
// eight leave some of them over).
struct DeviceInfo {
  std::once_flag once;
  bool ok = false;
  int n_sm = 0;
  int resident[kMaxCluster + 1] = {0};
  // the largest cluster of at most `most` CTAs for which all `heads` clusters run at the same time
  uint32_t fit(uint32_t heads, uint32_t most) const {
    uint32_t c = most;
    while (c > 1 && (uint32_t)resident[c] < heads) --c;
    return c;
  }
};

using DecKernel = void (*)(const DecParams);

// One kernel in its two forms; `split` may be null when the caller never splits it.
struct DecForm {
  DecKernel split, cluster;
  int threads;
  size_t smem;
  DeviceInfo *table;  // [64]
};

const DeviceInfo *device_info(const DecForm &f) {
  int dev = 0;
  if (check_cuda(cudaGetDevice(&dev)) != DF_OK || dev < 0 || dev >= 64) return nullptr;
  DeviceInfo &di = f.table[dev];
  std::call_once(di.once, [&]() {
    bool ok = cudaDeviceGetAttribute(&di.n_sm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
    for (DecKernel k : {f.split, f.cluster})
      ok = ok && (!k || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.smem) == cudaSuccess);
    ok = ok && cudaFuncSetAttribute(f.cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    for (int c = 1; ok && c <= kMaxCluster; ++c) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = c;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(c, 64);
      cfg.blockDim = dim3(f.threads);
      cfg.dynamicSmemBytes = f.smem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      ok = cudaOccupancyMaxActiveClusters(&di.resident[c], f.cluster, &cfg) == cudaSuccess;
    }
    di.ok = ok;
  });
  if (!di.ok) note_status(DF_ERR_CUDA);
  return di.ok ? &di : nullptr;
}

int launch_cluster(const DecForm &f, DecParams &p, uint32_t cluster, cudaStream_t s) {
  p.chunk = (p.T + cluster - 1) / cluster;
  p.n_chunks = cluster;
  const int st = check_cuda(launch_clusters(f.cluster, cluster, dim3(cluster, p.H), dim3(f.threads), f.smem, s, p));
  note_launch();
  return st;
}

// Chooses the form for `narrow` (256 threads, two CTAs per SM) and, where the kernel has one, `wide` (512 threads, one CTA
// per SM, the same ring per thread). `round` = tokens that a narrow CTA works on at a time. Measured on B200, one fp32 or
// bf16 cache, device time per call:
//  * up to 64 rounds per head (4096 tokens of 64 fp32 dims): a cluster that gives every CTA about a round, at most 8
//    (T = 300: 3.4 us with 8, 4.5 with 16; T = 4096: 8.1 with either);
//  * beyond that the chip has to be filled: the largest cluster for which all heads are resident at once (16 heads of 128
//    bf16 dims over 65537 tokens: 85 us with 13, 118 with 16, whose 16 clusters need a second wave);
//  * few heads leave SMs empty either way, and then bytes in flight per CTA decide: the wide CTA when twice its cluster
//    exceeds the narrow one (8 heads: 52 us with wide 10, 58 with narrow 16; 12 heads: equal; 16 heads: narrow);
//  * with scratch and clusters on less than 3/5 of the SMs, the split form, two CTAs per SM (8 heads: 46 us; 1 head of 64
//    fp32 dims over 200000 tokens: 28 us against 57).
int launch_form(const DecForm &narrow, const DecForm *wide, DecParams &p, uint32_t max_chunks, uint32_t round, cudaStream_t s) {
  const DeviceInfo *di = device_info(narrow);
  if (!di) return DF_ERR_CUDA;
  if (p.T <= 64 * round) {
    uint32_t cluster = 1;
    while (cluster < 8 && cluster * round < p.T) cluster *= 2;
    return launch_cluster(narrow, p, di->fit(p.H, cluster), s);
  }
  const DecForm *form = &narrow;
  uint32_t cluster = di->fit(p.H, kMaxCluster), filled = cluster;
  if (wide) {
    const DeviceInfo *dw = device_info(*wide);
    if (!dw) return DF_ERR_CUDA;
    const uint32_t c = dw->fit(p.H, kMaxCluster);
    if ((uint32_t)dw->resident[c] >= p.H && 2 * c > cluster) {
      form = wide;
      cluster = filled = c;
    }
  }
  if (max_chunks > cluster && (uint64_t)filled * p.H * 5 < (uint64_t)di->n_sm * 3) {
    uint32_t want = (2 * (uint32_t)di->n_sm + p.H - 1) / p.H;
    if (want > max_chunks) want = max_chunks;
    if (want > (uint32_t)kMaxChunks) want = kMaxChunks;
    p.chunk = (p.T + want - 1) / want;
    p.n_chunks = (p.T + p.chunk - 1) / p.chunk;
    launch_kernel(narrow.split, dim3(p.n_chunks, p.H), dim3(narrow.threads), narrow.smem, s, p);
    note_launch();
    if (check_cuda(cudaGetLastError()) != DF_OK) return DF_ERR_CUDA;
    return launch_reduce(p, s);
  }
  return launch_cluster(*form, p, cluster, s);
}

template <bool BF16, int GB, int LPT, int SLOTS>
int launch_ring(DecParams &p, uint32_t max_chunks, cudaStream_t s) {
  static DeviceInfo narrow_info[64], wide_info[64];
  constexpr int U = SLOTS == 1 ? 4 : 2;
  constexpr size_t kThreadBytes = (size_t)3 * U * 2 * SLOTS * GB;
  const DecForm narrow = {k_attn_decode_ring<BF16, GB, LPT, SLOTS, 256, true>, k_attn_decode_ring<BF16, GB, LPT, SLOTS, 256, false>, 256,
                          256 * kThreadBytes, narrow_info};
  const DecForm wide = {nullptr, k_attn_decode_ring<BF16, GB, LPT, SLOTS, 512, false>, 512, 512 * kThreadBytes, wide_info};
  return launch_form(narrow, &wide, p, max_chunks, 8 * (32 / LPT) * U, s);
}
template <bool BF16>
int launch_any(DecParams &p, uint32_t max_chunks, cudaStream_t s) {
  static DeviceInfo info[64];
  const DecForm narrow = {k_attn_decode_any<BF16, true>, k_attn_decode_any<BF16, false>, 256, 0, info};
  return launch_form(narrow, nullptr, p, max_chunks, 64, s);
}

}  // namespace

// Decode dispatch. partial_* may be null (scratch-free cluster form); otherwise they hold at least
// n_heads * max_chunks states, and the split form is used when it pays.
int decode_dispatch(const float *q, const void *k, const void *v, const int32_t *block_table, float *out,
                    float *partial_m, float *partial_l, float *partial_o, uint32_t max_chunks, uint32_t H,
                    uint32_t T, uint32_t D, float scale, uint32_t page_size, bool kv_bf16, cudaStream_t s) {
  DecParams p;
  p.q = q; p.k = k; p.v = v; p.block_table = block_table; p.out = out;
  p.pm = partial_m; p.pl = partial_l; p.po = partial_o;
  p.H = H; p.T = T; p.D = D; p.page_size = page_size ? page_size : 1;
  p.scale_log2 = scale * kLog2e;
  if (!(partial_m && partial_l && partial_o)) max_chunks = 0;
  // The widest granule that divides a head's row slice and every base address; lanes so that a row takes one or two slots.
  const uintptr_t bits = reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | (uintptr_t)(D * (kv_bf16 ? 2 : 4));
  if (kv_bf16) {
    if (bits % 16 == 0) return D <= 64 ? launch_ring<true, 16, 8, 1>(p, max_chunks, s) : launch_ring<true, 16, 16, 1>(p, max_chunks, s);
    if (bits % 8 == 0) return D <= 64 ? launch_ring<true, 8, 16, 1>(p, max_chunks, s) : launch_ring<true, 8, 16, 2>(p, max_chunks, s);
    return launch_any<true>(p, max_chunks, s);
  }
  if (bits % 16 == 0) return D <= 64 ? launch_ring<false, 16, 16, 1>(p, max_chunks, s) : launch_ring<false, 16, 16, 2>(p, max_chunks, s);
  return launch_any<false>(p, max_chunks, s);
}

}  // namespace df

// attn_generic.cu — the HBM-bound helper passes of the attention library: the delta pre-pass, the merge of partial
// results and the accumulation of per-block gradients.
#include <math.h>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {

namespace {

// ---------------------------------------------------------------------------------------
// delta pre-pass, HBM-bound: delta[b][h][i] = sum_d dO[b][i][h][d] * O[b][i][h][d].
// A block streams 32 consecutive rows (a contiguous 32*H*D chunk of both tensors) with 16-byte
// loads, LPS = D/4 lanes cooperate on one (row, head) segment, the 32*H sums are transposed
// through shared memory so the [B][H][S] output is written in full 128-byte lines.
// Algorithmic bytes: 2*B*S*H*D*4 read + B*H*S*4 written.
// ---------------------------------------------------------------------------------------
template <int LPS>
__global__ void __launch_bounds__(256) k_delta_vec(const float4 *__restrict__ o,
                                                   const float4 *__restrict__ g,
                                                   float *__restrict__ delta, uint32_t H,
                                                   uint32_t S, uint32_t tiles_per_batch, uint32_t R) {
  ptx::pdl_wait();
  extern __shared__ float s_sum[];  // [H][R], R = rows per block (32, or 8 when the grid would be too small)
  const uint32_t b = blockIdx.x / tiles_per_batch;
  const uint32_t i0 = (blockIdx.x % tiles_per_batch) * R;
  const uint32_t rows = (S - i0) < R ? (S - i0) : R;
  const uint32_t nseg = rows * H;  // segments in this chunk, index = ii*H + h
  const size_t chunk = ((size_t)b * S + i0) * H * LPS;  // in float4 units
  const uint32_t grp = threadIdx.x / LPS, lane = threadIdx.x % LPS;
  constexpr uint32_t kGroups = 256 / LPS;
  for (uint32_t sg0 = 0; sg0 < nseg; sg0 += kGroups * 4) {
    float acc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t sg = sg0 + u * kGroups + grp;
      acc[u] = 0.0f;
      if (sg < nseg) {
        const float4 a = __ldg(o + chunk + (size_t)sg * LPS + lane);
        const float4 c = __ldg(g + chunk + (size_t)sg * LPS + lane);
        acc[u] = a.x * c.x + a.y * c.y + a.z * c.z + a.w * c.w;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int off = LPS / 2; off > 0; off >>= 1) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], off);
      const uint32_t sg = sg0 + u * kGroups + grp;
      if (lane == 0 && sg < nseg) s_sum[(sg % H) * R + sg / H] = acc[u];
    }
  }
  __syncthreads();
  for (uint32_t idx = threadIdx.x; idx < R * H; idx += 256u) {
    const uint32_t h = idx / R, ii = idx % R;
    if (ii < rows) delta[((size_t)b * H + h) * S + i0 + ii] = s_sum[idx];
  }
}

// Any D / alignment: eight lanes per (b, i, h) segment, consecutive segments side by side in memory, 16-byte loads where
// VEC (D % 4 == 0 and aligned). One thread per segment, as before, read 32 distant lines per load: B=2, S=600, H=6, D=96
// 27.4 -> 3 us.
template <bool VEC>
__global__ void __launch_bounds__(256) k_delta_any(const float *__restrict__ o, const float *__restrict__ g, float *__restrict__ delta,
                                                   uint32_t B, uint32_t H, uint32_t S, uint32_t D) {
  ptx::pdl_wait();
  const size_t n = (size_t)B * H * S;
  const uint32_t lane = threadIdx.x & 7u;
  for (size_t u0 = blockIdx.x * (size_t)32; u0 < n; u0 += (size_t)gridDim.x * 32) {
    const size_t u = u0 + threadIdx.x / 8;
    float s = 0.0f;
    if (u < n) {
      if (VEC) {
        const float4 *o4 = reinterpret_cast<const float4 *>(o + u * D), *g4 = reinterpret_cast<const float4 *>(g + u * D);
        for (uint32_t d = lane; d < D / 4; d += 8) {
          const float4 a = __ldg(o4 + d), c = __ldg(g4 + d);
          s += (a.x * c.x + a.y * c.y) + (a.z * c.z + a.w * c.w);
        }
      } else {
        for (uint32_t d = lane; d < D; d += 8) s = fmaf(__ldg(o + u * D + d), __ldg(g + u * D + d), s);
      }
    }
#pragma unroll
    for (int x = 4; x >= 1; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
    if (u < n && lane == 0) delta[((u / H / S) * H + u % H) * S + (u / H) % S] = s;
  }
}

// Partial-result merge (ring step): one thread per (b, i, h, d); weights recomputed per element.
__global__ void k_merge_partials(float *__restrict__ o_a, float *__restrict__ lse_a,
                                 const float *__restrict__ o_b, const float *__restrict__ lse_b,
                                 uint32_t B, uint32_t H, uint32_t S, uint32_t D) {
  ptx::pdl_wait();
  const size_t n = (size_t)B * S * H * D;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t d = e % D, h = (e / D) % H, i = (e / ((size_t)D * H)) % S,
                 b = e / ((size_t)D * H * S);
    const size_t si = (b * H + h) * S + i;
    const float la = lse_a[si], lb = __ldg(lse_b + si);
    const float mx = fmaxf(la, lb);
    float res = 0.0f;
    if (mx != -INFINITY) {
      const float wa = expf(la - mx), wb = expf(lb - mx);
      res = (wa * o_a[e] + wb * __ldg(o_b + e)) / (wa + wb);
    }
    o_a[e] = res;
  }
}

// Second pass of the merge: the statistics themselves (kept separate so that every element
// thread of the first pass reads the un-merged lse_a).
__global__ void k_merge_lse(float *__restrict__ lse_a, const float *__restrict__ lse_b, size_t n) {
  ptx::pdl_wait();
  for (size_t u = blockIdx.x * (size_t)blockDim.x + threadIdx.x; u < n;
       u += (size_t)gridDim.x * blockDim.x) {
    const float la = lse_a[u], lb = __ldg(lse_b + u);
    const float mx = fmaxf(la, lb);
    if (mx != -INFINITY) lse_a[u] = mx + logf(expf(la - mx) + expf(lb - mx));
  }
}

__global__ void k_accumulate(float *__restrict__ dst, const float *__restrict__ src, size_t n) {
  ptx::pdl_wait();
  for (size_t u = blockIdx.x * (size_t)blockDim.x + threadIdx.x; u < n;
       u += (size_t)gridDim.x * blockDim.x)
    dst[u] += __ldg(src + u);
}

inline int grid_1d(size_t n, int threads) {
  size_t blocks = (n + threads - 1) / threads;
  const size_t cap = 148 * 16;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace

int delta_prepass(const AttnParams &p, cudaStream_t s) {
  if (p.Sq == 0 || p.B == 0 || p.H == 0) return DF_OK;
  const uint32_t D = p.D, H = p.H, S = p.Sq;
  const bool pow2 = (D & (D - 1)) == 0 && D >= 4;
  const bool aligned = ((reinterpret_cast<uintptr_t>(p.o_in) | reinterpret_cast<uintptr_t>(p.d_out)) & 15u) == 0;
  if (pow2 && aligned && H <= 256) {
    // 32 rows per block stream best on large inputs; small inputs get 8 rows so that the grid covers the GPU
    const uint32_t R = ((uint64_t)p.B * ((S + 31) / 32) < 148u * 8u) ? 8u : 32u;
    const uint32_t tiles = (S + R - 1) / R;
    const dim3 grid(p.B * tiles);
    const size_t smem = (size_t)H * R * sizeof(float);
    const float4 *o4 = reinterpret_cast<const float4 *>(p.o_in);
    const float4 *g4 = reinterpret_cast<const float4 *>(p.d_out);
    switch (D / 4) {
      case 1: launch_kernel(k_delta_vec<1>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
      case 2: launch_kernel(k_delta_vec<2>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
      case 4: launch_kernel(k_delta_vec<4>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
      case 8: launch_kernel(k_delta_vec<8>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
      case 16: launch_kernel(k_delta_vec<16>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
      default: launch_kernel(k_delta_vec<32>, grid, dim3(256), smem, s, o4, g4, p.delta, H, S, tiles, R); break;
    }
  } else {
    const size_t n = (size_t)p.B * H * S;
    if (D % 4 == 0 && aligned) launch_kernel(k_delta_any<true>, dim3(grid_1d(n * 8, 256)), dim3(256), 0, s, p.o_in, p.d_out, p.delta, p.B, H, S, D);
    else launch_kernel(k_delta_any<false>, dim3(grid_1d(n * 8, 256)), dim3(256), 0, s, p.o_in, p.d_out, p.delta, p.B, H, S, D);
  }
  note_launch();
  return check_cuda(cudaGetLastError());
}

int merge_partials(float *o_a, float *lse_a, const float *o_b, const float *lse_b, uint32_t B,
                   uint32_t H, uint32_t S, uint32_t D, cudaStream_t s) {
  const size_t n = (size_t)B * S * H * D;
  if (n == 0) return DF_OK;
  launch_kernel(k_merge_partials, dim3(grid_1d(n, 256)), dim3(256), 0, s, o_a, lse_a, o_b, lse_b, B, H, S, D);
  launch_kernel(k_merge_lse, dim3(grid_1d((size_t)B * H * S, 256)), dim3(256), 0, s, lse_a, lse_b, (size_t)B * H * S);
  note_launch(2);
  return check_cuda(cudaGetLastError());
}

int accumulate(float *dst, const float *src, uint64_t n, cudaStream_t s) {
  if (n == 0) return DF_OK;
  launch_kernel(k_accumulate, dim3(grid_1d(n, 256)), dim3(256), 0, s, dst, src, (size_t)n);
  note_launch();
  return check_cuda(cudaGetLastError());
}

}  // namespace df

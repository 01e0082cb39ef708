// linear_rows.cu - the projections of linear_sm100.cu for a handful of rows (generating text: one row per sequence):
//   out_j[M, N] = X[M, K] W_j[N, K]^T + b_j[N]  (+ residual[M, N], or GELU in the epilogue),  M <= 8.
//
// With so few rows the work is reading W once (2.4 MB for a 768 x 768 matrix): bytes and latency, not products. The tensor
// kernel's 128 x 256 tiles give such a matrix to three CTAs, which then read it at a fiftieth of the chip's rate. Here
// every warp takes one output feature, or a slice of one: it requests its whole slice of the row of W at once, multiplies in
// full fp32 and adds up over its lanes, and the warps that share a feature meet in shared memory. Slices are at most 1024
// elements (eight 16-byte loads per lane in flight) and as short as it takes to have eight warps per SM, down to 256.
// Measured on B200, 1 row: 768 -> 768 15.6 -> 2.6 us, 768 -> 3 x 768 15.9 -> 3.0, 768 -> 3072 16.1 -> 3.2, 3072 -> 768 40 -> 3.2.
#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace df {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kBatch = 8;  // 16-byte loads of W that a lane has in flight

struct RowsParams {
  const float *x, *w[3], *bias[3], *residual;
  float *out[3], *gelu_out;
  uint32_t M, N, K, features;  // features = N * matrices
  int store_pre;               // with gelu_out: also write the pre-activation
};

// MR: rows held per warp (M rounded up to a power of two); KS: warps per output feature.
template <int MR, int KS>
__global__ void __launch_bounds__(kThreads) k_linear_rows(const RowsParams p) {
  ptx::pdl_wait();
  __shared__ float part[kWarps][MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t f = blockIdx.x * (kWarps / KS) + warp / KS;
  const bool has = f < p.features;
  const uint32_t mat = has ? f / p.N : 0, n = has ? f - mat * p.N : 0;
  const uint32_t nv = p.K >> 2, slice = (nv + KS - 1) / KS, v0 = (warp % KS) * slice, v1 = min(nv, v0 + slice);
  const float *w_mat = mat == 0 ? p.w[0] : (mat == 1 ? p.w[1] : p.w[2]), *bias = mat == 0 ? p.bias[0] : (mat == 1 ? p.bias[1] : p.bias[2]);
  float *out = mat == 0 ? p.out[0] : (mat == 1 ? p.out[1] : p.out[2]);
  const float4 *w4 = reinterpret_cast<const float4 *>(w_mat + (size_t)n * p.K);
  const float4 *x4 = reinterpret_cast<const float4 *>(p.x);
  float acc[MR];
#pragma unroll
  for (int m = 0; m < MR; ++m) acc[m] = 0.0f;
  if (has) {
    for (uint32_t v = v0 + lane; v < v1; v += 32 * kBatch) {
      float4 w[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) w[i] = v + 32 * i < v1 ? __ldg(w4 + v + 32 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        if (v + 32 * i < v1) {
#pragma unroll
          for (int m = 0; m < MR; ++m) {
            if ((uint32_t)m < p.M) {
              const float4 x = __ldg(x4 + (size_t)m * nv + v + 32 * i);
              acc[m] = fmaf(w[i].x, x.x, fmaf(w[i].y, x.y, fmaf(w[i].z, x.z, fmaf(w[i].w, x.w, acc[m]))));
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
  float v = acc[0];
#pragma unroll
  for (int m = 1; m < MR; ++m)
    if (lane == m) v = acc[m];
  if (KS > 1) {
    if (lane < MR) part[warp][lane] = v;
    __syncthreads();
    if (warp % KS) return;
    v = 0.0f;
    if (lane < MR) {
#pragma unroll
      for (int k = 0; k < KS; ++k) v += part[warp + k][lane];
    }
  }
  if (!has || (uint32_t)lane >= p.M || lane >= MR) return;
  if (bias) v += __ldg(bias + n);
  const size_t at = (size_t)lane * p.N + n;
  if (p.residual) v += __ldg(p.residual + at);
  if (!p.gelu_out || p.store_pre) out[at] = v;
  if (p.gelu_out) p.gelu_out[at] = gelu_value(v);
}

template <int MR>
void launch(const RowsParams &p, int ks, cudaStream_t s) {
  const unsigned grid = (p.features * (unsigned)ks + kWarps - 1) / kWarps;
  switch (ks) {
    case 1: launch_kernel(k_linear_rows<MR, 1>, grid, dim3(kThreads), 0, s, p); break;
    case 2: launch_kernel(k_linear_rows<MR, 2>, grid, dim3(kThreads), 0, s, p); break;
    case 4: launch_kernel(k_linear_rows<MR, 4>, grid, dim3(kThreads), 0, s, p); break;
    default: launch_kernel(k_linear_rows<MR, 8>, grid, dim3(kThreads), 0, s, p); break;
  }
}

}  // namespace

// Same arguments, alignment and shape rules as tensor_linear; M <= kLinearRowsMax.
int rows_linear(const float *x, const float *const *w, const float *const *bias, float *const *out, const float *residual, float *gelu_out,
                int n_mats, uint32_t M, uint32_t K, uint32_t N, int n_sm, cudaStream_t s) {
  RowsParams p;
  p.x = x;
  for (int j = 0; j < 3; ++j) {
    const int jj = j < n_mats ? j : 0;
    p.w[j] = w[jj];
    p.bias[j] = bias ? bias[jj] : nullptr;
    p.out[j] = out[jj];
  }
  p.residual = residual;
  p.gelu_out = gelu_out;
  p.store_pre = (gelu_out && out[0] != gelu_out) ? 1 : 0;
  p.M = M; p.N = N; p.K = K;
  p.features = N * (uint32_t)n_mats;
  int ks = 1;
  while (ks < 8 && (K / ks > 1024 || p.features * ks < (uint32_t)n_sm * 8) && K / (2 * ks) >= 256) ks *= 2;
  if (M == 1) launch<1>(p, ks, s);
  else if (M == 2) launch<2>(p, ks, s);
  else if (M <= 4) launch<4>(p, ks, s);
  else launch<8>(p, ks, s);
  note_launch();
  return check_cuda(cudaGetLastError());
}

}  // namespace df

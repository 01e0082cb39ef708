// loss_ce.cu — the loss head's fused softmax + cross-entropy over one chunk of logits, for B200 (sm_100a).
//
// Drop-in for two symbols of darkforest-cuda/kernels/softmax.cu, which the reference's static step calls once per
// 512-row chunk of the vocabulary logits (darkforest-core/src/engine/static_gpt2.rs:1386-1418 through
// darkforest-cuda/src/lib.rs:1897-1945 and src/kernels.rs:531-600):
//   launch_fused_chunked_logit_ce  (softmax.cu:325-410)  logits -> probabilities in place, grad_logits =
//                                  (p - onehot(target)) / total_rows, loss += sum_rows -log(max(p_target, 1e-12)) / total_rows
//   launch_chunked_ce_eval         (softmax.cu:415-480)  loss += sum_rows (log(sum) - (z_target - max)) / total_rows
// Same arithmetic (max-subtracted softmax in fp32 with __expf / __logf); what differs is the traffic. The
// reference walks each row of [chunk_rows, vocab] three times through global memory (max; exp + write; normalise +
// two writes: 3 reads, 3 writes of the 200 KB row). Here a cluster of CTAs keeps the row in its shared memory, so
// the training form reads the logits once and writes probabilities and gradients once each (1 read + 2 writes, the
// algorithmic minimum); the eval form reads once with an online (max, sum) pair and writes nothing. Rows of an odd-length vocabulary are not
// 16-byte aligned: every row is processed as a scalar head up to the next 16-byte boundary, a float4 body and a scalar
// tail. Rows too long for a cluster's shared memory are walked in global memory.
#include <cooperative_groups.h>
#include <float.h>
#include <math.h>

#include <mutex>

#include "df_common.cuh"
#include "sm100_ptx.cuh"

namespace cg = cooperative_groups;

namespace df {
namespace {

constexpr int kCeThreads = 1024;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Block-wide reductions over kCeThreads threads; `red` holds 32 floats. Every thread gets the result.
__device__ __forceinline__ float block_max(float v, float *red) {
  v = warp_max(v);
  __syncthreads();  // the previous use of `red` is over
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[threadIdx.x & 31];  // kCeThreads / 32 = 32 warps: every slot is written
  return warp_max(r);
}
__device__ __forceinline__ float block_sum(float v, float *red) {
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = red[threadIdx.x & 31];
  return warp_sum(r);
}

// [0, head) scalar, [head, head + 4 * n4) as float4, rest scalar: `head` elements bring the row to a 16-byte boundary
__device__ __forceinline__ void split_row(const float *row, uint32_t cols, uint32_t *head, uint32_t *n4) {
  const uint32_t mis = (uint32_t)((reinterpret_cast<uintptr_t>(row) >> 2) & 3u);
  uint32_t h = (4u - mis) & 3u;
  if (h > cols) h = cols;
  *head = h;
  *n4 = (cols - h) >> 2;
}

// Training form, the row resident in the shared memory of a cluster of CTAs. What bounds it is HBM (1 read and 2 writes of
// the row); a CTA that owns a whole SM and a whole row, as before, alternates between reading and writing and leaves the
// last round of rows half empty (512 rows on 148 SMs). Here a row is cut into slices of at most 53 KB, one per CTA of
// a cluster (short rows: several rows per cluster), and four CTAs share an SM, so that one row's loads run under another's
// exponentials and stores. A thread copies its own 16-byte groups in with cp.async and reads back only those: no barrier until
// the CTAs exchange one (max, sum) each. A running cluster takes over rows whose cluster has not started yet (claim_request): with
// rows dealt out in advance the slowest SMs end 25 % after the others (2048 x 50257: 250 against 200 us), and with a cluster per
// row the loss would be rounded once per row. Probabilities go in place, gradients out, with streaming stores; SAME_PHASE: the
// gradient row lies at the same 16-byte phase as the logits row. Measured on B200 against the kernel before: 512 x 50257
// 76.0 -> 56.2 us (5.5 TB/s), 2048 x 50257 268 -> 200 us (6.2 TB/s), 32 x 50257 15.3 -> 8.2 us, 512 x 5000 11.4 -> 10.0 us.
constexpr int kSliceThreads = 256;
constexpr int kMaxCeCluster = 8;
constexpr uint32_t kSliceGroups = 13;     // groups of four floats per thread: 52 KB per CTA, four CTAs per SM
constexpr uint32_t kMaxSliceGroups = 54;  // one CTA per SM

template <bool SAME_PHASE>
__global__ void __launch_bounds__(kSliceThreads, 4)
k_logit_ce_cluster(float *__restrict__ logits, const uint32_t *__restrict__ targets, float *__restrict__ grad_logits,
                   float *__restrict__ loss, uint32_t chunk_rows, uint32_t cols, uint32_t slices, uint32_t groups, uint32_t more,
                   float inv_total_rows, unsigned int *status) {
  ptx::pdl_wait();
  extern __shared__ __align__(16) float4 slice[];  // [groups][kSliceThreads]
  __shared__ float red[kSliceThreads / 32];
  __shared__ float2 part[2][kMaxCeCluster];  // (max, sum) of every CTA of the cluster, for rows in turn
  __shared__ uint32_t next_unit[2];
  __shared__ __align__(16) uint4 claim;
  __shared__ uint64_t claim_bar;
  __shared__ uint32_t give_up;
  __shared__ float cluster_loss;  // of the cluster's rows (in its first CTA)
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t n_cta = cluster.num_blocks(), rank = cluster.block_rank(), t = threadIdx.x;
  const uint32_t slot = rank / slices, part_rank = rank - slot * slices, rows_per_cluster = n_cta / slices;
  const uint32_t a_claim = ptx::smem_u32(&claim), a_bar = ptx::smem_u32(&claim_bar);
  if (t == 0) {
    ptx::mbar_init(a_bar, 1);
    ptx::mbar_init_fence();
    give_up = 0;
    cluster_loss = 0.0f;
  }
  cluster.barrier_arrive();  // waited for before the first write to another CTA's shared memory
  auto reduce = [&](float v, bool is_max) {
    v = is_max ? warp_max(v) : warp_sum(v);
    __syncthreads();  // the previous use of `red` is over
    if ((t & 31) == 0) red[t >> 5] = v;
    __syncthreads();
    float r = red[0];
#pragma unroll
    for (int w = 1; w < kSliceThreads / 32; ++w) r = is_max ? fmaxf(r, red[w]) : r + red[w];
    return r;
  };
  const bool one_row = rows_per_cluster == 1 && !more;
  uint32_t turn = 0;
  for (uint32_t unit = blockIdx.x / n_cta; unit != ~0u; unit = more ? next_unit[turn] : ~0u, turn ^= 1) {
    if (more && rank == 0 && t == 0) {  // asked now, answered long before the exchange below
      ptx::fence_proxy_async_smem();
      ptx::mbar_arrive_expect_tx(a_bar, 16);
      ptx::claim_request(a_claim, a_bar);
    }
    const bool has = unit * rows_per_cluster + slot < chunk_rows;  // else this CTA only keeps the cluster's barriers company
    const uint32_t row = has ? unit * rows_per_cluster + slot : 0;
    float *grow = logits + (size_t)row * cols;
    const uint32_t target = __ldg(targets + row);
    uint32_t head, n4;
    split_row(grow, cols, &head, &n4);
    // this CTA: float4 groups [g0, g1) of the body; the first also has the row's scalar head, the last its scalar tail
    const uint32_t per = groups * kSliceThreads, g0 = min(n4, part_rank * per), g1 = has ? min(n4, g0 + per) : g0;
    const uint32_t body = head + 4u * n4;
    uint32_t extra = cols;  // the scalar element of this thread, if any
    if (has && part_rank == 0 && t < head) extra = t;
    if (has && part_rank == slices - 1 && t >= 32 && t - 32 < cols - body) extra = body + (t - 32);
    const float x_extra = extra < cols ? grow[extra] : 0.0f;
    const float4 *src = reinterpret_cast<const float4 *>(grow + head);
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(slice + t));
    for (uint32_t i = 0; i < groups; ++i) {
      const uint32_t g = g0 + i * kSliceThreads + t;
      if (g < g1) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * kSliceThreads * 16u), "l"(src + g) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const uint32_t mine = g1 > g0 + t ? (g1 - g0 - t + kSliceThreads - 1) / kSliceThreads : 0;  // groups of this thread
    float top = extra < cols ? x_extra : -FLT_MAX;
#pragma unroll 4
    for (uint32_t i = 0; i < mine; ++i) {
      const float4 x = slice[i * kSliceThreads + t];
      top = fmaxf(top, fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w)));
    }
    const float cta_max = reduce(top, true);
    float sum = extra < cols ? __expf(x_extra - cta_max) : 0.0f;
#pragma unroll 4
    for (uint32_t i = 0; i < mine; ++i) {
      const float4 x = slice[i * kSliceThreads + t];
      sum += (__expf(x.x - cta_max) + __expf(x.y - cta_max)) + (__expf(x.z - cta_max) + __expf(x.w - cta_max));
    }
    const float cta_sum = reduce(sum, false);
    if (unit == blockIdx.x / n_cta) cluster.barrier_wait();
    if (t < slices) cluster.map_shared_rank(&part[turn][0], slot * slices + t)[part_rank] = make_float2(cta_max, cta_sum);
    if (more && rank == 0 && t == 0) {
      const bool answered = ptx::mbar_wait(a_bar, turn, &give_up);
      const uint32_t first = answered ? ptx::claim_result(a_claim) : ~0u;
      if (!answered && status) atomicOr(status, DEV_STATUS_WAIT_EXPIRED);
      for (uint32_t r = 0; r < n_cta; ++r) cluster.map_shared_rank(next_unit, r)[turn] = first == ~0u ? ~0u : first / n_cta;
    }
    cluster.sync();
    float row_max = -FLT_MAX, row_sum = 0.0f;
    for (uint32_t r = 0; r < slices; ++r) row_max = fmaxf(row_max, part[turn][r].x);
    for (uint32_t r = 0; r < slices; ++r) row_sum += part[turn][r].y * __expf(part[turn][r].x - row_max);
    const float inv_sum = 1.0f / row_sum, g_scale = inv_total_rows;
    float *ggrad = grad_logits + (size_t)row * cols;
    float p_target = -1.0f;
    if (extra < cols) {
      const float p = __expf(x_extra - row_max) * inv_sum;
      grow[extra] = p;
      ggrad[extra] = (p - (extra == target ? 1.0f : 0.0f)) * g_scale;
      if (extra == target) p_target = p;
    }
    float4 *out = reinterpret_cast<float4 *>(grow + head);
#pragma unroll 2
    for (uint32_t i = 0; i < mine; ++i) {
      const uint32_t g = g0 + i * kSliceThreads + t;
      const float4 x = slice[i * kSliceThreads + t];
      const float4 p = make_float4(__expf(x.x - row_max) * inv_sum, __expf(x.y - row_max) * inv_sum, __expf(x.z - row_max) * inv_sum,
                                   __expf(x.w - row_max) * inv_sum);
      __stcs(out + g, p);
      // the target column (if it lies in this group of four) takes the scalar formula, (p - 1) * scale
      const uint32_t k = target - (head + 4u * g);  // unsigned: 4 or more when the target is elsewhere
      const float4 d = make_float4((p.x - (k == 0u ? 1.0f : 0.0f)) * g_scale, (p.y - (k == 1u ? 1.0f : 0.0f)) * g_scale,
                                   (p.z - (k == 2u ? 1.0f : 0.0f)) * g_scale, (p.w - (k == 3u ? 1.0f : 0.0f)) * g_scale);
      if (k < 4u) p_target = k == 0u ? p.x : (k == 1u ? p.y : (k == 2u ? p.z : p.w));
      float *gd = ggrad + head + 4u * g;
      if (SAME_PHASE) {
        __stcs(reinterpret_cast<float4 *>(gd), d);
      } else {
        gd[0] = d.x; gd[1] = d.y; gd[2] = d.z; gd[3] = d.w;
      }
    }
    if (p_target >= 0.0f)
      atomicAdd(one_row ? loss : cluster.map_shared_rank(&cluster_loss, 0), -__logf(fmaxf(p_target, 1e-12f)) * inv_total_rows);
  }
  if (one_row) return;
  // one addition per cluster: every further one would round the running loss once more
  cluster.barrier_arrive();
  if (rank == 0) {
    cluster.barrier_wait();
    if (t == 0 && cluster_loss != 0.0f) atomicAdd(loss, cluster_loss);
  }
}

// Training form for rows that do not fit a cluster's shared memory: max pass, sum pass and write pass from global memory.
__global__ void __launch_bounds__(kCeThreads, 1)
k_chunked_logit_ce_global(float *__restrict__ logits, const uint32_t *__restrict__ targets, float *__restrict__ grad_logits,
                          float *__restrict__ loss, uint32_t chunk_rows, uint32_t cols, float inv_total_rows) {
  ptx::pdl_wait();
  __shared__ float red[32];
  float cta_loss = 0.0f;
  for (uint32_t row = blockIdx.x; row < chunk_rows; row += gridDim.x) {
    float *grow = logits + (size_t)row * cols;
    float *ggrad = grad_logits + (size_t)row * cols;
    const uint32_t target = __ldg(targets + row);
    float tmax = -FLT_MAX;
    for (uint32_t i = threadIdx.x; i < cols; i += kCeThreads) tmax = fmaxf(tmax, grow[i]);
    const float row_max = block_max(tmax, red);
    float tsum = 0.0f;
    for (uint32_t i = threadIdx.x; i < cols; i += kCeThreads) tsum += __expf(grow[i] - row_max);
    const float inv_sum = 1.0f / block_sum(tsum, red);
    for (uint32_t i = threadIdx.x; i < cols; i += kCeThreads) {
      const float p = __expf(grow[i] - row_max) * inv_sum;
      grow[i] = p;
      ggrad[i] = (p - (i == target ? 1.0f : 0.0f)) * inv_total_rows;
      if (i == target) cta_loss += -__logf(fmaxf(p, 1e-12f)) * inv_total_rows;
    }
  }
  cta_loss = block_sum(cta_loss, red);
  if (threadIdx.x == 0 && cta_loss != 0.0f) atomicAdd(loss, cta_loss);
}

// Eval form: one read of the row, online (max, sum) per thread, nothing written but the loss. One row per CTA, four
// CTAs per SM. (The cluster form above, with the row in shared memory, was slower: 26 against 18 us at 512 x 50257.)
constexpr int kEvalThreads = 512;
__global__ void __launch_bounds__(kEvalThreads, 4)
k_chunked_ce_eval(const float *__restrict__ logits, const uint32_t *__restrict__ targets, float *__restrict__ loss,
                  uint32_t chunk_rows, uint32_t cols, float inv_total_rows) {
  ptx::pdl_wait();
  __shared__ float red[32];
  const uint32_t row = blockIdx.x;
  if (row >= chunk_rows) return;
  const float *grow = logits + (size_t)row * cols;
  const uint32_t target = __ldg(targets + row);
  uint32_t head, n4;
  split_row(grow, cols, &head, &n4);
  const uint32_t body_end = head + 4u * n4;
  const int n_warps = kEvalThreads / 32;
  auto reduce = [&](float v, bool is_max) {
    v = is_max ? warp_max(v) : warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = (int)(threadIdx.x & 31) < n_warps ? red[threadIdx.x & 31] : (is_max ? -FLT_MAX : 0.0f);
    return is_max ? warp_max(r) : warp_sum(r);
  };
  float m = -FLT_MAX, s = 0.0f;
  auto push = [&](float x) {
    if (x > m) {
      s = s * __expf(m - x) + 1.0f;
      m = x;
    } else {
      s += __expf(x - m);
    }
  };
  if (threadIdx.x < head) push(grow[threadIdx.x]);
  const float4 *g4 = reinterpret_cast<const float4 *>(grow + head);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < n4; i += kEvalThreads) {
    const float4 x = __ldcs(g4 + i);
    const float gm = fmaxf(fmaxf(x.x, x.y), fmaxf(x.z, x.w));
    if (gm > m) {
      s *= __expf(m - gm);
      m = gm;
    }
    s += __expf(x.x - m) + __expf(x.y - m) + __expf(x.z - m) + __expf(x.w - m);
  }
  if (body_end + threadIdx.x < cols) push(grow[body_end + threadIdx.x]);
  const float row_max = reduce(m, true);
  const float sum = reduce(s * __expf(m - row_max), false);  // a thread that saw nothing has s = 0
  if (threadIdx.x == 0 && target < cols)
    atomicAdd(loss, (-(grow[target] - row_max) + __logf(fmaxf(sum, 1e-12f))) * inv_total_rows);
}

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
    const int smem = (int)(kMaxSliceGroups * kSliceThreads * 16);
    d.ok = cudaFuncSetAttribute(k_logit_ce_cluster<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
           cudaFuncSetAttribute(k_logit_ce_cluster<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
           cudaDeviceGetAttribute(&d.n_sm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && d.n_sm > 0;
  });
  if (!d.ok) {
    note_status(DF_ERR_CUDA);
    return DF_ERR_CUDA;
  }
  *n_sm = d.n_sm;
  return DF_OK;
}

}  // namespace

int chunked_logit_ce(float *logits, const uint32_t *targets, float *grad_logits, float *loss, uint32_t chunk_rows, uint32_t cols,
                     uint32_t total_rows, cudaStream_t s) {
  if (chunk_rows == 0 || cols == 0) return DF_OK;
  if (!logits || !targets || !loss || total_rows == 0) return DF_ERR_INVALID_ARG;
  int n_sm = 0;
  if (device_info(&n_sm) != DF_OK) return DF_ERR_CUDA;
  const float inv = 1.0f / (float)total_rows;
  if (!grad_logits) {
    launch_kernel(k_chunked_ce_eval, dim3(chunk_rows), dim3(kEvalThreads), 0, s, logits, targets, loss, chunk_rows, cols, inv);
    note_launch();
    return check_cuda(cudaGetLastError());
  }
  // whether logits and grad_logits rows are misaligned alike (both stored with 16-byte accesses)
  const bool same_phase = ((reinterpret_cast<uintptr_t>(logits) ^ reinterpret_cast<uintptr_t>(grad_logits)) & 15u) == 0;
  // The smallest number of slices per row that leaves room for four CTAs per SM; more while the rows alone do not give every SM
  // two CTAs; beyond eight slices' worth of columns (106000) the slices grow to a whole SM each. From 257 rows on, clusters of
  // four CTAs take as many rows as they have slices for, which keeps the additions to the loss at 256 or fewer.
  const uint32_t n4 = cols / 4 + 1;
  uint32_t slices = 1;
  auto groups_of = [&](uint32_t c) { return (n4 + c * kSliceThreads - 1) / (c * kSliceThreads); };
  while (slices < (uint32_t)kMaxCeCluster && (groups_of(slices) > kSliceGroups ||
                                              ((uint64_t)chunk_rows * slices < 2u * (uint64_t)n_sm && groups_of(slices) > 2)))
    slices *= 2;
  const uint32_t groups = groups_of(slices), cluster = slices < 4 && chunk_rows > 256 ? 4 : slices;
  const uint32_t rows_per_cluster = cluster / slices, units = (chunk_rows + rows_per_cluster - 1) / rows_per_cluster;
  if (groups > kMaxSliceGroups || (uint64_t)units * cluster > 0x7fffffffull) {
    const unsigned grid = chunk_rows < (uint32_t)n_sm ? chunk_rows : (unsigned)n_sm;
    launch_kernel(k_chunked_logit_ce_global, grid, dim3(kCeThreads), 0, s, logits, targets, grad_logits, loss, chunk_rows, cols, inv);
    note_launch();
    return check_cuda(cudaGetLastError());
  }
  // running clusters take over further rows only where there are more than two machines full of them: asking costs about 1.5 us
  const uint32_t more = (uint64_t)units * cluster > 8u * (uint64_t)n_sm ? 1u : 0u;
  const int st = check_cuda(launch_clusters(same_phase ? k_logit_ce_cluster<true> : k_logit_ce_cluster<false>, cluster, dim3(units * cluster),
                                            dim3(kSliceThreads), (size_t)groups * kSliceThreads * 16, s, logits, targets, grad_logits, loss,
                                            chunk_rows, cols, slices, groups, more, inv, device_status_ptr()));
  note_launch();
  return st;
}

}  // namespace df

// spmspv.cu -- y = A x with a sparse x, pushed over the columns of A.
//
// segTACO's SpMSpV (spmspv_csr_gpu_taco.h:5-55; CPU reference
// spmspv_csr_gpu.h:9-32) stores A as the CSR of A^T and gives each stored x_j
// one thread that walks column j and adds A_ij * x_j into y[i] atomically.
// Here y is cleared by a kernel of its own, and the stored entries of x are dealt to
// warps, E to a warp, by a second one that starts while the first runs and waits for it
// only before its first add:
//   * a lane looks up one entry (its column's bounds), and the warp walks the
//     nonzeros of its entries as one flat range, whatever the columns' lengths:
//     position f belongs to the entry that a search of the lanes' prefix sums
//     finds, four positions per lane loading while the four before are added;
//   * columns of more than kLongCol nonzeros are left out of that range: the lane that
//     finds one writes it to a list in each CTA of its cluster of eight, whose 64 warps
//     take its pieces in turn, so a column of 50,000 nonzeros loads eight SMs instead of
//     one warp.  The lists are complete once every CTA has looked its entries up; no CTA
//     reads another's shared memory, so none waits for another to finish.
// What bounds it: one atomic add per nonzero at a random y[i] (a warp's 32
// adds are 32 separate requests to L2), and for few entries the launches and the chain
// of dependent loads x -> column bounds -> nonzeros -> add.  Measured on GB300, both
// kernels, K columns of Poisson lengths; one warp per column / lists read across the
// cluster, without the prefetch, after a memset / here: 1M columns of mean 2, 1000 entries
// 3.2 / 5.3 / 3.3 us, 100,000 11.2 / 7.6 / 5.2; mean 20, 10,000 5.3 / 7.3 / 5.1,
// 100,000 18.8 / 20.7 / 17.2, 250,000 36.9 / 41.3 / 36.7; 300,000 of mean 100, 10,000 10.1 /
// 11.7 / 10.2, 100,000 57.9 / 76.9 / 63.5; 1M Zipf lengths up to 50,000, 100,000 entries 655 /
// 31.7 / 23.8; 1M power-law rows by columns (adds meet in hot rows), 100,000 22.7 / 27.5 /
// 23.9.
// Without clusters (a CTA's warps share its long columns) the short columns' calls are
// 0.5 to 2 us faster, the Zipf ones with 10,000 and 100,000 entries 20 and 38 us.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "internal.h"

namespace segtaco {

constexpr int kLongCol = 512;    // nonzeros; longer columns are shared by the cluster
constexpr int kColPiece = 512;   // nonzeros of a long column that a warp takes at a time
constexpr int kCluster = 8;      // CTAs per cluster (the portable maximum)
constexpr int kPushWarps = kCta / 32;

struct LongCol {
  int p0, p1;
  float x;
};

// Adds the nonzeros of one column range [p0, p1) scaled by x into y.
__device__ __forceinline__ void push_range(const int *__restrict__ row_idx,
                                           const float *__restrict__ val, int p0, int p1, float x,
                                           float *__restrict__ y, int lane) {
  constexpr int U = 8;
  const int n = p1 - p0;
  for (int o = lane; o < n; o += 32 * U) {
    int i[U];
    float a[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool ok = o + 32 * u < n;
      i[u] = ok ? ld_stream(row_idx + (p0 + o + 32 * u)) : -1;
      a[u] = ok && val ? ld_stream(val + (p0 + o + 32 * u)) : 1.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i[u] >= 0) atomicAdd(y + i[u], a[u] * x);
  }
}

// y = 0.  The push kernel may start at once; it waits before it adds.
__global__ void __launch_bounds__(kCta) clear_y_kernel(float *__restrict__ y, unsigned n) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const unsigned lead = (unsigned)((16 - ((uintptr_t)y & 15)) & 15) / 4;
  const unsigned head = lead < n ? lead : n;  // up to the first 16-byte boundary
  const unsigned t = blockIdx.x * (unsigned)kCta + threadIdx.x;
  float4 *q = reinterpret_cast<float4 *>(y + head);
  const unsigned v = (n - head) / 4;
  for (unsigned i = t; i < v; i += gridDim.x * (unsigned)kCta) q[i] = make_float4(0, 0, 0, 0);
  if (t < head) y[t] = 0.0f;
  if (t < n - head - 4 * v) y[head + 4 * v + t] = 0.0f;
}

// (Six CTAs per SM, 40 registers: 100,000 entries, mean 20, 15 to a warp 19.9 -> 16.9 us
// against the 48 registers taken unasked; eight spill, 20.3.)
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kCta, 6)
    spmspv_kernel(const int *__restrict__ col_ptr, const int *__restrict__ row_idx,
                  const float *__restrict__ val, int nx, const int *__restrict__ x_idx,
                  const float *__restrict__ x_vals, float *__restrict__ y, int per_warp) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ LongCol list[];  // the cluster's entries: kCluster * kPushWarps * per_warp
  __shared__ int count;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  if (threadIdx.x == 0) count = 0;
  cluster.barrier_arrive();  // every CTA's count is 0 once all have arrived
  const long long e0 = ((long long)blockIdx.x * kPushWarps + warp) * per_warp;
  const bool has = lane < per_warp && e0 + lane < nx;
  int p0 = 0, len = 0;
  float xv = 0.0f;
  if (has) {
    const int j = __ldg(x_idx + e0 + lane);
    xv = __ldg(x_vals + e0 + lane);
    p0 = __ldg(col_ptr + j);
    len = __ldg(col_ptr + j + 1) - p0;
  }
  const bool is_long = len > kLongCol;
  cluster.barrier_wait();
  if (is_long) {
#pragma unroll 1
    for (int b = 0; b < kCluster; ++b) {
      const int at = atomicAdd(cluster.map_shared_rank(&count, b), 1);
      cluster.map_shared_rank(list, b)[at] = LongCol{p0, p0 + len, xv};
    }
    len = 0;
  }
  cluster.barrier_arrive();  // the lists are complete once every thread has arrived
  asm volatile("griddepcontrol.wait;" ::: "memory");  // y is clear
  if (per_warp == 1) {
    const int p = __shfl_sync(FULL, p0, 0);
    push_range(row_idx, val, p, p + __shfl_sync(FULL, len, 0), __shfl_sync(FULL, xv, 0), y, lane);
  } else {
    // Flat range of the warp's short columns: `end` = its position past lane's column.
    int end = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, end, o);
      if (lane >= o) end += t;
    }
    const int total = __shfl_sync(FULL, end, 31);
    const int shift = p0 - (end - len);  // nonzero index = position + shift of its column
    constexpr int U = 4;
    struct Batch {
      int i[U];
      float a[U], x[U];
    };
    auto fetch = [&](int f0, Batch &b) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int f = f0 + 32 * u + lane;
        int k = 0;  // columns that end at or before position f
#pragma unroll
        for (int st = 16; st > 0; st >>= 1)
          if (__shfl_sync(FULL, end, k + st - 1) <= f) k += st;
        const int sh = __shfl_sync(FULL, shift, k);
        b.x[u] = __shfl_sync(FULL, xv, k);
        const bool ok = f < total;
        b.i[u] = ok ? ld_stream(row_idx + (f + sh)) : -1;
        b.a[u] = ok && val ? ld_stream(val + (f + sh)) : 1.0f;
      }
    };
    Batch b;
    if (total > 0) fetch(0, b);
    for (int f0 = 0; f0 < total; f0 += 32 * U) {
      Batch next;
      if (f0 + 32 * U < total) fetch(f0 + 32 * U, next);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (b.i[u] >= 0) atomicAdd(y + b.i[u], b.a[u] * b.x[u]);
      b = next;
    }
  }
  cluster.barrier_wait();
  // The cluster's long columns: pieces in turn over its 64 warps, from a warp that the
  // column picks (the lists' order differs from CTA to CTA).
  constexpr int W = kCluster * kPushWarps;
  const int n = count, me = (int)cluster.block_rank() * kPushWarps + warp;
  for (int k = 0; k < n; ++k) {
    const LongCol c = list[k];
    const int pieces = (c.p1 - c.p0 - 1) / kColPiece + 1;
    for (int q = (me - (c.p0 >> 4)) & (W - 1); q < pieces; q += W) {
      const int s = c.p0 + q * kColPiece;
      push_range(row_idx, val, s, s + imin(kColPiece, c.p1 - s), c.x, y, lane);
    }
  }
}

int launch_spmspv(int M, int K, long long nnz, const int *col_ptr, const int *row_idx,
                  const float *val, int nx, const int *x_idx, const float *x_vals, float *y,
                  cudaStream_t s) {
  if (M <= 0) return SEGTACO_OK;
  if (nx <= 0)
    return check_cuda(cudaMemsetAsync(y, 0, (size_t)M * sizeof(float), s), "memset y");
  // Entries per warp, E: few of them hide the chain of loads behind other warps, many
  // fill the flat ranges of short columns and save warps.  Up to 2048 entries one;
  // beyond, E = sqrt(nx / 98 sqrt(m)) for columns of mean length m.  Measured on GB300, E = 3
  // / 6 / 11 / 15 / 24: 10,000 entries, random rows, m = 2 4.9 / 4.6 / 4.5 / 4.6 / 4.7 us, 20
  // 5.3 / 5.8 / 6.0 / 6.8 / 8.0, 100 10.2 / 10.9 / 12.5 / 15.2 / 21; 100,000 entries, 2 17.9 /
  // 11.0 / 8.0 / 5.9 / 5.5, 20 23.7 / 20.1 / 18.3 / 16.9 / 17.4, 100 62 / 62 / 63 / 66 / 68,
  // banded (72) 31.0 / 24.9 / 23.0 / 21.8 / 24; 300,000 entries, 2 46 / 26 / 15.8 / 12.5 / 9.8,
  // 20 63 / 49 / 43 / 41 / 40.  1000 entries, E = 1 / 3 / 8: 2 3.7 / 4.0 / 4.3, 100 4.3 / 6.3 /
  // 9.5.
  const double mean = K > 0 && nnz > K ? (double)nnz / K : 1.0;
  int per_warp = 1;
  const double unit = 98.0 * std::sqrt(mean);
  while (nx > 2048 && per_warp < 32 && unit * (per_warp + 1) * (per_warp + 1) <= nx) ++per_warp;
  const long long vecs = (long long)M / 4, each = kCta * 4;
  const long long blocks = std::min<long long>(8LL * device_sms(), (vecs + each - 1) / each);
  clear_y_kernel<<<(unsigned)std::max<long long>(blocks, 1), kCta, 0, s>>>(y, (unsigned)M);
  SEGTACO_TRY(check_launch("clear_y_kernel"));
  const long long warps = ((long long)nx + per_warp - 1) / per_warp;
  const long long clusters = (warps + kCluster * kPushWarps - 1) / (kCluster * kPushWarps);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * kCluster));
  cfg.blockDim = dim3(kCta);
  cfg.dynamicSmemBytes = (size_t)kCluster * kPushWarps * per_warp * sizeof(LongCol);
  cfg.stream = s;
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return check_cuda(cudaLaunchKernelEx(&cfg, spmspv_kernel, col_ptr, row_idx, val, nx, x_idx, x_vals,
                                       y, per_warp),
                    "spmspv_kernel");
}

}  // namespace segtaco

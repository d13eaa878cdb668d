// spmspv.cu -- y = A x with a sparse x, pushed over the columns of A.
//
// segTACO's SpMSpV (spmspv_csr_gpu_taco.h:5-55; CPU reference
// spmspv_csr_gpu.h:9-32) stores A as the CSR of A^T and gives each stored x_j
// one thread that walks column j and adds A_ij * x_j into y[i] atomically.
// Here the stored entries of x are dealt to warps, E to a warp, and y is
// cleared on the same stream first:
//   * a lane looks up one entry (its column's bounds), and the warp walks the
//     nonzeros of its entries as one flat range, whatever the columns' lengths:
//     position f belongs to the entry that a search of the lanes' prefix sums
//     finds, four positions per lane in flight;
//   * columns of more than kLongCol nonzeros are left out of that range and
//     listed in shared memory.  A cluster of eight CTAs then reads its CTAs' lists
//     through distributed shared memory and deals their pieces to its 64 warps,
//     so a column of 50,000 nonzeros loads eight SMs instead of one warp.  The
//     cluster barrier is only waited for after the short columns.
// What bounds it: one atomic add per nonzero at a random y[i] (a warp's 32
// adds are 32 separate requests to L2), and for few entries the chain of
// dependent loads x -> column bounds -> nonzeros -> add.  Measured on GB300,
// 1M x 1M with Zipf column lengths up to 50,000 and 100,000 entries (call and
// clearing of y): 35.5 us, against 594 us with one warp per column, where the
// longest column's warp was what the call waited for.
#include <cooperative_groups.h>

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

__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kCta)
    spmspv_kernel(const int *__restrict__ col_ptr, const int *__restrict__ row_idx,
                  const float *__restrict__ val, int nx, const int *__restrict__ x_idx,
                  const float *__restrict__ x_vals, float *__restrict__ y, int per_warp) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ LongCol list[kPushWarps * 32];
  __shared__ int count;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
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
  if (len > kLongCol) {
    list[atomicAdd(&count, 1)] = LongCol{p0, p0 + len, xv};
    len = 0;
  }
  cluster.barrier_arrive();  // the CTA's list is complete once every thread has arrived
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
  for (int f0 = 0; f0 < total; f0 += 32 * U) {
    int i[U];
    float a[U], x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int f = f0 + 32 * u + lane;
      int k = 0;  // columns that end at or before position f
#pragma unroll
      for (int st = 16; st > 0; st >>= 1)
        if (__shfl_sync(FULL, end, k + st - 1) <= f) k += st;
      const int sh = __shfl_sync(FULL, shift, k);
      x[u] = __shfl_sync(FULL, xv, k);
      const bool ok = f < total;
      i[u] = ok ? ld_stream(row_idx + (f + sh)) : -1;
      a[u] = ok && val ? ld_stream(val + (f + sh)) : 1.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i[u] >= 0) atomicAdd(y + i[u], a[u] * x[u]);
  }
  cluster.barrier_wait();
  // The cluster's long columns: piece k of all lists goes to warp k mod 64.
  const int me = (int)cluster.block_rank() * kPushWarps + warp;
  int piece = 0;
  for (int b = 0; b < kCluster; ++b) {
    const int n = *cluster.map_shared_rank(&count, b);
    const LongCol *l = cluster.map_shared_rank(list, b);
    for (int k = 0; k < n; ++k) {
      const LongCol c = l[k];
      const int pieces = (c.p1 - c.p0 + kColPiece - 1) / kColPiece;
      // first piece of this column at or after `piece` that is this warp's
      const int skip = (me - piece % (kCluster * kPushWarps) + kCluster * kPushWarps) %
                       (kCluster * kPushWarps);
      for (int q = skip; q < pieces; q += kCluster * kPushWarps) {
        const int s = c.p0 + q * kColPiece;
        push_range(row_idx, val, s, s + imin(kColPiece, c.p1 - s), c.x, y, lane);
      }
      piece += pieces;
    }
  }
  cluster.sync();  // no CTA leaves while another reads its list
}

int launch_spmspv(int M, int K, const int *col_ptr, const int *row_idx, const float *val, int nx,
                  const int *x_idx, const float *x_vals, float *y, cudaStream_t s) {
  (void)K;
  if (M > 0) SEGTACO_TRY(check_cuda(cudaMemsetAsync(y, 0, (size_t)M * sizeof(float), s), "memset y"));
  if (nx <= 0) return SEGTACO_OK;
  // Entries per warp: one while that gives no more than a resident wave of
  // warps (64 per SM), then more of them to a warp.
  int per_warp = 1;
  while (per_warp < 32 && nx / per_warp > 64 * device_sms()) per_warp <<= 1;
  const long long warps = ((long long)nx + per_warp - 1) / per_warp;
  const long long clusters = (warps + kCluster * kPushWarps - 1) / (kCluster * kPushWarps);
  spmspv_kernel<<<(unsigned)(clusters * kCluster), kCta, 0, s>>>(col_ptr, row_idx, val, nx, x_idx,
                                                                x_vals, y, per_warp);
  return check_launch("spmspv_kernel");
}

}  // namespace segtaco

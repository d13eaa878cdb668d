// spmm_join.cu -- rb_pr over uneven rows: merge-path chunks (spmm_split.cuh) that store
// their sums of cut rows instead of adding them to C, and the kernel here, which adds
// each cut row's sums in chunk order, so the result does not vary from run to run.
//
// A row-block warp that meets a row of tens of thousands of nonzeros walks it alone
// while the GPU waits; chunks share it out, as pieces do (spmm_long.cu), and walk the
// short rows several side by side too.  Both kernels search their chunk edges, so
// nothing is prepared.  Measured on GB300, power-law rows, row walk -> here: 17,801 rows
// (357,000 nonzeros), N = 97 679 -> 38 us, 20,000, N = 128 284 -> 20; pieces -> here:
// 60,000 rows, N = 64 108 -> 45, 400,000, N = 37 432 -> 183; the eb_pr product of the same
// shape, without the sums' traffic and this launch, 26, 19, 42 and 164.
//
// What bounds the kernel here: the latency of the edge search and of a row's sums; a
// row of many chunks is the CTA's, each warp every eighth sum.
#include "internal.h"
#include "spmm_launch.cuh"
#include "spmm_split.cuh"

namespace segtaco {
namespace {

constexpr int kJoinWarps = 8;
constexpr int kJoinShort = 16;  // sums that one warp adds up; more: the whole CTA

__device__ __forceinline__ void add4(float4 &a, const float4 &b) {
  a.x += b.x, a.y += b.y, a.z += b.z, a.w += b.w;
}

// Warp w takes the row cut by chunk w's first edge, if it ends in the chunk.  The row
// began in the chunk of its first nonzero (merge item row_ptr[r] + r); that chunk and
// those after it hold its open sums, chunk w its last one, if any of its nonzeros lie
// there.
__global__ void __launch_bounds__(kJoinWarps * 32) spmm_join_kernel(SpmmArgs<float> a, int D) {
  __shared__ int s_row[kJoinWarps], s_terms[kJoinWarps];
  __shared__ long long s_first[kJoinWarps];
  __shared__ bool s_head[kJoinWarps];
  __shared__ float4 s_sum[kJoinWarps][32];
  const int wid = threadIdx.x / 32, lane = threadIdx.x & 31;
  const long long w = (long long)blockIdx.x * kJoinWarps + wid;
  int row = -1, terms = 0;
  long long first = 0;
  bool head = false;
  if (w < a.units) {
    const ChunkEdges ce = search_edges(a, w, D, lane);
    if (ce.x1 > ce.x0) {
      const int rp0 = __ldg(a.row_ptr + ce.x0);
      if (rp0 < ce.y0) {
        row = ce.x0;
        first = ((long long)rp0 + ce.x0) / D;
        head = __ldg(a.row_ptr + ce.x0 + 1) > ce.y0;
        terms = (int)(w - first) + (head ? 1 : 0);
      }
    }
  }
  // Sums `from`, from + step, ... of a row at columns col .. col+3, in order (the row
  // pitch of the sums is a multiple of 4).
  auto add_up = [&](long long c0, int n, bool last_is_head, int from, int step, int col) {
    float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int i = from; i < n; i += step) {
      const long long at = 2 * (c0 + i) + (last_is_head && i == n - 1 ? 0 : 1);
      add4(t, *reinterpret_cast<const float4 *>(a.piece_part + at * a.piece_ld + col));
    }
    return t;
  };
  auto put = [&](int r, int col, const float4 &t) {
    float *dst = a.C + (long long)r * a.ldc + col;
    const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (col + k < a.N) dst[k] = v[k];
  };
  const bool far = terms > kJoinShort;
  if (row >= 0 && !far)
    for (int col = 4 * lane; col < a.N; col += 128)
      put(row, col, add_up(first, terms, head, 0, 1, col));
  if (lane == 0) {
    s_row[wid] = row;
    s_terms[wid] = far ? terms : 0;
    s_first[wid] = first;
    s_head[wid] = head;
  }
  __syncthreads();
  for (int k = 0; k < kJoinWarps; ++k) {
    if (s_terms[k] == 0) continue;  // the whole CTA agrees
    for (int c0 = 0; c0 < a.N; c0 += 128) {
      const int col = c0 + 4 * lane;
      if (col < a.N)
        s_sum[wid][lane] = add_up(s_first[k], s_terms[k], s_head[k], wid, kJoinWarps, col);
      __syncthreads();
      if (wid == 0 && col < a.N) {
        float4 t = s_sum[0][lane];
#pragma unroll
        for (int j = 1; j < kJoinWarps; ++j) add4(t, s_sum[j][lane]);
        put(s_row[k], col, t);
      }
      __syncthreads();  // s_sum is free for the next columns
    }
  }
}

}  // namespace

int launch_spmm_join(const SpmmLaunch &L, cudaStream_t s) {
  const SpmmArgs<float> a = make_spmm_args<float>(L);
  const unsigned grid = (unsigned)((L.units + kJoinWarps - 1) / kJoinWarps);
  spmm_join_kernel<<<grid, kJoinWarps * 32, 0, s>>>(a, L.split_items);
  return check_launch("spmm_join_kernel");
}

}  // namespace segtaco

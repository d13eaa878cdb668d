// spmv.cu -- y = A x, A CSR.
//
// A warp takes a chunk of consecutive nonzeros, 128 at a time with four gathers of x
// in flight per lane, so that every lane has a nonzero whatever the row lengths:
//   * where no row ends among the 128, each lane adds its products to a partial sum of
//     the open row;
//   * otherwise the products of 32 nonzeros are summed by rows with a segmented scan
//     (the rows' ends as a bit mask), and the lanes, one row each, fetch their row's
//     sum and store it, neighbouring rows together.
// The chunk's first row is searched in the kernel.  y is cleared first, so empty rows
// need no store; a row cut by a chunk edge receives an atomic add from each chunk that
// holds part of it, every other row one plain store.
//
// What bounds it: each 4-byte gather of x from a random position is a tag lookup and a
// 32-byte sector of its own in L1.  Measured on GB300, partition and the N = 1 row walk
// before -> here: 1M power-law rows (20M nonzeros) 127 -> 99 us, 400,000 lognormal rows
// 79 -> 36, 300,000 rows of 16 68 -> 37, 200,000 banded rows 88 -> 54, 1000 rows 21 -> 8.
// 2 / 6 / 8 batches in flight 121 / 102 / 112 us; 64 warps per SM (32 registers) 114.
#include <climits>

#include "common.cuh"
#include "internal.h"

namespace segtaco {

constexpr int kSpmvBatches = 4;  // batches of 32 nonzeros whose gathers are in flight

__global__ void __launch_bounds__(kCta, 6)
    spmv_kernel(int M, unsigned nnz, const int *__restrict__ row_ptr,
                const int *__restrict__ col, const float *__restrict__ val,
                const float *__restrict__ x, float *__restrict__ y, unsigned chunk) {
  constexpr int B = kSpmvBatches;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned long long first = ((unsigned long long)blockIdx.x * (kCta / 32) + threadIdx.x / 32) * chunk;
  if (first >= nnz) return;  // whole warp leaves together
  const unsigned p0 = (unsigned)first;
  const unsigned pe = nnz - p0 < chunk ? nnz : p0 + chunk;
  int open = warp_row_of(row_ptr, M, p0, lane);  // the row of the next nonzero
  const int cut = (unsigned)__ldg(row_ptr + open) < p0 ? open : -1;  // began in an earlier chunk
  // ends of rows wb .. wb+31
  int wb = open;
  auto window = [&](int b) {
    return b + lane < M ? (unsigned)__ldg(row_ptr + b + 1 + lane) : 0xffffffffu;
  };
  unsigned re = window(wb);
  unsigned oend = __shfl_sync(FULL, re, 0);  // end of row `open`
  float part = 0.0f;  // this lane's share of the open row's sum
  for (unsigned p = p0; p < pe; p += 32 * B) {
    float v[B];
    {
      int c[B];
      float a[B];
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const bool ok = p + 32 * b + lane < pe;
        c[b] = ok ? ld_stream(col + (p + 32 * b + lane)) : -1;
        a[b] = ok && val ? ld_stream(val + (p + 32 * b + lane)) : 1.0f;
      }
#pragma unroll
      for (int b = 0; b < B; ++b) v[b] = c[b] >= 0 ? a[b] * __ldg(x + c[b]) : 0.0f;
    }
    if (pe - p >= 32 * B && oend > p + 32 * B) {
#pragma unroll
      for (int b = 0; b < B; ++b) part += v[b];
      continue;
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const unsigned q = p + 32 * b;
      if (q >= pe) break;
      const unsigned qe = pe - q < 32 ? pe : q + 32;  // this batch: [q, qe)
      if (oend > qe) {  // no row ends here
        part += v[b];
        continue;
      }
      // The open row's sum so far joins the batch's first position.
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
      float s = lane == 0 ? v[b] + part : v[b];
      // Ends of rows inside the batch, over as many windows as it touches.
      const int wb0 = wb;
      unsigned ends = 0;
      for (;;) {
        ends |= __reduce_or_sync(FULL, re > q && re <= qe ? 1u << (re - 1 - q) : 0u);
        if (__shfl_sync(FULL, re, 31) > qe) break;
        wb += 32;
        re = window(wb);
      }
      // Segmented inclusive scan: sums from the row's first position here.
      const unsigned before = ends & ((1u << lane) - 1u);
      const int begin = 32 - __clz(before);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(FULL, s, o);
        if (lane - o >= begin) s += t;
      }
      // The rows that end here, one per lane of their window.
      for (int wx = wb0;; wx += 32) {
        const unsigned e = wx == wb ? re : window(wx);
        unsigned st = __shfl_up_sync(FULL, e, 1);
        if (lane == 0) st = wx == wb0 ? 0u : (unsigned)__ldg(row_ptr + wx);
        // (the first window's first row is the open one or has ended: never empty here)
        const bool mine = e > q && e <= qe && e != st;
        const float sum = __shfl_sync(FULL, s, mine ? (int)(e - 1 - q) : 0);
        if (mine) {
          if (wx + lane == cut)
            atomicAdd(y + cut, sum);
          else
            __stcs(y + wx + lane, sum);
        }
        if (wx == wb) break;
      }
      // The row open after the batch and its sum here.
      const unsigned later = __ballot_sync(FULL, re > qe);
      const int f = __ffs(later) - 1;  // the window's last end is past the batch
      open = wb + f;
      oend = __shfl_sync(FULL, re, f);
      const int n = (int)(qe - q);
      const float tail = __shfl_sync(FULL, s, n - 1);
      part = lane == 0 && !((ends >> (n - 1)) & 1u) ? tail : 0.0f;
    }
  }
  // The row open at the chunk's end continues in the next chunk.
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(FULL, part, o);
  if (lane == 0 && oend > pe && (unsigned)__ldg(row_ptr + open) < pe) atomicAdd(y + open, part);
}

int launch_spmv(int M, long long nnz, const int *row_ptr, const int *col, const float *val,
                const float *x, float *y, cudaStream_t s) {
  SEGTACO_TRY(check_cuda(cudaMemsetAsync(y, 0, (size_t)M * sizeof(float), s), "memset y"));
  if (nnz == 0) return SEGTACO_OK;
  // 1024 nonzeros per warp, down to 128 while that leaves fewer than two waves of warps.
  unsigned chunk = 1024;
  while (chunk > 128 && nnz / chunk < 2 * 48 * 152) chunk >>= 1;
  const long long warps = (nnz + chunk - 1) / chunk;
  spmv_kernel<<<(unsigned)((warps + kCta / 32 - 1) / (kCta / 32)), kCta, 0, s>>>(
      M, (unsigned)nnz, row_ptr, col, val, x, y, chunk);
  return check_launch("spmv_kernel");
}

}  // namespace segtaco

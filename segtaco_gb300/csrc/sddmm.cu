// sddmm.cu -- out[p] = vals[p] * <X[i,:], Y[j,:]> for every nonzero p = (i, j).
//
// segTACO's SDDMM (sddmm_csr_gpu_taco.h:5-150, CPU reference sddmm_csr_gpu.h:9-50)
// is element-balanced: nonzero blocks with start rows from
// taco_binarySearchBeforeBlock.  Here a warp takes a block of nonzeros (256 unless
// the call says otherwise) and groups of G lanes one dot product each.  Three kernels:
// the default (sddmm_gather_kernel, any D and alignment, its warps search their first
// row), the fixed shapes (sddmm_fixed_kernel: D of 512 bytes and more in 32-byte
// lanes, batches of problems, and explicit requests) and the general one
// (sddmm_kernel: explicit requests and row pitches from 4 GB).
#include <algorithm>
#include <atomic>
#include <climits>

#include "common.cuh"
#include "internal.h"

namespace segtaco {

constexpr int kSddmmBlock = 256;  // nonzeros per warp

template <typename XT, int V, int G, int U = (V == 8 ? 1 : 4)>
__global__ void __launch_bounds__(kCta, 3) sddmm_kernel(int M, long long nnz,
                                                    const int *__restrict__ row_ptr,
                                                    const int *__restrict__ col,
                                                    const float *__restrict__ val,
                                                    const XT *__restrict__ X,
                                                    const XT *__restrict__ Y, long long ldx,
                                                    long long ldy, int D, float *__restrict__ out,
                                                    const int *__restrict__ starts,
                                                    long long nblk, int blk) {
  constexpr int P = 32 / G;  // nonzeros per step
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane & (G - 1);
  const long long w = (long long)blockIdx.x * (kCta / 32) + threadIdx.x / 32;
  if (w >= nblk) return;
  const long long pb = w * blk;
  const long long pe = pb + blk < nnz ? pb + blk : nnz;
  int wb = __ldg(starts + w);  // row of nonzero pb
  int rw = (wb + lane < M) ? __ldg(row_ptr + wb + 1 + lane) : INT_MAX;
  for (long long p = pb; p < pe; p += 32) {
    const int nb = (int)(pe - p < 32 ? pe - p : 32);
    const int mc = lane < nb ? ld_stream(col + p + lane) : 0;
    const float mv = lane < nb ? (val ? ld_stream(val + p + lane) : 1.0f) : 0.0f;
    for (;;) {
      const int adv = __popc(__ballot_sync(FULL, (long long)rw <= p));
      if (adv == 0) break;
      wb += adv;
      rw = (wb + lane < M) ? __ldg(row_ptr + wb + 1 + lane) : INT_MAX;
    }
    const bool covered = (long long)__shfl_sync(FULL, rw, 31) > p + nb - 1;
    float res = 0.0f;
    const int nsteps = (nb + P - 1) / P;
    // Steps of P nonzeros, U at a time: every load of the U steps is issued
    // before the first multiply-add.
    for (int s0 = 0; s0 < nsteps; s0 += U) {
      int rows[U], js[U];
      bool ok[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int s = s0 + u;
        const int t = s * P + g;
        ok[u] = s < nsteps && t < nb;
        js[u] = __shfl_sync(FULL, mc, t & 31);
        int row = wb;
        if (covered) {
#pragma unroll
          for (int gg = 0; gg < P; ++gg) {
            const unsigned bal = __ballot_sync(FULL, (long long)rw <= p + s * P + gg);
            if (g == gg) row = wb + __popc(bal);
          }
        } else if (ok[u]) {
          int lo = wb, hi = M - 1;
          const long long q = p + t;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((long long)__ldg(row_ptr + mid) <= q)
              lo = mid;
            else
              hi = mid - 1;
          }
          row = lo;
        }
        rows[u] = row;
      }
      float acc[U];
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u] = 0.0f;
      for (int k = gl * V; k < D; k += G * V) {
        float xa[U][V], ya[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (ok[u]) {
            DenseLoad<XT, V, false>::run(X + (long long)rows[u] * ldx + k, xa[u], 0);
            DenseLoad<XT, V, false>::run(Y + (long long)js[u] * ldy + k, ya[u], 0);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (ok[u]) {
#pragma unroll
            for (int v = 0; v < V; ++v) acc[u] = fmaf(xa[u][v], ya[u][v], acc[u]);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float a = acc[u];
#pragma unroll
        for (int o = 1; o < G; o <<= 1) a += __shfl_xor_sync(FULL, a, o);
        // Nonzero t of step s was reduced by group t - s*P; lane t keeps it.
        const int s = s0 + u;
        const float r = __shfl_sync(FULL, a, ((lane - s * P) & (P - 1)) * G);
        if (lane / P == s) res = r;
      }
    }
    if (lane < nb) out[p + lane] = mv * res;
  }
}

// A row of X is read once, or for skewed rows by neighbouring warps: where X and Y do not
// stay in L2 from call to call, it leaves L2 to Y's rows (the results are streamed).
__device__ __forceinline__ uint64_t sddmm_policy_x(bool first) {
  return first ? l2_policy_evict_first() : l2_policy_evict_normal();
}

// The default kernel.  G lanes hold one dot product, each lane C chunks of E
// elements (32 bytes where D, ldx, ldy and the pointers allow it, else 16, else one
// or two elements), so the lanes of a group read whole lines of Y[j]; a group takes
// U consecutive nonzeros per step and issues the loads of all of them, and of X for
// the rows of its first and last nonzero, before the first multiply-add.  X stays
// in registers while the row does.  The U sums over G lanes are reduced together,
// each exchange halving the values a lane still holds (U = 4, G = 8: 4 shuffles
// instead of 12).  FULL: D = G*E*C, so no lane is idle and one pass covers D;
// otherwise idle chunks load zeros and D beyond G*E*C goes in passes.
//
// What bounds it: the gathers of Y in flight (300,000 power-law rows, D = 128 bf16: long-
// scoreboard stalls first, 61 % of issue slots, 8.5 TB/s of Y rows, 70 % of them from L2,
// whose pipe and L1's are under 50 % busy).  The row of a warp's first nonzero is searched in the kernel,
// so a call is one launch and needs no scratch.  Measured on GB300, call time, the
// kernels below (block starts, then the fixed-shape or general kernel) -> here:
// 300,000 power-law rows, D = 128 bf16 196 -> 184 us, D = 64 fp32 170 -> 162; 100,000
// lognormal rows, fp32, D = 16 / 32 17.9 -> 13.3, 24 -> 18; 85 204 -> 60; 40 84 -> 30;
// 243,068 rows, D = 70 bf16 522 -> 79; 5000 rows, D = 64 19 -> 5.
// U: 4, or 2 for 32-byte lanes on 8 lanes and more, which keeps 64 registers without
// spills (300,000 power-law rows, D = 128 bf16: 185 us with 2, 221 with 4).
template <int BYTES, int G> __host__ __device__ constexpr int sddmm_steps() {
  return G < 4 ? G : BYTES == 32 && G >= 8 ? 2 : 4;
}

template <typename XT, int E, int C, int G, bool FULL>
__global__ void __launch_bounds__(kCta, 4) sddmm_gather_kernel(
    int M, unsigned nnz, const int *__restrict__ row_ptr, const int *__restrict__ col,
    const float *__restrict__ val, const XT *__restrict__ X, const XT *__restrict__ Y,
    unsigned ldx, unsigned ldy, int D, float *__restrict__ out, unsigned nblk, unsigned blk,
    bool x_first) {
  constexpr int P = 32 / G;
  constexpr int U = sddmm_steps<E * (int)sizeof(XT), G>();
  using Dv = Dense<XT, E>;
  const unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane & (G - 1);
  const unsigned w = blockIdx.x * (kCta / 32) + threadIdx.x / 32;
  if (w >= nblk) return;  // whole warp leaves together
  const uint64_t pol = l2_policy_evict_normal();
  const uint64_t polx = sddmm_policy_x(x_first);
  const unsigned pb = w * blk;
  const unsigned pe = nnz - pb < blk ? nnz : pb + blk;
  auto load_cols = [&](unsigned p) { return p + lane < pe ? ld_stream(col + (p + lane)) : 0; };
  auto load_vals = [&](unsigned p) {
    return val && p + lane < pe ? ld_stream(val + (p + lane)) : 1.0f;
  };
  int mc = load_cols(pb);
  float mv = load_vals(pb);
  int wb = warp_row_of(row_ptr, M, pb, lane);
  // ends of rows wb .. wb+31
  unsigned rw = wb + lane < M ? (unsigned)__ldg(row_ptr + wb + 1 + lane) : 0xffffffffu;
  // ldx and ldy are in bytes
  const char *Xg = reinterpret_cast<const char *>(X + gl * E);
  const char *Yg = reinterpret_cast<const char *>(Y + gl * E);
  typename Dv::raw_t xa[C];  // X of row xrow (in one pass only)
  int xrow = -1;
  for (unsigned p = pb; p < pe; p += 32) {
    const int nb = pe - p < 32 ? (int)(pe - p) : 32;
    const int mcn = load_cols(p + 32);
    const float mvn = load_vals(p + 32);
    for (;;) {
      const int adv = __popc(__ballot_sync(ALL, rw <= p));
      if (adv == 0) break;
      wb += adv;
      rw = wb + lane < M ? (unsigned)__ldg(row_ptr + wb + 1 + lane) : 0xffffffffu;
    }
    // Row of nonzero p + lane (positions past the block: the block's last row).
    const unsigned q = p + (lane < nb ? lane : nb - 1);
    int myrow;
    if (__shfl_sync(ALL, rw, 31) > p + (nb - 1)) {  // the window holds the batch
      int rr = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1)
        if (__shfl_sync(ALL, rw, rr + st - 1) <= q) rr += st;
      myrow = wb + rr;
    } else {
      int lo = wb, hi = M - 1;
      while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if ((unsigned)__ldg(row_ptr + mid) <= q)
          lo = mid;
        else
          hi = mid - 1;
      }
      myrow = lo;
    }
#pragma unroll 1
    for (int s0 = 0; s0 < nb; s0 += P * U) {
      const int t0 = s0 + g * U;  // this group's nonzeros t0 .. t0+U-1 of the batch
      float sum[U];
#pragma unroll
      for (int u = 0; u < U; ++u) sum[u] = 0.0f;
      const int r0 = __shfl_sync(ALL, myrow, t0), r1 = __shfl_sync(ALL, myrow, t0 + U - 1);
      const bool one_row = U == 1 || __all_sync(ALL, r0 == r1);
      for (int k0 = 0; k0 < (FULL ? 1 : D); k0 += FULL ? 1 : G * E * C) {
        const int left = FULL ? D : D - k0 - gl * E;
        const int chunks = left <= 0 ? 0 : imin(C, (left + G * E - 1) / (G * E));
        const size_t kb = FULL ? 0 : (size_t)(left > 0 ? k0 : 0) * sizeof(XT);
        auto load = [&](const char *base, int r, unsigned ld, typename Dv::raw_t(&d)[C],
                        uint64_t hint) {
          const XT *p_ = reinterpret_cast<const XT *>(base + (size_t)(unsigned)r * ld + kb);
#pragma unroll
          for (int c = 0; c < C; ++c)
            d[c] = FULL ? Dv::load(p_ + c * (G * E), hint)
                        : Dv::load_if(p_ + c * (G * E), hint, c < chunks);
        };
        typename Dv::raw_t y[U][C];
#pragma unroll
        for (int u = 0; u < U; ++u) load(Yg, __shfl_sync(ALL, mc, t0 + u), ldy, y[u], pol);
        if (r0 != xrow || (!FULL && D > G * E * C)) load(Xg, r0, ldx, xa, polx);
        auto dot = [&](int u) {
#pragma unroll
          for (int c = 0; c < C; ++c)
#pragma unroll
            for (int e = 0; e < E; ++e)
              sum[u] = fmaf(Dv::get(xa[c], e), Dv::get(y[u][c], e), sum[u]);
        };
        if (one_row) {
#pragma unroll
          for (int u = 0; u < U; ++u) dot(u);
        } else {
          typename Dv::raw_t xb[C];
          load(Xg, r1, ldx, xb, polx);
          int at = r0;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int r = __shfl_sync(ALL, myrow, t0 + u);
            if (r != at) {
              at = r;
              if (r == r1) {
#pragma unroll
                for (int c = 0; c < C; ++c) xa[c] = xb[c];
              } else {
                load(Xg, r, ldx, xa, polx);
              }
            }
            __syncwarp();
            dot(u);
          }
        }
      }
      xrow = r1;
      // Sums over the group's lanes; lane gl ends with that of nonzero t0 + first.
      int first = 0;
      bool owner = true;
      {
        int n = U;
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) {
          const bool hi = (lane & o) != 0;
          if (n > 1) {
            n /= 2;
#pragma unroll
            for (int i = 0; i < U / 2; ++i) {
              if (i < n) {
                const float keep = hi ? sum[i + n] : sum[i];
                const float send = hi ? sum[i] : sum[i + n];
                sum[i] = keep + __shfl_xor_sync(ALL, send, o);
              }
            }
            if (hi) first += n;
          } else {
            sum[0] += __shfl_xor_sync(ALL, sum[0], o);
            if (hi) owner = false;
          }
        }
      }
      const float v = __shfl_sync(ALL, mv, t0 + first);
      if (owner && t0 + first < nb) __stcs(out + (p + (t0 + first)), v * sum[0]);
    }
    mc = mcn;
    mv = mvn;
  }
}

// Sixteen-byte vectors and D = G*V*KI: G lanes per dot product, each lane
// KI vector loads of X[i] and of Y[j] (KI = 4 whenever D allows), so one step
// covers P = 32/G nonzeros and its reduction takes only log2(G) shuffles.  The
// row of every nonzero of a batch is found once (a search of the 32-row
// window, or of row_ptr when the batch leaves it) and passed by one shuffle
// per step.  A group keeps its slice of X[i] in registers until its row
// changes.  Raw vectors stay in registers until their multiply-adds.
template <typename XT, int V, int G, int KI>
__device__ __forceinline__ void sddmm_fixed_block(
    int M, long long nnz, const int *__restrict__ row_ptr, const int *__restrict__ col,
    const float *__restrict__ val, const XT *__restrict__ X, const XT *__restrict__ Y,
    long long ldx, long long ldy, float *__restrict__ out, const int *__restrict__ starts,
    long long w, int blk, bool x_first) {
  constexpr int P = 32 / G;
  using Dv = Dense<XT, V>;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane & (G - 1);
  const uint64_t pol = l2_policy_evict_normal();
  const uint64_t polx = sddmm_policy_x(x_first);
  const long long pb = w * blk;
  const long long pe = pb + blk < nnz ? pb + blk : nnz;
  int mcn = pb + lane < pe ? ld_stream(col + pb + lane) : 0;
  float mvn = pb + lane < pe && val ? ld_stream(val + pb + lane) : 1.0f;
  int wb = starts ? __ldg(starts + w) : warp_row_of(row_ptr, M, pb, lane);  // row of nonzero pb
  int rw = (wb + lane < M) ? __ldg(row_ptr + wb + 1 + lane) : INT_MAX;
  // The group's slice of X[xrow] stays in registers while its nonzeros stay in
  // that row (consecutive nonzeros of a row go to the same group's steps).
  typename Dv::raw_t xa[KI];
  int xrow = -1;
  for (long long p = pb; p < pe; p += 32) {
    const int nb = (int)(pe - p < 32 ? pe - p : 32);
    const int mc = mcn;  // columns and values of this batch; the next one's load meanwhile
    const float mv = mvn;
    mcn = p + 32 + lane < pe ? ld_stream(col + p + 32 + lane) : 0;
    mvn = p + 32 + lane < pe && val ? ld_stream(val + p + 32 + lane) : 1.0f;
    for (;;) {
      const int adv = __popc(__ballot_sync(FULL, (long long)rw <= p));
      if (adv == 0) break;
      wb += adv;
      rw = (wb + lane < M) ? __ldg(row_ptr + wb + 1 + lane) : INT_MAX;
    }
    // Row of nonzero p + lane.
    const long long q = p + lane;
    int myrow;
    if ((long long)__shfl_sync(FULL, rw, 31) > p + nb - 1) {  // the window holds the batch
      int rr = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1)
        if ((long long)__shfl_sync(FULL, rw, rr + st - 1) <= q) rr += st;
      myrow = wb + rr;
    } else {
      int lo = wb, hi = M - 1;
      if (lane < nb) {
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if ((long long)__ldg(row_ptr + mid) <= q)
            lo = mid;
          else
            hi = mid - 1;
        }
      }
      myrow = lo;
    }
    float res = 0.0f;
    const int nsteps = (nb + P - 1) / P;
    for (int s = 0; s < nsteps; ++s) {
      const int t = s * P + g;
      const int j = __shfl_sync(FULL, mc, t & 31);
      const int row = __shfl_sync(FULL, myrow, t & 31);
      float acc = 0.0f;
      if (t < nb) {
        if (row != xrow) {  // a new row for this group: its slice of X[i]
          const XT *xr = X + (long long)row * ldx + gl * V;
#pragma unroll
          for (int k = 0; k < KI; ++k) xa[k] = Dv::load(xr + k * G * V, polx);
          xrow = row;
        }
        const XT *yr = Y + (long long)j * ldy + gl * V;
        typename Dv::raw_t ya[KI];
#pragma unroll
        for (int k = 0; k < KI; ++k) ya[k] = Dv::load(yr + k * G * V, pol);
#pragma unroll
        for (int k = 0; k < KI; ++k) {
#pragma unroll
          for (int v = 0; v < V; ++v) acc = fmaf(Dv::get(xa[k], v), Dv::get(ya[k], v), acc);
        }
      }
#pragma unroll
      for (int o = 1; o < G; o <<= 1) acc += __shfl_xor_sync(FULL, acc, o);
      const float r = __shfl_sync(FULL, acc, ((lane - s * P) & (P - 1)) * G);
      if (lane / P == s) res = r;
    }
    if (lane < nb) __stcs(out + (p + lane), mv * res);
  }
}

template <typename XT, int V, int G, int KI>
__global__ void __launch_bounds__(kCta, 4) sddmm_fixed_kernel(
    int M, long long nnz, const int *__restrict__ row_ptr, const int *__restrict__ col,
    const float *__restrict__ val, const XT *__restrict__ X, const XT *__restrict__ Y,
    long long ldx, long long ldy, float *__restrict__ out, const int *__restrict__ starts,
    long long nblk, int blk, bool x_first) {
  const long long w = (long long)blockIdx.x * (kCta / 32) + threadIdx.x / 32;
  if (w >= nblk) return;  // whole warp leaves together
  sddmm_fixed_block<XT, V, G, KI>(M, nnz, row_ptr, col, val, X, Y, ldx, ldy, out, starts, w,
                                  blk, x_first);
}

// Several problems of one shape in one launch: warp w takes block
// w - blk_begin[p] of the last problem p with blk_begin[p] <= w.
template <typename XT, int V, int G, int KI>
__global__ void __launch_bounds__(kCta, 4) sddmm_fixed_multi_kernel(
    const SddmmProblem *__restrict__ probs, int nprobs, long long total) {
  const long long w = (long long)blockIdx.x * (kCta / 32) + threadIdx.x / 32;
  if (w >= total) return;  // whole warp leaves together
  int lo = 0, hi = nprobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].blk_begin <= w)
      lo = mid;
    else
      hi = mid - 1;
  }
  const SddmmProblem &a = probs[lo];
  sddmm_fixed_block<XT, V, G, KI>(a.M, a.nnz, a.row_ptr, a.col, a.val,
                                  static_cast<const XT *>(a.X), static_cast<const XT *>(a.Y),
                                  a.ldx, a.ldy, a.out, a.starts, w - a.blk_begin, kSddmmBlock,
                                  false);
}

// Blocks of at most P nonzeros per warp that fill whole waves of resident warps, so that
// the last of a few waves is not nearly empty.  Measured on GB300, blocks of 256 /
// here: rows of 16, 1.26M nonzeros (1.01 waves), D = 128 fp32 80 / 56 us, D = 64 51 / 35; 3.2M
// (2.6 waves), D = 128 163 / 150; 1.8M lognormal (1.5 waves), D = 100 113 / 97; 60,000
// power-law rows (1.1 waves), D = 64 47 / 39; from four waves on it makes no difference.
struct SddmmGrid {
  long long blk, nblk;
  unsigned ctas;
};
template <auto Kernel> SddmmGrid sddmm_grid(long long nnz, int P) {
  static std::atomic<int> per_sm{0};
  int n = per_sm.load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, kCta, 0) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 4;
    }
    per_sm.store(n, std::memory_order_relaxed);
  }
  const long long slots = (long long)device_sms() * n * (kCta / 32);
  const long long waves = (nnz + P * slots - 1) / (P * slots);
  SddmmGrid g;
  g.blk = P;
  if (waves > 1 && waves <= 4) {
    const long long each = (nnz + waves * slots - 1) / (waves * slots);
    g.blk = std::min<long long>(P, (each + 15) / 16 * 16);
  }
  g.nblk = (nnz + g.blk - 1) / g.blk;
  g.ctas = (unsigned)((g.nblk + kCta / 32 - 1) / (kCta / 32));
  return g;
}

// Fixed shapes (KI, G) of each family, for both launches.
#define SEGTACO_SDDMM_SHAPES32(X_) \
  X_(1, 1) X_(1, 2) X_(1, 4) X_(2, 4) X_(2, 8) X_(2, 16) X_(1, 8) X_(1, 16) X_(1, 32)
#define SEGTACO_SDDMM_SHAPES16(X_) \
  X_(1, 1) X_(2, 1) X_(4, 1) X_(4, 2) X_(4, 4) X_(4, 8) X_(4, 16) X_(4, 32)

// Fixed shape of an SDDMM (shared by the single and the multi-problem launch):
// family 1 = fp32 32-byte lanes (V = 8), 2 = bf16 32-byte lanes (V = 16),
// 3 = 16-byte lanes (V = 16 / element size), 0 = the general kernel.
SddmmShape sddmm_shape(int x_dtype, int D, long long ldx, long long ldy, const void *X,
                       const void *Y, int lanes) {
  SddmmShape sh;
  const int esz = x_dtype == SEGTACO_BF16 ? 2 : 4;
  const uintptr_t al = (uintptr_t)X | (uintptr_t)Y;
  int V = 16 / esz;
  while (V > 1 && (D % V != 0 || ldx % V != 0 || ldy % V != 0 || (al % (V * esz)) != 0)) V >>= 1;
  sh.V = V;
  // 32-byte lanes (one ld.global.v8), G >= 4 lanes reading whole 128-byte lines
  // of a row per load instruction (16-byte lanes read each line of Y in two
  // halves, and the kernel is bound by the L1 data pipe); KI <= 2 loads per
  // lane keep the variants within 64 registers.
  const int w32 = 32 / esz;
  if (V * esz == 16 && D % w32 == 0 && ldx % w32 == 0 && ldy % w32 == 0 && (al % 32) == 0) {
    const int T = D / w32;
    if (T >= 1 && T <= 32 && (T & (T - 1)) == 0) {
      sh.family = esz == 4 ? 1 : 2;
      sh.G = T < 4 ? T : (T / 2 > 4 ? T / 2 : 4);
      // A requested lane count with one load per lane, or two from 4 lanes
      // (the compiled shapes); other requests keep the default.
      if (lanes > 0 && (lanes & (lanes - 1)) == 0 && T % lanes == 0 &&
          (T / lanes == 1 || (T / lanes == 2 && lanes >= 4)))
        sh.G = lanes;
      sh.KI = T / sh.G;
      return sh;
    }
  }
  // Sixteen-byte vectors with D / V a power of two up to 128 (KI <= 4 loads).
  if (V * esz == 16 && D % V == 0) {
    const int T = D / V;
    if (T >= 1 && T <= 128 && (T & (T - 1)) == 0) {
      sh.family = 3;
      sh.KI = T < 4 ? T : 4;
      // A requested lane count with four loads per lane (the compiled
      // shapes); other requests keep the default.
      if (lanes > 0 && (lanes & (lanes - 1)) == 0 && T >= 4 && T % lanes == 0 && T / lanes == 4)
        sh.KI = 4;
      sh.G = T / sh.KI;
    }
  }
  return sh;
}

namespace {
// Switch over the family's shapes, each case launching CASE_(XT, V, KI, G).
#define SEGTACO_SDDMM_SWITCH(sh, x_dtype)                                                  \
  switch ((sh).family * 10000 + (sh).KI * 100 + (sh).G) {                                \
    SEGTACO_SDDMM_SHAPES32(SEGTACO_SDDMM_F1) SEGTACO_SDDMM_SHAPES32(SEGTACO_SDDMM_F2)     \
    default:                                                                             \
      if ((sh).family == 3 && (x_dtype) == SEGTACO_BF16) {                               \
        switch ((sh).KI * 100 + (sh).G) {                                                \
          SEGTACO_SDDMM_SHAPES16(SEGTACO_SDDMM_F3B)                                      \
          default: return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no fixed shape");      \
        }                                                                                \
      } else if ((sh).family == 3) {                                                     \
        switch ((sh).KI * 100 + (sh).G) {                                                \
          SEGTACO_SDDMM_SHAPES16(SEGTACO_SDDMM_F3F)                                      \
          default: return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no fixed shape");      \
        }                                                                                \
      } else {                                                                           \
        return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no fixed shape");                 \
      }                                                                                  \
  }
#define SEGTACO_SDDMM_F1(KI_, G_) \
  case 10000 + KI_ * 100 + G_: CASE_(float, 8, KI_, G_) break;
#define SEGTACO_SDDMM_F2(KI_, G_) \
  case 20000 + KI_ * 100 + G_: CASE_(uint16_t, 16, KI_, G_) break;
#define SEGTACO_SDDMM_F3B(KI_, G_) \
  case KI_ * 100 + G_: CASE_(uint16_t, 8, KI_, G_) break;
#define SEGTACO_SDDMM_F3F(KI_, G_) \
  case KI_ * 100 + G_: CASE_(float, 4, KI_, G_) break;

int launch_fixed_single(const SddmmShape &sh, int x_dtype, dim3 grid, int M, long long nnz,
                        const int *row_ptr, const int *col, const float *val, const void *X,
                        const void *Y, long long ldx, long long ldy, float *out, const int *starts,
                        long long nblk, int blk, bool x_first, cudaStream_t s) {
#define CASE_(XT, V, KI, G)                                                                \
  {                                                                                        \
    SddmmGrid b{blk, nblk, grid.x};                                                        \
    if (!starts) b = sddmm_grid<&sddmm_fixed_kernel<XT, V, G, KI>>(nnz, blk);              \
    sddmm_fixed_kernel<XT, V, G, KI><<<b.ctas, kCta, 0, s>>>(                              \
        M, nnz, row_ptr, col, val, static_cast<const XT *>(X), static_cast<const XT *>(Y), ldx, \
        ldy, out, starts, b.nblk, (int)b.blk, x_first);                                    \
  }
  SEGTACO_SDDMM_SWITCH(sh, x_dtype)
#undef CASE_
  return check_launch("sddmm_fixed_kernel");
}

int launch_fixed_multi(const SddmmShape &sh, int x_dtype, dim3 grid, const SddmmProblem *probs,
                       int nprobs, long long total, cudaStream_t s) {
#define CASE_(XT, V, KI, G) \
  sddmm_fixed_multi_kernel<XT, V, G, KI><<<grid, kCta, 0, s>>>(probs, nprobs, total);
  SEGTACO_SDDMM_SWITCH(sh, x_dtype)
#undef CASE_
  return check_launch("sddmm_fixed_multi_kernel");
}

}  // namespace

#define SEGTACO_SDDMM_CASE(XT, V, G)                                                          \
  case V * 100 + G:                                                                           \
    sddmm_kernel<XT, V, G><<<grid, kCta, 0, s>>>(M, nnz, row_ptr, col, val,                   \
                                                 static_cast<const XT *>(X),                  \
                                                 static_cast<const XT *>(Y), ldx, ldy, D, out, \
                                                 starts, nblk, P);                            \
    break;

// Lane shapes (E, C, G) of the default kernel: 32- and 16-byte chunks (bf16: and
// 8-byte ones), one per lane, and one to four 1- or 2-element chunks.
#define SEGTACO_SDDMM_NARROW(X_, XT, E) \
  X_(XT, E, 1, 1) X_(XT, E, 1, 2) X_(XT, E, 1, 4) X_(XT, E, 1, 8) X_(XT, E, 2, 8) X_(XT, E, 3, 8) \
  X_(XT, E, 4, 8) X_(XT, E, 5, 8) X_(XT, E, 3, 16) X_(XT, E, 4, 16) X_(XT, E, 2, 32) X_(XT, E, 3, 32) \
  X_(XT, E, 4, 32)
#define SEGTACO_SDDMM_WIDE(X_, XT, E) \
  X_(XT, E, 1, 1) X_(XT, E, 1, 2) X_(XT, E, 1, 4) X_(XT, E, 1, 8) X_(XT, E, 1, 16) X_(XT, E, 1, 32)
#define SEGTACO_SDDMM_KEY(E, C, G) ((E)*10000 + (C)*100 + (G))
#define SEGTACO_SDDMM_RUN(XT, E, C, G, F)                                                  \
  {                                                                                        \
    const SddmmGrid b = sddmm_grid<&sddmm_gather_kernel<XT, E, C, G, F>>(nnz, P);          \
    sddmm_gather_kernel<XT, E, C, G, F><<<b.ctas, kCta, 0, s>>>(                           \
        M, (unsigned)nnz, row_ptr, col, val, static_cast<const XT *>(X),                   \
        static_cast<const XT *>(Y), (unsigned)(ldx * sizeof(XT)), (unsigned)(ldy * sizeof(XT)), \
        D, out, (unsigned)b.nblk, (unsigned)b.blk, x_first);                               \
  }
#define SEGTACO_SDDMM_NARROW_CASE(XT, E, C, G)  \
  case SEGTACO_SDDMM_KEY(E, C, G):              \
    SEGTACO_SDDMM_RUN(XT, E, C, G, false)       \
    break;
#define SEGTACO_SDDMM_WIDE_CASE(XT, E, C, G)    \
  case SEGTACO_SDDMM_KEY(E, C, G):              \
    if (D == (E) * (C) * (G))                   \
      SEGTACO_SDDMM_RUN(XT, E, C, G, true)      \
    else                                        \
      SEGTACO_SDDMM_RUN(XT, E, C, G, false)     \
    break;

// X and Y from 64 MB on do not stay in L2 beside the pattern, the results and what runs
// between the calls.  Measured on GB300, repeated calls, X normal / leaving first: 90,000
// lognormal rows, D = 128 bf16 (46 MB) 32.0 / 34.3 us; 100,000 power-law rows, D = 64 fp32
// (51 MB) 45 / 49, 100 bf16 (40 MB) 73 / 82; 300,000, D = 64 bf16 (77 MB) 115.6 / 114.2, 32
// fp32 (77 MB) 103.2 / 101.5, 128 bf16 (154 MB) 185 / 180; 90,000 lognormal rows, D = 128 fp32
// (92 MB) 49.4 / 46.3, 400,000 (410 MB) 296 / 290.  (The choice in the kernel costs nothing.)
bool sddmm_x_first(int M, int K, int D, int x_dtype) {
  const long long esz = x_dtype == SEGTACO_BF16 ? 2 : 4;
  return ((long long)M + K) * D * esz > (64LL << 20);
}

bool sddmm_gather_applies(int x_dtype, long long ldx, long long ldy) {
  const int esz = x_dtype == SEGTACO_BF16 ? 2 : 4;
  return ldx * esz < (1LL << 32) && ldy * esz < (1LL << 32);
}

int launch_sddmm_gather(int M, long long nnz, const int *row_ptr, const int *col,
                        const float *val, const void *X, const void *Y, int x_dtype,
                        long long ldx, long long ldy, int D, float *out, int P,
                        bool x_first, cudaStream_t s) {
  const int esz = x_dtype == SEGTACO_BF16 ? 2 : 4;
  const uintptr_t al = (uintptr_t)X | (uintptr_t)Y;
  int E = 32 / esz;
  while (E > 1 && (D % E != 0 || ldx % E != 0 || ldy % E != 0 || (al % (E * esz)) != 0)) E >>= 1;
  // As many lanes as D needs chunks of 16 and 32 bytes; fewer lanes with up to five
  // chunks of 1 and 2 elements each (more nonzeros per step), until a load
  // instruction would touch too many lines.  Measured on GB300, 100,000 lognormal
  // rows (1.2M nonzeros), fp32, 8 / 16 / 32 lanes: D = 17 24.0 / 32.3 / 47.8 us, 37
  // 32.1 / 35.4 / 51.4, 61 57.0 / 39.4 / 51.8, 127 - / 85.3 / 70.0.
  const int n = (D + E - 1) / E;
  int C = 1, G = 1;
  if (E == 4 && esz == 2 && n > 16 && n <= 32) {
    G = 16, C = 2;  // bf16 in 8-byte chunks: D = 100 44 us against 58 with 32 lanes
  } else if (E >= 4 || n <= 8) {
    while (G < 32 && G < n) G <<= 1;
  } else {
    G = n <= 40 ? 8 : n <= 64 && E == 1 ? 16 : 32;
    C = (n + G - 1) / G;
    if (C > 4 && G == 32) C = 4;
  }
  if (x_dtype == SEGTACO_BF16) {
    switch (SEGTACO_SDDMM_KEY(E, C, G)) {
      SEGTACO_SDDMM_WIDE(SEGTACO_SDDMM_WIDE_CASE, uint16_t, 16)
      SEGTACO_SDDMM_WIDE(SEGTACO_SDDMM_WIDE_CASE, uint16_t, 8)
      SEGTACO_SDDMM_WIDE(SEGTACO_SDDMM_NARROW_CASE, uint16_t, 4)
      SEGTACO_SDDMM_NARROW_CASE(uint16_t, 4, 2, 16)
      SEGTACO_SDDMM_NARROW(SEGTACO_SDDMM_NARROW_CASE, uint16_t, 2)
      SEGTACO_SDDMM_NARROW(SEGTACO_SDDMM_NARROW_CASE, uint16_t, 1)
      default:
        return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no bf16 shape E=%d C=%d G=%d", E, C, G);
    }
  } else {
    switch (SEGTACO_SDDMM_KEY(E, C, G)) {
      SEGTACO_SDDMM_WIDE(SEGTACO_SDDMM_WIDE_CASE, float, 8)
      SEGTACO_SDDMM_WIDE(SEGTACO_SDDMM_WIDE_CASE, float, 4)
      SEGTACO_SDDMM_NARROW(SEGTACO_SDDMM_NARROW_CASE, float, 2)
      SEGTACO_SDDMM_NARROW(SEGTACO_SDDMM_NARROW_CASE, float, 1)
      default:
        return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no f32 shape E=%d C=%d G=%d", E, C, G);
    }
  }
  return check_launch("sddmm_gather_kernel");
}

int launch_sddmm(int M, long long nnz, const int *row_ptr, const int *col, const float *val,
                 const void *X, const void *Y, int x_dtype, long long ldx, long long ldy, int D,
                 float *out, int *starts, int P, long long nblk, cudaStream_t s,
                 bool starts_ready, int lanes, int kernel, bool x_first) {
  if (nnz == 0) return SEGTACO_OK;
  if (!starts_ready && starts)
    SEGTACO_TRY(launch_block_starts_canonical(row_ptr, M, P, nblk, starts, s));
  const dim3 grid((unsigned)((nblk + (kCta / 32) - 1) / (kCta / 32)));
  // The fixed-shape kernel where D and the operands allow it (unless the
  // general one is asked for); the general kernel (V-wide vectors, G lanes
  // covering D) otherwise.
  const SddmmShape sh = sddmm_shape(x_dtype, D, ldx, ldy, X, Y, lanes);
  if (sh.family != 0 && kernel != SEGTACO_SDDMM_GENERAL)
    return launch_fixed_single(sh, x_dtype, grid, M, nnz, row_ptr, col, val, X, Y, ldx, ldy, out,
                               starts, nblk, P, x_first, s);
  const int V = sh.V;
  // Lanes per dot product: enough to cover D in one pass, at most 32.
  int G = 1;
  while (G < 32 && G * V < D) G <<= 1;
  if (x_dtype == SEGTACO_BF16) {
    switch (V * 100 + G) {
      SEGTACO_SDDMM_CASE(uint16_t, 8, 1) SEGTACO_SDDMM_CASE(uint16_t, 8, 2)
      SEGTACO_SDDMM_CASE(uint16_t, 8, 4) SEGTACO_SDDMM_CASE(uint16_t, 8, 8)
      SEGTACO_SDDMM_CASE(uint16_t, 8, 16) SEGTACO_SDDMM_CASE(uint16_t, 8, 32)
      SEGTACO_SDDMM_CASE(uint16_t, 4, 1) SEGTACO_SDDMM_CASE(uint16_t, 4, 2)
      SEGTACO_SDDMM_CASE(uint16_t, 4, 4) SEGTACO_SDDMM_CASE(uint16_t, 4, 8)
      SEGTACO_SDDMM_CASE(uint16_t, 4, 16) SEGTACO_SDDMM_CASE(uint16_t, 4, 32)
      SEGTACO_SDDMM_CASE(uint16_t, 2, 1) SEGTACO_SDDMM_CASE(uint16_t, 2, 2)
      SEGTACO_SDDMM_CASE(uint16_t, 2, 4) SEGTACO_SDDMM_CASE(uint16_t, 2, 8)
      SEGTACO_SDDMM_CASE(uint16_t, 2, 16) SEGTACO_SDDMM_CASE(uint16_t, 2, 32)
      SEGTACO_SDDMM_CASE(uint16_t, 1, 1) SEGTACO_SDDMM_CASE(uint16_t, 1, 2)
      SEGTACO_SDDMM_CASE(uint16_t, 1, 4) SEGTACO_SDDMM_CASE(uint16_t, 1, 8)
      SEGTACO_SDDMM_CASE(uint16_t, 1, 16) SEGTACO_SDDMM_CASE(uint16_t, 1, 32)
      default:
        return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no bf16 variant V=%d G=%d", V, G);
    }
  } else {
    switch (V * 100 + G) {
      SEGTACO_SDDMM_CASE(float, 4, 1) SEGTACO_SDDMM_CASE(float, 4, 2)
      SEGTACO_SDDMM_CASE(float, 4, 4) SEGTACO_SDDMM_CASE(float, 4, 8)
      SEGTACO_SDDMM_CASE(float, 4, 16) SEGTACO_SDDMM_CASE(float, 4, 32)
      SEGTACO_SDDMM_CASE(float, 2, 1) SEGTACO_SDDMM_CASE(float, 2, 2)
      SEGTACO_SDDMM_CASE(float, 2, 4) SEGTACO_SDDMM_CASE(float, 2, 8)
      SEGTACO_SDDMM_CASE(float, 2, 16) SEGTACO_SDDMM_CASE(float, 2, 32)
      SEGTACO_SDDMM_CASE(float, 1, 1) SEGTACO_SDDMM_CASE(float, 1, 2)
      SEGTACO_SDDMM_CASE(float, 1, 4) SEGTACO_SDDMM_CASE(float, 1, 8)
      SEGTACO_SDDMM_CASE(float, 1, 16) SEGTACO_SDDMM_CASE(float, 1, 32)
      default:
        return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no f32 variant V=%d G=%d", V, G);
    }
  }
  return check_launch("sddmm_kernel");
}

int launch_sddmm_multi(const SddmmShape &sh, int x_dtype, const SddmmProblem *probs, int nprobs,
                      long long total_blocks, cudaStream_t s) {
  if (total_blocks <= 0 || nprobs <= 0) return SEGTACO_OK;
  if (sh.family == 0) return set_error(SEGTACO_EUNSUPPORTED, "sddmm: no fixed shape to batch");
  const dim3 grid((unsigned)((total_blocks + (kCta / 32) - 1) / (kCta / 32)));
  return launch_fixed_multi(sh, x_dtype, grid, probs, nprobs, total_blocks, s);
}

long long sddmm_block_nnz() { return kSddmmBlock; }

}  // namespace segtaco

// spmm_split.cuh -- the split walk of merge-path chunks: the element-balanced
// SpMM schedules (eb_sr, eb_pr) for products launched alone and in batches.
//
// A warp owns one merge-path chunk (D rows + nonzeros) and one slab of W = G*E*C
// dense columns.  Its lanes form P = 32/G slots, and the chunk's nonzeros are cut
// into P equal runs, one per slot: every slot has the same number of gathers
// whatever the row lengths are, so no slot waits for another's longer row and
// short rows need no batch of their own.  A slot walks its run in storage order, four
// nonzeros a step with their gathers in flight together; terms of a row are summed by
// themselves, four or two at a time, and then added to the row's sum, so that a long row is
// rounded once for them instead of once a term (error against FP64, one chain per row /
// here: 77,777 lognormal rows, N = 37 9.3e-8 / 7.2e-8, N = 128 9.8e-8 / 6.9e-8; 60,000
// power-law rows, N = 64 2.3e-7 / 1.6e-7; 0 to 3 % of the time, rows of 16 1 to 5 %
// faster):
//   * a row that begins and ends in the run is stored as it ends;
//   * the first row end of a run whose row began earlier keeps its partial sum in
//     shared memory, and the row still open at the run's end leaves its sum there
//     too; after the walk each such row is summed from the runs it spans;
//   * a row cut by the chunk's edge is zeroed by the partition kernel and
//     receives one red.global.add from each chunk that holds part of it; every
//     other row is stored once, so C needs no memset.
// The chunk's row ends, column indices and values are staged in shared memory by
// coalesced loads issued together, so that between the partition entry and the
// gathers there is one round trip; a step's four indices are one broadcast
// 16-byte shared load.  A step in which no slot meets a row end (long rows) takes
// the path without checks.
//
// Lane columns: C chunks of E consecutive elements, G*E apart.  C = 1 with 16- or
// 32-byte chunks where N, ldb and the base pointers allow them; otherwise (odd
// N) up to four 1- or 2-element chunks per lane on 8, 16 or 32 lanes, so that one
// pass over A covers up to 128 columns.
//
// What bounds it: the gathers' round trips to L2 (31 warps per SM, 60 % of issue
// slots used, long-scoreboard stalls first; 12.9 TB/s of gathers on 250,000
// power-law rows, N = 64, against ~17 TB/s for bare random 128-byte rows).  Eight
// loads in flight per lane cost registers and L1 and were slower (115 us against
// 104), as were 40 and 48 warps per SM at 48 and 40 registers (122 / 148 us).
// Measured on GB300, partition and product, before (row, flat and sequential
// walks of spmm_kernels.cuh) -> here, fp32 unless noted: 250,000 power-law rows,
// N = 64, eb_sr 184 -> 103 us, eb_pr 120 -> 103; 77,777 lognormal rows (mean 12),
// N = 32 / 64 / 37 / 126 25.2 -> 18.9, 33.5 -> 25.8, 77 -> 26, 102 -> 60 us; 200,000
// rows, N = 64, bf16 84 -> 48; 400,000 rows, N = 128 380 -> 248, N = 127 986 -> 401.
// 1M power-law rows, N = 128: bf16 801 -> 686 us; fp32 keeps the row walk's 8
// columns per lane (1.10 ms against 1.18).
#pragma once

#include <type_traits>

#include "spmm_kernels.cuh"

namespace segtaco {

constexpr int kSplitStep = 4;  // positions per slot and step: one 16-byte index load
template <int N> using Int = std::integral_constant<int, N>;

// Shared memory of one warp, in 4-byte words: the columns and values of the
// chunk's nonzeros (whole steps from a multiple of 4, and one step more), its row
// ends after them -- rows and nonzeros of a chunk are D together -- and the partial
// sums of the runs' first row ends (`head`).  The open sums of the runs reuse the
// columns' and values' space.  What is not shared memory is L1, and the gathers in
// flight need it (D = 256, 36 warps: 96 KB of 256).
template <int V> __host__ __device__ inline int split_head(int D) {
  const int staged = 2 * (D + 3 + 2 * kSplitStep) + 2, open = 32 * V;
  return ((staged > open ? staged : open) + 3) & ~3;
}
template <int V> __host__ __device__ inline int split_words(int D) {
  return split_head<V>(D) + 32 * V;
}

// Edges of a chunk: row and nonzero coordinates of its first and last merge item.
struct ChunkEdges {
  int x0, y0, x1, y1;
};
template <typename BT>
__device__ __forceinline__ ChunkEdges chunk_edges(const SpmmArgs<BT> &a, long long w) {
  return {__ldg(a.part_x + w), __ldg(a.part_y + w), __ldg(a.part_x + w + 1),
          __ldg(a.part_y + w + 1)};
}
// The same without partition arrays: lanes 0-15 search the chunk's first diagonal,
// lanes 16-31 its last, 16 probes a round (the row coordinate is the number of row
// ends r with row_ptr[r + 1] + r + 1 <= d, as in merge_path_x).
template <typename BT>
__device__ __forceinline__ ChunkEdges search_edges(const SpmmArgs<BT> &a, long long w, int D,
                                                  int lane) {
  const unsigned FULL = 0xffffffffu;
  const int l = lane & 15;
  const long long total = (long long)a.M + a.nnz;
  long long d = (w + (lane >> 4)) * (long long)D;
  if (d > total) d = total;
  long long lo = d > a.nnz ? d - a.nnz : 0, hi = d < a.M ? d : a.M;  // lo <= x <= hi
  while (__any_sync(FULL, lo < hi)) {
    // row ends lo .. hi-1 are open; probe l asks for row lo + (l + 1) step - 1
    const long long step = (hi - lo + 15) / 16;
    const long long at = lo + (l + 1) * step - 1;
    const bool past = at >= hi || (long long)__ldg(a.row_ptr + at + 1) + at + 1 > d;
    const unsigned m = (__ballot_sync(FULL, past) >> (lane & 16)) & 0xffffu;
    if (lo < hi) {
      const int f = m ? __ffs(m) - 1 : 16;  // probes 0 .. f-1 have ended
      const long long nhi = lo + (f + 1) * step - 1;
      lo += f * step;
      if (lo > hi) lo = hi;
      if (f < 16 && nhi < hi) hi = nhi;
    }
  }
  const int x = (int)lo, y = (int)(d - lo);
  return {__shfl_sync(FULL, x, 0), __shfl_sync(FULL, y, 0), __shfl_sync(FULL, x, 16),
          __shfl_sync(FULL, y, 16)};
}

// JOIN (rb_pr, spmm_join.cu): chunk w's sums of rows cut by its edges are stored in
// a.piece_part -- two rows of a.piece_ld floats, the row it starts in, then the row
// open at its end -- instead of being added to C.
template <typename BT, int E, int C, int G, bool JOIN = false>
__device__ __forceinline__ void spmm_split_unit(const SpmmArgs<BT> &a, const ChunkEdges ce,
                                                int slab, int lane, int D,
                                                int *__restrict__ sm, long long w = 0) {
  constexpr int P = 32 / G;
  constexpr int V = E * C;
  constexpr int S = kSplitStep;
  static_assert(S == 4, "a step is summed as four terms or two pairs");
  using Dn = Dense<BT, E>;
  const unsigned FULL = 0xffffffffu;
  int *cs = sm;
  float *head = reinterpret_cast<float *>(sm + split_head<V>(D)) + lane * V;
  float *open = reinterpret_cast<float *>(sm);
  const int slot = lane / G, gl = lane & (G - 1);
  const int M = a.M;
  const int col0 = slab * (G * V) + gl * E;
  // chunks of this lane inside N (N is a multiple of E): a prefix
  const int left = a.N - col0;
  const int chunks = left <= 0 ? 0 : imin(C, (left + G * E - 1) / (G * E));
  const uint64_t pol = l2_policy(a.l2_hints);
  // Lanes past N load column 0 and never store.  Strides in bytes fit 32 bits
  // (the planner's condition), so a gather's address is one multiply-add.
  const char *Bc = reinterpret_cast<const char *>(a.B + (left > 0 ? col0 : 0));
  const unsigned ldb = (unsigned)a.ldb * (unsigned)sizeof(BT);
  char *Cc = reinterpret_cast<char *>(a.C + col0);
  const unsigned ldc = (unsigned)a.ldc * 4u;

  const int x0 = ce.x0, y0 = ce.y0, x1 = ce.x1, y1 = ce.y1;
  const int rp0 = x0 < M ? __ldg(a.row_ptr + x0) : y0;
  // Row x0 began in an earlier chunk; row x1 holds nonzeros here and ends later.
  const bool head_split = rp0 < y0;
  const int nrows = x1 - x0;  // rows that end in this chunk
  // Staged positions start at a multiple of 4 (the first y0 - ybase are not
  // ours) and are dealt to the runs in whole steps; the first `extra` runs have
  // one step more than the others.
  const int ybase = y0 & ~(S - 1);
  const int nn = y1 - ybase;
  const int all = y1 > y0 ? (nn + S - 1) / S : 0;
  const int steps = all / P, extra = all - steps * P;
  float *vs = reinterpret_cast<float *>(cs + (all + 1) * S);
  int *re = cs + 2 * (all + 1) * S;  // nrows + 1 of them
  for (int i = lane; i < (all + 1) * S; i += 32) {
    const bool ok = i < nn && ybase + i >= y0;
    cs[i] = ok ? ld_stream(a.col + (ybase + i)) : 0;
    vs[i] = ok ? ld_val(a.val, ybase + i) : 0.0f;
  }
  float acc[V];
  zero<V>(acc);
  auto store = [&](float *dst, bool add) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if (c < chunks) put_c<E>(dst + c * (G * E), acc + c * E, add);
    }
  };
  auto c_row = [&](int r) { return reinterpret_cast<float *>(Cc + (size_t)(unsigned)r * ldc); };
  // Row ends, and zeros for the empty rows (P rows at a time).
  for (int b = 0; b < nrows; b += 32) {
    const int i = b + lane;
    const int e = i < nrows ? __ldg(a.row_ptr + (x0 + i + 1)) : INT_MAX;
    if (i < nrows) re[i] = e;
    int s = __shfl_up_sync(FULL, e, 1);
    if (lane == 0) s = b == 0 ? rp0 : re[b - 1];
    unsigned m = __ballot_sync(FULL, i < nrows && s == e);
    while (m) {
      int at = -1;  // slot k takes the k-th of the next P empty rows
#pragma unroll 1
      for (int k = 0; k < P && m; ++k, m &= m - 1)
        if (k == slot) at = __ffs(m) - 1;
      if (at >= 0) store(c_row(x0 + b + at), false);
    }
    __syncwarp();  // re[b + 31] is read by lane 0 next
  }
  if (lane == 0) re[nrows] = INT_MAX;  // the row open at the chunk's end
  __syncwarp();
  if (all == 0) return;  // only row ends: an edge row's earlier chunks hold its sum

  // The slot's run [lo, hi) and its first row.
  const int p0 = (slot * steps + imin(slot, extra)) * S;
  const int lo = imax(ybase + p0, y0);
  const int hi = imin(ybase + p0 + (steps + (slot < extra ? 1 : 0)) * S, y1);
  int row = 0;  // first row whose end is past lo
  {
    int n = nrows;  // re[nrows] qualifies
    while (n > 0) {
      const int h = n >> 1;
      if (re[row + h] <= lo) {
        row += h + 1;
        n -= h + 1;
      } else {
        n = h;
      }
    }
  }
  int rend = re[row];
  // its row began before the run
  bool first = (row > 0 ? re[row - 1] : rp0) < lo;
  int hrow = -1;  // row whose end this run holds and whose partial sum waits in `head`
  bool ended = false;
  auto flush = [&]() {
    if (first) {
      hrow = row;
      first = false;
#pragma unroll
      for (int v = 0; v < V; ++v) head[v] = acc[v];
    } else {
      store(c_row(x0 + row), false);
    }
    ended = true;
    zero<V>(acc);
  };
  auto next_row = [&](int pos) {
    flush();
    do {  // rows without nonzeros are zeroed already
      rend = re[++row];
    } while (rend <= pos);
  };
  const bool ragged0 = y0 != ybase, ragged1 = (nn & (S - 1)) != 0;
  const int last = steps + (extra > 0 ? 1 : 0);
#pragma unroll 1
  for (int t = 0; t < last; ++t) {
    // a run that has ended reads the step of zeros past the chunk (B row 0)
    const int q = t < steps || slot < extra ? p0 + t * S : all * S;
    const int4 c4 = *reinterpret_cast<const int4 *>(cs + q);
    const int cc[S] = {c4.x, c4.y, c4.z, c4.w};
    typename Dn::raw_t b[S][C];
#pragma unroll
    for (int u = 0; u < S; ++u) {
      const BT *p = reinterpret_cast<const BT *>(Bc + (size_t)(unsigned)cc[u] * ldb);
#pragma unroll
      for (int c = 0; c < C; ++c)
        b[u][c] = C == 1 ? Dn::load(p, pol) : Dn::load_if(p + c * (G * E), pol, c < chunks);
    }
    const float4 v4 = *reinterpret_cast<const float4 *>(vs + q);
    const float vv[S] = {v4.x, v4.y, v4.z, v4.w};
    // acc += the `count` terms from `first` on, summed by themselves
    auto add = [&](auto first, auto count) {
      constexpr int U = decltype(first)::value, K = decltype(count)::value;
#pragma unroll
      for (int c = 0; c < C; ++c)
#pragma unroll
        for (int e = 0; e < E; ++e) {
          if constexpr (K == 1) {
            acc[c * E + e] = fmaf(vv[U], Dn::get(b[U][c], e), acc[c * E + e]);
          } else {
            float x = vv[U] * Dn::get(b[U][c], e);
#pragma unroll
            for (int k = 1; k < K; ++k) x = fmaf(vv[U + k], Dn::get(b[U + k][c], e), x);
            acc[c * E + e] += x;
          }
        }
    };
    const int p = ybase + q;
    auto ends_at = [&](int pos) {  // closes the rows that end there
      if (__any_sync(FULL, pos == rend)) {
        if (pos == rend) next_row(pos);
        __syncwarp();
      }
    };
    if (t == steps || (t == 0 && ragged0) || (t == steps - 1 && ragged1)) {
      // positions outside the chunk, or runs that have ended
      auto one = [&](auto first) {
        constexpr int U = decltype(first)::value;
        if (p + U >= lo && p + U < hi) {
          if (p + U == rend) next_row(p + U);
          add(first, Int<1>());
        }
      };
      one(Int<0>()), one(Int<1>()), one(Int<2>()), one(Int<3>());
      continue;
    }
    if (E <= 4) ends_at(p);
    if (__all_sync(FULL, p + S <= rend)) {  // no row ends in the step
      add(Int<0>(), Int<4>());
    } else if constexpr (E <= 4) {  // two by two, cut where a row ends between them
      auto pair = [&](auto first, auto second) {
        constexpr int U = decltype(first)::value;
        if (U > 0) ends_at(p + U);
        if (__any_sync(FULL, p + U + 1 == rend)) {
          add(first, Int<1>());
          if (p + U + 1 == rend) next_row(p + U + 1);
          __syncwarp();
          add(second, Int<1>());
        } else {
          add(first, Int<2>());
        }
      };
      pair(Int<0>(), Int<1>());
      pair(Int<2>(), Int<3>());
    } else {
      // 8 bf16 elements per lane: one by one.  Two by two 250,000 power-law rows, bf16, N =
      // 64 85 / 89 us, N = 128 144 / 150, for the same error (1.5e-7); lognormal rows
      // 7.9e-8 / 7.3e-8.  All terms of a row kept apart until the step's end: 6.4e-8, but 64
      // registers, and 400,000 lognormal rows, N = 128 158 / 187 us.
      auto one = [&](auto first) {
        ends_at(p + decltype(first)::value);
        add(first, Int<1>());
      };
      one(Int<0>()), one(Int<1>()), one(Int<2>()), one(Int<3>());
    }
  }
  if (lo < hi && rend <= hi) flush();

  // Rows that span runs: the partial sum of the run that holds the row's end plus
  // the open sums of the runs before it, back to the run it began in (the
  // nearest one that holds a row end, or the first).
  __syncwarp();  // columns and values are read
#pragma unroll
  for (int v = 0; v < V; ++v) open[lane * V + v] = acc[v];
  const unsigned ends = __ballot_sync(FULL, ended);
  __syncwarp();
  auto add_open = [&](int s) {  // open sums of runs s, s-1, ... of one row
    for (; s >= 0; --s) {
#pragma unroll
      for (int v = 0; v < V; ++v) acc[v] += open[(s * G + gl) * V + v];
      if ((ends >> (s * G)) & 1) break;
    }
  };
  if (hrow >= 0) {
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = head[v];
    add_open(slot - 1);
    const bool cut = hrow == 0 && head_split;
    store(JOIN && cut ? a.piece_part + 2 * w * a.piece_ld + col0 : c_row(x0 + hrow), !JOIN && cut);
  }
  // The row open at the chunk's end (it ends in a later chunk).
  if (slot == 0 && x1 < M && __ldg(a.row_ptr + x1) < y1) {
    zero<V>(acc);
    add_open(P - 1);
    store(JOIN ? a.piece_part + (2 * w + 1) * a.piece_ld + col0 : c_row(x1), !JOIN);
  }
}

// Warps per SM: 36 at 56 registers, 32 at 64 for several chunks per lane.
template <typename BT, int E, int C, int G> constexpr int split_min_ctas() {
  return (C > 1 ? 32 : 36) / kSpmmWarps;
}

// a.part_x null: the chunk's edges are searched here (and, but for JOIN, C is zero on
// entry).
template <typename BT, int E, int C, int G, bool JOIN = false>
__global__ void __launch_bounds__(kSpmmCta, split_min_ctas<BT, E, C, G>())
    spmm_split_kernel(SpmmArgs<BT> a, int D) {
  extern __shared__ __align__(16) int split_sm[];
  const long long w = (long long)blockIdx.x * kSpmmWarps + threadIdx.x / 32;
  if (w >= a.units) return;  // whole warp leaves together
  const int lane = threadIdx.x & 31;
  const ChunkEdges ce = a.part_x ? chunk_edges(a, w) : search_edges(a, w, D, lane);
  spmm_split_unit<BT, E, C, G, JOIN>(a, ce, blockIdx.y, lane, D,
                                     split_sm + threadIdx.x / 32 * split_words<E * C>(D), w);
}

}  // namespace segtaco

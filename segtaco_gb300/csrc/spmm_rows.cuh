// spmm_rows.cuh -- the row-slot walk of row blocks (rb_sr, rb_pr) whose rows are known to
// be even.
//
// A warp owns a block of R consecutive rows and one slab of W = G*E*C dense columns
// (lanes as in spmm_split.cuh).  Its P = 32/G slots take the block's rows, slot s rows
// s, s + P, ..., each slot on its own: one fmaf chain per column and row in storage
// order, so rb_sr's results are those of the one-slot row walk bit for bit, while P
// rows are in flight instead of one, and 16-byte lanes serve narrow N.  Per round trip
// a slot reads eight column indices and values with its lanes (the next eight, of this
// row or its next one, loading meanwhile) and issues up to eight gathers.
//
// rb_pr (COOP) leaves rows of kCoopRow nonzeros and more to the end, where the whole
// warp takes them one after another, the slots eight nonzeros each in turn, and folds
// the slots' sums.
//
// Rows of a.long_row nonzeros and more are left to the long-row CTAs (spmm_long.cu).
//
// What bounds it: the gathers' round trips while rows are even; with uneven rows the
// slots that wait for the longest one.  Measured figures stand at the planner's rule
// (api.cu).
#pragma once

#include "spmm_split.cuh"

namespace segtaco {

constexpr int kCoopRow = 128;
constexpr int kRowStep = 8;  // nonzeros of a slot per round trip

template <typename BT, int E, int C, int G, bool COOP>
__device__ __forceinline__ void spmm_rows_unit(const SpmmArgs<BT> &a, long long w, int slab,
                                               int lane) {
  constexpr int P = 32 / G;
  constexpr int V = E * C;
  constexpr int S = kRowStep;
  constexpr int L = G >= S ? 1 : S / G;  // indices per lane and round trip
  using Dn = Dense<BT, E>;
  const unsigned FULL = 0xffffffffu;
  const int slot = lane / G, gl = lane & (G - 1);
  const int col0 = slab * (G * V) + gl * E;
  const int left = a.N - col0;
  const int chunks = left <= 0 ? 0 : imin(C, (left + G * E - 1) / (G * E));
  const uint64_t pol = l2_policy(a.l2_hints);
  const char *Bc = reinterpret_cast<const char *>(a.B + (left > 0 ? col0 : 0));
  const unsigned ldb = (unsigned)a.ldb * (unsigned)sizeof(BT);
  char *Cc = reinterpret_cast<char *>(a.C + col0);
  const unsigned ldc = (unsigned)a.ldc * 4u;
  const long long r0 = w * a.rows_per_unit;
  const int R = (int)(a.M - r0 < a.rows_per_unit ? a.M - r0 : a.rows_per_unit);
  // lane l: start and end of row r0 + l (R <= 32)
  const int rs = lane < R ? __ldg(a.row_ptr + (r0 + lane)) : 0;
  const int re = lane < R ? __ldg(a.row_ptr + (r0 + lane + 1)) : 0;
  // rows that the slots leave out
  const bool skip = (a.long_row > 0 && re - rs >= a.long_row) || (COOP && re - rs >= kCoopRow);
  const unsigned slots_rows = __ballot_sync(FULL, lane < R && !skip);
  float acc[V];
  zero<V>(acc);
  auto store = [&](int r) {
    float *dst = reinterpret_cast<float *>(Cc + (size_t)(unsigned)(r0 + r) * ldc);
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (c < chunks) put_c<E>(dst + c * (G * E), acc + c * E, false);
  };
  // (unsigned: a position past the last nonzero stays above it)
  auto load_idx = [&](unsigned p, unsigned end, int(&mc)[L], float(&mv)[L]) {
#pragma unroll
    for (int i = 0; i < L; ++i) {
      const unsigned o = gl + i * G;
      const bool ok = o < S && p < end && o < end - p;
      mc[i] = ok ? ld_stream(a.col + (p + o)) : 0;
      mv[i] = ok ? ld_val(a.val, p + o) : 0.0f;
    }
  };
  // Gathers and multiply-adds of the slot's n (at most S) loaded nonzeros.
  auto walk = [&](int n, const int(&mc)[L], const float(&mv)[L]) {
    typename Dn::raw_t b[S][C];
    float vv[S];
    const bool deep = __any_sync(FULL, n > S / 2);
#pragma unroll
    for (int u = 0; u < S; ++u) {
      if (u < S / 2 || deep) {
        // (lanes of a slot hold its index u at lane u % G; past the row's end: B row 0)
        const int j = __shfl_sync(FULL, mc[u / G < L ? u / G : 0], u & (G - 1), G);
        vv[u] = __shfl_sync(FULL, mv[u / G < L ? u / G : 0], u & (G - 1), G);
        const BT *p = reinterpret_cast<const BT *>(Bc + (size_t)(unsigned)j * ldb);
#pragma unroll
        for (int c = 0; c < C; ++c)
          b[u][c] = C == 1 ? Dn::load(p, pol) : Dn::load_if(p + c * (G * E), pol, c < chunks);
      }
    }
#pragma unroll
    for (int u = 0; u < S; ++u) {
      if (u < n) {
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
          for (int e = 0; e < E; ++e)
            acc[c * E + e] = fmaf(vv[u], Dn::get(b[u][c], e), acc[c * E + e]);
      }
    }
  };
  // ---- one row per slot at a time ----
  // Slot's next row at or after r (r = slot + k P), or R.
  auto next_row = [&](int r) {
    while (r < R && !((slots_rows >> r) & 1u)) r += P;
    return r < R ? r : R;
  };
  int r = next_row(slot);
  int p = __shfl_sync(FULL, rs, r & 31), end = __shfl_sync(FULL, re, r & 31);
  if (r >= R) p = end = 0;
  int mc[L];
  float mv[L];
  load_idx(p, end, mc, mv);
  while (__any_sync(FULL, r < R)) {
    const int n = end - p;
    // where this slot goes on: the row's next nonzeros or its next row
    const bool more = n > S;
    const int nr = more ? r : next_row(r + P);
    int np = __shfl_sync(FULL, rs, nr & 31), nend = __shfl_sync(FULL, re, nr & 31);
    if (more) np = p + S;
    if (nr >= R) np = nend = 0;
    int nc[L];
    float nv[L];
    load_idx(np, nend, nc, nv);
    if (__any_sync(FULL, n > 0)) walk(n, mc, mv);
    if (r < R && !more) {
      store(r);
      zero<V>(acc);
    }
    r = nr;
    p = np;
    end = nend;
#pragma unroll
    for (int i = 0; i < L; ++i) {
      mc[i] = nc[i];
      mv[i] = nv[i];
    }
  }
  // ---- rb_pr's longer rows, the whole warp on each ----
  if constexpr (COOP) {
    unsigned rows = __ballot_sync(FULL, lane < R && re - rs >= kCoopRow &&
                                            !(a.long_row > 0 && re - rs >= a.long_row));
    while (rows) {
      const int rr = __ffs(rows) - 1;
      rows &= rows - 1;
      const unsigned q1 = __shfl_sync(FULL, re, rr);
      unsigned q = __shfl_sync(FULL, rs, rr) + slot * S;
      load_idx(q, q1, mc, mv);
      // (every slot takes part until the row's last nonzero)
      for (unsigned base = q - slot * S; base < q1; base += P * S) {
        int nc[L];
        float nv[L];
        load_idx(q + P * S, q1, nc, nv);
        walk((int)(q1 - q), mc, mv);
        q += P * S;
#pragma unroll
        for (int i = 0; i < L; ++i) {
          mc[i] = nc[i];
          mv[i] = nv[i];
        }
      }
      fold_slots<G, V>(acc);
      if (slot == 0) store(rr);
      zero<V>(acc);
    }
  }
}

template <typename BT, int E, int C, int G, bool COOP>
__global__ void __launch_bounds__(kSpmmCta, 32 / kSpmmWarps) spmm_rows_kernel(SpmmArgs<BT> a) {
  const long long w = (long long)blockIdx.x * kSpmmWarps + threadIdx.x / 32;
  if (w >= a.units) return;  // whole warp leaves together
  spmm_rows_unit<BT, E, C, G, COOP>(a, w, blockIdx.y, threadIdx.x & 31);
}

}  // namespace segtaco

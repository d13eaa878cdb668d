// api.cu -- the extern "C" entry points of include/segtaco.h, argument checks,
// scratch handling and the SpMM planner (schedule / slab width / vector width).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#include "internal.h"

namespace segtaco {

static thread_local std::string g_last_error;

int set_error(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

int check_cuda(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return SEGTACO_OK;
  const int code = (e == cudaErrorMemoryAllocation) ? SEGTACO_ENOMEM : SEGTACO_ECUDA;
  return set_error(code, "%s: %s", what, cudaGetErrorString(e));
}

int check_launch(const char *what) { return check_cuda(cudaGetLastError(), what); }

// One memory pool per device for the scratch of calls that bring no workspace.
// The device's default pool hands everything back to the driver at each
// synchronisation, so a call after one paid for mapping its scratch again:
// measured on GB300, an SpMM of 1000 rows (N = 16) without a workspace took
// 232 us when each call was waited for, 23 us otherwise.  This pool keeps at most
// kScratchKeep bytes across synchronisations (segtaco_taco_release() gives
// them back); the driver makes it safe for several threads and streams.
constexpr unsigned long long kScratchKeep = 64ull << 20;
constexpr int kMaxDevices = 64;
static std::mutex g_scratch_mu;
// A device's pool and the id of the context that it was made in: cudaDeviceReset ends
// both, and the next call makes another.
struct ScratchPool {
  std::atomic<unsigned long long> context{0};
  std::atomic<cudaMemPool_t> pool{nullptr};
};
static ScratchPool g_scratch_pool[kMaxDevices];

// Id of the current context; 0 where there is none.
static unsigned long long context_id() {
  static const auto get = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return reinterpret_cast<PFN_cuCtxGetId_v12000>(p);
  }();
  unsigned long long id = 0;
  return get && get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// The current device's pool; nullptr where there is none (the caller then
// allocates from the default pool).
static cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
  const unsigned long long id = context_id();
  if (id == 0) return nullptr;
  ScratchPool &slot = g_scratch_pool[dev];
  if (slot.context.load(std::memory_order_acquire) == id)
    return slot.pool.load(std::memory_order_relaxed);
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  if (slot.context.load(std::memory_order_acquire) == id)
    return slot.pool.load(std::memory_order_relaxed);
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  unsigned long long keep = kScratchKeep;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  slot.pool.store(pool, std::memory_order_relaxed);
  slot.context.store(id, std::memory_order_release);
  return pool;
}

void trim_scratch_pools() {
  std::lock_guard<std::mutex> lk(g_scratch_mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  for (int d = 0; d < kMaxDevices; ++d) {
    const cudaMemPool_t pool = g_scratch_pool[d].pool.load(std::memory_order_relaxed);
    if (!pool || cudaSetDevice(d) != cudaSuccess) continue;
    if (g_scratch_pool[d].context.load(std::memory_order_acquire) == context_id())
      cudaMemPoolTrimTo(pool, 0);
  }
  cudaSetDevice(dev);
}

Scratch::~Scratch() {
  if (owned_) cudaFreeAsync(owned_, s_);
}

int Scratch::reserve(size_t total) {
  total_ = total;
  used_ = 0;
  if (total == 0) return SEGTACO_OK;
  if (user_) {
    if (cap_ < total)
      return set_error(SEGTACO_EINVAL, "workspace too small: %zu bytes given, %zu needed", cap_,
                       total);
    if (((uintptr_t)user_) & 255)
      return set_error(SEGTACO_EINVAL, "workspace must be 256-byte aligned");
    base_ = static_cast<char *>(user_);
    return SEGTACO_OK;
  }
  // Inside a capture the allocation becomes a node of the graph, which owns it:
  // the default pool, as outside the library.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(s_, &cap) != cudaSuccess) {
    cudaGetLastError();
    cap = cudaStreamCaptureStatusActive;
  }
  cudaMemPool_t pool = cap == cudaStreamCaptureStatusNone ? scratch_pool() : nullptr;
  SEGTACO_TRY(check_cuda(pool ? cudaMallocFromPoolAsync(&owned_, total, pool, s_)
                              : cudaMallocAsync(&owned_, total, s_),
                         "cudaMallocAsync(workspace)"));
  base_ = static_cast<char *>(owned_);
  return SEGTACO_OK;
}

void *Scratch::take(size_t bytes) {
  void *p = base_ + used_;
  used_ += align256(bytes);
  return p;
}

// ---------------------------------------------------------------------------
// SpMM planner
// ---------------------------------------------------------------------------
static bool is_pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

// Products of at most this many elements of C search their chunk edges in the split
// walk's kernel and clear C whole, instead of running the partition kernel: one
// launch and no scratch.  Measured on GB300, partition / search, device time of a
// call: 1000 lognormal rows, N = 16 7.8 / 5.9 us; 10,000, N = 61 18.3 / 9.8; 28,000, N =
// 128 (3.6M elements) 23.6 / 21.9; 200,000 power-law rows, N = 16 (3.2M) 39.9 / 41.4;
// 77,777 rows, N = 128 (10M) 38.2 / 43.2.  An untuned call of 1000 rows from Python 15.5
// -> 10.3 us without the scratch.
constexpr long long kSearchMaxElems = 2LL << 20;
// Merge-path chunks up to this many items take the split walk (a warp stages
// its chunk in shared memory).
constexpr long long kSplitMaxItems = 512;

// The lane shape of the split walk (spmm_split.cuh) for N columns: E elements
// per chunk (the widest load of at most 16 bytes that N, ldb and the pointers
// allow: `fits`), C chunks per lane on G lanes.  False where no shape serves the
// request: explicit narrow lanes, and fp32's 32-byte lanes, whose row walk is the
// faster one for skewed rows over a B beyond L2 (1M x 1M power law, N = 128:
// 1.10 ms against 1.18).
template <typename F>
static bool split_shape(const segtaco_config &c, int N, int K, int esz, F fits, SpmmPlan *plan) {
  const int wide = 16 / esz;  // elements of a 16-byte chunk
  if (c.vec > 0 && (c.vec < wide || (esz == 4 && c.vec > wide))) return false;
  int E = wide;
  while (E > 1 && !fits(E)) E >>= 1;
  // Columns per slab: all of them up to 128, so that A is walked once and a slot's
  // gather brings whole 128-byte lines.  Measured on GB300, lognormal rows (mean
  // 12), fp32, slabs of 32 / 64 / 128 columns: 100,000 rows, N = 128, 71.6 / 56.9
  // / 46.2 us; N = 127 109.9 / 85.3 / 69.7.  fp32 in 16-byte chunks over a B beyond
  // L2: 64 (400,000 rows, N = 128: 258 / 253 / 280 us).
  int cap = 128;
  if (esz == 4 && E == wide && (double)K * N * esz > 96e6) cap = 64;
  if (c.col_tile > 0 && c.col_tile < cap) cap = c.col_tile;
  const int slabs = (N + cap - 1) / cap;
  const int n = ((N + slabs - 1) / slabs + E - 1) / E;  // chunks of a slab
  int C = 1, G;
  if (E >= 4) {
    G = 1;
    while (G < 32 && 2 * G * E <= cap && G < n) G <<= 1;
  } else if (n <= 8) {
    G = 1;
    while (G < n) G <<= 1;
  } else {
    // Several chunks per lane.  More lanes mean fewer 128-byte lines per load
    // instruction and fewer slots: 77,777 rows, N = 37, 8 / 16 / 32 lanes 28.4 /
    // 26.1 / 30.9 us; N = 17 20.4 / 23.1 / 28.3; N = 61 48.1 / 30.5 / 33.0.
    G = n <= 24 ? 8 : n <= 64 && E == 1 ? 16 : 32;
    C = (n + G - 1) / G;
  }
  plan->split_elems = E;
  plan->V = E * C;
  plan->G = G;
  plan->W = G * E * C;
  plan->slabs = (N + plan->W - 1) / plan->W;
  return true;
}

// Whether a configuration asks for rb_pr's joined chunks (spmm_join.cu): depth 8 with
// SEGTACO_FLAG_LONG_ROWS, and from 1M nonzeros on the default threshold (another one asks
// for pieces of the rows it names).
static bool asks_join(const segtaco_config &c, long long nnz) {
  return c.schedule == SEGTACO_RB_PR && nnz > 0 && c.depth == 8 && c.k_parts <= 1 &&
         (c.flags & SEGTACO_FLAG_LONG_ROWS) &&
         !(c.flags & (SEGTACO_FLAG_ROW_WALK | SEGTACO_FLAG_FLAT_WALK)) &&
         (nnz < kLongRowsMinNnz || c.items_per_unit <= 0 || c.items_per_unit == kPieceThreshold);
}
// Where the sums of joined chunks (two rows of C per chunk of up to 512 items) outgrow the
// scratch kept between calls and C's own traffic, the pieces are the faster: rows of 500
// nonzeros, 233,000, N = 128 3.77 ms joined and waited for, 3.12 in pieces (with a workspace
// 3.33 / 3.10); of 1500, 50,000, N = 64 and 256 1.24 / 1.03 and 4.72 / 3.94; of 100, 200,000,
// N = 256 1.38 / 1.31.  Not beyond 256 columns, where the pieces walk A for each 32 of
// them (rows of 500, N = 512 15.3 / 25.7), nor for rows of 20 (400,000, N = 512 1.39 / 2.11).
static bool sums_too_large(int M, long long nnz, int N, double bytes) {
  return nnz >= kLongRowsMinNnz && N <= 256 && nnz > 32LL * M && bytes > (double)kScratchKeep;
}

int plan_spmm(int M, int K, long long nnz, int N, int b_dtype, long long ldb, long long ldc,
              const void *B, const float *C, const segtaco_config *cfg, SpmmPlan *plan,
              LongRowScratch scratch) {
  segtaco_config c{};
  c.schedule = SEGTACO_AUTO;
  if (cfg) c = *cfg;
  const int esz = b_dtype == SEGTACO_BF16 ? 2 : 4;
  // A configuration for joined chunks (below) planned without them: over a B beyond L2
  // the lanes that segtaco_autotune_heuristic chooses for pieces.  Measured on GB300,
  // segtaco_spmm_noalloc, lognormal rows, fp32, 16-byte / 32-byte lanes: 400,000, N = 64
  // 244 / 208 us, 128 526 / 474; 100,000, N = 128 125 / 111.
  if (scratch != LongRowScratch::kJoin && asks_join(c, nnz) && c.vec == 0 && c.col_tile == 0 &&
      (double)K * N * esz > 48e6 && N % (32 / esz) == 0)
    c.vec = 32 / esz;
  // Vector width: the widest 16-byte-or-less load that N, the strides and the
  // base pointers allow, for both the B loads and the C stores.
  // fp32 also takes vec = 8 on request: one 32-byte load per lane.
  int V = c.vec > 0 ? c.vec : 16 / esz;
  if (V > (esz == 2 ? 16 : 8) || !is_pow2(V))
    return set_error(SEGTACO_EINVAL, "vec=%d not in {1,2,4,8} (bf16: up to 16)", c.vec);
  auto fits = [&](int v) {
    const int vc = v < 4 ? v : 4;           // C is stored in float4 pieces
    const int ab = v * esz;                  // one B load of v elements per lane
    return N % v == 0 && ldb % v == 0 && ((uintptr_t)B % ab) == 0 && ldc % vc == 0 &&
           ((uintptr_t)C % (vc * 4)) == 0;
  };
  while (V > 1 && !fits(V)) V >>= 1;
  int schedule = c.schedule;
  // Without row-length statistics the merge path is the safe default: its
  // work per unit is bounded whatever the row-length skew.
  if (schedule == SEGTACO_AUTO) schedule = SEGTACO_EB_PR;
  if (schedule < SEGTACO_RB_SR || schedule > SEGTACO_EB_PR)
    return set_error(SEGTACO_EINVAL, "unknown schedule %d", schedule);
  // The slot walk keeps every row of a chunk in one slot, in storage order,
  // so eb_sr may use several slots there; elsewhere a sequential schedule is
  // one slot of 32 lanes.
  const bool slot_walk = (c.flags & SEGTACO_FLAG_SLOT_WALK) &&
                         (schedule == SEGTACO_EB_SR || schedule == SEGTACO_EB_PR);
  const bool sequential = (schedule == SEGTACO_RB_SR || schedule == SEGTACO_EB_SR) && !slot_walk;
  // Slab width W = G*V columns.  Sequential schedules use one slot (G = 32);
  // parallel ones use P = 32/G >= 2 slots, by default a 128-byte B segment per
  // nonzero (32 fp32 / 64 bf16 columns).
  int G;
  // 16-element (32-byte bf16) lanes exist for G <= 4 only: the sequential
  // schedules (G = 32) take at most 8.
  if (sequential && V > 8) V = 8;
  if (sequential) {
    G = 32;
    if (c.col_tile > 0 && c.vec <= 0) {
      // A requested slab width picks the vector width (W = 32*V).
      while (V > 1 && 32 * V > c.col_tile) V >>= 1;
    }
    // No idle half-slab: N = 32 takes one column per lane, not 8 lanes of 4.
    if (c.vec <= 0)
      while (V > 1 && 32 * (V / 2) >= N) V >>= 1;
  } else {
    int W = c.col_tile > 0 ? c.col_tile : 128 / esz;
    if (V > 8 && W / V > 4) V = 8;  // 16-element lanes: G <= 4
    G = W / V;
    if (G < 1) G = 1;
    if (G > 16) G = 16;
    while (!is_pow2(G)) --G;
    while (G > 1 && (G / 2) * V >= N) G >>= 1;  // no idle half-slots
  }
  const int W = G * V;
  plan->schedule = schedule;
  plan->V = V;
  plan->G = G;
  plan->W = W;
  plan->slabs = (N + W - 1) / W;
  plan->l2_hints = (c.flags & SEGTACO_FLAG_L2_HINTS) != 0;
  // TMA bulk copies need 16-byte lane vectors and 16-byte aligned segments
  // (V == 16/esz already implies N, ldb and B are multiples / aligned).
  plan->use_tma = (c.flags & SEGTACO_FLAG_SMEM_RING) && V * esz == 16;
  plan->bulk_copies = (c.flags & SEGTACO_FLAG_TMA_BULK) != 0;
  if (c.depth != 0 && c.depth != 4 && c.depth != 8)
    return set_error(SEGTACO_EINVAL, "depth=%d not in {0, 4, 8}", c.depth);
  plan->deep = c.depth == 8;
  // Walk, where neither the split walk nor row slots nor joined chunks apply (below):
  // the flat walk by default for eb_sr (one slot over merge-path chunks:
  // short rows share a batch of 32 nonzeros instead of a round trip each;
  // measured on GB300 1.44 vs 1.53 ms on the 1M x 1M power-law SpMM), the row
  // walk everywhere else (rb units are too small to amortise the flat walk's
  // per-unit setup, and with several slots its flush bookkeeping costs more
  // instructions than the row walk); the flags force either.  Walks other
  // than the 4-load row walk exist for sixteen-byte vectors only.
  const bool wide = V * esz == 16;
  if ((c.flags & SEGTACO_FLAG_ROW_WALK) && (c.flags & SEGTACO_FLAG_FLAT_WALK))
    return set_error(SEGTACO_EINVAL, "ROW_WALK and FLAT_WALK are exclusive");
  const bool flat = wide && ((c.flags & SEGTACO_FLAG_FLAT_WALK) ||
                             (schedule == SEGTACO_EB_SR && G == 32 &&
                              !(c.flags & SEGTACO_FLAG_ROW_WALK)));
  plan->walk = flat ? 2 : (plan->deep && wide ? 1 : 0);
  // The slot walk (every slot its own merge-path chunk) on request, for the
  // element-balanced schedules and the lane shapes it is compiled for.
  const bool eb = schedule == SEGTACO_EB_SR || schedule == SEGTACO_EB_PR;
  if ((c.flags & SEGTACO_FLAG_SLOT_WALK) && eb && !plan->use_tma) {
    const int k = V * 100 + G;
    const bool ok = esz == 4 ? (k == 804 || k == 408 || k == 808 || k == 404 || k == 416 ||
                                k == 101)
                             : (k == 1604 || k == 804 || k == 808);
    if (ok) plan->walk = 3;
  }
  // eb_sr with 8-byte lanes (bf16 over 128-column slabs, fp32 over 64): the
  // sequential walk with staged indices (spmm_seq_unit), unless a walk is
  // forced.
  if (schedule == SEGTACO_EB_SR && G == 32 && !plan->use_tma && plan->walk == 0 &&
      !(c.flags & (SEGTACO_FLAG_ROW_WALK | SEGTACO_FLAG_FLAT_WALK)) && V * esz == 8)
    plan->walk = 4;
  plan->rows_per_unit = c.rows_per_unit > 0 ? c.rows_per_unit : 1;
  plan->items_per_unit = 0;
  plan->nchunks = (M + plan->rows_per_unit - 1) / plan->rows_per_unit;  // rb: row blocks
  plan->workspace = 0;
  plan->long_row = 0;
  plan->piece_len = 0;
  plan->piece_parts = 1;
  plan->px_entries = plan->py_entries = 0;
  if (schedule == SEGTACO_EB_SR || schedule == SEGTACO_EB_PR) {
    // merge-path items per chunk: one chunk per warp (512, fewer for small
    // products), or per slot in the slot walk (64, so a warp still covers
    // about 512)
    long long D = c.items_per_unit > 0   ? c.items_per_unit
                  : plan->walk == 3 ? 64
                                    : default_chunk_items(M, nnz);
    if (D < 1) D = 1;
    const long long total = (long long)M + nnz;
    long long nch = (total + D - 1) / D;
    if (nch < 1) nch = 1;
    plan->items_per_unit = D;
    plan->nchunks = nch;
    plan->px_entries = plan->py_entries = nch + 1;
  } else if (nnz >= kLongRowsMinNnz && (c.flags & SEGTACO_FLAG_LONG_ROWS) &&
             plan->walk != 2 && !plan->use_tma) {
    const int epc = 16 / esz;
    if (schedule == SEGTACO_RB_PR && scratch != LongRowScratch::kList) {
      // rb_pr: long rows as pieces of kPieceLen nonzeros in the row-block
      // launch (spmm_long.cu), over the same column slabs; rows from
      // kPieceThreshold nonzeros by default.
      long long T = c.items_per_unit > 0 ? c.items_per_unit : kPieceThreshold;
      if (T > nnz) T = nnz;
      plan->long_row = (int)T;
      // passes over ranges of B's rows (a launch of their own before the row
      // blocks) on request
      int parts = c.k_parts > 0 ? c.k_parts : 1;
      if (parts > kMaxPieceParts) parts = kMaxPieceParts;
      if (parts > K) parts = K > 0 ? K : 1;
      plan->piece_parts = parts;
      plan->piece_len = (int)(parts > 1 ? kPassPieceLen : kPieceLen);
      plan->px_entries = piece_layout(nnz, T, plan->piece_len, plan->slabs, W, parts).entries;
      plan->py_entries = 4;  // the count
    } else if (N % epc == 0 && ldb % epc == 0 && ((uintptr_t)B % 16) == 0) {
      // Long rows to CTAs of their own (spmm_long.cu): their ring copies
      // 16-byte chunks of B rows, so B, ldb and N must allow 16-byte pieces.
      long long T = long_row_threshold(c);
      if (T > nnz) T = nnz;
      long long hi, lo;
      long_list_caps(nnz, T, &hi, &lo);
      plan->long_row = (int)T;
      plan->px_entries = hi + lo;
      plan->py_entries = 4;  // the two parts' counts, 64-bit work queue
    }
  }
  // Merge-path chunks take the split walk unless another walk or a chunk beyond
  // its staging is asked for.
  if (eb && !plan->use_tma && plan->walk != 3 && plan->items_per_unit <= kSplitMaxItems &&
      !(c.flags & (SEGTACO_FLAG_ROW_WALK | SEGTACO_FLAG_FLAT_WALK)) && c.depth != 8 &&
      ldb * esz < (1LL << 32) && ldc * 4 < (1LL << 32) &&
      split_shape(c, N, K, esz, fits, plan))
    plan->walk = kWalkSplit;
  plan->window_halo = -1;
  plan->band_halo = -1;
  if ((c.flags & SEGTACO_FLAG_WINDOW) && schedule == SEGTACO_RB_PR && plan->long_row == 0 &&
      !plan->use_tma && nnz > 0 && K > 0 && N >= 64 && N % 16 == 0 &&
      ((uintptr_t)B % 16) == 0 && (ldb * esz) % 16 == 0 && ((uintptr_t)C % 16) == 0 &&
      ldc % 4 == 0) {
    // rb_pr on a banded matrix: 32-row blocks with the band of A as a dense
    // tile and B's window of 32 + 2H rows by TMA (spmm_band_kernel).
    const long long H = c.items_per_unit > 0 ? c.items_per_unit : 32;
    if (32 + 2 * H <= 256) plan->band_halo = (int)H;
  }
  if ((c.flags & SEGTACO_FLAG_WINDOW) && plan->band_halo < 0 && plan->long_row == 0 &&
      !plan->use_tma && nnz > 0 && K > 0 &&
      (schedule == SEGTACO_RB_SR || schedule == SEGTACO_RB_PR) && plan->walk != 2) {
    // TMA needs B 16-byte aligned and its row pitch a multiple of 16 bytes;
    // the window's rows (4 per-warp row blocks plus two halos) fit one box.
    const long long H = c.items_per_unit > 0 ? c.items_per_unit : 32;
    const long long wrows = 4 * plan->rows_per_unit + 2 * H;
    if (((uintptr_t)B % 16) == 0 && (ldb * esz) % 16 == 0 && wrows <= 256 &&
        (size_t)wrows * W * esz <= 60 * 1024 && window_variant_exists(b_dtype, V, G))
      plan->window_halo = (int)H;
  }
  // Row blocks of rows known to be even (depth 4, which segtaco_autotune_heuristic sets
  // for them) without pieces, band or window take the row-slot walk (spmm_rows.cuh)
  // where a warp holds at least two rows side by side, or the operands allow only 1- or
  // 2-element lanes.  Measured on GB300, fp32, row walk / row-slot walk: 16,384 rows of
  // 16, N = 32, rb_sr 9.4 / 4.3 us, rb_pr 8.6 / 4.5; 300,000, N = 16 rb_sr 117 / 30; N = 64
  // 150 / 97; 20,000 banded rows, N = 37 47 / 26.  Uneven rows keep the row walk: a
  // slot's trips through a long row cost more instructions than a whole warp's (20,000
  // power-law rows, N = 37, rb_sr 309 / 937 us).  rb_pr's row walk also splits rows of
  // more than 32 nonzeros over its slots (50,000 banded rows of 73, N = 32: 29.8 us against
  // 31.1, N = 16 bf16 23.3 / 27.8; rb_sr 56 / 31).
  if ((schedule == SEGTACO_RB_SR || schedule == SEGTACO_RB_PR) && c.depth == 4 &&
      !plan->use_tma && plan->piece_len == 0 && plan->band_halo < 0 && plan->window_halo < 0 &&
      !(c.flags & (SEGTACO_FLAG_ROW_WALK | SEGTACO_FLAG_FLAT_WALK)) &&
      ldb * esz < (1LL << 32) && ldc * 4 < (1LL << 32)) {
    segtaco_config rc = c;
    if (rc.vec >= 16 / esz) rc.vec = 0;  // (wider lanes: the 16-byte ones)
    SpmmPlan t = *plan;
    if (split_shape(rc, N, K, esz, fits, &t) &&
        (t.split_elems <= 2 ||
         (t.G < 32 && (schedule == SEGTACO_RB_SR || nnz <= 32LL * M)))) {
      *plan = t;
      plan->walk = kWalkRowSlots;
      const int P = 32 / t.G;
      int rows = P;  // up to four rows per slot, while the warps fill two waves
      while (2 * rows <= 32 && rows < 4 * P && M / (2 * rows) >= 2 * 152 * 32) rows *= 2;
      plan->rows_per_unit = rows;
      plan->nchunks = (M + rows - 1) / rows;
    }
  }
  // rb_pr over rows known to be uneven (asks_join, as segtaco_autotune_heuristic sets for
  // them): merge-path chunks whose sums of cut rows are added in order (spmm_join.cu)
  // instead of pieces and row blocks.  fp32's explicit 32-byte lanes (split_shape) and
  // passes over B keep the pieces.
  if (scratch == LongRowScratch::kJoin && asks_join(c, nnz) && !plan->use_tma &&
      plan->band_halo < 0 && plan->window_halo < 0) {
    SpmmPlan t = *plan;
    if (split_shape(c, N, K, esz, fits, &t)) {
      t.walk = kWalkSplitJoin;
      t.long_row = t.piece_len = 0;
      t.piece_parts = 1;
      t.items_per_unit = default_chunk_items(M, nnz);
      t.nchunks = (M + nnz + t.items_per_unit - 1) / t.items_per_unit;
      t.px_entries = 2 * t.nchunks * (((long long)N + 3) & ~3LL);
      t.py_entries = 0;
      if (ldb * esz >= (1LL << 32) || ldc * 4 >= (1LL << 32) ||
          sums_too_large(M, nnz, N, t.px_entries * 4.0))
        return plan_spmm(M, K, nnz, N, b_dtype, ldb, ldc, B, C, cfg, plan,
                         LongRowScratch::kPieces);
      *plan = t;
    }
  }
  if (plan->px_entries)
    plan->workspace = align256((size_t)plan->px_entries * sizeof(int)) +
                      align256((size_t)plan->py_entries * sizeof(int));
  return SEGTACO_OK;
}

int run_spmm_planned(const SpmmPlan &plan, int M, int K, long long nnz, const int *row_ptr,
                     const int *col, const float *vals, const void *B, int b_dtype, long long ldb,
                     float *C, long long ldc, int N, int *px, int *py, cudaStream_t s,
                     bool partition_ready) {
  if (M == 0 || N == 0) return SEGTACO_OK;
  SpmmLaunch L;
  L.dtype = b_dtype;
  L.V = plan.V;
  L.G = plan.G;
  L.l2_hints = plan.l2_hints;
  L.M = M;
  L.K = K;
  L.N = N;
  L.nnz = nnz;
  L.row_ptr = row_ptr;
  L.col = col;
  L.val = vals;
  L.B = B;
  L.ldb = ldb;
  L.C = C;
  L.ldc = ldc;
  L.part_x = px;
  L.part_y = py;
  L.units = plan.nchunks;
  L.rows_per_unit = (int)plan.rows_per_unit;
  L.use_tma = plan.use_tma;
  L.bulk_copies = plan.bulk_copies;
  L.deep = plan.deep;
  L.walk = plan.walk;
  L.no_fork = plan.no_fork;
  L.split_elems = plan.split_elems;
  L.coop = plan.schedule == SEGTACO_RB_PR;
  L.window_halo = plan.window_halo;
  L.band_halo = plan.band_halo;
  const bool bf16 = b_dtype == SEGTACO_BF16;
  switch (plan.schedule) {
    case SEGTACO_RB_SR:
    case SEGTACO_RB_PR:
      if (L.use_tma) return bf16 ? launch_spmm_tma_bf16(L, true, s) : launch_spmm_tma_f32(L, true, s);
      if (plan.band_halo >= 0) return launch_spmm_band(L, s);
      if (plan.window_halo >= 0) return launch_spmm_window(L, s);
      if (plan.walk == kWalkSplitJoin) {
        L.part_x = L.part_y = nullptr;  // the edges are searched in the kernels
        L.split_items = (int)plan.items_per_unit;
        L.piece_part = reinterpret_cast<float *>(px);
        L.piece_ld = ((long long)N + 3) & ~3LL;
        SEGTACO_TRY(bf16 ? launch_spmm_join_bf16(L, s) : launch_spmm_join_f32(L, s));
        return launch_spmm_join(L, s);
      }
      if (plan.long_row > 0 && plan.piece_len > 0) {
        L.long_row = plan.long_row;
        if (!partition_ready)
          SEGTACO_TRY(launch_long_pieces_list(row_ptr, M, nnz, plan.long_row, plan.piece_len,
                                              plan.slabs, plan.W, plan.piece_parts, px, py, s));
        const PieceLayout pl = piece_layout(nnz, plan.long_row, plan.piece_len, plan.slabs,
                                            plan.W, plan.piece_parts);
        L.piece_len = plan.piece_len;
        L.pieces = px;
        L.piece_count = py;
        L.piece_ctr = reinterpret_cast<unsigned *>(px + pl.ctr);
        L.piece_part = reinterpret_cast<float *>(px + pl.part);
        L.piece_cap = pl.cap;
        L.piece_multi = pl.multi;
        L.piece_ld = pl.ld;
        L.piece_parts = plan.piece_parts;
        // count[2..3]: the passes' work counter (the count array is 256-byte aligned)
        L.piece_queue = reinterpret_cast<unsigned long long *>(py + 2);
        if (plan.piece_parts > 1) {
          // the pieces' passes, then the row blocks of the short rows alone
          SEGTACO_TRY(bf16 ? launch_spmm_pieces_bf16(L, s) : launch_spmm_pieces_f32(L, s));
          L.piece_len = 0;
          L.piece_cap = 0;
        }
        return bf16 ? launch_spmm_bf16_rows(L, s) : launch_spmm_f32_rows(L, s);
      }
      if (plan.long_row > 0) {
        L.long_row = plan.long_row;
        if (!partition_ready)
          SEGTACO_TRY(launch_long_rows_list(row_ptr, M, nnz, plan.long_row, px, py, s));
        return launch_spmm_long_rows(L, px, py, s);
      }
      return bf16 ? launch_spmm_bf16_rows(L, s) : launch_spmm_f32_rows(L, s);
    case SEGTACO_EB_SR:
    case SEGTACO_EB_PR:
      if (px == nullptr)  // no partition arrays: rows cut by a chunk edge are added to zeros
        SEGTACO_TRY(check_cuda(
            ldc == N ? cudaMemsetAsync(C, 0, (size_t)M * N * sizeof(float), s)
                     : cudaMemset2DAsync(C, ldc * sizeof(float), 0, N * sizeof(float), M, s),
            "clearing C"));
      else if (!partition_ready)
        SEGTACO_TRY(launch_merge_path(row_ptr, M, nnz, plan.items_per_unit, plan.nchunks, px, py,
                                      C, ldc, N, s));
      if (L.use_tma) return bf16 ? launch_spmm_tma_bf16(L, false, s) : launch_spmm_tma_f32(L, false, s);
      if (plan.walk == kWalkSplit) {
        L.split_items = (int)plan.items_per_unit;
        return bf16 ? launch_spmm_split_bf16(L, s) : launch_spmm_split_f32(L, s);
      }
      return bf16 ? launch_spmm_bf16_chunks(L, s) : launch_spmm_f32_chunks(L, s);
    default:
      return set_error(SEGTACO_EINVAL, "unknown schedule %d", plan.schedule);
  }
}

long long sddmm_block_nnz();

// Host-side checks of the CSR arguments; `need_col` is false for the calls
// that only read row_ptr (partitions, row ids).
static int check_csr_args(int M, int K, long long nnz, const int *row_ptr, const int *col,
                          bool need_col = true) {
  if (M < 0 || K < 0 || nnz < 0) return set_error(SEGTACO_EINVAL, "negative size");
  if (nnz > 0x7fffffffLL) return set_error(SEGTACO_EINVAL, "nnz exceeds int32 indices");
  if (M > 0 && row_ptr == nullptr) return set_error(SEGTACO_EINVAL, "row_ptr is NULL");
  if (need_col && nnz > 0 && col == nullptr) return set_error(SEGTACO_EINVAL, "col is NULL");
  return SEGTACO_OK;
}

}  // namespace segtaco

using namespace segtaco;

extern "C" {

const char *segtaco_version(void) { return "segtaco-gb300 0.1 (sm_103a)"; }

const char *segtaco_last_error(void) { return g_last_error.c_str(); }

int segtaco_device_available(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n > 0 ? 1 : 0;
}

int segtaco_autotune_heuristic(int32_t M, int32_t K, int64_t nnz, int32_t N, int32_t b_dtype,
                               int64_t max_row_len, segtaco_config *cfg) {
  if (!cfg) return set_error(SEGTACO_EINVAL, "cfg is NULL");
  const int requested = cfg->schedule;
  const bool banded = (cfg->flags & SEGTACO_FLAG_WINDOW) != 0;
  memset(cfg, 0, sizeof(*cfg));
  const double mean = M > 0 ? (double)nnz / M : 0.0;
  // Row-balanced when rows are short and even; merge path otherwise.
  const bool even = max_row_len >= 0 && mean > 0.0 && (double)max_row_len <= 4.0 * mean + 8.0;
  const int schedule = (requested >= SEGTACO_RB_SR && requested <= SEGTACO_EB_PR)
                           ? requested
                           : (even ? SEGTACO_RB_PR : SEGTACO_EB_PR);
  cfg->schedule = schedule;
  const int esz = b_dtype == SEGTACO_BF16 ? 2 : 4;
  const bool sequential = schedule == SEGTACO_RB_SR || schedule == SEGTACO_EB_SR;
  // Column slab: the B slab should stay in L2 (measured on GB300: 128-byte
  // segments for the parallel schedules; the sequential ones take 16-byte
  // vectors on all 32 lanes).  A B that fits L2 whole is one slab.
  const double bbytes = (double)K * N * esz;
  const bool skewed = mean > 0.0 && (double)max_row_len > 8.0 * mean;
  if (sequential) {
    // The narrowest lanes that still cover N in one slab (N = 32: one column
    // per lane, all 32 lanes busy; measured on GB300, 16,384^2 with 16
    // nonzeros per row, N = 32: 16-byte lanes left 24 of 32 lanes idle).
    int v = 16 / esz;
    while (v > 1 && 32 * (v / 2) >= N) v >>= 1;
    cfg->col_tile = 32 * v;
  } else
    cfg->col_tile = bbytes <= 48e6 ? (N <= 64 * 4 / esz ? N : 64 * 4 / esz) : 128 / esz;
  // Row-block schedules from 1M nonzeros whose longest row reaches the
  // long-row threshold hand those rows to CTAs of their own (spmm_long.cu;
  // without row statistics they stay in the row-block kernel: the long-row
  // launch costs its L1 carveout, banded 262,144 rows N = 64 rb_pr 0.344 ->
  // 0.435 ms).  rb_sr's row-block kernel then takes 128-column slabs also for
  // bf16 (8-byte lanes).  Measured on GB300, 1M x 1M power law, N = 128:
  // fp32 2.32 ms (64-column slabs: 2.45), bf16 2.29 ms (256: 2.52).
  const bool long_rows =
      (schedule == SEGTACO_RB_SR || schedule == SEGTACO_RB_PR) && nnz >= kLongRowsMinNnz &&
      max_row_len >= (schedule == SEGTACO_RB_PR ? kPieceThreshold : kLongRowDefault);
  if (schedule == SEGTACO_RB_SR && long_rows) cfg->col_tile = 128;
  // fp32 with B beyond L2 (32-column slabs): 8 columns per lane (one 32-byte
  // load, 4 lanes per 128-byte segment, 8 slots), so a warp step covers 8 rows
  // or 8 nonzeros instead of 4.  Measured on GB300: 1M x 1M power law (skewed
  // rows), N = 128, eb_pr 1.33 -> 1.15 ms, rb_pr 2.84 -> 2.49 ms; banded
  // 262,144 rows (even rows, 19M nonzeros), N = 64, rb_pr 0.368 -> 0.344 ms.
  // Even rows with few nonzeros keep 4 (the 256-matrix pool, products of at
  // most a few million nonzeros, 3.74 -> 3.87 ms with 8); with B in L2
  // (64-column slabs: 8 lanes per slot, 24 warps per SM) the pool lost more
  // (4.38 ms).
  if (!sequential && esz == 4 && bbytes > 48e6 && N % 8 == 0 && (skewed || nnz >= 4000000))
    cfg->vec = 8;
  // eb_pr takes the split walk with the planner's lanes (spmm_split.cuh) instead,
  // unless most nonzeros are in long rows (a longest row of 256 means and more)
  // over a B beyond L2.  Measured on GB300, N = 128, fp32, 8 columns per lane /
  // split walk: 1M power-law rows 1.10 / 1.18 ms, 400,000 349 / 365 us; 400,000
  // lognormal rows (longest 64 means) 380 / 250 us; B in L2 (250,000 power-law rows,
  // N = 64) 120 / 105.
  const bool heavy = (double)max_row_len > 256.0 * mean && bbytes > 96e6;
  const bool split = schedule == SEGTACO_EB_PR && !(heavy && N % (32 / esz) == 0);
  // rb_pr takes chunks whose cut rows are joined (spmm_join.cu) from the same longest
  // rows as the pieces, and below 1M nonzeros from 640, with the same exception for
  // fp32.  Measured on GB300, row walk / joined chunks (longest row): 1000 power-law
  // rows, N = 16 8.2 / 9.3 us (513), 1473, N = 114 26.0 / 11.7 (1267), 17,801, N = 97 679 / 38
  // (26,528); lognormal rows, N = 64, 3000 8.6 / 10.9 (209), 80,000 39.6 / 31.4 (796).
  // Pieces / joined chunks, power-law rows: 60,000, N = 64 108 / 45, 400,000, N = 37 432 /
  // 183, N = 128 372 / 420 fp32 and 301 / 274 bf16; 400,000 lognormal rows, N = 128 395 / 278.
  const bool join = schedule == SEGTACO_RB_PR && !even && !(heavy && esz == 4 && N % 8 == 0) &&
                    (long_rows || (nnz < kLongRowsMinNnz && max_row_len >= kJoinRow &&
                                   !(banded && N >= 64 && N % 16 == 0)));
  // A B that fits L2 whole (up to ~96 MB) under a large product: one slab of
  // up to 64 columns (8 per lane, G = 8), so A is read once.  Measured on
  // GB300, banded 262,144 rows (19.1M nonzeros), N = 64, rb_pr: 0.248 ms
  // against 0.323 ms with two 32-column slabs.
  if (!sequential && esz == 4 && bbytes > 48e6 && bbytes <= 96e6 && nnz >= 4000000 &&
      N % 8 == 0 && !skewed)
    cfg->col_tile = N < 64 ? N : 64;
  // bf16 likewise: 16 columns per lane (one 32-byte load) on 64-column slabs.
  // Measured on GB300: 1M x 1M power law, N = 128, eb_pr 0.996 -> 0.823 ms;
  // with B in L2 (banded, N = 64) 8 stays faster (0.224 vs 0.235 ms).
  if (!sequential && esz == 2 && bbytes > 48e6 && N % 16 == 0 && (skewed || nnz >= 4000000))
    cfg->vec = 16;
  // (joined chunks: a slab for the pieces that may take their place, where it covers N and
  // so changes nothing for the chunks.  segtaco_spmm_noalloc, 100,000 lognormal rows, 32
  // fp32 / 64 bf16 columns against 64 / 128: N = 64 fp32 65 / 55 us, N = 128 bf16 88 / 70;
  // 60,000 power-law rows, N = 64 67 / 108.)
  const bool piece_tile = join && !((double)max_row_len > 256.0 * mean) && N <= 256 / esz &&
                          bbytes <= 48e6;
  if (split || join) cfg->vec = 0;
  if (split || join) cfg->col_tile = piece_tile ? 256 / esz : 0;
  // eb: merge-path items per chunk; rb: the long-row threshold.
  cfg->items_per_unit = (schedule == SEGTACO_RB_SR || schedule == SEGTACO_RB_PR)
                            ? (int)kLongRowDefault
                            : (int)default_chunk_items(M, nnz);
  cfg->rows_per_unit = schedule == SEGTACO_RB_PR || schedule == SEGTACO_RB_SR ? 4 : 1;
  // rb_sr walks its rows one after another in one slot: fewer rows per warp
  // while the rows are few.  Measured on GB300, 16,384 x 16,384 with 16
  // nonzeros per row, N = 32: 0.0174 ms with 4 rows, 0.0154 with 2.
  if (schedule == SEGTACO_RB_SR)
    while (cfg->rows_per_unit > 1 && M / cfg->rows_per_unit < 8192) cfg->rows_per_unit >>= 1;
  // rb: 8 loads in flight in the row walk, or (4) even rows side by side.
  // (rb_pr's rows of more than 32 nonzeros in 16-byte lanes stay with the row walk;
  // 8 with long rows would ask for joined chunks, even rows keep the pieces.  Even rows
  // of rb_sr that fill the lanes, fp32 beyond 64 columns, get the row walk with 4 loads: 8
  // / 4 loads, rows of 16, N = 96 and 128, 16,384 10.8 / 10.2 and 11.0 / 10.7 us, 100,000
  // 50.7 / 49.7 and 54.7 / 54.7; 100,000 banded rows of 73 175 / 168 and 179 / 168.)
  const bool side_by_side =
      even &&
      (schedule == SEGTACO_RB_SR || nnz <= 32LL * M || N % (16 / esz) != 0 || long_rows);
  cfg->depth = (schedule == SEGTACO_RB_SR || schedule == SEGTACO_RB_PR) && !side_by_side ? 8 : 4;
  cfg->flags = long_rows || join ? SEGTACO_FLAG_LONG_ROWS : 0;
  // rb_pr's long rows as pieces of the row-block launch (rows of >= 512
  // nonzeros, pieces of 4096); the rows left are short, so a warp takes 64 of
  // them to fill its slots (32 while that leaves fewer than 8192 warps).
  // Measured on GB300, 1M x 1M power law, N = 128: 1.69 ms with the long-row
  // CTAs (threshold 2048, 4 rows per warp), 1.58 with pieces of 512, 1.22
  // with 32 rows per warp (2 rows: 2.01); pieces of 4096: 1.119 ms with 32
  // rows, 1.114 with 64 (the 10M-nonzero Zipf 1.922 matrix 0.697 / 0.689).
  // Rows of ~73 nonzeros (banded, N = 64) keep 4: 0.251 ms against 0.266
  // with 16.
  if (schedule == SEGTACO_RB_PR && long_rows) {
    cfg->items_per_unit = (int)kPieceThreshold;
    if (mean < 32.0) cfg->rows_per_unit = M / 64 >= 8192 ? 64 : 32;
  }
  // fp32 B beyond L2 under skewed rows: the gathered B rows evict_last in L2
  // (A and C stream with evict-first loads and stores).  Measured on GB300,
  // 1M x 1M power law, N = 128, three alternations: eb_pr 1.128 -> 1.110 ms,
  // rb_pr (pieces, 32 rows per warp) 1.219 -> 1.201; rb_sr unchanged (1.683
  // / 1.687).
  if (!sequential && esz == 4 && bbytes > 48e6 && skewed) cfg->flags |= SEGTACO_FLAG_L2_HINTS;
  // Rows known to lie near the diagonal (the caller's segtaco_band_stats):
  // rb_pr takes the band kernel (32-row blocks, the band of A as a dense tile,
  // B's window by TMA, 4 x 4 register tiles; spmm_window.cu) with a halo of
  // 32.  Measured on GB300, banded-plus-random 262,144 rows (half band 32, 8
  // off-band nonzeros per row): fp32 N = 64 0.2465 -> 0.178 ms, bf16 B
  // 0.2323 -> 0.112 ms, fp32 N = 128 0.650 -> 0.455 ms (halo 16: 0.61 ms,
  // 48: 0.29 ms at fp32 N = 64).  The staged window for the row-block walk
  // (still one gathered B slice per nonzero, from shared memory instead of
  // L1) measured slower than the plain row blocks (0.373 vs 0.248 ms) and is
  // not chosen; rb_sr keeps the plain row blocks.
  if (banded && schedule == SEGTACO_RB_PR && !long_rows && N >= 64 && N % 16 == 0) {
    cfg->flags |= SEGTACO_FLAG_WINDOW;
    cfg->items_per_unit = 32;
  }
  return SEGTACO_OK;
}

int segtaco_spmm_plan_name(int32_t M, int32_t K, int64_t nnz, int32_t N, int32_t b_dtype,
                           const void *B, int64_t ldb, const segtaco_config *cfg, char *out,
                           size_t len) {
  if (!out || len == 0) return set_error(SEGTACO_EINVAL, "out is NULL");
  SpmmPlan plan;
  SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, ldb, N, B, nullptr, cfg, &plan));
  static const char *sched[] = {"rb_sr", "rb_pr", "eb_sr", "eb_pr"};
  const char *kernel = plan.use_tma         ? "tma_ring"
                       : plan.band_halo >= 0   ? "band"
                       : plan.window_halo >= 0 ? "window"
                       : plan.long_row > 0 ? (plan.piece_len > 0 ? "pieces" : "long_rows")
                       : (plan.schedule >= SEGTACO_EB_SR) ? "chunks" : "rows";
  snprintf(out, len, "%s %s V=%d G=%d W=%d slabs=%d walk=%d halo=%d rows_per_unit=%lld parts=%d",
           sched[plan.schedule], kernel, plan.V, plan.G, plan.W, plan.slabs, plan.walk,
           plan.band_halo >= 0 ? plan.band_halo : plan.window_halo,
           (long long)plan.rows_per_unit, plan.piece_len > 0 ? plan.piece_parts : 1);
  return SEGTACO_OK;
}

int segtaco_spmm_workspace_size(int32_t M, int32_t K, int64_t nnz, int32_t N, int32_t b_dtype,
                                const segtaco_config *cfg, size_t *bytes) {
  if (!bytes) return set_error(SEGTACO_EINVAL, "bytes is NULL");
  SpmmPlan plan;
  // Alignment does not change the workspace: plan with aligned stand-ins.
  SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, N, N, nullptr, nullptr, cfg, &plan));
  *bytes = plan.workspace;
  if (plan.walk == kWalkSplitJoin) {  // (row pitches from 4 GB keep the pieces)
    SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, N, N, nullptr, nullptr, cfg, &plan,
                          LongRowScratch::kPieces));
    *bytes = std::max(*bytes, plan.workspace);
  }
  return SEGTACO_OK;
}

// Whether a caller's workspace holds the sums of joined chunks.
static bool holds_sums(const SpmmPlan &plan, const void *workspace, size_t bytes) {
  return bytes >= plan.workspace && ((uintptr_t)workspace & 255) == 0;
}

// Whether segtaco_spmm_partition, which knows neither B nor its pitch, made what `plan`
// reads from this workspace.  Another alignment or pitch of B can change the lanes, and
// with them the pieces' layout or the chunks' size, and a row pitch from 4 GB takes
// pieces where the partition had joined chunks in mind and prepared nothing.
static bool partition_serves(const SpmmPlan &plan, int M, int K, long long nnz, int N, int b_dtype,
                             const float *C, long long ldc, const segtaco_config *cfg,
                             const void *workspace, size_t bytes) {
  SpmmPlan p;
  if (plan_spmm(M, K, nnz, N, b_dtype, N, ldc, nullptr, C, cfg, &p) != SEGTACO_OK) return false;
  if (p.walk == kWalkSplitJoin && !holds_sums(p, workspace, bytes) &&
      plan_spmm(M, K, nnz, N, b_dtype, N, ldc, nullptr, C, cfg, &p, LongRowScratch::kPieces) !=
          SEGTACO_OK)
    return false;
  const bool pieces = plan.piece_len > 0;
  return p.px_entries == plan.px_entries && p.py_entries == plan.py_entries &&
         p.items_per_unit == plan.items_per_unit && p.long_row == plan.long_row &&
         p.piece_len == plan.piece_len && p.piece_parts == plan.piece_parts &&
         (!pieces || (p.slabs == plan.slabs && p.W == plan.W));
}

int segtaco_spmm(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr, const int32_t *col,
                 const float *vals, const void *B, int32_t b_dtype, int64_t ldb, float *C,
                 int64_t ldc, int32_t N, const segtaco_config *cfg, void *workspace,
                 size_t workspace_bytes, void *stream) {
  SEGTACO_TRY(check_csr_args(M, K, nnz, row_ptr, col));
  if (N < 0) return set_error(SEGTACO_EINVAL, "negative N");
  if (b_dtype != SEGTACO_F32 && b_dtype != SEGTACO_BF16)
    return set_error(SEGTACO_EINVAL, "unknown dense dtype %d", b_dtype);
  if (M == 0 || N == 0) return SEGTACO_OK;
  if (C == nullptr) return set_error(SEGTACO_EINVAL, "C is NULL");
  if (nnz > 0 && B == nullptr) return set_error(SEGTACO_EINVAL, "B is NULL");
  if (ldb < N || ldc < N) return set_error(SEGTACO_EINVAL, "ldb/ldc smaller than N");
  SpmmPlan plan;
  SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, ldb, ldc, B, C, cfg, &plan));
  // A caller's workspace that cannot hold the sums of cut rows: the pieces or row blocks
  if (plan.walk == kWalkSplitJoin && workspace && !holds_sums(plan, workspace, workspace_bytes))
    SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, ldb, ldc, B, C, cfg, &plan,
                          LongRowScratch::kPieces));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bool ready = cfg && (cfg->flags & SEGTACO_FLAG_PARTITION_READY);
  if (ready && workspace && plan.workspace)
    ready = partition_serves(plan, M, K, nnz, N, b_dtype, C, ldc, cfg, workspace, workspace_bytes);
  const bool search = !ready && plan.walk == kWalkSplit && (long long)M * N <= kSearchMaxElems;
  Scratch scratch(workspace, workspace_bytes, s);
  if (workspace || !search)  // (a caller's workspace is checked, if not needed)
    SEGTACO_TRY(scratch.reserve(plan.workspace));
  int *px = nullptr, *py = nullptr;
  if (plan.workspace && !search) {
    px = static_cast<int *>(scratch.take(plan.px_entries * sizeof(int)));
    py = static_cast<int *>(scratch.take(plan.py_entries * sizeof(int)));
  }
  // (below the pieces' size rb_pr has nothing prepared and needs no caller's workspace)
  if (ready && plan.workspace && !workspace &&
      (plan.walk != kWalkSplitJoin || nnz >= kLongRowsMinNnz))
    return set_error(SEGTACO_EINVAL, "PARTITION_READY needs the caller's workspace");
  return run_spmm_planned(plan, M, K, nnz, row_ptr, col, vals, B, b_dtype, ldb, C, ldc, N, px, py,
                          s, ready);
}

int segtaco_spmm_partition(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr, float *C,
                           int64_t ldc, int32_t N, int32_t b_dtype, const segtaco_config *cfg,
                           void *workspace, size_t workspace_bytes, void *stream) {
  SEGTACO_TRY(check_csr_args(M, K, nnz, row_ptr, nullptr, false));
  if (M == 0 || N == 0) return SEGTACO_OK;
  if (C == nullptr || ldc < N) return set_error(SEGTACO_EINVAL, "C is NULL or ldc < N");
  SpmmPlan plan;
  SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, N, ldc, nullptr, C, cfg, &plan));
  if (plan.walk == kWalkSplitJoin && workspace && holds_sums(plan, workspace, workspace_bytes))
    return SEGTACO_OK;  // nothing to prepare
  if (plan.walk == kWalkSplitJoin)
    SEGTACO_TRY(plan_spmm(M, K, nnz, N, b_dtype, N, ldc, nullptr, C, cfg, &plan,
                          LongRowScratch::kPieces));
  if (!plan.workspace) return SEGTACO_OK;
  if (!workspace) return set_error(SEGTACO_EINVAL, "segtaco_spmm_partition needs a workspace");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Scratch scratch(workspace, workspace_bytes, s);
  SEGTACO_TRY(scratch.reserve(plan.workspace));
  int *px = static_cast<int *>(scratch.take(plan.px_entries * sizeof(int)));
  int *py = static_cast<int *>(scratch.take(plan.py_entries * sizeof(int)));
  if (plan.long_row > 0 && plan.piece_len > 0)
    return launch_long_pieces_list(row_ptr, M, nnz, plan.long_row, plan.piece_len, plan.slabs,
                                   plan.W, plan.piece_parts, px, py, s);
  if (plan.long_row > 0) return launch_long_rows_list(row_ptr, M, nnz, plan.long_row, px, py, s);
  return launch_merge_path(row_ptr, M, nnz, plan.items_per_unit, plan.nchunks, px, py, C, ldc, N,
                           s);
}

int segtaco_block_starts_taco(int32_t M, int64_t nnz, const int32_t *row_ptr, int32_t P,
                              int32_t *out, void *stream) {
  SEGTACO_TRY(check_csr_args(M, 0, nnz, row_ptr, nullptr, false));
  if (P <= 0 || out == nullptr) return set_error(SEGTACO_EINVAL, "P must be > 0, out non-NULL");
  const long long nblk = (nnz + P - 1) / P;
  return launch_block_starts_taco(row_ptr, M, P, nblk, out, static_cast<cudaStream_t>(stream));
}

int segtaco_block_starts_canonical(int32_t M, int64_t nnz, const int32_t *row_ptr, int32_t P,
                                   int32_t *out, void *stream) {
  SEGTACO_TRY(check_csr_args(M, 0, nnz, row_ptr, nullptr, false));
  if (P <= 0 || out == nullptr) return set_error(SEGTACO_EINVAL, "P must be > 0, out non-NULL");
  const long long nblk = (nnz + P - 1) / P;
  return launch_block_starts_canonical(row_ptr, M, P, nblk, out,
                                       static_cast<cudaStream_t>(stream));
}

int segtaco_merge_path(int32_t M, int64_t nnz, const int32_t *row_ptr, int64_t D, int32_t *out_x,
                       int32_t *out_y, void *stream) {
  SEGTACO_TRY(check_csr_args(M, 0, nnz, row_ptr, nullptr, false));
  if (D <= 0 || !out_x || !out_y) return set_error(SEGTACO_EINVAL, "D must be > 0, outputs non-NULL");
  long long nch = ((long long)M + nnz + D - 1) / D;
  if (nch < 1) nch = 1;
  return launch_merge_path(row_ptr, M, nnz, D, nch, out_x, out_y, nullptr, 0, 0,
                           static_cast<cudaStream_t>(stream));
}

int segtaco_row_ids(int32_t M, int64_t nnz, const int32_t *row_ptr, int32_t *out, void *stream) {
  SEGTACO_TRY(check_csr_args(M, 0, nnz, row_ptr, nullptr, false));
  if (nnz > 0 && out == nullptr) return set_error(SEGTACO_EINVAL, "out is NULL");
  return launch_row_ids(row_ptr, M, out, static_cast<cudaStream_t>(stream));
}

int segtaco_csr_validate(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr,
                         const int32_t *col, void *stream) {
  SEGTACO_TRY(check_csr_args(M, K, nnz, row_ptr, col));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Scratch scratch(nullptr, 0, s);
  SEGTACO_TRY(scratch.reserve(256));
  int *err = static_cast<int *>(scratch.take(2 * sizeof(int)));
  SEGTACO_TRY(check_cuda(cudaMemsetAsync(err, 0, 2 * sizeof(int), s), "memset"));
  SEGTACO_TRY(launch_validate(row_ptr, M, K, nnz, col, err, s));
  int h[2] = {0, 0};
  SEGTACO_TRY(check_cuda(cudaMemcpyAsync(h, err, sizeof(h), cudaMemcpyDeviceToHost, s), "copy"));
  SEGTACO_TRY(check_cuda(cudaStreamSynchronize(s), "sync"));
  static const char *what[] = {"", "row_ptr[0] != 0", "row_ptr[M] != nnz",
                               "row_ptr decreases at row", "col out of [0, K) at nonzero"};
  if (h[0] != 0) return set_error(SEGTACO_EINVAL, "malformed CSR: %s %d", what[h[0] & 7], h[1]);
  return SEGTACO_OK;
}

// The workspace that segtaco_spmv accepts: the partition of 512-item merge-path
// chunks (spmv.cu needs none).
static segtaco_config spmv_config() {
  segtaco_config c = {};
  c.schedule = SEGTACO_EB_PR;
  c.col_tile = 1;
  c.vec = 1;
  c.items_per_unit = 512;
  c.flags = SEGTACO_FLAG_ROW_WALK;
  return c;
}

int segtaco_spmv_workspace_size(int32_t M, int64_t nnz, size_t *bytes) {
  if (!bytes) return set_error(SEGTACO_EINVAL, "bytes is NULL");
  if (M < 0 || nnz < 0) return set_error(SEGTACO_EINVAL, "negative size");
  const segtaco_config c = spmv_config();
  SpmmPlan plan;
  SEGTACO_TRY(plan_spmm(M, 1, nnz, 1, SEGTACO_F32, 1, 1, nullptr, nullptr, &c, &plan));
  *bytes = plan.workspace;
  return SEGTACO_OK;
}

int segtaco_spmv(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr, const int32_t *col,
                 const float *vals, const float *x, float *y, void *workspace,
                 size_t workspace_bytes, void *stream) {
  SEGTACO_TRY(check_csr_args(M, K, nnz, row_ptr, col));
  if (M == 0) return SEGTACO_OK;
  if (y == nullptr || (nnz > 0 && x == nullptr)) return set_error(SEGTACO_EINVAL, "x/y is NULL");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (workspace) {  // checked, if no longer needed
    size_t need = 0;
    SEGTACO_TRY(segtaco_spmv_workspace_size(M, nnz, &need));
    Scratch scratch(workspace, workspace_bytes, s);
    SEGTACO_TRY(scratch.reserve(need));
  }
  return launch_spmv(M, nnz, row_ptr, col, vals, x, y, s);
}

int segtaco_sddmm_autotune(int32_t M, int32_t K, int64_t nnz, int32_t D, int32_t x_dtype,
                           int64_t max_row_len, segtaco_sddmm_config *cfg) {
  if (!cfg) return set_error(SEGTACO_EINVAL, "cfg is NULL");
  if (M < 0 || K < 0 || nnz < 0 || D < 0) return set_error(SEGTACO_EINVAL, "negative size");
  const bool banded = cfg->kernel == SEGTACO_SDDMM_BAND;
  memset(cfg, 0, sizeof(*cfg));
  cfg->kernel = SEGTACO_SDDMM_AUTO;
  // Rows known to lie near the diagonal: the band kernel (sddmm_band.cu).
  // Measured on GB300, banded-plus-random 262,144 rows, D = 64: fp32 0.330 ->
  // 0.191 ms, bf16 factors 0.303 -> 0.150 ms.
  if (banded && D == 64) cfg->kernel = SEGTACO_SDDMM_BAND;
  (void)x_dtype;
  // Blocks of 256 nonzeros per warp; smaller for small problems, so that the
  // launch still holds about a wave of warps (152 SMs x 32).  Measured on GB300,
  // default kernel, blocks of 32 / 64 / 128 / 256: 1.2M nonzeros, D = 16 - / 17.1 /
  // 14.5 / 13.3 us, D = 64 bf16 - / 25.2 / 22.9 / 21.6; 58,751, D = 64 4.9 / 6.3 / 9.6
  // / 16.8.
  int blk = 256;
  while (blk > 32 && nnz / blk < 4096) blk >>= 1;
  cfg->block_nnz = blk;
  cfg->lanes = 0;  // from D (sddmm_shape)
  (void)max_row_len;
  (void)K;
  return SEGTACO_OK;
}

int segtaco_sddmm_ex(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr,
                     const int32_t *col, const float *vals, const void *X, const void *Y,
                     int32_t x_dtype, int64_t ldx, int64_t ldy, int32_t D, float *out,
                     const segtaco_sddmm_config *cfg, void *stream) {
  SEGTACO_TRY(check_csr_args(M, K, nnz, row_ptr, col));
  if (x_dtype != SEGTACO_F32 && x_dtype != SEGTACO_BF16)
    return set_error(SEGTACO_EINVAL, "unknown dense dtype %d", x_dtype);
  if (nnz == 0) return SEGTACO_OK;
  if (D < 0 || ldx < D || ldy < D) return set_error(SEGTACO_EINVAL, "bad D/ldx/ldy");
  if (!X || !Y || !out) return set_error(SEGTACO_EINVAL, "X/Y/out is NULL");
  segtaco_sddmm_config c;
  if (cfg)
    c = *cfg;
  else
    SEGTACO_TRY(segtaco_sddmm_autotune(M, K, nnz, D, x_dtype, -1, &c));
  const long long P = c.block_nnz > 0 ? c.block_nnz : sddmm_block_nnz();
  if (P < 32 || P > 4096 || (P & (P - 1)))
    return set_error(SEGTACO_EINVAL, "block_nnz=%lld not a power of two in [32, 4096]", P);
  if (c.lanes < 0 || c.lanes > 32 || (c.lanes & (c.lanes - 1)))
    return set_error(SEGTACO_EINVAL, "lanes=%d not 0 or a power of two up to 32", c.lanes);
  if (c.kernel < SEGTACO_SDDMM_AUTO || c.kernel > SEGTACO_SDDMM_BAND)
    return set_error(SEGTACO_EINVAL, "unknown SDDMM kernel %d", c.kernel);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (c.kernel == SEGTACO_SDDMM_BAND && sddmm_band_applies(x_dtype, D, ldx, ldy, X, Y))
    return launch_sddmm_band(M, K, nnz, row_ptr, col, vals, X, Y, x_dtype, ldx, ldy, D, out, s);
  if (c.kernel == SEGTACO_SDDMM_BAND) c.kernel = SEGTACO_SDDMM_AUTO;
  const long long nblk = (nnz + P - 1) / P;
  const bool x_first = sddmm_x_first(M, K, D, x_dtype);
  if (c.kernel == SEGTACO_SDDMM_AUTO && c.lanes == 0 && sddmm_gather_applies(x_dtype, ldx, ldy)) {
    // Dot products of 512 bytes and more in 32-byte lanes stay with the fixed-shape
    // kernel, two loads per lane (banded, 100,000 rows, D = 128 fp32: 219 us against
    // 232; lognormal rows 55.5 / 55.7), also without a pass for the block starts.
    const SddmmShape sh = sddmm_shape(x_dtype, D, ldx, ldy, X, Y, 0);
    if ((sh.family == 1 || sh.family == 2) && sh.KI == 2 && sh.G >= 8)
      return launch_sddmm(M, nnz, row_ptr, col, vals, X, Y, x_dtype, ldx, ldy, D, out, nullptr,
                          (int)P, nblk, s, false, 0, SEGTACO_SDDMM_FIXED, x_first);
    return launch_sddmm_gather(M, nnz, row_ptr, col, vals, X, Y, x_dtype, ldx, ldy, D, out, (int)P,
                               x_first, s);
  }
  Scratch scratch(nullptr, 0, s);
  SEGTACO_TRY(scratch.reserve(align256((size_t)(nblk + 1) * sizeof(int))));
  int *starts = static_cast<int *>(scratch.take((nblk + 1) * sizeof(int)));
  return launch_sddmm(M, nnz, row_ptr, col, vals, X, Y, x_dtype, ldx, ldy, D, out, starts, (int)P,
                      nblk, s, false, c.lanes, c.kernel, x_first);
}

int segtaco_sddmm(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr, const int32_t *col,
                  const float *vals, const void *X, const void *Y, int32_t x_dtype, int64_t ldx,
                  int64_t ldy, int32_t D, float *out, void *stream) {
  return segtaco_sddmm_ex(M, K, nnz, row_ptr, col, vals, X, Y, x_dtype, ldx, ldy, D, out, nullptr,
                          stream);
}

int segtaco_spmspv(int32_t M, int32_t K, int64_t nnz, const int32_t *col_ptr,
                   const int32_t *row_idx, const float *vals, int32_t nx, const int32_t *x_idx,
                   const float *x_vals, float *y, void *stream) {
  SEGTACO_TRY(check_csr_args(K, M, nnz, col_ptr, row_idx));
  if (nx < 0) return set_error(SEGTACO_EINVAL, "negative nx");
  if (M > 0 && y == nullptr) return set_error(SEGTACO_EINVAL, "y is NULL");
  if (nx > 0 && (!x_idx || !x_vals)) return set_error(SEGTACO_EINVAL, "x is NULL");
  return launch_spmspv(M, K, nnz, col_ptr, row_idx, vals, nx, x_idx, x_vals, y,
                       static_cast<cudaStream_t>(stream));
}

}  // extern "C"

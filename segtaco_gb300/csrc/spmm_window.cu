// spmm_window.cu -- row-block SpMM with the reused B rows staged by TMA.
//
// For matrices whose nonzeros cluster around the diagonal (banded, block
// diagonal, meshes), the rows of a row block gather B rows from a short range
// around the block: rows i0 .. i1-1 touch B rows near [i0 - H, i1 + H).  Each
// 128-thread CTA here owns a block of 4 * rows_per_unit rows and one column
// slab; one thread brings the window B[i0 - H .. i1 + H) x slab into shared
// memory with a single cp.async.bulk.tensor.2d copy (a tensor map over B,
// box = window rows x slab columns; rows outside [0, K) are zero-filled by the
// copy engine), completing on an mbarrier.  Then the four warps walk their row
// blocks exactly as the row-block kernel does (spmm_walk_unit), except that a
// gather of a B row inside the window reads the shared copy; rows outside it
// (the off-band nonzeros) are still gathered from global memory.  So every
// in-band B row crosses L2 once per row block instead of once per nonzero.
//
// The wait is bounded: after kWindowSpin polls the CTA records SEGTACO_ETIMEOUT
// in the device status word (segtaco_device_status), waits once more, bounded,
// for its copy, and leaves its rows unwritten.
//
// Same results as the row-block kernel: the walk, its summation order and its
// stores are unchanged, only where a B value is read from.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <atomic>
#include <cfloat>
#include <mutex>

#include "mma.cuh"
#include "spmm_launch.cuh"

namespace segtaco {
namespace {

constexpr long long kWindowSpin = 1LL << 22;

__device__ __forceinline__ uint32_t sm_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool window_wait(uint32_t bar) {
  for (long long i = 0; i < kWindowSpin; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(0)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Most gathers come from shared memory here, so fewer resident warps hide
// the latency: 16 warps per SM, whose registers hold the walk and both
// gather paths without spilling.
template <typename BT, int V, int G> constexpr int window_min_ctas() {
  return 16 / kSpmmWarps;
}

template <typename BT, int V, int G>
__global__ void __launch_bounds__(kSpmmCta, window_min_ctas<BT, V, G>())
    spmm_window_kernel(SpmmArgs<BT> a, const __grid_constant__ CUtensorMap tm, int halo,
                       int *status) {
  constexpr int W = G * V;
  extern __shared__ __align__(128) unsigned char smem[];
  const long long rows_blk = (long long)kSpmmWarps * a.rows_per_unit;
  const int wrows = (int)(rows_blk + 2 * halo);
  BT *win = reinterpret_cast<BT *>(smem);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (((size_t)wrows * W * sizeof(BT) + 15) & ~size_t(15)));
  const int wlo = (int)((long long)blockIdx.x * rows_blk - halo);
  const uint32_t b = sm_u32(bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)((size_t)wrows * W * sizeof(BT));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes)
                 : "memory");
    // x = the slab's first column (a multiple of W: 16-byte aligned), y = the
    // window's first row (negative at the top edge: zero-filled)
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(sm_u32(win)),
        "l"(&tm), "r"((int)(blockIdx.y * W)), "r"(wlo), "r"(b)
        : "memory");
  }
  if (!window_wait(b)) {
    if (threadIdx.x == 0) atomicExch(status, SEGTACO_ETIMEOUT);
    window_wait(b);  // the copy may still land: wait for it once more, bounded
    return;
  }
  const long long w = (long long)blockIdx.x * kSpmmWarps + threadIdx.x / 32;
  if (w >= a.units) return;
  Window<BT> wv;
  wv.base = win;
  wv.lo = wlo;
  wv.rows = wrows;
  spmm_walk_unit<BT, V, G, true, false, true>(a, w, blockIdx.y, threadIdx.x & 31, wv);
}

// ---------------------------------------------------------------------------
// Banded row blocks for rb_pr (SEGTACO_FLAG_WINDOW with a parallel reduction), fp32
// B; bf16 B: spmm_band_mma_kernel below.
//
// On a banded matrix the plain row blocks deliver each nonzero's 64-column B
// slice to registers (256 bytes for 64 multiply-adds), and that load/store
// data pipe is their bound; the window kernel above only moves the same bytes
// from shared memory instead of L1.  Here B values are reused from registers:
// a CTA owns kBandRows = 32 consecutive rows and a slab of 64 columns, brings
// the band window B[jw0 .. jw0 + win) x slab (win = 32 + 2H rows around the
// diagonal, column i0 * K / M of its first row) into shared memory with one
// TMA tensor copy, and scatters its rows' in-window nonzeros into a dense
// tile At[win][32] (row pitch kBandPitch = 36 floats: 16-byte aligned, and
// the scatter's consecutive columns of one row spread over 8 banks).  Thread
// (rb, cb) then keeps rows 4rb .. 4rb+3 x columns 4cb .. 4cb+3 in registers
// and, for every window row j, reads At[j][4rb .. 4rb+3] and B[j][4cb ..
// 4cb+3] (two 16-byte shared loads) for 16 multiply-adds: 2 bytes to
// registers per multiply-add.  The tile holds zeros where a row has no
// nonzero (win steps per row instead of ~2H + 1 nonzeros), and the summation
// order within a row differs from the storage order, which the parallel
// reduction allows; duplicate entries of a row add up in the tile.
//
// The scatter reads the block's nonzeros (contiguous in A) coalesced, 20 per thread in
// flight, one exchange per nonzero (with 8, a row search each and float adds in shared
// memory: banded 262,144 rows, N = 64 195 us, now 181; 100,000, N = 128 144, now 133).
// Off-band nonzeros (outside the window) go to a per-row list of kBandList entries,
// and each thread gathers its 4 columns of them from global memory, 8 at a time (a
// row with more walks its nonzeros in global memory instead).  The tile's zeros make
// NaN of infinities in the window's unused rows: a thread that ends with an infinity
// or NaN sums that row again, nonzero by nonzero.  (Five CTAs per SM, what the shared
// memory allows: 93 registers, banded 262,144 rows, N = 64 183.5 -> 177.8 us against the 79
// the compiler takes unasked.)  The TMA wait is bounded as in the window kernel
// (SEGTACO_ETIMEOUT, rows left unwritten).
constexpr int kBandRows = 32;
constexpr int kBandCols = 64;
constexpr int kBandList = 16;
constexpr int kBandPitch = 36;

__device__ __forceinline__ float4 band_b4(const float *p) {
  return __ldg(reinterpret_cast<const float4 *>(p));
}
__device__ __forceinline__ void band_fma4(float (&acc)[4], float x, const float4 &b) {
  acc[0] = fmaf(x, b.x, acc[0]);
  acc[1] = fmaf(x, b.y, acc[1]);
  acc[2] = fmaf(x, b.z, acc[2]);
  acc[3] = fmaf(x, b.w, acc[3]);
}

// Shared-memory layout of a band CTA (byte offsets; win = window rows).
struct BandSmem {
  size_t at, rp, cnt, lcol, lval, bar, bytes;
};
__host__ __device__ inline BandSmem band_smem(int win) {
  BandSmem m;
  size_t o = ((size_t)win * kBandCols * sizeof(float) + 127) & ~size_t(127);  // B window first
  m.at = o;
  o += (size_t)win * kBandPitch * 4;
  m.rp = o;
  o += (kBandRows + 1) * 4;
  m.cnt = o;
  o += kBandRows * 4;
  m.lcol = o;
  o += kBandRows * kBandList * 4;
  m.lval = o;
  o += kBandRows * kBandList * 4;
  m.bar = (o + 7) & ~size_t(7);
  m.bytes = m.bar + 8;
  return m;
}

__global__ void __launch_bounds__(kSpmmCta, 5)
    spmm_band_kernel(SpmmArgs<float> a, const __grid_constant__ CUtensorMap tm, int halo,
                     int *status) {
  const int win = kBandRows + 2 * halo;
  const BandSmem L = band_smem(win);
  extern __shared__ __align__(128) unsigned char smem[];
  float *bw = reinterpret_cast<float *>(smem);  // [win][kBandCols]
  float *at = reinterpret_cast<float *>(smem + L.at);  // [win][kBandPitch]
  int *rp = reinterpret_cast<int *>(smem + L.rp);
  int *cnt = reinterpret_cast<int *>(smem + L.cnt);
  int *lcol = reinterpret_cast<int *>(smem + L.lcol);
  float *lval = reinterpret_cast<float *>(smem + L.lval);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L.bar);
  const int t = threadIdx.x;
  const int M = a.M;
  const int i0 = blockIdx.x * kBandRows;
  const int jw0 = (int)((long long)i0 * a.K / M) - halo;
  const uint32_t b = sm_u32(bar);
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b),
                 "r"((uint32_t)((size_t)win * kBandCols * sizeof(float)))
                 : "memory");
    // x = the slab's first column (a multiple of 64 elements), y = the
    // window's first row (negative at the top edge: zero-filled)
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(sm_u32(bw)),
        "l"(&tm), "r"((int)(blockIdx.y * kBandCols)), "r"(jw0), "r"(b)
        : "memory");
  }
  // Scatter the block's nonzeros, SQ per thread per pass with every load in flight;
  // the first pass loads before the tile is cleared.  An exchange puts a value in
  // the tile; where it returns another entry of the same position, that one is added
  // back (the native exchange is one instruction, an add of floats in shared memory a
  // loop).
  constexpr int SQ = 20;
  const int k_beg = __ldg(a.row_ptr + i0), k_end = __ldg(a.row_ptr + min(i0 + kBandRows, M));
  int cj[SQ];
  float cv[SQ];
  auto load = [&](int n0) {  // nonzeros k_beg + n0 + t + 128 q
#pragma unroll
    for (int q = 0; q < SQ; ++q) {
      const bool has = n0 + t + q * kSpmmCta < k_end - k_beg;
      cj[q] = has ? __ldg(a.col + (k_beg + n0 + t + q * kSpmmCta)) : 0;
      cv[q] = has ? ld_val(a.val, k_beg + n0 + t + q * kSpmmCta) : 0.0f;
    }
  };
  load(0);
  for (int e = t; e < win * kBandPitch / 4; e += kSpmmCta)
    reinterpret_cast<float4 *>(at)[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (t <= kBandRows) rp[t] = __ldg(a.row_ptr + min(i0 + t, M));
  if (t < kBandRows) cnt[t] = 0;
  __syncthreads();
  for (int n0 = 0; n0 < k_end - k_beg; n0 += SQ * kSpmmCta) {
    if (n0 > 0) load(n0);
    int r = 0;  // the last row whose start is <= the thread's first nonzero
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (r + step <= kBandRows - 1 && rp[r + step] - k_beg <= n0 + t) r += step;
    int rend = rp[r + 1] - k_beg;
#pragma unroll
    for (int q = 0; q < SQ; ++q) {
      const int n = n0 + t + q * kSpmmCta;
      if (n < k_end - k_beg) {
        while (n >= rend) rend = rp[++r + 1] - k_beg;  // n < rp[kBandRows] - k_beg
        const unsigned d = (unsigned)(cj[q] - jw0);
        if (d < (unsigned)win) {
          float *cell = at + d * kBandPitch + r;
          const float old = atomicExch(cell, cv[q]);
          if (old != 0.0f) atomicAdd(cell, old);
        } else {
          const int slot = atomicAdd(cnt + r, 1);
          if (slot < kBandList) {
            lcol[r * kBandList + slot] = cj[q];
            lval[r * kBandList + slot] = cv[q];
          }
        }
      }
    }
  }
  __syncthreads();
  if (!window_wait(b)) {
    if (t == 0) atomicExch(status, SEGTACO_ETIMEOUT);
    window_wait(b);  // the copy may still land: wait for it once more, bounded
    return;
  }
  const int rb = t >> 4, cb = t & 15;
  const int c0 = blockIdx.y * kBandCols + 4 * cb;  // this thread's first column
  if (c0 >= a.N) return;                           // N is a multiple of 16
  float acc[4][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0f;
  // The first off-band gathers of row 4rb, issued before the tile product so
  // that their latency hides behind it.
  const int n0 = cnt[4 * rb];
  const int pre = n0 <= kBandList ? min(n0, 8) : 0;
  float4 g0[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    // slots past the row's list gather B row 0 (in bounds) and are not used
    const int j = e < pre ? lcol[4 * rb * kBandList + e] : 0;
    g0[e] = band_b4(a.B + (size_t)(unsigned)j * a.ldb + c0);
  }
  const float *acol = at + 4 * rb;
  const float *bcol = bw + 4 * cb;
#pragma unroll 4
  for (int j = 0; j < win; ++j) {
    const float4 x = *reinterpret_cast<const float4 *>(acol + j * kBandPitch);
    const float4 bv = *reinterpret_cast<const float4 *>(bcol + j * kBandCols);
    band_fma4(acc[0], x.x, bv);
    band_fma4(acc[1], x.y, bv);
    band_fma4(acc[2], x.z, bv);
    band_fma4(acc[3], x.w, bv);
  }
  // Off-band nonzeros of the thread's four rows, from global memory.
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (e < pre) band_fma4(acc[0], lval[4 * rb * kBandList + e], g0[e]);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = 4 * rb + q;
    const int n = cnt[r];
    if (n <= kBandList) {
      for (int e0 = q == 0 ? pre : 0; e0 < n; e0 += 8) {
        float4 g[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int ee = e0 + e < n ? e0 + e : e0;
          g[e] = band_b4(a.B + (size_t)(unsigned)lcol[r * kBandList + ee] * a.ldb + c0);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (e0 + e < n) band_fma4(acc[q], lval[r * kBandList + e0 + e], g[e]);
      }
    } else {
      // more off-band nonzeros than the list holds: walk the row
      for (int k = rp[r]; k < rp[r + 1]; ++k) {
        const int j = __ldg(a.col + k);
        if ((unsigned)(j - jw0) >= (unsigned)win)
          band_fma4(acc[q], ld_val(a.val, k),
                    band_b4(a.B + (size_t)(unsigned)j * a.ldb + c0));
      }
    }
  }
  // An infinity or NaN: from the row's own terms, or from a zero of the tile times an
  // infinity of the window.  The row again, nonzero by nonzero.
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float amax = max_nan(max_nan(acc[q][0], acc[q][1]), max_nan(acc[q][2], acc[q][3]));
    if (!(fabsf(amax) <= FLT_MAX)) {
      acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = 0.0f;
#pragma unroll 1
      for (int k = rp[4 * rb + q]; k < rp[4 * rb + q + 1]; ++k)
        band_fma4(acc[q], ld_val(a.val, k),
                  band_b4(a.B + (size_t)(unsigned)__ldg(a.col + k) * a.ldb + c0));
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = i0 + 4 * rb + q;
    if (i < M)
      __stcs(reinterpret_cast<float4 *>(a.C + (long long)i * a.ldc + c0),
             make_float4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]));
  }
}

// ---------------------------------------------------------------------------
// The band tile on the tensor cores, for a bf16 dense operand.
//
// The tile product At x B is a dense contraction (32 x win by win x 64 per CTA), and
// its multiply-adds, two shared loads per 16 of them, were the kernel's time.  Here
// it runs as mma.m16n8k16 with fp32 accumulation.  A's values are fp32: each is split
// into three bf16 parts (x = hi + mid + lo, mma.cuh), so three
// products per step give the exact products x*b that the multiply-add form rounds
// once; the parts of a step are summed from zero, lowest first, and added to the
// running sum in fp32.  (tcgen05 needs 64 or 128 rows per tile: a 32-row block's
// band fills 68 % of its 96-column window, a 128-row block's 34 % of 192.)
//
// Warp w: rows 16 (w & 1) .. +15, all 64 columns, every other half of the window
// steps (w >> 1).  B's window comes by TMA with the 128-byte swizzle and is read
// with ldmatrix.trans.  The two halves' sums go to shared memory (the tile's space),
// and eight lanes per row then add its off-band nonzeros (16 bytes of B per lane) and
// store whole lines of C.
//
// Splitting an infinity or NaN, or multiplying a zero part by one, makes NaN, a value
// next to the largest splits into infinite parts, and one below 2^-103 has no three
// parts: a CTA that finds an infinity or NaN among its sums, or such a value in its
// tile, sums its rows nonzero by nonzero instead.
//
// What bounds it now: instructions (56 % of issue slots with 23 warps per SM), most of
// them in the scatter and the off-band rows; the tensor pipe is 14 % busy.  Measured
// on GB300, banded-plus-random 262,144 rows (half band 32, 8 off-band nonzeros per
// row), bf16 B, N = 64: 160 us with multiply-adds -> 112 (without the product 97,
// without the off-band rows 97); error against FP64 1.5e-7 -> 9.3e-8.  20 nonzeros in
// flight per thread instead of 10 117.5 -> 115.6 us; a warp per row instead of the flat
// scatter 122; seven CTAs per SM 120; all three parts summed in the tensor cores'
// accumulators 120 us and an error of 1.57e-7.
constexpr int kBandAPad = 8;   // tile pitch win + 8: conflict-free 8-byte fragment loads
constexpr int kBandCPad = 4;   // pitch of the summed rows: 68 floats

struct BandMmaSmem {
  size_t at, list, rp, cnt, bar, bytes;
};
__host__ __device__ inline int band_mma_win(int halo) { return (kBandRows + 2 * halo + 15) & ~15; }
__host__ __device__ inline BandMmaSmem band_mma_smem(int win) {
  BandMmaSmem m;
  m.at = (size_t)win * 128;  // B window first: 64 bf16 per row
  size_t o = m.at + (size_t)kBandRows * (win + kBandAPad) * 4;
  const size_t sums = (size_t)2 * kBandRows * (kBandCols + kBandCPad) * 4;
  if (o < sums) o = sums;
  m.list = o;  // (column, value bits)
  o += (size_t)kBandRows * kBandList * 8;
  m.rp = o;
  o += (kBandRows + 1) * 4;
  m.cnt = o;
  o += kBandRows * 4;
  m.bar = (o + 7) & ~size_t(7);
  m.bytes = m.bar + 8;
  return m;
}

__global__ void __launch_bounds__(kSpmmCta, 6)
    spmm_band_mma_kernel(SpmmArgs<uint16_t> a, const __grid_constant__ CUtensorMap tm, int halo,
                         int *status) {
  const int win = band_mma_win(halo);
  const int pitch = win + kBandAPad;
  const BandMmaSmem L = band_mma_smem(win);
  extern __shared__ __align__(1024) unsigned char swz[];  // the 128-byte swizzle's period
  float *at = reinterpret_cast<float *>(swz + L.at);  // [kBandRows][pitch]
  float *sums = reinterpret_cast<float *>(swz);       // [2][kBandRows][68], after the product
  int2 *list = reinterpret_cast<int2 *>(swz + L.list);
  int *rp = reinterpret_cast<int *>(swz + L.rp);
  int *cnt = reinterpret_cast<int *>(swz + L.cnt);
  uint64_t *bar = reinterpret_cast<uint64_t *>(swz + L.bar);
  const int t = threadIdx.x, lane = t & 31;
  const int M = a.M;
  const int i0 = blockIdx.x * kBandRows;
  const int jw0 = (int)((long long)i0 * a.K / M) - halo;
  const uint32_t b = sm_u32(bar);
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b),
                 "r"((uint32_t)(win * 128))
                 : "memory");
    // x = the slab's first column (a multiple of 64 elements), y = the
    // window's first row (negative at the top edge: zero-filled)
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(sm_u32(swz)),
        "l"(&tm), "r"((int)(blockIdx.y * kBandCols)), "r"(jw0), "r"(b)
        : "memory");
  }
  // Scatter the block's nonzeros, SQ per thread per pass with every load in flight;
  // the first pass loads before the tile is cleared.  An exchange puts a value in
  // the tile; where it returns another entry of the same position, that one is added
  // back (the native exchange is one instruction, an add of floats in shared memory a
  // loop).
  constexpr int SQ = 20;
  const int k_beg = __ldg(a.row_ptr + i0), k_end = __ldg(a.row_ptr + min(i0 + kBandRows, M));
  int cj[SQ];
  float cv[SQ];
  auto load = [&](int n0) {  // nonzeros k_beg + n0 + t + 128 q
#pragma unroll
    for (int q = 0; q < SQ; ++q) {
      const bool has = n0 + t + q * kSpmmCta < k_end - k_beg;
      cj[q] = has ? __ldg(a.col + (k_beg + n0 + t + q * kSpmmCta)) : 0;
      cv[q] = has ? ld_val(a.val, k_beg + n0 + t + q * kSpmmCta) : 0.0f;
    }
  };
  load(0);
  for (int e = t; e < kBandRows * pitch / 4; e += kSpmmCta)
    reinterpret_cast<float4 *>(at)[e] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (t <= kBandRows) rp[t] = __ldg(a.row_ptr + min(i0 + t, M));
  if (t < kBandRows) cnt[t] = 0;
  __syncthreads();
  for (int n0 = 0; n0 < k_end - k_beg; n0 += SQ * kSpmmCta) {
    if (n0 > 0) load(n0);
    int r = 0;  // the last row whose start is <= the thread's first nonzero
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (r + step <= kBandRows - 1 && rp[r + step] - k_beg <= n0 + t) r += step;
    int rend = rp[r + 1] - k_beg;
#pragma unroll
    for (int q = 0; q < SQ; ++q) {
      const int n = n0 + t + q * kSpmmCta;
      if (n < k_end - k_beg) {
        while (n >= rend) rend = rp[++r + 1] - k_beg;  // n < rp[kBandRows] - k_beg
        const unsigned d = (unsigned)(cj[q] - jw0);
        if (d < (unsigned)win) {
          float *cell = at + r * pitch + d;
          const float old = atomicExch(cell, cv[q]);
          if (old != 0.0f) atomicAdd(cell, old);
        } else {
          const int slot = atomicAdd(cnt + r, 1);
          if (slot < kBandList) list[r * kBandList + slot] = make_int2(cj[q], __float_as_int(cv[q]));
        }
      }
    }
  }
  __syncthreads();
  if (!window_wait(b)) {
    if (t == 0) atomicExch(status, SEGTACO_ETIMEOUT);
    window_wait(b);  // the copy may still land: wait for it once more, bounded
    return;
  }
  // ---- the tile product --------------------------------------------------
  float acc[8][4];
#pragma unroll
  for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
  const int w = t >> 5;
  const int steps = win / 16, half = (steps + 1) / 2;
  const int s0 = w < 2 ? 0 : half, s1 = w < 2 ? half : steps;
  // A fragment: rows 16 (w & 1) + lane / 4 (and + 8), columns 2 (lane % 4) (and + 8)
  const float *arow = at + (16 * (w & 1) + (lane >> 2)) * pitch + 2 * (lane & 3);
  // B fragments of two n-tiles: lanes 0-15 rows k .. k+15 of columns 8n, 16-31 of 8n + 8
  const uint32_t brow = sm_u32(swz) + (uint32_t)(lane & 15) * 128;
  uint32_t least = 0xffffffffu;  // the tile's smallest nonzero magnitude
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    uint32_t hi[4], mid[4], lo[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // a0: row, a1: row + 8, a2, a3: columns + 8
      const float2 v =
          *reinterpret_cast<const float2 *>(arow + (q & 1) * 8 * pitch + 16 * s + (q >> 1) * 8);
      least = min_nonzero(min_nonzero(least, v.x), v.y);
      split3(v.x, v.y, hi[q], mid[q], lo[q]);
    }
    const uint32_t row = brow + (uint32_t)s * 16 * 128;
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
      uint32_t bf[4];
      ldmatrix_x4_trans(bf, row + ((((uint32_t)(2 * n2 + (lane >> 4))) ^ ((row >> 7) & 7)) << 4));
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float d[4];
        mma_bf16_zero(d, lo, bf[2 * h], bf[2 * h + 1]);
        mma_bf16(d, mid, bf[2 * h], bf[2 * h + 1]);
        mma_bf16(d, hi, bf[2 * h], bf[2 * h + 1]);
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[2 * n2 + h][q] += d[q];
      }
    }
  }
  float amax = 0.0f;  // the sums' largest magnitude, or NaN
#pragma unroll
  for (int q = 0; q < 32; ++q) amax = max_nan(amax, acc[q / 4][q % 4]);
  const bool odd = !(fabsf(amax) <= FLT_MAX) || least < kSplitMin;
  const bool direct = __syncthreads_or(odd) != 0;  // the tile and the window are free now
  {
    float *s = sums + (w >> 1) * kBandRows * (kBandCols + kBandCPad) +
               (16 * (w & 1) + (lane >> 2)) * (kBandCols + kBandCPad) + 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      *reinterpret_cast<float2 *>(s + 8 * n) = make_float2(acc[n][0], acc[n][1]);
      *reinterpret_cast<float2 *>(s + 8 * (kBandCols + kBandCPad) + 8 * n) =
          make_float2(acc[n][2], acc[n][3]);
    }
  }
  __syncthreads();
  // ---- off-band nonzeros and the store: eight lanes per row, 8 columns each ----
  const int l = t & 7;
  const int c0 = blockIdx.y * kBandCols + 8 * l;
  if (c0 >= a.N) return;  // N is a multiple of 16
  auto gather = [&](int j) {
    return __ldg(reinterpret_cast<const uint4 *>(a.B + (size_t)(unsigned)j * a.ldb + c0));
  };
#pragma unroll 1
  for (int r = t >> 3; r < kBandRows; r += kSpmmCta / 8) {
    if (i0 + r >= M) return;
    float s[8];
    auto add = [&](float x, const uint4 &g) {
      const uint32_t wd[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s[2 * q] = fmaf(x, bf16lo(wd[q]), s[2 * q]);
        s[2 * q + 1] = fmaf(x, bf16hi(wd[q]), s[2 * q + 1]);
      }
    };
    const int n = cnt[r];
    if (direct) {
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q] = 0.0f;
      for (int k = rp[r]; k < rp[r + 1]; ++k) add(ld_val(a.val, k), gather(__ldg(a.col + k)));
    } else {
      const float *p0 = sums + r * (kBandCols + kBandCPad) + 8 * l;
      const float *p1 = p0 + kBandRows * (kBandCols + kBandCPad);
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q] = p0[q] + p1[q];
      if (n <= kBandList) {
        for (int e0 = 0; e0 < n; e0 += 8) {
          uint4 g[8];
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int2 it = list[r * kBandList + (e0 + e < n ? e0 + e : e0)];
            g[e] = gather(it.x);
            x[e] = __int_as_float(it.y);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (e0 + e < n) add(x[e], g[e]);
        }
      } else {
        // more off-band nonzeros than the list holds: walk the row
        for (int k = rp[r]; k < rp[r + 1]; ++k) {
          const int j = __ldg(a.col + k);
          if ((unsigned)(j - jw0) >= (unsigned)win) add(ld_val(a.val, k), gather(j));
        }
      }
    }
    float *dst = a.C + (long long)(i0 + r) * a.ldc + c0;
    __stcs(reinterpret_cast<float4 *>(dst), make_float4(s[0], s[1], s[2], s[3]));
    __stcs(reinterpret_cast<float4 *>(dst) + 1, make_float4(s[4], s[5], s[6], s[7]));
  }
}

// cuTensorMapEncodeTiled from the driver, looked up once.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

template <typename BT, int V, int G> int launch_window_variant(const SpmmLaunch &L, cudaStream_t s) {
  constexpr int W = G * V;
  const long long rows_blk = (long long)kSpmmWarps * L.rows_per_unit;
  const long long wrows = rows_blk + 2LL * L.window_halo;
  if (wrows > 256)
    return set_error(SEGTACO_EINVAL, "window of %lld rows (4*rows_per_unit + 2*halo) > 256",
                     wrows);
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return set_error(SEGTACO_EUNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  CUtensorMap tm;
  const cuuint64_t dims[2] = {(cuuint64_t)L.N, (cuuint64_t)L.K};
  const cuuint64_t strides[1] = {(cuuint64_t)L.ldb * sizeof(BT)};
  const cuuint32_t box[2] = {(cuuint32_t)W, (cuuint32_t)wrows};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = enc(&tm, sizeof(BT) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                               : CU_TENSOR_MAP_DATA_TYPE_UINT16,
                         2, const_cast<void *>(L.B), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(SEGTACO_EINVAL, "window: tensor map of B rejected (CUresult %d)", (int)r);
  const size_t bytes = (((size_t)wrows * W * sizeof(BT) + 15) & ~size_t(15)) + 16;
  auto kern = spmm_window_kernel<BT, V, G>;
  // The shared-memory opt-in, once per device.
  static std::atomic<unsigned long long> opted{0};
  int dev = 0;
  SEGTACO_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(opted.load() & bit)) {
    SEGTACO_TRY(check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)(64 * 1024)),
                           "cudaFuncSetAttribute(spmm_window_kernel)"));
    opted.fetch_or(bit);
  }
  if (bytes > 64 * 1024) return set_error(SEGTACO_EINVAL, "window of %zu bytes > 64 KB", bytes);
  int *status = nullptr;
  SEGTACO_TRY(tma_status_ptr(&status));
  const SpmmArgs<BT> a = make_spmm_args<BT>(L);
  const dim3 grid = spmm_grid(L);
  kern<<<grid, kSpmmCta, bytes, s>>>(a, tm, L.window_halo, status);
  return check_launch("spmm_window_kernel");
}

template <typename BT> int launch_window(const SpmmLaunch &L, cudaStream_t s) {
  switch (L.V * 100 + L.G) {
#define SEGTACO_WINDOW_CASE(V, G) \
  case V * 100 + G:               \
    return launch_window_variant<BT, V, G>(L, s);
    SEGTACO_WINDOW_CASE(8, 4)
    SEGTACO_WINDOW_CASE(4, 8)
    SEGTACO_WINDOW_CASE(8, 8)
    SEGTACO_WINDOW_CASE(4, 16)
    SEGTACO_WINDOW_CASE(8, 16)
    SEGTACO_WINDOW_CASE(1, 32)
    SEGTACO_WINDOW_CASE(2, 32)
#undef SEGTACO_WINDOW_CASE
    default:
      break;
  }
  if constexpr (sizeof(BT) == 2) {
    if (L.V == 16 && L.G == 4) return launch_window_variant<BT, 16, 4>(L, s);
  }
  return set_error(SEGTACO_EUNSUPPORTED, "window: no variant V=%d G=%d", L.V, L.G);
}

// The band kernels: fp32 B with multiply-adds, bf16 B on the tensor cores (its
// window in the 128-byte swizzle, rows rounded up to whole 16-row steps).
template <typename BT> int launch_band_typed(const SpmmLaunch &L, cudaStream_t s) {
  constexpr bool kMma = sizeof(BT) == 2;
  const int win = kMma ? band_mma_win(L.band_halo) : kBandRows + 2 * L.band_halo;
  if (L.band_halo < 0 || win > 256)
    return set_error(SEGTACO_EINVAL, "band window of %d rows (32 + 2*halo) > 256", win);
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return set_error(SEGTACO_EUNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  CUtensorMap tm;
  const cuuint64_t dims[2] = {(cuuint64_t)L.N, (cuuint64_t)L.K};
  const cuuint64_t strides[1] = {(cuuint64_t)L.ldb * sizeof(BT)};
  const cuuint32_t box[2] = {(cuuint32_t)kBandCols, (cuuint32_t)win};
  const cuuint32_t es[2] = {1, 1};
  const CUresult r = enc(&tm, sizeof(BT) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                               : CU_TENSOR_MAP_DATA_TYPE_UINT16,
                         2, const_cast<void *>(L.B), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE,
                         kMma ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return set_error(SEGTACO_EINVAL, "band: tensor map of B rejected (CUresult %d)", (int)r);
  void (*kern)(SpmmArgs<BT>, const CUtensorMap, int, int *);
  size_t bytes;
  if constexpr (kMma) {
    kern = spmm_band_mma_kernel;
    bytes = band_mma_smem(win).bytes;
  } else {
    kern = spmm_band_kernel;
    bytes = band_smem(win).bytes;
  }
  static std::atomic<unsigned long long> opted{0};
  int dev = 0;
  SEGTACO_TRY(check_cuda(cudaGetDevice(&dev), "cudaGetDevice"));
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(opted.load() & bit)) {
    SEGTACO_TRY(check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)(200 * 1024)),
                           "cudaFuncSetAttribute(spmm_band_kernel)"));
    opted.fetch_or(bit);
  }
  if (bytes > 200 * 1024) return set_error(SEGTACO_EINVAL, "band tiles of %zu bytes > 200 KB", bytes);
  int *status = nullptr;
  SEGTACO_TRY(tma_status_ptr(&status));
  const SpmmArgs<BT> a = make_spmm_args<BT>(L);
  const dim3 grid((unsigned)((L.M + kBandRows - 1) / kBandRows),
                  (unsigned)((L.N + kBandCols - 1) / kBandCols), 1);
  kern<<<grid, kSpmmCta, bytes, s>>>(a, tm, L.band_halo, status);
  return check_launch("spmm_band_kernel");
}

// Nonzeros within `halo` of the diagonal (row i scaled to column i*K/M).
// A warp per 32 consecutive rows: lane l reads the bounds of row r0 + l, then
// the warp walks each of the 32 rows with its lanes striding the row's
// nonzeros (coalesced; a row of 50,000 nonzeros costs its warp ~1,600 steps
// instead of one thread 50,000).
__global__ void band_stats_kernel(const int *__restrict__ row_ptr, const int *__restrict__ col,
                                  int M, int K, int halo, unsigned long long *out) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  unsigned long long n = 0;
  const long long warps = (long long)gridDim.x * (blockDim.x / 32);
  for (long long r0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32; r0 < M;
       r0 += warps * 32) {
    const long long rl = r0 + lane;
    const int b = rl < M ? __ldg(row_ptr + rl) : 0;
    const int e = rl < M ? __ldg(row_ptr + rl + 1) : 0;
    for (int i = 0; i < 32; ++i) {
      const int bi = __shfl_sync(FULL, b, i), ei = __shfl_sync(FULL, e, i);
      const long long d = (r0 + i) * (long long)K / M;
      for (int p = bi + lane; p < ei; p += 32) {
        const long long c = __ldg(col + p);
        n += (c >= d - halo && c <= d + halo) ? 1 : 0;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(out, n);
}

}  // namespace

int launch_band_stats(const int *row_ptr, const int *col, int M, int K, int halo,
                      unsigned long long *out, cudaStream_t s) {
  SEGTACO_TRY(check_cuda(cudaMemsetAsync(out, 0, sizeof(unsigned long long), s), "memset"));
  if (M <= 0) return SEGTACO_OK;
  long long blocks = (M + 255) / 256;  // 8 warps of 32 rows per block
  if (blocks > 4096) blocks = 4096;
  band_stats_kernel<<<(unsigned)blocks, 256, 0, s>>>(row_ptr, col, M, K, halo, out);
  return check_launch("band_stats_kernel");
}

bool window_variant_exists(int dtype, int V, int G) {
  const int k = V * 100 + G;
  if (k == 804 || k == 408 || k == 808 || k == 416 || k == 816 || k == 132 || k == 232)
    return true;
  return dtype == SEGTACO_BF16 && k == 1604;
}

int launch_spmm_window(const SpmmLaunch &L, cudaStream_t s) {
  return L.dtype == SEGTACO_BF16 ? launch_window<uint16_t>(L, s) : launch_window<float>(L, s);
}

int launch_spmm_band(const SpmmLaunch &L, cudaStream_t s) {
  return L.dtype == SEGTACO_BF16 ? launch_band_typed<uint16_t>(L, s)
                                 : launch_band_typed<float>(L, s);
}

}  // namespace segtaco

using namespace segtaco;

extern "C" int segtaco_band_stats(int32_t M, int32_t K, int64_t nnz, const int32_t *row_ptr,
                                  const int32_t *col, int32_t halo, int64_t *in_band,
                                  void *stream) {
  if (M < 0 || K < 0 || nnz < 0 || halo < 0 || !in_band)
    return set_error(SEGTACO_EINVAL, "segtaco_band_stats: bad arguments");
  *in_band = 0;
  if (M == 0 || nnz == 0) return SEGTACO_OK;
  if (!row_ptr || !col) return set_error(SEGTACO_EINVAL, "segtaco_band_stats: NULL CSR");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Scratch scratch(nullptr, 0, s);
  SEGTACO_TRY(scratch.reserve(256));
  auto *d = static_cast<unsigned long long *>(scratch.take(sizeof(unsigned long long)));
  SEGTACO_TRY(launch_band_stats(row_ptr, col, M, K, halo, d, s));
  unsigned long long h = 0;
  SEGTACO_TRY(check_cuda(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, s), "copy"));
  SEGTACO_TRY(check_cuda(cudaStreamSynchronize(s), "sync"));
  *in_band = (int64_t)h;
  return SEGTACO_OK;
}

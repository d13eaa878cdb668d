// sddmm_band.cu -- SDDMM on banded matrices: out[k] = val[k] * <X[i], Y[j]> for
// the nonzeros (i, j) of A that lie near the diagonal.
//
// The warp-block SDDMM kernels (sddmm.cu) gather Y[j] once per nonzero (256
// bytes for D = 64 fp32) and keep X[i] in registers while a row lasts; on a
// banded matrix those gathers hit L1 and the load/store data pipe bounds them.
// Rows i and i + 1 share almost all of their band, so here a CTA owns 32
// consecutive rows and computes every dot product of its band at once: the dense
// tile <X[i0 + r], Y[jw0 + j]> of its 32 rows and the 32 + 2 kSbHalo window rows
// around the diagonal (column i0 * K / M of its first row), a 32 x 96 x 64
// contraction that runs as mma.m16n8k16 with fp32 accumulation.  bf16 factors take one
// product per step.  fp32 factors are split into three bf16 parts (hi + mid + lo, rounded
// to nearest: mma.cuh) and six of the nine products summed per step of 16 elements,
// hi x hi by itself and the others the smallest first, both then added to the running
// sum in fp32; what is left out is below 2^-24 of a product, either way.  Warp w takes window rows 24 w .. +23 and
// all 32 rows; a lane's four elements of a row are one load of 16 (8) bytes, in the
// same order for X and Y, so neither needs transposing or, for Y, shared memory.  The
// tile then goes to shared memory and every nonzero of the block reads its dot product
// there.  Nonzeros outside the window (off band) are listed (kSbList per block) and then
// computed by 16 lanes each, 4 elements per lane from the X block and Y[j] in global
// memory, summed by shuffles; beyond the list a thread computes the dot product alone.
// The tile holds dot products for window positions without a nonzero too (96 per row
// instead of ~2 kSbHalo + 1).  Splitting an infinity or NaN makes NaN of both, and a
// value next to the largest splits into infinite parts; one below 2^-103 has no three
// parts.  A CTA with fp32 factors that meets such a sum or value computes its dot
// products one by one instead.
//
// What bounds it: the sampling of the tile and the off-band gathers, each about half
// of what the product leaves (without the off-band list 136 us, without the product
// 158).  Measured on GB300, banded-plus-random 262,144 rows, half band 32, 8 off-band
// nonzeros per row, multiply-adds on 4 x 6 register tiles -> here: fp32 246 -> 191 us,
// bf16 222 -> 150; error against FP64 1.4e-7 -> 6.0e-8 and 5.0e-8 -> 4.6e-8.  Eight
// off-band steps in flight instead of four 206 -> 195 us; 20 sampled nonzeros in flight
// instead of 10 spill (258); a warp per row in the sampling 252.
#include <cfloat>

#include "common.cuh"
#include "internal.h"
#include "mma.cuh"

namespace segtaco {
namespace {

constexpr int kSbRows = 32;                     // rows per CTA
constexpr int kSbHalo = 32;                     // window rows on either side
constexpr int kSbWin = kSbRows + 2 * kSbHalo;  // 96 window rows
constexpr int kSbD = 64;                        // dot-product length
constexpr int kSbTP = kSbWin + 8;  // pitch of the tile: conflict-free 8-byte stores
constexpr int kSbXP = kSbD + 16;   // pitch of the X block: conflict-free 16-byte loads
constexpr int kSbCta = 128;
constexpr int kSq = 10;       // nonzeros in flight per thread of the sampling pass
constexpr int kSbList = 512;  // off-band nonzeros listed per block

// Four consecutive X or Y values as floats (fp32: 16 bytes; bf16: 8 bytes).
template <typename XT> __device__ __forceinline__ float4 sb_ld4(const XT *p) {
  if constexpr (sizeof(XT) == 4) {
    return __ldg(reinterpret_cast<const float4 *>(p));
  } else {
    const uint2 x = __ldg(reinterpret_cast<const uint2 *>(p));
    return make_float4(bf16lo(x.x), bf16hi(x.x), bf16lo(x.y), bf16hi(x.y));
  }
}
// Two floats as a bf16 pair (exact for values that are bf16).
__device__ __forceinline__ uint32_t sb_pair(float x, float y) {
  return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

template <typename XT>
__global__ void __launch_bounds__(kSbCta, sizeof(XT) == 4 ? 5 : 6)  // 96 / 80 registers
    sddmm_band_kernel(int M, int K, const int *__restrict__ row_ptr, const int *__restrict__ col,
                      const float *__restrict__ val, const XT *__restrict__ X,
                      const XT *__restrict__ Y, long long ldx, long long ldy,
                      float *__restrict__ out) {
  constexpr bool kSplit = sizeof(XT) == 4;
  constexpr int kParts = kSplit ? 3 : 1;
  __shared__ __align__(16) float xr[kSbRows * kSbXP];    // X block, row-major
  __shared__ __align__(16) float tile[kSbRows * kSbTP];  // tile[r][window row]
  __shared__ int4 lst[kSbList];                          // (k, row, column, value bits)
  __shared__ int rp[kSbRows + 1];
  __shared__ int lcount;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int i0 = blockIdx.x * kSbRows;
  const int jw0 = (int)((long long)i0 * K / M) - kSbHalo;
  // Y: lane g = lane / 4 of n-tile n holds window row 24 w + 8 n + g, elements
  // 16 s + 4 (lane % 4) .. +3 in step s; rows outside [0, K) are zeros.
  const int e4 = 4 * (lane & 3);
  const XT *yrow[3];
  bool yok[3];
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const int j = jw0 + 24 * w + 8 * n + (lane >> 2);
    yok[n] = j >= 0 && j < K;
    yrow[n] = Y + (size_t)(yok[n] ? j : 0) * ldy + e4;
  }
  uint32_t least = 0xffffffffu;  // the fp32 factors' smallest nonzero magnitude
  auto note = [&](const float4 &v) {
    if constexpr (kSplit)
      least = min_nonzero(min_nonzero(min_nonzero(min_nonzero(least, v.x), v.y), v.z), v.w);
  };
  auto load_y = [&](int s, float4(&y)[3]) {
#pragma unroll
    for (int n = 0; n < 3; ++n)
      y[n] = yok[n] ? sb_ld4<XT>(yrow[n] + 16 * s) : make_float4(0, 0, 0, 0);
  };
  float4 ycur[3];
  load_y(0, ycur);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int e = t + u * kSbCta;  // 0 .. 511: row e / 16, elements 4 (e % 16) ..
    const int i = i0 + e / (kSbD / 4);
    const float4 x =
        i < M ? sb_ld4<XT>(X + (size_t)i * ldx + 4 * (e % (kSbD / 4))) : make_float4(0, 0, 0, 0);
    *reinterpret_cast<float4 *>(xr + (e / (kSbD / 4)) * kSbXP + 4 * (e % (kSbD / 4))) = x;
    note(x);
  }
  if (t <= kSbRows) rp[t] = __ldg(row_ptr + min(i0 + t, M));
  if (t == 0) lcount = 0;
  __syncthreads();
  // ---- the dense tile ----
  float acc[2][3][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 3; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
#pragma unroll 1
  for (int s = 0; s < kSbD / 16; ++s) {
    float4 ynext[3];
    if (s + 1 < kSbD / 16) load_y(s + 1, ynext);
    uint32_t xa[2][kParts][4];  // [m-tile][part][register]
#pragma unroll
    for (int h = 0; h < 4; ++h) {  // rows g, g + 8, g + 16, g + 24
      const float4 x = *reinterpret_cast<const float4 *>(xr + (8 * h + (lane >> 2)) * kSbXP +
                                                         16 * s + e4);
      uint32_t(&p)[kParts][4] = xa[h >> 1];
      const int q = h & 1;  // registers q (elements 0, 1) and q + 2 (elements 2, 3)
      if constexpr (kSplit) {
        split3(x.x, x.y, p[0][q], p[1][q], p[2][q]);
        split3(x.z, x.w, p[0][q + 2], p[1][q + 2], p[2][q + 2]);
      } else {
        p[0][q] = sb_pair(x.x, x.y);
        p[0][q + 2] = sb_pair(x.z, x.w);
      }
    }
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      uint32_t yb[kParts][2];
      const float4 y = ycur[n];
      note(y);
      if constexpr (kSplit) {
        split3(y.x, y.y, yb[0][0], yb[1][0], yb[2][0]);
        split3(y.z, y.w, yb[0][1], yb[1][1], yb[2][1]);
      } else {
        yb[0][0] = sb_pair(y.x, y.y);
        yb[0][1] = sb_pair(y.z, y.w);
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        float d[4];
        mma_bf16_zero(d, xa[m][0], yb[0][0], yb[0][1]);  // hi hi
        if constexpr (kSplit) {
          float e[4];
          mma_bf16_zero(e, xa[m][0], yb[2][0], yb[2][1]);  // hi lo
          mma_bf16(e, xa[m][2], yb[0][0], yb[0][1]);       // lo hi
          mma_bf16(e, xa[m][1], yb[1][0], yb[1][1]);       // mid mid
          mma_bf16(e, xa[m][0], yb[1][0], yb[1][1]);       // hi mid
          mma_bf16(e, xa[m][1], yb[0][0], yb[0][1]);       // mid hi
#pragma unroll
          for (int q = 0; q < 4; ++q) d[q] += e[q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[m][n][q] += d[q];
      }
    }
#pragma unroll
    for (int n = 0; n < 3; ++n) ycur[n] = ynext[n];
  }
  constexpr int SQ = kSq;
  const int k_beg = rp[0], len = rp[kSbRows] - k_beg;
  int cj[SQ];
  float cv[SQ];
  auto load_nz = [&](int n0) {
#pragma unroll
    for (int u = 0; u < SQ; ++u) {
      const bool has = n0 + u * kSbCta < len;
      cj[u] = has ? __ldg(col + (k_beg + n0 + u * kSbCta)) : 0;
      cv[u] = has && val ? __ldg(val + (k_beg + n0 + u * kSbCta)) : 1.0f;
    }
  };
  load_nz(t);
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      float *dst = tile + (16 * m + (lane >> 2)) * kSbTP + 24 * w + 8 * n + 2 * (lane & 3);
      *reinterpret_cast<float2 *>(dst) = make_float2(acc[m][n][0], acc[m][n][1]);
      *reinterpret_cast<float2 *>(dst + 8 * kSbTP) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
  // An infinity or NaN among the tile's sums, or a tiny factor: every dot product by itself.
  float amax = 0.0f;
  if constexpr (kSplit) {
#pragma unroll
    for (int q = 0; q < 24; ++q) amax = max_nan(amax, acc[q / 12][q / 4 % 3][q % 4]);
  }
  const bool direct = __syncthreads_or(kSplit && (!(fabsf(amax) <= FLT_MAX) || least < kSplitMin)) != 0;
  // The block's nonzeros, coalesced, kSq per thread per pass.
  for (int n0 = t; n0 < len; n0 += SQ * kSbCta) {
    if (n0 != t) load_nz(n0);
    int r = 0;  // the last row whose start is <= the thread's first nonzero
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (r + step <= kSbRows - 1 && rp[r + step] - k_beg <= n0) r += step;
    int rend = rp[r + 1] - k_beg;
#pragma unroll
    for (int u = 0; u < SQ; ++u) {
      const int n = n0 + u * kSbCta;
      if (n < len) {
        while (n >= rend) rend = rp[++r + 1] - k_beg;  // n < rp[kSbRows] - k_beg
        const int k = k_beg + n;
        const unsigned dj = (unsigned)(cj[u] - jw0);
        if (dj < (unsigned)kSbWin && !direct) {
          out[k] = cv[u] * tile[r * kSbTP + dj];
        } else {
          const int slot = atomicAdd(&lcount, 1);
          if (slot < kSbList) {
            lst[slot] = make_int4(k, r, cj[u], __float_as_int(cv[u]));
          } else {
            // past the list: the dot product by this thread alone
            const XT *yr = Y + (size_t)(unsigned)cj[u] * ldy;
            float sum = 0.0f;
#pragma unroll 4
            for (int q = 0; q < kSbD / 4; ++q) {
              const float4 y = sb_ld4<XT>(yr + 4 * q);
              const float4 x = *reinterpret_cast<const float4 *>(xr + r * kSbXP + 4 * q);
              sum = fmaf(x.x, y.x, sum);
              sum = fmaf(x.y, y.y, sum);
              sum = fmaf(x.z, y.z, sum);
              sum = fmaf(x.w, y.w, sum);
            }
            out[k] = cv[u] * sum;
          }
        }
      }
    }
  }
  __syncthreads();
  // Listed off-band nonzeros: 16 lanes each (lane l: elements 4l .. 4l+3); a
  // warp takes two per step, eight steps with their gathers in flight at once,
  // and every lane of it takes part in the shuffles.
  const int n = min(lcount, kSbList);
  const int hw = (t >> 4) & 1, l = t & 15;
  constexpr int kSteps = 8, kStride = kSbCta / 16;  // 8 entries per step over the CTA
  for (int e0 = 2 * w; e0 < n; e0 += kSteps * kStride) {
    int4 it[kSteps];
    float4 y[kSteps];
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
      const int e = e0 + u * kStride + hw;
      it[u] = lst[e < n ? e : e0];  // past the list: entry e0 again, not stored
      y[u] = sb_ld4<XT>(Y + (size_t)(unsigned)it[u].z * ldy + 4 * l);
    }
#pragma unroll
    for (int u = 0; u < kSteps; ++u) {
      const float4 x = *reinterpret_cast<const float4 *>(xr + it[u].y * kSbXP + 4 * l);
      float s = x.x * y[u].x;
      s = fmaf(x.y, y[u].y, s);
      s = fmaf(x.z, y[u].z, s);
      s = fmaf(x.w, y[u].w, s);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, 16);
      if (e0 + u * kStride + hw < n && l == 0) out[it[u].x] = __int_as_float(it[u].w) * s;
    }
  }
}

}  // namespace

bool sddmm_band_applies(int x_dtype, int D, long long ldx, long long ldy, const void *X,
                        const void *Y) {
  const int esz = x_dtype == SEGTACO_BF16 ? 2 : 4;
  const uintptr_t al = (uintptr_t)X | (uintptr_t)Y;
  return D == kSbD && ldx % 4 == 0 && ldy % 4 == 0 && (al % (4 * esz)) == 0;
}

int launch_sddmm_band(int M, int K, long long nnz, const int *row_ptr, const int *col,
                      const float *val, const void *X, const void *Y, int x_dtype, long long ldx,
                      long long ldy, int D, float *out, cudaStream_t s) {
  if (nnz == 0 || M == 0) return SEGTACO_OK;
  if (!sddmm_band_applies(x_dtype, D, ldx, ldy, X, Y))
    return set_error(SEGTACO_EINVAL,
                     "sddmm band kernel: needs D = 64, ldx and ldy multiples of 4 and X, Y "
                     "aligned to 4 elements");
  const dim3 grid((unsigned)((M + kSbRows - 1) / kSbRows));
  if (x_dtype == SEGTACO_BF16)
    sddmm_band_kernel<uint16_t><<<grid, kSbCta, 0, s>>>(
        M, K, row_ptr, col, val, static_cast<const uint16_t *>(X),
        static_cast<const uint16_t *>(Y), ldx, ldy, out);
  else
    sddmm_band_kernel<float><<<grid, kSbCta, 0, s>>>(M, K, row_ptr, col, val,
                                                     static_cast<const float *>(X),
                                                     static_cast<const float *>(Y), ldx, ldy, out);
  return check_launch("sddmm_band_kernel");
}

}  // namespace segtaco

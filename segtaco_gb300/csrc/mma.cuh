// mma.cuh -- warp-level tensor-core steps of the band kernels (bf16 operands, fp32
// accumulation) and the split of fp32 values into bf16 parts.
#pragma once

#include <stdint.h>

namespace segtaco {

// x = hi + mid + lo for two values, each part a bf16 pair, rounded to nearest, so that
// |mid| <= 2^-8 and |lo| <= 2^-17 of x's leading bit and neither has x's sign for good: the
// products of mid and lo that a caller leaves out are below 2^-24 of the whole and
// cancel (cut off instead, mid and lo reach 2^-7 and 2^-15, all one way: up to 4.7e-7
// of a product).  Values from the middle between bf16's largest and 2^128 on give
// infinite and NaN parts, as infinities and NaN do.
__device__ __forceinline__ uint32_t round_bf16x2(float x, float y) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
  return r;
}
__device__ __forceinline__ void split3(float x, float y, uint32_t &hi, uint32_t &mid,
                                       uint32_t &lo) {
  hi = round_bf16x2(x, y);
  const float xr = x - __uint_as_float(hi << 16);
  const float yr = y - __uint_as_float(hi & 0xffff0000u);
  mid = round_bf16x2(xr, yr);
  lo = __byte_perm(__float_as_uint(xr - __uint_as_float(mid << 16)),
                   __float_as_uint(yr - __uint_as_float(mid & 0xffff0000u)), 0x7632);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a x b (from zero).
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                              uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// Smallest nonzero magnitude: the smaller of `least` (start: 0xffffffff) and twice x's
// bits less one (zeros wrap to the top).  Below kSplitMin the parts of a value can fall
// under bf16's smallest normal number, 2^-126, where the last bits of `lo` are lost or left
// to the tensor cores' treatment of subnormals; a kernel that splits sends such values
// another way.
constexpr uint32_t kSplitMin = 2u * ((127u - 103u) << 23) - 1u;  // |x| = 2^-103
__device__ __forceinline__ uint32_t min_nonzero(uint32_t least, float x) {
  const uint32_t b = __float_as_uint(x);
  return min(least, b + b - 1u);
}
// The larger magnitude (its sign is no use), NaN if either is NaN.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.xorsign.abs.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

}  // namespace segtaco

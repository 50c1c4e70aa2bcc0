// f32x2.cuh — packed pairs of FP32 values (one instruction issues both).
#pragma once

#include <cuda_runtime.h>

namespace gg {

// Two FP32 lanes in one 64-bit register pair; every operation rounds each
// half as the scalar one does.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a + b for an `a` that is a product: written as add2(mul2(..), b) it was
// contracted to a fused multiply-add and the sums differed by an ulp, so the
// sum is a fused multiply-add itself, of a factor 1 that the compiler does
// not know (`ones` comes with the kernel's arguments).
__device__ __forceinline__ f32x2 add_product2(f32x2 a, f32x2 ones, f32x2 b) { return fma2(a, ones, b); }
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The correctly rounded square roots of two normal numbers: an approximate
// reciprocal root y, then s = x y and one residual correction
// s + (x - s^2) (y / 2) in fused arithmetic (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990).
// tests/test_upsample_pairs.py compares it with sqrtf for every float from
// 1e-30 up.  An infinite or NaN operand gives NaN.
__device__ __forceinline__ f32x2 sqrt2(f32x2 x) {
  float a, b;
  unpack2(x, a, b);
  const f32x2 y = pack2(rsqrt_approx(a), rsqrt_approx(b));
  const f32x2 s = mul2(x, y);
  const f32x2 neg_s = s ^ 0x8000000080000000ull;
  return fma2(fma2(neg_s, s, x), mul2(y, pack2(0.5f, 0.5f)), s);
}

// max(x, lo) that keeps a NaN.
__device__ __forceinline__ float max_nan(float x, float lo) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(lo));
  return r;
}

}  // namespace gg

// f32x2.cuh -- packed FP32 pairs (sm_100's f32x2 instructions): two values in
// one 64-bit register pair, one instruction for both.  Each operation is the
// IEEE single-precision operation of each half, the same result as two scalar
// ones; but ptxas fuses an f2_mul whose result only feeds an f2_add or f2_sub
// (f2_fma(a, b, 0) keeps the product's own rounding).
#pragma once

namespace qpsdm {

using f2 = unsigned long long;

__device__ __forceinline__ f2 f2_pack(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 f2_dup(float a) { return f2_pack(a, a); }
__device__ __forceinline__ float2 f2_unpack(f2 r) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a + b rounded towards zero
__device__ __forceinline__ f2 f2_add_rz(f2 a, f2 b) {
  f2 r;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

}  // namespace qpsdm

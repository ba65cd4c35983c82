// f32x2.cuh -- two single-precision operations an instruction, each rounded as its scalar form.
#pragma once
#include <cuda_runtime.h>

namespace pmcmc {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return mul2(a, b); }

// A formula for one value (V = float) or two (V = F2).
template <typename V>
__device__ __forceinline__ V same(float x);
template <>
__device__ __forceinline__ float same<float>(float x) {
  return x;
}
template <>
__device__ __forceinline__ F2 same<F2>(float x) {
  return pack2(x, x);
}
__device__ __forceinline__ float fma_of(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ F2 fma_of(F2 a, F2 b, F2 c) { return fma2(a, b, c); }

}  // namespace pmcmc

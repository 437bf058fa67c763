// pdot_pairs.cuh — FP32 screening of point pairs, for passes that want one maximum or
// minimum of FP64 over all pairs: squared distances of a point to four others at a time.
#pragma once
#include "pdot_common.cuh"

namespace pdot {
namespace {

constexpr float kUnit = 5.9604645e-8f;  // 2^-24, the relative error of one FP32 rounding

// Two FP32 operations in one instruction, each rounded as the scalar one, and a minimum
// and maximum of three that pass over a NaN as fminf and fmaxf do.
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ float unpack_low(unsigned long long r) { return __uint_as_float((unsigned)r); }
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Squared distances of the point -minus[D] (each coordinate twice) to four points from
// t on of a tile that holds its coordinates apart.
template <int D>
__device__ __forceinline__ void sqdist4(const unsigned long long* minus, const ulonglong2* c, unsigned long long* s) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const unsigned long long e0 = add2(c[d].x, minus[d]), e1 = add2(c[d].y, minus[d]);
    s[0] = d == 0 ? mul2(e0, e0) : fma2(e0, e0, s[0]);
    s[1] = d == 0 ? mul2(e1, e1) : fma2(e1, e1, s[1]);
  }
}

// The larger of `top` and the four distances.
template <int D>
__device__ __forceinline__ float max_sqdist4(const unsigned long long* minus, const ulonglong2* c, float top) {
  unsigned long long s[2];
  sqdist4<D>(minus, c, s);
  float s0, s1, s2, s3;
  unpack2(s[0], s0, s1);
  unpack2(s[1], s2, s3);
  return max3(max3(top, s0, s1), s2, s3);
}

}  // namespace
}  // namespace pdot

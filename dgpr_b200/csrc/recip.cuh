// Reciprocal, quotient, square root and reciprocal square root for the
// pointwise physics: the hardware's approximation (rcp.approx / rsqrt.approx,
// good to about 2^-22) refined by one step of Householder's iteration, of
// third order in FP64
//   1/x:       y + y (e + e^2),           e = 1 - x y
//   1/sqrt(x): y + y (e / 2 + 3 e^2 / 8), e = 1 - x y^2
// and of second order (Newton) in FP32, and for the square root and the
// quotient a step on the remainder.  Measured against the division and square
// root operators over 1e-17 .. 1e17 (FP64) and 2e-9 .. 5e8 (FP32): FP64
// reciprocal within 1.0 eps, reciprocal square root 1.2, square root equal;
// FP32 reciprocal, quotient and square root rounded to nearest (the
// refinement leaves 2^-45, so a result differs once in some 2^20).  For
// normal arguments with normal results, which densities, sound speeds and
// Jacobians are; zero, infinite and NaN arguments give NaN or infinity, as
// the quotients they replace did once they met a momentum or a pressure.
// Against the operators they have no range check, branch or call: with seven
// of them a face point, those kept the compiler from interleaving the rest
// (FP64 stage at 32^3, p = 3: 383 -> 369 us; paired FP32 stage: 250 -> 234 us).
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "pair.cuh"

namespace dgb {

__host__ __device__ __forceinline__ double rcp(double x)
{
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = ::fma(-x, y, 1.0);
  return ::fma(::fma(e, e, e), y, y);
#else
  return 1.0 / x;
#endif
}

__host__ __device__ __forceinline__ double rsqrt_(double x)
{
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = ::fma(-x * y, y, 1.0);
  return ::fma(::fma(0.375, e, 0.5), y * e, y);
#else
  return 1.0 / ::sqrt(x);
#endif
}

__host__ __device__ __forceinline__ float rcp_approx(float x)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}

__host__ __device__ __forceinline__ float rsqrt_approx(float x)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / ::sqrtf(x);
#endif
}

__host__ __device__ __forceinline__ float rcp(float x)
{
  const float y = rcp_approx(x);
  return ::fmaf(::fmaf(-x, y, 1.0f), y, y);
}

__host__ __device__ __forceinline__ float rsqrt_(float x)
{
  const float y = rsqrt_approx(x);
  return ::fmaf(0.5f * y, ::fmaf(-x * y, y, 1.0f), y);
}

__host__ __device__ __forceinline__ f2 rcp(f2 x)
{
  const f2 y(rcp_approx(x.v.x), rcp_approx(x.v.y));
  return fma(fma(-x, y, f2(1.0f)), y, y);
}

__host__ __device__ __forceinline__ f2 rsqrt_(f2 x)
{
  const f2 y(rsqrt_approx(x.v.x), rsqrt_approx(x.v.y));
  return fma(f2(f2(0.5f) * y), fma(f2(-x * y), y, f2(1.0f)), y);
}

// a / b
template <class T>
__host__ __device__ __forceinline__ T quot(T a, T b)
{
  const T r = rcp(b), q = a * r;
  const T d = fma(-q, b, a);
  return fma(d, r, q);
}

// sqrt(x) = x / sqrt(x), with the remainder of its square folded back in
template <class T>
__host__ __device__ __forceinline__ T sqrt_of(T x, T is)
{
  const T s = x * is;
  const T d = fma(-s, s, x);
  return fma(T(T(0.5) * is), d, s);
}

}  // namespace dgb

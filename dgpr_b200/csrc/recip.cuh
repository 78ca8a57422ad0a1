// Reciprocal, quotient, square root and reciprocal square root for the
// pointwise physics: the hardware's approximation (rcp.approx / rsqrt.approx,
// good to about 2^-22) refined
//   1/x:       by Newton's iteration y + y (1 - x y), twice in FP64, once in FP32,
//   1/sqrt(x): by one step of Householder's iteration of third order in FP64,
//              y + y (e / 2 + 3 e^2 / 8), e = 1 - x y^2, of Newton's in FP32
//              (y + y e / 2),
// and the quotient and the square root by a step on their remainder, exact in
// a fused multiply-add (P. Markstein, Computation of elementary functions on
// the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  What is
// left before the last rounding is 2^-39 units in the last place in FP64 and
// 2^-20 in FP32, so reciprocal, quotient, square root and the reciprocal of
// that root (rcp_from) round as the operators do but in such near-ties:
// measured within 0.5 + 2^-10 units over 1e-17 .. 1e17 (FP64) and 0.5 + 2^-20
// over 2e-9 .. 5e8 (FP32), tests/test_gpu_recip.py.  rsqrt_ itself, which
// sqrt_of and rcp_from start from, is within 1.5 units; no value of the physics
// is one of it.  For normal arguments with normal results, which densities,
// sound speeds and Jacobians are; zero, infinite and NaN arguments give NaN or
// infinity, as the quotients they replace did once they met a momentum or a
// pressure.
// Against the operators they have no range check, branch or call: with seven
// of them a face point, those kept the compiler from interleaving the rest
// (FP64 stage at 32^3, p = 3: 383 -> 369 us; paired FP32 stage: 250 -> 234 us).
// (One third-order step for the FP64 reciprocal, 1/c straight from rsqrt_ and
// the lifting scales as products are 0.6% faster per step at 32^3, p = 3, and
// reach 0.506, 0.99 and 1.0 units.)
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
  y = ::fma(::fma(-x, y, 1.0), y, y);
  return ::fma(::fma(-x, y, 1.0), y, y);
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

// 1 / x from an approximation y of it
template <class T>
__host__ __device__ __forceinline__ T rcp_from(T x, T y)
{
  return fma(fma(T(-x), y, T(1)), y, y);
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

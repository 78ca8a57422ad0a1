// Check hooks (include/dgb200_check.h): the pointwise physics the kernels use
// and its hand-written reverse mode, run on the CPU so tests can compare the
// VJPs with finite differences without a GPU; and the reciprocals and roots of
// recip.cuh on the GPU, whose arithmetic the CPU does not have.
#include <cstring>

#include "../../include/dgb200.h"
#include "../../include/dgb200_check.h"
#include "host.hpp"
#include "adjoint.hpp"
#include "physics_vjp.cuh"

using namespace dgb;

namespace {

// f(a, b) at i: rcp, quot, sqrt_of, 1 / sqrt, rsqrt_
template <class T>
__host__ __device__ T arithmetic(int f, T a, T b)
{
  const T rs = rsqrt_(a);
  switch (f) {
    case 0: return rcp(a);
    case 1: return quot(a, b);
    case 2: return sqrt_of(a, rs);
    case 3: return rcp_from(sqrt_of(a, rs), rs);
  }
  return rs;
}

// the same through the operators
template <class T>
__device__ T operators(int f, T a, T b)
{
  return f == 0 ? T(1) / a : f == 1 ? a / b : f == 2 ? sqrt(a) : T(1) / sqrt(a);
}

__global__ void arithmetic_kernel(int f, int type, long n, const double* a, const double* b, double* y)
{
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (type == 0) {
    y[i] = arithmetic<double>(f, a[i], b[i]);
    y[n + i] = operators<double>(f, a[i], b[i]);
  } else if (type == 1) {
    y[i] = arithmetic<float>(f, (float)a[i], (float)b[i]);
    y[n + i] = operators<float>(f, (float)a[i], (float)b[i]);
  } else {
    const f2 v = arithmetic<f2>(f, f2((float)a[i], (float)a[n - 1 - i]), f2((float)b[i], (float)b[n - 1 - i]));
    y[i] = v.v.x;
    y[n + n - 1 - i] = v.v.y;
  }
}

}  // namespace

extern "C" int dgb_check_arithmetic(int f, int type, long long n, const double* a, const double* b, double* y)
{
  if (f < 0 || f > 4 || type < 0 || type > 2 || n < 1 || !a || !b || !y) return DGB_ERR_ARG;
  double* d = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  cudaError_t e = cudaMalloc(&d, 4 * bytes);
  if (e != cudaSuccess) return DGB_ERR_CUDA;
  e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    arithmetic_kernel<<<(unsigned)((n + 255) / 256), 256>>>(f, type, (long)n, d, d + n, d + 2 * n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, d + 2 * n, 2 * bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? DGB_OK : DGB_ERR_CUDA;
}

extern "C" int dgb_check_prepare(int p, int precision, int curved)
{
  const int P = p + 1;
  cudaError_t e = prepare_kernels(P, precision);
  if (e == cudaSuccess) e = prepare_gauss(P, precision);
  if (e == cudaSuccess) e = prepare_adjoint(P, curved != 0);
  return e == cudaSuccess ? DGB_OK : DGB_ERR_CUDA;
}

extern "C" int dgb_check_pointwise(int which, const double* x, const double* ybar, const double* aux, double* y,
                                   double* xbar)
{
  if (!x || !aux || !y) return DGB_ERR_ARG;
  switch (which) {
    case DGB_CHECK_EULER_FLUX: {  // x = U[5], aux = {gamma}
      double F[3][5];
      euler_flux(x, aux[0], F);
      std::memcpy(y, F, sizeof F);
      if (xbar && ybar) {
        double Fb[3][5];
        std::memcpy(Fb, ybar, sizeof Fb);
        for (int i = 0; i < 5; ++i) xbar[i] = 0.;
        euler_flux_vjp(x, aux[0], Fb, xbar);
      }
      return DGB_OK;
    }
    case DGB_CHECK_EULER_FLUX_N: {  // x = U[5], aux = {gamma, n[3]}
      euler_flux_n(x, aux[0], aux + 1, y);
      if (xbar && ybar) {
        for (int i = 0; i < 5; ++i) xbar[i] = 0.;
        euler_flux_n_vjp(x, aux[0], aux + 1, ybar, xbar);
      }
      return DGB_OK;
    }
    case DGB_CHECK_VISC_FLUX:       // x = S[5] G[3][5], aux = {mu}
    case DGB_CHECK_VISC_FLUX_HEAT: {  // aux = {mu, kq}
      const double kq = which == DGB_CHECK_VISC_FLUX_HEAT ? aux[1] : 0.;
      double G[3][5], Q[3][5];
      std::memcpy(G, x + 5, sizeof G);
      visc_flux(x, G, aux[0], Q, kq);
      std::memcpy(y, Q, sizeof Q);
      if (xbar && ybar) {
        double Qb[3][5], Gb[3][5] = {};
        std::memcpy(Qb, ybar, sizeof Qb);
        for (int i = 0; i < 5; ++i) xbar[i] = 0.;
        visc_flux_vjp(x, G, aux[0], Qb, xbar, Gb, kq);
        std::memcpy(xbar + 5, Gb, sizeof Gb);
      }
      return DGB_OK;
    }
    case DGB_CHECK_VISC_RANK1:       // x = S[5] d[5], aux = {mu, n[3]}
    case DGB_CHECK_VISC_RANK1_HEAT: {  // aux = {mu, n[3], kq}
      const double kq = which == DGB_CHECK_VISC_RANK1_HEAT ? aux[4] : 0.;
      double Q[3][5];
      visc_rank1(x, x + 5, aux + 1, aux[0], Q, kq);
      std::memcpy(y, Q, sizeof Q);
      if (xbar && ybar) {
        double Qb[3][5];
        std::memcpy(Qb, ybar, sizeof Qb);
        for (int i = 0; i < 10; ++i) xbar[i] = 0.;
        visc_rank1_vjp(x, x + 5, aux + 1, aux[0], Qb, xbar, xbar + 5, kq);
      }
      return DGB_OK;
    }
    case DGB_CHECK_VISC_JUMP_N:       // x = S[5] d[5], aux = {mu, n[3]}
    case DGB_CHECK_VISC_JUMP_N_HEAT: {  // aux = {mu, n[3], kq}
      const double kq = which == DGB_CHECK_VISC_JUMP_N_HEAT ? aux[4] : 0.;
      visc_jump_n(x, x + 5, aux + 1, aux[0], y, kq);
      if (xbar && ybar) {
        for (int i = 0; i < 10; ++i) xbar[i] = 0.;
        visc_jump_n_vjp(x, x + 5, aux + 1, aux[0], ybar, xbar, xbar + 5, kq);
      }
      return DGB_OK;
    }
    case DGB_CHECK_ROE: {  // x = Ul[5] Ur[5], aux = {gamma, n[3]}
      roe_flux(x, x + 5, aux + 1, aux[0], y);
      if (xbar && ybar) {
        for (int i = 0; i < 10; ++i) xbar[i] = 0.;
        roe_flux_vjp(x, x + 5, aux + 1, aux[0], ybar, xbar, xbar + 5);
      }
      return DGB_OK;
    }
    case DGB_CHECK_BOUNDARY_STATE: {  // x = UL[5], aux = {btype, n[3], gamma, R, P, Pt, Tt, Ufr[5] (, Tw)}
      DevParams prm{};
      prm.gamma = aux[4];
      prm.R = aux[5];
      prm.P = aux[6];
      prm.Pt = aux[7];
      prm.Tt = aux[8];
      for (int r = 0; r < 5; ++r) prm.Ufr[r] = aux[9 + r];
      const int bt = (int)aux[0];
      if (bt == -8) prm.Tw = aux[14];
      if (boundary_state(bt, x, aux + 1, prm, y)) return DGB_ERR_BOUNDARY;
      if (xbar && ybar) {
        for (int i = 0; i < 5; ++i) xbar[i] = 0.;
        if (boundary_state_vjp(bt, x, aux + 1, prm, ybar, xbar)) return DGB_ERR_UNSUPPORTED;
      }
      return DGB_OK;
    }
    case DGB_CHECK_FACE_MATCH:  // x = {n_own[3], n_nbr[3], fJ_own, fJ_nbr}
      y[0] = face_mismatch(x, x + 3, 1, x[6], x[7]) ? 1. : 0.;
      return DGB_OK;
  }
  return DGB_ERR_ARG;
}

// The FP64 residual of a nodal state and its vector-Jacobian product through
// the kernels whose lanes own lines of Gauss points (lstage.cuh,
// ladjoint.cuh), which change the basis on the element as they load and store
// it: P = 2..5, meshes of full line kernels (line_kernels).  The residual takes
// the nodal kernels' face traces (enqueue_residual); the VJP, which is linear in
// lam and does not multiply a jump by more than it is worth, traces from the
// Gauss points: its error against a float64 autodifferentiation is the nodal
// kernels' (2.75e-15 against 2.77e-15 at 12^3, p = 4, 1.6e-15 to 2.4e-15
// elsewhere, within 8% of theirs either way).
//
// The nodal kernels (stage_kernel, adjA_kernel, adjB_kernel) interpolate,
// project and apply the inverse mass matrix with a thread per node, reading
// each contraction's inputs from shared memory, and the face phase's two
// tangential passes as well.  Whole calls before and now: residual 193 -> 109
// us at 24^3 p = 2, 187 -> 109 at 20^3 p = 3, 163 -> 96 at 14^3 p = 4;
// residual and VJP 709 -> 438 at 24^3 p = 2, 649 -> 427 at 20^3 p = 3,
// 477 -> 292 at 12^3 p = 4.
#include "../../include/dgb200.h"
#include "ladjoint.cuh"

namespace dgb {

namespace {

template <int P, bool CV, bool HT>
cudaError_t vjp_line(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW;
  const unsigned grid = (unsigned)((L.E + EPW - 1) / EPW);
  const auto trace = [&](auto kernel) {
    kernel<<<grid, 32, LStage<P, H>::TOTAL, st>>>(L.E, v.U, line_ops<P>(L.table), L.geo, L.gf, s.trace, L.prm);
  };
  if (!CV && L.axis)
    trace(ltrace_kernel<P, H, CV, HT, !CV, true>);
  else
    trace(ltrace_kernel<P, H, CV, HT, false, true>);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ladj_launch<P, CV, HT, true>(L, v, s, s.trace, st) : e;
}

// f(P, curved, heat) with the launch's values as types
template <class F>
cudaError_t dispatch(const KLaunch& L, F f)
{
  const auto geometry = [&](auto p) {
    const auto heat = [&](auto cv) {
      return L.prm.kq != 0. ? f(p, cv, std::true_type()) : f(p, cv, std::false_type());
    };
    return L.gv ? heat(std::true_type()) : heat(std::false_type());
  };
  switch (L.P) {
    case 2: return geometry(std::integral_constant<int, 2>());
    case 3: return geometry(std::integral_constant<int, 3>());
    case 4: return geometry(std::integral_constant<int, 4>());
    case 5: return geometry(std::integral_constant<int, 5>());
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_residual_line(const KLaunch& L, const double* U, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  if (L.prm.kq != 0.) return cudaErrorInvalidValue;  // (see enqueue_residual)
  return dispatch(L, [&](auto p, auto cv, auto) {
    return llaunch_residual_pc<decltype(p)::value, decltype(cv)::value, false>(L, U, Tin, sa, st);
  });
}

cudaError_t launch_residual_vjp_line(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  return dispatch(L, [&](auto p, auto cv, auto ht) {
    return vjp_line<decltype(p)::value, decltype(cv)::value, decltype(ht)::value>(L, v, s, st);
  });
}

}  // namespace dgb

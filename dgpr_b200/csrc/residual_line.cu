// The FP64 residual of a nodal state and its vector-Jacobian product through
// the kernels whose lanes own lines of Gauss points (lstage.cuh,
// ladjoint.cuh), which change the basis on the element as they load and store
// it: P = 2..5, meshes that take them (line_adjoint).  The residual takes
// the nodal kernels' face traces (enqueue_residual); the VJP, which is linear in
// lam and does not multiply a jump by more than it is worth, traces from the
// Gauss points: its error against a float64 autodifferentiation is the nodal
// kernels' (2.75e-15 against 2.77e-15 at 12^3, p = 4, 1.6e-15 to 2.4e-15
// elsewhere, within 8% of theirs either way).
//
// The nodal kernels (stage_kernel, adjA_kernel, adjB_kernel) interpolate,
// project and apply the inverse mass matrix with a thread per node, reading
// each contraction's inputs from shared memory, and the face phase's two
// tangential passes as well.  Whole calls on device
// arrays, nodal kernels against these: residual 183 -> 120 us at 24^3 p = 2,
// 175 -> 120 at 20^3 p = 3, 152 -> 98 at 14^3 p = 4; residual and VJP 540 ->
// 320, 491 -> 314, 482 -> 274.
#include "../../include/dgb200.h"
#include "ladjoint.cuh"

namespace dgb {

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

template <int P>
cudaError_t residual_line_p(const KLaunch& L, const double* U, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  if constexpr (P >= 2 && P <= 5)
    return L.gv ? llaunch_residual_pc<P, true, false>(L, U, Tin, sa, st)
                : llaunch_residual_pc<P, false, false>(L, U, Tin, sa, st);
  return cudaErrorInvalidValue;
}

template <int P>
cudaError_t vjp_line_p(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  if constexpr (P >= 2 && P <= 5) {
    const bool heat = L.prm.kq != 0.;
    if (L.gv) return heat ? vjp_line<P, true, true>(L, v, s, st) : vjp_line<P, true, false>(L, v, s, st);
    return heat ? vjp_line<P, false, true>(L, v, s, st) : vjp_line<P, false, false>(L, v, s, st);
  }
  return cudaErrorInvalidValue;
}

#define DGB_LINE_ORDER(EXTERN, P)                                                                              \
  EXTERN template cudaError_t residual_line_p<P>(const KLaunch&, const double*, const void*, const StageArgs&, \
                                                 cudaStream_t);                                                \
  EXTERN template cudaError_t vjp_line_p<P>(const KLaunch&, const VjpArgs&, const VjpScratch&, cudaStream_t);

#ifdef DGB_ORDER
DGB_LINE_ORDER(, DGB_ORDER)
#else
#define DGB_X(P) DGB_LINE_ORDER(extern, P)
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

cudaError_t launch_residual_line(const KLaunch& L, const double* U, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  if (L.prm.kq != 0.) return cudaErrorInvalidValue;  // (see enqueue_residual)
  switch (L.P) {
    case 2: return residual_line_p<2>(L, U, Tin, sa, st);
    case 3: return residual_line_p<3>(L, U, Tin, sa, st);
    case 4: return residual_line_p<4>(L, U, Tin, sa, st);
    case 5: return residual_line_p<5>(L, U, Tin, sa, st);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_residual_vjp_line(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  switch (L.P) {
    case 2: return vjp_line_p<2>(L, v, s, st);
    case 3: return vjp_line_p<3>(L, v, s, st);
    case 4: return vjp_line_p<4>(L, v, s, st);
    case 5: return vjp_line_p<5>(L, v, s, st);
  }
  return cudaErrorInvalidValue;
}

#endif  // DGB_ORDER

}  // namespace dgb

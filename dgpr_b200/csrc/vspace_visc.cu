// The viscous terms of the FP64 Gauss-point residual alone (the stage kernels
// with VO): the derivative of the residual in the viscosity, for the
// parameter gradients of the adjoint sweep.
#include "../../include/dgb200.h"
#include "vspace.cuh"

namespace dgb {

template <int P, bool CV, bool HT>
cudaError_t visc_launch_k(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  constexpr bool kAlways = P == 3 || P == 4;
  if constexpr (UseLine<P, double>::value)
    if (L.ladj || kAlways) return llaunch_visc_pc<P, CV, HT>(L, Vs, Tin, sa, st);
  if constexpr (!kAlways) {
    using K = VStageSmem<P, double>;
    const cudaError_t e = allow_shared(vstage_kernel<P, double, CV, HT, true>, K::TOTAL);
    if (e != cudaSuccess) return e;
    vstage_kernel<P, double, CV, HT, true><<<(unsigned)L.E, Cfg<P>::NTS, K::TOTAL, st>>>(
        L.E, Vs, reinterpret_cast<const double*>(Tin), reinterpret_cast<const double*>(L.ops), L.opsd, L.geo,
        CV ? L.gv : nullptr, CV ? L.gf : nullptr, L.nbr, L.prm, element_order(sa, L.E, 1),
        vline_ops<P, double>(L.table));
    return cudaGetLastError();
  }
  return cudaErrorInvalidValue;
}

template <int P>
cudaError_t visc_launch_p(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  const bool heat = L.prm.kq != 0.;
  if (L.gv)
    return heat ? visc_launch_k<P, true, true>(L, Vs, Tin, sa, st) : visc_launch_k<P, true, false>(L, Vs, Tin, sa, st);
  return heat ? visc_launch_k<P, false, true>(L, Vs, Tin, sa, st) : visc_launch_k<P, false, false>(L, Vs, Tin, sa, st);
}

#ifdef DGB_ORDER
template cudaError_t visc_launch_p<DGB_ORDER>(const KLaunch&, const double*, const void*, const StageArgs&,
                                              cudaStream_t);
#else
#define DGB_X(P)                                                                                             \
  extern template cudaError_t visc_launch_p<P>(const KLaunch&, const double*, const void*, const StageArgs&, \
                                               cudaStream_t);
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

cudaError_t vlaunch_stage_visc(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                               cudaStream_t st)
{
  if (L.precision != DGB_FP64 || sa.mode != MODE_RESIDUAL || sa.ecount) return cudaErrorInvalidValue;
  switch (L.P) {
    case 1: return visc_launch_p<1>(L, Vs, Tin, sa, st);
    case 2: return visc_launch_p<2>(L, Vs, Tin, sa, st);
    case 3: return visc_launch_p<3>(L, Vs, Tin, sa, st);
    case 4: return visc_launch_p<4>(L, Vs, Tin, sa, st);
    case 5: return visc_launch_p<5>(L, Vs, Tin, sa, st);
    case 6: return visc_launch_p<6>(L, Vs, Tin, sa, st);
    case 7: return visc_launch_p<7>(L, Vs, Tin, sa, st);
  }
  return cudaErrorInvalidValue;
}

#endif  // DGB_ORDER

}  // namespace dgb

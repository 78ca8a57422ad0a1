// Gauss-point stage kernels (vspace.cuh) in FP64 without the heat flux, the
// basis change, and the dispatch of the Gauss-point form on compute type and
// heat flag (dgb_step).
#include "../../include/dgb200.h"
#include "vspace.cuh"

namespace dgb {

template <int P>
cudaError_t gauss_basis_p(const KLaunch& L, const double* in, double* out, int mode, cudaStream_t st,
                          double* out2)
{
  const unsigned g = (unsigned)L.E;
  switch (mode) {
    case GB_TO_GAUSS: gauss_basis_kernel<P, GB_TO_GAUSS><<<g, Cfg<P>::NT, 0, st>>>(L.E, in, out, L.opsd, out2); break;
    case GB_TO_NODAL: gauss_basis_kernel<P, GB_TO_NODAL><<<g, Cfg<P>::NT, 0, st>>>(L.E, in, out, L.opsd, out2); break;
    case GB_ADJ_TO_GAUSS:
      gauss_basis_kernel<P, GB_ADJ_TO_GAUSS><<<g, Cfg<P>::NT, 0, st>>>(L.E, in, out, L.opsd, out2);
      break;
    case GB_ADJ_TO_NODAL:
      gauss_basis_kernel<P, GB_ADJ_TO_NODAL><<<g, Cfg<P>::NT, 0, st>>>(L.E, in, out, L.opsd, out2);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

#ifdef DGB_ORDER
DGB_VSPACE_ORDER(, DGB_ORDER, double, false)
template cudaError_t gauss_basis_p<DGB_ORDER>(const KLaunch&, const double*, double*, int, cudaStream_t, double*);
#else
#define DGB_X(P)                              \
  DGB_VSPACE_ORDER(extern, P, double, false) \
  extern template cudaError_t gauss_basis_p<P>(const KLaunch&, const double*, double*, int, cudaStream_t, double*);
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

// A line kernel gives an element a third to a half of the lanes that the
// CTA-per-element kernels give it and needs about half their instructions, so
// it wins where the mesh fills the machine and loses on latency where it does
// not, and in a second wave that is nearly empty.  How much it needs goes by the
// geometry: boxes along the axes have their own kernels; a metric of nine
// entries, from the record or per point, costs its few lanes more than the many
// of the others.  RK4 steps, time of the CTA kernel (with line items at P = 5, a
// warp group's) over the line kernel's, boxes; sheared; curved elements:
//   p = 1: 1089 elements 0.98; 0.77; 0.78, 1188 1.07; 0.83; 0.83, 2366 1.23; 0.96; 0.92,
//          2535 1.45; 1.12; 1.12, 13824 2.0; 1.5; 1.4
//   p = 2: 1089 0.88; 0.70; 0.70 (each line over two lanes: 0.82; 0.76; 0.76, while its
//          one-element warps fit the 148 SMs 8 at a time, 1.2 to 1.3 from 1188),
//          1188 0.99; 0.80; 0.78, 2366 1.10; 0.85; 0.86, 2535 1.45; 1.11; 1.17, 5202 1.73;
//          1.34; 1.34, 5491 1.22; 0.96; 0.90 (a wave is 5328: 12 warps of 3 elements on
//          148 SMs), 6137 1.25; 0.99; 0.92, 6859 1.31; 1.02; 0.97, 13824 1.5; 1.2; 1.1
//   p = 3: 60 1.25; 1.08; 1.17, 2366 1.53; 1.22; 1.16, 2535 1.26; 1.02; 0.91 (a wave is 2368),
//          2925 1.28; 1.03; 0.97, 3375 1.55; 1.28; 1.25, 13824 1.40; 1.10; 1.16
//   p = 4: 512 0.93; 0.79; 0.78, 648 1.03; 0.81; 0.79, 900 1.22; 0.92; 0.88, 2535 1.21; 0.98;
//          0.87, 7200 1.23; 1.00; 0.87
LineKernels line_kernels(int P, long E, bool axis, bool curved)
{
  constexpr long kSM = 148;
  switch (P) {
    case 2: return E > (axis ? 8 : 16) * kSM ? LINE_FULL : LINE_NONE;
    case 3:
      if (axis) return E > 8 * kSM ? LINE_FULL : LINE_SPLIT;
      return E > 16 * kSM && !(E > 36 * kSM && E <= 44 * kSM) ? LINE_FULL : LINE_NONE;
    case 4: return curved && E > 16 * kSM && E <= 20 * kSM ? LINE_NONE : LINE_FULL;
    case 5: return axis && E >= 600 ? LINE_FULL : LINE_NONE;
  }
  return LINE_NONE;
}

// Both sides: enqueue_residual.
bool line_adjoint(int P, long E)
{
  switch (P) {
    case 2: return E >= 216;
    case 3: return E > 148 * 8;
    case 4: return true;
    case 5: return E >= 350;
  }
  return false;
}

cudaError_t vprepare_fp64(int P, bool heat)
{
  cudaError_t e = vprepare_t<double, false>(P);
  return e == cudaSuccess && heat ? vprepare_fp64_heat(P) : e;
}

cudaError_t vlaunch_trace_fp64(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  return L.prm.kq != 0. ? vlaunch_trace_fp64_heat(L, V, Tout, st) : vlaunch_trace_t<double, false>(L, V, Tout, st);
}

cudaError_t vlaunch_stage_fp64(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                               cudaStream_t st)
{
  return L.prm.kq != 0. ? vlaunch_stage_fp64_heat(L, Vs, Tin, sa, st)
                        : vlaunch_stage_t<double, false>(L, Vs, Tin, sa, st);
}

cudaError_t prepare_gauss(int P, int precision)
{
  cudaError_t e = precision == DGB_MIXED_FP32 ? vprepare_fp32(P, true) : vprepare_fp64(P, true);
  return e;
}

cudaError_t launch_vtrace(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  return L.precision == DGB_MIXED_FP32 ? vlaunch_trace_fp32(L, V, Tout, st) : vlaunch_trace_fp64(L, V, Tout, st);
}

cudaError_t launch_vstage(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  return L.precision == DGB_MIXED_FP32 ? vlaunch_stage_fp32(L, Vs, Tin, sa, st)
                                       : vlaunch_stage_fp64(L, Vs, Tin, sa, st);
}

cudaError_t launch_gauss_basis_mode(const KLaunch& L, const double* in, double* out, int mode, cudaStream_t st,
                                    double* out2)
{
  switch (L.P) {
    case 1: return gauss_basis_p<1>(L, in, out, mode, st, out2);
    case 2: return gauss_basis_p<2>(L, in, out, mode, st, out2);
    case 3: return gauss_basis_p<3>(L, in, out, mode, st, out2);
    case 4: return gauss_basis_p<4>(L, in, out, mode, st, out2);
    case 5: return gauss_basis_p<5>(L, in, out, mode, st, out2);
    case 6: return gauss_basis_p<6>(L, in, out, mode, st, out2);
    case 7: return gauss_basis_p<7>(L, in, out, mode, st, out2);
  }
  return cudaErrorInvalidValue;
}

#endif  // DGB_ORDER

}  // namespace dgb

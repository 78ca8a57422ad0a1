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
// not (stage times, box meshes, line against CTA kernel):
//   p = 1: 8^3 10.5 / 10.5 us, 4^3 10.5 / 8.5, 36^3 80 / 193
//   p = 2: 12^3 18.7 / 18.8, 10^3 16.6 / 16.2, 36^3 219 / 362; with each line
//          over two lanes 8^3 12.6 / 14.6, 10^3 14.5 / 15.9, 12^3 24.9: that
//          form while its one-element warps fit the 148 SMs 8 at a time
//   p = 3: 4^3 12.6 / 16.6, 32^3 268 / 372
//   p = 4: 8^3 22.8 / 25.6, 6^3 22.8 / 18.8, 24^3 266 / 434
LineKernels line_kernels(int P, long E)
{
  switch (P) {
    case 2: return E >= 216 ? LINE_FULL : LINE_NONE;
    case 3: return E > 148 * 8 ? LINE_FULL : LINE_SPLIT;
    case 4: return LINE_FULL;
    case 5: return E >= 350 ? LINE_FULL : LINE_NONE;
  }
  return LINE_NONE;
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

// Discrete adjoint of the FP64 residual in the Gauss-point form (the VJP of
// f_V, vspace.cuh), without the heat flux: the kernels of adjoint_kernels.cuh
// instantiated with GS = true, compiled apart so that the forms build in
// parallel.
#include "adjoint_kernels.cuh"
#include "ladjoint.cuh"

namespace dgb {

#ifdef DGB_ORDER
DGB_ADJOINT_ORDER(, DGB_ORDER, false, true)
#else
#define DGB_X(P) DGB_ADJOINT_ORDER(extern, P, false, true)
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

cudaError_t prepare_adjoint_gauss(int P, bool curved)
{
  cudaError_t e = prepare_adj_t<false, true>(P, curved);
  return e == cudaSuccess ? prepare_adj_t_gauss_heat(P, curved) : e;
}

cudaError_t launch_vjp_gauss_plain(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  return launch_vjp_t<false, true>(L, v, s, st);
}

#endif  // DGB_ORDER

}  // namespace dgb

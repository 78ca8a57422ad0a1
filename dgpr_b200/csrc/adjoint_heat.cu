// Discrete adjoint of the FP64 residual with the heat flux: the kernels of
// adjoint_kernels.cuh instantiated with HT = true, compiled apart from the
// plain ones so that both build in parallel.
#include "adjoint_kernels.cuh"

namespace dgb {

#ifdef DGB_ORDER
DGB_ADJOINT_ORDER(, DGB_ORDER, true, false)
#else
#define DGB_X(P) DGB_ADJOINT_ORDER(extern, P, true, false)
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

cudaError_t prepare_adjoint_heat(int P, bool curved) { return prepare_adj_t<true, false>(P, curved); }

cudaError_t launch_residual_vjp_heat(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, cudaStream_t st)
{
  return launch_vjp_t<true, false>(L, v, s, st);
}

#endif  // DGB_ORDER

}  // namespace dgb

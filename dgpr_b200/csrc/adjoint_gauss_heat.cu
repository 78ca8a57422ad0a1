// Discrete adjoint of the FP64 residual in the Gauss-point form with the heat
// flux: the kernels of adjoint_kernels.cuh instantiated with HT = GS = true.
#include "adjoint_kernels.cuh"
#include "ladjoint.cuh"

namespace dgb {

#ifdef DGB_ORDER
DGB_ADJOINT_ORDER(, DGB_ORDER, true, true)
#else
#define DGB_X(P) DGB_ADJOINT_ORDER(extern, P, true, true)
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

cudaError_t prepare_adj_t_gauss_heat(int P, bool curved) { return prepare_adj_t<true, true>(P, curved); }

cudaError_t launch_residual_vjp_gauss_heat(const KLaunch& L, const VjpArgs& v, const VjpScratch& s,
                                           cudaStream_t st)
{
  return launch_vjp_t<true, true>(L, v, s, st);
}

#endif  // DGB_ORDER

}  // namespace dgb

// Gauss-point stage kernels (vspace.cuh) in FP32 (the mixed form) without
// the heat flux: the paired kernels where they apply, else one element per CTA.
#include "vspace.cuh"

namespace dgb {

#ifdef DGB_ORDER
DGB_VSPACE_ORDER(, DGB_ORDER, float, false)
DGB_PAIR_ORDER(, DGB_ORDER, false)
#else
#define DGB_X(P) DGB_VSPACE_ORDER(extern, P, float, false) DGB_PAIR_ORDER(extern, P, false)
DGB_EACH_ORDER(DGB_X)
#undef DGB_X

// A line kernel gives an element (or pair) P^2 or 2 P^2 lanes against P^3 and
// more, so it loses on latency while the CTA kernels hold the mesh in a wave or
// little more, and wins above; at P = 4, with as many lanes as the warp group's
// kernel, it also wins where 16 elements per SM (of the 20 warps that MStage
// compiles single elements for) are the whole mesh, and loses in between, where
// its second wave is nearly empty.  The lines are measured, not derived: 148 * 16
// is the multiple of the SMs that they lie by.  Whole RK4 steps, CTA against line
// kernel:
//   pairs   p = 1: 16^3 54 / 60 us, 18^3 79 / 68, 36^3 467 / 317
//           p = 2: 24^3 302 / 348, 36^3 1005 / 1006: never
//           p = 3: 16^3 136 / 145, 18^3 217 / 209, 32^3 1011 / 957
//   single  p = 1: 13^3 41 / 41, 15^3 68 / 46, 35^3 579 / 274
//           p = 2: 13^3 62 / 85, 15^3 100 / 92, 35^3 1020 / 881
//           p = 3: 11^3 77 / 67, 15^3 142 / 143, 19^3 271 / 251, 31^3 1088 / 1035;
//                  curved 12^3 86 / 77, 16^3 175 / 190, 28^3 871 / 881
bool mixed_line(int P, long E, bool pair, bool curved)
{
  constexpr long kWave = 148 * 16;
  switch (P) {
    case 2: return E > (pair ? 2 * kWave : kWave);
    case 3: return !pair && E > kWave;
    case 4: return pair ? E >= 5000 : E <= kWave || (!curved && E >= 5000);
  }
  return false;
}

cudaError_t vprepare_fp32(int P, bool heat)
{
  cudaError_t e = vprepare_t<float, false>(P);
  if (e == cudaSuccess) e = vprepare2_t<false>(P);
  return e == cudaSuccess && heat ? vprepare_fp32_heat(P) : e;
}

cudaError_t vlaunch_trace_fp32(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  if (L.prm.kq != 0.) return vlaunch_trace_fp32_heat(L, V, Tout, st);
  return use_pair(L) ? vlaunch_trace2_t<false>(L, V, Tout, st) : vlaunch_trace_t<float, false>(L, V, Tout, st);
}

cudaError_t vlaunch_stage_fp32(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                               cudaStream_t st)
{
  if (L.tc) return vlaunch_stage_tc(L, Vs, Tin, sa, st);
  if (L.prm.kq != 0.) return vlaunch_stage_fp32_heat(L, Vs, Tin, sa, st);
  return use_pair(L) ? vlaunch_stage2_t<false>(L, Vs, Tin, sa, st) : vlaunch_stage_t<float, false>(L, Vs, Tin, sa, st);
}

#endif  // DGB_ORDER

}  // namespace dgb

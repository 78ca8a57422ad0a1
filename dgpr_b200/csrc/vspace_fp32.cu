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
// little more, and wins above, but in a second wave of its own that is nearly
// empty (at p = 2 a wave is 7104 elements: 16 warps of 3 on 148 SMs; at p = 3 4736 in
// pairs); at P = 4, with as many lanes as the warp group's kernel, it also wins
// on the smallest meshes.  RK4 steps, time of the CTA or warp-group kernel over the
// line kernel's, all sides periodic / with walls:
//   pairs   p = 1: 4352 elements 0.94 / 0.91, 5202 1.14 / 1.07, 13824 1.47 / 1.44
//           p = 2: 24^3 302 / 348 us, 36^3 1005 / 1006: never
//           p = 3: 5202 0.83 / 0.89, 5832 1.05 / 1.06, 8000 1.05 / 1.02, 13824 1.04 / 1.03
//   single  p = 1: 2197 1.01 / 0.97, 2535 1.32 / 1.28, 9261 2.05 / 1.96; curved 2366 0.97 /
//                  0.90, 2535 1.32 / 1.26, 13824 1.58 / 1.56
//           p = 2: 2925 0.86 / 0.88, 3375 1.07 / 1.12, 6859 1.14 / 1.14; curved 2366 0.73 /
//                  0.71, 2535 1.05 / 1.08, 6859 1.09 / 1.10, 7200 0.91 / 0.94, 9261 0.91 /
//                  0.93, 13824 1.10 / 1.11
//           p = 3: 343 1.12 / 1.08, 2197 1.07 / 1.05, 3375 0.95 / 0.92, 4913 1.16 / 1.14, 9261
//                  0.97 / 0.97; curved 60 1.14 / 1.15, 2366 1.09 / 1.06, 3375 0.89 / 0.87
bool mixed_line(int P, long E, bool pair, bool curved)
{
  constexpr long kSM = 148;
  switch (P) {
    case 2: return E > (pair ? 32 : 16) * kSM;
    case 3: return !pair && (curved ? E > 16 * kSM && !(E > 48 * kSM && E <= 64 * kSM) : E > 21 * kSM);
    case 4: return pair ? E > 38 * kSM : E <= 16 * kSM || (!curved && E >= 5000);
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

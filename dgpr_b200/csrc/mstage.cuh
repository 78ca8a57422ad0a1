// The mixed form's Gauss-point stage and trace kernels with lanes owning lines
// of Gauss points (lstage.cuh), for one element (T = float) or a pair of
// elements (T = f2) at a time, P = 2..4.
//
// The arithmetic is that of the kernels with a thread per Gauss point
// (vstage_kernel, vstage2_kernel, wstage2_kernel), sum by sum in their order,
// so the FP32 values come out the same bits: the volume term of all three axes
// before the first face, the faces one after the other, tangential sums over
// the face's points in ascending order, the nodal residual of the norm along
// x, y, z.  (FP32 rounding in another order would move a mixed state by 1e-8
// within a few steps.)
//
// The kernels with a thread per point are bound by their shared-memory reads
// and, at P <= 3, by lanes without a point (P = 2: 8 of 32).  Here a warp holds
// 4 (P = 2), 3 (P = 3) or one (P = 4) elements or pairs, reads each value of a
// line once, and keeps the face exchange in registers.  Bound by the latency
// of dependent instructions at 12 to 20 warps per SM.  Stage, point -> line:
// pairs P = 2 36^3 119 -> 75 us, P = 4 32^3 227 -> 205; single elements P = 2
// 36^3 156 -> 63, P = 3 239 -> 195, P = 4 8^3 14.6 -> 12.7.  Pairs at P = 3 and
// all at P = 5 gained less than the line items of vspace.cuh give the point
// kernels, and keep those.
#pragma once

#include "vspace.cuh"

namespace dgb {

// 1D operators in the compute type, passed as a kernel parameter.
template <int P, class T>
struct MOps {
  T Dq[P * P], EL[2 * P], DL[2 * P], w[P], B[P * P], cend[2];
  double iw[P];
};

template <int P, int H, class T>
struct MStage {
  using L = LStage<P, H>;
  static_assert(P % H == 0, "a lane owns all its points");
  static constexpr int ST = (int)sizeof(T);
  static constexpr int oGeo = align16(3 * L::A * ST);
  static constexpr int oGeoF = oGeo + align16(kGeoStride * ST);  // pairs: each element's own record
  static constexpr int UNIT = oGeoF + (is_pair<T>::value ? 2 * kGeoStride * 4 : 0);
  static constexpr int TOTAL = L::EPW * UNIT;
  static_assert(TOTAL <= kSharedDefault, "shared memory of the line kernels");
  static constexpr int MINB = sizeof(T) == 4 && H == 2 ? 20 : 16;  // warps per SM
};

// The state at the lane's points of the x-lines from memory (a pair: both).
template <int P, int H, class T, int NPL>
__device__ __forceinline__ void mline_from_memory(const LLane<P, H>& ln, const double* Vs, long e, T (&t)[5][NPL])
{
  constexpr int NB = P * P * P, W = is_pair<T>::value ? 2 : 1;
  double v[W][5][NPL];
#pragma unroll
  for (int i = 0; i < W; ++i)
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      const double* p = Vs + ((e + i) * 5 + r) * NB + P * ln.l;
      if constexpr (P % 2 == 0 && NPL == 2) {
        const double2 d = *reinterpret_cast<const double2*>(p + ln.q(0));
        v[i][r][0] = d.x;
        v[i][r][1] = d.y;
      } else {
#pragma unroll
        for (int j = 0; j < NPL; ++j) v[i][r][j] = p[ln.q(j)];
      }
    }
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      if constexpr (is_pair<T>::value)
        t[r][j] = T((float)v[0][r][j], (float)v[1][r][j]);
      else
        t[r][j] = T(v[0][r][j]);
    }
}

template <int P, int H, class T>
__device__ __forceinline__ void mgeo_to_shared(const LLane<P, H>& ln, const double* __restrict__ geo, long e, T* sg,
                                               float* sgf)
{
  if (!ln.active) return;
  for (int i = ln.l * H + ln.h; i < kGeoStride; i += P * P * H) {
    if constexpr (is_pair<T>::value) {
      const float g0 = (float)geo[e * kGeoStride + i], g1 = (float)geo[(e + 1) * kGeoStride + i];
      sg[i] = T(g0, g1);
      sgf[i] = g0;
      sgf[kGeoStride + i] = g1;
    } else {
      sg[i] = T(geo[e * kGeoStride + i]);
    }
  }
}

// vtrace_half at the lane's face points, of the state in the tiles
// (line_spread).
template <int P, int H, class T, bool CV>
__device__ __forceinline__ void mline_traces(const LLane<P, H>& ln, const MOps<P, T>& op, const T* tiles, const T* sg,
                                             const double* gfe, T mu, T kq, T* __restrict__ Te)
{
  constexpr int VS = LTile<P>::VS;
#pragma unroll 1
  for (int f = 0; f < 6 / H; ++f) {
    const int ax = H == 2 ? f : f >> 1, end = H == 2 ? ln.h : f & 1;
    const T* tile = tiles + ax * (5 * VS);
    T S[5], dn[5], g[3][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) S[r] = dn[r] = T(0);
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const T ev = op.EL[end * P + k], dv = op.DL[end * P + k];
      const int o = ln.at(k);
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        const T u = tile[r * VS + o];
        S[r] = fma(ev, u, S[r]);
        dn[r] = fma(dv, u, dn[r]);
      }
    }
    T d1[5], d2[5];
#pragma unroll
    for (int r = 0; r < 5; ++r) d1[r] = d2[r] = T(0);
    if (mu != T(0)) {
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const T c1 = op.Dq[ln.a * P + k], c2 = op.Dq[ln.b * P + k];
        const int s1 = ln.lane_of(k, ln.b), s2 = ln.lane_of(ln.a, k);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          d1[r] = fma(c1, shfl_line(S[r], s1), d1[r]);
          d2[r] = fma(c2, shfl_line(S[r], s2), d2[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      g[0][r] = ax == 0 ? dn[r] : d1[r];
      g[1][r] = ax == 0 ? d1[r] : (ax == 1 ? dn[r] : d2[r]);
      g[2][r] = ax == 2 ? dn[r] : d2[r];
    }
    if (ln.active) trace_point_store<P, T, CV>(2 * ax + end, ln.l, S, g, sg, gfe, mu, kq, Te);
  }
}

template <int P, int H, class T, bool CV, bool HT>
__global__ void __launch_bounds__(32, 16)
mtrace_kernel(long count, const double* __restrict__ V, const __grid_constant__ MOps<P, T> op,
              const double* __restrict__ geo, const double* __restrict__ gf, T* __restrict__ Tr, DevParams prm)
{
  using L = MStage<P, H, T>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * L::UNIT;
  T* S1 = reinterpret_cast<T*>(eb);
  T* sg = reinterpret_cast<T*>(eb + L::oGeo);
  const long e = is_pair<T>::value ? 2 * ln.u : ln.u;
  T t[5][L::L::NPL];
  mline_from_memory(ln, V, e, t);
  line_spread<0, false>(ln, S1, t);
  mgeo_to_shared(ln, geo, e, sg, reinterpret_cast<float*>(eb + L::oGeoF));
  __syncwarp();
  mline_traces<P, H, T, CV>(ln, op, S1, sg, CV ? gf + e * 6 * kFaceC * P * P : nullptr, T(prm.mu),
                            HT ? T(prm.kq) : T(0), Tr + ln.u * 60 * P * P);
}

// One RK stage; arguments as vstage_kernel and vstage2_kernel.  sof: the FP32
// operator table, for the boundary lanes of pairs.
template <int P, int H, class T, bool CV, bool HT>
__global__ void __launch_bounds__(32, (MStage<P, H, T>::MINB))
mstage_kernel(long count, const double* Vs, const T* __restrict__ Tr, const __grid_constant__ MOps<P, T> op,
              const float* __restrict__ sof, const double* __restrict__ geo, const double* __restrict__ gv,
              const double* __restrict__ gf, const int* __restrict__ nbr, const __grid_constant__ DevParams prm,
              const __grid_constant__ StageArgs sa)
{
  using L = MStage<P, H, T>;
  constexpr bool PR = is_pair<T>::value;
  constexpr int NB = P * P * P, NQF = P * P, VS = LTile<P>::VS, A = 5 * VS, NPL = L::L::NPL;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * L::UNIT;
  T* S1 = reinterpret_cast<T*>(eb);  // tiles as in lstage_kernel
  T* sg = reinterpret_cast<T*>(eb + L::oGeo);
  float* sgf = reinterpret_cast<float*>(eb + L::oGeoF);
  const bool active = ln.active;
  const long k = sa.ebase + sa.estep * ln.u, e = PR ? 2 * k : k;
  const int fq = ln.l;
  int* const flag = active ? sa.flag : nullptr;

  T Sv[5][NPL];  // the state at the lane's points of its x-line
  mline_from_memory(ln, Vs, e, Sv);
#pragma unroll
  for (int r = 0; r < 5; ++r) line_store<0, 0>(ln, S1 + r * VS, Sv[r]);
  mgeo_to_shared(ln, geo, e, sg, sgf);
  __syncwarp();

  const T gamma = T(prm.gamma), mu = T(prm.mu), kq = HT ? T(prm.kq) : T(0);
  const double* gve = CV ? gv + e * kVolC * NB : nullptr;
  const double* gfe = CV ? gf + e * 6 * kFaceC * NQF : nullptr;

  // ---------------- volume integral (solve.cpp:276-341) + source (345-360)
  {  // reference derivatives along y, z, x (in place of the state)
    T c[NPL][P];
#pragma unroll
    for (int j = 0; j < NPL; ++j)
#pragma unroll
      for (int m = 0; m < P; ++m) c[j][m] = op.Dq[ln.q(j) * P + m];
    auto derivative = [&](auto axis) {
      constexpr int ax = decltype(axis)::value;
      T d[5][NPL];
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const T v = S1[r * VS + ln.template to<ax, 0>(m)];
#pragma unroll
          for (int j = 0; j < NPL; ++j) d[r][j] = m ? fma(c[j][m], v, d[r][j]) : T(c[j][m] * v);
        }
      if (ax == 0) __syncwarp();  // all have read the state
#pragma unroll
      for (int r = 0; r < 5; ++r) line_store<ax, ax>(ln, S1 + ax * A + r * VS, d[r]);
    };
    derivative(std::integral_constant<int, 1>());
    derivative(std::integral_constant<int, 2>());
    derivative(std::integral_constant<int, 0>());
  }
  __syncwarp();
#pragma unroll 1
  for (int j = 0; j < NPL; ++j) {  // the flux at the lane's points
    const int i = ln.q(j), o = ln.at(i), oy = ln.template to<0, 1>(i), oz = ln.template to<0, 2>(i);
    T Jbuf[9], wJ;
    if constexpr (CV) {
      const double* gq = gve + i + P * ln.l;
#pragma unroll
      for (int c = 0; c < 9; ++c) Jbuf[c] = T(gq[c * NB]);
      wJ = op.w[i] * op.w[ln.a] * op.w[ln.b] * T(gq[kVolDetJ * NB]);
    } else {
      wJ = op.w[i] * op.w[ln.a] * op.w[ln.b] * sg[kGeoDetJ];
    }
    T S[5], g[3][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      S[r] = Sv[r][0];
      g[0][r] = S1[r * VS + o];
      g[1][r] = S1[A + r * VS + oy];
      g[2][r] = S1[2 * A + r * VS + oz];
    }
    const bool own = ln.owns(j);
    vpoint_core<T, false>(S, g, CV ? Jbuf : sg + kGeoJinv, wJ, gamma, mu, kq, [&](int m, int r, T v) {
      if (own) S1[m * A + r * VS + (m == 0 ? o : m == 1 ? oy : oz)] = v;
    });
#pragma unroll
    for (int r = 0; r < 5; ++r)  // the next point's state
#pragma unroll
      for (int m = 1; m < NPL; ++m) Sv[r][m - 1] = Sv[r][m];
  }
  __syncwarp();
  T yl[5][NPL];  // Y at the lane's points of its line
  {
    T c[NPL][P];
#pragma unroll
    for (int j = 0; j < NPL; ++j)
#pragma unroll
      for (int m = 0; m < P; ++m) c[j][m] = op.Dq[m * P + ln.q(j)];
    auto divergence = [&](auto axis) {
      constexpr int ax = decltype(axis)::value;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        T y[NPL];
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const T f = S1[ax * A + r * VS + ln.at(m)];
#pragma unroll
          for (int j = 0; j < NPL; ++j) y[j] = m ? fma(c[j][m], f, y[j]) : T(c[j][m] * f);
        }
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          if (ax == 0) {
            yl[r][j] = y[j];
          } else {
            yl[r][j] = S1[r * VS + ln.at(ln.q(j))] + y[j];
          }
        }
      }
      if (ax == 2) {
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          const int q = ln.q(j);
          const T wJ = op.w[ln.a] * op.w[ln.b] * op.w[q] *
                       (CV ? T(gve[kVolDetJ * NB + fq + NQF * q]) : sg[kGeoDetJ]);
#pragma unroll
          for (int r = 0; r < 5; ++r) yl[r][j] = yl[r][j] - T(prm.src[r]) * wJ;
        }
      }
      __syncwarp();  // all have read tile 0
#pragma unroll
      for (int r = 0; r < 5; ++r) line_store<ax, ax == 2 ? 0 : ax + 1>(ln, S1 + r * VS, yl[r]);
      __syncwarp();
    };
    divergence(std::integral_constant<int, 0>());
    divergence(std::integral_constant<int, 1>());
    divergence(std::integral_constant<int, 2>());
  }

  // ---------------- faces (solve.cpp:393-794), one after the other
#pragma unroll 1
  for (int ax = 0; ax < 3; ++ax) {
    const int ax1 = ax == 0 ? 1 : 0, ax2 = ax == 2 ? 1 : 2;
    T ga[5], gb[4], pa[5], pb[4];  // the (last) end's values, the other's
#pragma unroll 1
    for (int f = 0; f < 2 / H; ++f) {
      const int end = H == 2 ? ln.h : f, lf = 2 * ax + end;
      T fa[5], fb[12];  // fb rows: the two tangential axes, the normal axis
      const T* To = Tr + (k * 6 + lf) * 10 * NQF + fq;
      const int nb = nbr[e * 6 + lf], nb1 = PR ? nbr[e * 6 + 6 + lf] : 0;
      const double* gp = CV ? gfe + lf * kFaceC * NQF + fq : nullptr;
      T n[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) n[c] = CV ? T(gp[(kFaceN + c) * NQF]) : sg[kGeoN + 3 * lf + c];
      const T fJ = CV ? T(gp[kFaceFJ * NQF]) : sg[kGeoFJ + lf];
      const T fw = fJ * op.w[ln.a] * op.w[ln.b];
      auto Jf = [&]() {  // rows in fb's order
        if constexpr (CV)
          return JacobianRows<T>(gp, NQF, ax1, ax2, ax);
        else
          return JacobianRows<T>(sg + kGeoJinv, 1, ax1, ax2, ax);
      };
      auto lift = [&]() { return CV ? T(gp[kFaceLift * NQF]) : quot(op.cend[end], sg[kGeoDetJ]); };
      bool lanes = false;  // a pair with a boundary in either element
      if constexpr (PR) lanes = nb < 0 || nb1 < 0;
      if (!lanes) {
        T Uo[5], Qo[5], Un[5], Qn[5], lift_n = T(0);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          Uo[r] = To[r * NQF];
          Qo[r] = To[(5 + r) * NQF];
        }
        if constexpr (PR) {
          const long i0 = ((long)(nb / 2) * 6 + (lf ^ 1)) * 10 * NQF + fq;
          const long i1 = ((long)(nb1 / 2) * 6 + (lf ^ 1)) * 10 * NQF + fq;
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            Un[r] = T(pair_lane(Tr, i0 + r * NQF, nb), pair_lane(Tr, i1 + r * NQF, nb1));
            Qn[r] = T(pair_lane(Tr, i0 + (5 + r) * NQF, nb), pair_lane(Tr, i1 + (5 + r) * NQF, nb1));
          }
          lift_n = quot(op.cend[end ^ 1], T((float)geo[(long)nb * kGeoStride + kGeoDetJ],
                                            (float)geo[(long)nb1 * kGeoStride + kGeoDetJ]));
        } else if (nb >= 0) {
          const T* Tn = Tr + ((long)nb * 6 + (lf ^ 1)) * 10 * NQF + fq;
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            Un[r] = Tn[r * NQF];
            Qn[r] = Tn[(5 + r) * NQF];
          }
          lift_n = CV ? T(gf[(((long)nb * 6 + (lf ^ 1)) * kFaceC + kFaceLift) * NQF + fq])
                      : quot(op.cend[end ^ 1], T(geo[(long)nb * kGeoStride + kGeoDetJ]));
        }
        face_flux_core<T, 1, false, true>(end, PR ? 0 : nb, Uo, Qo, Un, Qn, lift_n, n, fJ, fw, Jf, lift, prm, gamma,
                                          mu, kq, flag, fa, fb);
      }
      if constexpr (PR) {
        if (lanes) {  // each element through the scalar routine
          T ta[5], tb[12];
#pragma unroll 1
          for (int j = 0; j < 2; ++j)
            pair_face_lane<P, HT, 1>(j, j ? nb1 : nb, lf, fq, To - fq, Tr, sof, sgf + j * kGeoStride, geo, prm, flag, ta,
                                     tb);
#pragma unroll
          for (int r = 0; r < 5; ++r) fa[r] = ta[r];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int r = 0; r < 4; ++r) fb[i * 4 + r] = tb[(i == 0 ? ax1 : i == 1 ? ax2 : ax) * 4 + r];
        }
        __syncwarp();
      }
      if (mu != T(0)) {  // tangential test derivatives, the face's points in ascending order
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const T d1 = op.Dq[m * P + ln.a], d2 = op.Dq[m * P + ln.b];
          const int s1 = ln.lane_of(m, ln.b), s2 = ln.lane_of(ln.a, m);
          T x1[4], x2[4];
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            x1[r] = shfl_line(fb[r], s1);
            x2[r] = shfl_line(fb[4 + r], s2);
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            fa[1 + r] = fma(d1, x1[r], fa[1 + r]);
            fa[1 + r] = fma(d2, x2[r], fa[1 + r]);
          }
        }
      }
      if constexpr (H == 1) {
        if (f == 0) {
#pragma unroll
          for (int r = 0; r < 5; ++r) pa[r] = fa[r];
#pragma unroll
          for (int r = 0; r < 4; ++r) pb[r] = fb[8 + r];
        }
      }
#pragma unroll
      for (int r = 0; r < 5; ++r) ga[r] = fa[r];
#pragma unroll
      for (int r = 0; r < 4; ++r) gb[r] = fb[8 + r];
    }
    if constexpr (H == 2) {  // the low end's in pa, pb, the high end's in ga, gb
      const int s = ln.partner();
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        const T x = shfl_line(ga[r], s);
        pa[r] = ln.h ? x : ga[r];
        ga[r] = ln.h ? ga[r] : x;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const T x = shfl_line(gb[r], s);
        pb[r] = ln.h ? x : gb[r];
        gb[r] = ln.h ? gb[r] : x;
      }
    }
    // onto the lane's points of the line
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int q = ln.q(j), o = ln.at(q);
      const T ev0 = op.EL[q], dv0 = op.DL[q], ev1 = op.EL[P + q], dv1 = op.DL[P + q];
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        T y = S1[r * VS + o];
        if (r == 0) {
          y += ev0 * pa[0];
          y += ev1 * ga[0];
        } else {
          y += ev0 * pa[r] + dv0 * pb[r > 0 ? r - 1 : 0];
          y += ev1 * ga[r] + dv1 * gb[r > 0 ? r - 1 : 0];
        }
        yl[r][j] = y;
      }
    }
    if (ax < 2) {
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          const int q = ln.q(j);
          if (ln.owns(j)) S1[r * VS + (ax == 0 ? ln.template to<0, 1>(q) : ln.template to<1, 2>(q))] = yl[r][j];
        }
      __syncwarp();
    }
  }

  // ---------------- norm partial: the nodal residual R = B3^T Y, along x, y, z
  if (sa.part) {
    T t[5][NPL], c[NPL][P];
    T* N = S1 + A;
#pragma unroll
    for (int j = 0; j < NPL; ++j)
#pragma unroll
      for (int m = 0; m < P; ++m) c[j][m] = op.B[m * P + ln.q(j)];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int j = 0; j < NPL; ++j) t[r][j] = yl[r][j];
    auto contraction = [&](auto axis) {
      constexpr int ax = decltype(axis)::value;
#pragma unroll
      for (int r = 0; r < 5; ++r) line_store<ax == 0 ? 2 : ax - 1, ax>(ln, N + r * VS, t[r]);
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        T v[P];
        line_load(ln, N + r * VS, v);
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          t[r][j] = c[j][0] * v[0];
#pragma unroll
          for (int m = 1; m < P; ++m) t[r][j] = fma(c[j][m], v[m], t[r][j]);
        }
      }
      __syncwarp();
    };
    contraction(std::integral_constant<int, 0>());
    contraction(std::integral_constant<int, 1>());
    contraction(std::integral_constant<int, 2>());
    double s[PR ? 2 : 1] = {};
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int j = 0; j < NPL; ++j)
        if (ln.owns(j)) {
          if constexpr (PR) {
            s[0] += double(t[r][j].lane(0)) * double(t[r][j].lane(0));
            s[1] += double(t[r][j].lane(1)) * double(t[r][j].lane(1));
          } else {
            s[0] += double(t[r][j]) * double(t[r][j]);
          }
        }
    const int i = ln.l * H + ln.h;
#pragma unroll
    for (int j = 0; j < (PR ? 2 : 1); ++j) {  // over the element's lanes, in a fixed order
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        const double o = __shfl_down_sync(0xffffffffu, s[j], off);
        if (i + off < L::L::LE) s[j] += o;
      }
      if (active && i == 0) sa.part[e + j] = s[j];
    }
  }

  // ---------------- f_V = -Y / (w detJ) in FP64, RK update, on the z-line
  {
    const double iwab = op.iw[ln.a] * op.iw[ln.b];
#pragma unroll
    for (int i = 0; i < (PR ? 2 : 1); ++i) {
      double sc[NPL];
      const double id = CV ? 0. : -1.0 / geo[(e + i) * kGeoStride + kGeoDetJ];
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        const int q = ln.q(j);
        if constexpr (CV)
          sc[j] = -iwab * op.iw[q] / gve[kVolDetJ * NB + fq + NQF * q];
        else
          sc[j] = iwab * op.iw[q] * id;
      }
      const long base = (e + i) * 5 * NB + fq + NQF * ln.q(0);
      // all the operands are loaded before any result is stored
      RkOperands o[5][NPL];
      if (sa.mode != MODE_RESIDUAL) {
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
          for (int j = 0; j < NPL; ++j) {
            const long g = base + r * NB + NQF * j;
            o[r][j] = rk_stage_load(sa, g, Vs + g);
          }
      }
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          const long g = base + r * NB + NQF * j;
          double y;
          if constexpr (PR)
            y = double(yl[r][j].lane(i));
          else
            y = double(yl[r][j]);
          if (!active) continue;
          if (sa.mode == MODE_RESIDUAL) {
            sa.fout[g] = y * sc[j];
            continue;
          }
          const double un = rk_stage_apply(sa, g, y * sc[j], o[r][j]);
          sa.Uout[g] = un;
          if constexpr (PR) {  // the new state, for the traces
            if (i == 0)
              yl[r][j].v.x = (float)un;
            else
              yl[r][j].v.y = (float)un;
          } else {
            yl[r][j] = T(un);
          }
        }
    }
  }
  // ---------------- face traces of the new state for the next stage
  if (sa.Tnext) {
    __syncwarp();  // the tiles are free
    line_spread<2, false>(ln, S1, yl);
    __syncwarp();
    mline_traces<P, H, T, CV>(ln, op, S1, sg, gfe, mu, kq, reinterpret_cast<T*>(sa.Tnext) + k * 60 * NQF);
  }
}

// ------------------------------------------------------------ host launchers

template <int P, class T>
MOps<P, T> mline_ops(const double* table)
{
  using C = Cfg<P>;
  MOps<P, T> o;
  const auto t = [&](int i) { return T((float)table[i]); };
  for (int i = 0; i < P * P; ++i) {
    o.Dq[i] = t(C::oDq + i);
    o.B[i] = t(C::oB + i);
  }
  for (int i = 0; i < 2 * P; ++i) {
    o.EL[i] = t(C::oEh + i);
    o.DL[i] = t(C::oDh + i);
  }
  for (int i = 0; i < P; ++i) {
    o.w[i] = t(C::oW + i);
    o.iw[i] = 1.0 / table[C::oW + i];
  }
  for (int i = 0; i < 2; ++i) o.cend[i] = t(C::oC + i);
  return o;
}

template <int P, class T, bool CV, bool HT>
cudaError_t mllaunch_stage_pc(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                              cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW, W = is_pair<T>::value ? 2 : 1;
  const long count = (sa.ecount ? sa.ecount : L.E) / W;
  mstage_kernel<P, H, T, CV, HT><<<(unsigned)((count + EPW - 1) / EPW), 32, MStage<P, H, T>::TOTAL, st>>>(
      count, Vs, reinterpret_cast<const T*>(Tin), mline_ops<P, T>(L.table), reinterpret_cast<const float*>(L.ops), L.geo,
      L.gv, L.gf, L.nbr, L.prm, element_order(sa, L.E, W));
  return cudaGetLastError();
}

template <int P, class T, bool CV, bool HT>
cudaError_t mllaunch_trace_pc(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW;
  const long count = L.E / (is_pair<T>::value ? 2 : 1);
  mtrace_kernel<P, H, T, CV, HT><<<(unsigned)((count + EPW - 1) / EPW), 32, MStage<P, H, T>::TOTAL, st>>>(
      count, V, mline_ops<P, T>(L.table), L.geo, L.gf, reinterpret_cast<T*>(Tout), L.prm);
  return cudaGetLastError();
}

}  // namespace dgb

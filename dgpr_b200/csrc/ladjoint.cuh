// The residual VJP in the Gauss-point form (adjA_kernel and adjB_kernel of
// adjoint_kernels.cuh) with lanes owning lines of Gauss points (lstage.cuh).
//
// ladjA_kernel, per element: mu = -lam / (w detJ), the transpose of
// the volume term into the volume part, and at each face point the adjoints of
// this element's trace and of the neighbour's values.  Its tiles hold the
// reference derivatives of the state and of mu, along each axis in that axis'
// line order; the pointwise reverse leaves the adjoints of the derivatives in
// the latter's places, and they go back along the lines as a stage's fluxes
// do.
//
// ladjB_kernel (P = 2..5), per element: the adjoints of its face traces,
// gathered from its own and its neighbours' trace adjoints, through the
// transpose of the trace map, added to the volume part.  The face value and
// gradient of the state come from the lane's line and shuffles, as in
// line_trace; the transpose sends a face point's value adjoint and the
// tangential derivatives' (exchanged by shuffles) to the points of its normal
// line, as the stage does with its face fluxes.
//
// The thread-per-point kernels were latency-bound with their contractions'
// reads of shared memory leading; at 16^3, p = 3: adjA 75 -> 62 us,
// adjB 41 -> 28 us a launch (ncu durations).
//
// NOD: U, lam and the result are nodal (residual_line.cu); the basis changes
// on the element as they are loaded and stored.
#pragma once

#include "adjoint_kernels.cuh"
#include "vspace.cuh"

namespace dgb {

// Shared memory of ladjA_kernel per element: the state's derivative tiles,
// mu's, the geometry record.
template <int P, int H>
struct LAdjA {
  using L = LStage<P, H>;
  static constexpr int oGeo = align16(6 * L::A * 8);
  static constexpr int UNIT = oGeo + align16(kGeoStride * 8);
  static constexpr int TOTAL = L::EPW * UNIT;
  static_assert(TOTAL <= kSharedDefault, "shared memory of the line kernels");
  // Warps per SM.  Without spills the pointwise reverse and the face VJPs take
  // 240 registers; measured on the reverse sweep at 16^3 and 24^3, p = 3:
  // 9.22 and 26.4 ms with 8 warps, 9.42 and 26.7 with 11 (168 registers),
  // 9.86 and 28.2 with 16
  static constexpr int MINB = 8;
};

// Reference derivatives along y, z and (H = 2) x of the field in the first
// of three tiles (x order) into them, the last in its place.
template <int P, int H, int ND>
__device__ __forceinline__ void line_derivatives(const LLane<P, H>& ln, const LOps<P>& op, double* tiles)
{
  constexpr int VS = LTile<P>::VS, A = 5 * VS, NPL = LStage<P, H>::NPL;
  double c[NPL][P];
#pragma unroll
  for (int j = 0; j < NPL; ++j)
#pragma unroll
    for (int m = 0; m < P; ++m) c[j][m] = op.Dq[ln.q(j) * P + m];
  auto derivative = [&](auto axis) {
    constexpr int ax = decltype(axis)::value;
    double d[ND][NPL];
#pragma unroll
    for (int r = 0; r < ND; ++r)
#pragma unroll
      for (int m = 0; m < P; ++m) {
        const double v = tiles[r * VS + ln.template to<ax, 0>(m)];
#pragma unroll
        for (int j = 0; j < NPL; ++j) d[r][j] = m ? fma(c[j][m], v, d[r][j]) : c[j][m] * v;
      }
    if (ax == 0) __syncwarp();  // all have read the field
#pragma unroll
    for (int r = 0; r < ND; ++r) line_store<ax, ax>(ln, tiles + ax * A + r * VS, d[r]);
  };
  derivative(std::integral_constant<int, 1>());
  derivative(std::integral_constant<int, 2>());
  if constexpr (H == 2) derivative(std::integral_constant<int, 0>());
}

template <int P, int H, bool CV, bool HT, bool NOD>
__global__ void __launch_bounds__(32, (LAdjA<P, H>::MINB))
ladjA_kernel(long count, const double* __restrict__ V, const double* __restrict__ Tr, const __grid_constant__ VjpArgs v,
             const __grid_constant__ LOps<P> op, const double* __restrict__ geo, const double* __restrict__ gv,
             const double* __restrict__ gf, const int* __restrict__ nbr, const __grid_constant__ DevParams prm,
             double* __restrict__ part, double* __restrict__ TA, int* flag)
{
  using L = LStage<P, H>;
  using K = LAdjA<P, H>;
  constexpr int NB = P * P * P, NQF = P * P, VS = LTile<P>::VS, NPL = L::NPL;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * K::UNIT;
  double* S1 = reinterpret_cast<double*>(eb);  // the state, its derivatives; then the volume part in tile 0
  double* N1 = S1 + 3 * L::A;                  // mu, its derivatives, the adjoints of the state's; then mu again
  double* sg = reinterpret_cast<double*>(eb + K::oGeo);
  const long e = ln.u;
  const int fq = ln.l;
  const double gamma = prm.gamma, mu = prm.mu, kq = HT ? prm.kq : 0.;
  const double* gve = CV ? gv + e * kVolC * NB : nullptr;
  const double* gfe = CV ? gf + e * 6 * kFaceC * NQF : nullptr;
  const double wab = op.w[ln.a] * op.w[ln.b], iwab = op.iw[ln.a] * op.iw[ln.b];

  double Sv[5][NPL], Mv[5][NPL];  // the state and mu at the lane's points of its x-line
  auto load = [&](const double* src, double (&t)[5][NPL]) {
    if constexpr (NOD)
      zline_from_memory(ln, src, e, t);
    else
      line_from_memory(ln, src, e, t);
  };
  load(V, Sv);
  load(v.X, Mv);
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j) Mv[r][j] *= v.cx;
  const double* more[2] = {v.Y, v.Z};
  const double cs[2] = {v.cy, v.cz};
#pragma unroll
  for (int m = 0; m < 2; ++m)
    if (more[m]) {
      double t[5][NPL];
      load(more[m], t);
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) Mv[r][j] = fma(cs[m], t[r][j], Mv[r][j]);
    }
  if constexpr (NOD) {  // V = B3 U, dJ/dV = B3^-T dJ/dU
    line_basis<false>(ln, op.B, S1, Sv);
    line_basis<true>(ln, op.Bi, S1, Mv);
  }
  geo_to_shared(ln, geo, e, sg);
  __syncwarp();
#pragma unroll
  for (int j = 0; j < NPL; ++j) {  // mu = -lam / (w detJ)
    const int q = ln.q(j);
    const double sc = -iwab * op.iw[q] / (CV ? gve[kVolDetJ * NB + q + P * ln.l] : sg[kGeoDetJ]);
#pragma unroll
    for (int r = 0; r < 5; ++r) Mv[r][j] *= sc;
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    line_store<0, 0>(ln, S1 + r * VS, Sv[r]);
    line_store<0, 0>(ln, N1 + r * VS, Mv[r]);
  }
  __syncwarp();

  // ---- the volume term's transpose: derivatives of the state (of the energy
  // only for the heat flux) and of mu, then the pointwise reverse
  constexpr int ND = HT ? 5 : 4;
  line_derivatives<P, H, ND>(ln, op, S1);
  line_derivatives<P, H, 5>(ln, op, N1);
  __syncwarp();
#pragma unroll 1
  for (int j = 0; j < NPL; ++j) {
    const int i = ln.q(j), o = ln.at(i), oy = ln.template to<0, 1>(i), oz = ln.template to<0, 2>(i);
    double Jbuf[9], wJ;
    if constexpr (CV) {
      const double* gq = gve + i + P * ln.l;
#pragma unroll
      for (int c = 0; c < 9; ++c) Jbuf[c] = gq[c * NB];
      wJ = op.w[i] * wab * gq[kVolDetJ * NB];
    } else {
      wJ = op.w[i] * wab * sg[kGeoDetJ];
    }
    const double* Jq = CV ? Jbuf : sg + kGeoJinv;
    auto along_x = [&](const double (&t)[5][NPL], const double* tile, int r) {
      if constexpr (H == 2) {
        return tile[r * VS + o];
      } else {
        double g = op.Dq[i * P] * t[r][0];
#pragma unroll
        for (int m = 1; m < P; ++m) g = fma(op.Dq[i * P + m], t[r][m], g);
        return g;
      }
    };
    double S[5], Hb[3][5], Sb[5], Gb[3][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      S[r] = H == 2 ? Sv[r][0] : S1[r * VS + o];
      const double n0 = along_x(Mv, N1, r), n1 = N1[L::A + r * VS + oy], n2 = N1[2 * L::A + r * VS + oz];
#pragma unroll
      for (int c = 0; c < 3; ++c) Hb[c][r] = wJ * (n0 * Jq[c] + n1 * Jq[3 + c] + n2 * Jq[6 + c]);  // adjoint of Q - F
      Sb[r] = 0.;
    }
    euler_flux_vjp(S, gamma, Hb, Sb);
#pragma unroll
    for (int r = 0; r < 5; ++r) Sb[r] = -Sb[r];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < 5; ++r) Gb[c][r] = 0.;
    if (mu != 0.) {
      double Gp[3][5];
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        const double g0 = r < ND ? along_x(Sv, S1, r) : 0., g1 = r < ND ? S1[L::A + r * VS + oy] : 0.,
                     g2 = r < ND ? S1[2 * L::A + r * VS + oz] : 0.;
#pragma unroll
        for (int c = 0; c < 3; ++c) Gp[c][r] = r < ND ? Jq[c] * g0 + Jq[3 + c] * g1 + Jq[6 + c] * g2 : 0.;
      }
      visc_flux_vjp(S, Gp, mu, Hb, Sb, Gb, kq);
    }
    if (ln.owns(j)) {
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        S1[r * VS + o] = Sb[r];
        if (r < ND) {
          N1[r * VS + o] = Jq[0] * Gb[0][r] + Jq[1] * Gb[1][r] + Jq[2] * Gb[2][r];
          N1[L::A + r * VS + oy] = Jq[3] * Gb[0][r] + Jq[4] * Gb[1][r] + Jq[5] * Gb[2][r];
          N1[2 * L::A + r * VS + oz] = Jq[6] * Gb[0][r] + Jq[7] * Gb[1][r] + Jq[8] * Gb[2][r];
        }
      }
    }
    if constexpr (H == 2) {  // the next point's state
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int m = 1; m < NPL; ++m) Sv[r][m - 1] = Sv[r][m];
    }
  }
  __syncwarp();
  {  // S-bar + sum_i Dq_i^T g-bar_i along the lines of each axis, handed on in tile 0 of S1
    double c[NPL][P];
#pragma unroll
    for (int j = 0; j < NPL; ++j)
#pragma unroll
      for (int m = 0; m < P; ++m) c[j][m] = op.Dq[m * P + ln.q(j)];
    auto divergence = [&](auto axis) {
      constexpr int ax = decltype(axis)::value;
      double y[5][NPL];
#pragma unroll
      for (int r = 0; r < 5; ++r) {
#pragma unroll
        for (int j = 0; j < NPL; ++j) y[r][j] = S1[r * VS + ln.at(ln.q(j))];
        if (r < ND)
#pragma unroll
          for (int m = 0; m < P; ++m) {
            const double f = N1[ax * L::A + r * VS + ln.at(m)];
#pragma unroll
            for (int j = 0; j < NPL; ++j) y[r][j] = fma(c[j][m], f, y[r][j]);
          }
      }
      __syncwarp();
      if constexpr (ax < 2) {
#pragma unroll
        for (int r = 0; r < 5; ++r) line_store<ax, ax + 1>(ln, S1 + r * VS, y[r]);
      } else {
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
          for (int j = 0; j < NPL; ++j)
            if (ln.owns(j)) part[e * 5 * NB + r * NB + fq + NQF * ln.q(j)] = y[r][j];
      }
    };
    divergence(std::integral_constant<int, 0>());
    __syncwarp();
    divergence(std::integral_constant<int, 1>());
    __syncwarp();
    divergence(std::integral_constant<int, 2>());
  }
  line_spread<0, false>(ln, N1, Mv);
  __syncwarp();

  // ---- faces.  The lifting's transpose is pointwise like the lifting.
#pragma unroll 1
  for (int f = 0; f < 6 / H; ++f) {
    const int ax = H == 2 ? f : f >> 1, end = H == 2 ? ln.h : f & 1, lf = 2 * ax + end;
    const int ax1 = ax == 0 ? 1 : 0, ax2 = ax == 2 ? 1 : 2;
    const double* tile = N1 + ax * L::A;
    const int nb = nbr[e * 6 + lf];
    const double* To = Tr + (e * 6 + lf) * 10 * NQF + fq;
    double Uo[5], Un[5], lift_n = 0.;
#pragma unroll
    for (int r = 0; r < 5; ++r) Uo[r] = To[r * NQF];
    if (nb >= 0) {
      const double* Tn = Tr + ((long)nb * 6 + (lf ^ 1)) * 10 * NQF + fq;
#pragma unroll
      for (int r = 0; r < 5; ++r) Un[r] = Tn[r * NQF];
      lift_n = CV ? gf[(((long)nb * 6 + (lf ^ 1)) * kFaceC + kFaceLift) * NQF + fq]
                  : quot(op.cend[end ^ 1], geo[(long)nb * kGeoStride + kGeoDetJ]);
    }
    const double* gp = CV ? gfe + lf * kFaceC * NQF + fq : nullptr;
    double n[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) n[c] = CV ? gp[(kFaceN + c) * NQF] : sg[kGeoN + 3 * lf + c];
    const double fJ = CV ? gp[kFaceFJ * NQF] : sg[kGeoFJ + lf];
    const double fw = fJ * wab;
    const double lift = CV ? gp[kFaceLift * NQF] : quot(op.cend[end], sg[kGeoDetJ]);
    // mu and, for the viscous terms, its gradient at the face point
    double Sm[5], dcb[3][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) Sm[r] = 0.;
    {
      double dn[5] = {0., 0., 0., 0., 0.};
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const double ev = op.EL[end * P + k], dv = op.DL[end * P + k];
        const int o = ln.at(k);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          const double u = tile[r * VS + o];
          Sm[r] = fma(ev, u, Sm[r]);
          if (r > 0) dn[r] = fma(dv, u, dn[r]);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 5; ++r) dcb[c][r] = 0.;
      if (mu != 0.) {
        double d1[5], d2[5];
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const double c1 = op.Dq[ln.a * P + (ln.a + m) % P], c2 = op.Dq[ln.b * P + (ln.b + m) % P];
          const int s1 = ln.s1(m), s2 = ln.s2(m);
#pragma unroll
          for (int r = 1; r < 5; ++r) {
            d1[r] = m ? fma(c1, shfl_line(Sm[r], s1), d1[r]) : c1 * Sm[r];
            d2[r] = m ? fma(c2, shfl_line(Sm[r], s2), d2[r]) : c2 * Sm[r];
          }
        }
        // adjoint of the dual-consistency tensor: dc_bar[c] = -fw sum_i Jinv[i][c] grad_i(mu)
        const JacobianRows<double> J(CV ? gp : sg + kGeoJinv, CV ? NQF : 1, ax1, ax2, ax);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
          for (int r = 1; r < 5; ++r) dcb[c][r] = -fw * (J(0, c) * d1[r] + J(1, c) * d2[r] + J(2, c) * dn[r]);
      }
    }
    double* TAe = TA + ((e * 6 + lf) * kTraceAdj) * NQF + fq;
    const double ef = prm.eta * (nb >= 0 ? 0.5 : 1.0);
    if (nb >= 0) {
      double Uob[5] = {0., 0., 0., 0., 0.}, Unb[5] = {0., 0., 0., 0., 0.};
      const double iro = rcp(Uo[0]), irn = rcp(Un[0]);
      {  // in the element's own orientation: as a function the Roe flux is antisymmetric under swapping the sides
        double fb[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) fb[r] = fw * Sm[r];
        roe_flux_vjp_r(Uo, Un, iro, irn, n, gamma, fb, Uob, Unb);
      }
      if (mu != 0.) {
        double d[5], dbar[5] = {0., 0., 0., 0., 0.};
#pragma unroll
        for (int r = 0; r < 5; ++r) d[r] = Uo[r] - 0.5 * (Uo[r] + Un[r]);
        visc_rank1_vjp_r(Uo, iro, d, n, mu, dcb, Uob, dbar, kq);
        double rob[5], rnb[5];
        rob[0] = rnb[0] = 0.;  // the lifting has no mass component
#pragma unroll
        for (int r = 1; r < 5; ++r) {
          const double zb = ef * fJ * Sm[r];
          rob[r] = 0.5 * fw * lift * zb;
          rnb[r] = 0.5 * fw * lift_n * zb;
        }
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          Uob[r] += 0.5 * dbar[r];
          Unb[r] -= 0.5 * dbar[r];
          d[r] = Uo[r] - Un[r];
          dbar[r] = 0.;
        }
        visc_jump_n_vjp_r(Uo, iro, d, n, mu, rob, Uob, dbar, kq);
        visc_jump_n_vjp_r(Un, irn, d, n, mu, rnb, Unb, dbar, kq);
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          Uob[r] += dbar[r];
          Unb[r] -= dbar[r];
        }
      }
      if (ln.active) {
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          TAe[r * NQF] = Uob[r];
          TAe[(5 + r) * NQF] = -0.5 * fw * Sm[r];
          TAe[(10 + r) * NQF] = Unb[r];
        }
      }
    } else if (ln.active) {  // a call, so its registers stay out of the interior path
      AdjWallIn in;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        in.Uo[r] = Uo[r];
        in.ab[r] = Sm[r];
        in.zb[r] = r ? ef * fJ * Sm[r] : 0.;
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        in.n[c] = n[c];
#pragma unroll
        for (int r = 0; r < 5; ++r) in.dcb[c][r] = dcb[c][r];
      }
      in.fw = fw;
      in.lift = lift;
      adj_boundary_face_point(in, nb, prm, gamma, mu, kq, flag, TAe, NQF);
    }
    __syncwarp();
  }
}

template <int P, int H, bool CV, bool HT, bool NOD>
__global__ void __launch_bounds__(32, (LStage<P, H>::MINB))
ladjB_kernel(long count, const double* __restrict__ V, const double* __restrict__ TA, const __grid_constant__ LOps<P> op,
             const double* __restrict__ geo, const double* __restrict__ gf, const int* __restrict__ nbr,
             const __grid_constant__ DevParams prm, const double* __restrict__ part, const __grid_constant__ VjpArgs v)
{
  using L = LStage<P, H>;
  constexpr int NB = P * P * P, NQF = P * P, VS = LTile<P>::VS, NPL = L::NPL;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * L::UNIT;
  double* S1 = reinterpret_cast<double*>(eb);
  double* sg = reinterpret_cast<double*>(eb + L::oGeo);
  const long e = ln.u;
  const int fq = ln.l;
  const double mu = prm.mu, kq = HT ? prm.kq : 0.;
  {
    double t[5][NPL];
    if constexpr (NOD) {
      zline_from_memory(ln, V, e, t);
      line_basis<false>(ln, op.B, S1, t);
    } else {
      line_from_memory(ln, V, e, t);
    }
    line_spread<0, false>(ln, S1, t);
  }
  geo_to_shared(ln, geo, e, sg);
  __syncwarp();
  double yl[5][NPL];  // the adjoint at the lane's points of its line
#pragma unroll 1
  for (int ax = 0; ax < 3; ++ax) {
    const int ax1 = ax == 0 ? 1 : 0, ax2 = ax == 2 ? 1 : 2;
    const double* tile = S1 + ax * L::A;
    double ga[5], gb[5], pa[5], pb[5];  // value and normal-derivative adjoints: the (last) end's, the other's
#pragma unroll 1
    for (int f = 0; f < 2 / H; ++f) {
      const int end = H == 2 ? ln.h : f, lf = 2 * ax + end;
      // the trace adjoints: the element's own and the neighbour's side
      double vb[5], qb[5];
      {
        const int nb = nbr[e * 6 + lf];
        const double* To = TA + (e * 6 + lf) * kTraceAdj * NQF + fq;
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          vb[r] = To[r * NQF];
          qb[r] = To[(5 + r) * NQF];
        }
        if (nb >= 0) {
          const double* Tn = TA + ((long)nb * 6 + (lf ^ 1)) * kTraceAdj * NQF + fq;
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            vb[r] += Tn[(10 + r) * NQF];
            qb[r] -= Tn[(5 + r) * NQF];
          }
        }
      }
      double gn[5] = {0., 0., 0., 0., 0.};
      if (mu != 0.) {
        double S[5], dn[5], d1[5], d2[5];
#pragma unroll
        for (int r = 0; r < 5; ++r) S[r] = dn[r] = 0.;
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const double ev = op.EL[end * P + k], dv = op.DL[end * P + k];
          const int o = ln.at(k);
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            const double u = tile[r * VS + o];
            S[r] = fma(ev, u, S[r]);
            dn[r] = fma(dv, u, dn[r]);
          }
        }
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const double c1 = op.Dq[ln.a * P + (ln.a + m) % P], c2 = op.Dq[ln.b * P + (ln.b + m) % P];
          const int s1 = ln.s1(m), s2 = ln.s2(m);
#pragma unroll
          for (int r = 0; r < (HT ? 5 : 4); ++r) {
            d1[r] = m ? fma(c1, shfl_line(S[r], s1), d1[r]) : c1 * S[r];
            d2[r] = m ? fma(c2, shfl_line(S[r], s2), d2[r]) : c2 * S[r];
          }
        }
        // Qn = A(S, grad S) . n; rows of the inverse Jacobian: t1, t2, n
        const double* gp = CV ? gf + ((e * 6 + lf) * kFaceC) * NQF + fq : nullptr;
        const JacobianRows<double> J(CV ? gp : sg + kGeoJinv, CV ? NQF : 1, ax1, ax2, ax);
        double n[3], G[3][5], Gb[3][5];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          n[c] = CV ? gp[(kFaceN + c) * NQF] : sg[kGeoN + 3 * lf + c];
#pragma unroll
          for (int r = 0; r < 5; ++r)
            G[c][r] = r < 4 || HT ? J(0, c) * d1[r] + J(1, c) * d2[r] + J(2, c) * dn[r] : 0.;
        }
        visc_flux_n_vjp(S, G, n, mu, qb, vb, Gb, kq);
        double g1[5], g2[5];
#pragma unroll
        for (int r = 0; r < (HT ? 5 : 4); ++r) {
          g1[r] = J(0, 0) * Gb[0][r] + J(0, 1) * Gb[1][r] + J(0, 2) * Gb[2][r];
          g2[r] = J(1, 0) * Gb[0][r] + J(1, 1) * Gb[1][r] + J(1, 2) * Gb[2][r];
          gn[r] = J(2, 0) * Gb[0][r] + J(2, 1) * Gb[1][r] + J(2, 2) * Gb[2][r];
        }
#pragma unroll
        for (int m = 0; m < P; ++m) {  // the tangential derivatives' transposes
          const double c1 = op.Dq[((ln.a + m) % P) * P + ln.a], c2 = op.Dq[((ln.b + m) % P) * P + ln.b];
          const int s1 = ln.s1(m), s2 = ln.s2(m);
#pragma unroll
          for (int r = 0; r < (HT ? 5 : 4); ++r) {
            vb[r] = fma(c1, m ? shfl_line(g1[r], s1) : g1[r], vb[r]);
            vb[r] = fma(c2, m ? shfl_line(g2[r], s2) : g2[r], vb[r]);
          }
        }
      }
      if constexpr (H == 1) {
        if (f == 0) {
#pragma unroll
          for (int r = 0; r < 5; ++r) {
            pa[r] = vb[r];
            pb[r] = gn[r];
          }
        }
      }
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        ga[r] = vb[r];
        gb[r] = gn[r];
      }
    }
    if constexpr (H == 2) {
      const int s = ln.partner();
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        pa[r] = shfl_line(ga[r], s);
        pb[r] = r < 4 || HT ? shfl_line(gb[r], s) : 0.;
      }
    }
    const int eg = H == 2 ? ln.h : 1;  // the end of ga, gb
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int q = ln.q(j);
      const double ev = op.EL[eg * P + q], dv = op.DL[eg * P + q];
      const double eo = op.EL[(eg ^ 1) * P + q], dw = op.DL[(eg ^ 1) * P + q];
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        double y = fma(eo, pa[r], ev * ga[r]);
        if (r < 4 || HT) y = fma(dw, pb[r], fma(dv, gb[r], y));
        yl[r][j] = y + (ax > 0 ? S1[r * VS + ln.at(q)] : 0.);
      }
    }
    if (ax < 2) {  // on to the next axis' lines, in tile 0
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          const int q = ln.q(j);
          if (ln.owns(j))
            S1[r * VS + (ax == 0 ? ln.template to<0, 1>(q) : ln.template to<1, 2>(q))] = yl[r][j];
        }
      __syncwarp();
    }
  }
  // with the volume part; the running sum loaded before any store (acc_out may be acc_in)
  const long base = e * 5 * NB;
  double ai[5][NPL];
  auto point = [&](int r, int j) { return base + r * NB + (NOD ? P * fq + ln.q(j) : fq + NQF * ln.q(j)); };
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      yl[r][j] += part[base + r * NB + fq + NQF * ln.q(j)];
      ai[r][j] = v.acc_out && v.acc_in ? v.acc_in[point(r, j)] : 0.;
    }
  if constexpr (NOD) {  // dJ/dU = B3^T dJ/dV
    __syncwarp();
    line_basis<true>(ln, op.B, S1, yl);
  }
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      if (!ln.owns(j)) continue;
      if (v.a_out) v.a_out[point(r, j)] = yl[r][j];
      if (v.acc_out) v.acc_out[point(r, j)] = ai[r][j] + yl[r][j];
    }
}

// ------------------------------------------------------------ host launchers

template <int P, bool CV, bool HT, bool NOD>
cudaError_t ladj_launch(const KLaunch& L, const VjpArgs& v, const VjpScratch& s, const double* Tr, cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW;
  const LOps<P> op = line_ops<P>(L.table);
  const unsigned grid = (unsigned)((L.E + EPW - 1) / EPW);
  ladjA_kernel<P, H, CV, HT, NOD><<<grid, 32, LAdjA<P, H>::TOTAL, st>>>(L.E, v.U, Tr, v, op, L.geo, L.gv, L.gf, L.nbr,
                                                                        L.prm, s.part, s.ta, s.flag);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  ladjB_kernel<P, H, CV, HT, NOD><<<grid, 32, LStage<P, H>::TOTAL, st>>>(L.E, v.U, s.ta, op, L.geo, L.gf, L.nbr, L.prm,
                                                                         s.part, v);
  return cudaGetLastError();
}

}  // namespace dgb

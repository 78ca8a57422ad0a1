// The Gauss-point RK stage and trace kernels with lanes owning lines of Gauss
// points, P = 2..5.
//
// The P^2 lines of an element in each direction go to P^2 x H lanes: lane
// (a, b, h) owns, in turn, the x-line through (y, z) = (a, b), the y-line
// through (x, z) and the z-line through (x, y): all of it and both its end
// face points (H = 1), or half of its points and one end (H = 2, even P).  A
// warp takes 32 / (P^2 H) elements.  A contraction along a line reads the
// line once and gives all the lane's points of it, so an element tile crosses
// shared memory a few times per stage instead of P times per contraction; the
// element's lanes sit in one warp, so the phases are ordered by __syncwarp and
// what face points exchange (tangential derivatives, the two ends of a line)
// goes through shuffles.
//
// Per stage:
//   the state into a tile; the reference derivatives along y, z and x into
//   tiles (x in place of the state, which stays in registers)
//   volume flux at the lane's points, in place of the derivatives
//   per direction: the face fluxes at the line's ends, the divergence along
//   the line, Y handed on in the first tile
//   on z-lines the RK update, then the new state's tiles and its face traces
// A tile that is read along an axis lies in that axis' line order, so every
// phase addresses its lines alike, whatever the axis.
//
// What bounded the kernels before (a thread per Gauss point, each contraction
// reading its P inputs from shared memory): the shared-memory pipe, 75% busy
// at p = 3 with the FP64 pipe at 41% and the issue slots at 43%.  Here, at
// 24^3, p = 3 (one stage): 4.2 + 3.8 M shared-memory wavefronts instead of
// 22.2 + 8.0 M, 60.9 M warp instructions instead of 81.7 M, no pipe above 65%
// (shared memory and shuffles; FP64 36%, issue 49%): what is left is the
// latency of dependent instructions and of the face points' global loads at
// 15 warps an SM.  Stage at 32^3, p = 3: 369 -> 272 us on boxes along the axes,
// 345 us on other affine elements; p = 4 at 24^3 434 -> 273, p = 2 at 36^3 362 ->
// 222, p = 1 at 36^3 193 -> 82; trace kernel at 32^3, p = 3 115 -> 76 us.
#pragma once

#include "vspace.cuh"

namespace dgb {

// 1D operators, passed as a kernel parameter.
template <int P>
struct LOps {
  double Dq[P * P];             // Dq[q * P + k] = L_k'(x_q)
  double EL[2 * P], DL[2 * P];  // values and derivatives of L_q at the line's ends
  double w[P], cend[2];
  double B[P * P], Bi[P * P];   // nodal polynomials at the Gauss points, and the inverse
  double iw[P];                 // 1 / w
};

// Tile of one variable: point (x, y, z) at (x ^ y) + 4 y + 20 z at P = 4 (the
// lanes of a half-warp, each on its own line in any direction, fall in
// distinct 8-byte banks), else in plain order (odd strides; P = 2 is small).
template <int P>
struct LTile {
  static constexpr int PS = P == 4 ? 20 : P * P;
  static constexpr int VS = P == 4 ? 76 : P * P * P;  // entries per variable
};

template <int P, int H>
struct LStage {
  static constexpr int NPL = (P + H - 1) / H;  // points of a line per lane (odd P, H = 2: the second lane's last is no point)
  static constexpr int LE = P * P * H;    // lanes per element (or pair)
  static constexpr int EPW = 32 / LE;     // elements (or pairs) per warp
  static constexpr int ST = (int)sizeof(double);
  static constexpr int A = 5 * LTile<P>::VS;  // entries of one tile of five variables
  static constexpr int oGeo = align16(3 * A * ST);
  static constexpr int UNIT = oGeo + align16(kGeoStride * ST);
  static constexpr int TOTAL = EPW * UNIT;
  static_assert(TOTAL <= kSharedDefault, "shared memory of the line kernels");
  // Warps per SM the kernel is compiled for: the most whose registers hold a
  // lane's values.  Registers come per scheduler, so 16 warps have 128 each,
  // 12 have 168.  Measured: p = 3 at 32^3 267 us with 16, 310 with 20 (96
  // registers, spills), 365 with 12 (before AX: 355 with 16); p = 2 at 36^3
  // 219 us with 12, 236 with 16.
  static constexpr int MINB = P % H ? 8 : H == 2 ? 16 : 12;  // (P % H: small meshes only)
};

__device__ __forceinline__ double shfl_line(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float shfl_line(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ f2 shfl_line(f2 v, int src)
{
  return f2(__shfl_sync(0xffffffffu, v.v.x, src), __shfl_sync(0xffffffffu, v.v.y, src));
}

// A lane's place in its warp: its element (or pair) number u of the launch,
// active unless it has none (such a lane repeats another's loads and stores
// nothing); the line (a, b) and the part h of it; where lines lie in a tile.
template <int P, int H>
struct LLane {
  static constexpr int LE = P * P * H, EPW = 32 / LE, NPL = (P + H - 1) / H;
  using TL = LTile<P>;
  int slot, l, a, b, h;  // l = a + P b
  bool active;
  long u;
  __device__ explicit LLane(long count)
  {
    const int lane = threadIdx.x;
    slot = lane / LE < EPW ? lane / LE : EPW - 1;
    const int i = lane < EPW * LE ? lane - slot * LE : lane - EPW * LE;
    l = i / H;
    h = i % H;
    a = l % P;
    b = l / P;
    const long u0 = (long)blockIdx.x * EPW + slot;
    active = lane < EPW * LE && u0 < count;
    u = u0 < count ? u0 : count - 1;
  }
  __device__ int lane_of(int a_, int b_) const { return slot * LE + (a_ + P * b_) * H + h; }
  __device__ int partner() const { return slot * LE + l * H + (H - 1 - h); }
  // lanes m further along the face's first and second axis, cyclic
  __device__ int s1(int m) const { return lane_of((a + m) % P, b); }
  __device__ int s2(int m) const { return lane_of(a, (b + m) % P); }
  // the lane's j-th point of a line, if it is one (else some point)
  __device__ int q(int j) const
  {
    if (H == 1) return j;
    return P % H == 0 || h * NPL + j < P ? h * NPL + j : P - 1;
  }
  __device__ bool owns(int j) const { return active && (P % H == 0 || h * NPL + j < P); }
  // The place of entry k of line (a_, b_) in a tile of that line order: lines
  // follow one another in a, then b.
  __device__ static int place(int k, int a_, int b_) { return (P == 4 ? k ^ a_ : k) + P * a_ + TL::PS * b_; }
  __device__ int at(int k) const { return place(k, a, b); }  // of the lane's own line
  // point k of the lane's line along FROM in the line order of axis TO
  // (x-lines (y, z), y-lines (x, z), z-lines (x, y))
  template <int FROM, int TO>
  __device__ int to(int k) const
  {
    const int x = FROM == 0 ? k : a, y = FROM == 0 ? a : FROM == 1 ? k : b, z = FROM == 2 ? k : b;
    return TO == 0 ? place(x, y, z) : TO == 1 ? place(y, x, z) : place(z, x, y);
  }
};

// Variable r of the axis frame of AX elements (components n, t1, t2; the
// conserved order otherwise) along axis ax.
template <bool AX>
__device__ __forceinline__ constexpr int frame_var(int ax, int r)
{
  return !AX || r == 0 || r == 4 ? r : r == 1 ? 1 + ax : r == 2 ? (ax == 0 ? 2 : 1) : (ax == 2 ? 2 : 3);
}
// ... and the place of variable v in that frame
template <bool AX>
__device__ __forceinline__ constexpr int frame_slot(int ax, int v)
{
  for (int r = 1; r < 4; ++r)
    if (frame_var<AX>(ax, r) == v) return r;
  return v;
}

template <int P, int H, class T>
__device__ __forceinline__ void line_load(const LLane<P, H>& ln, const T* tile, T* v)
{
#pragma unroll
  for (int k = 0; k < P; ++k) v[k] = tile[ln.at(k)];
}

// the lane's own points of its line along FROM, into the line order of TO
template <int FROM, int TO, int P, int H, class T>
__device__ __forceinline__ void line_store(const LLane<P, H>& ln, T* tile, const T* v)
{
#pragma unroll
  for (int j = 0; j < LStage<P, H>::NPL; ++j)
    if (ln.owns(j)) tile[ln.template to<FROM, TO>(ln.q(j))] = v[j];
}

// The lane's points of the element's x-lines from memory.
template <int P, int H>
__device__ __forceinline__ void line_from_memory(const LLane<P, H>& ln, const double* Vs, long e, double (&t)[5][LStage<P, H>::NPL])
{
  constexpr int NB = P * P * P, NPL = LStage<P, H>::NPL;
  const double* g = Vs + e * 5 * NB + P * ln.l;
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    if constexpr (P % 2 == 0 && NPL == 2) {
      const double2 d = *reinterpret_cast<const double2*>(g + r * NB + ln.q(0));
      t[r][0] = d.x;
      t[r][1] = d.y;
    } else {
#pragma unroll
      for (int k = 0; k < NPL; ++k) t[r][k] = g[r * NB + ln.q(k)];
    }
  }
}

// The lane's points of the element's z-lines, from memory.
template <int P, int H>
__device__ __forceinline__ void zline_from_memory(const LLane<P, H>& ln, const double* Vs, long e,
                                                  double (&t)[5][LStage<P, H>::NPL])
{
  constexpr int NB = P * P * P, NQF = P * P, NPL = LStage<P, H>::NPL;
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j) t[r][j] = Vs[(e * 5 + r) * NB + ln.l + NQF * ln.q(j)];
}

// The lane's points of the element's x-lines, to memory.
template <int P, int H>
__device__ __forceinline__ void xline_to_memory(const LLane<P, H>& ln, double* Vs, long e,
                                                const double (&t)[5][LStage<P, H>::NPL])
{
  constexpr int NB = P * P * P, NPL = LStage<P, H>::NPL;
#pragma unroll
  for (int r = 0; r < 5; ++r)
#pragma unroll
    for (int j = 0; j < NPL; ++j)
      if (ln.owns(j)) Vs[(e * 5 + r) * NB + P * ln.l + ln.q(j)] = t[r][j];
}

// M x M x M (TR: its transpose) applied to five fields: values at the lane's
// points of its z-lines in, of its x-lines out.  tile: scratch of five fields,
// free before and after.
template <bool TR, int P, int H>
__device__ __forceinline__ void line_basis(const LLane<P, H>& ln, const double* M, double* tile,
                                           double (&t)[5][LStage<P, H>::NPL])
{
  constexpr int VS = LTile<P>::VS, NPL = LStage<P, H>::NPL;
  double c[NPL][P];
#pragma unroll
  for (int j = 0; j < NPL; ++j)
#pragma unroll
    for (int m = 0; m < P; ++m) c[j][m] = TR ? M[m * P + ln.q(j)] : M[ln.q(j) * P + m];
  auto contraction = [&](auto axis) {
    constexpr int ax = decltype(axis)::value;
#pragma unroll
    for (int r = 0; r < 5; ++r) line_store<ax == 2 ? 2 : ax + 1, ax>(ln, tile + r * VS, t[r]);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      double v[P];
      line_load(ln, tile + r * VS, v);
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        t[r][j] = c[j][0] * v[0];
#pragma unroll
        for (int m = 1; m < P; ++m) t[r][j] = fma(c[j][m], v[m], t[r][j]);
      }
    }
    __syncwarp();
  };
  contraction(std::integral_constant<int, 2>());
  contraction(std::integral_constant<int, 1>());
  contraction(std::integral_constant<int, 0>());
}

// The values t at the lane's points of its lines along FROM (variables in
// that axis' frame) into three tiles, one in the line order and the frame of
// each axis.
template <int FROM, bool AX, int P, int H, class T, int NPL>
__device__ __forceinline__ void line_spread(const LLane<P, H>& ln, T* tiles, const T (&t)[5][NPL])
{
  constexpr int VS = LTile<P>::VS, A = 5 * VS;
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    constexpr bool ax_ = AX;
    const int v = frame_var<ax_>(FROM, r);
    line_store<FROM, 0>(ln, tiles + frame_slot<ax_>(0, v) * VS, t[r]);
    line_store<FROM, 1>(ln, tiles + A + frame_slot<ax_>(1, v) * VS, t[r]);
    line_store<FROM, 2>(ln, tiles + 2 * A + frame_slot<ax_>(2, v) * VS, t[r]);
  }
}

// The element's geometry record into shared memory.
template <int P, int H>
__device__ __forceinline__ void geo_to_shared(const LLane<P, H>& ln, const double* __restrict__ geo, long e, double* sg)
{
  if (!ln.active) return;
  for (int i = ln.l * H + ln.h; i < kGeoStride; i += P * P * H) sg[i] = geo[e * kGeoStride + i];
}

// ---------------------------------------------------------------- axis frames
//
// Boxes along the coordinate axes (their nodes exactly so, geo_element_kernel)
// have a diagonal inverse Jacobian and face normals +-e_a.  Their kernels (AX) take
// the vectors of a line's phase in the frame of its axis, components (n, t1,
// t2) = (ax, ax1, ax2), by permuted addresses: metric products become scalings,
// normal components are components, and tensor entries that vanish for such a
// normal are neither formed nor exchanged.

// Components of A(S, g) e_n in the frame, from velocity derivatives
// dn[i] = d vel_i / d x_n and du[t] = d vel_n / d x_t, div: t = tau e_n.
__device__ __forceinline__ void axis_stress(double mu, const double* dn, double dv1, double dv2, double div, double* t)
{
  t[0] = 2. * mu * dn[0] - (2. / 3.) * mu * div;
  t[1] = mu * (dn[1] + dv1);
  t[2] = mu * (dn[2] + dv2);
}

// The ghost state in the frame of axis ax, outward sign s.
__device__ __forceinline__ int axis_boundary_state(int bt, const double* U, double s, int ax, const DevParams& prm, double* Ub)
{
  const double n[3] = {s, 0., 0.};
  const int bad = boundary_state_call(bt, U, n, prm, Ub);
  if (bt == DGB_BT_FREESTREAM) {
    Ub[1] = prm.Ufr[1 + ax];
    Ub[2] = prm.Ufr[ax == 0 ? 2 : 1];
    Ub[3] = prm.Ufr[ax == 2 ? 2 : 3];
  }
  return bad;
}

// face_flux_core for a face normal to an axis: states and fluxes in the frame
// (components n, t1, t2), fb rows t1, t2, n; j1, j2, jn: the diagonal of the
// inverse Jacobian.  Interior faces: both elements form the same bits of the
// Roe flux along +e_n (its central part and averages are symmetric in the two
// states, with no product fused into their sums, and its dissipation is odd
// in their difference), so what they add stays antisymmetric.  Boundary
// faces take the ghost state's Euler flux; the viscous terms are the interior
// ones with the ghost's weights.  VO: the viscous terms alone.
template <bool VO>
__device__ __forceinline__ void axis_face_flux(int ax, int end, int nb, const double* Uo, const double* Qo, double* Un, const double* Qn,
                                               double lift_n, double lift_o, double fJ, double fw, double j1, double j2, double jn,
                                               const DevParams& prm, double gamma, double mu, double kq, int* flag, double* fa, double* fb)
{
  const double s = end ? 1. : -1., gm1 = gamma - 1.;
  double lo, ln, half;  // weights of the lifting sources of both sides, and of the dual term
  double vo[3], vn[3], io, in;
  if (nb >= 0) {
    const double le = 0.25 * prm.eta * fJ;
    lo = le * lift_o;
    ln = le * lift_n;
    half = 0.5;
  } else {
    const int bad = axis_boundary_state(nb, Uo, s, ax, prm, Un);
    if (bad && flag) atomicOr(flag, 2);
    lo = 0.;
    ln = prm.eta * fJ * lift_o;
    half = 1.;
  }
  io = rcp(Uo[0]);
  in = rcp(Un[0]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    vo[i] = Uo[1 + i] * io;
    vn[i] = Un[1 + i] * in;
  }
  const double pn = gm1 * (Un[4] - 0.5 * (Un[1] * vn[0] + Un[2] * vn[1] + Un[3] * vn[2]));
  const double Hn = (Un[4] + pn) * in;
  double F[5] = {Un[1], Un[1] * vn[0] + pn, Un[1] * vn[1], Un[1] * vn[2], Un[1] * Hn};
  if constexpr (VO) {
#pragma unroll
    for (int r = 0; r < 5; ++r) fa[r] = nb >= 0 ? -0.5 * (Qo[r] - Qn[r]) : -Qo[r];
  } else if (nb >= 0) {
    const double po = gm1 * (Uo[4] - 0.5 * (Uo[1] * vo[0] + Uo[2] * vo[1] + Uo[3] * vo[2]));
    const double Ho = (Uo[4] + po) * io;
    const double sc = 0.5 * s;
    F[0] = sc * (F[0] + Uo[1]);
    F[1] = sc * (F[1] + (Uo[1] * vo[0] + po));
    F[2] = sc * __dadd_rn(F[2], __dmul_rn(Uo[1], vo[1]));
    F[3] = sc * __dadd_rn(F[3], __dmul_rn(Uo[1], vo[2]));
    F[4] = sc * __dadd_rn(F[4], __dmul_rn(Uo[1], Ho));
    const double so = sqrt_of(Uo[0], rsqrt_(Uo[0])), sn = sqrt_of(Un[0], rsqrt_(Un[0]));
    const double id = rcp(so + sn);
    auto mean = [&](double x, double y) { return __dadd_rn(__dmul_rn(so, x), __dmul_rn(sn, y)) * id; };
    const double u = mean(vo[0], vn[0]), v = mean(vo[1], vn[1]), w = mean(vo[2], vn[2]), H = mean(Ho, Hn);
    const double q2 = 0.5 * (u * u + v * v + w * w);
    const double c2 = gm1 * (H - q2);
    const double rc = rsqrt_(c2), c = sqrt_of(c2, rc), ic = rcp_from(c, rc);
    const double l1 = u + c, l2 = u - c, eps = 0.05 * c, e2 = eps * eps, i2e = 10. * ic;
    double a1 = fabs(l1), a2 = fabs(l2), a3 = fabs(u);
    a1 = select_lt(a1, eps, (e2 + l1 * l1) * i2e, a1);
    a2 = select_lt(a2, eps, (e2 + l2 * l2) * i2e, a2);
    a3 = select_lt(a3, eps, (e2 + u * u) * i2e, a3);
    const double s1 = 0.5 * (a1 + a2) - a3, s2 = 0.5 * (a1 - a2);
    double d[5];  // half the jump Un - Uo
#pragma unroll
    for (int r = 0; r < 5; ++r) d[r] = 0.5 * (Un[r] - Uo[r]);
    const double G1 = gm1 * (q2 * d[0] - (u * d[1] + v * d[2] + w * d[3]) + d[4]) * ic;
    const double G2 = d[1] - u * d[0];
    const double C1 = (G1 * s1 + G2 * s2) * ic, C2 = G1 * s2 + G2 * s1;
    F[0] -= a3 * d[0] + C1;
    F[1] -= a3 * d[1] + C1 * u + C2;
    F[2] -= a3 * d[2] + C1 * v;
    F[3] -= a3 * d[3] + C1 * w;
    F[4] -= a3 * d[4] + C1 * H + C2 * u;
#pragma unroll
    for (int r = 0; r < 5; ++r) fa[r] = F[r] - 0.5 * (Qo[r] - Qn[r]);
  } else {
#pragma unroll
    for (int r = 0; r < 5; ++r) fa[r] = s * F[r] - Qo[r];
  }
  if (mu != 0.) {
    const double lam = -(2. / 3.) * mu, m2 = 2. * mu + lam;
    double d[5], ao[3], an[3];
#pragma unroll
    for (int r = 0; r < 5; ++r) d[r] = Uo[r] - Un[r];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      ao[i] = (d[1 + i] - d[0] * vo[i]) * io;
      an[i] = (d[1 + i] - d[0] * vn[i]) * in;
    }
    {  // BR2 lifting sources of both sides
      const double o0 = lo * (m2 * ao[0]), o1 = lo * (mu * ao[1]), o2 = lo * (mu * ao[2]);
      const double n0 = ln * (m2 * an[0]), n1 = ln * (mu * an[1]), n2 = ln * (mu * an[2]);
      fa[1] += o0 + n0;
      fa[2] += o1 + n1;
      fa[3] += o2 + n2;
      fa[4] += vo[0] * o0 + vo[1] * o1 + vo[2] * o2 + (vn[0] * n0 + vn[1] * n1 + vn[2] * n2);
      if (kq != 0.) fa[4] += kq * (lo * heat_y(Uo, d) + ln * heat_y(Un, d));
    }
    // dual consistency
    const double b = -half * s * fw, b1 = b * j1, b2 = b * j2, bn = b * jn;
    fb[0] = b1 * (mu * ao[1]);
    fb[1] = b1 * (lam * ao[0]);
    fb[2] = 0.;
    fb[3] = vo[0] * fb[0] + vo[1] * fb[1];
    fb[4] = b2 * (mu * ao[2]);
    fb[5] = 0.;
    fb[6] = b2 * (lam * ao[0]);
    fb[7] = vo[0] * fb[4] + vo[2] * fb[6];
    fb[8] = bn * (m2 * ao[0]);
    fb[9] = bn * (mu * ao[1]);
    fb[10] = bn * (mu * ao[2]);
    fb[11] = vo[0] * fb[8] + vo[1] * fb[9] + vo[2] * fb[10];
    if (kq != 0.) fb[11] += bn * (kq * heat_y(Uo, d));
  } else {
#pragma unroll
    for (int i = 0; i < 12; ++i) fb[i] = 0.;
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) fa[r] *= fw;
}

// A(S, grad S) n at a face normal to an axis, outward sign s, in the frame:
// derivatives in physical coordinates along n (of the energy only with the
// heat flux), and along t1, t2 of the density, the normal momentum and that
// axis' own.
__device__ __forceinline__ void axis_visc_flux(const double* S, const double* gn, const double* g1, const double* g2, double s, double mu, double* Qn,
                                               double kq)
{
  const double ir = rcp(S[0]);
  const double v[3] = {S[1] * ir, S[2] * ir, S[3] * ir};
  double dn[3], t[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) dn[i] = (gn[1 + i] - gn[0] * v[i]) * ir;
  const double d1n = (g1[1] - g1[0] * v[0]) * ir, d11 = (g1[2] - g1[0] * v[1]) * ir;
  const double d2n = (g2[1] - g2[0] * v[0]) * ir, d22 = (g2[2] - g2[0] * v[2]) * ir;
  axis_stress(s * mu, dn, d1n, d2n, dn[0] + d11 + d22, t);
  Qn[0] = 0.;
  Qn[1] = t[0];
  Qn[2] = t[1];
  Qn[3] = t[2];
  Qn[4] = v[0] * t[0] + v[1] * t[1] + v[2] * t[2];
  if (kq != 0.) Qn[4] += s * kq * heat_y(S, gn);
}

// The face traces at the face point (ax, end) of the lane's line, of the state
// in the tile of axis ax (line_spread), into Te (the element's slice of the trace buffer): value and
// normal derivative from the line, tangential derivatives from the face's
// other points by shuffles, then A(U, grad U) . n.
template <int P, int H, bool CV, bool HT, bool AX>
__device__ __forceinline__ void line_trace(const LLane<P, H>& ln, const LOps<P>& op, int ax, int end, const double* tile,
                                           const double* sg, const double* gfe, double mu, double kq, double* __restrict__ Te)
{
  constexpr int NQF = P * P, VS = LTile<P>::VS;
  const int lf = 2 * ax + end, fq = ln.l;
  const int ax1 = ax == 0 ? 1 : 0, ax2 = ax == 2 ? 1 : 2;
  const int var[5] = {0, AX ? 1 + ax : 1, AX ? 1 + ax1 : 2, AX ? 1 + ax2 : 3, 4};  // frame_var
  double S[5], dn[5], Qn[5];
#pragma unroll
  for (int r = 0; r < 5; ++r) S[r] = dn[r] = Qn[r] = 0.;
#pragma unroll
  for (int k = 0; k < P; ++k) {
    const double ev = op.EL[end * P + k], dv = op.DL[end * P + k];
    const int o = ln.at(k);
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      const double v = tile[r * VS + o];
      S[r] = fma(ev, v, S[r]);
      if (r < 4 || HT) dn[r] = fma(dv, v, dn[r]);
    }
  }
  if (mu != 0.) {
    // the tangential derivatives that the flux needs: of the energy only with
    // the heat flux, and none there or of the other tangential momentum (AX)
    double d1[5], d2[5];
#pragma unroll
    for (int m = 0; m < P; ++m) {
      const double c1 = op.Dq[ln.a * P + (ln.a + m) % P], c2 = op.Dq[ln.b * P + (ln.b + m) % P];
      const int s1 = ln.s1(m), s2 = ln.s2(m);
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        if (AX ? r != 4 && r != 3 : r < 4 || HT) d1[r] = m ? fma(c1, shfl_line(S[r], s1), d1[r]) : c1 * S[r];
        if (AX ? r != 4 && r != 2 : r < 4 || HT) d2[r] = m ? fma(c2, shfl_line(S[r], s2), d2[r]) : c2 * S[r];
      }
    }
    if constexpr (AX) {
      const double jn = sg[kGeoJinv + 4 * ax], j1 = sg[kGeoJinv + 4 * ax1], j2 = sg[kGeoJinv + 4 * ax2];
      const double g1[3] = {j1 * d1[0], j1 * d1[1], j1 * d1[2]}, g2[3] = {j2 * d2[0], j2 * d2[1], j2 * d2[3]};
#pragma unroll
      for (int r = 0; r < 5; ++r) dn[r] *= jn;
      axis_visc_flux(S, dn, g1, g2, end ? 1. : -1., mu, Qn, kq);
    } else {
      // rows of the inverse Jacobian: the face's two tangential axes, its normal axis
      double G[3][5], n[3];
      const double* gp = CV ? gfe + lf * kFaceC * NQF + fq : nullptr;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double j1 = CV ? gp[(3 * ax1 + c) * NQF] : sg[kGeoJinv + 3 * ax1 + c];
        const double j2 = CV ? gp[(3 * ax2 + c) * NQF] : sg[kGeoJinv + 3 * ax2 + c];
        const double jn = CV ? gp[(3 * ax + c) * NQF] : sg[kGeoJinv + 3 * ax + c];
        n[c] = CV ? gp[(kFaceN + c) * NQF] : sg[kGeoN + 3 * lf + c];
#pragma unroll
        for (int r = 0; r < 5; ++r) G[c][r] = r < 4 || HT ? (j1 * d1[r] + j2 * d2[r] + jn * dn[r]) : 0.;
      }
      visc_flux_n(S, G, n, mu, Qn, kq);
    }
  }
  if (ln.active) {
    double* Tq = Te + lf * 10 * NQF + fq;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      Tq[var[r] * NQF] = S[r];
      Tq[(5 + var[r]) * NQF] = Qn[r];
    }
  }
}

// the lane's face points of all directions
template <int P, int H, bool CV, bool HT, bool AX>
__device__ __forceinline__ void line_traces(const LLane<P, H>& ln, const LOps<P>& op, const double* tiles, const double* sg,
                                            const double* gfe, double mu, double kq, double* __restrict__ Te)
{
#pragma unroll 1
  for (int f = 0; f < 6 / H; ++f) {
    const int ax = H == 2 ? f : f >> 1, end = H == 2 ? ln.h : f & 1;
    line_trace<P, H, CV, HT, AX>(ln, op, ax, end, tiles + ax * (5 * LTile<P>::VS), sg, gfe, mu, kq, Te);
  }
}

// Face traces of a Gauss-point state V into Tr.  NOD: of a nodal state.
template <int P, int H, bool CV, bool HT, bool AX, bool NOD = false>
__global__ void __launch_bounds__(32, 16)
ltrace_kernel(long count, const double* __restrict__ V, const __grid_constant__ LOps<P> op,
              const double* __restrict__ geo, const double* __restrict__ gf, double* __restrict__ Tr, DevParams prm)
{
  using L = LStage<P, H>;
  constexpr int NQF = P * P;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * L::UNIT;
  double* S1 = reinterpret_cast<double*>(eb);
  double* sg = reinterpret_cast<double*>(eb + L::oGeo);
  const long e = ln.u;
  double t[5][L::NPL];
  if constexpr (NOD) {
    zline_from_memory(ln, V, e, t);
    line_basis<false>(ln, op.B, S1, t);
  } else {
    line_from_memory(ln, V, e, t);
  }
  line_spread<0, AX>(ln, S1, t);
  geo_to_shared(ln, geo, e, sg);
  __syncwarp();
  line_traces<P, H, CV, HT, AX>(ln, op, S1, sg, CV ? gf + e * 6 * kFaceC * NQF : nullptr, prm.mu,
                           HT ? prm.kq : 0., Tr + ln.u * 60 * NQF);
}

// One RK stage; arguments as vstage_kernel.  VO: the viscous terms alone.
// NOD: the residual of a nodal state (MODE_RESIDUAL), f and R nodal too.
template <int P, int H, bool CV, bool HT, bool AX, bool VO = false, bool NOD = false>
__global__ void __launch_bounds__(32, (LStage<P, H>::MINB))
lstage_kernel(long count, const double* Vs, const double* __restrict__ Tr, const __grid_constant__ LOps<P> op,
              const double* __restrict__ geo, const double* __restrict__ gv, const double* __restrict__ gf,
              const int* __restrict__ nbr, const __grid_constant__ DevParams prm,
              const __grid_constant__ StageArgs sa)
{
  using L = LStage<P, H>;
  constexpr int NB = P * P * P, NQF = P * P, VS = LTile<P>::VS, NPL = L::NPL;
  extern __shared__ __align__(16) unsigned char smraw[];
  const LLane<P, H> ln(count);
  unsigned char* eb = smraw + ln.slot * L::UNIT;
  // tile 0: the state, its x derivatives (H = 2), the x fluxes, Y; tiles 1, 2:
  // the y and z derivatives, then fluxes; all three: the new state
  double* S1 = reinterpret_cast<double*>(eb);
  double* sg = reinterpret_cast<double*>(eb + L::oGeo);
  const bool active = ln.active;
  const long e = sa.ebase + sa.estep * ln.u;
  const int fq = ln.l;  // the lane's face point
  int* const flag = active ? sa.flag : nullptr;  // (a lane without an element has no normal either)
  const double* Ve = Vs + e * 5 * NB;

  double Sv[5][NPL];  // the state at the lane's points of its x-line
  if constexpr (NOD) {
    zline_from_memory(ln, Vs, e, Sv);
    line_basis<false>(ln, op.B, S1, Sv);
  } else {
    line_from_memory(ln, Vs, e, Sv);
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) line_store<0, 0>(ln, S1 + r * VS, Sv[r]);
  geo_to_shared(ln, geo, e, sg);
  __syncwarp();

  const double gamma = prm.gamma, mu = prm.mu, kq = HT ? prm.kq : 0.;
  const double wab = op.w[ln.a] * op.w[ln.b];
  const double* gve = CV ? gv + e * kVolC * NB : nullptr;
  const double* gfe = CV ? gf + e * 6 * kFaceC * NQF : nullptr;

  // ---------------- reference derivatives along y, z and (H = 2; else from
  // the registers at each point) x, the last in place of the state; the
  // energy's only for the heat flux
  constexpr int ND = HT ? 5 : 4;
  {
    double c[NPL][P];
#pragma unroll
    for (int j = 0; j < NPL; ++j)
#pragma unroll
      for (int m = 0; m < P; ++m) c[j][m] = op.Dq[ln.q(j) * P + m];
    auto derivative = [&](auto axis) {
      constexpr int ax = decltype(axis)::value;
      double d[ND][NPL];
#pragma unroll
      for (int r = 0; r < ND; ++r) {
#pragma unroll
        for (int m = 0; m < P; ++m) {
          const double v = S1[r * VS + ln.template to<ax, 0>(m)];
#pragma unroll
          for (int j = 0; j < NPL; ++j) d[r][j] = m ? fma(c[j][m], v, d[r][j]) : c[j][m] * v;
        }
      }
      if (ax == 0) __syncwarp();  // all have read the state
#pragma unroll
      for (int r = 0; r < ND; ++r) line_store<ax, ax>(ln, S1 + ax * L::A + r * VS, d[r]);
    };
    derivative(std::integral_constant<int, 1>());
    derivative(std::integral_constant<int, 2>());
    if constexpr (H == 2) derivative(std::integral_constant<int, 0>());
  }
  __syncwarp();

  // ---------------- volume flux (solve.cpp:276-341) at the lane's points
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
    double S[5], Gp[3][5], F[3][5];
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      S[r] = H == 2 ? Sv[r][0] : S1[r * VS + o];
      if (r == 4 && !HT) {
        Gp[0][r] = Gp[1][r] = Gp[2][r] = 0.;
        continue;
      }
      double gx;
      if constexpr (H == 2) {
        gx = S1[r * VS + o];
      } else {
        gx = op.Dq[i * P] * Sv[r][0];
#pragma unroll
        for (int m = 1; m < P; ++m) gx = fma(op.Dq[i * P + m], Sv[r][m], gx);
      }
      const double gy = S1[L::A + r * VS + oy], gz = S1[2 * L::A + r * VS + oz];
      if constexpr (AX) {
        Gp[0][r] = Jq[0] * gx;
        Gp[1][r] = Jq[4] * gy;
        Gp[2][r] = Jq[8] * gz;
      } else {
#pragma unroll
        for (int c = 0; c < 3; ++c) Gp[c][r] = Jq[c] * gx + Jq[3 + c] * gy + Jq[6 + c] * gz;
      }
    }
    if constexpr (VO) {
      visc_flux(S, Gp, mu, F, kq);
    } else if (euler_flux(S, gamma, F); mu != 0.) {
      double Q[3][5];
      visc_flux(S, Gp, mu, Q, kq);
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 5; ++r) F[c][r] = Q[c][r] - F[c][r];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int r = 0; r < 5; ++r) F[c][r] = -F[c][r];
    }
    if (ln.owns(j)) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        const double wj = AX ? (wJ * Jq[4 * m]) : wJ;
#pragma unroll
        for (int r = 0; r < 5; ++r)
          S1[m * L::A + frame_slot<AX>(m, r) * VS + (m == 0 ? o : m == 1 ? oy : oz)] =
              AX ? (wj * F[m][r]) : wj * (Jq[3 * m] * F[0][r] + Jq[3 * m + 1] * F[1][r] + Jq[3 * m + 2] * F[2][r]);
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

  double yl[5][NPL];  // Y at the lane's points of its line (AX: in the axis frame)
#pragma unroll 1
  for (int ax = 0; ax < 3; ++ax) {
    const int ax1 = ax == 0 ? 1 : 0, ax2 = ax == 2 ? 1 : 2;
    const int var[5] = {0, AX ? 1 + ax : 1, AX ? 1 + ax1 : 2, AX ? 1 + ax2 : 3, 4};
    // ---------------- the faces at the line's ends (solve.cpp:393-794)
    double ga[5], gb[4];  // what the end (H = 1: the last one) adds through EL and DL; H = 1: the first end's
    double pa[5], pb[4];
#pragma unroll 1
    for (int f = 0; f < 2 / H; ++f) {
      const int end = H == 2 ? ln.h : f, lf = 2 * ax + end;
      double fa[5], fb[12];  // fb rows: the two tangential axes, the normal axis
      const double* To = Tr + (e * 6 + lf) * 10 * NQF + fq;
      const int nb = nbr[e * 6 + lf];
      const double* gp = CV ? gfe + lf * kFaceC * NQF + fq : nullptr;
      double n[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) n[c] = CV ? gp[(kFaceN + c) * NQF] : sg[kGeoN + 3 * lf + c];
      const double fJ = CV ? gp[kFaceFJ * NQF] : sg[kGeoFJ + lf];
      const double fw = fJ * wab;
      auto Jf = [&]() {  // rows in fb's order
        if constexpr (CV)
          return JacobianRows<double>(gp, NQF, ax1, ax2, ax);
        else
          return JacobianRows<double>(sg + kGeoJinv, 1, ax1, ax2, ax);
      };
      auto lift = [&]() { return CV ? gp[kFaceLift * NQF] : quot(op.cend[end], sg[kGeoDetJ]); };
      double Uo[5], Qo[5], Un[5], Qn[5], lift_n = 0.;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        Uo[r] = To[var[r] * NQF];
        Qo[r] = To[(5 + var[r]) * NQF];
      }
      if (nb >= 0) {
        const double* Tn = Tr + ((long)nb * 6 + (lf ^ 1)) * 10 * NQF + fq;
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          Un[r] = Tn[var[r] * NQF];
          Qn[r] = Tn[(5 + var[r]) * NQF];
        }
        lift_n = CV ? gf[(((long)nb * 6 + (lf ^ 1)) * kFaceC + kFaceLift) * NQF + fq]
                    : quot(op.cend[end ^ 1], geo[(long)nb * kGeoStride + kGeoDetJ]);
      }
      if constexpr (AX)
        axis_face_flux<VO>(ax, end, nb, Uo, Qo, Un, Qn, lift_n, lift(), fJ, fw, sg[kGeoJinv + 4 * ax1],
                       sg[kGeoJinv + 4 * ax2], sg[kGeoJinv + 4 * ax], prm, gamma, mu, kq, flag, fa, fb);
      else
        face_flux_core<double, 1, VO, true>(end, nb, Uo, Qo, Un, Qn, lift_n, n, fJ, fw, Jf, lift, prm, gamma, mu, kq,
                                          flag, fa, fb);
      if (mu != 0.) {  // tangential test derivatives: Dq^double fb along the face's two axes (AX: fb[2] = fb[5] = 0)
        const double c1 = op.Dq[ln.a * P + ln.a], c2 = op.Dq[ln.b * P + ln.b];
        double g[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          g[r] = AX && r == 2 ? fa[1 + r] : fma(c1, fb[r], fa[1 + r]);
          if (!AX || r != 1) g[r] = fma(c2, fb[4 + r], g[r]);
        }
#pragma unroll
        for (int m = 1; m < P; ++m) {
          const double d1 = op.Dq[((ln.a + m) % P) * P + ln.a], d2 = op.Dq[((ln.b + m) % P) * P + ln.b];
          const int s1 = ln.s1(m), s2 = ln.s2(m);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (!AX || r != 2) g[r] = fma(d1, shfl_line(fb[r], s1), g[r]);
            if (!AX || r != 1) g[r] = fma(d2, shfl_line(fb[4 + r], s2), g[r]);
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) fa[1 + r] = g[r];
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
    if constexpr (H == 2) {  // the other end's, from the lane that has it
      const int s = ln.partner();
#pragma unroll
      for (int r = 0; r < 5; ++r) pa[r] = shfl_line(ga[r], s);
#pragma unroll
      for (int r = 0; r < 4; ++r) pb[r] = mu != 0. ? shfl_line(gb[r], s) : 0.;
    }
    // ---------------- both onto the lane's points of the line, the divergence
    // along it, and Y so far
    {
      const int eg = H == 2 ? ln.h : 1;  // the end of ga, gb
      double ev[NPL], dv[NPL], eo[NPL], dw[NPL];
#pragma unroll
      for (int j = 0; j < NPL; ++j) {
        ev[j] = op.EL[eg * P + ln.q(j)];
        dv[j] = op.DL[eg * P + ln.q(j)];
        eo[j] = op.EL[(eg ^ 1) * P + ln.q(j)];
        dw[j] = op.DL[(eg ^ 1) * P + ln.q(j)];
      }
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          double y = fma(eo[j], pa[r], ev[j] * ga[r]);
          if (r > 0) y = fma(dw[j], pb[r - 1 < 0 ? 0 : r - 1], fma(dv[j], gb[r - 1 < 0 ? 0 : r - 1], y));
          yl[r][j] = y;
        }
    }
    {
      double c[NPL][P];
#pragma unroll
      for (int j = 0; j < NPL; ++j)
#pragma unroll
        for (int m = 0; m < P; ++m) c[j][m] = op.Dq[m * P + ln.q(j)];
      const double* F = S1 + ax * L::A;
#pragma unroll
      for (int r = 0; r < 5; ++r) {
        double f[P];
        line_load(ln, F + r * VS, f);
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          if (ax > 0) yl[r][j] += S1[r * VS + ln.at(ln.q(j))];
#pragma unroll
          for (int m = 0; m < P; ++m) yl[r][j] = fma(c[j][m], f[m], yl[r][j]);
        }
      }
    }
    if (ax < 2) {  // Y on to the next axis' lines, in its frame
      __syncwarp();  // all have read tile 0
      {
#pragma unroll
        for (int r = 0; r < 5; ++r) {
          constexpr bool ax_ = AX;
          const int slot = ax == 0 ? frame_slot<ax_>(1, frame_var<ax_>(0, r)) : frame_slot<ax_>(2, frame_var<ax_>(1, r));
#pragma unroll
          for (int j = 0; j < NPL; ++j) {
            const int q = ln.q(j);
            if (ln.owns(j))
              S1[slot * VS + (ax == 0 ? ln.template to<0, 1>(q) : ln.template to<1, 2>(q))] = yl[r][j];
          }
        }
      }
      __syncwarp();
    }
  }
  constexpr int zv[5] = {0, AX ? 3 : 1, AX ? 1 : 2, AX ? 2 : 3, 4};  // the variables of yl on z-lines
#pragma unroll
  for (int j = 0; j < NPL; ++j) {  // the source (solve.cpp:345-360), tested with w detJ
    const int q = ln.q(j);
    const double wJ = op.w[q] * wab * (CV ? gve[kVolDetJ * NB + fq + NQF * q] : sg[kGeoDetJ]);
#pragma unroll
    for (int r = 0; r < 5; ++r) yl[r][j] -= prm.src[zv[r]] * wJ;
  }

  // ---------------- norm partial: the nodal residual R = B3^double Y
  if (sa.part) {
    double s = 0., t[5][NPL];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int j = 0; j < NPL; ++j) t[r][j] = yl[r][j];
    line_basis<true>(ln, op.B, S1 + L::A, t);  // (in the y fluxes' place)
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int j = 0; j < NPL; ++j)
        if (ln.owns(j)) s += t[r][j] * t[r][j];
    // over the element's lanes, in a fixed order
    const int i = ln.l * H + ln.h;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double o = __shfl_down_sync(0xffffffffu, s, off);
      if (i + off < L::LE) s += o;
    }
    if (active && i == 0) sa.part[e] = s;
  }

  // ---------------- f_V = -Y / (w detJ), RK update, on the z-line
  {
    const double iwab = op.iw[ln.a] * op.iw[ln.b];
    const double id = CV ? 0. : -1.0 / sg[kGeoDetJ];
    const long base = e * 5 * NB + fq + NQF * ln.q(0);
    double sc[NPL];
#pragma unroll
    for (int j = 0; j < NPL; ++j) {
      const int q = ln.q(j);
      if constexpr (CV)
        sc[j] = -iwab * op.iw[q] / gve[kVolDetJ * NB + fq + NQF * q];
      else
        sc[j] = iwab * op.iw[q] * id;
    }
    if constexpr (NOD) {  // R = B3^T Y, f = B3^-1 (-Y / (w detJ))
      double t[5][NPL];
      __syncwarp();
      if (sa.Rout) {
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
          for (int j = 0; j < NPL; ++j) t[zv[r]][j] = yl[r][j];
        line_basis<true>(ln, op.B, S1, t);
        xline_to_memory(ln, sa.Rout, e, t);
      }
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) t[zv[r]][j] = yl[r][j] * sc[j];
      line_basis<false>(ln, op.Bi, S1, t);
      xline_to_memory(ln, sa.fout, e, t);
      return;
    }
    // the operands of RC variables are all loaded before any result is stored
    constexpr int RC = NPL > 4 ? 3 : 5;
#pragma unroll
    for (int r0 = 0; r0 < 5; r0 += RC) {
      RkOperands o[RC][NPL];
      if (sa.mode != MODE_RESIDUAL) {
#pragma unroll
        for (int r = r0; r < 5 && r < r0 + RC; ++r)
#pragma unroll
          for (int j = 0; j < NPL; ++j) {
            const long g = base + zv[r] * NB + NQF * (P % H == 0 ? j : ln.q(j) - ln.q(0));
            o[r - r0][j] = rk_stage_load(sa, g, Vs + g);
          }
      }
#pragma unroll
      for (int r = r0; r < 5 && r < r0 + RC; ++r)
#pragma unroll
        for (int j = 0; j < NPL; ++j) {
          const long g = base + zv[r] * NB + NQF * (P % H == 0 ? j : ln.q(j) - ln.q(0));
          if (!ln.owns(j)) continue;
          if (sa.mode == MODE_RESIDUAL) {
            sa.fout[g] = yl[r][j] * sc[j];
          } else {  // yl: the new state, for the traces
            yl[r][j] = rk_stage_apply(sa, g, yl[r][j] * sc[j], o[r - r0][j]);
            sa.Uout[g] = yl[r][j];
          }
        }
    }
  }
  // ---------------- face traces of the new state for the next stage
  if (sa.Tnext) {
    __syncwarp();  // the tiles are free
    line_spread<2, AX>(ln, S1, yl);
    __syncwarp();
    line_traces<P, H, CV, HT, AX>(ln, op, S1, sg, gfe, mu, kq, reinterpret_cast<double*>(sa.Tnext) + e * 60 * NQF);
  }
}

// ------------------------------------------------------------ host launchers

template <int P>
LOps<P> line_ops(const double* table)
{
  using C = Cfg<P>;
  LOps<P> o;
  for (int i = 0; i < P * P; ++i) {
    o.Dq[i] = table[C::oDq + i];
    o.B[i] = table[C::oB + i];
    o.Bi[i] = table[C::oBi + i];
  }
  for (int i = 0; i < 2 * P; ++i) {
    o.EL[i] = table[C::oEh + i];
    o.DL[i] = table[C::oDh + i];
  }
  for (int i = 0; i < P; ++i) {
    o.w[i] = table[C::oW + i];
    o.iw[i] = 1.0 / table[C::oW + i];
  }
  for (int i = 0; i < 2; ++i) o.cend[i] = table[C::oC + i];
  return o;
}

template <int P, int H, bool CV, bool HT>
cudaError_t llaunch_stage_ph(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                             cudaStream_t st)
{
  constexpr int EPW = LStage<P, H>::EPW;
  const long count = sa.ecount ? sa.ecount : L.E;
  const StageArgs so = element_order(sa, L.E, 1);
  const auto launch = [&](auto kernel) {
    kernel<<<(unsigned)((count + EPW - 1) / EPW), 32, LStage<P, H>::TOTAL, st>>>(
        count, Vs, reinterpret_cast<const double*>(Tin), line_ops<P>(L.table), L.geo, L.gv, L.gf, L.nbr, L.prm, so);
  };
  if constexpr (!CV)
    if (L.axis) {
      launch(lstage_kernel<P, H, CV, HT, true>);
      return cudaGetLastError();
    }
  launch(lstage_kernel<P, H, CV, HT, false>);
  return cudaGetLastError();
}

// the viscous terms alone (sa.mode MODE_RESIDUAL), any mesh of line kernels
template <int P, bool CV, bool HT>
cudaError_t llaunch_visc_pc(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW, smem = LStage<P, H>::TOTAL;
  const StageArgs so = element_order(sa, L.E, 1);
  const auto launch = [&](auto kernel) {
    kernel<<<(unsigned)((L.E + EPW - 1) / EPW), 32, smem, st>>>(L.E, Vs, reinterpret_cast<const double*>(Tin),
                                                                line_ops<P>(L.table), L.geo, L.gv, L.gf, L.nbr, L.prm,
                                                                so);
    return cudaGetLastError();
  };
  if constexpr (!CV)
    if (L.axis) return launch(lstage_kernel<P, H, CV, HT, true, true>);
  return launch(lstage_kernel<P, H, CV, HT, false, true>);
}

// f and R of a nodal state with its traces Tin
template <int P, bool CV, bool HT>
cudaError_t llaunch_residual_pc(const KLaunch& L, const double* U, const void* Tin, const StageArgs& sa, cudaStream_t st)
{
  constexpr int H = LineShape<P>::H, EPW = LStage<P, H>::EPW, smem = LStage<P, H>::TOTAL;
  const auto launch = [&](auto kernel) {
    kernel<<<(unsigned)((L.E + EPW - 1) / EPW), 32, smem, st>>>(L.E, U, reinterpret_cast<const double*>(Tin),
                                                                line_ops<P>(L.table), L.geo, L.gv, L.gf, L.nbr, L.prm,
                                                                element_order(sa, L.E, 1));
    return cudaGetLastError();
  };
  if constexpr (!CV)
    if (L.axis) return launch(lstage_kernel<P, H, CV, HT, true, false, true>);
  return launch(lstage_kernel<P, H, CV, HT, false, false, true>);
}

template <int P, bool CV, bool HT>
cudaError_t llaunch_stage_pc(const KLaunch& L, const double* Vs, const void* Tin, const StageArgs& sa,
                             cudaStream_t st)
{
  if constexpr (LineShape<P>::SPLIT != LineShape<P>::H)
    if (L.line == LINE_SPLIT) return llaunch_stage_ph<P, LineShape<P>::SPLIT, CV, HT>(L, Vs, Tin, sa, st);
  return llaunch_stage_ph<P, LineShape<P>::H, CV, HT>(L, Vs, Tin, sa, st);
}

template <int P, int H, bool CV, bool HT>
cudaError_t llaunch_trace_ph(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  using K = LStage<P, H>;
  const auto launch = [&](auto kernel) {
    kernel<<<(unsigned)((L.E + K::EPW - 1) / K::EPW), 32, K::TOTAL, st>>>(
        L.E, V, line_ops<P>(L.table), L.geo, L.gf, reinterpret_cast<double*>(Tout), L.prm);
  };
  if constexpr (!CV)
    if (L.axis) {
      launch(ltrace_kernel<P, H, CV, HT, true>);
      return cudaGetLastError();
    }
  launch(ltrace_kernel<P, H, CV, HT, false>);
  return cudaGetLastError();
}

template <int P, bool CV, bool HT>
cudaError_t llaunch_trace_pc(const KLaunch& L, const double* V, void* Tout, cudaStream_t st)
{
  if constexpr (LineShape<P>::SPLIT != LineShape<P>::H)
    if (L.line == LINE_SPLIT) return llaunch_trace_ph<P, LineShape<P>::SPLIT, CV, HT>(L, V, Tout, st);
  return llaunch_trace_ph<P, LineShape<P>::H, CV, HT>(L, V, Tout, st);
}

}  // namespace dgb

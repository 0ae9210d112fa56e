// Per-voxel update of the pseudo-time Stokes sweep (the body of
// central_diff5, src/solver.cc:136-220 of the reference) in two arithmetic
// forms:
//   * update_exact: the reference's operation order term by term (translation
//     units that use it are compiled with -fmad=false), bit-identical to the
//     reference CPU program;
//   * update_fast: the same linear map regrouped into a coefficient form with
//     FMAs (31 FP64 instructions per fluid voxel in FP64, where the relaxation
//     is folded into the coefficients and the centre coefficient comes from a
//     16-entry table; about 39 in FP32; instead of ~70 plus three divisions),
//     used by the FP64 fast sweeps, the FP64 residual and the FP32 correction
//     sweeps of the mixed-precision form.
#pragma once

#include "pm_internal.h"

namespace pm {

// Values of the 4 fields a fluid voxel reads (axis-aligned offsets only).
template <typename T>
struct Stencil {
  T uc, uxm, uxp, uym, uyp, uymm, uypp, uzm, uzp, uzmm, uzpp;
  T vc, vxm, vxp, vxmm, vxpp, vym, vyp, vzm, vzp, vzmm, vzpp;
  T wc, wxm, wxp, wxmm, wxpp, wym, wyp, wymm, wypp, wzm, wzp;
  T pc, pxm, pym, pzm;
};

// code byte 1..216 -> neighbourhood cases (cx, cy, cz) in 1..6 (the
// split_number of src/solver.cc:94-109 applied to 100cx + 10cy + cz).
__device__ __forceinline__ void decode_cases(int code, int& cx, int& cy, int& cz) {
  int c = code - 1;
  int a = c / 36;
  int rem = c - a * 36;
  int b = rem / 6;
  cx = a + 1;
  cy = b + 1;
  cz = rem - b * 6 + 1;
}

// The left neighbour along an axis is solid exactly for cases 1, 2 and 4 of
// eval_geometry (src/geometry.cc:273-296).
__device__ __forceinline__ bool left_solid(int cs) { return cs == 1 || cs == 2 || cs == 4; }

// get_2nd_derivation, src/solver.cc:57-91, operand order preserved.
__device__ __forceinline__ double d2_exact(int cs, double ll, double l, double m, double r,
                                           double rr) {
  double d = 0.0;
  if (cs == 1) d = -8.0 * m;
  else if (cs == 2) d = 8.0 / 3.0 * r - 16.0 / 3.0 * m;
  else if (cs == 3) d = 8.0 / 3.0 * l - 16.0 / 3.0 * m;
  else if (cs == 4) d = 2.0 * r - 5.0 * m - 1.0 / 5.0 * rr;
  else if (cs == 5) d = 2.0 * l - 1.0 / 5.0 * ll - 5.0 * m;
  else if (cs == 6) d = l - 2.0 * m + r;
  return d;
}

// Whether x is +0 or -0, without the FP64 pipe.
__device__ __forceinline__ bool zero_bits(double x) {
  return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) == 0u;
}

// x / kRe, correctly rounded, in three FP64 instructions instead of the
// general division: kInvRe is the correctly rounded reciprocal, x * kInvRe is
// less than an ulp from the quotient (the reciprocal is off by 0.19 of half an
// ulp, the product by half an ulp), and one residual step then rounds
// correctly (Markstein 1990; Brisebarre, Muller and Raina, IEEE TC 53, 2004).
// The step needs the residual exact and the product finite; arguments for
// which that is not sure take the division.  Zero, whose sign the step would
// lose, is its own quotient.
__device__ __forceinline__ double div_re_step(double x) {
  constexpr double kInvRe = 1.0 / kRe;
  static_assert(kRe == 0.01, "the product's error bound above is for this divisor");
  const double q = x * kInvRe;
  const double r = __fma_rn(__fma_rn(-kRe, q, x), kInvRe, q);
  return zero_bits(x) ? x : r;
}
__device__ __forceinline__ bool div_re_holds(double x) {
  return zero_bits(x) || (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - 64u < 1900u;
}
__device__ __noinline__ static double div_re_general(double x) { return x / kRe; }
__device__ __forceinline__ double div_re(double x) {
  const double r = div_re_step(x);
  return div_re_holds(x) ? r : div_re_general(x);
}

// central_diff5 body (src/solver.cc:142-219) for one fluid voxel.
template <int SOLVER>
__device__ __forceinline__ void update_exact(const Stencil<double>& s, int code, double& un,
                                             double& vn, double& wn, double& pn) {
  int cx, cy, cz;
  decode_cases(code, cx, cy, cz);
  const bool lx = left_solid(cx), ly = left_solid(cy), lz = left_solid(cz);
  double dp_dz = lz ? 0. : -s.pzm + s.pc;
  double dp_dy = ly ? 0. : -s.pym + s.pc;
  double dp_dx = lx ? 0. : -s.pxm + s.pc;
  double uxx = (s.uxm - 2 * s.uc + s.uxp);
  double vyy = (s.vym - 2 * s.vc + s.vyp);
  double wzz = (s.wzm - 2 * s.wc + s.wzp);
  double vxx = d2_exact(cx, s.vxmm, s.vxm, s.vc, s.vxp, s.vxpp);
  double wxx = d2_exact(cx, s.wxmm, s.wxm, s.wc, s.wxp, s.wxpp);
  double uyy = d2_exact(cy, s.uymm, s.uym, s.uc, s.uyp, s.uypp);
  double wyy = d2_exact(cy, s.wymm, s.wym, s.wc, s.wyp, s.wypp);
  double uzz = d2_exact(cz, s.uzmm, s.uzm, s.uc, s.uzp, s.uzpp);
  double vzz = d2_exact(cz, s.vzmm, s.vzm, s.vc, s.vzp, s.vzpp);
  double fu = uxx + uyy + uzz;
  double fv = vyy + vzz + vxx;
  double fw = wzz + wxx + wyy;
  double v_sum = 0.0;
  if (SOLVER == 1) v_sum = (s.wzp - s.wc + s.vyp - s.vc + s.uxp - s.uc);
  if (SOLVER == 1 || SOLVER == 2) {
    un = lx ? 0.0 : s.uc + (-dp_dx + div_re(fu)) * kDt;
    vn = ly ? 0.0 : s.vc + (-dp_dy + div_re(fv)) * kDt;
    wn = lz ? 0.0 : s.wc + (-dp_dz + div_re(fw)) * kDt;
  } else {
    un = (1.0 - kOmega) * s.uc + kOmega * (-dp_dx + div_re(fu)) * kDt;
    vn = (1.0 - kOmega) * s.vc + kOmega * (-dp_dy + div_re(fv)) * kDt;
    wn = (1.0 - kOmega) * s.wc + kOmega * (-dp_dz + div_re(fw)) * kDt;
  }
  if (SOLVER == 2 || SOLVER == 3) v_sum = (s.wzp - wn + s.vyp - vn + s.uxp - un);
  pn = s.pc - kC2 * v_sum * kDt;
}

// Coefficient form.  Each wall-aware stencil of case cs is
//   a(cs) * centre + cA(cs) * A + cB(cs) * B
// with A, B the (at most two) off-centre points it uses.
template <typename T>
struct CaseCoef {
  T a, cA, cB;
};

// Coefficients per case: 1 (-8, 0, 0); 2, 3 (-16/3, 8/3, 0); 4, 5 (-5, 2, -0.2);
// 6 (-2, 1, 1).  In FP32 as selects on three comparisons (no branches; the
// FP32 correction sweep measured 20.5 us against 22.6 us with a switch on the
// 128^3 sphere pack); in FP64 as a switch (the FP64 Jacobi sweep measured
// 68 us against 76 us with selects, which cost register pairs).
template <typename T>
__device__ __forceinline__ CaseCoef<T> case_coef(int cs) {
  CaseCoef<T> k;
  if (sizeof(T) == 8) {
    switch (cs) {
      case 1: k.a = T(-8.0); k.cA = T(0.0); k.cB = T(0.0); break;
      case 2: case 3: k.a = T(-16.0 / 3.0); k.cA = T(8.0 / 3.0); k.cB = T(0.0); break;
      case 4: case 5: k.a = T(-5.0); k.cA = T(2.0); k.cB = T(-0.2); break;
      default: k.a = T(-2.0); k.cA = T(1.0); k.cB = T(1.0); break;
    }
    return k;
  }
  const bool c1 = cs == 1, le3 = cs <= 3, le5 = cs <= 5;
  k.a = c1 ? T(-8.0) : (le3 ? T(-16.0 / 3.0) : (le5 ? T(-5.0) : T(-2.0)));
  k.cA = c1 ? T(0.0) : (le3 ? T(8.0 / 3.0) : (le5 ? T(2.0) : T(1.0)));
  k.cB = le3 ? T(0.0) : (le5 ? T(-0.2) : T(1.0));
  return k;
}

// A = left for cases 3, 5, 6, else right; B = second right (4), second left
// (5), right (6); unused (coefficient 0) otherwise.
template <typename T>
__device__ __forceinline__ void case_pick(int cs, T ll, T l, T r, T rr, T& A, T& B) {
  A = (cs == 3 || cs == 5 || cs == 6) ? l : r;
  B = cs == 4 ? rr : (cs == 5 ? ll : r);
}

// One velocity component: the along-axis 3-point term plus two cross-axis
// wall stencils, the pressure difference, and the solver's relaxation.
// Group of a case by its centre coefficient a: 1 -> 0, 2/3 -> 1, 4/5 -> 2, 6 -> 3.
__device__ __forceinline__ int case_group(int cs) {
  return cs == 1 ? 0 : (cs <= 3 ? 1 : (cs <= 5 ? 2 : 3));
}

// Centre coefficient a of a case group (the FP64 form's centre table is built
// from it: see centre64).
__device__ __forceinline__ double group_a(int g) {
  return g == 0 ? -8.0 : (g == 1 ? -16.0 / 3.0 : (g == 2 ? -5.0 : -2.0));
}

// FP64 form: the relaxation of the solver is folded into the coefficients,
// so a new velocity is one FMA chain over its nine stencil values
//   v' = Cc c + K' (am + ap + cA1 A1 + cB1 B1 + cA2 A2 + cB2 B2) - dt' (pc - pm)
// with K' = dt/Re, dt' = dt (solvers 1, 2) or K' = omega dt/Re, dt' = omega dt
// (solver 3, whose update is (1 - omega) c + omega dt (-dp + f/Re)), and the
// centre coefficient Cc = 1 + K' ctr (solvers 1, 2) or (1 - omega) + K' ctr
// (solver 3), ctr = -2 + a1 + a2.  -dt' pc is shared by the three velocities.
// 31 FP64 instructions per fluid voxel instead of 36 (SOR) / 33: GB300's
// FP64 pipe (1/64 of the FP32 rate) bounds the FP64 sweeps.
template <int SOLVER>
struct Relax64 {
  static constexpr double K = SOLVER == 3 ? kDt / kRe * kOmega : kDt / kRe;
  static constexpr double Dt = SOLVER == 3 ? kDt * kOmega : kDt;
  static constexpr double Base = SOLVER == 3 ? 1.0 - kOmega : 1.0;
};

template <int SOLVER>
__device__ __forceinline__ double centre64(int g1, int g2) {
  const double ctr = (-2.0 + group_a(g1)) + group_a(g2);
  return __fma_rn(Relax64<SOLVER>::K, ctr, Relax64<SOLVER>::Base);
}

// Off-centre coefficients of a wall stencil of case cs times K' (see case_coef).
template <int SOLVER>
__device__ __forceinline__ void case_coef64(int cs, double& cA, double& cB) {
  constexpr double K = Relax64<SOLVER>::K;
  switch (cs) {
    case 1: cA = 0.0; cB = 0.0; break;
    case 2: case 3: cA = K * (8.0 / 3.0); cB = 0.0; break;
    case 4: case 5: cA = K * 2.0; cB = K * -0.2; break;
    default: cA = K; cB = K; break;
  }
}

template <int SOLVER>
__device__ __forceinline__ double2 case_coef64(int cs) {
  double2 k;
  case_coef64<SOLVER>(cs, k.x, k.y);
  return k;
}

// A block's shared tables: centre coefficients by the two case groups,
// off-centre ones by case, the cases (cx | cy << 4 | cz << 8) of a code byte.
struct Tables64 {
  double centre[16];
  double2 coef[8];
  unsigned short cases[256];
};

template <int SOLVER>
__device__ __forceinline__ void fill_centre64(double* centre) {
  for (int i = threadIdx.x; i < 16; i += blockDim.x) centre[i] = centre64<SOLVER>(i >> 2, i & 3);
}

template <int SOLVER>
__device__ __forceinline__ void fill_tables64(Tables64& t) {
  fill_centre64<SOLVER>(t.centre);
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    if (i < 8) t.coef[i] = case_coef64<SOLVER>(i);
    int cx, cy, cz;
    decode_cases(i >= 1 && i <= 216 ? i : 216, cx, cy, cz);
    t.cases[i] = (unsigned short)(cx | cy << 4 | cz << 8);
  }
}

// tab: the block's tables, or null (then computed per voxel).
template <int SOLVER>
__device__ __forceinline__ double vel64(double c, double am, double ap, int cs1, double A1,
                                        double B1, int cs2, double A2, double B2, double pm,
                                        double P, bool lsolid, const Tables64* tab) {
  const double2 k1 = tab ? tab->coef[cs1] : case_coef64<SOLVER>(cs1);
  const double2 k2 = tab ? tab->coef[cs2] : case_coef64<SOLVER>(cs2);
  constexpr double K = Relax64<SOLVER>::K;
  const double Cc = tab ? tab->centre[case_group(cs1) * 4 + case_group(cs2)]
                        : centre64<SOLVER>(case_group(cs1), case_group(cs2));
  // no pressure difference where the left neighbour is solid
  double t = lsolid ? 0.0 : fma(Relax64<SOLVER>::Dt, pm, P);
  t = fma(Cc, c, t);
  t = fma(K, am, t);
  t = fma(K, ap, t);
  t = fma(k1.x, A1, t);
  t = fma(k1.y, B1, t);
  t = fma(k2.x, A2, t);
  t = fma(k2.y, B2, t);
  return (SOLVER != 3 && lsolid) ? 0.0 : t;
}

template <typename T, int SOLVER>
__device__ __forceinline__ T vel_fast(T c, T am, T ap, int cs1, T ll1, T l1, T r1, T rr1, int cs2,
                                      T ll2, T l2, T r2, T rr2, T dp, bool zero) {
  const CaseCoef<T> k1 = case_coef<T>(cs1), k2 = case_coef<T>(cs2);
  T A1, B1, A2, B2;
  case_pick<T>(cs1, ll1, l1, r1, rr1, A1, B1);
  case_pick<T>(cs2, ll2, l2, r2, rr2, A2, B2);
  T f = am + ap;
  f = fma(k1.cA, A1, f);
  f = fma(k1.cB, B1, f);
  f = fma(k2.cA, A2, f);
  f = fma(k2.cB, B2, f);
  const T centre = T(-2.0) + k1.a + k2.a;  // centre coefficient (exact small sums)
  f = fma(centre, c, f);
  const T K = T(kDt / kRe);
  if (SOLVER == 3) {
    // (1 - w) c + w (-dp + f / Re) dt
    T t = fma(T(kDt / kRe * kOmega), f, T(1.0 - kOmega) * c);
    return fma(T(-kDt * kOmega), dp, t);
  }
  T t = fma(K, f, c);
  t = fma(T(-kDt), dp, t);
  return zero ? T(0.0) : t;
}

template <typename T, int SOLVER>
__device__ __forceinline__ void update_fast_cases(const Stencil<T>& s, int cx, int cy, int cz,
                                                  T& un, T& vn, T& wn, T& pn) {
  const bool lx = left_solid(cx), ly = left_solid(cy), lz = left_solid(cz);
  const T dpx = lx ? T(0) : s.pc - s.pxm;
  const T dpy = ly ? T(0) : s.pc - s.pym;
  const T dpz = lz ? T(0) : s.pc - s.pzm;
  T div0 = T(0);
  if (SOLVER == 1) div0 = ((s.wzp - s.wc) + (s.vyp - s.vc)) + (s.uxp - s.uc);
  // u: along x, cross y (cy) and z (cz)
  un = vel_fast<T, SOLVER>(s.uc, s.uxm, s.uxp, cy, s.uymm, s.uym, s.uyp, s.uypp, cz, s.uzmm,
                           s.uzm, s.uzp, s.uzpp, dpx, lx);
  // v: along y, cross x (cx) and z (cz)
  vn = vel_fast<T, SOLVER>(s.vc, s.vym, s.vyp, cx, s.vxmm, s.vxm, s.vxp, s.vxpp, cz, s.vzmm,
                           s.vzm, s.vzp, s.vzpp, dpy, ly);
  // w: along z, cross x (cx) and y (cy)
  wn = vel_fast<T, SOLVER>(s.wc, s.wzm, s.wzp, cx, s.wxmm, s.wxm, s.wxp, s.wxpp, cy, s.wymm,
                           s.wym, s.wyp, s.wypp, dpz, lz);
  T div = (SOLVER == 1) ? div0 : ((s.wzp - wn) + (s.vyp - vn)) + (s.uxp - un);
  pn = fma(T(-kC2 * kDt), div, s.pc);
}

template <typename T, int SOLVER>
__device__ __forceinline__ void update_fast(const Stencil<T>& s, int code, T& un, T& vn, T& wn,
                                            T& pn) {
  int cx, cy, cz;
  decode_cases(code, cx, cy, cz);
  update_fast_cases<T, SOLVER>(s, cx, cy, cz, un, vn, wn, pn);
}

// Gather of the stencil values of one interior voxel, through the read-only
// path, from L2, or with plain loads (values a kernel whose end this one waits
// for itself wrote).
constexpr int kLdCg = 0, kLdNc = 1, kLdPlain = 2;
template <typename T>
__device__ __forceinline__ T ldA(const T* p, int how) {
  return how == kLdNc ? __ldg(p) : how == kLdPlain ? *p : __ldcg(p);
}

// P3 selects how the centre pressure of a voxel on the last interior plane
// (z = NZ-3) is read.  The out-of-place orderings store the swept,
// pre-reapply pressure there (their -x/-y neighbours on that plane must see it,
// as in the reference's in-place order, boundary_conditions.cc:46-79 runs only
// after the sweep) and imply the reapplied value 3 for the voxel itself:
//   0: stored value (in-place reference order, explicit reapply)
//   1: 3 (FP64 state)         2: 0 (homogeneous correction of the mixed form)
template <typename T, int PHASE, int NC = kLdNc, int P3 = 1>
__device__ __forceinline__ void gather(Stencil<T>& s, const Fields<T>& A, const Fields<T>& B,
                                       long long c, int x, int y, int z, const Grid& g,
                                       long long px, long long pl) {
  const long long sx = 1, sy = px, sz = pl;
  // PHASE 2 (black): interior +-1 neighbours are red and already updated (in
  // B); every other read (centre, +-2, halos) is the previous iterate (A).
  // (one load from a selected base: the red values this pass reads from B are
  // not written by it)
  auto P = [&](const T* a, const T* b, long long o, bool interior) -> T {
    if (PHASE == 2) return ldA((interior ? b : a) + c + o, NC);
    return ldA(a + c + o, NC);
  };
  const bool ixm = x - 1 >= 2, ixp = x + 1 <= g.NX - 3;
  const bool iym = y - 1 >= 2, iyp = y + 1 <= g.NY - 3;
  const bool izm = z - 1 >= 2, izp = z + 1 <= g.NZ - 3;
  s.uc = ldA(A.u + c, NC);
  s.vc = ldA(A.v + c, NC);
  s.wc = ldA(A.w + c, NC);
  s.pc = (P3 != 0 && z == g.NZ - 3) ? T(P3 == 1 ? 3.0 : 0.0) : ldA(A.p + c, NC);
  s.uxm = P(A.u, B.u, -sx, ixm); s.uxp = P(A.u, B.u, sx, ixp);
  s.uym = P(A.u, B.u, -sy, iym); s.uyp = P(A.u, B.u, sy, iyp);
  s.uzm = P(A.u, B.u, -sz, izm); s.uzp = P(A.u, B.u, sz, izp);
  s.uymm = ldA(A.u + c - 2 * sy, NC); s.uypp = ldA(A.u + c + 2 * sy, NC);
  s.uzmm = ldA(A.u + c - 2 * sz, NC); s.uzpp = ldA(A.u + c + 2 * sz, NC);
  s.vxm = P(A.v, B.v, -sx, ixm); s.vxp = P(A.v, B.v, sx, ixp);
  s.vym = P(A.v, B.v, -sy, iym); s.vyp = P(A.v, B.v, sy, iyp);
  s.vzm = P(A.v, B.v, -sz, izm); s.vzp = P(A.v, B.v, sz, izp);
  s.vxmm = ldA(A.v + c - 2 * sx, NC); s.vxpp = ldA(A.v + c + 2 * sx, NC);
  s.vzmm = ldA(A.v + c - 2 * sz, NC); s.vzpp = ldA(A.v + c + 2 * sz, NC);
  s.wxm = P(A.w, B.w, -sx, ixm); s.wxp = P(A.w, B.w, sx, ixp);
  s.wym = P(A.w, B.w, -sy, iym); s.wyp = P(A.w, B.w, sy, iyp);
  s.wzm = P(A.w, B.w, -sz, izm); s.wzp = P(A.w, B.w, sz, izp);
  s.wxmm = ldA(A.w + c - 2 * sx, NC); s.wxpp = ldA(A.w + c + 2 * sx, NC);
  s.wymm = ldA(A.w + c - 2 * sy, NC); s.wypp = ldA(A.w + c + 2 * sy, NC);
  s.pxm = P(A.p, B.p, -sx, ixm);
  s.pym = P(A.p, B.p, -sy, iym);
  s.pzm = P(A.p, B.p, -sz, izm);
}

// The FP64 coefficient form of one voxel.  Only the values its cases use are
// loaded: per velocity the centre, the two neighbours along its axis and two
// (A, B) of each cross axis, whose offsets the cases give -- 25 loads instead
// of the stencil's 37, and no selects between loaded values.  Buffers and the
// centre pressure as in gather (PHASE, P3); F[1 - b] - F[b] is the same for
// the four fields.  o: the voxel's own values as read.
// Overlapped Jacobi sweeps of a 128^3 pack take 46.3 us with the whole stencil
// and 44.0 so, red-black half-sweeps of a 97x61x118 pack 12.3 and 10.9.
struct Own64 {
  double u, v, w, p;
};

// A load whose line may be the first to leave L2 (first), or a plain one.
__device__ __forceinline__ double ld_last(const double* p, bool first) {
  unsigned long long go, stay;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(go));
  asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(stay));
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;"
               : "=d"(v)
               : "l"(p), "l"(first ? go : stay));
  return v;
}

template <int SOLVER, int PHASE, int LD, int P3 = 1>
__device__ __forceinline__ void update64(const Fields<double>& A, const Fields<double>& B,
                                         long long c, int x, int y, int z, const Grid& g, int code,
                                         const Tables64* tab, Own64& o, double& un, double& vn,
                                         double& wn, double& pn) {
  int cx, cy, cz;
  if (tab) {
    const unsigned cs = tab->cases[code];
    cx = cs & 15;
    cy = (cs >> 4) & 15;
    cz = cs >> 8;
  } else {
    decode_cases(code, cx, cy, cz);
  }
  const long long sx = 1, sy = g.px64, sz = g.pl64;
  // PHASE 2: interior neighbours at distance 1 are read in B
  const long long d = PHASE == 2 ? B.u - A.u : 0;
  const long long xm = (PHASE == 2 && x - 1 >= 2 ? d : 0) - sx;
  const long long xp = (PHASE == 2 && x + 1 <= g.NX - 3 ? d : 0) + sx;
  const long long ym = (PHASE == 2 && y - 1 >= 2 ? d : 0) - sy;
  const long long yp = (PHASE == 2 && y + 1 <= g.NY - 3 ? d : 0) + sy;
  const long long zm = (PHASE == 2 && z - 1 >= 2 ? d : 0) - sz;
  const long long zp = (PHASE == 2 && z + 1 <= g.NZ - 3 ? d : 0) + sz;
  // A = left for cases 3, 5, 6, else right; B = second right (4), second left
  // (5), right otherwise (as case_pick)
  auto first = [](int cs, long long m, long long p) { return cs == 3 || cs >= 5 ? m : p; };
  auto second = [](int cs, long long s, long long p) {
    return cs == 4 ? 2 * s : (cs == 5 ? -2 * s : p);
  };
  const long long ax = first(cx, xm, xp), bx = second(cx, sx, xp);
  const long long ay = first(cy, ym, yp), by = second(cy, sy, yp);
  const long long az = first(cz, zm, zp), bz = second(cz, sz, zp);
  const double *U = A.u + c, *V = A.v + c, *W = A.w + c, *Q = A.p + c;
  // the black pass's own values: the last use of the old state's lines (but for
  // second neighbours), which make room for the new state, all of it read by
  // the next sweep.  Where L2 holds one state and not both (128^3 pack): 57.7 ->
  // 55.7 us; where it holds both (97x61x118, 112^3) as before; where it does not
  // hold one, without the hint (160^3 98 against 96 us, 224^3 217 against 203).
  // The same hint on a Jacobi sweep's reads of the plane below: 44.1 -> 45.1.
  const bool one_fits = g.pl64 * g.NZ <= (long long)kL2Bytes / 32;
  auto own = [&](const double* q) { return PHASE == 2 ? ld_last(q, one_fits) : ldA(q, LD); };
  o.u = own(U);
  o.v = own(V);
  o.w = own(W);
  o.p = (P3 != 0 && z == g.NZ - 3) ? (P3 == 1 ? 3.0 : 0.0) : own(Q);
  const double uxp = ldA(U + xp, LD), vyp = ldA(V + yp, LD), wzp = ldA(W + zp, LD);
  const bool lx = left_solid(cx), ly = left_solid(cy), lz = left_solid(cz);
  const double P = -Relax64<SOLVER>::Dt * o.p;
  un = vel64<SOLVER>(o.u, ldA(U + xm, LD), uxp, cy, ldA(U + ay, LD), ldA(U + by, LD), cz,
                     ldA(U + az, LD), ldA(U + bz, LD), ldA(Q + xm, LD), P, lx, tab);
  vn = vel64<SOLVER>(o.v, ldA(V + ym, LD), vyp, cx, ldA(V + ax, LD), ldA(V + bx, LD), cz,
                     ldA(V + az, LD), ldA(V + bz, LD), ldA(Q + ym, LD), P, ly, tab);
  wn = vel64<SOLVER>(o.w, ldA(W + zm, LD), wzp, cx, ldA(W + ax, LD), ldA(W + bx, LD), cy,
                     ldA(W + ay, LD), ldA(W + by, LD), ldA(Q + zm, LD), P, lz, tab);
  const double dv = SOLVER == 1 ? ((wzp - o.w) + (vyp - o.v)) + (uxp - o.u)
                                : ((wzp - wn) + (vyp - vn)) + (uxp - un);
  pn = fma(-kC2 * kDt, dv, o.p);
}

// The same update from the whole stencil (update64 loads only what the cases
// use, so its addresses wait for the code byte; here the 37 loads do not).
// centre: the block's table of centre coefficients; the others from selects on
// the cases.
template <int SOLVER>
__device__ __forceinline__ double vel64_whole(double c, double am, double ap, int cs1, double ll1,
                                              double l1, double r1, double rr1, int cs2,
                                              double ll2, double l2, double r2, double rr2,
                                              double pm, double P, bool lsolid,
                                              const double* centre) {
  double cA1, cB1, cA2, cB2, A1, B1, A2, B2;
  case_coef64<SOLVER>(cs1, cA1, cB1);
  case_coef64<SOLVER>(cs2, cA2, cB2);
  case_pick<double>(cs1, ll1, l1, r1, rr1, A1, B1);
  case_pick<double>(cs2, ll2, l2, r2, rr2, A2, B2);
  constexpr double K = Relax64<SOLVER>::K;
  const double Cc = centre[case_group(cs1) * 4 + case_group(cs2)];
  double t = lsolid ? 0.0 : fma(Relax64<SOLVER>::Dt, pm, P);
  t = fma(Cc, c, t);
  t = fma(K, am, t);
  t = fma(K, ap, t);
  t = fma(cA1, A1, t);
  t = fma(cB1, B1, t);
  t = fma(cA2, A2, t);
  t = fma(cB2, B2, t);
  return (SOLVER != 3 && lsolid) ? 0.0 : t;
}

template <int SOLVER, int PHASE>
__device__ __forceinline__ void update64_whole(const Fields<double>& A, const Fields<double>& B,
                                               long long c, int x, int y, int z, const Grid& g,
                                               int code, const double* centre, Own64& o,
                                               double& un, double& vn, double& wn, double& pn) {
  Stencil<double> s;
  gather<double, PHASE>(s, A, B, c, x, y, z, g, g.px64, g.pl64);
  o = {s.uc, s.vc, s.wc, s.pc};
  int cx, cy, cz;
  decode_cases(code, cx, cy, cz);
  const bool lx = left_solid(cx), ly = left_solid(cy), lz = left_solid(cz);
  const double P = -Relax64<SOLVER>::Dt * s.pc;
  double d0 = 0.0;
  if (SOLVER == 1) d0 = ((s.wzp - s.wc) + (s.vyp - s.vc)) + (s.uxp - s.uc);
  un = vel64_whole<SOLVER>(s.uc, s.uxm, s.uxp, cy, s.uymm, s.uym, s.uyp, s.uypp, cz, s.uzmm,
                           s.uzm, s.uzp, s.uzpp, s.pxm, P, lx, centre);
  vn = vel64_whole<SOLVER>(s.vc, s.vym, s.vyp, cx, s.vxmm, s.vxm, s.vxp, s.vxpp, cz, s.vzmm,
                           s.vzm, s.vzp, s.vzpp, s.pym, P, ly, centre);
  wn = vel64_whole<SOLVER>(s.wc, s.wzm, s.wzp, cx, s.wxmm, s.wxm, s.wxp, s.wxpp, cy, s.wymm,
                           s.wym, s.wyp, s.wypp, s.pzm, P, lz, centre);
  const double dv = SOLVER == 1 ? d0 : ((s.wzp - wn) + (s.vyp - vn)) + (s.uxp - un);
  pn = fma(-kC2 * kDt, dv, s.pc);
}

// Write the new values of interior voxel (x, y, z) and, on periodic axes,
// its halo copies (the halo exchange fused into the sweep).  The pressure
// reapply is fused too: the z-halo copies on planes 1 and NZ-2 hold nz+2 and 2
// (their geometry is this fluid voxel); x/y halo copies and the last interior
// plane keep the swept, pre-reapply value, as the reference's
// exchange-then-reapply order leaves the halos (the 3 of the last plane is
// implied, see gather).  HOMOG (correction sweeps of the mixed form) writes 0
// where the reapply writes a constant.
template <typename T, bool HOMOG>
__device__ __forceinline__ void write_voxel(const Fields<T>& B, long long c, int x, int y, int z,
                                            const Grid& g, long long px, long long pl, T un,
                                            T vn, T wn, T pn) {
  const T pin = HOMOG ? T(0) : T(g.nz + 2), pout = HOMOG ? T(0) : T(2.0);
  B.u[c] = un;
  B.v[c] = vn;
  B.w[c] = wn;
  B.p[c] = pn;  // last interior plane: swept value stored, reapplied 3 implied
  auto put = [&](long long o, T pv) {
    B.u[c + o] = un; B.v[c + o] = vn; B.w[c + o] = wn; B.p[c + o] = pv;
  };
  if (g.per[0]) {
    if (x < 4) put((long long)g.nx, pn);
    if (x >= g.nx) put(-(long long)g.nx, pn);
  }
  if (g.per[1]) {
    if (y < 4) put((long long)g.ny * px, pn);
    if (y >= g.ny) put(-(long long)g.ny * px, pn);
  }
  if (g.per[2]) {
    if (z < 4) put((long long)g.nz * pl, z == 2 ? pout : pn);
    if (z >= g.nz) put(-(long long)g.nz * pl, z == g.nz + 1 ? pin : pn);
  }
}


// ------------------------------------------------------------------ per-voxel bodies
// Shared by the single-problem kernels and the batched (many-sample) kernels,
// so a sample computes exactly the same values alone and in a batch.

// Interior linear index (x fastest) -> padded coordinates.
__device__ __forceinline__ unsigned div_magic(unsigned n, unsigned long long m, int s) {
  return (unsigned)(((unsigned long long)n * m) >> (32 + s));
}

__device__ __forceinline__ void lin_to_xyz(int lin, const Grid& g, int& x, int& y, int& z) {
  const unsigned r = div_magic((unsigned)lin, g.mnx, g.snx);  // lin / nx
  const unsigned zz = div_magic(r, g.mny, g.sny);             // r / ny
  x = lin - (int)r * g.nx + 2;
  y = (int)r - (int)zz * g.ny + 2;
  z = (int)zz + 2;
}

// One voxel of an FP64 sweep (Jacobi phase 0, red 1, black 2) from A into B.
// whole: the table of centre coefficients, for update64_whole.
template <int SOLVER, int PHASE, bool EXACT, int LD = kLdNc>
__device__ __forceinline__ void sweep64_voxel(const Fields<double>& A, const Fields<double>& B,
                                              const uint8_t* codes, const Grid& g, int lin,
                                              const Tables64* tab = nullptr,
                                              const double* whole = nullptr) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  if (PHASE && (((x + y + z) & 1) != PHASE - 1)) return;  // (x+y+z) - 6 has the same parity
  const long long px = g.px64, pl = g.pl64;
  int code = codes[((long long)z * g.NY + y) * g.pxc + x];
  long long c = (long long)z * pl + (long long)y * px + x;
  double un, vn, wn, pn;
  if (EXACT) {
    Stencil<double> s;
    gather<double, PHASE, LD>(s, A, B, c, x, y, z, g, px, pl);
    update_exact<SOLVER>(s, code, un, vn, wn, pn);
  } else if (whole) {
    Own64 o;
    update64_whole<SOLVER, PHASE>(A, B, c, x, y, z, g, code, whole, o, un, vn, wn, pn);
  } else {
    Own64 o;
    update64<SOLVER, PHASE, LD>(A, B, c, x, y, z, g, code, tab, o, un, vn, wn, pn);
  }
  write_voxel<double, false>(B, c, x, y, z, g, px, pl, un, vn, wn, pn);
}

// ---- interleaved FP32 correction fields (float4 u, v, w, p per voxel)

// The stencil of one voxel from the correction: the union of its offsets is
// 13 points, each one 128-bit load.  The voxel's own pressure on the last
// interior plane is the reapplied (fixed) value, whose correction is 0.
__device__ __forceinline__ void gather4(Stencil<float>& s, const float4* E, long long c, int z,
                                        const Grid& g) {
  const long long px = g.px4, pl = g.pl4;
  const float4 C = __ldg(E + c);
  const float4 XM = __ldg(E + c - 1), XP = __ldg(E + c + 1);
  const float4 XMM = __ldg(E + c - 2), XPP = __ldg(E + c + 2);
  const float4 YM = __ldg(E + c - px), YP = __ldg(E + c + px);
  const float4 YMM = __ldg(E + c - 2 * px), YPP = __ldg(E + c + 2 * px);
  const float4 ZM = __ldg(E + c - pl), ZP = __ldg(E + c + pl);
  const float4 ZMM = __ldg(E + c - 2 * pl), ZPP = __ldg(E + c + 2 * pl);
  s.uc = C.x; s.uxm = XM.x; s.uxp = XP.x; s.uym = YM.x; s.uyp = YP.x;
  s.uymm = YMM.x; s.uypp = YPP.x; s.uzm = ZM.x; s.uzp = ZP.x; s.uzmm = ZMM.x; s.uzpp = ZPP.x;
  s.vc = C.y; s.vxm = XM.y; s.vxp = XP.y; s.vxmm = XMM.y; s.vxpp = XPP.y; s.vym = YM.y;
  s.vyp = YP.y; s.vzm = ZM.y; s.vzp = ZP.y; s.vzmm = ZMM.y; s.vzpp = ZPP.y;
  s.wc = C.z; s.wxm = XM.z; s.wxp = XP.z; s.wxmm = XMM.z; s.wxpp = XPP.z; s.wym = YM.z;
  s.wyp = YP.z; s.wymm = YMM.z; s.wypp = YPP.z; s.wzm = ZM.z; s.wzp = ZP.z;
  s.pc = (z == g.NZ - 3) ? 0.f : C.w;
  s.pxm = XM.w; s.pym = YM.w; s.pzm = ZM.w;
}

// write_voxel for the interleaved correction (homogeneous boundary values).
__device__ __forceinline__ void write_voxel4(float4* B, long long c, int x, int y, int z,
                                             const Grid& g, float un, float vn, float wn,
                                             float pn) {
  const long long px = g.px4, pl = g.pl4;
  const float4 val = make_float4(un, vn, wn, pn);
  B[c] = val;
  if (g.per[0]) {
    if (x < 4) B[c + g.nx] = val;
    if (x >= g.nx) B[c - g.nx] = val;
  }
  if (g.per[1]) {
    if (y < 4) B[c + (long long)g.ny * px] = val;
    if (y >= g.ny) B[c - (long long)g.ny * px] = val;
  }
  if (g.per[2]) {
    // the z copies landing on planes NZ-2 and 1 hold reapplied pressure: 0
    if (z < 4) B[c + (long long)g.nz * pl] = make_float4(un, vn, wn, z == 2 ? 0.f : pn);
    if (z >= g.nz)
      B[c - (long long)g.nz * pl] = make_float4(un, vn, wn, z == g.nz + 1 ? 0.f : pn);
  }
}

// r = F(x) - x (FP64, stored FP32) and the first correction e1 = r.  On the
// last interior plane the state stores the swept pressure (the reapplied 3 is
// implied), so its residual is taken against that stored value.
template <int SOLVER>
__device__ __forceinline__ void dc_residual_voxel(const Fields<double>& X, float4* R, float4* E,
                                                  const uint8_t* codes, const Grid& g, int lin,
                                                  const double* centre) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  int code = codes[((long long)z * g.NY + y) * g.pxc + x];
  long long c = (long long)z * g.pl64 + (long long)y * g.px64 + x;
  Own64 o;
  double un, vn, wn, pn;
  update64_whole<SOLVER, 0>(X, X, c, x, y, z, g, code, centre, o, un, vn, wn, pn);
  const double pstored = (z == g.NZ - 3) ? __ldg(X.p + c) : o.p;
  float ru = (float)(un - o.u), rv = (float)(vn - o.v), rw = (float)(wn - o.w),
        rp = (float)(pn - pstored);
  long long c4 = (long long)z * g.pl4 + (long long)y * g.px4 + x;
  R[c4] = make_float4(ru, rv, rw, rp);
  write_voxel4(E, c4, x, y, z, g, ru, rv, rw, rp);
}

// e2 = L(e) + r (FP32 correction sweep).
template <int SOLVER>
__device__ __forceinline__ void dc_inner_voxel(const float4* E, float4* E2, const float4* R,
                                               const uint8_t* codes, const Grid& g, int lin) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  int code = codes[((long long)z * g.NY + y) * g.pxc + x];
  long long c = (long long)z * g.pl4 + (long long)y * g.px4 + x;
  Stencil<float> s;
  gather4(s, E, c, z, g);
  float un, vn, wn, pn;
  update_fast<float, SOLVER>(s, code, un, vn, wn, pn);
  const float4 r = __ldg(R + c);
  write_voxel4(E2, c, x, y, z, g, un + r.x, vn + r.y, wn + r.z, pn + r.w);
}

// x += e at a fluid voxel and at every halo copy a sweep writes for it (the
// only places where e can be non-zero).
__device__ __forceinline__ void dc_correct_voxel(const Fields<double>& X, const float4* E,
                                                 const Grid& g, int lin) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  auto add = [&](int xx, int yy, int zz) {
    long long c64 = (long long)zz * g.pl64 + (long long)yy * g.px64 + xx;
    const float4 e = E[(long long)zz * g.pl4 + (long long)yy * g.px4 + xx];
    X.u[c64] += (double)e.x;
    X.v[c64] += (double)e.y;
    X.w[c64] += (double)e.z;
    X.p[c64] += (double)e.w;
  };
  add(x, y, z);
  if (g.per[0]) {
    if (x < 4) add(x + g.nx, y, z);
    if (x >= g.nx) add(x - g.nx, y, z);
  }
  if (g.per[1]) {
    if (y < 4) add(x, y + g.ny, z);
    if (y >= g.ny) add(x, y - g.ny, z);
  }
  if (g.per[2]) {
    if (z < 4) add(x, y, z + g.nz);
    if (z >= g.nz) add(x, y, z - g.nz);
  }
}

}  // namespace pm

// Model-5 (six-equation multi-material flow with hyperelastic solids, ghost-fluid
// coupling, pressure relaxation) FP64 stage kernels.
//
// Compiled with --fmad=false and written in the operation order of the reference's C
// code (m5_*.c, state_equation.c, F_pe-free relaxation modes 1 and 3), so that the only
// rounding differences from the reference come from pow(): CUDA's and glibc's pow differ
// in the last bit for some arguments.
//
// The kernels are bound by the FP64 pipe: comparisons, clamps, halvings and sign tests work on
// the bit patterns, quotients by one divisor share its reciprocal (ffv_fp64.cuh), and terms that
// are exactly zero -- the deformation of a fluid cell (A = 0), the components of a face's unit
// normal -- are left out.  None of this changes a bit of the result.  The consistent flux form,
// which has no reference to equal bit for bit, also takes its own Newton iteration
// (relaxationvec).
//
// One stage:
//   m5_recon_slopes (cell, axis)  MUSCL states of the two faces (m5_faceinterp_V1 /
//                                  m5_reconctruct_V1)
//   m5_relax_faces  (cell, face)  their pressure relaxation, in place (m5_relaxationvec)
//   m5_face_flux    (cell, face)  HLLC or ghost-fluid HLLC per face or subface; a 1:1 face
//                                  is evaluated once, by the cell first in leaf order, and
//                                  the other takes its negative (the reference's flux
//                                  reuse, m5_residual.c:59-173)
//   m5_cell_update  (cell)        residual sum + non-conservative terms (m5_residual.c:175-215),
//                                  RK stage (m5_RK.c), positivity and ZEROU masks
//   m5_gfm_seq                    cells whose solid fraction crosses AVF_LIM in stage 1, in
//                                  leaf order (m5_gfm.c reads earlier neighbours' new state)
//   m5_relax_cell   (cell)        cell pressure relaxation (m5_relaxation_solid.c)
//   m5_gfm_seq (relax)            relaxation-crossing cells in leaf order (m5_gfm_rel.c)
#include <math.h>

#include "ffv_device.cuh"
#include "ffv_fp64.cuh"
#include "ffv_m5.cuh"
#include "ffv_m5_frame.cuh"
#include "ffv_plastic.cuh"

namespace {

// ------------------------------------------------------------------ EOS (state_equation.c)
// every entry of a deformation tensor is a zero: a fluid cell
__device__ __forceinline__ bool no_deformation(const double A[9]) {
  uint64_t any = 0;
#pragma unroll
  for (int q = 0; q < 9; q++) any |= f64::abs_bits(A[q]);
  return any == 0;
}

// G = A A^T (symmetric to the bit: the reference's two expressions of an off-diagonal entry have
// the same products in the same order) and the powers of its determinant that the elastic energy
// and stress of every solid take; solid: the determinant is not zero
struct Elastic {
  double G[6];  // G00, G11, G22, G01, G02, G12
  double p13, p16;
  bool solid;
};

// (1 + t)^a for |t| <= 1/32, a a unit fraction: 1 + t P(t), P the binomial series to t^9 (the first
// omitted term is below 3e-18), rounded once
template <int INV>
__device__ __forceinline__ double root_near_one(double t) {
  constexpr double a = 1.0 / INV;
  constexpr double c1 = a, c2 = c1 * (a - 1) / 2, c3 = c2 * (a - 2) / 3, c4 = c3 * (a - 3) / 4,
                   c5 = c4 * (a - 4) / 5, c6 = c5 * (a - 5) / 6, c7 = c6 * (a - 6) / 7,
                   c8 = c7 * (a - 7) / 8, c9 = c8 * (a - 8) / 9, c10 = c9 * (a - 9) / 10;
  double r = fma(c10, t, c9);
  r = fma(r, t, c8);
  r = fma(r, t, c7);
  r = fma(r, t, c6);
  r = fma(r, t, c5);
  r = fma(r, t, c4);
  r = fma(r, t, c3);
  r = fma(r, t, c2);
  r = fma(r, t, c1);
  return fma(r, t, 1.0);
}

__device__ __forceinline__ void elastic_of(const M5Consts &k, const double A[9], Elastic &e) {
  e.solid = false;
  if (k.nsolids == 0 || no_deformation(A)) return;
  const double G0 = A[0] * A[0] + A[1] * A[1] + A[2] * A[2];
  const double G1 = A[0] * A[3] + A[1] * A[4] + A[2] * A[5];
  const double G2 = A[0] * A[6] + A[1] * A[7] + A[2] * A[8];
  const double G4 = A[3] * A[3] + A[4] * A[4] + A[5] * A[5];
  const double G5 = A[3] * A[6] + A[4] * A[7] + A[5] * A[8];
  const double G8 = A[6] * A[6] + A[7] * A[7] + A[8] * A[8];
  const double Gmag = G0 * (G4 * G8 - G5 * G5) - G1 * (G1 * G8 - G5 * G2) + G2 * (G1 * G5 - G4 * G2);
  e.G[0] = G0;
  e.G[1] = G4;
  e.G[2] = G8;
  e.G[3] = G1;
  e.G[4] = G2;
  e.G[5] = G5;
  if (f64::abs_bits(Gmag) == 0) return;
  e.solid = true;
  // a solid's determinant is within its volume strain of 1: the consistent flux form, which has no
  // reference to equal bit for bit, takes the series instead of two powers of ~90 instructions
  // each (wall mesh of 0.41 M cells, 45 % of them solid)
  const double t = Gmag - 1.0;
  if (k.flux_form == FFV_FLUX_CONSISTENT && f64::abs_bits(t) <= 0x3fa0000000000000ull) {
    e.p13 = root_near_one<3>(t);
    e.p16 = root_near_one<6>(t);
  } else {
    e.p13 = pow(fabs(Gmag), 1.0 / 3.0);
    e.p16 = pow(fabs(Gmag), 1.0 / 6.0);
  }
}

// state_equation.c:269-317 and :217-267
__device__ __forceinline__ double elastic_energy(const Elastic &e, double mu) {
  if (!e.solid || mu == 0.0) return 0.0;
  const double g13 = f64::is_nan(e.p13) ? 0.0 : e.p13;
  const double d0 = e.G[0] - g13, d1 = e.G[1] - g13, d2 = e.G[2] - g13;
  const double a = e.G[3], b = e.G[4], c = e.G[5];
  const double tr1 = (d0 * d0 + a * a + b * b) + (a * a + d1 * d1 + c * c) + (b * b + c * c + d2 * d2);
  return mu / (4.0 * e.p16) * tr1;
}

// state_equation.c:143-204, accumulated into st (and stored in ast when given)
__device__ __forceinline__ void eos_stress_acc(double st[3][3], double avf, double pr,
                                               const Elastic &e, double mu, double (*ast)[3]) {
  const double press = -avf * pr;
  if (e.solid && mu != 0.0) {
    const double G0 = e.G[0], G4 = e.G[1], G8 = e.G[2], G1 = e.G[3], G2 = e.G[4], G5 = e.G[5];
    const double q0 = G0 * G0 + G1 * G1 + G2 * G2, q4 = G1 * G1 + G4 * G4 + G5 * G5,
                 q8 = G2 * G2 + G5 * G5 + G8 * G8, q1 = G0 * G1 + G1 * G4 + G2 * G5,
                 q2 = G0 * G2 + G1 * G5 + G2 * G8, q5 = G1 * G2 + G4 * G5 + G5 * G8;
    const f64::Rcp three{3.0, 1.0 / 3.0};
    const double J1 = f64::div(G0 + G4 + G8, three), J2 = f64::div(q0 + q4 + q8, three);
    const double f = mu / e.p16;
    const double s0 = press - f * (q0 - J2 - e.p13 * (G0 - J1)),
                 s4 = press - f * (q4 - J2 - e.p13 * (G4 - J1)),
                 s8 = press - f * (q8 - J2 - e.p13 * (G8 - J1));
    const double s1 = -f * (q1 - e.p13 * G1), s2 = -f * (q2 - e.p13 * G2), s5 = -f * (q5 - e.p13 * G5);
    const double s[3][3] = {{s0, s1, s2}, {s1, s4, s5}, {s2, s5, s8}};
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        if (j >= i) st[i][j] += s[i][j];
        else st[i][j] = st[j][i];
        if (ast) ast[i][j] = s[i][j];
      }
  } else {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      st[i][i] += press;
      if (ast)
        for (int j = 0; j < 3; j++) ast[i][j] = i == j ? press : 0.0;
    }
  }
}

// a volume fraction between amin / 100 and 1 - amin / 100
__device__ __forceinline__ double clamp_vf(const M5Consts &k, double a) {
  return f64::le(a, k.lo) ? k.lo : (f64::ge(a, k.hi) ? k.hi : a);
}

// phi[0] (m5_facevalues.c:83-99): the solid fraction(s) against AVF_LIM; ac the cell's fractions
template <int N>
__device__ __forceinline__ double phi0_of(const M5Consts &k, double a0, double a1) {
  const double c0 = clamp_vf(k, a0);
  if (N > 2 && k.nsolids == 2 && k.mu[0] != 0.0) {
    const double c1 = clamp_vf(k, a1);
    return (f64::gt(c0, c1) ? c0 : c1) - k.avf_lim;
  }
  return c0 - k.avf_lim;
}

template <int N>
struct Sol {
  double r, u, v, w, e, ut, vt, wt, phi0, c2;
  double ra[N], avf[N], are[N], p[N];
  double A[9], st[3][3];
  double vec[K5<N>::NC];  // conservative part of the state vector (HLLC corrections)
  bool flat;              // A = 0
};

// m5_facevalues.c:3-192 (from_face false: U is a cell state) and m5_facercnstr.c:3-191
// (from_face true: U is a face state); phi0 from the cell-centre state's volume fractions.
// ast (optional) receives each material's stress.
template <int N>
__device__ void make_sol(const M5Consts &k, const double *U, double phi0, bool from_face,
                         Sol<N> &s, double (*ast)[3][3] = nullptr) {
  using C = K5<N>;
  s.r = U[0];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (i) s.r += U[i];
    s.ra[i] = U[i];
    s.vec[i] = U[i];
  }
  const f64::Rcp r = f64::rcp(s.r);
  s.u = f64::div(U[C::i1 + 0], r);
  s.v = f64::div(U[C::i1 + 1], r);
  s.w = f64::div(U[C::i1 + 2], r);
  s.vec[C::i1 + 0] = U[C::i1 + 0];
  s.vec[C::i1 + 1] = U[C::i1 + 1];
  s.vec[C::i1 + 2] = U[C::i1 + 2];
  s.e = f64::div(U[C::i2], r);
  s.vec[C::i2] = U[C::i2];
  double at[N], sum = 0.0;
#pragma unroll
  for (int i = 0; i < N - 1; ++i) {
    at[i] = clamp_vf(k, U[C::i3 + i]);
    sum = i ? sum + at[i] : at[i];
  }
  double last = 1.0 - sum;  // the last fraction; avf[N - 1] sums the scaled ones once more
  at[N - 1] = last;
  if (f64::gt(sum, k.hi)) {
    const double dif = sum - k.hi;
    const f64::Rcp rs = f64::rcp(sum);
    sum = 0.0;
#pragma unroll
    for (int j = 0; j < N - 1; ++j) {
      at[j] = at[j] - f64::div(at[j], rs) * dif;
      sum = j ? sum + at[j] : at[j];
    }
    at[N - 1] = 1.0 - k.hi;
    last = 1.0 - sum;
  }
#pragma unroll
  for (int i = 0; i < N - 1; ++i) s.avf[i] = at[i];
  s.avf[N - 1] = last;
  s.phi0 = phi0;
#pragma unroll
  for (int i = 0; i < N; ++i) s.are[i] = U[C::i4 + i];
#pragma unroll
  for (int q = 0; q < 9; q++) s.A[q] = U[C::i5 + q];
  s.flat = no_deformation(s.A);
  Elastic el;
  elastic_of(k, s.A, el);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) s.st[i][j] = 0.0;
  double c2 = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double ael = elastic_energy(el, k.mu[i]);
    const double a = from_face ? s.avf[i] : at[i];
    const double press = (k.gm1[i] * (s.are[i] - ael) / a) - k.gpi[i];
    c2 += f64::div(a, r) * k.gamma[i] * (press + k.pinf[i]);
    s.p[i] = press;
    eos_stress_acc(s.st, s.avf[i], press, el, k.mu[i], ast ? ast[i] : nullptr);
  }
  s.c2 = c2;
}

// the same with phi0 from the cell state Sc
template <int N>
__device__ __forceinline__ double phi0_state(const M5Consts &k, const double *Sc) {
  return phi0_of<N>(k, Sc[K5<N>::i3], N > 2 ? Sc[K5<N>::i3 + 1] : 0.0);
}

// m5_bc.c (m5_bc_symmetry) / bc_reflective.c / bc_wall.c: ghost velocity
template <int F, int N>
__device__ __forceinline__ void ghost(const Sol<N> &L, int bc, Sol<N> &R) {
  R = L;
  if (bc == 1 || bc == 4 || bc == 5) {
    const double v3[3] = {L.u, L.v, L.w};
    const double ul = loc<F, 0>(v3), vl = loc<F, 1>(v3), wl = loc<F, 2>(v3);
    const double ur = -ul, vr = bc == 5 ? -vl : vl, wr = bc == 5 ? -wl : wl;
    R.u = glob<F, 0>(ur, vr, wr);
    R.v = glob<F, 1>(ur, vr, wr);
    R.w = glob<F, 2>(ur, vr, wr);
  }
}

template <int N>
struct NC {
  double unc[3], avf[N], are[N], A[9];
};

// m5_star_region.c:3-158
template <int F, int N>
__device__ unsigned star_region(const M5Consts &k, const Sol<N> &s, double rL, double rR,
                                bool both_solid, bool leftside, double u_S, double SL, double SR,
                                double uL, double vL, double wL, double uR, double vR, double wR,
                                const double sL[3], const double sR[3], double *Us, NC<N> &nc) {
  using C = K5<N>;
  const double SK = leftside ? SL : SR, uK = leftside ? uL : uR, vK = leftside ? vL : vR,
               wK = leftside ? wL : wR, s11K = leftside ? sL[0] : sR[0],
               s12K = leftside ? sL[1] : sR[1], s13K = leftside ? sL[2] : sR[2];
  // SK - u* and u* - SK are each other's negation to the bit, and so are quotients by them
  const f64::Rcp dS = f64::rcp(SK - u_S);
  const double dK = SK - uK;
  double ar_S[N], r_S = 0.0;
#pragma unroll
  for (int v = 0; v < N; ++v) {
    ar_S[v] = f64::div(s.ra[v] * dK, dS);
    r_S = v ? r_S + ar_S[v] : ar_S[v];
  }
  const double mR = (uR - SR) * rR, mL = (uL - SL) * rL, mLR = mL * (uR - SR) * rR;
  const f64::Rcp den = f64::rcp(mR - mL);
  const double s11_S = f64::div(mR * (sL[0]) - mL * (sR[0]) + mLR * (uR - uL), den);
  double s12_S = 0.0, s13_S = 0.0;
  if (both_solid) {
    s12_S = f64::div(mR * (sL[1]) - mL * (sR[1]) + mLR * (vR - vL), den);
    s13_S = f64::div(mR * (sL[2]) - mL * (sR[2]) + mLR * (wR - wL), den);
  }
  const double j12 = s12_S - s12K, j13 = s13_S - s13K;
  double v_S = vK + 0.0, w_S = wK + 0.0;
  if (f64::abs_bits(j12) | f64::abs_bits(j13)) {
    const f64::Rcp dv = f64::rcp((uK - SK) * s.r);
    v_S = vK + f64::div(j12, dv);
    w_S = wK + f64::div(j13, dv);
  }
  const double vel[3] = {glob<F, 0>(u_S, v_S, w_S), glob<F, 1>(u_S, v_S, w_S),
                         glob<F, 2>(u_S, v_S, w_S)};
  const double re = s.r * s.e;
  // the reference's expression, or the Rankine-Hugoniot energy jump across the S_K wave
  // (FFV_FLUX_CONSISTENT, include/ffv.h)
  const double sg11 = k.flux_form == FFV_FLUX_CONSISTENT ? f64::neg(s11K) : s11K;
  const double Em_S = (re * (uK - SK) + sg11 * uK - s12K * vK - s13K * wK + s11_S * u_S + s12_S * v_S +
                       s13_S * w_S) /
                      (r_S * (k.flux_form == FFV_FLUX_CONSISTENT ? u_S - SK : u_S + SK));
  Elastic el;
  el.solid = false;
  double Ag[3][3];
  if (!s.flat) {
    double Am[3][3], Al[3][3], AS[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) Am[i][j] = s.A[3 * i + j];
    tens_to_local<F>(Am, Al);
    const double ju = uK - SK, jv = vK - v_S, jw = wK - w_S;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      AS[0][j] = f64::neg(f64::div(Al[0][j] * ju - Al[1][j] * jv + Al[2][j] * jw, dS));
      AS[1][j] = Al[1][j];
      AS[2][j] = Al[2][j];
    }
    tens_to_global<F>(AS, Ag);
    elastic_of(k, &Ag[0][0], el);
  } else {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) Ag[i][j] = 0.0;
  }
#pragma unroll
  for (int v = 0; v < N; ++v) {
    const double rm = (s.ra[v] / s.avf[v]);
    const double rm_S = f64::neg(f64::div(rm * (uK - SK), dS));
    const double p_k = -s.p[v];
    const double ga = k.gamma[v], pi = k.pinf[v], gp1 = ga + 1.0, gm1 = k.gm1[v];
    const double p_S = (p_k + pi) * ((gm1 * rm + gp1 * rm_S) / (gm1 * rm_S + gp1 * rm)) - pi;
    const double ael = elastic_energy(el, k.mu[v]);
    double e_S = (p_S + k.gpi[v]) / (rm_S * gp1);
    // (a zero elastic energy adds a zero; rm_S or a fraction of zero makes it 0 / 0)
    const double den_e = s.avf[v] * rm_S;
    if (f64::abs_bits(ael) || !f64::moderate(den_e)) e_S += ael / den_e;
    nc.are[v] = ar_S[v] * e_S;
  }
#pragma unroll
  for (int v = 0; v < N; ++v) Us[C::i0 + v] = ar_S[v];
#pragma unroll
  for (int v = 0; v < 3; ++v) Us[C::i1 + v] = r_S * vel[v];
  Us[C::i2] = r_S * Em_S;
#pragma unroll
  for (int d = 0; d < 3; d++) nc.unc[d] = vel[d];
#pragma unroll
  for (int v = 0; v < N - 1; ++v) nc.avf[v] = s.avf[v];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) nc.A[3 * i + j] = Ag[i][j];
  unsigned st = 0;
#pragma unroll
  for (int iv = 0; iv < C::NC; ++iv)
    if (f64::is_nan(Us[iv])) st |= FFV_ST_NAN;
  return st;
}

// m5_flux.c (gfm false) / m5_flux_gfm.c (gfm true), normal component along face F:
// Fn[iv] = sum_d F[iv][d] n_d with n the signed unit axis of F.
template <int F, int N>
__device__ void flux_n(const Sol<N> &s, int flag, bool gfm, bool cons, NC<N> &nc, double *Fn) {
  using C = K5<N>;
  constexpr int a = Fr<F, 0>::ax, sg = Fr<F, 0>::sg;
  const double vu = gfm ? s.ut : s.u, vv = gfm ? s.vt : s.v, vw = gfm ? s.wt : s.w;
  const double vel[3] = {vu, vv, vw};
  const double va = vel[a];
#pragma unroll
  for (int v = 0; v < N; v++) Fn[C::i0 + v] = sgn<sg>(va * s.ra[v]);
#pragma unroll
  for (int b = 0; b < 3; b++)
    Fn[C::i1 + b] = sgn<sg>((gfm || cons) ? va * vel[b] * s.r - s.st[b][a]
                                          : va * vel[b] * s.r + s.st[b][a]);
  Fn[C::i2] = sgn<sg>(s.r * s.e * va - s.st[a][0] * vu - s.st[a][1] * vv - s.st[a][2] * vw);
  if (flag == 0 || flag == 3) {
#pragma unroll
    for (int d = 0; d < 3; d++) nc.unc[d] = vel[d];
#pragma unroll
    for (int v = 0; v < N - 1; ++v) nc.avf[v] = s.avf[v];
#pragma unroll
    for (int v = 0; v < N; ++v) nc.are[v] = s.are[v];
#pragma unroll
    for (int q = 0; q < 9; q++) nc.A[q] = (gfm || cons) ? s.A[q] : -s.A[q];
  } else if (flag == 4) {  // symmetry face (m5_flux.c:58-66): the velocity is the caller's
#pragma unroll
    for (int v = 0; v < N - 1; ++v) nc.avf[v] = s.avf[v];
#pragma unroll
    for (int v = 0; v < N; ++v) nc.are[v] = s.are[v];
#pragma unroll
    for (int q = 0; q < 9; q++) nc.A[q] = s.A[q];
  }
  const double ua = nc.unc[a];
#pragma unroll
  for (int v = 0; v < N - 1; ++v) Fn[C::i3 + v] = sgn<sg>(ua * nc.avf[v]);
#pragma unroll
  for (int v = 0; v < N; ++v) Fn[C::i4 + v] = sgn<sg>(ua * nc.are[v]);
  if (s.flat) {  // a fluid state: the star state's deformation is zero too
#pragma unroll
    for (int q = 0; q < 9; q++) Fn[C::i5 + q] = 0.0;
  } else {
#pragma unroll
    for (int q = 0; q < 9; q++) Fn[C::i5 + q] = sgn<sg>(ua * nc.A[q]);
  }
}

// K = a ? A : B, field by field (selects: the states stay in registers)
template <int N>
__device__ __forceinline__ void select_sol(bool a, const Sol<N> &A, const Sol<N> &B, Sol<N> &K) {
  K.r = a ? A.r : B.r;
  K.u = a ? A.u : B.u;
  K.v = a ? A.v : B.v;
  K.w = a ? A.w : B.w;
  K.e = a ? A.e : B.e;
  K.ut = a ? A.ut : B.ut;
  K.vt = a ? A.vt : B.vt;
  K.wt = a ? A.wt : B.wt;
#pragma unroll
  for (int i = 0; i < N; i++) {
    K.ra[i] = a ? A.ra[i] : B.ra[i];
    K.avf[i] = a ? A.avf[i] : B.avf[i];
    K.are[i] = a ? A.are[i] : B.are[i];
    K.p[i] = a ? A.p[i] : B.p[i];
  }
  K.flat = a ? A.flat : B.flat;
#pragma unroll
  for (int q = 0; q < 9; q++) K.A[q] = a ? A.A[q] : B.A[q];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) K.st[i][j] = a ? A.st[i][j] : B.st[i][j];
#pragma unroll
  for (int q = 0; q < K5<N>::NC; q++) K.vec[q] = a ? A.vec[q] : B.vec[q];
}

// m5_hllc.c:3-95 / m5_hllc_gfm.c:3-100 with the wave speeds, accumulated as
// m5_residual.c:155-165: ff += A (F.n + corr); unc receives the face velocity.  The solver's four
// branches share one star-region and one physical-flux evaluation, on the state of the contact's
// upwind side: lanes of a warp on different sides of the contact do not run one after the other.
template <int F, int N>
__device__ unsigned hllc_acc(const M5Consts &k, Sol<N> L, Sol<N> R, int bc, bool gfm,
                             double Area, double *ff, double unc[3]) {
  using C = K5<N>;
  const double vl3[3] = {L.u, L.v, L.w}, vr3[3] = {R.u, R.v, R.w};
  const double uL = loc<F, 0>(vl3), vL = loc<F, 1>(vl3), wL = loc<F, 2>(vl3);
  double uR = loc<F, 0>(vr3), vR = loc<F, 1>(vr3), wR = loc<F, 2>(vr3);
  if (gfm) {
    vR = vL;
    wR = wL;
    L.ut = L.u;
    L.vt = L.v;
    L.wt = L.w;
    R.ut = glob<F, 0>(uR, vR, wR);
    R.vt = glob<F, 1>(uR, vR, wR);
    R.wt = glob<F, 2>(uR, vR, wR);
    R.vec[C::i1 + 0] = R.ut * R.r;
    R.vec[C::i1 + 1] = R.vt * R.r;
    R.vec[C::i1 + 2] = R.wt * R.r;
    R.vec[C::i2] = R.r * R.e;
  }
  const double ruL = L.r * uL, ruR = R.r * uR;
  const double cL = sqrt(L.c2), cR = sqrt(R.c2);
  double a = uL + cL, b = uR + cR;
  const double SR = (a > b) ? a : b;
  a = uL - cL;
  b = uR - cR;
  const double SL = (a < b) ? a : b;
  double TL[3][3], TR[3][3];
  tens_to_local<F>(L.st, TL);
  tens_to_local<F>(R.st, TR);
  const double sL[3] = {TL[0][0], TL[0][1], TL[0][2]}, sR[3] = {TR[0][0], TR[0][1], TR[0][2]};
  double u_S = ((L.r * (uL * uL) - (sL[0])) - (R.r * (uR * uR) - (sR[0])) - (SL * ruL) +
                (SR * ruR)) / (ruL - ruR - (SL * L.r) + (SR * R.r));
  unsigned st = (f64::is_nan(u_S) || f64::is_nan(SR) || f64::is_nan(SL)) ? FFV_ST_NAN_SPEED : 0u;
  if (!gfm && bc == 4) u_S = 0.0;
  NC<N> nc;
  double Fn[C::NEQ], Us[C::NC];
  // 0: supersonic from the left, 1: left star state, 2: right star state, 3: supersonic from
  // the right
  const bool left_star = (gfm ? f64::lt0(SL) : f64::le0(SL)) && f64::ge0(u_S);
  const bool right_star = gfm ? (f64::lt0(u_S) && f64::gt0(SR)) : (f64::le0(u_S) && f64::ge0(SR));
  const int branch = f64::ge0(SL) ? 0 : left_star ? 1 : right_star ? 2 : f64::le0(SR) ? 3 : -1;
  if (branch < 0) {
    st |= FFV_ST_NO_BRANCH;
#pragma unroll
    for (int d = 0; d < 3; d++) unc[d] = 0.0;
    return st;  // adds nothing
  }
  const bool left = branch <= 1, starred = branch == 1 || branch == 2;
  Sol<N> K;
  select_sol<N>(left, L, R, K);
  const double SK = left ? SL : SR;
  if (starred)
    st |= star_region<F>(k, K, L.r, R.r, f64::gt0(L.phi0) && f64::gt0(R.phi0), left, u_S, SL, SR,
                         uL, vL, wL, uR, vR, wR, sL, sR, Us, nc);
  flux_n<F>(K, branch, gfm, k.flux_form == FFV_FLUX_CONSISTENT, nc, Fn);
#pragma unroll
  for (int iv = 0; iv < C::NC; ++iv) {
    const double corr = starred ? SK * (Us[iv] - K.vec[iv]) : 0.0;
    ff[iv] += (Area) * (Fn[iv] + corr);
  }
#pragma unroll
  for (int iv = C::NC; iv < C::i5; ++iv) ff[iv] += (Area) * Fn[iv];
  // (the deformation's flux of a fluid state is a zero)
  if (!K.flat)
#pragma unroll
    for (int iv = C::i5; iv < C::NEQ; ++iv) ff[iv] += (Area) * Fn[iv];
#pragma unroll
  for (int d = 0; d < 3; d++) unc[d] = nc.unc[d];
  return st;
}

// m5_hllc.c:56-85, a symmetry face (bc 1): the mean of the physical fluxes of the cell's own
// state (m5_facevalues.c, not the reconstructed face state) and of its mirror image
// (m5_bc_symmetry: normal velocity reversed), the advected volume fractions, energies and
// deformation moving with the mean velocity, no HLLC part; accumulated as m5_residual.c:155-165
template <int F, int N>
__device__ void symmetry_acc(const Sol<N> &Lc, bool cons, double Area, double *ff, double unc[3]) {
  using C = K5<N>;
  Sol<N> Rc;
  ghost<F, N>(Lc, 1, Rc);
  NC<N> nc;
  nc.unc[0] = 0.5 * (Lc.u + Rc.u);
  nc.unc[1] = 0.5 * (Lc.v + Rc.v);
  nc.unc[2] = 0.5 * (Lc.w + Rc.w);
  double FL[C::NEQ], FR[C::NEQ];
  flux_n<F>(Lc, 4, false, cons, nc, FL);
  flux_n<F>(Rc, 4, false, cons, nc, FR);
#pragma unroll
  for (int iv = 0; iv < C::NEQ; ++iv) ff[iv] += (Area) * ((0.5 * FL[iv]) + (0.5 * FR[iv]));
#pragma unroll
  for (int d = 0; d < 3; d++) unc[d] = nc.unc[d];
}

// ------------------------------------------------------------ relaxation (m5_relaxationvec.c)
// the N - 1 fractions scaled so that their sum is the upper bound
template <int N>
__device__ __forceinline__ void scale_vf(const M5Consts &k, double *avf, double sum) {
  const double dif = sum - k.hi;
  const f64::Rcp rs = f64::rcp(sum);
#pragma unroll
  for (int j = 0; j < N - 1; ++j) avf[j] = avf[j] - f64::div(avf[j], rs) * dif;
}

template <int N>
__device__ __forceinline__ void vf_limit_relax(const M5Consts &k, double *avf, bool elseif) {
  double sum = 0.0;
#pragma unroll
  for (int i = 0; i < N - 1; ++i) {
    if (f64::le(avf[i], k.lo)) avf[i] = k.lo;
    else if (f64::ge(avf[i], k.hi)) avf[i] = k.hi;
    if (!elseif && f64::ge(avf[i], k.hi)) avf[i] = k.hi;  // two ifs: a lower bound above the upper
    sum = i ? sum + avf[i] : avf[i];
  }
  if (f64::ge(sum, k.hi)) {
    scale_vf<N>(k, avf, sum);
    sum = k.hi;
  }
  avf[N - 1] = 1.0 - sum;
}

// 1 / x to about an ulp, for 1e-37 < |x| < 1e37: the FP32 reciprocal (conversions on the integer
// pipe) and two Newton-Raphson steps of x r = 1
__device__ __forceinline__ double rcp_near(double x) {
  double r = f64_of_f32(1.0f / f32_of_f64(x));
  r = fma(fma(-x, r, 1.0), r, r);
  return fma(fma(-x, r, 1.0), r, r);
}
// y / x, the quotient from that reciprocal corrected by its remainder (Markstein): the rounded
// quotient but where it lies within ~2^-100 of a midpoint.  Divisors beyond the reciprocal's range (a
// material thinned out to 1e-38 kg/m^3) take the division.
__device__ __forceinline__ double div_near(double y, double x) {
  if (((uint32_t)(f64::bits(x) >> 52) & 0x7FFu) - 901u > 244u) return f64::div_plain(y, x);
  const double r = rcp_near(x), q = y * r;
  return fma(fma(-q, x, y), r, q);
}

// Newton on sum_k alpha_k(p) = 1 along each material's isentrope (m5_relaxationvec.c:456-490), to
// |F| <= 1e-12 or the reference's cap of 500 iterations; alpha[k] receives the last iterate's
// fractions, the return value is true when an iterate is NaN.  The reference's arithmetic: an
// iterate that repeats bitwise is a fixed point (F, dF and the densities repeat with it), so
// leaving there gives exactly the reference's result.  Most non-converging face states of a stiff
// two-phase interface reach such a point within a few iterations and would otherwise spin to the
// cap.
template <int N>
__device__ __forceinline__ bool newton_reference(const M5Consts &k, const double *avf,
                                                 const double *ar, const bool *live,
                                                 const double *pk, double p, double *alpha) {
  double rk[N];
  f64::Rcp den[N];
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    alpha[iv] = 0.0;
    if (live[iv]) {
      rk[iv] = ar[iv] / avf[iv];
      den[iv] = f64::rcp(pk[iv] + k.pinf[iv]);
    }
  }
  double F = 1.0e-9, dF = 1.0e9, p_prev = NAN;
#pragma unroll 1
  for (int iter = 0; f64::abs_gt(F, 1.0e-12) && iter < 500; iter++) {
    p = p - F / dF;
#pragma unroll
    for (int iv = 0; iv < N; ++iv)
      if (f64::lt(p, k.pfloor[iv])) p = k.preset[iv];
    F = -1.0;
    dF = 0.0;
#pragma unroll
    for (int iv = 0; iv < N; ++iv) {
      if (live[iv]) {
        const double pp = p + k.pinf[iv];
        const double rho = rk[iv] * pow(f64::div(pp, den[iv]), k.igam[iv]);
        alpha[iv] = ar[iv] / rho;
        F = F + alpha[iv];
        dF = dF - ar[iv] / (k.gamma[iv] * rho * pp);
      }
    }
    if (f64::is_nan(p) || f64::is_nan(F) || f64::is_nan(dF)) return true;
    if (p == p_prev) break;
    p_prev = p;
  }
  return false;
}

// The same iteration without a reference to equal bit for bit (the consistent flux form).  The
// ratio x = (p + p_inf) / (p_k + p_inf) is near 1 in all but the cells of an interface or a strong
// shock: for |x - 1| <= 1/32 the power is 1 + t P(t), t = x - 1 (exact), P the binomial series to t^9
// (the first omitted term is below 3e-18), rounded once -- an error of at most 0.53 ulp, below
// pow's -- and the two other quotients start from Newton-Raphson reciprocals.  35 FP64 instructions
// per material and iteration against ~110 with pow and three divisions.  The iterates are the
// reference's but where the two powers round differently, so that the stopping test, |F| <= 1e-12,
// falls alike: with derivatives good to an ulp only, or a series in p - p_k (more exact still), it
// fell otherwise in one state of ~200,000 and moved a fraction by 1e-12.
template <int N>
__device__ __forceinline__ bool newton_series(const M5Consts &k, const double *avf,
                                              const double *ar, const bool *live,
                                              const double *pk, double p, double *alpha) {
  double rk[N];
  f64::Rcp den[N];
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    alpha[iv] = 0.0;
    if (live[iv]) {
      rk[iv] = ar[iv] / avf[iv];
      den[iv] = f64::rcp(pk[iv] + k.pinf[iv]);
    }
  }
  double F = 1.0e-9, dF = 1.0e9, p_prev = NAN;
#pragma unroll 1
  for (int iter = 0; f64::abs_gt(F, 1.0e-12) && iter < 500; iter++) {
    p = p - F / dF;
#pragma unroll
    for (int iv = 0; iv < N; ++iv)
      if (f64::lt(p, k.pfloor[iv])) p = k.preset[iv];
    F = -1.0;
    dF = 0.0;
#pragma unroll
    for (int iv = 0; iv < N; ++iv) {
      if (live[iv]) {
        const double pp = p + k.pinf[iv], x = f64::div(pp, den[iv]), t = x - 1.0;
        double pw;
        if (f64::abs_bits(t) <= 0x3fa0000000000000ull) {  // 1/32
          const double *c = k.binom[iv];
          pw = c[9];
#pragma unroll
          for (int j = 8; j >= 0; j--) pw = fma(pw, t, c[j]);
          pw = fma(pw, t, 1.0);
        } else {
          pw = pow(x, k.igam[iv]);
        }
        const double rho = rk[iv] * pw;
        alpha[iv] = div_near(ar[iv], rho);
        F = F + alpha[iv];
        dF = dF - div_near(ar[iv], k.gamma[iv] * rho * pp);
      }
    }
    if (f64::is_nan(p) || f64::is_nan(F) || f64::is_nan(dF)) return true;
    if (p == p_prev) break;
    p_prev = p;
  }
  return false;
}

template <int N, bool FAST>
__device__ unsigned relaxationvec(const M5Consts &k, double *V) {
  using C = K5<N>;
  double ar[N], are[N], avf[N], avf0[N], ael[N];
  double rho = 0.0;
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    ar[iv] = V[iv + C::i0];
    are[iv] = V[iv + C::i4];
    rho = iv ? rho + ar[iv] : ar[iv];
  }
  const f64::Rcp rr = f64::rcp(rho);
  const double u = f64::div(V[C::i1 + 0], rr), v = f64::div(V[C::i1 + 1], rr),
               w = f64::div(V[C::i1 + 2], rr);
  const double rE = V[C::i2];
#pragma unroll
  for (int iv = 0; iv < N - 1; ++iv) avf[iv] = V[iv + C::i3];
  vf_limit_relax<N>(k, avf, true);
#pragma unroll
  for (int iv = 0; iv < N; ++iv) avf0[iv] = avf[iv];
  {
    Elastic el;
    elastic_of(k, V + C::i5, el);
#pragma unroll
    for (int iv = 0; iv < N; ++iv) ael[iv] = elastic_energy(el, k.mu[iv]);
  }
  const double eps_sml = 1.0e-12;
  unsigned st = 0;
  int i_as = 0;
  if (N == 2 && k.prelax == 1) {  // closed form for two materials (only)
    double t0[N], p0[N];
#pragma unroll
    for (int iv = 0; iv < N; ++iv) {
      t0[iv] = 1.0 / (ar[iv] / avf[iv]);
      p0[iv] = (k.gm1[iv] * (are[iv] - ael[iv]) / avf[iv]) - k.gpi[iv];
    }
    const double *ga = k.gamma, *pi = k.pinf;
    const double A_1 = (avf[0] / ga[0]) * (p0[0] + pi[0]) / ((avf[0] / ga[0]) + (avf[1] / ga[1]));
    const double A_2 = (avf[1] / ga[1]) * (p0[1] + pi[1]) / ((avf[0] / ga[0]) + (avf[1] / ga[1]));
    const double d = (A_2 - A_1 - (pi[1] - pi[0]));
    const double pe = 0.5 * (A_1 + A_2 - (pi[0] + pi[1])) + sqrt(0.25 * (d * d) + A_1 * A_2);
    if (f64::is_nan(pe)) st |= FFV_ST_NAN;
#pragma unroll
    for (int iv = 0; iv < N; ++iv) {
      const double t1 = t0[iv] * (p0[iv] + ga[iv] * pi[iv] + (ga[iv] - 1.0) * pe) /
                        (pe + ga[iv] * pi[iv] + (ga[iv] - 1.0) * pe);
      const double rm = 1.0 / t1;
      avf[iv] = ar[iv] / rm;
    }
    vf_limit_relax<N>(k, avf, false);
  } else {  // PRELAX 3
    double pkinit[N];
    bool live[N], irelax = true;
#pragma unroll
    for (int iv = 0; iv < N; ++iv) {
      if (f64::lt0(avf[iv]) || f64::lt0(ar[iv])) {
        avf[iv] = eps_sml;
        ar[iv] = eps_sml;
        are[iv] = eps_sml;
      }
      if (f64::ge(avf[iv], 1.0)) avf[iv] = 1.0 - eps_sml;
    }
#pragma unroll
    for (int iv = 0; iv < N; ++iv)
      if (f64::gt(avf[iv], 1.0 - eps_sml)) irelax = false;
    if (irelax) {
      double p0 = 0.0;
#pragma unroll
      for (int iv = 0; iv < N; ++iv) {
        live[iv] = f64::gt(avf[iv], eps_sml);
        pkinit[iv] = 0.0;
        if (live[iv]) {
          pkinit[iv] = (k.gm1[iv] * (are[iv] - ael[iv]) / avf[iv]) - k.gpi[iv];
          if (f64::le(pkinit[iv], k.pfloor[iv])) pkinit[iv] = k.pfloor[iv];
        }
        p0 += avf[iv] * pkinit[iv];
      }
      double alpha[N];
      const bool nan = FAST ? newton_series<N>(k, avf, ar, live, pkinit, p0, alpha)
                            : newton_reference<N>(k, avf, ar, live, pkinit, p0, alpha);
      if (nan) st |= FFV_ST_NAN;
#pragma unroll
      for (int iv = 0; iv < N; ++iv)
        if (live[iv]) avf[iv] = alpha[iv];
      vf_limit_relax<N>(k, avf, true);
    }
    i_as = (k.mu[1] != 0.0 && avf[0] < avf[1]) ? 1 : 0;
  }
  // the deformation scales with the solid's fraction; a fluid's is zero
  if (!no_deformation(V + C::i5)) {
    const double ratio = avf[i_as] / avf0[i_as];
#pragma unroll
    for (int q = 0; q < 9; q++) V[q + C::i5] = V[q + C::i5] * ratio;
  }
  double e_elast = 0.0;
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    // a zero elastic energy adds a zero (where the quotients are defined)
    if (f64::abs_bits(ael[iv]) == 0 && f64::moderate(ar[iv]) && f64::moderate(rho)) continue;
    const double eK = ael[iv] / (ar[iv]);
    const double Ys = f64::div(ar[iv], rr);
    e_elast += Ys * eK;
  }
  const double e_hyd = f64::div(rE, rr) - 0.5 * (u * u + v * v + w * w) - e_elast;
  double num = 0.0, den = 0.0;
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    const f64::Rcp g1{k.gm1[iv], k.ig1[iv]};
    num += f64::div(avf[iv] * k.gamma[iv] * k.pinf[iv], g1);
    den += f64::div(avf[iv], g1);
  }
  const double p_relaxed = (rho * e_hyd - num) / den;
#pragma unroll
  for (int iv = 0; iv < N - 1; ++iv) {
    if (f64::is_nan(avf[iv])) st |= FFV_ST_NAN;
    V[iv + C::i3] = avf[iv];
  }
#pragma unroll
  for (int iv = 0; iv < N; iv++) {
    const f64::Rcp g1{k.gm1[iv], k.ig1[iv]};
    const double a2 = f64::div(avf[iv] * (p_relaxed + k.gpi[iv]), g1) + ael[iv];
    if (f64::is_nan(a2)) st |= FFV_ST_NAN;
    V[iv + C::i4] = a2;
  }
  return st;
}

// avf_limit.c:3-21 on a state vector
template <int N>
__device__ __forceinline__ void avf_limit(const M5Consts &k, double *S) {
  using C = K5<N>;
  double sum = 0.0;
#pragma unroll
  for (int v = 0; v < N - 1; ++v) {
    S[C::i3 + v] = clamp_vf(k, S[C::i3 + v]);
    sum = v ? sum + S[C::i3 + v] : S[C::i3 + v];
  }
  if (f64::gt(sum, k.hi)) scale_vf<N>(k, S + C::i3, sum);
}

template <int N>
__device__ __forceinline__ void load_state(const double *__restrict__ S, int64_t n, int64_t c,
                                           double *U) {
#pragma unroll
  for (int v = 0; v < K5<N>::NEQ; v++) U[v] = S[(int64_t)v * n + c];
}

// m5_facevalues_MUSCL.c:3-45 (iside 1): value across face f, volume fractions limited.  At a
// boundary the ghost's state vector is the cell's own with the clamped volume fractions of
// m5_facevalues.c:46-80 (the bc only changes the ghost's primitive velocity).
template <int N>
__device__ __forceinline__ void value_across(const M5Consts &k, const ffv_dmesh &m,
                                             const double *__restrict__ S, int64_t c, int f,
                                             uint32_t kind, const double *Sc, double *X) {
  using C = K5<N>;
  if (kind & FFV_FK_BC) {
#pragma unroll
    for (int i = 0; i < C::NEQ; i++) X[i] = Sc[i];
    avf_limit<N>(k, X);
  } else if (kind == FFV_FK_FINER) {
    const int32_t *sg = m.sub + 4 * (int64_t)m.nbr[(int64_t)f * m.n + c];
    const int64_t s0 = sg[0], s1 = sg[1], s2 = sg[2], s3 = sg[3];
#pragma unroll
    for (int i = 0; i < C::NEQ; i++) {
      const double *Sv = S + (int64_t)i * m.n;
      X[i] = ((Sv[s0] / 4.0 + Sv[s1] / 4.0) + Sv[s2] / 4.0) + Sv[s3] / 4.0;
    }
  } else {
    load_state<N>(S, m.n, m.nbr[(int64_t)f * m.n + c], X);
  }
  avf_limit<N>(k, X);
}

// ------------------------------------------------------------------------------ kernels
// m5_reconctruct.c:144-179: volume-fraction limits of a face state
template <int N>
__device__ __forceinline__ void face_vf_limit(const M5Consts &k, double *avf) {
  const double top = 1.0 - (2.0 * k.lo);
  double sum = 0.0;
#pragma unroll
  for (int iv = 0; iv < N - 1; ++iv) {
    if (f64::le(avf[iv], k.lo)) avf[iv] = k.lo;
    else if (f64::ge(avf[iv], top)) avf[iv] = top;
    sum = iv ? sum + avf[iv] : avf[iv];
  }
  if (f64::ge(sum, k.hi)) scale_vf<N>(k, avf, sum);
}

// The limited, not yet relaxed states of the two faces of one axis (blockIdx.y) of every cell:
// both faces' increments come from the same two one-sided slopes.  Between neighbours of the
// cell's own level at a power-of-two spacing the limiter works on bit patterns
// (f64::minmod_pair): four FP64 instructions per variable and axis, against ~50 with four divisions
// per face.  The internal energies keep the cell's value (the reference multiplies their slope
// by zero).  The states go to memory and m5_relax_faces relaxes them there: with six face
// states per cell in flight separately the FP64 pipe has more warps to take from, and the
// extra traffic (2 KB per cell) is 2 % of the FP64 time.
template <int N, int FA, int FB>
__device__ __forceinline__ void slopes_axis(const ffv_dmesh &m, const ffv_geom &g,
                                            const M5Consts &k, const double *__restrict__ S,
                                            double *__restrict__ SF, int64_t c) {
  using C = K5<N>;
  static_assert(fr_opp(FA) == FB, "opposite faces");
  const uint32_t info = m.info[c];
  const int l = ffv_info_level(info);
  const uint32_t ka = ffv_face_kind(info, FA), kb = ffv_face_kind(info, FB);
  double SL[C::NEQ], XA[C::NEQ], XB[C::NEQ];
  load_state<N>(S, m.n, c, SL);
  value_across<N>(k, m, S, c, FA, ka, SL, XA);
  value_across<N>(k, m, S, c, FB, kb, SL, XB);
  avf_limit<N>(k, SL);
  const bool plain = ka == FFV_FK_SAME && kb == FFV_FK_SAME && ((g.pow2 >> l) & 1u);
  const f64::Rcp da{g.dcc[l][face_class(ka)], g.rdcc[l][face_class(ka)]};
  const f64::Rcp db{g.dcc[l][face_class(kb)], g.rdcc[l][face_class(kb)]};
  const double fa = g.dcf[l][face_class(ka)], fb = g.dcf[l][face_class(kb)];
  const bool ba = (ka & FFV_FK_BC) != 0, bb = (kb & FFV_FK_BC) != 0;
#pragma unroll
  for (int i = 0; i < C::NEQ; i++) {
    double cA = 0.0, cB = 0.0;
    if (i < C::i4 || i >= C::i5) {
      const double dA = XA[i] - SL[i], dB = XB[i] - SL[i];
      if (plain) {
        f64::minmod_pair(dA, dB, da.r, cA, cB);
      } else if (!(ba || bb) || (i >= C::i3 && i < C::i4)) {
        // (next to a boundary only a volume fraction scaled twice can differ from the cell's: the
        // other variables' slopes there are 0 / 0)
        const double a = f64::div(dA, da), b = f64::div(dB, db);
        const bool opposed = f64::gt0(f64::neg(b) * a);
        const double ga = f64::abs_gt(b, a) ? a : f64::neg(b);
        const double gb = f64::abs_gt(a, b) ? b : f64::neg(a);
        if (!ba && opposed && f64::abs_gt(dA, 1e-10)) cA = fa * ga;
        if (!bb && opposed && f64::abs_gt(dB, 1e-10)) cB = fb * gb;
      }
    }
    XA[i] = SL[i] + cA;
    XB[i] = SL[i] + cB;
  }
  face_vf_limit<N>(k, XA + C::i3);
  face_vf_limit<N>(k, XB + C::i3);
#pragma unroll
  for (int i = 0; i < C::NEQ; i++) {
    SF[((int64_t)FA * C::NEQ + i) * m.n + c] = XA[i];
    SF[((int64_t)FB * C::NEQ + i) * m.n + c] = XB[i];
  }
}

template <int N>
__global__ void __launch_bounds__(128) m5_recon_slopes(ffv_dmesh m, ffv_geom g, M5Consts k,
                                                       const double *__restrict__ S,
                                                       double *__restrict__ SF) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  if (blockIdx.y == 0) slopes_axis<N, 0, 2>(m, g, k, S, SF, c);
  else if (blockIdx.y == 1) slopes_axis<N, 3, 1>(m, g, k, S, SF, c);
  else slopes_axis<N, 4, 5>(m, g, k, S, SF, c);
}

// Pressure relaxation of every face state (blockIdx.y the face), in place.  FP64 pipe 84 % busy; a
// warp runs as long as its slowest lane's Newton iteration (3.9 iterations on the wall mesh, 6 on
// the bubble's, the mean lane 2.8 and 3.9).  Slopes and relaxation in one kernel with the plain
// arithmetic took 11.35 ms per stage on the wall mesh (0.41 M cells); now 0.58 + 5.0 ms, and in
// the reference's form on the bubble mesh (51,584 cells) 1.94-2.54 ms against 0.11 + 1.5-2.1 ms.
template <int N, bool FAST>
__global__ void __launch_bounds__(128) m5_relax_faces(int64_t n, M5Consts k, double *SF,
                                                      unsigned *__restrict__ status) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double *U = SF + (int64_t)blockIdx.y * C::NEQ * n + c;
  double V[C::NEQ];
#pragma unroll
  for (int i = 0; i < C::NEQ; i++) V[i] = U[(int64_t)i * n];
  const unsigned st = relaxationvec<N, FAST>(k, V);
#pragma unroll
  for (int i = C::i3; i < C::NEQ; i++) U[(int64_t)i * n] = V[i];  // the rest is unchanged
  if (st) atomicOr(status, st);
}

template <int N>
__device__ __forceinline__ void load_face_state(const double *__restrict__ SF, int64_t n, int f,
                                                int64_t c, double *U) {
#pragma unroll
  for (int v = 0; v < K5<N>::NEQ; v++) U[v] = SF[((int64_t)f * K5<N>::NEQ + v) * n + c];
}

// Flux of cell c through face F -- its only neighbour there (same level or coarser), boundary or
// finer neighbour q -- into ff (area-weighted, from zero), the face velocity into un.  Returns
// whether it is a ghost-fluid face.
template <int N, int ORDER, int F>
__device__ bool face_flux(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k,
                          const double *__restrict__ S, const double *__restrict__ SF, int64_t c,
                          uint32_t info, int q, double *ff, double un[3], unsigned &st) {
  using C = K5<N>;
  constexpr int FO = fr_opp(F);
  const uint32_t kind = ffv_face_kind(info, F);
  const int l = ffv_info_level(info);
  double U[C::NEQ];
#pragma unroll
  for (int iv = 0; iv < C::NEQ; iv++) ff[iv] = 0.0;
  const auto phi_at = [&](int64_t o) {
    return phi0_of<N>(k, S[(int64_t)C::i3 * m.n + o], N > 2 ? S[(int64_t)(C::i3 + 1) * m.n + o] : 0.0);
  };
  Sol<N> L, R;
  if (kind == (FFV_FK_BC | FFV_BC_SYMMETRY)) {
    // the cell's own state, not the face state; the HLLC flux the reference computes first
    // for this face is discarded (m5_hllc.c:59-63)
    load_state<N>(S, m.n, c, U);
    make_sol<N>(k, U, 0.0, false, L);
    symmetry_acc<F, N>(L, k.flux_form == FFV_FLUX_CONSISTENT, g.area[l], ff, un);
    return false;
  }
  if (ORDER == 2) load_face_state<N>(SF, m.n, F, c, U);
  else load_state<N>(S, m.n, c, U);
  make_sol<N>(k, U, phi_at(c), ORDER == 2, L);
  const int bc = (kind & FFV_FK_BC) ? (int)(kind & 7u) : 0;
  if (bc) {
    ghost<F, N>(L, bc, R);
  } else {
    int64_t o = m.nbr[(int64_t)F * m.n + c];
    if (kind == FFV_FK_FINER) o = m.sub[4 * o + q];
    if (ORDER == 2) load_face_state<N>(SF, m.n, FO, o, U);
    else load_state<N>(S, m.n, o, U);
    make_sol<N>(k, U, phi_at(o), ORDER == 2, R);
  }
  const bool gfm = (f64::gt0(L.phi0) && f64::lt0(R.phi0)) || (f64::lt0(L.phi0) && f64::gt0(R.phi0));
  st |= hllc_acc<F, N>(k, L, R, bc, gfm, g.area[kind == FFV_FK_FINER ? l + 1 : l], ff, un);
  return gfm;
}

template <int N>
__device__ __forceinline__ void store_flux(int64_t n, int f, int64_t c, const double *ff,
                                           const double un[3], bool gfm, double *__restrict__ FF,
                                           double *__restrict__ UF, uint8_t *__restrict__ GF) {
  using C = K5<N>;
#pragma unroll
  for (int iv = 0; iv < C::NEQ; iv++) FF[((int64_t)f * C::NEQ + iv) * n + c] = ff[iv];
#pragma unroll
  for (int d = 0; d < 3; d++) UF[((int64_t)f * 3 + d) * n + c] = un[d];
  GF[(int64_t)f * n + c] = gfm ? FFV_FACE_GFM : 0;
}

template <int N, int ORDER, int F>
__device__ __forceinline__ void owner_flux(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k,
                                           const double *__restrict__ S,
                                           const double *__restrict__ SF, double *__restrict__ FF,
                                           double *__restrict__ UF, uint8_t *__restrict__ GF,
                                           unsigned *status, int64_t c) {
  if (c >= m.n) return;
  const uint32_t info = m.info[c];
  // a 1:1 face is evaluated by its earlier cell, and m5_cell_update takes the negative for the
  // other, as the reference's flux reuse does (m5_residual.c:80-99)
  if (ffv_face_kind(info, F) != FFV_FK_SAME || m.nbr[(int64_t)F * m.n + c] < c) return;
  double ff[K5<N>::NEQ], un[3];
  unsigned st = 0;
  const bool gfm = face_flux<N, ORDER, F>(m, g, k, S, SF, c, info, 0, ff, un, st);
  store_flux<N>(m.n, F, c, ff, un, gfm, FF, UF, GF);
  if (st) atomicOr(status, st);
}

template <int N, int ORDER, int F>
__device__ __forceinline__ void listed_flux(const ffv_dmesh &m, const ffv_geom &g,
                                            const M5Consts &k, const double *__restrict__ S,
                                            const double *__restrict__ SF, int64_t c, bool finer,
                                            bool live, double *__restrict__ FF,
                                            double *__restrict__ UF, uint8_t *__restrict__ GF,
                                            unsigned *status) {
  using C = K5<N>;
  const int q = finer ? (int)(threadIdx.x & 3) : 0;
  double ff[C::NEQ], un[3] = {0.0, 0.0, 0.0};
  unsigned st = 0;
  bool gfm = false;
  if (live) gfm = face_flux<N, ORDER, F>(m, g, k, S, SF, c, m.info[c], q, ff, un, st);
  if (finer) {
    // four lanes hold the four subfaces: their sum in order, the last one's velocity divided by
    // four (m5_residual.c:163-165)
    const int first = (threadIdx.x & 31) & ~3;
#pragma unroll
    for (int iv = 0; iv < C::NEQ; iv++) {
      const double x = ff[iv];
      double sum = __shfl_sync(0xffffffffu, x, first);
#pragma unroll
      for (int j = 1; j < 4; j++) sum += __shfl_sync(0xffffffffu, x, first + j);
      ff[iv] = sum;
    }
#pragma unroll
    for (int d = 0; d < 3; d++) un[d] = __shfl_sync(0xffffffffu, un[d], first + 3) * 0.25;
    gfm = (__ballot_sync(0xffffffffu, gfm) >> first) & 15u;
  }
  if (live && q == 0) store_flux<N>(m.n, F, c, ff, un, gfm, FF, UF, GF);
  if (st) atomicOr(status, st);
}

// All face fluxes in one launch.  The first blocks take the boundary, coarser and finer faces from
// the mesh's list of them (0.2 to 0.3 per cell on a refined mesh; as single lanes of the warps over
// all cells and faces they took a third to a half of the kernel), the others the faces between
// cells of one level, each once: the positive face of one axis of FFV_LIST_TPB cells.  FP64 pipe
// ~80 % busy; with the list 40.1 -> 19.5 ms per step on the wall mesh of 0.41 M cells (21.3 before
// it), 5.87 -> 3.83 ms on the bubble mesh of 51,584 (4.30).
template <int N, int ORDER>
__global__ void __launch_bounds__(FFV_LIST_TPB) m5_face_flux(ffv_dmesh m, ffv_geom g, M5Consts k,
                                                             ffv_face_list fl,
                                                             const double *__restrict__ S,
                                                             const double *__restrict__ SF,
                                                             double *__restrict__ FF,
                                                             double *__restrict__ UF,
                                                             uint8_t *__restrict__ GF,
                                                             unsigned *__restrict__ status) {
  int axis;
  int64_t c;
  if (ffv_owner_block(fl, m.n, axis, c)) {
    if (axis == 0) owner_flux<N, ORDER, owner_face(0)>(m, g, k, S, SF, FF, UF, GF, status, c);
    else if (axis == 1) owner_flux<N, ORDER, owner_face(1)>(m, g, k, S, SF, FF, UF, GF, status, c);
    else owner_flux<N, ORDER, owner_face(2)>(m, g, k, S, SF, FF, UF, GF, status, c);
    return;
  }
  bool live, finer;
  const int f = ffv_listed_face(fl, c, live, finer);
  switch (f) {
    case 0: listed_flux<N, ORDER, 0>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
    case 1: listed_flux<N, ORDER, 1>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
    case 2: listed_flux<N, ORDER, 2>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
    case 3: listed_flux<N, ORDER, 3>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
    case 4: listed_flux<N, ORDER, 4>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
    default: listed_flux<N, ORDER, 5>(m, g, k, S, SF, c, finer, live, FF, UF, GF, status); break;
  }
}

// Residual sum and non-conservative terms (m5_residual.c:171-214) for face F.  The reference
// multiplies every component with the unit normal's; on a Cartesian forest two of the three are
// zero and the third +-1, so one component's terms remain: u . n = sg u_a, and of the
// deformation's terms those of the face's axis.
template <int N, int F>
__device__ __forceinline__ void nonconservative(const ffv_geom &g, const Sol<N> &Cs,
                                                const double (*ast)[3][3], uint32_t info, int l,
                                                const double un[3], double *rhs) {
  using C = K5<N>;
  const uint32_t kind = ffv_face_kind(info, F);
  // (the reference sums four subface areas: a power-of-two multiple, the same double)
  const double Af = kind == FFV_FK_FINER ? 4.0 * g.area[l + 1] : g.area[l];
  constexpr int a = Fr<F, 0>::ax, b = a == 0 ? 1 : 0, d = a == 2 ? 1 : 2;
  constexpr int sg = Fr<F, 0>::sg;
#pragma unroll
  for (int iv = 0; iv < N - 1; ++iv) rhs[C::i3 + iv] += Af * sgn<sg>(Cs.avf[iv] * un[a]);
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    const double(*t)[3] = ast[iv];
    double x;
    if (Cs.flat) x = sgn<sg>(t[a][a] * un[a]);  // a pressure
    else x = sgn<sg>(t[a][0] * un[0]) + sgn<sg>(t[a][1] * un[1]) + sgn<sg>(t[a][2] * un[2]);
    rhs[C::i4 + iv] += Af * x;
  }
  if (Cs.flat) return;
  // row a: the other two rows with their velocities, the second subtracted
  // (m5_residual.c:199-214); the other rows: themselves with the normal velocity
  const double *A = Cs.A;
  double *R5 = rhs + C::i5;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    R5[3 * a + j] += Af * (sgn<sg>(A[3 * b + j] * un[b]) + sgn<-sg>(A[3 * d + j] * un[d]));
    R5[3 * b + j] += Af * sgn<sg>(A[3 * b + j] * un[a]);
    R5[3 * d + j] += Af * sgn<sg>(A[3 * d + j] * un[a]);
  }
}

template <int N>
__device__ __forceinline__ void clamp_zerou(const M5Consts &k, double *s, const double *sn) {
  using C = K5<N>;
#pragma unroll
  for (int v = 0; v < N; v++)
    if (f64::lt0(s[C::i0 + v])) s[C::i0 + v] = sn[C::i0 + v];
  constexpr int e5 = C::i5;
  if (k.zerou[0]) {
    s[C::i1 + 0] = sn[C::i1 + 0];
    s[e5 + 1] = sn[e5 + 1]; s[e5 + 2] = sn[e5 + 2]; s[e5 + 3] = sn[e5 + 3]; s[e5 + 6] = sn[e5 + 6];
  }
  if (k.zerou[1]) {
    s[C::i1 + 1] = sn[C::i1 + 1];
    s[e5 + 1] = sn[e5 + 1]; s[e5 + 3] = sn[e5 + 3]; s[e5 + 5] = sn[e5 + 5]; s[e5 + 7] = sn[e5 + 7];
  }
  if (k.zerou[2]) {
    s[C::i1 + 2] = sn[C::i1 + 2];
    s[e5 + 2] = sn[e5 + 2]; s[e5 + 5] = sn[e5 + 5]; s[e5 + 6] = sn[e5 + 6]; s[e5 + 7] = sn[e5 + 7];
  }
}

// residual + RK stage (m5_RK.c): writes RHS and the new state into Snew; stage-1 cells
// whose solid fraction crosses AVF_LIM get the partial update and a flag for m5_gfm_seq
template <int N>
__global__ void __launch_bounds__(128) m5_cell_update(ffv_dmesh m, ffv_geom g, M5Consts k,
                                                      const double *__restrict__ S,
                                                      double *__restrict__ SN,
                                                      const double *__restrict__ FF,
                                                      const double *__restrict__ UF,
                                                      double *__restrict__ RHS,
                                                      double *__restrict__ Snew,
                                                      uint8_t *__restrict__ flag,
                                                      int32_t *__restrict__ list,
                                                      const double *__restrict__ dtp, int irk,
                                                      unsigned *__restrict__ status) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  const uint32_t info = m.info[c];
  const int l = ffv_info_level(info);
  double s[C::NEQ], rhs[C::NEQ];
  load_state<N>(S, m.n, c, s);
  Sol<N> Cs;
  double ast[N][3][3];
  make_sol<N>(k, s, 0.0, false, Cs, ast);
#pragma unroll
  for (int iv = 0; iv < C::NEQ; iv++) rhs[iv] = 0.0;
#define FACE(F)                                                                          \
  {                                                                                      \
    int64_t fc = c;                                                                      \
    int ff = F;                                                                          \
    bool other = false;                                                                  \
    if (ffv_face_kind(info, F) == FFV_FK_SAME) {                                         \
      const int64_t o = m.nbr[(int64_t)F * m.n + c];                                     \
      if (o < c) {                                                                       \
        fc = o;                                                                          \
        ff = fr_opp(F);                                                                  \
        other = true;                                                                    \
      }                                                                                  \
    }                                                                                    \
    _Pragma("unroll") for (int iv = 0; iv < C::NEQ; iv++) {                              \
      const double x = FF[((int64_t)ff * C::NEQ + iv) * m.n + fc];                       \
      rhs[iv] += other ? f64::neg(x) : x;                                                \
    }                                                                                    \
    double un[3];                                                                        \
    _Pragma("unroll") for (int d = 0; d < 3; d++) {                                      \
      const double x = UF[((int64_t)ff * 3 + d) * m.n + fc];                             \
      un[d] = other ? f64::neg(x) : x;                                                   \
    }                                                                                    \
    nonconservative<N, F>(g, Cs, ast, info, l, un, rhs);                                 \
  }
  FACE(0) FACE(1) FACE(2) FACE(3) FACE(4) FACE(5)
#undef FACE
  // a non-positive density in the stage's input is reported (the arithmetic is untouched)
  unsigned st = f64::le0(Cs.r) ? FFV_ST_NEG_DENSITY : 0u;
#pragma unroll
  for (int iv = 0; iv < C::NEQ; iv++) {
    if (f64::is_nan(rhs[iv])) st |= FFV_ST_NAN;
    RHS[(int64_t)iv * m.n + c] = rhs[iv];
  }
  const double dt = *dtp, iV = g.inv_vol[l];
  const f64::Rcp V{g.vol[l], iV};
  double sn[C::NEQ];
  if (irk == 1) {
#pragma unroll
    for (int e = 0; e < C::NEQ; e++) {
      sn[e] = s[e];
      SN[(int64_t)e * m.n + c] = s[e];
    }
  } else {
    load_state<N>(SN, m.n, c, sn);
  }
  bool gfm = false;
  if (irk == 1) {
#pragma unroll
    for (int v = 0; v < N - 1; ++v) {
      if (k.mu[v] != 0.0) {
        const int e = C::i3 + v;
        const double phi_old = s[e] - k.avf_lim;
        const double buf = iV * rhs[e];
        const double as_new = sn[e] + dt * buf;
        if (phi_old * (as_new - k.avf_lim) < 0.0) gfm = true;
      }
    }
#pragma unroll
    for (int e = 0; e < C::NEQ; e++)
      if (!gfm || e >= C::i2) s[e] = sn[e] + dt * (iV * rhs[e]);
  } else {
    const double a = irk == 2 ? 3.0 / 4.0 : (irk == 3 ? 1.0 / 3.0 : 1.0 / 2.0);
    const double b = irk == 2 ? 1.0 / 4.0 : (irk == 3 ? 2.0 / 3.0 : 1.0 / 2.0);
    const double bdt = b * dt;
#pragma unroll
    for (int e = 0; e < C::NEQ; e++) s[e] = a * sn[e] + b * s[e] + f64::div(bdt * rhs[e], V);
  }
  if (!gfm) clamp_zerou<N>(k, s, sn);
#pragma unroll
  for (int e = 0; e < C::NEQ; e++) Snew[(int64_t)e * m.n + c] = s[e];
  flag[c] = gfm ? 1 : 0;
  if (gfm) list[1 + atomicAdd(list, 1)] = (int32_t)c;
  if (st) atomicOr(status, st);
}

// cell pressure relaxation (m5_relaxation_solid.c:16-32); flags and lists solid-fraction crossings
template <int N, bool FAST>
__global__ void __launch_bounds__(128) m5_relax_cell(int64_t n, M5Consts k,
                                                     const double *__restrict__ Sin,
                                                     double *__restrict__ Sout,
                                                     uint8_t *__restrict__ flag,
                                                     int32_t *__restrict__ list,
                                                     unsigned *__restrict__ status) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double s[C::NEQ];
  load_state<N>(Sin, n, c, s);
  const double phi_old = s[C::i3] - k.avf_lim;
  const unsigned st = relaxationvec<N, FAST>(k, s);
  // the plastic return where the reference's prototype would run it (m5_relaxation_solid.c:14),
  // after the relaxation so that the stored state lies on or inside the yield surface
  if (k.plastic) plastic_return<N>(k, s);
  // phi_new[0] exists in the reference only for a solid material 0 (else no trigger)
  const double phi_new = (k.mu[0] != 0.0) ? s[C::i3] - k.avf_lim : phi_old;
  const bool crossed = phi_old * phi_new < 0.0;
  flag[c] = crossed ? 1 : 0;
  if (crossed) list[1 + atomicAdd(list, 1)] = (int32_t)c;
#pragma unroll
  for (int e = 0; e < C::NEQ; e++) Sout[(int64_t)e * n + c] = s[e];
  if (st) atomicOr(status, st);
}

// The flagged cells in leaf order.  The kernels append them to list[1 ..], count list[0], as they come.
// Up to GFM_SORT are ranked in shared memory, by the first block alone.  More are collected anew from the
// flags: each of FFV_GFM_PARTS blocks takes a run of cells, writes the flagged ones to the start of that
// run's places in the list and their number to list_parts, and the last block to finish (it waits for
// none) goes on with all runs one after the other.  One block over all flags, 2048 cells a turn, took
// 19.5 ms on 16.8 M cells, beside 71 to 88 ms of fixes of some ten thousand; now 0.1 ms.
constexpr int GFM_TPB = 256, GFM_SORT = 2048, GFM_RUN = GFM_TPB * 16;
__host__ __device__ inline int64_t gfm_run(int64_t n) {
  return ((n + FFV_GFM_PARTS - 1) / FFV_GFM_PARTS + GFM_RUN - 1) / GFM_RUN * GFM_RUN;
}

// the flagged cells of this block's run, collected in order
__device__ void collect_run(int64_t n, const uint8_t *flag, int32_t *list, int32_t *parts) {
  __shared__ int warp_total[2][GFM_TPB / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t run = gfm_run(n), first = blockIdx.x * run, last = first + run < n ? first + run : n;
  int32_t *out = list + 1 + first;
  int found = 0, turn = 0;
  for (int64_t c0 = first; c0 < last; c0 += GFM_RUN) {
    const int64_t c = c0 + (int64_t)t * 16;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (c + 16 <= last) {  // 16-byte loads: the runs begin at multiples of that
      const uint4 v = *reinterpret_cast<const uint4 *>(flag + c);
      w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
      for (int i = 0; i < 16; i++)
        if (c + i < last) w[i >> 2] |= (uint32_t)flag[c + i] << (8 * (i & 3));
    }
    const int mine = __popc(w[0]) + __popc(w[1]) + __popc(w[2]) + __popc(w[3]);  // flags are 0 or 1
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    if (lane == 31) warp_total[turn][warp] = upto;
    __syncthreads();
    int at = found + upto - mine;
#pragma unroll
    for (int j = 0; j < GFM_TPB / 32; j++) {
      if (j < warp) at += warp_total[turn][j];
      found += warp_total[turn][j];
    }
    turn ^= 1;  // the next turn's totals go beside those that others may still read
    if (mine) {
#pragma unroll
      for (int i = 0; i < 16; i++)
        if ((w[i >> 2] >> (8 * (i & 3))) & 1u) out[at++] = (int32_t)(c + i);
    }
  }
  if (t == 0) parts[blockIdx.x] = found;
}

// m5_gfm.c (relax false) / m5_gfm_rel.c (relax true) for the flagged cells, one warp, in
// leaf order.  A neighbour earlier in leaf order is read from Snew (its final state of this
// pass), a later one from Sold, as the reference's in-place list walk sees them.  One launch of a few
// blocks, which end at once where no cell is flagged: a count, a scan and a scatter over all cells
// before it took 12-15 us of every pass on meshes that the step itself crosses in 80 us.
template <int N>
__global__ void __launch_bounds__(GFM_TPB) m5_gfm_seq(ffv_dmesh m, ffv_geom g, M5Consts k,
                                                      const uint8_t *__restrict__ flag,
                                                      int32_t *list, int32_t *parts,
                                                      const double *__restrict__ Sold,
                                                      double *__restrict__ Snew,
                                                      const double *__restrict__ SN,
                                                      const double *__restrict__ RHS,
                                                      const uint8_t *__restrict__ GF,
                                                      const double *__restrict__ dtp, int relax) {
  using C = K5<N>;
  __shared__ double s_phiR[6], s_vel[6][3], s_own[C::NEQ];
  __shared__ int32_t found[GFM_SORT], sorted[GFM_SORT];
  __shared__ bool last_block;
  const int cnt = *(volatile int32_t *)list;
  if (cnt == 0) return;
  const bool few = cnt <= GFM_SORT;
  if (few) {
    // (a block that starts after the first one has cleared the count finds none)
    if (blockIdx.x != 0) return;
    for (int i = threadIdx.x; i < cnt; i += GFM_TPB) found[i] = list[1 + i];
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += GFM_TPB) {
      const int32_t v = found[i];
      int r = 0;
      for (int j = 0; j < cnt; j++) r += found[j] < v;
      sorted[r] = v;
    }
    __syncthreads();
  } else {
    collect_run(m.n, flag, list, parts);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_block = atomicAdd(parts + FFV_GFM_PARTS, 1) == FFV_GFM_PARTS - 1;
    __syncthreads();
    if (!last_block) return;
    __threadfence();
    if (threadIdx.x == 0) parts[FFV_GFM_PARTS] = 0;
  }
  if (threadIdx.x == 0) list[0] = 0;  // for the next pass
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  const double DT = *dtp;
  // the run, its number of cells, the place in it
  int part = 0, left = few ? cnt : __ldcg(parts), at = 0;
  const int64_t run = gfm_run(m.n);
  for (int idx = 0; idx < cnt; idx++, at++) {
    while (at == left && part < FFV_GFM_PARTS - 1) {
      part++;
      left = __ldcg(parts + part);
      at = 0;
    }
    if (at == left) break;  // (the flags and the count agree)
    const int64_t c = few ? sorted[at] : __ldcg(list + 1 + part * run + at);
    const uint32_t info = m.info[c];
    const int l = ffv_info_level(info);
    if (lane == 0)
      for (int e = 0; e < C::NEQ; e++) s_own[e] = Snew[(int64_t)e * m.n + c];
    __syncwarp();
    double own[C::NEQ];
#pragma unroll
    for (int e = 0; e < C::NEQ; e++) own[e] = s_own[e];
    Sol<N> L;
    make_sol<N>(k, own, phi0_state<N>(k, own), false, L);
    if (lane < 6) {
      const int f = lane;
      const uint32_t kind = ffv_face_kind(info, f);
      double phiR = 0.0, vr[3] = {0.0, 0.0, 0.0};
      if (GF[(int64_t)f * m.n + c] & FFV_FACE_GFM) {
        Sol<N> R;
        if (kind & FFV_FK_BC) {
          const int bc = (int)(kind & 7u);
          switch (f) {
            case 0: ghost<0, N>(L, bc, R); break;
            case 1: ghost<1, N>(L, bc, R); break;
            case 2: ghost<2, N>(L, bc, R); break;
            case 3: ghost<3, N>(L, bc, R); break;
            case 4: ghost<4, N>(L, bc, R); break;
            default: ghost<5, N>(L, bc, R); break;
          }
        } else {
          const int64_t o = kind == FFV_FK_FINER ? m.sub[4 * (int64_t)m.nbr[(int64_t)f * m.n + c]]
                                                 : m.nbr[(int64_t)f * m.n + c];
          double so[C::NEQ];
          load_state<N>(o < c ? Snew : Sold, m.n, o, so);
          make_sol<N>(k, so, phi0_state<N>(k, so), false, R);
        }
        phiR = R.phi0;
        vr[0] = R.u;
        vr[1] = R.v;
        vr[2] = R.w;
      }
      s_phiR[f] = phiR;
      s_vel[f][0] = vr[0];
      s_vel[f][1] = vr[1];
      s_vel[f][2] = vr[2];
    }
    __syncwarp();
    if (lane == 0) {
      double s[C::NEQ], sn[C::NEQ];
#pragma unroll
      for (int e = 0; e < C::NEQ; e++) {
        s[e] = own[e];
        sn[e] = SN[(int64_t)e * m.n + c];
      }
      const double V = g.vol[l];
      double rho_new = 0.0, ut, vt, wt;
      if (!relax) {
        for (int v = 0; v < N; ++v) rho_new += s[v] + (DT / V) * RHS[(int64_t)v * m.n + c];
        ut = s[C::i1 + 0] + (DT / V) * RHS[(int64_t)(C::i1 + 0) * m.n + c];
        vt = s[C::i1 + 1] + (DT / V) * RHS[(int64_t)(C::i1 + 1) * m.n + c];
        wt = s[C::i1 + 2] + (DT / V) * RHS[(int64_t)(C::i1 + 2) * m.n + c];
        ut = ut / rho_new;
        vt = vt / rho_new;
        wt = wt / rho_new;
      } else {
        for (int v = 0; v < N; ++v) rho_new += s[v];
        ut = s[C::i1 + 0] / rho_new;
        vt = s[C::i1 + 1] / rho_new;
        wt = s[C::i1 + 2] / rho_new;
      }
      double nxi = 0.0, nyi = 0.0, nzi = 0.0, total = 0.0, ug[6], vg[6], wg[6];
      int nint = 0;
      for (int f = 0; f < 6; f++) {
        if (GF[(int64_t)f * m.n + c] & FFV_FACE_GFM) {
          const double phi = (L.phi0 + s_phiR[f]) / 2.0;
          const double A = g.area[ffv_face_kind(info, f) == FFV_FK_FINER ? l + 1 : l];
          const int ax = fr_n_axis(f), sg = fr_n_sign(f);
          const double nv[3] = {ax == 0 ? (double)sg : 0.0, ax == 1 ? (double)sg : 0.0,
                                ax == 2 ? (double)sg : 0.0};
          if (relax) {
            nxi += phi * A * nv[0];
            nyi += phi * A * nv[1];
            nzi += phi * A * nv[2];
          } else {
            nxi = phi * A * nv[0];
            nyi = phi * A * nv[1];
            nzi = phi * A * nv[2];
          }
          ug[nint] = s_vel[f][0];
          vg[nint] = s_vel[f][1];
          wg[nint] = s_vel[f][2];
          total += A;
          nint++;
        }
      }
      if (nint != 0) {
        const double norm = sqrt(nxi * nxi + nyi * nyi + nzi * nzi);
        nxi = -nxi / norm;
        nyi = -nyi / norm;
        nzi = -nzi / norm;
        double n1x, n1y, n1z;
        if (fabs(nzi) < 0.99) {
          n1x = nyi;
          n1y = -nxi;
          n1z = 0.0;
        } else {
          n1x = nzi;
          n1y = 0.0;
          n1z = -nxi;
        }
        const double n2x = nyi * n1z - nzi * n1y, n2y = nzi * n1x - nxi * n1z,
                     n2z = nxi * n1y - nyi * n1x;
        const double ul = ut * nxi + vt * nyi + wt * nzi;
        double vnl = 0.0, wnl = 0.0;
        int ft = 0;
        for (int f = 0; f < 6; f++) {
          if (GF[(int64_t)f * m.n + c] & FFV_FACE_GFM) {
            const double A = g.area[ffv_face_kind(info, f) == FFV_FK_FINER ? l + 1 : l];
            const double vl = ug[ft] * n1x + vg[ft] * n1y + wg[ft] * n1z;
            const double wl = ug[ft] * n2x + vg[ft] * n2y + wg[ft] * n2z;
            vnl = vl * (A / total);
            wnl = wl * (A / total);
            ft++;
          }
        }
        const double ung = ul * nxi + vnl * n1x + wnl * n2x;
        const double vng = ul * nyi + vnl * n1y + wnl * n2y;
        const double wng = ul * nzi + vnl * n1z + wnl * n2z;
        if (!relax)
          for (int v = 0; v < N; ++v) s[v] = s[v] + (DT / V) * RHS[(int64_t)v * m.n + c];
        s[C::i1 + 0] = rho_new * ung;
        s[C::i1 + 1] = rho_new * vng;
        s[C::i1 + 2] = rho_new * wng;
        s[C::i2] -= rho_new * 0.5 * (ut * ut + vt * vt + wt * wt);
        s[C::i2] += rho_new * 0.5 * (ung * ung + vng * vng + wng * wng);
      } else if (!relax) {
        for (int v = 0; v < N; ++v) s[v] = s[v] + (DT / V) * RHS[(int64_t)v * m.n + c];
        for (int d = 0; d < 3; d++)
          s[C::i1 + d] = s[C::i1 + d] + (DT / V) * RHS[(int64_t)(C::i1 + d) * m.n + c];
      }
      if (!relax) clamp_zerou<N>(k, s, sn);
      for (int e = 0; e < C::NEQ; e++) Snew[(int64_t)e * m.n + c] = s[e];
    }
    __syncwarp();
  }
}

// Whether a cell's speed over h is certainly below `fastest` and the cell certainly has one: an upper
// bound of m5_cfl_kernel's speed in FP32.  c^2 cancels -- a nearly absent stiff material's energy
// against its p_inf, the liquid's against its own -- so the bound is raised by the rounding of the terms
// and not of their sum: nine roundings of 6e-8 in all, taken as 1e-6.  The last fraction is formed as a
// double-float difference (1 - alpha in FP32 is off by 3e-8, of which p_inf = 3.2e10 beside a gas makes
// 3 % of c^2), and the fractions are within what the exact form leaves alone but for 1e-4 of the limit.
// The elastic energy only lowers c^2.  It is left out, but where it, or a value that is not finite,
// could leave a cell without a speed, the cell is not passed over: with eps^2 = |A A^T - I|^2 <= 0.01 it
// is below 2 mu eps^2 (eigenvalues 1 + l of G, |l| <= eps, sum (l - g)^2 <= (1 + sqrt 3)^2 eps^2 and
// |G|^(1/6) >= 0.948).
template <int N>
__device__ __forceinline__ bool certainly_slower(const M5Consts &k, const double *s, float ih,
                                                 float fastest) {
  using C = K5<N>;
  bool sure = true;
  float rf = 0.0f, uf = 0.0f, cf = 0.0f, err = 0.0f, softer = 0.0f;
  df rest = df_make(1.0f);
  float deformed = 0.0f;  // eps^2, rounding included
  if (k.nsolids != 0) {
    float A[9];
    bool any = false;
#pragma unroll
    for (int q = 0; q < 9; q++) {
      A[q] = f32_of_f64(s[C::i5 + q]);
      any |= f64::abs_bits(s[C::i5 + q]) != 0;
    }
    if (any) {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
          const float e = (A[3 * i] * A[3 * j] + A[3 * i + 1] * A[3 * j + 1] + A[3 * i + 2] * A[3 * j + 2]) -
                          (i == j ? 1.0f : 0.0f);
          deformed += (i == j ? 1.0f : 2.0f) * e * e;
        }
      sure = deformed <= 0.01f;  // (not where it is NaN)
      deformed = deformed * 1.02f + 1.0e-10f;
    }
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float r = f32_of_f64(s[i]);
    sure &= r >= 0.0f;
    rf += r;
    float a;
    if (i < N - 1) {
      const df x = df_from_double(s[C::i3 + (i < N - 1 ? i : 0)]);
      a = x.hi;
      sure &= a >= k.alo_f && a <= k.ahi_f;
      rest = df_sub(rest, x);
    } else {
      a = rest.hi;
      sure &= a >= 0.9999f * k.alo_f;
    }
    const float w = k.gamma_f[i] * (k.gamma_f[i] - 1.0f), e = f32_of_f64(s[C::i4 + i]);
    cf += w * (e - a * k.pinf_f[i]);
    err += w * (1.0e-6f * (fabsf(e) + a * k.pinf_f[i]) + 1.0e-4f * k.alo_f * k.pinf_f[i]);
    softer += w * 2.0f * k.mu_f[i] * deformed;
  }
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float u = fabsf(f32_of_f64(s[C::i1 + d]));
    sure &= u <= 3.0e38f;
    uf = fmaxf(uf, u);
  }
  sure &= rf > 1.0e-20f && rf < 1.0e30f && cf > 1.0e-20f && cf > 1.01f * (err + softer);
  return sure && (uf / rf + sqrtf((cf + err) / rf)) * ih * 1.001f < fastest;
}

// CFL (new, the reference has a fixed DT): dt = h / (max_a |u_a| + c), mixture sound speed
// c^2 = sum_k (alpha_k / rho) gamma_k (p_k + p_inf_k) as m5_wave_speeds.c:43-50 forms it.  With the
// pressure put in, alpha_k (p_k + p_inf_k) = (gamma_k - 1) (alpha rho e_k - e_el - alpha_k p_inf_k)
// needs no division by a fraction; at a power-of-two spacing the smallest dt is the reciprocal of
// the largest speed over h.  A cell certainly slower than the thread's largest so far is passed
// over.  The rest are bound by the FP64 pipe: ffv_cfl_dt took 298 / 1404 / 6186 us on wall meshes of
// 0.41, 2.5 and 10.1 M cells with all cells in FP64, now 150 / 433 / 1773 us (a bound that left out the
// deformation and the rounding of the terms 112 / 409 / 1331 us).
template <int N>
__global__ void m5_cfl_kernel(ffv_dmesh m, ffv_geom g, M5Consts k, const double *__restrict__ S,
                              unsigned long long *out) {
  using C = K5<N>;
  double best = INFINITY;
  uint64_t fastest = 0;  // bits of the largest speed / h (NaN above all)
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < m.n;
       c += (int64_t)gridDim.x * blockDim.x) {
    double s[C::NEQ];
    load_state<N>(S, m.n, c, s);
    const int l = ffv_info_level(m.info[c]);
    const bool scaled = (g.pow2 >> l) & 1u;
    if (scaled && fastest && certainly_slower<N>(k, s, g.idcc_f[l][0], f32_of_f64(f64::of_bits(fastest)))) continue;
    double r = s[0];
#pragma unroll
    for (int i = 1; i < N; ++i) r += s[i];
    const f64::Rcp rr = f64::rcp(r);
    avf_limit<N>(k, s);
    double last = 1.0 - s[C::i3];
    if (N > 2) last = 1.0 - (s[C::i3] + s[C::i3 + 1]);
    Elastic el;
    elastic_of(k, s + C::i5, el);
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const double a = i < N - 1 ? s[C::i3 + (i < N - 1 ? i : 0)] : last;
      sum += k.gamma[i] * k.gm1[i] * ((s[C::i4 + i] - elastic_energy(el, k.mu[i])) - a * k.pinf[i]);
    }
    uint64_t um = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) um = um > f64::abs_bits(s[C::i1 + d]) ? um : f64::abs_bits(s[C::i1 + d]);
    const double sp = f64::of_bits(f64::abs_bits(f64::div(f64::of_bits(um), rr))) + sqrt(f64::div(sum, rr));
    if (scaled) {
      const uint64_t v = f64::bits(sp * g.rdcc[l][0]);
      fastest = v > fastest ? v : fastest;  // a speed is not negative; NaN sorts above infinity
    } else {
      const double dt = g.h[l] / sp;
      best = (dt < best || isnan(dt)) ? dt : best;
    }
  }
  if (fastest) {
    const double dt = 1.0 / f64::of_bits(fastest);
    best = (dt < best || isnan(dt)) ? dt : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double other = __shfl_xor_sync(0xffffffffu, best, o);
    best = (other < best || isnan(other)) ? other : best;
  }
  if ((threadIdx.x & 31) == 0) {
    // a cell without a speed leaves no stable step: 0 (as NaN it would lose to every other warp's
    // step, and its own warp's cells with it)
    atomicMin(out, best >= 0.0 ? (unsigned long long)__double_as_longlong(best) : 0ULL);
  }
}

// ------------------------------------------------------------------ refinement tags
// neighbour q (< count) of cell c across face f; count 0 for boundary faces
__device__ __forceinline__ int face_neighbours(const ffv_dmesh &m, int64_t c, uint32_t info, int f,
                                               int64_t nb[4]) {
  const uint32_t kind = ffv_face_kind(info, f);
  if (kind & FFV_FK_BC) return 0;
  const int32_t s = m.nbr[(int64_t)f * m.n + c];
  if (kind == FFV_FK_FINER) {
#pragma unroll
    for (int q = 0; q < 4; q++) nb[q] = m.sub[4 * (int64_t)s + q];
    return 4;
  }
  nb[0] = s;
  return 1;
}

// the sign of phi[v], v = 0, 1 (m5_facevalues.c:83-99): the clamped volume fractions against AVF_LIM
// (phi[0] the larger of two solids' fractions when there are two); two bits each: 0 below, 1 equal
// (or NaN), 2 above
__device__ __forceinline__ uint32_t phi_code(double a, double lim) {
  const int64_t x = f64::order_key(a + 0.0), y = f64::order_key(lim + 0.0);  // (-0 as +0)
  return f64::is_nan(a) || x == y ? 1u : (x < y ? 0u : 2u);
}
// What the criterion reads of every cell, made once: the signs of phi, the density and (where a
// pressure criterion is on) the alpha-weighted pressure sum_k alpha_k p_k from the reference's cell
// primitives (make_sol of the cell state), each also rounded to FP32 for the jumps' screen.
struct TagCells {
  double *pr, *rho;
  float *pr_f, *rho_f;
  uint8_t *phi;
};
template <int N>
__global__ void __launch_bounds__(128) m5_tag_cells(int64_t n, M5Consts k, bool prs, bool rho,
                                                    const double *__restrict__ S, TagCells t) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const double a0 = clamp_vf(k, S[(int64_t)C::i3 * n + c]);
  uint32_t code;
  if (N > 2) {
    const double a1 = clamp_vf(k, S[(int64_t)(C::i3 + 1) * n + c]);
    code = phi_code(k.nsolids == 2 && k.mu[0] != 0.0 && !f64::gt(a0, a1) ? a1 : a0, k.avf_lim) |
           phi_code(a1, k.avf_lim) << 2;
  } else {
    code = phi_code(a0, k.avf_lim) | 1u << 2;
  }
  t.phi[c] = (uint8_t)code;
  if (prs) {
    double s[C::NEQ];
    load_state<N>(S, n, c, s);
    Sol<N> q;
    make_sol<N>(k, s, 0.0, false, q);
    double p = 0.0;
#pragma unroll
    for (int iv = 0; iv < N; ++iv) p += q.avf[iv] * q.p[iv];
    t.pr[c] = p;
    t.pr_f[c] = f32_of_f64(p);
  }
  if (rho) {
    double r = S[c];
#pragma unroll
    for (int i = 1; i < N; ++i) r += S[(int64_t)i * n + c];
    t.rho[c] = r;
    t.rho_f[c] = f32_of_f64(r);
  }
}

// Interface layers: one word per cell, SI[0] in its low half, SI[1] in the high one; W is 32 bits wide,
// or 64 where layers beyond 65535 can be asked for (a mesh of more cells than that and as many layers:
// one word is half the bytes, and 16 bits are enough for all others).
template <typename W>
__device__ __forceinline__ int si_low(W w) { return (int)(w & ((W(1) << (4 * sizeof(W))) - 1)); }
template <typename W>
__device__ __forceinline__ int si_high(W w) { return (int)(w >> (4 * sizeof(W))); }

// what the neighbours across a face show: hit(neighbour) of any of them, bit v for SI[v]
template <typename Hit>
__device__ __forceinline__ int face_shows(const ffv_dmesh &m, uint32_t kind, int32_t nb, Hit hit) {
  if (kind & FFV_FK_BC) return 0;
  if (kind != FFV_FK_FINER) return hit(nb);
  const int4 s = *reinterpret_cast<const int4 *>(m.sub + 4 * (int64_t)nb);
  return hit(s.x) | hit(s.y) | hit(s.z) | hit(s.w);
}
// the first face (in order) that shows any bit of `want`: its bits.  All six faces' loads are in
// flight together.
template <typename Hit>
__device__ __forceinline__ int first_face(const ffv_dmesh &m, int64_t c, int want, Hit hit) {
  const uint32_t info = m.info[c];
  int32_t nb[6];
#pragma unroll
  for (int f = 0; f < 6; f++) nb[f] = m.nbr[(int64_t)f * m.n + c];
  int shows[6];
#pragma unroll
  for (int f = 0; f < 6; f++) shows[f] = face_shows(m, ffv_face_kind(info, f), nb[f], hit);
  int set = 0;
#pragma unroll
  for (int f = 0; f < 6; f++)
    if (set == 0) set = shows[f] & want;
  return set;
}

// interface_location.c:17-46: SI = 1 where phi changes sign across a face (the face loop
// stops after the first face that shows a change); those cells are listed (list nullable)
template <typename W>
__global__ void __launch_bounds__(128) m5_si_first(ffv_dmesh m, const uint8_t *__restrict__ phi,
                                                   W *__restrict__ SI,
                                                   int32_t *__restrict__ list,
                                                   int32_t *__restrict__ count) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int set = 0;
  if (c < m.n) {
    const uint32_t own = phi[c];
    set = first_face(m, c, 3, [&](int32_t o) {
      const uint32_t x = own ^ phi[o];
      return ((x & 3u) == 2u ? 1 : 0) | ((x >> 2) == 2u ? 2 : 0);
    });
    SI[c] = (W)(set & 1) | (W)(set >> 1) << (4 * sizeof(W));
  }
  if (!list) return;
  const unsigned b = __ballot_sync(0xffffffffu, set != 0);
  if (b == 0) return;
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(count, __popc(b));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (set) list[at + __popc(b & ((1u << lane) - 1u))] = (int32_t)c;
}

// interface_location.c:52-80 for one cell: what layer lvl sets in it (bit v), from its
// neighbours' layer lvl - 1.  The reference updates in place in leaf order, but a cell only reads
// neighbours' lvl - 1 entries and only writes lvl into entries that were 0, so updating in place in
// any order gives the same result (an entry that already is lvl was 0 before this layer).
template <typename W>
__device__ __forceinline__ int si_free(W w, int lvl) {
  const int s0 = si_low(w), s1 = si_high(w);
  return (s0 == 0 || s0 == lvl ? 1 : 0) | (s1 == 0 || s1 == lvl ? 2 : 0);
}
template <typename W>
__device__ __forceinline__ int si_is(W w, int lvl) {
  return (si_low(w) == lvl ? 1 : 0) | (si_high(w) == lvl ? 2 : 0);
}
template <typename W>
__device__ __forceinline__ int si_set(const ffv_dmesh &m, int lvl, const W *SI, int64_t c, int free) {
  return first_face(m, c, free, [&](int32_t o) { return si_is(__ldcg(SI + o), lvl - 1); });
}
template <typename W>
__device__ __forceinline__ W si_word(int set, int lvl) {
  return (set & 1 ? (W)lvl : W(0)) | (set & 2 ? (W)lvl << (4 * sizeof(W)) : W(0));
}

// Layer lvl from the cells that layer lvl - 1 set: only their neighbours can be next to it.  A
// neighbour of several is evaluated by each, with the same outcome; the one that sets its first
// entry lists it for the next layer.  Bound by the latency of its chain of loads, so every SM is
// filled.  The criterion's device part (cells, fourteen layers, split) took ~2.9 ms on the wall mesh
// of 2.5 M cells with every layer over all cells and FP64 jumps and signs; now ~0.8 ms.
template <typename W>
__global__ void __launch_bounds__(128) m5_si_grow(ffv_dmesh m, int lvl, W *SI,
                                                  const int32_t *__restrict__ from,
                                                  int32_t *__restrict__ to, int32_t *count) {
  const int n_from = count[(lvl - 1) % 3];
  if (blockIdx.x == 0 && threadIdx.x == 0) count[(lvl + 1) % 3] = 0;  // the next layer's
  // eight threads per cell: six faces
  const int face = threadIdx.x & 7;
  if (face >= 6) return;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; i < n_from;
       i += ((int64_t)gridDim.x * blockDim.x) >> 3) {
    const int64_t b = from[i];
    const int mine = si_is(__ldcg(SI + b), lvl - 1);
    const auto visit = [&](int32_t c) {
      const int free = si_free(__ldcg(SI + c), lvl);
      if (!(free & mine)) return 0;
      const int set = si_set(m, lvl, SI, c, free);
      if (!set) return 0;
      const W before = atomicOr(SI + c, si_word<W>(set, lvl));
      // the first of its visitors to set its first entry
      if ((set & 1 ? si_low(before) : si_high(before)) == 0) to[atomicAdd(count + lvl % 3, 1)] = c;
      return 0;
    };
    face_shows(m, ffv_face_kind(m.info[b], face), m.nbr[(int64_t)face * m.n + b], visit);
  }
}

// layer lvl over all cells: meshes whose neighbour relation is not symmetric (a part of a forest:
// a fine cell sees a coarser one whose own face towards it became a boundary)
template <typename W>
__global__ void __launch_bounds__(128) m5_si_layer(ffv_dmesh m, int lvl, W *SI) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  const W w = SI[c];
  const int free = si_free(w, lvl);
  if (free == 0) return;
  const int set = si_set(m, lvl, SI, c, free);
  if (set) SI[c] = w | si_word<W>(set, lvl);
}

// the layers as two arrays
template <typename W>
__global__ void __launch_bounds__(256) m5_si_unpack(int64_t n, const W *__restrict__ SI,
                                                    int32_t *__restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const W w = SI[c];
  out[c] = si_low(w);
  out[n + c] = si_high(w);
}

// relative jump |x_nb - x| / max(|x_nb|, |x|) (criterionsplt.c:83-89), 0 below 1e-8
__device__ __forceinline__ double rel_jump(double x_cur, double x_nb) {
  const double eps = 1.0e-8;
  if ((fabs(x_nb) > eps) || (fabs(x_cur) > eps)) {
    const double a = fabs(x_nb), b = fabs(x_cur);
    return fabs(x_nb - x_cur) / ((a > b) ? a : b);
  }
  return 0.0;
}

// Whether a neighbour's jump reaches the threshold.  The FP32 values decide where the jump is not
// within 1e-6 of it -- their rounding moves the ratio by less than 3e-7 -- and the magnitudes are
// ordinary; the rest take the FP64 expression.
__device__ __forceinline__ bool jump_reaches(double thr, float thr_f, const double *x,
                                             const float *xf, int64_t c, int64_t o) {
  const float a = xf[c], b = xf[o];
  const float d = fabsf(b - a), big = fmaxf(fabsf(a), fabsf(b));
  if (big > 1e-6f && big < 1e30f) {
    if (d > (thr_f + 1e-6f) * big) return true;
    if (d < (thr_f - 1e-6f) * big) return false;
  }
  return rel_jump(x[c], x[o]) >= thr;
}

// criterionsplt.c:3-140 per cell: the uniform level, the gradient criterion over every
// sub-neighbour (largest jump against the threshold: any neighbour's reaches it) and the interface
// layers
template <typename W>
__global__ void __launch_bounds__(128) m5_tag_split(ffv_dmesh m, ffv_m5_tagc t, TagCells x,
                                                    const W *__restrict__ SI,
                                                    int32_t *__restrict__ split) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  int level = 1;
  if (t.uniform == 1) level = level > t.lvl_uniform ? level : t.lvl_uniform;
  if (t.prs == 1 || t.rho == 1 || t.vel == 1) {
    const uint32_t info = m.info[c];
    // (no neighbour jumps by less than zero: a threshold at or below it is always reached)
    bool hp = 0.0 >= t.thr_prs, hr = 0.0 >= t.thr_rho, hv = 0.0 >= t.thr_vel;
    const float fp = (float)t.thr_prs, fr = (float)t.thr_rho, fv = (float)t.thr_vel;
    for (int f = 0; f < 6; f++) {
      int64_t nb[4];
      const int cnt = face_neighbours(m, c, info, f, nb);
      for (int q = 0; q < cnt; q++) {
        if (t.prs == 1 && !hp) hp = jump_reaches(t.thr_prs, fp, x.pr, x.pr_f, c, nb[q]);
        if (t.rho == 1 && !hr) hr = jump_reaches(t.thr_rho, fr, x.rho, x.rho_f, c, nb[q]);
        // the reference's velocity criterion takes the density jump (criterionsplt.c:120), which
        // it has where the density criterion is on
        if (t.vel == 1 && t.rho == 1 && !hv) hv = jump_reaches(t.thr_vel, fv, x.rho, x.rho_f, c, nb[q]);
      }
    }
    int lt = 1;
    if (t.prs == 1 && hp) lt = t.lvl_prs;
    if (t.rho == 1 && hr) lt = t.lvl_rho;
    if (t.vel == 1 && hv) lt = t.lvl_vel;
    level = level > lt ? level : lt;
  }
  if (t.inter0 != 0) {
    for (int v = 0; v < 2; ++v) {
      const int si = v ? si_high(SI[c]) : si_low(SI[c]);
      if (si >= 1 && si < t.lrs0) level = level > t.lvl0 ? level : t.lvl0;
      if (si >= t.lrs0 && si < t.lrs1) level = level > t.lvl1 ? level : t.lvl1;
    }
  }
  split[c] = level;
}

// exported fields (FP64): rho, u, v, w, sum_k alpha_k p_k, alpha_k, p_k, von Mises stress
// of the reference's cell primitives (make_sol of the cell state)
template <int N>
__global__ void __launch_bounds__(128) m5_export_fields(int64_t n, M5Consts k,
                                                        const double *__restrict__ S,
                                                        double *__restrict__ F) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double s[C::NEQ];
  load_state<N>(S, n, c, s);
  Sol<N> q;
  make_sol<N>(k, s, 0.0, false, q);
  double p = 0.0;
#pragma unroll
  for (int iv = 0; iv < N; ++iv) p += q.avf[iv] * q.p[iv];
  const double tr = (q.st[0][0] + q.st[1][1] + q.st[2][2]) / 3.0;
  double j2 = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double d = q.st[i][j] - (i == j ? tr : 0.0);
      j2 += d * d;
    }
  F[c] = q.r;
  F[n + c] = -q.u;  // the state holds the negated momentum in this node layout
  F[2 * n + c] = -q.v;
  F[3 * n + c] = -q.w;
  F[4 * n + c] = p;
#pragma unroll
  for (int iv = 0; iv < N; ++iv) {
    F[(int64_t)(5 + iv) * n + c] = q.avf[iv];
    F[(int64_t)(5 + N + iv) * n + c] = q.p[iv];
  }
  F[(int64_t)(5 + 2 * N) * n + c] = sqrt(1.5 * j2);
}

// merged cells of a mesh adaptation (map < 0): the reference's relaxation of the merged
// state (merge.c:52-57)
template <int N, bool FAST>
__global__ void __launch_bounds__(128) m5_relax_merged(int64_t n, M5Consts k,
                                                       const int64_t *__restrict__ map,
                                                       double *__restrict__ S) {
  using C = K5<N>;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n || map[c] >= 0) return;
  double s[C::NEQ];
  load_state<N>(S, n, c, s);
  relaxationvec<N, FAST>(k, s);
#pragma unroll
  for (int e = 0; e < C::NEQ; e++) S[(int64_t)e * n + c] = s[e];
}

}  // namespace

void ffv_m5_relax_merged(int64_t n, const M5Consts &k, const int64_t *map, double *S,
                         cudaStream_t st) {
  const unsigned gc = (unsigned)((n + 127) / 128);
  const bool fast = k.flux_form == FFV_FLUX_CONSISTENT;
  if (k.nmat == 2) (fast ? m5_relax_merged<2, true> : m5_relax_merged<2, false>)<<<gc, 128, 0, st>>>(n, k, map, S);
  else (fast ? m5_relax_merged<3, true> : m5_relax_merged<3, false>)<<<gc, 128, 0, st>>>(n, k, map, S);
}

void ffv_m5_export_fields(int64_t n, const M5Consts &k, const double *S, double *F,
                          cudaStream_t st) {
  const unsigned gc = (unsigned)((n + 127) / 128);
  if (k.nmat == 2) m5_export_fields<2><<<gc, 128, 0, st>>>(n, k, S, F);
  else m5_export_fields<3><<<gc, 128, 0, st>>>(n, k, S, F);
}

namespace {
template <typename W>
void tags_impl(const ffv_dmesh &m, const M5Consts &k, const ffv_m5_tagc &t, bool symmetric, const double *S,
               W *SI, int32_t *lists, int32_t *split, double *pr, cudaStream_t st) {
  const unsigned gc = (unsigned)((m.n + 127) / 128);
  // pr: pressure, density [n] doubles each, then both as floats; the phi codes wait in split
  float *f = reinterpret_cast<float *>(pr + 2 * m.n);
  const TagCells x{pr, pr + m.n, f, f + m.n, reinterpret_cast<uint8_t *>(split)};
  const bool prs = t.prs == 1, rho = t.rho == 1 || t.vel == 1;
  if (t.inter0 != 0 || prs || rho) {
    if (k.nmat == 2) m5_tag_cells<2><<<gc, 128, 0, st>>>(m.n, k, prs, rho, S, x);
    else m5_tag_cells<3><<<gc, 128, 0, st>>>(m.n, k, prs, rho, S, x);
  }
  if (t.inter0 != 0) {
    // two lists of at most n cells and the counts of three layers
    int32_t *list[2] = {lists, lists + m.n}, *count = lists + 2 * m.n;
    cudaMemsetAsync(count, 0, 3 * sizeof(int32_t), st);
    m5_si_first<<<gc, 128, 0, st>>>(m, x.phi, SI, symmetric ? list[1] : nullptr, count + 1);
    for (int lvl = 2; lvl < t.si_max; lvl++) {
      if (symmetric) m5_si_grow<<<152 * 16, 128, 0, st>>>(m, lvl, SI, list[(lvl - 1) & 1], list[lvl & 1], count);
      else m5_si_layer<<<gc, 128, 0, st>>>(m, lvl, SI);
    }
  } else {
    cudaMemsetAsync(SI, 0, sizeof(W) * m.n, st);
  }
  m5_tag_split<<<gc, 128, 0, st>>>(m, t, x, SI, split);
}
}  // namespace

void ffv_m5_tags(const ffv_dmesh &m, const M5Consts &k, const ffv_m5_tagc &t, bool symmetric,
                 const double *S, void *SI, bool wide, int32_t *lists, int32_t *split, double *pr,
                 cudaStream_t st) {
  if (wide) tags_impl(m, k, t, symmetric, S, static_cast<unsigned long long *>(SI), lists, split, pr, st);
  else tags_impl(m, k, t, symmetric, S, static_cast<uint32_t *>(SI), lists, split, pr, st);
}

void ffv_m5_si_unpack(int64_t n, const void *SI, bool wide, int32_t *out, cudaStream_t st) {
  const unsigned g = (unsigned)((n + 255) / 256);
  if (wide) m5_si_unpack<<<g, 256, 0, st>>>(n, static_cast<const unsigned long long *>(SI), out);
  else m5_si_unpack<<<g, 256, 0, st>>>(n, static_cast<const uint32_t *>(SI), out);
}

void ffv_m5_cfl(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k, const double *S,
                unsigned long long *d_out, cudaStream_t st) {
  if (k.nmat == 2) m5_cfl_kernel<2><<<152 * 4, 128, 0, st>>>(m, g, k, S, d_out);
  else m5_cfl_kernel<3><<<152 * 4, 128, 0, st>>>(m, g, k, S, d_out);
}

int ffv_m5_neq(int nmat) { return 3 * nmat + 12; }

struct Rec {
  cudaEvent_t *ev;
  int i;
  const char **names;
  cudaStream_t st;
  void operator()(const char *name) {
    if (ev) {
      names[i] = name;
      cudaEventRecord(ev[++i], st);
    }
  }
};

template <int N>
static void stage_impl(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k,
                       const ffv_m5_bufs &b, int irk, bool follows, cudaStream_t st,
                       cudaEvent_t *ev, const char **names) {
  const int tpb = 128;
  const unsigned gc = (unsigned)((m.n + tpb - 1) / tpb);
  Rec rec{ev, 0, names, st};
  if (ev) cudaEventRecord(ev[0], st);
  const bool f32 = k.precision == FFV_FP32_FLUX, fast = k.flux_form == FFV_FLUX_CONSISTENT;
  // the FP32 form keeps its face states and fluxes in the same buffers, as floats
  float *SFf = (float *)b.SF, *FFf = (float *)b.FF, *UFf = (float *)b.UF;
  if (k.order == 2) {
    if (f32) {
      // the FP32 copy of the state lives in RHS, which m5_cell_update writes later
      ffv_m5f_shadow(m.n, k, b.S, (float *)b.RHS, b.flat, follows, st);
      rec("m5f_shadow");
      ffv_m5f_recon(m, g, k, (float *)b.RHS, b.flat, SFf, b.status, st);
      rec("m5f_recon_face");
    } else {
      m5_recon_slopes<N><<<dim3(gc, 3), tpb, 0, st>>>(m, g, k, b.S, b.SF);
      rec("m5_recon_slopes");
      (fast ? m5_relax_faces<N, true> : m5_relax_faces<N, false>)<<<dim3(gc, 6), tpb, 0, st>>>(
          m.n, k, b.SF, b.status);
      rec("m5_relax_faces");
    }
  }
  if (f32)
    ffv_m5f_flux(m, g, k, b.S, k.order == 2 ? (const float *)b.RHS : nullptr, SFf, b.flat, FFf, UFf,
                 b.GF, b.list_faces, b.status, st);
  else
    (k.order == 2 ? m5_face_flux<N, 2> : m5_face_flux<N, 1>)
        <<<ffv_flux_blocks(b.list_faces, m.n), FFV_LIST_TPB, 0, st>>>(
            m, g, k, b.list_faces, b.S, b.SF, b.FF, b.UF, b.GF, b.status);
  rec(f32 ? "m5f_face_flux" : "m5_face_flux");
  if (f32)
    ffv_m5f_cell_update(m, g, k, b.S, b.SN, FFf, UFf, b.GF, b.flat, b.RHS, b.Snew, b.flag, b.list,
                        b.dt, irk, b.status, st);
  else
    m5_cell_update<N><<<gc, tpb, 0, st>>>(m, g, k, b.S, b.SN, b.FF, b.UF, b.RHS, b.Snew,
                                          b.flag, b.list, b.dt, irk, b.status);
  rec(f32 ? "m5f_cell_update" : "m5_cell_update");
  if (irk == 1) {
    m5_gfm_seq<N><<<FFV_GFM_PARTS, GFM_TPB, 0, st>>>(m, g, k, b.flag, b.list, b.list_parts, b.S, b.Snew,
                                                     b.SN, b.RHS, b.GF, b.dt, 0);
    rec("m5_gfm_seq");
  }
  if (f32) ffv_m5f_relax_cell(m.n, k, b.Snew, b.flat, b.S, b.flag, b.list, b.status, st);
  else
    (fast ? m5_relax_cell<N, true> : m5_relax_cell<N, false>)<<<gc, tpb, 0, st>>>(
        m.n, k, b.Snew, b.S, b.flag, b.list, b.status);
  rec(f32 ? "m5f_relax_cell" : "m5_relax_cell");
  // relaxed states are in S; a later neighbour is still unrelaxed (Snew)
  m5_gfm_seq<N><<<FFV_GFM_PARTS, GFM_TPB, 0, st>>>(m, g, k, b.flag, b.list, b.list_parts, b.Snew, b.S,
                                                   b.SN, b.RHS, b.GF, b.dt, 1);
  rec("m5_gfm_seq(relax)");
}

void ffv_m5_fp64_stage(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k,
                       const ffv_m5_bufs &b, int irk, bool follows, cudaStream_t st,
                       cudaEvent_t *ev, const char **names) {
  if (k.nmat == 2) stage_impl<2>(m, g, k, b, irk, follows, st, ev, names);
  else stage_impl<3>(m, g, k, b, irk, follows, st, ev, names);
}

int ffv_m5_launches_per_stage(const M5Consts &k, int irk) {
  const int recon = k.order == 2 ? 2 : 0;
  return recon + 2 + (irk == 1 ? 1 : 0) + 2;
}

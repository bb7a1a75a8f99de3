// Model-0 (Euler, stiffened gas) FP64 stage kernels.
//
// Compiled with --fmad=false: every multiply and add rounds separately, in the operation
// order of the reference's C code, so results are bit-identical to the reference
// (m0_*.c) on Cartesian forests.  Face frames are axis-aligned there, so the rotations of
// m0_wave_speeds.c:16-28 / m0_star_region.c:27-30 reduce to picking a component with a
// sign; that is exact (the other terms are products with 0.0).
//
// Per stage three kernels run:
//   m0_recon      grad_scheme -> m0_faceinterp_V1 (m0_faceinterp.c:59-88): limited face states
//                 SF of every cell, one thread per cell and axis;
//   m0_face_flux  the HLLC flux of every face between two cells of one level, once, from the
//                 side of the cell that comes first in leaf order (m0_residual.c:112-129 reuses
//                 that flux for the other side); it overwrites the first cell's face state,
//                 which nothing else reads;
//   m0_update     RHS -> m0_residual (m0_residual.c:7-141) fused with the RK stage update
//                 (RK.c:3-53): each cell gathers its own faces' fluxes (no atomics), negated
//                 where the other side evaluated them, and evaluates its boundary, coarser and
//                 finer faces itself.
// The stage is bound by the FP64 pipe (ffv_fp64.cuh).
#include <math.h>

#include "ffv_device.cuh"
#include "ffv_fp64.cuh"

namespace {

constexpr int NV = 5;

// gamma - 1, gamma and the pressure constants of the stiffened gas
struct Gas {
  double gamma, gm1, pinf, gpi;
};

struct Sol {
  double r, u, v, w, e, er, p, c;  // er = e / r
  double vec[NV];
};

// m0_facercnstr.c:29-43: face state vector -> primitive state; the five quotients by the density
// share its reciprocal
__device__ __forceinline__ void to_sol(const double U[NV], const Gas &k, Sol &s) {
  s.r = U[0];
  const f64::Rcp r = f64::rcp(s.r);
  s.u = f64::div(U[1], r);
  s.v = f64::div(U[2], r);
  s.w = f64::div(U[3], r);
#pragma unroll
  for (int i = 0; i < NV; i++) s.vec[i] = U[i];
  s.e = U[4];
  s.er = f64::div(s.e, r);
  double ei = s.er - 0.5 * (s.u * s.u + s.v * s.v + s.w * s.w);
  s.p = s.r * k.gm1 * ei - k.gpi;
  s.c = sqrt(f64::div(k.gamma * (s.p + k.pinf), r));
}

template <int A>
__device__ __forceinline__ double vc(const Sol &s) {
  return A == 0 ? s.u : (A == 1 ? s.v : s.w);
}
template <int S>
__device__ __forceinline__ double sgn(double x) {
  return S > 0 ? x : -x;
}
// components of the velocity in the frame of face F (m0_wave_speeds.c:21-35)
template <int F> __device__ __forceinline__ double rot_n(const Sol &s) { return sgn<fr_n_sign(F)>(vc<fr_n_axis(F)>(s)); }
template <int F> __device__ __forceinline__ double rot_t1(const Sol &s) { return sgn<fr_t1_sign(F)>(vc<fr_t1_axis(F)>(s)); }
template <int F> __device__ __forceinline__ double rot_t2(const Sol &s) { return sgn<fr_t2_sign(F)>(vc<fr_t2_axis(F)>(s)); }
// global component A of a*n + b*t1 + c*t2 (m0_star_region.c:27-29, bc_reflective.c:26-28)
template <int F, int A>
__device__ __forceinline__ double unrot(double a, double b, double c) {
  return fr_n_axis(F) == A ? sgn<fr_n_sign(F)>(a)
                           : (fr_t1_axis(F) == A ? sgn<fr_t1_sign(F)>(b) : sgn<fr_t2_sign(F)>(c));
}

// m0_bc.c:3-31: ghost state of a boundary face; only the velocity changes
// (bc_reflective.c for 1 and 4, bc_wall.c for 5).
template <int F>
__device__ __forceinline__ void ghost(const Sol &L, int bc, Sol &R) {
  R = L;
  if (bc == 1 || bc == 4 || bc == 5) {
    double ul = rot_n<F>(L), vl = rot_t1<F>(L), wl = rot_t2<F>(L);
    double ur = -ul, vr = bc == 5 ? -vl : vl, wr = bc == 5 ? -wl : wl;
    R.u = unrot<F, 0>(ur, vr, wr);
    R.v = unrot<F, 1>(ur, vr, wr);
    R.w = unrot<F, 2>(ur, vr, wr);
  }
}

// m0_flux.c:3-28, normal component along face F: sum_d F[i][d] n_d
template <int F>
__device__ __forceinline__ void flux_n(const Sol &s, double Fn[NV]) {
  constexpr int a = fr_n_axis(F);
  const double va = vc<a>(s);
  Fn[0] = sgn<fr_n_sign(F)>(va * s.r);
  Fn[1] = sgn<fr_n_sign(F)>(a == 0 ? s.r * s.u * s.u + s.p : s.r * s.u * va);
  Fn[2] = sgn<fr_n_sign(F)>(a == 1 ? s.r * s.v * s.v + s.p : s.r * s.v * va);
  Fn[3] = sgn<fr_n_sign(F)>(a == 2 ? s.r * s.w * s.w + s.p : s.r * s.w * va);
  Fn[4] = sgn<fr_n_sign(F)>(va * (s.e + s.p));
}

// m0_star_region.c:3-31
template <int F>
__device__ __forceinline__ void star(const Sol &s, double S_S, double SK, double uK, double vK,
                                     double wK, double Us[NV]) {
  const double d = SK - uK, rd = s.r * d;
  double const_S = rd / (SK - S_S);
  Us[0] = const_S;
  Us[1] = const_S * unrot<F, 0>(S_S, vK, wK);
  Us[2] = const_S * unrot<F, 1>(S_S, vK, wK);
  Us[3] = const_S * unrot<F, 2>(S_S, vK, wK);
  Us[4] = const_S * (s.er + (S_S - uK) * (S_S + (s.p / rd)));
}

// m0_hllc.c:3-59 with m0_wave_speeds.c:3-135, accumulated as m0_residual.c:178-184:
// ff[i] += -(A) * (F.n + HLLC correction).  Returns status bits.  The four branches share one
// star region and one physical flux, evaluated on the state of the contact's upwind side (the
// branches of one warp would otherwise run one after the other).
template <int F>
__device__ __forceinline__ unsigned hllc_acc(const Sol &L, const Sol &R, bool bc4, double A,
                                             double ff[NV]) {
  double uL = rot_n<F>(L), vL = rot_t1<F>(L), wL = rot_t2<F>(L);
  double uR = rot_n<F>(R), vR = rot_t1<F>(R), wR = rot_t2<F>(R);
  double ruL = L.r * uL, ruR = R.r * uR;
  double a = uL + L.c, b = uR + R.c;
  double SR = (a > b) ? a : b;
  a = uL - L.c;
  b = uR - R.c;
  double SL = (a < b) ? a : b;
  // s11 of the rotated stress tensor p I is p (rotate_vectors.c:73-106, unit normal)
  double S_S = ((L.r * (uL * uL) + L.p) - (R.r * (uR * uR) + R.p) - (SL * ruL) + (SR * ruR)) /
               (ruL - ruR - (SL * L.r) + (SR * R.r));
  unsigned st = f64::is_nan(S_S) ? FFV_ST_NAN_SPEED : 0u;
  if (bc4) S_S = 0.0;
  // 0: supersonic from the left, 1: left star state, 2: right star state, 3: supersonic from
  // the right
  const int branch = f64::ge0(SL) ? 0
                     : (f64::le0(SL) && f64::ge0(S_S)) ? 1
                     : (f64::le0(S_S) && f64::ge0(SR)) ? 2
                     : f64::le0(SR) ? 3 : -1;
  double Fn[NV] = {0.0, 0.0, 0.0, 0.0, 0.0}, corr[NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (branch < 0) {
    st |= FFV_ST_NO_BRANCH;
  } else {
    const bool left = branch <= 1;
    Sol K;
    K.r = left ? L.r : R.r;
    K.u = left ? L.u : R.u;
    K.v = left ? L.v : R.v;
    K.w = left ? L.w : R.w;
    K.e = left ? L.e : R.e;
    K.er = left ? L.er : R.er;
    K.p = left ? L.p : R.p;
    flux_n<F>(K, Fn);
    if (branch == 1 || branch == 2) {
      const double SK = left ? SL : SR;
      double Us[NV];
      star<F>(K, S_S, SK, left ? uL : uR, left ? vL : vR, left ? wL : wR, Us);
#pragma unroll
      for (int i = 0; i < NV; i++) corr[i] = SK * (Us[i] - (left ? L.vec[i] : R.vec[i]));
    }
  }
#pragma unroll
  for (int i = 0; i < NV; i++) ff[i] += -(A) * (Fn[i] + corr[i]);
  return st;
}

// Face-state access: ORDER 2 reads SF[f][v][c]; ORDER 1 reads a stage-start copy of S, which
// m0_copy_state put into the first face's slots.
template <int ORDER>
__device__ __forceinline__ void load_face(const double *__restrict__ FS, int64_t n, int f,
                                          int64_t c, double U[NV]) {
#pragma unroll
  for (int v = 0; v < NV; v++)
    U[v] = ORDER == 2 ? FS[((int64_t)f * NV + v) * n + c] : FS[(int64_t)v * n + c];
}

// The flux of the positive face of one axis (blockIdx.y) of every cell with a neighbour of its
// own level there, into that face's slots of SF: five values over the cell's own face state,
// which this thread alone reads (order 1: over slots that hold nothing).  About 190 FP64
// instructions per face, the FP64 pipe 83 % busy: 43 us per stage at 32,768 cells, 457 us at
// 465,704, and m0_update 29 and 406 us; evaluating each such face from both sides in one kernel
// with the update took 1770 per cell, 150 and 2926 us.
template <int ORDER, int F>
__device__ __forceinline__ void owner_flux(const ffv_dmesh &m, const ffv_geom &g, double *SF,
                                           int64_t c, uint32_t info, const Gas &k,
                                           unsigned *status) {
  if (ffv_face_kind(info, F) != FFV_FK_SAME) return;
  const int64_t o = m.nbr[(int64_t)F * m.n + c];
  if (o < c) return;
  double U[NV], ff[NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
  Sol L, R;
  load_face<ORDER>(SF, m.n, F, c, U);
  to_sol(U, k, L);
  load_face<ORDER>(SF, m.n, fr_opp(F), o, U);
  to_sol(U, k, R);
  const unsigned st = hllc_acc<F>(L, R, false, g.area[ffv_info_level(info)], ff);
#pragma unroll
  for (int v = 0; v < NV; v++) SF[((int64_t)F * NV + v) * m.n + c] = ff[v];
  if (st) atomicOr(status, st);
}

template <int ORDER>
__global__ void __launch_bounds__(128) m0_face_flux(ffv_dmesh m, ffv_geom g, double *SF, Gas k,
                                                    unsigned *__restrict__ status) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  const uint32_t info = m.info[c];
  if (blockIdx.y == 0) owner_flux<ORDER, owner_face(0)>(m, g, SF, c, info, k, status);
  else if (blockIdx.y == 1) owner_flux<ORDER, owner_face(1)>(m, g, SF, c, info, k, status);
  else owner_flux<ORDER, owner_face(2)>(m, g, SF, c, info, k, status);
}

constexpr int UPD = 128;  // threads of an update block

// work space of one face direction of an update block: the boundary, coarser and finer faces of
// its cells (four items for a finer face), compacted, and their fluxes
struct FaceItems {
  uint16_t item[4 * UPD];  // thread of the cell | subface << 8
  double flux[NV][4 * UPD];
  int warp_total[UPD / 32];
};

// Face F's residual of every cell of the block: the flux m0_face_flux left, its neighbour's
// negated, or an evaluation here of a boundary, coarser or finer face.  Such faces are a few per
// warp on a refined mesh, so a warp that evaluated its own would run the whole solver for one or
// two lanes: the block lists them and evaluates the list with full warps (465,704 cells: 989 to
// 406 us per stage).
template <int ORDER, int F>
__device__ __forceinline__ void block_residual(const ffv_dmesh &m, const ffv_geom &g,
                                               const double *__restrict__ FS, int64_t c,
                                               uint32_t info, const Gas &k, FaceItems &sh,
                                               unsigned &st, double rhs[NV]) {
  constexpr int FO = fr_opp(F);
  const bool live = c < m.n;
  const uint32_t kind = ffv_face_kind(info, F);
  const int cnt = !live || kind == FFV_FK_SAME ? 0 : (kind == FFV_FK_FINER ? 4 : 1);
  double ff[NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (live && cnt == 0) {
    const int64_t o = m.nbr[(int64_t)F * m.n + c];
    const bool own = o > c;
    const double *f = FS + (int64_t)(own ? F : FO) * NV * m.n + (own ? c : o);
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const double t = f[(int64_t)i * m.n];
      ff[i] = own ? t : f64::neg(t);
    }
  }
  if (__syncthreads_or(cnt)) {
    const unsigned before = (1u << (threadIdx.x & 31)) - 1u;
    const unsigned one = __ballot_sync(0xffffffffu, cnt == 1), four = __ballot_sync(0xffffffffu, cnt == 4);
    if ((threadIdx.x & 31) == 0) sh.warp_total[threadIdx.x >> 5] = __popc(one) + 4 * __popc(four);
    __syncthreads();
    int at = __popc(one & before) + 4 * __popc(four & before), total = 0;
#pragma unroll
    for (int w = 0; w < UPD / 32; w++) {
      if (w < (int)(threadIdx.x >> 5)) at += sh.warp_total[w];
      total += sh.warp_total[w];
    }
    for (int q = 0; q < cnt; q++) sh.item[at + q] = (uint16_t)(threadIdx.x | (q << 8));
    __syncthreads();
    for (int i = threadIdx.x; i < total; i += UPD) {
      const int64_t ci = c - threadIdx.x + (sh.item[i] & 255);
      const uint32_t in = m.info[ci], ki = ffv_face_kind(in, F);
      const int l = ffv_info_level(in);
      double U[NV], t[NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
      Sol L, R;
      load_face<ORDER>(FS, m.n, F, ci, U);
      to_sol(U, k, L);
      const int bc = (ki & FFV_FK_BC) ? (int)(ki & 7u) : 0;
      if (bc) {
        ghost<F>(L, bc, R);
      } else {
        const int64_t s = m.nbr[(int64_t)F * m.n + ci];
        load_face<ORDER>(FS, m.n, FO, ki == FFV_FK_FINER ? m.sub[4 * s + (sh.item[i] >> 8)] : s, U);
        to_sol(U, k, R);
      }
      st |= hllc_acc<F>(L, R, bc == 4, g.area[ki == FFV_FK_FINER ? l + 1 : l], t);
#pragma unroll
      for (int v = 0; v < NV; v++) sh.flux[v][i] = t[v];
    }
    __syncthreads();
    for (int q = 0; q < cnt; q++)
#pragma unroll
      for (int v = 0; v < NV; v++) ff[v] += sh.flux[v][at + q];
  }
#pragma unroll
  for (int i = 0; i < NV; i++) rhs[i] += ff[i];
}

template <int ORDER>
__global__ void __launch_bounds__(UPD) m0_update(ffv_dmesh m, ffv_geom g,
                                                 const double *__restrict__ FS,
                                                 double *__restrict__ S, double *__restrict__ SN,
                                                 const double *__restrict__ dtp, Gas gas, int irk,
                                                 unsigned *__restrict__ status) {
  __shared__ FaceItems sh;
  const int64_t c = (int64_t)blockIdx.x * UPD + threadIdx.x;
  const uint32_t info = c < m.n ? m.info[c] : 0u;
  const int l = ffv_info_level(info);
  double rhs[NV] = {0.0, 0.0, 0.0, 0.0, 0.0};
  unsigned st = 0;
  block_residual<ORDER, 0>(m, g, FS, c, info, gas, sh, st, rhs);
  block_residual<ORDER, 1>(m, g, FS, c, info, gas, sh, st, rhs);
  block_residual<ORDER, 2>(m, g, FS, c, info, gas, sh, st, rhs);
  block_residual<ORDER, 3>(m, g, FS, c, info, gas, sh, st, rhs);
  block_residual<ORDER, 4>(m, g, FS, c, info, gas, sh, st, rhs);
  block_residual<ORDER, 5>(m, g, FS, c, info, gas, sh, st, rhs);
  if (c >= m.n) {
    if (st) atomicOr(status, st);
    return;
  }
  // a non-positive density in the stage's input (the reference runs on into a NaN sound
  // speed there); the status word reports it, the arithmetic is untouched
  if (f64::le0(S[c])) st |= FFV_ST_NEG_DENSITY;
#pragma unroll
  for (int i = 0; i < NV; i++)
    if (f64::is_nan(rhs[i])) st |= FFV_ST_NAN;
  // RK.c:21-45 (stage 1 also performs RK(0): SN = S, RK.c:17-20)
  const double dt = *dtp, iV = g.inv_vol[l];
  const f64::Rcp V{g.vol[l], iV};
#pragma unroll
  for (int e = 0; e < NV; e++) {
    const int64_t k = (int64_t)e * m.n + c;
    const double s = S[k];
    double out;
    if (irk == 1) {
      SN[k] = s;
      out = s - dt * iV * rhs[e];
    } else {
      const double sn = SN[k];
      if (irk == 2)
        out = (3.0 / 4.0) * sn + (1.0 / 4.0) * s - f64::div((1.0 / 4.0) * dt * rhs[e], V);
      else if (irk == 3)
        out = (1.0 / 3.0) * sn + (2.0 / 3.0) * s - f64::div((2.0 / 3.0) * dt * rhs[e], V);
      else
        out = (1.0 / 2.0) * sn + (1.0 / 2.0) * s - f64::div((1.0 / 2.0) * dt * rhs[e], V);
    }
    S[k] = out;
    if (e == 0 && f64::le0(out)) st |= FFV_ST_NEG_DENSITY;
  }
  if (st) atomicOr(status, st);
}

// m0_facevalues_MUSCL.c:3-56 (iside 1): value across face F
template <int F>
__device__ __forceinline__ void across(const ffv_dmesh &m, const double *__restrict__ S,
                                       int64_t c, uint32_t info, const double Sc[NV],
                                       double out[NV]) {
  const uint32_t kind = ffv_face_kind(info, F);
  if (kind & FFV_FK_BC) {
#pragma unroll
    for (int v = 0; v < NV; v++) out[v] = Sc[v];
  } else if (kind == FFV_FK_FINER) {
    const int32_t *sg = m.sub + 4 * (int64_t)m.nbr[(int64_t)F * m.n + c];
    const int64_t s0 = sg[0], s1 = sg[1], s2 = sg[2], s3 = sg[3];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const double *Sv = S + (int64_t)v * m.n;
      double a = 0.0;
      a += Sv[s0] / 4.0;
      a += Sv[s1] / 4.0;
      a += Sv[s2] / 4.0;
      a += Sv[s3] / 4.0;
      out[v] = a;
    }
  } else {
    const int64_t o = m.nbr[(int64_t)F * m.n + c];
#pragma unroll
    for (int v = 0; v < NV; v++) out[v] = S[(int64_t)v * m.n + o];
  }
}

// m0_deltavalues.c:23-57 + m0_reconctruct.c:160-207 for the two faces of one axis: both limited
// increments come from the same two one-sided slopes.  Between neighbours of the cell's own
// level at a power-of-two spacing the whole limiter is integer work (f64::minmod_pair); other
// faces take the reference's quotients.  One thread per cell and axis (blockIdx.y): the FP64
// work is 4 instructions per variable and axis there, against 57 with four divisions per face
// (per stage at 32,768 cells 83 to 15 us, at 465,704 cells 865 to 262 us).
template <int FA, int FB>
__device__ __forceinline__ void recon_axis(const ffv_dmesh &m, const ffv_geom &g,
                                           const double *__restrict__ S, double *__restrict__ SF,
                                           int64_t c) {
  static_assert(fr_opp(FA) == FB, "opposite faces");
  const uint32_t info = m.info[c];
  const int l = ffv_info_level(info);
  double Sc[NV], XA[NV], XB[NV], cA[NV], cB[NV];
#pragma unroll
  for (int v = 0; v < NV; v++) Sc[v] = S[(int64_t)v * m.n + c];
  across<FA>(m, S, c, info, Sc, XA);
  across<FB>(m, S, c, info, Sc, XB);
  const uint32_t ka = ffv_face_kind(info, FA), kb = ffv_face_kind(info, FB);
  if ((ka | kb) & FFV_FK_BC) {
    // no slope next to a boundary: its own face has none, and the opposite face's one-sided
    // slope across the boundary is 0 / 0
#pragma unroll
    for (int v = 0; v < NV; v++) cA[v] = cB[v] = 0.0;
  } else if (ka == FFV_FK_SAME && kb == FFV_FK_SAME && ((g.pow2 >> l) & 1u)) {
    const double ih = g.rdcc[l][0];
#pragma unroll
    for (int v = 0; v < NV; v++) f64::minmod_pair(XA[v] - Sc[v], XB[v] - Sc[v], ih, cA[v], cB[v]);
  } else {
    const f64::Rcp da{g.dcc[l][face_class(ka)], g.rdcc[l][face_class(ka)]};
    const f64::Rcp db{g.dcc[l][face_class(kb)], g.rdcc[l][face_class(kb)]};
    const double fa = g.dcf[l][face_class(ka)], fb = g.dcf[l][face_class(kb)];
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const double dA = XA[v] - Sc[v], dB = XB[v] - Sc[v];
      const double a = f64::div(dA, da), b = f64::div(dB, db);
      const bool opposed = f64::gt0(-b * a);
      const double ga = f64::abs_gt(b, a) ? a : f64::neg(b), gb = f64::abs_gt(a, b) ? b : f64::neg(a);
      cA[v] = fa * (opposed && f64::abs_gt(dA, 1e-10) ? ga : 0.0);
      cB[v] = fb * (opposed && f64::abs_gt(dB, 1e-10) ? gb : 0.0);
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    SF[((int64_t)FA * NV + v) * m.n + c] = Sc[v] + cA[v];
    SF[((int64_t)FB * NV + v) * m.n + c] = Sc[v] + cB[v];
  }
}

__global__ void __launch_bounds__(128) m0_recon(ffv_dmesh m, ffv_geom g,
                                                const double *__restrict__ S,
                                                double *__restrict__ SF) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.n) return;
  if (blockIdx.y == 0) recon_axis<0, 2>(m, g, S, SF, c);
  else if (blockIdx.y == 1) recon_axis<3, 1>(m, g, S, SF, c);
  else recon_axis<4, 5>(m, g, S, SF, c);
}

__global__ void m0_copy_state(int64_t count, const double *__restrict__ S, double *__restrict__ D) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    D[i] = S[i];
}

}  // namespace

int ffv_m0_launches_per_stage(int order) { return 3; (void)order; }

const char *ffv_m0_fp64_kernel_name(int order, int i) {
  static const char *o2[3] = {"m0_recon", "m0_face_flux<2>", "m0_update<2>"};
  static const char *o1[3] = {"m0_copy_state", "m0_face_flux<1>", "m0_update<1>"};
  if (i < 0 || i > 2) return "";
  return order == 2 ? o2[i] : o1[i];
}

template <int ORDER>
static void m0_stage(const ffv_dmesh &m, const ffv_geom &g, const ffv_m0_bufs &b, const Gas &gas,
                     int irk, cudaStream_t st, cudaEvent_t *ev) {
  const int tpb = 128;
  const unsigned blocks = (unsigned)((m.n + tpb - 1) / tpb);
  if (ev) cudaEventRecord(ev[0], st);
  if (ORDER == 2) m0_recon<<<dim3(blocks, 3), tpb, 0, st>>>(m, g, b.S, b.SF);
  else m0_copy_state<<<1024, 256, 0, st>>>(NV * m.n, b.S, b.SF);
  if (ev) cudaEventRecord(ev[1], st);
  m0_face_flux<ORDER><<<dim3(blocks, 3), tpb, 0, st>>>(m, g, b.SF, gas, b.status);
  if (ev) cudaEventRecord(ev[2], st);
  m0_update<ORDER><<<blocks, tpb, 0, st>>>(m, g, b.SF, b.S, b.SN, b.dt, gas, irk, b.status);
  if (ev) cudaEventRecord(ev[3], st);
}

void ffv_m0_fp64_stage(const ffv_dmesh &m, const ffv_geom &g, const ffv_m0_bufs &b,
                       const ffv_m0_consts &k, int irk, cudaStream_t st, cudaEvent_t *ev) {
  const Gas gas{k.gamma, k.gamma - 1.0, k.pinf, k.gamma * k.pinf};
  if (k.order == 2) m0_stage<2>(m, g, b, gas, irk, st, ev);
  else m0_stage<1>(m, g, b, gas, irk, st, ev);
}

// Model-5 launch interface (ffv_m5_fp64.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ffv_device.cuh"
#include "ffv_df.cuh"

struct M5Consts {
  int nmat, order, prelax, nsolids;
  int precision;  // FFV_FP64 or FFV_FP32_FLUX
  int flux_form;  // FFV_FLUX_REFERENCE or FFV_FLUX_CONSISTENT
  int zerou[3];
  double gamma[FFV_MAX_MATERIALS], pinf[FFV_MAX_MATERIALS], mu[FFV_MAX_MATERIALS];
  double amin, avf_lim;
  double yield[FFV_MAX_MATERIALS];  // von Mises yield stress per material, 0 = none
  int plastic;                      // a solid material has a yield stress
  // per material, for the FP32-flux form: gamma p_inf, 1 / (gamma - 1),
  // gamma p_inf / (gamma - 1), 1 / gamma
  double gpi[FFV_MAX_MATERIALS], ig1[FFV_MAX_MATERIALS], gpg[FFV_MAX_MATERIALS],
      igam[FFV_MAX_MATERIALS];
  // FP64 form: gamma - 1, the relaxation's pressure floor -(1 - 1e-8) p_inf + 1e-8 and reset value,
  // AMIN / 100 and 1 - AMIN / 100, and the binomial coefficients of (1 + t)^(1 / gamma), t^1..t^10
  double gm1[FFV_MAX_MATERIALS], pfloor[FFV_MAX_MATERIALS], preset[FFV_MAX_MATERIALS];
  double lo, hi;
  double binom[3][10];
  // the same in FP32: p_inf, 1 / gamma, mu, gamma, the relaxation's pressure floor and reset
  // value, AMIN / 100 and 1 - AMIN / 100
  float pinf_f[FFV_MAX_MATERIALS], igam_f[FFV_MAX_MATERIALS], mu_f[FFV_MAX_MATERIALS],
      gamma_f[FFV_MAX_MATERIALS], plo_f[FFV_MAX_MATERIALS], preset_f[FFV_MAX_MATERIALS];
  float alo_f, ahi_f;
  // AVF_LIM in FP32, and whether phi0 takes the larger of two solid fractions (two solids,
  // the first one elastic): the FP32-flux form's phi0 needs no FP64 instruction
  float avf_lim_f;
  int phi_pair;
  // (a - j) / (j + 1), j = 1..6, a = -1 / gamma: the FP32 Newton iteration's binomial series
  float bin_f[FFV_MAX_MATERIALS][6];
  // double-float pairs for the FP32-flux form's pressure recovery: gamma - 1, gamma p_inf,
  // 1 / (gamma - 1), gamma p_inf / (gamma - 1), p_inf, the relaxation's pressure floor; and
  // AMIN / 100, 1 - AMIN / 100, 1 - 2 AMIN / 100, 1e-12, 1 - 1e-12
  df gm1_d[FFV_MAX_MATERIALS], gpi_d[FFV_MAX_MATERIALS], ig1_d[FFV_MAX_MATERIALS],
      gpg_d[FFV_MAX_MATERIALS], pinf_d[FFV_MAX_MATERIALS], floor_d[FFV_MAX_MATERIALS];
  df alo_d, ahi_d, a2lo_d, eps_d, oneeps_d;
};

// bits of a face's mark (GF): a ghost-fluid face; its deformation flux is stored (FP32-flux form)
#define FFV_FACE_GFM 1
#define FFV_FACE_DEFORMS 2

// FP32-flux form: flat cells and face states, whose deformation is zero and kept nowhere but in S
struct FlatMarks {
  uint8_t *cell;  // [n]: the stage's input state
  uint8_t *next;  // [n]: the state the cell update made (before it: this one's calm cells)
  uint8_t *base;  // [n]: SN (its deformation is then not stored)
  uint8_t *face;  // [6][n]: face states
};

// blocks of a ghost-fluid pass, where many cells are flagged (m5_gfm_seq)
#define FFV_GFM_PARTS 16

struct ffv_m5_bufs {
  double *S, *SN, *Snew, *SF, *FF, *UF, *RHS, *dt;
  uint8_t *GF, *flag;  // GF [6][n]: marks of faces, as the cell that evaluates the face sees them
  FlatMarks flat;
  // [1 + n]: the number of cells the last pass flagged, then the cells; list_parts [FFV_GFM_PARTS + 1]:
  // the number of them in each block's run of cells, and the blocks that have finished (0 between passes)
  int32_t *list, *list_parts;
  unsigned int *status;
  ffv_face_list list_faces;
};

int ffv_m5_neq(int nmat);
// ev (nullable): an event before the first and after every kernel; names[i] receives
// kernel i's name.  follows: the stage before ran on this state and nothing else has touched it.
void ffv_m5_fp64_stage(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k,
                       const ffv_m5_bufs &b, int irk, bool follows, cudaStream_t st,
                       cudaEvent_t *ev, const char **names);
int ffv_m5_launches_per_stage(const M5Consts &k, int irk);

// FP32-flux form (ffv_m5_fp32.cu): face states and face fluxes in FP32.
//   Sf:  [neq][n] float copy of the state, made by ffv_m5f_shadow (scratch)
//   SFf: [6][neq + 2][n] float -- the reconstructed, relaxed face state followed by the last
//        volume fraction and the relaxed pressure
//   FFf: [6][neq][n] float face fluxes (area-weighted), UFf: [6][3][n] float face velocity
// known: the marks of the previous stage's cell update hold for S
void ffv_m5f_shadow(int64_t n, const M5Consts &k, const double *S, float *Sf, const FlatMarks &fm,
                    bool known, cudaStream_t st);
void ffv_m5f_recon(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k, const float *Sf,
                   const FlatMarks &fm, float *SFf, unsigned *status, cudaStream_t st);
// Sf: the FP32 copy of the state (order 2), or nullptr (order 1: phi0 from S)
void ffv_m5f_flux(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k, const double *S,
                  const float *Sf, const float *SFf, const FlatMarks &fm, float *FFf, float *UFf,
                  uint8_t *GF, const ffv_face_list &fl, unsigned *status, cudaStream_t st);
// residual + RK stage of the FP32-flux form (the face fluxes of all but the deformation summed as
// double-float pairs)
void ffv_m5f_cell_update(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k, const double *S,
                         double *SN, const float *FFf, const float *UFf, const uint8_t *GF,
                         const FlatMarks &fm, double *RHS, double *Snew, uint8_t *flag,
                         int32_t *list, const double *dt, int irk, unsigned *status,
                         cudaStream_t st);
// where the indicator's fields of a cell go: F [5][n], or, with R, one 16-byte record [n] of the five
// normalised by norm (means, standard deviations) and rounded to BF16, as the perceptron takes them
struct ffv_field_out {
  float *F;
  uint4 *R;
  const float *norm;
  __device__ __forceinline__ void put(int64_t n, int64_t c, const float f[5]) const {
    if (!R) {
#pragma unroll
      for (int q = 0; q < 5; q++) F[q * n + c] = f[q];
      return;
    }
    uint32_t h[5];
#pragma unroll
    for (int q = 0; q < 5; q++)
      h[q] = __bfloat16_as_ushort(__float2bfloat16_rn((f[q] - norm[q]) * (1.0f / norm[5 + q])));
    R[c] = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4], 0u);
  }
};
// the indicator's fields of a model-5 state (log rho, log p, alpha_0, |u|, von Mises stress; FP32
// with double-float pressure recovery; ffv_mlp.cu gathers them)
void ffv_m5f_indicator_fields(int64_t n, const M5Consts &k, const double *S, const ffv_field_out &out,
                              cudaStream_t st);
// cell pressure relaxation: the Newton iteration in FP32, the pressure recovery and the
// energy-consistent pressure and internal energies in double-float
void ffv_m5f_relax_cell(int64_t n, const M5Consts &k, const double *Sin, const FlatMarks &fm,
                        double *Sout, uint8_t *flag, int32_t *list, unsigned *status,
                        cudaStream_t st);
void ffv_m5_cfl(const ffv_dmesh &m, const ffv_geom &g, const M5Consts &k, const double *S,
                unsigned long long *d_out, cudaStream_t st);

// refinement criteria (criterionsplt.c, interface_location.c) with the derived values the
// reference forms from its input (m5_input.c:50-57): lrs1 = lrs0 + lrs1 as given,
// si_max = ADAPT_INTER_MAX
struct ffv_m5_tagc {
  int uniform, lvl_uniform, prs, lvl_prs, rho, lvl_rho, vel, lvl_vel;
  int inter0, lvl0, lrs0, inter1, lvl1, lrs1, si_max;
  double thr_prs, thr_rho, thr_vel;
};
// SI [n]: interface layers, SI[0] | SI[1] << 16, or in 64 bits SI[0] | SI[1] << 32 (wide: layers of
// 2^16 and more); lists scratch [2 n + 3]; split [n]; symmetric: every cell's face neighbours have it as theirs
// pr: scratch [3][n] doubles (each cell's mixture pressure and density, made once)
void ffv_m5_tags(const ffv_dmesh &m, const M5Consts &k, const ffv_m5_tagc &t, bool symmetric,
                 const double *S, void *SI, bool wide, int32_t *lists, int32_t *split, double *pr,
                 cudaStream_t st);
// the layers as [2][n]
void ffv_m5_si_unpack(int64_t n, const void *SI, bool wide, int32_t *out, cudaStream_t st);

// exported per-leaf fields, F [nf][n] double (ffv_export_fields)
void ffv_m5_export_fields(int64_t n, const M5Consts &k, const double *S, double *F,
                          cudaStream_t st);
void ffv_m0_export_fields(int64_t n, double gamma, double pinf, const double *S, double *F,
                          cudaStream_t st);

// model 0 (ffv_m0_tags.cu): the relative-jump criterion on cell states and the indicator
// fields (log rho, log p, 1, |u|, 0)
void ffv_m0_tags(const ffv_dmesh &m, double gamma, double pinf, const ffv_m5_tagc &t,
                 const double *S, int32_t *split, cudaStream_t st);
void ffv_m0_indicator_fields(int64_t n, double gamma, double pinf, const double *S,
                             const ffv_field_out &out, cudaStream_t st);

// the reference's FP64 relaxation of the cells a mesh adaptation merged (map < 0)
void ffv_m5_relax_merged(int64_t n, const M5Consts &k, const int64_t *map, double *S,
                         cudaStream_t st);

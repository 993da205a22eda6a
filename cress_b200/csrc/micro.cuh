// Cold-rain microphysics kernels (internal interface).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include "common.cuh"
#include "hevi.cuh"

namespace cress {

// What the process rates take from a level alone, formed once per level on
// the host (float, from the base columns and the microphysics step): every
// cell of the level would otherwise spend a third of its exponentials,
// logarithms and square roots on them.  With this and one logarithm per
// species' mean diameter, k_micro_src, which is bound by the issue of such
// chains, takes 1462 us at 512 x 512 x 64 instead of 1698.
struct alignas(16) MicroLevel {
  float ptbr, rbr, rbv, pbr;    // rbv = 1/rbr
  float sr0v;                   // sqrt(r0 rbv): (r0/rbr)^gur of termblk.f90, gur = gus = gug = 0.5
  float sr0r, srbr;             // sqrt(r0 rbr), sqrt(rbr)
  float ncc;                    // diagnosed cloud number (diagnw.f90)
  float agin, cnis;             // rbr (cagin/rbr)^(1/3) of aggregat.f90 and convers.f90
  float cncr;                   // autoconversion's level factor (convers.f90)
  float rstv;                   // 1/rst
};
// The same for constants of the scheme and the step.
struct MicroConst {
  float cnu, cdv;               // nu0^.57013 / t0, dv0^.55249 / t0
  float cvntr, cvnts, cvntg;    // ventilation coefficients (setblk.f90:789-830)
  float agsn;                   // snow aggregation (aggregat.f90)
  float diaqs0;                 // diameter of the smallest snow (convers.f90)
};

struct MicroArgs {
  Grid g;
  const MicroLevel* lv;   // rows k = 0..nk
  MicroConst mc;
  const float* col;  // 1-D base columns (C_PTBR, C_RBR, C_PBR, C_JCB, C_RST used)
  // past level t-dt (pp: pressure perturbation for p and the Exner function)
  const float *ptpp, *qvp, *qcp, *qrp, *qip, *qsp, *qgp, *nip, *nsp, *ngp, *ppp;
  // future level t+dt (updated)
  float *ptpf, *qvf, *qcf, *qrf, *qif, *qsf, *qgf, *nif, *nsf, *ngf;
  float* prec;       // 10 planes (px*py): prc, prr, pri, prs, prg x (rate, accumulated)
  float* uspd;       // fall speeds of rain, snow and graupel (past level), written by the process-rate kernels
  int* dtp_bits;     // domain minimum of the sedimentation step (float bits, positive)
  float dtb;         // microphysics step = 2*dtb of the leapfrog (cloudphy.f90:282)
  float dz, thresq;
  int defer_adjstni; // 1: the final adjstni is left to k_moist_post (large step)
};

// Rows 0..nk of the level table for base columns col (col[f*(nk+1) + k]) and
// a microphysics step dtb, and the constants of that step.
void micro_levels(const float* col, int nk, float dtb, MicroLevel* out);
MicroConst micro_const(float dtb);
// Koenig table upload (once per device); returns a CRESS status.
int micro_init_tables();
// s_cloudphy for cphopt=3: source terms and sedimentation; or the two
// halves (process rates with the sub-step minimum, then sedimentation).
int launch_cloudphy(const MicroArgs& a, cudaStream_t st);
int launch_cloudphy_src(const MicroArgs& a, cudaStream_t st);
int launch_cloudphy_fall(const MicroArgs& a, cudaStream_t st);

struct SatArgs {
  Grid g;
  const float* col;  // C_PTBR, C_PBR
  const float* pp;
  float *ptp, *qv, *qc, *qi, *ni;
  float thresq;
};
int launch_satadjst(const SatArgs& a, cudaStream_t st);

// After the moist step's s_cloudphy: the Asselin filter of the nine moist
// fields (when `filter`) and s_satadjst on t and t+dt, pointwise in one
// pass.  Field order qv, qc, qr, qi, qs, qg, ni, ns, ng.
struct MoistPostArgs {
  Grid g;
  const float* col;
  float* c[9];          // t (filtered in place, then adjusted)
  float* f[9];          // t+dt (adjusted)
  const float* p[9];    // t-dt
  float* ptpc; const float* ppc;   // theta', p' at t (already filtered)
  float* ptpf; const float* ppf;   // theta', p' at t+dt
  float filcoe, thresq;
  int filter;
  int adjstni;          // 1: apply cloudphy's final adjstni to t+dt first (coldblk.f90:469)
};
int launch_moist_post(const MoistPostArgs& a, cudaStream_t st);

// Learned form of the process-rate part (the MLP of mlp.cu).
struct Mlp;
struct LearnedBuffers {
  bool fused = false;             // one persistent fused kernel (fb_list holds every cell)
  int chunk = 0;                  // cells per inference chunk (multiple of 128), chunked path
  __nv_bfloat16* xb = nullptr;    // [chunk][64] standardized inputs
  __nv_bfloat16* h0 = nullptr;    // [chunk][256] activations (ping)
  __nv_bfloat16* h1 = nullptr;    // [chunk][256] activations (pong)
  float* y = nullptr;             // [chunk][64] outputs
  unsigned char* env = nullptr;   // [chunk] inside the training envelope
  int* fb_list = nullptr;         // [chunk] cells sent to the plain scheme
  int* fb_count = nullptr;
  unsigned long long* stats = nullptr;   // MLP cells, fallback cells
  int* err = nullptr;
};
int launch_cloudphy_learned(const MicroArgs& a, const float* w, Mlp* m, const LearnedBuffers& L, float resid_tol,
                            cudaStream_t st, long long* launches);
int launch_cloudphy_fused(const MicroArgs& a, const float* w, Mlp* m, const LearnedBuffers& L, float resid_tol,
                          cudaStream_t st, long long* launches);
int launch_collect_tuples(const MicroArgs& a, const float* w, Mlp* m, int stride, float keep_zero,
                          unsigned long long seed, unsigned long long* count_d, cudaStream_t st);

}  // namespace cress

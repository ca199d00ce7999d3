// Device-side model description and the pointwise helpers every kernel shares.
//
// All device arrays keep the reference layout X(k,j,i) = base[i + (j+1)*iadim + k*n2]
// (include/epic.h:407-449), so host upload/download are plain copies.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cfloat>
#include <type_traits>
#include "dd_math.cuh"
#include "df.cuh"

// kernel groups whose block size the autotuner picks (DevModel::tb)
enum TuneGroup { TB_UV_CORE = 0, TB_PGRAD, TB_HSU, TB_VISC, TB_DIAG, TB_UPDATE, TB_COLUMN, TB_POINT, TB_ROW,
                 TB_HSU_MERID_VARIANT,   // not a block size: 0 automatic, else a HsuForm (kernels.h)
                 TB_COUNT };
#define TB(M, g) ((M).tb[g] > 0 ? (M).tb[g] : 128)

#define EPIC_MAX_NK 126      // column kernels keep per-column arrays of nk+2 entries
#define EPIC_MAX_NI 1024     // row kernels keep one row of ni entries in shared memory
#define EPIC_TURB_MAX_NK 64  // the turbulence closure's column solves keep nk+3 entries per array

namespace epic {

// Quantities of the latitude rows that the stencils divide or convert once per cell otherwise, made at
// model creation in each compute type (k_row_tables) with the expressions of the kernels: row j's h
// point is half-level 2j+1, its v point 2j.
enum RowTab { RT_NINV_H, RT_MINV_V, RT_MINV_H, RT_MNINV_H, RT_MNINV_V, RT_MNPV, RT_GDX, RT_GDY, RT_M_H, RT_M_V, RT_N_V, RT_MN_H, RT_F_V,
              RT_COUNT = 16 };

constexpr int SCRATCH_VOLUMES = 8;   // gz, unity, old, work0..3, lp3
constexpr int TABLE_SETS = 4;        // ptable, once per field of the 3-D filter
// Which volumes are work0..3 of a branch of the step (scratch_sets).  Concurrent branches keep theirs apart
// in volumes that nothing else uses at the time, so that they cost a model no memory: GZ until the 3-D
// filter needs it, OLD before THETA's and after NU_TURB's advection, UNITY after advection, DZDT3 until
// store_pgrad_vars writes every cell that the branch does (rows 0..nj of layers 1..nk), lp3 in the FP64 form.
enum ScratchSet { WS_MAIN = 0,      // the model's own
                  WS_KIN_TURB,      // uv_core beside source_sink_turb: KIN in lp3
                  WS_UNITY,         // UNITY's Akima fluxes in DZDT3
                  WS_THETA,         // THETA's hyperviscosity in GZ and OLD, its Akima fluxes in GZ
                  WS_THETA_TURB,    // THETA's hyperviscosity beside HDRY's and NU_TURB's: in work0 and work3
                  WS_NU,            // NU_TURB's diffusion and hyperviscosity in GZ, OLD and lp3, its Akima fluxes in GZ
                  WS_V };           // V's hyperviscosity and filtered copy beside U's: in UNITY and OLD

// Time-plane indices and step counters live on the device so that one captured CUDA graph
// serves every step (the reference rotates IT_ZERO/IT_MINUS1/IT_MINUS2 on the host,
// src/shared/epic_timestep.c:257-274).
// What every kernel reads before its first useful load comes first, in one cache line.
struct Ctl {
  int it_zero, it_minus1, it_minus2;
  int it_uv, it_uv_dis, it_uv_tend;
  int halted;                          // set between steps once err_code is set: every kernel of the
                                       // model then returns at entry (the reference stops the run at
                                       // its first epic_error); cleared by an upload
  long long itime, model_time;
  int err_code, err_k, err_j, err_i;   // first model error (0 = none)
  double err_val;
  double ab[2][3];                     // Adams-Bashforth coefficients chosen for u, v this step
  float2 abf[2][3];                    // the same as double-floats (the mixed forms' update)
  int lf_first[2];                     // leapfrog: forward (Euler) first step for u, v
};

enum ErrCode { ERR_NONE = 0, ERR_GZ_MONOTONE = 1, ERR_CALC_W_P = 2, ERR_PCHIP_X = 3, ERR_NONFINITE = 4, ERR_TIMEOUT = 5,
               ERR_TURB = 6 };

// double-float constants of the mixed form (DevModel::dfc), split on the host
enum { DFC_KAPPA, DFC_KAPPA_INV, DFC_KAPPA1, DFC_SIGMA_SIGMA, DFC_ZETA0, DFC_ZETA1, DFC_G_COEFF, DFC_ALPHA, DFC_LOG_P0,
       DFC_COUNT };

struct DevModel {
  // sizes
  int ni, nj, nk, iadim, jadim, kadim;
  long long n2, n3;
  int nvp, ntp;
  // scalars
  int uv_scheme, k_sigma, k_sponge, newt_cool_on, drag_v, drag_zonal_avg, rayleigh_on;
  int akima;   // advection scheme: 0 Hsu-Konor-Arakawa predictor-corrector, 1 Akima
  double dt, press0, topo_scale, prandtl, tau_drag, nudiv;
  double zeta0, zeta1, alpha, sigma_sigma, g_coeff;   // g_coeff = 1/(1-exp(-alpha*(1-sigma_sigma)))
  double kappa, cp, cpr, rgas, mu_dry, hs_kf, lat0, m0, eps13;
  double coef[9], nu[9];
  // 1-D grid arrays (device copies)
  const double *lon, *lat, *rln, *rlt, *f, *m, *n, *mn, *grav, *mn_inv;
  const double *sgth, *dsgth, *dsgth_inv, *h_min, *t_sponge_inv;
  const double *high_lat_h, *high_lat_pv;   // [(nj+3)*(ni+2)] 2-D like the reference
  int filt_south_h, filt_north_h, filt_south_v, filt_north_v;   // the rows that the zonal filter changes, |lat| >=
                                            // lat0: j up to filt_south and from filt_north on, h rows and v rows
                                            // (scalars: a run-time index would put a kernel's DevModel in memory)
  int filt_bands;                           // 0: not two such bands (row_is_filtered compares the latitude)
  const double *h_coef, *v_coef;            // d2dy2 coefficients, 3 per row
  const double *rt64;                       // RowTab of rows 0..nj+1, RT_COUNT values each, in binary64 ...
  const float *rt32;                        // ... and in binary32
  const double *vt64;                       // d2dy2's coefficients times the orders' 2, 4, 6 and 8: 12 a row, h rows
  const float *vt32;                        // 0..nj+1, then v rows (k_visc_tables), in both compute types
  const double *tw;                         // realft/four1 twiddles (see k_filter.cu)
  const double *coslat;                     // cos(lat[2j+1] deg), j = 0..nj, from the host libm
  const double *coslat4;                    // pow(coslat[j], 4.) correctly rounded (t_rad's cos^4)
  const MathTable *lt;                      // double-double tables for cr_log/cr_exp/cr_pow
  const float *twf;                         // the twiddles rounded to float (mixed form)
  const void *fop_map;                      // tensor-core filter (mixed form): the TMA tensor map of the
                                            // operator tiles of the filtered rows (k_filter_gemm.cu), or null
  const int *fop_slot;                      // their slot of each row j = -1..nj+1, h rows then v rows; -1
                                            // where the row is not filtered
  const float2 *exp2tab;                    // 2^(j/32), j = 0..31, as double-floats (exp_df)
  float2 dfc[DFC_COUNT];                    // kappa, 1/kappa, kappa+1, the hybrid-coordinate constants
                                            // and log(press0) as double-floats (hi, lo)
  double x_h2, x_he, x_3;                   // hydrogen thermodynamics when x_h2 > 0 (FP64 form)
  const double *thermo;                     // thermo_setup's tables (thermo_tables in epic_model.cu)
  int gas_giant;                            // planet->type "gas-giant": GZ_SURFACE from gz_from_u in store_pgrad_vars
  int jtp;                                  // grid.jtp: the row where gz_from_u puts GZ_SURFACE's zero
  // the Spalart-Allmaras DES turbulence closure (FP64 form; k_turb.cu)
  int turb;                                 // epic_grid.turbulence on
  int turb_h, turb_v;                       // horizontal / vertical subgrid diffusion (grid.diffusion_direction)
  int stab;                                 // grid.stability_factor "Collins et al. (2004)" (else "off")
  double kinvisc, dynvisc, max_nu2;         // planet->kinvisc, planet->dynvisc, set_max_nu's max_nu[2]
  double *nu_turb, *dc_uv, *dc_theta, *dc_mass;   // NU_TURB and DIFFUSION_COEF_UV, _THETA, _MASS
  double *turb_tau;                         // scratch: the wall stresses, one per column
  double *turb_pole;                        // scratch: the polar TAU12 rows of uv_horizontal_diffusion
  const double *turb_maxnu2;                // set_diffusion_coef's taper max_nu[2] MIN(1, (dy0 m)^-2), j = 0..nj
  int mixed;                                // FP32 stencils, advection, hyperviscosity, filter, physics
  int col64;                                // mixed, with the vertical pressure/geopotential integration
                                            // (set_p2etc, store_pgrad_vars) and the pressure gradient in FP64
  int cr;                                   // binary64 log/exp/pow correctly rounded (the drop-in form);
                                            // else the libdevice functions
  // state
  double *u, *v, *dudt, *dvdt, *hdry, *theta, *p3, *h3, *p2, *theta2, *t2, *t3, *rho2, *rho3, *exner3;
  double *gz3, *mont3, *heat3, *pv3, *ri2, *div_uv3, *w3, *dzdt3, *u_spinup, *gz_surface;
  // scratch
  double *gz, *unity, *old, *work0, *work1, *work2, *work3, *ptable;
  int wset, tset;   // which ScratchSet this launch's work0..3 are and which of the TABLE_SETS copies of
                    // ptable its ptable is (on a member's own description both are 0)
  float2 *lp3;   // log P3 at every interface as a double-float: written by set_p2etc of the mixed
                 // form (stage 11), read by its store_pgrad_vars (stage 19); P3 does not change
                 // between the two
  Ctl *ctl;
  // batch: the members' descriptions on the device (nullptr for a single model); kernels
  // launched over a batch take member blockIdx.z's description on entry (EPIC_MEMBER)
  const DevModel *batch;
  int nbatch;
  int hetero;          // batch launch over members of different ni / nj (epic_member relocates
                       // pointer arguments field by field); the launch description then carries
                       // the largest sizes of its members, and member 0's arrays
  long long reloc_n3;  // a launch description's field size of member 0 (whose arrays it carries)
  int fop_shared;      // a batch whose members all filter with member 0's operator tiles (same grid)
  char *pool_base;   // start of the model's device pool (state, scratch and tables)
  int sms;           // the model's device (host side only): its SMs, which the launch rules fill,
  int sa_cluster;    // and the blocks of the closure's wavefront cluster
  // launch shapes (host side only): threads per block of each kernel group, set by the
  // autotuner; they change no result (every tuned kernel is pointwise or per row)
  int tb[TB_COUNT];

  // Offsets within one 3-D field of one model: 32-bit arithmetic (epic_model_create rejects
  // grids whose wind arrays, up to three time planes, reach 2^31 elements).
  __host__ __device__ __forceinline__ int at(int k, int j, int i) const { return i + (j + 1) * iadim + k * (int)n2; }
  __host__ __device__ __forceinline__ int at2(int j, int i) const { return i + (j + 1) * iadim; }
};

// A pointer into member 0's arrays, moved to the same place in member `to`'s arrays.  The pool of
// a model (epic_model_create) packs the state arrays back to back as planes of n3 values (u and v
// value planes, the tendency planes, then the single fields), and carves the scratch volumes gz,
// unity, old, work0..3, lp3 one after another, each rounded up to 256 bytes (and, with the turbulence
// closure, NU_TURB and the three diffusivities the same way); so the plane (or volume) index and
// the offset inside it follow from the address by integer arithmetic, and map to the member's
// pool with its own n3.  A pointer outside these regions (a table) is returned as is.
__host__ __device__ __forceinline__ long long scratch_stride(long long n3) { return ((n3 * 8 + 255) / 256) * 256; }
template <class P>
__device__ __forceinline__ P *relocate_field(const DevModel &from, const DevModel &to, P *p) {
  const char *c = reinterpret_cast<const char *>(p);
  const long long n3 = from.reloc_n3;
  const char *s0 = reinterpret_cast<const char *>(from.gz);
  const long long st0 = scratch_stride(n3);
  if (c >= s0 && c < s0 + SCRATCH_VOLUMES * st0) {
    const long long o = c - s0, q = o / st0;
    return reinterpret_cast<P *>(reinterpret_cast<char *>(to.gz) + q * scratch_stride(to.n3) + (o - q * st0));
  }
  if (from.nu_turb) {   // the turbulence closure's four volumes (NU_TURB, the diffusivities), one stride apart
    const char *t0 = reinterpret_cast<const char *>(from.nu_turb);
    if (c >= t0 && c < t0 + 4 * st0) {
      const long long o = c - t0, q = o / st0;
      return reinterpret_cast<P *>(reinterpret_cast<char *>(to.nu_turb) + q * scratch_stride(to.n3) + (o - q * st0));
    }
  }
  const char *b0 = reinterpret_cast<const char *>(from.u);
  const long long planes = 2LL * from.nvp + 2LL * from.ntp + 20;
  if (c >= b0 && c < b0 + planes * n3 * 8) {
    const long long o = (c - b0) / 8, q = o / n3;
    return reinterpret_cast<P *>(to.u + q * to.n3 + (o - q * n3));
  }
  return p;
}

// Entry of every kernel: in a batch launch, take member blockIdx.z's description and move the
// state pointers passed as arguments (addresses in the launch description's arrays) to the same
// places in the member's arrays: by offset when the members share the pool layout (same sizes),
// array by array when they do not.  Returns true when the model is halted (a step found a fatal
// error): the kernel then returns at once.  Ctl::halted changes only in k_itime_advance, between
// steps, so every thread of a launch reads the same value.
template <class P>
__device__ __forceinline__ P *member_ptr(const DevModel &M, const DevModel &mem, P *p) {
  if (!p) return p;
  if (M.hetero) return relocate_field(M, mem, p);
  return (P *)(mem.pool_base + ((const char *)p - M.pool_base));
}
// Point work0..3 and ptable of a description that has its own at sets ws and ts.
__host__ __device__ __forceinline__ void scratch_sets(DevModel &M, int ws, int ts) {
  if (ws) {
    double *lp3 = reinterpret_cast<double *>(M.lp3);
    switch (ws) {
      case WS_KIN_TURB: M.work0 = lp3; break;
      case WS_UNITY: M.work3 = M.dzdt3; break;
      case WS_THETA: M.work1 = M.gz; M.work2 = M.old; M.work3 = M.gz; break;
      case WS_THETA_TURB: M.work1 = M.work0; M.work2 = M.work3; break;
      case WS_NU: M.work0 = M.gz; M.work1 = M.old; M.work2 = lp3; M.work3 = M.gz; break;
      case WS_V: M.work1 = M.unity; M.work2 = M.old; break;
    }
    M.wset = ws;
  }
  if (ts) {
    M.ptable += (long long)ts * 3 * (M.nj + 3) * (M.nk + 2);
    M.tset = ts;
  }
}
template <class... P>
__device__ __forceinline__ bool epic_member(DevModel &M, P *&...ptrs) {
  if (M.batch) {
    const DevModel &mem = M.batch[blockIdx.z];
    ((ptrs = member_ptr(M, mem, ptrs)), ...);
    const int ws = M.wset, ts = M.tset;
    M = mem;
    scratch_sets(M, ws, ts);
  }
  return M.ctl->halted != 0;
}

// ---- pointwise helpers: restatements of the reference routines named beside each ----

__device__ __forceinline__ double dmaxr(double x, double y) { return x > y ? x : y; }   // MAX, include/epic.h:144
__device__ __forceinline__ double dminr(double x, double y) { return x < y ? x : y; }   // MIN, include/epic.h:138

// fcmp, src/shared/epic_funcs_util.c:4275-4330.  delta is two units of the last place of the larger
// magnitude, so values of one sign whose bit patterns lie more than 8 apart are ordered as their
// patterns are, and opposite signs as their signs: the usual answers, on the integer pipe (the
// comparison itself is four binary64 operations, 16 clocks a warp each).  The rest -- near neighbours,
// zeros, very small or infinite magnitudes, NaN -- takes the reference's own arithmetic.
static __device__ __noinline__ int fcmp_near(double x1, double x2) {
  int e;
  frexp(fabs(x1) > fabs(x2) ? x1 : x2, &e);
  const double delta = ldexp(DBL_EPSILON, e);
  const double d = x1 - x2;
  return d > delta ? 1 : (d < -delta ? -1 : 0);
}
__device__ __forceinline__ int fcmp(double x1, double x2) {
  const long long u1 = __double_as_longlong(x1), u2 = __double_as_longlong(x2);
  const unsigned e1 = (unsigned)(u1 >> 52) & 0x7ffu, e2 = (unsigned)(u2 >> 52) & 0x7ffu;
  const long long d = u1 - u2;
  const bool same = (u1 ^ u2) >= 0, apart = same ? d > 8 || d < -8 : true;
  if (e1 - 64u < 1983u && e2 - 64u < 1983u && apart) return (same ? (d > 0) != (u1 < 0) : u2 < 0) ? 1 : -1;
  return fcmp_near(x1, x2);
}

// THETA2 at an isentropic layer (set_p2etc, K > k_sigma-1) interpolates linearly in the table
// (sigmatheta[2K+1], THETA(K)), K = nk down to k_sigma-1, at sigmatheta[2K] (linint after
// find_place_in_table, epic_funcs_diag.c:3553-3561, epic_funcs_util.c:636-648,2908-2976).  The interval
// found depends on the vertical grid alone: a column kernel finds it once per level for the whole
// block (theta2_intervals, before its first barrier) instead of once per column -- the search's
// fcmp calls are binary64 operations.  kay indexes the ascending table x = sigmatheta[2(nk-kay)+1].
__device__ __forceinline__ int theta2_interval(const DevModel &M, int k) {
  const int nk = M.nk, nkay = nk - (M.k_sigma - 1) + 1;
  const double sg = M.sgth[2 * k];
  auto X = [&](int kay) { return M.sgth[2 * (nk - kay) + 1]; };
  if (fcmp(sg, X(0)) <= 0) return 0;
  if (fcmp(sg, X(nkay - 1)) >= 0) return nkay - 2;
  int il = -1, iu = nkay;
  while (iu - il > 1) {
    const int im = (iu + il) >> 1;
    if (fcmp(sg, X(im)) >= 0) il = im; else iu = im;
  }
  return il;
}
// the intervals of levels k_sigma..nk, and for the binary32 forms (w != nullptr) the weights
// (sigmatheta[2k] - x0) / (x1 - x0) rounded to binary32
__device__ __forceinline__ void theta2_intervals(const DevModel &M, int *kay, float *w) {
  for (int k = M.k_sigma + (int)threadIdx.x; k <= M.nk; k += (int)blockDim.x) {
    const int q = theta2_interval(M, k);
    kay[k] = q;
    if (w) {
      const double x0 = M.sgth[2 * (M.nk - q) + 1], x1 = M.sgth[2 * (M.nk - q - 1) + 1];
      w[k] = (float)((M.sgth[2 * k] - x0) / (x1 - x0));
    }
  }
}

// In the drop-in form the transcendentals are correctly rounded (dd_math.cuh) so that they agree
// with the reference's libm; the mixed form's binary64 kernels take the libdevice functions.
__device__ __forceinline__ double xlog(const DevModel &M, double x) { return M.cr ? cr_log(x, *M.lt) : ::log(x); }
__device__ __forceinline__ double xexp(const DevModel &M, double x) { return M.cr ? cr_exp(x, *M.lt) : ::exp(x); }
__device__ __forceinline__ double xpow(const DevModel &M, double x, double y) { return M.cr ? cr_pow(x, y, *M.lt) : ::pow(x, y); }
// f_sigma(s), with g_sigma(s) returned in g (epic_funcs_diag.c:1238-1314, 1751-1770; get_sigma, get_p_sigma and
// return_sigmatheta are parts of the column kernels): one exponential and each comparison (a binary64 operation)
// serve both.
__device__ __forceinline__ double f_and_g_sigma(const DevModel &M, double s, double &g) {
  if (s <= M.sigma_sigma) {
    g = 0.;
    return s < 0. ? M.zeta0 : M.zeta0 + s * (M.zeta1 - M.zeta0);
  }
  if (s >= 1.) {
    g = 1.;
    return 0.;
  }
  g = M.g_coeff * (1. - xexp(M, -M.alpha * (s - M.sigma_sigma)));
  return (1. - g) * (M.zeta0 + s * (M.zeta1 - M.zeta0));
}
// return_density (ideal gas); return_temp and return_enthalpy below (the ideal gas, or hydrogen)
// The hydrogen thermodynamics of thermo_setup's tables (x_h2 > 0; normal hydrogen, fpara = 0.25,
// the para fraction the reference takes when the fpara tracer is off, epic_funcs_diag.c:3709;
// ideal equation of state).  Layout of DevModel::thermo: T(fp, theta_mean) [16][128], the ortho
// and para enthalpies [2][128], the temperature grid [128], the mean potential temperature grid
// [128], the para fractions [16].
constexpr int TH_M = 128, TH_N = 16;
constexpr double TH_FP = 0.25;
__device__ __forceinline__ const double *th_t(const DevModel &M) { return M.thermo; }
__device__ __forceinline__ const double *th_h(const DevModel &M, int q) { return M.thermo + TH_N * TH_M + q * TH_M; }
__device__ __forceinline__ const double *th_tgrid(const DevModel &M) { return M.thermo + TH_N * TH_M + 2 * TH_M; }
__device__ __forceinline__ const double *th_thgrid(const DevModel &M) { return M.thermo + TH_N * TH_M + 3 * TH_M; }
__device__ __forceinline__ const double *th_fpdat(const DevModel &M) { return M.thermo + TH_N * TH_M + 4 * TH_M; }

// return_temp, epic_funcs_diag.c:6112-6210: the ideal relation, or with hydrogen the table of
// temperature against para fraction and mean potential temperature (bilinear).  The hydrogen
// part, from the ideal-gas temperature theta1 = theta (p/p0)^kappa (which the mixed forms' column
// kernels evaluate with their own power):
__device__ __forceinline__ double hydrogen_temp(const DevModel &M, double theta1) {
  if (theta1 <= 20.) return theta1;
  if (theta1 >= 600.)
    return xexp(M, (M.cpr * xlog(M, theta1) - 2.5 * M.x_h2 * ((1. - TH_FP) * -2.105769 + TH_FP * -1.666421)) /
                       (2.5 * M.x_he + 3.5 * (1. - M.x_he)));
  const double *fpdat = th_fpdat(M), *thg = th_thgrid(M), *t = th_t(M);
  const double en = div_rn((double)(TH_N - 1) * (TH_FP - fpdat[0]), fpdat[TH_N - 1] - fpdat[0]);
  int n = (int)en;
  double ffp, fth;
  if (n > TH_N - 2) { n = TH_N - 2; ffp = 1.; }
  else if (n < 0) { n = 0; ffp = 0.; }
  else ffp = fmod(en, 1.);
  const double em = div_rn((double)(TH_M - 1) * (theta1 - thg[0]), thg[TH_M - 1] - thg[0]);
  int m = (int)em;
  if (m > TH_M - 2) { m = TH_M - 2; fth = 1.; }
  else if (m < 0) { m = 0; fth = 0.; }
  else fth = fmod(em, 1.);
  return t[n * TH_M + m] * (1. - fth) * (1. - ffp) + t[(n + 1) * TH_M + m] * (1. - fth) * (ffp) +
         t[n * TH_M + m + 1] * (fth) * (1. - ffp) + t[(n + 1) * TH_M + m + 1] * (fth) * (ffp);
}
__device__ __forceinline__ double return_temp(const DevModel &M, double p, double theta) {
  if (M.x_h2 == 0.) return theta * xpow(M, div_rn(p, M.press0), M.kappa);
  return hydrogen_temp(M, theta * xpow(M, div_rn(p, M.press0), M.kappa));
}
__device__ __forceinline__ double return_density(double p, double t, double mu) { return div_rn(p * mu, 8.314472e+3 * t); }
__device__ __forceinline__ double return_enthalpy(const DevModel &M, double t) {
  if (M.x_h2 == 0. || t <= 20.) return (M.cpr * t) * M.rgas;
  double enthalpy;
  if (t > 500.) {   // hydrogen above the table, epic_funcs_diag.c:6699-6712
    const double ho = 1545.3790 + 3.5 * (t - 500.), hp = 1720.3776 + 3.5 * (t - 500.);
    enthalpy = (M.x_h2) * ((1. - TH_FP) * ho + TH_FP * hp) + (M.x_he * 2.5 + M.x_3 * 3.5) * t;
  } else {          // :6713-6735
    const double *tg = th_tgrid(M), *ho = th_h(M, 0), *hp = th_h(M, 1);
    const double em = div_rn((double)(TH_M - 1) * (t - tg[0]), tg[TH_M - 1] - tg[0]);
    int m = (int)em;
    double fract;
    if (m == TH_M - 1) { m--; fract = 1.; }
    else fract = fmod(em, 1.);
    const double h0 = (1. - fract) * ho[m] + (fract) * ho[m + 1], h1 = (1. - fract) * hp[m] + (fract) * hp[m + 1];
    enthalpy = (M.x_h2) * ((1. - TH_FP) * h0 + (TH_FP) * h1) + (M.x_he * 2.5 + M.x_3 * 3.5) * t;
  }
  return enthalpy * M.rgas;
}

// ---- binary64 <-> binary32 conversions on the integer pipe ----
//
// GB300 executes FP64 arithmetic and the F64<->F32 conversion instructions on the same narrow
// FP64 unit, about 1.7 operations per clock per SM against ~114 for FP32 adds (measured).  The
// mixed form reads its binary64 state in every kernel, so it converts with a few integer
// operations and selects instead (no branch).  For every normal binary32 result, zero,
// infinity and overflow the bits are those of the hardware's round-to-nearest-even conversion;
// a NaN stays a NaN; binary32 subnormals (magnitudes below 1.2e-38, which the model's fields
// never hold except as exact zeros) are flushed to signed zero in both directions.
__device__ __forceinline__ float d2f(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned a = hi & 0x7fffffffu;
  // round the 64-bit pattern to nearest-even at bit 29 (a carry may bump the exponent), then
  // take the 8 low exponent bits and the 23 leading mantissa bits and rebias the exponent
  const unsigned long long v = (((unsigned long long)hi << 32) | lo) + (0x0fffffffull + ((lo >> 29) & 1u));
  unsigned u = (__funnelshift_l((unsigned)v, (unsigned)(v >> 32), 3) - (896u << 23)) | (hi & 0x80000000u);
  if (a - 0x38100000u >= 0x0fe00000u)   // |x| < FLT_MIN (to signed zero), or beyond FLT_MAX, inf, NaN
    u = (hi & 0x80000000u) | (a < 0x38100000u ? 0u : ((a | (lo != 0u)) > 0x7ff00000u ? 0x7fc00000u : 0x7f800000u));
  return __uint_as_float(u);
}
__device__ __forceinline__ double f2d(float f) {
  const unsigned w = __float_as_uint(f), a = w & 0x7fffffffu;
  unsigned hi = (a >> 3) + (896u << 20), lo = a << 29;
  hi = a >= 0x7f800000u ? hi + (896u << 20) : hi;            // infinity, NaN: exponent 2047
  hi = a < 0x00800000u ? 0u : hi;
  lo = a < 0x00800000u ? 0u : lo;
  return __hiloint2double((int)(hi | (w & 0x80000000u)), (int)lo);
}

// ---- binary64 <-> double-float without the FP64 unit ----
//
// The double-float form of x is (hi, lo) = (RN32(x), RN32(x - hi)) and its binary64 value is
// RN64(hi + lo): one FP64 subtraction or addition each, at the FP64 unit's rate.  The mixed
// form's column kernels convert several values per level, so both are computed on the integer
// and FP32 pipes instead, with the same bits: the residual x - hi is the part of x's 53-bit
// significand below hi's rounding point, an integer r (|r| <= 2^28) in units of x's last place,
// rounded to binary32 by one fused multiply-add of two exact halves; hi + lo moves hi's binary64
// significand by lo in units of its last place, rounded to nearest-even by the conversion to
// integer (in the binade below a power of two when lo takes hi towards zero, whose unit is half
// as large; a normalised lo, |lo| <= ulp32(hi)/2, never takes the sum out of those binades).
// Magnitudes below 2^-74 (5e-23, far below any value of the model's fields but exact zeros) keep
// binary32 precision: lo is zero there, and a hi that small converts without its lo.
__device__ __forceinline__ dfl d2df(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned a = hi & 0x7fffffffu;
  const unsigned half = 0x0fffffffu + ((lo >> 29) & 1u);   // d2f's rounding increment
  const unsigned long long v = (((unsigned long long)hi << 32) | lo) + half;
  unsigned u = (__funnelshift_l((unsigned)v, (unsigned)(v >> 32), 3) - (896u << 23)) | (hi & 0x80000000u);
  if (a - 0x38100000u >= 0x0fe00000u)
    u = (hi & 0x80000000u) | (a < 0x38100000u ? 0u : ((a | (lo != 0u)) > 0x7ff00000u ? 0x7fc00000u : 0x7f800000u));
  // x - hi in units of x's last place: the 29 bits below the rounding point, less the carry
  const int r = (int)((unsigned)v & 0x1fffffffu) - (int)half;
  const int rs = (int)hi < 0 ? -r : r;
  // rs = 64 q + b with |q| <= 2^22 and 0 <= b < 64, both exact in binary32 by the 1.5 2^23 and
  // 2^23 shifts; lo = RN32(rs 2^(E-1075)), E the binary64 exponent field, normal for E >= 949
  const float fq = __uint_as_float(0x4B400000u + (unsigned)(rs >> 6)) - 12582912.f;
  const float fb = __uint_as_float(0x4B000000u + ((unsigned)rs & 63u)) - 8388608.f;
  const unsigned e = a >> 20;
  const float sc = e - 949u < 202u ? __uint_as_float((e - 948u) << 23) : 0.f;
  return dfl(__uint_as_float(u), fmaf(fq, 64.f * sc, fb * sc));
}
__device__ __forceinline__ double df2d(dfl x) {
  const unsigned wh = __float_as_uint(x.hi), wl = __float_as_uint(x.lo), ah = wh & 0x7fffffffu, eh = ah >> 23;
  // lo towards zero from a power of two: the binade below, its unit half as large
  const unsigned down = (ah & 0x007fffffu) == 0u && ((wl ^ wh) & 0x80000000u) && (wl & 0x7fffffffu) ? 1u : 0u;
  const bool ok = eh - 52u - down < 202u - down;   // 2^-74 <= |hi| (2^-73 going down), finite
  // lo in units of the last place of hi's binary64 significand: lo 2^(52 - (eh - 127) + down)
  const float sc = __uint_as_float(((ok ? 306u - eh : 127u) + down) << 23);
  const int k = ok ? __float2int_rn(x.lo * sc) : 0;
  unsigned long long mag = ((unsigned long long)ah << 29) + (896ull << 52);
  mag = ah >= 0x7f800000u ? mag + (896ull << 52) : (ah < 0x00800000u ? 0ull : mag);   // f2d's cases
  mag += (long long)((int)wh < 0 ? -k : k);
  return __longlong_as_double((long long)(mag | ((unsigned long long)(wh & 0x80000000u) << 32)));
}

// ---- compute-type helpers for kernels instantiated in FP64 (R = double: the drop-in form,
// bit-identical to the reference's arithmetic) and FP32 (R = float: the mixed form) ----

// a binary64 value in the compute type, and a compute-type value back in binary64
template <class R> __device__ __forceinline__ R cv(double x);
template <> __device__ __forceinline__ double cv<double>(double x) { return x; }
template <> __device__ __forceinline__ float cv<float>(double x) { return d2f(x); }
template <> __device__ __forceinline__ dfl cv<dfl>(double x) { return d2df(x); }
// a model constant in the compute type: the double-float ones come split from the host (the
// same bits as cv<dfl> of the binary64 value), the others by cv
template <class R> __device__ __forceinline__ R mconst(const DevModel &, int, double v) { return cv<R>(v); }
template <> __device__ __forceinline__ dfl mconst<dfl>(const DevModel &M, int q, double) { return dfl(M.dfc[q].x, M.dfc[q].y); }
__device__ __forceinline__ double to_d(double x) { return x; }
__device__ __forceinline__ double to_d(float x) { return f2d(x); }
__device__ __forceinline__ double to_d(dfl x) { return df2d(x); }

template <class R> __device__ __forceinline__ R rmax(R x, R y) { return x > y ? x : y; }
template <class R> __device__ __forceinline__ R rmin(R x, R y) { return x < y ? x : y; }
// a / b: the IEEE quotient (binary64 on the integer pipe)
template <class R> __device__ __forceinline__ R qdiv(R a, R b) { return a / b; }
template <> __device__ __forceinline__ double qdiv<double>(double a, double b) { return div_rn(a, b); }
// x 2^-E in the compute type: binary64 on the integer pipe (the exponent less E; zeros as they are,
// magnitudes at the ends of the range by the multiplication).  The rare branch holds no call, so that
// loads after it can be issued before it.
template <int E, class R> __device__ __forceinline__ R scale_down(R x) {
  if constexpr (std::is_same_v<R, double>) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const unsigned e = (unsigned)hi & 0x7ff00000u;
    const bool zero = (((unsigned)hi << 1) | (unsigned)lo) == 0u;
    double r = __hiloint2double(zero ? hi : hi - (E << 20), lo);
    if (!zero && e - ((unsigned)(E + 1) << 20) >= 0x7ff00000u - ((unsigned)(E + 1) << 20)) r = (1. / (1 << E)) * x;
    return r;
  } else {
    return R(1. / (1 << E)) * x;
  }
}
template <class R> __device__ __forceinline__ R half_of(R x) { return scale_down<1>(x); }
// 2 x likewise
template <class R> __device__ __forceinline__ R twice_of(R x) {
  if constexpr (std::is_same_v<R, double>) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const unsigned e = (unsigned)hi & 0x7ff00000u;
    const bool zero = (((unsigned)hi << 1) | (unsigned)lo) == 0u;
    double r = __hiloint2double(zero ? hi : hi + 0x00100000, lo);
    if (!zero && e - 0x00100000u >= 0x7fd00000u) r = 2. * x;
    return r;
  } else {
    return R(2.) * x;
  }
}

template <class R> struct RMath;
template <> struct RMath<double> {
  static __device__ __forceinline__ double log(const DevModel &M, double x) { return xlog(M, x); }
  static __device__ __forceinline__ double exp(const DevModel &M, double x) { return xexp(M, x); }
  static __device__ __forceinline__ double pow(const DevModel &M, double x, double y) { return xpow(M, x, y); }
  static __device__ __forceinline__ int cmp(double x1, double x2) { return fcmp(x1, x2); }
  static __device__ __forceinline__ double log_pow(const DevModel &M, double x, double y, double &lg) {
    if (!M.cr) { lg = ::log(x); return ::pow(x, y); }
    return cr_log_pow(x, y, *M.lt, lg);
  }
  static __device__ __forceinline__ double cos4(const DevModel &M, int j) { return M.coslat4[j]; }
};
template <> struct RMath<dfl> {
  static __device__ __forceinline__ dfl log(const DevModel &M, dfl x) { return log_df(x, M.exp2tab); }
  static __device__ __forceinline__ dfl exp(const DevModel &M, dfl x) { return exp_df(x, M.exp2tab); }
  static __device__ __forceinline__ dfl pow(const DevModel &M, dfl x, dfl y) { return exp_df(y * log_df(x, M.exp2tab), M.exp2tab); }
};
template <> struct RMath<float> {
  static __device__ __forceinline__ float log(const DevModel &, float x) { return logf(x); }
  static __device__ __forceinline__ float exp(const DevModel &, float x) { return expf(x); }
  static __device__ __forceinline__ float pow(const DevModel &, float x, float y) { return powf(x, y); }
  static __device__ __forceinline__ float log_pow(const DevModel &, float x, float y, float &lg) {
    lg = logf(x);
    return powf(x, y);
  }
  static __device__ __forceinline__ float cos4(const DevModel &M, int j) { return (float)M.coslat4[j]; }
  // fcmp with the float epsilon
  static __device__ __forceinline__ int cmp(float x1, float x2) {
    int e;
    frexpf(fabsf(x1) > fabsf(x2) ? x1 : x2, &e);
    const float delta = ldexpf(FLT_EPSILON, e);
    const float d = x1 - x2;
    return d > delta ? 1 : (d < -delta ? -1 : 0);
  }
};

// ---- the corrector of hsu_advection at one face (epic_flux.c:717-1484, all three directions) ----
//
// The reference splits the face's velocity into max(0, w) and min(0, w) and sums the corrections of
// both; one of the two is zero, and so is every finite term it multiplies.  hsu_face
// evaluates the upwind side alone: one square root and two quotients a face instead of two and
// three, half the products -- the same value, a zero term added nowhere changing it.
// w: the face's velocity; w_up: the velocity at the next face upstream; a_u, a_d: the field in the
// cells upstream and downstream; ap_d: the predicted field downstream; d_up: predicted minus field
// across the upstream face; aa: the squared second difference in the upstream cell; min_u, min_d: the
// field's floor in the two cells; c: the metric
// factor of the Courant number (times dt in the reference's order: |w| c DT).
template <class R> __device__ __forceinline__ bool is_neg(R w);   // the sign bit
template <> __device__ __forceinline__ bool is_neg<double>(double w) { return __double2hiint(w) < 0; }
template <> __device__ __forceinline__ bool is_neg<float>(float w) { return __float_as_int(w) < 0; }
template <class R> __device__ __forceinline__ R qsqrt(R x) { return sqrt(x); }
template <> __device__ __forceinline__ double qsqrt<double>(double x) { return sqrt_rn(x); }
// A term of the other side that is not finite makes the reference's sums NaNs (zero times it).  The kernels
// that hold a row or column add them where they can occur at all: a value that is not finite leaves its
// predicted one so, and a velocity the fluxes and predicted values beside it, so one look at the predicted
// values says whether the face fluxes have to be gone over (hsu_upwind_tainted, hsu_tainted).  With the look
// at every face instead, 12 steps of 128x64x20 took 10.13 ms against 10.04.
// the magnitude's bits from the exponent's top down, as an unsigned number, and its value from which on (infinity) a
// number is not finite
__device__ __forceinline__ unsigned top_bits(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
__device__ __forceinline__ unsigned top_bits(float x) { return (unsigned)__float_as_int(x) & 0x7fffffffu; }
template <class R> constexpr unsigned NONFINITE_BITS = std::is_same_v<R, double> ? 0x7ff00000u : 0x7f800000u;
template <class R> __device__ __forceinline__ bool nonfinite(R x) { return top_bits(x) >= NONFINITE_BITS<R>; }
template <class R> __device__ __forceinline__ R quiet_nan() { return std::is_same_v<R, double> ? R(__longlong_as_double(0x7ff8000000000000ll)) : R(__int_as_float(0x7fc00000)); }
// the face flux; w_dn: the velocity at the next face downstream; a_dd: the field in the cell beyond the
// downstream one (any finite number where there is none); ap_u: the predicted field upstream
template <class R>
__device__ __forceinline__ bool hsu_tainted(bool neg, R w_up, R w_dn, R a_dd, R ap_u) {
  if (max(max(top_bits(w_up), top_bits(w_dn)), max(top_bits(a_dd), top_bits(ap_u))) < NONFINITE_BITS<R>) return false;
  // an infinite velocity counts where its sign is that of the side it is split into
  return nonfinite(a_dd) || nonfinite(ap_u) || w_up != w_up || w_dn != w_dn || (nonfinite(w_dn) && is_neg(w_dn) != neg);
}
template <class R>
__device__ __forceinline__ R hsu_face(R w, R w_up, R a_u, R a_d, R ap_d, R d_up, R aa, R min_u, R min_d, R c, R DT) {
  const bool neg = is_neg(w);
  const R wu = is_neg(w_up) == neg ? w_up : R(0.);
  R f = half_of(w * (ap_d + a_u));
  R what = qsqrt<R>(w * wu);
  what = neg ? -what : what;
  const R mu = fabs(w) * c * DT;
  const R al = qdiv(R(1.) + mu, R(6.));
  R g = qdiv(aa, aa + (a_u - min_u) * (a_d - min_d));
  g = g * g;
  const R be = R(1.) + (qdiv(R(1.), twice_of(al)) - R(1.)) * g;
  return f + -al * (w * be * (ap_d - a_u) - what * (R(1.) - g) * d_up);
}
// the predictor's flux: the upwind cell's value carried by w (the other side's term is zero)
template <class R>
__device__ __forceinline__ R hsu_upwind(R w, R a_minus, R a_plus) { return w * (is_neg(w) ? a_minus : a_plus); }
template <class R>
__device__ __forceinline__ bool hsu_upwind_tainted(R w, R a_minus, R a_plus) { return nonfinite(is_neg(w) ? a_plus : a_minus); }

template <class R> __device__ __forceinline__ R rt(const DevModel &M, int j, int q);
template <> __device__ __forceinline__ double rt<double>(const DevModel &M, int j, int q) { return M.rt64[j * RT_COUNT + q]; }
template <> __device__ __forceinline__ float rt<float>(const DevModel &M, int j, int q) { return M.rt32[j * RT_COUNT + q]; }

// the three coefficients of d2dy2 of an order (2, 4, 6, 8) at row j
template <class R> __device__ __forceinline__ const R *visc_coef(const DevModel &M, int vgrid, int order, int j);
template <> __device__ __forceinline__ const double *visc_coef<double>(const DevModel &M, int vgrid, int order, int j) {
  return M.vt64 + ((vgrid ? M.nj + 2 : 0) + j) * 12 + 3 * (order / 2 - 1);
}
template <> __device__ __forceinline__ const float *visc_coef<float>(const DevModel &M, int vgrid, int order, int j) {
  return M.vt32 + ((vgrid ? M.nj + 2 : 0) + j) * 12 + 3 * (order / 2 - 1);
}

// 1 / n for a power of 2 (ni): a product with it is the quotient, without a division's chain of 64-cycle operations
__device__ __forceinline__ double inv_pow2(int n) { return __hiloint2double((1023 + __clz(n) - 31) << 20, 0); }

struct Trip { double x, y, z; };

__device__ __forceinline__ double pchst(double a, double b) {
  if (a == 0.0) return 0.0;
  if (a < 0.0) return b < 0.0 ? 1.0 : (b == 0.0 ? 0.0 : -1.0);
  return b < 0.0 ? -1.0 : (b == 0.0 ? 0.0 : 1.0);
}
// get_kin (the Suarez-Takacs blend for the Sadourney scheme, epic_funcs_diag.c:2694-2847) at h-point
// (j, i) of the layer planes Uk, Vk
template <class R>
__device__ __forceinline__ R kin_at(const DevModel &M, const double *Uk, const double *Vk, int j, int i) {
  const int jj = 2 * j;
  const R mn1 = cv<R>(M.mn[jj + 1]), mni0 = cv<R>(M.mn_inv[jj]), mni2 = cv<R>(M.mn_inv[jj + 2]);
  R u2 = cv<R>(Uk[M.at2(j, i)]), u4 = cv<R>(Uk[M.at2(j, i + 1)]), v2 = cv<R>(Vk[M.at2(j, i)]), v4 = cv<R>(Vk[M.at2(j + 1, i)]);
  const R kin_c = (u2 * u2 + u4 * u4 + mn1 * (v2 * v2 * mni0 + v4 * v4 * mni2)) * R(.25);
  if (j == 0 || j == M.nj) return kin_c;
  u2 = R(.5) * (cv<R>(Uk[M.at2(j + 1, i)]) + cv<R>(Uk[M.at2(j - 1, i)]));
  u4 = R(.5) * (cv<R>(Uk[M.at2(j + 1, i + 1)]) + cv<R>(Uk[M.at2(j - 1, i + 1)]));
  v2 = R(.5) * (cv<R>(Vk[M.at2(j, i + 1)]) + cv<R>(Vk[M.at2(j, i - 1)]));
  v4 = R(.5) * (cv<R>(Vk[M.at2(j + 1, i + 1)]) + cv<R>(Vk[M.at2(j + 1, i - 1)]));
  const R kin_s = (u2 * u2 + u4 * u4 + mn1 * (v2 * v2 * mni0 + v4 * v4 * mni2)) * R(.25);
  return (R(5.) / R(6.)) * kin_c + (R(1.) / R(6.)) * kin_s;
}
// Record the first model error (the reference would epic_error() and exit).
__device__ __forceinline__ void flag_error(Ctl *c, int code, int k, int j, int i, double v) {
  if (atomicCAS(&c->err_code, 0, code) == 0) {
    c->err_k = k; c->err_j = j; c->err_i = i; c->err_val = v;
  }
}

// The mixed forms' pressure gradient reads GZ3 and P2 as (hi, lo) binary32 splits, hi = float(x),
// lo = float(x - hi), kept in the scratch volumes work1 (GZ3) and work2 (P2) from the kernels that
// write the two fields before it (store_pgrad_vars and set_p2etc of stages 19 and 11, and the
// polar rows of GZ3 in uv_pgrad itself) to the pressure gradient.
__device__ __forceinline__ void put_split(double *work, long long x, double v) {
  const dfl d = d2df(v);
  reinterpret_cast<float2 *>(work)[x] = make_float2(d.hi, d.lo);
}

// Zonal periodicity of one row: pads i = 0 and i = ni+1 (bc_lateral, src/single/s_epic_functions.c:55-59).
// Called by the thread that owns interior cell i after it wrote the final value.
__device__ __forceinline__ void write_with_pads(double *a, const DevModel &M, long long rowbase, int i, double val) {
  a[rowbase + i] = val;
  if (i == M.ni) a[rowbase] = val;
  if (i == 1) a[rowbase + M.ni + 1] = val;
}

}  // namespace epic

// Kernel launch helpers.
#define EPIC_CUDA_CHECK(x)                                                     \
  do {                                                                         \
    cudaError_t e_ = (x);                                                      \
    if (e_ != cudaSuccess) return epic::set_error(EPIC_ERR_CUDA, "%s: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

inline unsigned epic_blocks(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

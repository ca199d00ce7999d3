// Launchers of the step kernels (each returns 0; launch errors surface through cudaGetLastError).
#pragma once
#include <cuda_runtime.h>
#include "device_common.cuh"
#include "epic_gb300.h"

namespace epic {

// Which time plane of a wind array a kernel works on; the index itself lives in Ctl so that
// one captured graph serves every step.
enum PlaneSel { PL_NONE = 0, PL_UV = 1, PL_UV_DIS = 2, PL_UV_TEND = 3 };

__device__ __forceinline__ int plane_offset(const DevModel &M, int sel) {
  const Ctl *c = M.ctl;
  switch (sel) {
    case PL_UV: return c->it_uv * (int)M.n3;
    case PL_UV_DIS: return c->it_uv_dis * (int)M.n3;
    case PL_UV_TEND: return c->it_uv_tend * (int)M.n3;
    default: return 0;
  }
}

// Grid of a launch over every member of a batch: blockIdx.z selects the member (one member
// when the model is not a batch).
inline dim3 zg(dim3 g, const DevModel &M) {
  g.z = M.nbatch > 1 ? (unsigned)M.nbatch : 1u;
  return g;
}

// Kernels that march up the rows: thread = one column i of one level, ROWS latitude rows from
// j0 = jlo + blockIdx.y ROWS (per member), carrying what neighbouring rows share -- values already loaded and
// converted, the products and faces between two rows -- in registers.  As many rows a thread as leave
// 512 threads per SM, up to 4; a template parameter, so that a single row is straight code.
inline int march_rows(const DevModel &M, int nkk) {
  const long long cells = (long long)M.ni * nkk * (M.nj + 1) * (M.nbatch > 1 ? M.nbatch : 1);
  return cells >= 4LL * M.sms * 512 ? 4 : (cells >= 2LL * M.sms * 512 ? 2 : 1);
}
struct March { int k, i, j0, j1; };
// rows jlo..jhi; false for a thread without work
template <int ROWS>
__device__ __forceinline__ bool march(const DevModel &M, int k0, int nkk, int jlo, int jhi, March &s) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, ni = (unsigned)M.ni;
  s.j0 = jlo + (int)blockIdx.y * ROWS;
  s.j1 = ROWS == 1 ? s.j0 : min(s.j0 + ROWS - 1, jhi);
  if (t >= (unsigned)nkk * ni || s.j0 > jhi) return false;
  s.k = k0 + (int)(t / ni);
  s.i = 1 + (int)(t - (unsigned)(s.k - k0) * ni);
  return true;
}
#define EPIC_MARCH_R(R, kern, nkk, nrows, block, stream, ...)                                                         \
  do {                                                                                                                \
    const int rows_ = march_rows(M, (nkk));                                                                           \
    const dim3 grid_ = zg(dim3(epic_blocks((long long)(nkk) * M.ni, (block)), epic_blocks((nrows), rows_)), M);       \
    if (rows_ == 4) kern<R, 4><<<grid_, (block), 0, (stream)>>>(__VA_ARGS__);                                         \
    else if (rows_ == 2) kern<R, 2><<<grid_, (block), 0, (stream)>>>(__VA_ARGS__);                                    \
    else kern<R, 1><<<grid_, (block), 0, (stream)>>>(__VA_ARGS__);                                                    \
  } while (0)
#define EPIC_MARCH(mixed, kern, nkk, nrows, block, stream, ...)                                                       \
  do {                                                                                                                \
    if (mixed) EPIC_MARCH_R(float, kern, nkk, nrows, block, stream, __VA_ARGS__);                                     \
    else EPIC_MARCH_R(double, kern, nkk, nrows, block, stream, __VA_ARGS__);                                          \
  } while (0)

// Launch the FP32 (mixed form) or FP64 instantiation of a kernel template over every member
// (the launcher's `M` sets the batch).
#define EPIC_LAUNCH_R(mixed, kern, grid, block, smem, stream, ...)                              \
  do {                                                                                          \
    if (mixed) kern<float><<<zg((grid), M), (block), (smem), (stream)>>>(__VA_ARGS__);          \
    else kern<double><<<zg((grid), M), (block), (smem), (stream)>>>(__VA_ARGS__);              \
  } while (0)

// k_filter.cu -- zonal filter (epic_adjust.c) and the zonal pass of hsu_advection.
// fp32: filter in FP32 (the mixed forms; on the tensor cores for ni a multiple of 128).
// shift (tensor-core path only): filter x - x(i=1) of each row and add x(i=1) back in binary64,
// for fields whose zonal variations are small beside their value (the geopotential).
// filtered_rows_only: on the tensor-core path only the rows the filter changes are written (an in-place
// call whose rows 0..nj(+1) already carry their periodic pads, or one beside launch_filter_rest).
int launch_filter_planes(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s,
                         int fp32 = 0, int shift = 0, int filtered_rows_only = 0);
// The other rows of an out-of-place call (the tensor-core path; nothing on the others): copied, with their
// pads, on a stream of their own choice.
int launch_filter_rest(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s, int fp32);
int launch_varz_filter(const DevModel &M, double *buff, int sel, int index, int kstart, int kend, cudaStream_t s);
int launch_hsu_zonal(const DevModel &M, double *buff, int kind, int kstart, cudaStream_t s);
int filter_kernels_init(int ni);
// k_filter_gemm.cu -- the plane filter as a tcgen05 (3xTF32) operator product, mixed form
bool filter_gemm_usable(const DevModel &M);
int launch_filter_planes_gemm(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s,
                              int shift = 0);
int filter_gemm_init(int ni);

// k_column_acc.cu -- set_p2etc and store_pgrad_vars (column part) of the mixed form, with the
// quantities feeding the pressure gradient in double-float.
__global__ void k_set_p2etc_acc(DevModel M, int update_theta, int layers);
__global__ void k_pgrad_vars_column_acc(DevModel M);
__global__ void k_gz3_column_acc(DevModel M);   // GZ3 alone (the call before the filtered-GZ copy)
__global__ void k_pgrad_vars_column_acc_h2(DevModel M);   // the two above with hydrogen thermodynamics
__global__ void k_gz3_column_acc_h2(DevModel M);
int column_acc_kernels_init();
void fill_filter_kernels(int ni, int nj, const double *hl_h, const double *hl_pv, long long iadim, float *fh, float *fv);
bool filter_operator_wanted(const epic_grid &g, int precision);
size_t filter_operator_bytes(const epic_grid &g);
int filter_operator_create(const epic_grid &g, const double *hl_h, const double *hl_pv, long long iadim, cudaStream_t s, DevModel &d,
                           void **mem, uint64_t *hash, const char **why);
void filter_operator_release(void *mem);
size_t twiddle_doubles(int ni);
void fill_twiddles(int ni, double *tw);

// k_column.cu -- vertical (column) work
int launch_source_sink(const DevModel &M, cudaStream_t s);
// with_source_sink: source_sink first, in the same kernel (the step calls the two in a row)
int launch_calc_w(const DevModel &M, cudaStream_t s, bool with_source_sink = false);
int launch_uv_drag(const DevModel &M, cudaStream_t s);
int launch_hsu_vertical(const DevModel &M, double *buff, int kind, cudaStream_t s);
int launch_restore_mass(const DevModel &M, cudaStream_t s);
// early: the step's calls inside advection (set_p2etc) and before the filtered-GZ copy
// (store_pgrad_vars), whose outputs but P3, HDRY and GZ3 stage 11 and stage 19 rewrite before
// anything reads them: only those are computed (EPIC_PREC_MIXED with its
// double-float kernels, which also leave the interfaces' logarithms for store_pgrad_vars:
// GZ3 places the 3-D filter's profiles, so it needs their accuracy; EPIC_PREC_MIXED_FAST with
// its FP32 ones; the FP64 form in binary64, where a power takes as long as ten products).
int launch_set_p2etc(const DevModel &M, int update_theta, cudaStream_t s, bool early = false);
// dzdt: its horizontal part of DZDT3 too (launch_pgrad_dzdt).
int launch_store_pgrad_vars(const DevModel &M, cudaStream_t s, bool early = false, bool dzdt = true);
int launch_pgrad_dzdt(const DevModel &M, cudaStream_t s);
int launch_gz_monotone(const DevModel &M, cudaStream_t s);
int launch_calc_heating(const DevModel &M, cudaStream_t s);
int launch_advection_prep(const DevModel &M, int phase, cudaStream_t s);
int column_kernels_init(int nk);

// k_stencil.cu -- horizontal stencils and the time update
// the row tables (DevModel::rt64, rt32, vt64, vt32) from the 1-D grid arrays; once per model
int launch_row_tables(const DevModel &M, cudaStream_t s);
int launch_zero_tend(const DevModel &M, cudaStream_t s);
int launch_uv_core(const DevModel &M, cudaStream_t s);
// uv_pgrad_finite_volume: GZ3's pole rows, then DUDT (lon) and DVDT (lat), independent of each other
int launch_pgrad_poles(const DevModel &M, cudaStream_t s);
int launch_pgrad_lon(const DevModel &M, cudaStream_t s);
int launch_pgrad_lat(const DevModel &M, cudaStream_t s);
int launch_hsu_meridional(const DevModel &M, double *buff, int kind, cudaStream_t s);
enum HsuForm { HSU_MARCH = 1, HSU_PASSES = 2, HSU_TILES = 3 };   // the tuning table's TB_HSU_MERID_VARIANT (0: by size)
int hsu_meridional_form(const DevModel &M, int nkk);             // the form that nkk planes take
// akima_advection (epic_flux.c:1502-1940), the other advection scheme: vertical (k_column.cu),
// meridional (k_stencil.cu) and zonal (k_filter.cu) passes, arguments as their Hsu counterparts
int launch_akima_vertical(const DevModel &M, double *buff, int kind, cudaStream_t s);
int launch_akima_meridional(const DevModel &M, double *buff, int kind, cudaStream_t s);
int launch_akima_zonal(const DevModel &M, double *buff, int kind, int kstart, cudaStream_t s);
// meridional, then zonal hyperviscosity; index: 0 = U, 1 = V, 2 = HDRY (with restore_mass), 3 = THETA, 4 = NU_TURB
int launch_hyperviscosity(const DevModel &M, int index, double *var, int sel, cudaStream_t s);
int stencil_kernels_init();
int launch_divergence_damping(const DevModel &M, cudaStream_t s);
// the time update: which scheme coefficients this step takes (decide: from the tendency planes of
// earlier steps alone), the update, the rotation of the time-plane indices
int launch_uv_decide(const DevModel &M, cudaStream_t s);
int launch_uv_update(const DevModel &M, cudaStream_t s);
int launch_uv_rotate(const DevModel &M, cudaStream_t s);
// store_diag: the filtered copies of V (into work1) and U (into work2), PV3 from the first with its
// polar values, DIV_UV3 from the second, RI2
int launch_diag_filter_v(const DevModel &M, cudaStream_t s, cudaStream_t rest);   // rest: launch_filter_rest's stream
int launch_diag_filter_u(const DevModel &M, cudaStream_t s, cudaStream_t rest);
int launch_diag_pv(const DevModel &M, cudaStream_t s);
int launch_diag_pv_poles(const DevModel &M, cudaStream_t s);
int launch_diag_div(const DevModel &M, cudaStream_t s);
int launch_diag_ri2(const DevModel &M, cudaStream_t s);
int launch_itime_advance(const DevModel &M, cudaStream_t s);
int launch_set_itime(const DevModel &M, long long itime, cudaStream_t s);

// k_turb.cu -- the Spalart-Allmaras DES turbulence closure (FP64 form): source_sink_turb,
// scalar_horizontal_diffusion (with its set_p2etc), scalar_vertical_diffusion (with its
// set_p2etc), uv_horizontal_diffusion, uv_vertical_diffusion, set_diffusion_coef, and
// restore_mass(NU_TURB_INDEX); scratch work0..3 and the model's turbulence arrays
int launch_source_sink_turb(const DevModel &M, cudaStream_t s);
int launch_theta_hdiff(const DevModel &M, cudaStream_t s, bool early);   // with the set_p2etc that follows (early: launch_set_p2etc's)
int launch_nu_hdiff(const DevModel &M, cudaStream_t s);      // with restore_mass
int launch_tau_wall_h(const DevModel &M, cudaStream_t s);   // NU_TURB's wall stresses, of the winds, GZ3 and RHO3 alone
int launch_theta_vdiff(const DevModel &M, cudaStream_t s, bool early);   // with the set_p2etc that follows
int launch_nu_vdiff(const DevModel &M, cudaStream_t s);   // with restore_mass
int turb_kernels_init(int device, int *cluster);   // on the current device; *cluster: DevModel::sa_cluster
// uv_horizontal_diffusion: COEFFD and H_RHO; the filtered copies of them (0, 1: after coef), U and V (2, 3); the rest
int launch_uvh_coef(const DevModel &M, cudaStream_t s);
int launch_uvh_filter(const DevModel &M, int which, cudaStream_t s);
int launch_uvh_apply(const DevModel &M, cudaStream_t s);
int launch_uv_vdiff(const DevModel &M, cudaStream_t s);
int launch_set_diffusion_coef(const DevModel &M, cudaStream_t s);
int launch_restore_nu(const DevModel &M, cudaStream_t s);
// cfl_dt's three limits as the bits of positive binary64 values, minimised into lim[0..2]
// (x, y, z), which the caller sets to DBL_MAX's bits first
int launch_cfl_dt(const DevModel &M, unsigned long long *lim, cudaStream_t s);

}  // namespace epic

// The Spalart-Allmaras DES turbulence closure of the FP64 form: source_sink_turb, the horizontal
// and vertical subgrid diffusion of THETA, NU_TURB and the winds, and set_diffusion_coef
// (src/shared/epic_subgrid.c), with crank_nicolson's banded solve (src/shared/epic_funcs_util.c).
// Every expression is the reference's, in its order, in binary64 with the correctly rounded
// log/exp/pow/atan/cos of dd_math.cuh, so each kernel's output equals the CPU restatement's bit
// for bit.  The parallel decomposition is this file's own:
//   - source_sink_SA updates NU_TURB in place in K, J, I order (each point reads the new values of
//     its K-1, J-1 and I-1 neighbours, the old ones of K+1, J+1, I+1).  Its NU_TURB-free part
//     (strain, wall distance, Brunt-Vaisala frequency) is one pointwise pass; the rest runs as
//     wavefronts K + J + I = d, every point of a front independent of the others, in one kernel per
//     model whose blocks form a cluster with a barrier between fronts;
//   - the Laplacians of laplacian_h are three pointwise passes around the row filter, all layers
//     at once (each layer's Laplacian reads only its own plane);
//   - the implicit vertical diffusions take a tile of 32 columns per block: the set-up of the bands and
//     the residual are pointwise in the levels, the band solver's recurrences one warp's;
//   - uv_horizontal_diffusion's stresses are recomputed where the wind updates read them.
#include <map>
#include <mutex>
#include "device_common.cuh"
#include "kernels.h"
#include "epic_common.h"
#include "epic_gb300.h"

namespace epic {

namespace {

constexpr double SA_CV1_3 = 7.1 * 7.1 * 7.1;   // cv1^3, epic_subgrid.c:2186-2187
enum { WALL_U, WALL_V, WALL_H };               // law_of_the_wall's grids: U_INDEX, V_INDEX, the h-grid

__device__ __forceinline__ double nu_floor(const DevModel &M) { return 1.e-4 * M.kinvisc; }

// D_WALL as dwall_SA sets it before each use (:2716-2770): the height above the surface, or
// FLOAT_MAX on a gas giant
__device__ __forceinline__ double d_wall(const DevModel &M, int k, int j, int i) {
  if (M.gas_giant) return DBL_MAX;
  return div_rn(M.gz3[M.at(k, j, i)] - M.topo_scale * M.gz_surface[M.at2(j, i)], M.grav[2 * j + 1]);
}

__device__ __forceinline__ double limit_range(double lo, double x, double hi) { return x < lo ? lo : (x > hi ? hi : x); }

// func_utau, :3112-3165
__device__ double func_utau(const DevModel &M, double u_tau, double u_tan, double dwall, int j, int i) {
  const double C = 5., const1 = 0.127, const2 = 1. / .41, const3 = 0.41 * 1.43e-3, one_third = 1. / 3., pi_six = M_PI / 6.;
  const double sqrt_one_third = sqrt(1. / 3.);
  const MathTable &T = *M.lt;
  double u_plus = 0.;
  if (u_tau != 0.) u_plus = div_rn(u_tan, u_tau);
  else flag_error(M.ctl, ERR_TURB, -1, j, i, u_tau);
  const double y_plus = fabs(div_rn(u_tau * dwall, M.kinvisc));
  if (u_plus < 0.1) return 1.e+20;
  if (y_plus < 5.) return y_plus - u_plus;
  if (y_plus < 70.) {
    const double yy = const1 * y_plus;
    return div_rn(one_third * cr_log(div_rn(1. + yy, sqrt_rn(yy * (yy - 1.) + 1.)), T) +
                      sqrt_one_third * (cr_atan(sqrt_one_third * (2. * yy - 1.), T) + pi_six), const1) +
           .25 * const2 * cr_log(1. + const3 * cr_pow(y_plus, 4., T), T) - u_plus;
  }
  return const2 * cr_log(y_plus, T) + C - u_plus;
}

// law_of_the_wall, :2995-3105: secant iterations on the wall law for the friction velocity
// (the reference scales its t_vis argument by fv1 and leaves it unused)
__device__ double law_of_the_wall(const DevModel &M, int k, int j, int i, int index, double u_tan) {
  const double kinvisc = M.kinvisc, tol = 1.e-6;
  if (M.gas_giant) return 1.0e-4 * kinvisc;
  double dwall;
  if (index == WALL_U) dwall = 0.5 * (d_wall(M, k, j, i) + d_wall(M, k, j, i - 1));
  else if (index == WALL_V) dwall = 0.5 * M.m[2 * j] * (div_rn(d_wall(M, k, j, i), M.m[2 * j + 1]) + div_rn(d_wall(M, k, j - 1, i), M.m[2 * j - 1]));
  else dwall = d_wall(M, k, j, i);
  if (dwall * u_tan < 0.00023) return 0.01 * kinvisc;
  double dwall_inv = 0.;
  if (dwall > 0.) dwall_inv = div_rn(1., dwall);
  else flag_error(M.ctl, ERR_TURB, k, j, i, dwall);
  const double x1 = sqrt_rn(kinvisc * (1. + 0.01) * u_tan * dwall_inv);
  const double x2 = sqrt_rn(kinvisc * (1. + 20.) * u_tan * dwall_inv);
  double fl = func_utau(M, x1, u_tan, dwall, j, i), f = func_utau(M, x2, u_tan, dwall, j, i), rts, xl;
  if (fabs(fl) < fabs(f)) {
    rts = x1; xl = x2;
    const double sw = fl; fl = f; f = sw;
  } else {
    xl = x1; rts = x2;
  }
  double u_tau = 0.;
  int iter;
  for (iter = 0; iter < 30; iter++) {
    const double dx = div_rn((xl - rts) * f, f - fl);
    xl = rts;
    fl = f;
    rts += dx;
    f = func_utau(M, rts, u_tan, dwall, j, i);
    if (f > .99e+20) return 0.01 * kinvisc;
    if (fabs(dx) < tol || f == 0.0) {
      u_tau = rts;
      break;
    }
  }
  if (iter < 30) return dmaxr(div_rn(u_tau * u_tau * dwall, u_tan) - kinvisc, 0.01 * kinvisc);
  return 20. * kinvisc;
}

// invert_fv1, :3172-3226
__device__ double invert_fv1(const DevModel &M, double t_vis, int j, int i) {
  const double pi_factor = M_PI * 0.5 / 30.0;
  if (t_vis < 0.) flag_error(M.ctl, ERR_TURB, -1, j, i, t_vis);
  const double chi = div_rn(t_vis, M.kinvisc);
  if (chi > 30) return t_vis;
  if (chi < 0.4) return M.kinvisc * cr_pow(chi * SA_CV1_3, .25, *M.lt);
  double fv1 = cr_cos(pi_factor * cr_pow(chi, 0.35, *M.lt), *M.lt);
  fv1 = 1.0 - fv1 * fv1;
  return div_rn(M.kinvisc * chi, fv1);
}

// get_kin at h-point (j, i) of layer k of the wind time plane `sel`; i = 0 is the pad (bc_lateral)
__device__ __forceinline__ double kin_plane(const DevModel &M, int sel, int k, int j, int i) {
  if (i == 0) i = M.ni;
  const long long off = plane_offset(M, sel) + (long long)k * M.n2;
  return kin_at<double>(M, M.u + off, M.v + off, j, i);
}

// The wall stress of tau_surface (:2819-2988) under the wind component `index` at (j, i), from
// layer K = nk-1 and the winds of plane it_uv
__device__ double tau_wall(const DevModel &M, int index, int j, int i) {
  if (M.gas_giant) return 0.;
  const int k = M.nk - 1;
  const double *U = M.u + plane_offset(M, PL_UV), *V = M.v + plane_offset(M, PL_UV);
  auto rho3 = [&](int jj, int ii) { return M.rho3[M.at(k, jj, ii)]; };
  auto gz = [&](int kk, int jj, int ii) { return M.gz3[M.at(kk, jj, ii)]; };
  if (index == WALL_U) {
    const double rho = .5 * (rho3(j, i) + rho3(j, i - 1));
    const double dz = div_rn(.5 * (gz(k, j, i) + gz(k, j, i - 1) - gz(k + 1, j, i) - gz(k + 1, j, i - 1)), M.grav[2 * j + 1]);
    const double kin = .5 * (kin_plane(M, PL_UV, k, j, i) + kin_plane(M, PL_UV, k, j, i - 1));
    const double u_tan = sqrt_rn(2. * kin);
    const double dc = law_of_the_wall(M, k, j, i, WALL_U, u_tan);
    return div_rn((M.dynvisc + rho * dc) * (U[M.at(k, j, i)] - 0.), dz);
  }
  if (index == WALL_V) {
    const double rho = .5 * (rho3(j, i) + rho3(j - 1, i));
    const double dz = div_rn(.5 * (gz(k, j, i) + gz(k, j - 1, i) - gz(k + 1, j, i) - gz(k + 1, j - 1, i)), M.grav[2 * j]);
    const double kin = .5 * (kin_plane(M, PL_UV, k, j, i) + kin_plane(M, PL_UV, k, j - 1, i));
    const double u_tan = sqrt_rn(2. * kin);
    const double dc = law_of_the_wall(M, k, j, i, WALL_V, u_tan);
    return div_rn((M.dynvisc + rho * dc) * (V[M.at(k, j, i)] - 0.), dz);
  }
  const double rho = rho3(j, i);
  const double dz = div_rn(gz(k, j, i) - gz(k + 1, j, i), M.grav[2 * j + 1]);
  const double kin = kin_plane(M, PL_UV, k, j, i);
  const double u_tan = sqrt_rn(2. * kin);
  const double dc = law_of_the_wall(M, k, j, i, WALL_H, u_tan);
  const double nu = invert_fv1(M, dc, j, i);
  return div_rn((M.dynvisc + rho * nu) * (u_tan - 0.), dz);
}

// ---------------------------------------------------------------------------------------------
// source_sink_SA, :2434-2711
// ---------------------------------------------------------------------------------------------

// get_brunt2 on the interface kk = 2k+1, 1 <= k < nk (np = 1, fpara off, Held-Suarez cp),
// epic_funcs_diag.c:2885-3075
__device__ double brunt2_iface(const DevModel &M, int k, int j, int i) {
  const long long x = M.at(k, j, i);
  const double pressure = M.p3[x], temperature = M.t3[x], density = M.rho3[x];
  const double cp = 1004., mu = M.mu_dry;
  const double deltap = 0.001 * pressure, deltaT = 0.001 * temperature;
  auto dens = [&](double p, double t) { return div_rn(p * mu, 8.314472e+3 * t); };   // return_density
  const double drho_dp_T = div_rn(dens(pressure + deltap, temperature) - dens(pressure - deltap, temperature), 2. * deltap);
  const double drho_dT_p = div_rn(dens(pressure, temperature + deltaT) - dens(pressure, temperature - deltaT), 2. * deltaT);
  const double Drho_Dp = div_rn(M.rho2[M.at(k + 1, j, i)] - M.rho2[x], M.p2[M.at(k + 1, j, i)] - M.p2[x]);
  const double g = M.grav[2 * j + 1];
  return g * g * (Drho_Dp - drho_dp_T + div_rn(temperature, cp * density * density) * drho_dT_p * drho_dT_p);
}

// Everything of a point's update but the three gradient terms, at every point k = 1..nk-1,
// j = 0..nj, i = 1..ni: the terms that read only the point's own NU_TURB (which the sweep has not
// changed when it reaches the point) and the NU_TURB-free strain, wall distance and buoyancy.
// work0 = the production cb1 S~ NU, work1 = the destruction cw1 fw (NU/d~)^2, work3 = the buoyancy
// term (0 where N^2 >= 0, which subtracts nothing), work2 = 1/dz.
__global__ void k_sa_prep(DevModel M) {
  if (epic_member(M)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  if (t >= (unsigned)(M.nk - 1) * nr * ni) return;
  const unsigned r = t / ni, q = r / nr;
  const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = 1 + (int)q;
  const double cw2 = 0.3, cw3_6 = 64., cb1 = 0.1355, cb2 = 0.622, sigma = 2. / 3., kappa = 0.41;
  const double kappa_2 = kappa * kappa, cw1 = (cb1 / kappa_2) + ((1. + cb2) / sigma), nu_turb_limiter = 3000.;
  const MathTable &T = *M.lt;
  const long long off = plane_offset(M, PL_UV_DIS);
  const double *U = M.u + off, *V = M.v + off;
  auto u = [&](int kk, int jj, int ii) { return U[M.at(kk, jj, ii)]; };
  auto v = [&](int kk, int jj, int ii) { return V[M.at(kk, jj, ii)]; };
  auto w3 = [&](int kk, int jj, int ii) { return M.w3[M.at(kk, jj, ii)]; };
  auto gz3 = [&](int kk) { return M.gz3[M.at(kk, j, i)]; };
  const int jj = 2 * j, kk = 2 * k + 1;
  const double m_2jp1 = M.m[jj + 1], n_2jp1 = M.n[jj + 1];
  // delta_SA (:2774-2808), for k < nk
  const double dx = div_rn(1., M.m[jj + 1]), dy = div_rn(1., M.n[jj + 1]);
  const double dz = div_rn(gz3(k - 1) - gz3(k + 1), M.grav[jj + 1]);
  double delta = dminr(dx, dy);
  delta = dminr(delta, dz);
  const double d_tilda = dminr(d_wall(M, k, j, i), 0.65 * delta);
  const double dz_inv = div_rn(M.grav[jj + 1], gz3(k - 1) - gz3(k + 1));
  // U on the v-grid (zero on the polar rows) and V on the u-grid, layer k
  auto u2d = [&](int J) -> double {
    if (J == 0 || J == M.nj + 1) return 0.;
    const int JJ = 2 * J;
    const double inv_m = div_rn(1., M.mn[JJ - 1]), inv_p = div_rn(1., M.mn[JJ + 1]), mn_v = div_rn(.5, inv_m + inv_p);
    return ((u(k, J, i) + u(k, J, i + 1)) * inv_p + (u(k, J - 1, i) + u(k, J - 1, i + 1)) * inv_m) * mn_v;
  };
  auto v2d = [&](int I) -> double {
    if (I == M.ni + 1) I = 1;
    const double inv_m = div_rn(1., M.mn[jj]), inv_p = div_rn(1., M.mn[jj + 2]), mn_u = div_rn(.5, inv_m + inv_p);
    return ((v(k, j, I) + v(k, j, I - 1)) * inv_m + (v(k, j + 1, I) + v(k, j + 1, I - 1)) * inv_p) * mn_u;
  };
  const double s11 = (u(k, j, i + 1) - u(k, j, i)) * m_2jp1;
  const double s22 = (v(k, j + 1, i) - v(k, j, i)) * n_2jp1;
  const double s33 = div_rn(w3(k - 1, j, i) - w3(k + 1, j, i), M.sgth[kk - 2] - M.sgth[kk + 2]);
  const double s12 = .5 * ((u2d(j + 1) - u2d(j)) * n_2jp1 + (v2d(i + 1) - v2d(i)) * m_2jp1);
  const double u_var3 = 0.5 * (u(k + 1, j, i) + u(k + 1, j, i + 1));
  const double u_var1 = 0.5 * (u(k - 1, j, i) + u(k - 1, j, i + 1));
  double w_var3 = 0.5 * (w3(k, j, i) + w3(k, j, i + 1));
  double w_var1 = 0.5 * (w3(k, j, i) + w3(k, j, i - 1));
  const long long x = M.at(k, j, i);
  const double h_rho = div_rn(M.h3[x], M.rho3[x]);
  const double s13 = .5 * ((u_var1 - u_var3) * dz_inv + h_rho * (w_var3 - w_var1) * m_2jp1);
  const double v_var3 = 0.5 * (v(k + 1, j, i) + v(k + 1, j + 1, i));
  const double v_var1 = 0.5 * (v(k - 1, j, i) + v(k - 1, j + 1, i));
  w_var3 = 0.5 * (w3(k, j, i) + w3(k, j + 1, i));
  w_var1 = 0.5 * (w3(k, j, i) + w3(k, j - 1, i));
  const double s23 = .5 * ((v_var1 - v_var3) * dz_inv + h_rho * (w_var3 - w_var1) * n_2jp1);
  const double S = sqrt_rn(2. * (s11 * s11 + s22 * s22 + s33 * s33 + 2. * (s12 * s12 + s13 * s13 + s23 * s23)));
  // the point's own NU_TURB terms
  const double nu = M.nu_turb[x];
  const double chi = div_rn(nu, M.kinvisc);
  const double chi3 = cr_pow(chi, 3., T);
  const double fv1 = div_rn(chi3, chi3 + SA_CV1_3);
  const double fv2 = 1. - div_rn(chi, 1. + chi * fv1);
  const double tmp1 = kappa_2 * d_tilda * d_tilda;
  const double S_tilda = S + div_rn(nu * fv2, tmp1);
  const double tmp2 = S_tilda * tmp1;
  double fw = 1.;
  if (tmp2 != 0.) {
    const double r_sa = div_rn(nu, tmp2);
    if (r_sa < 0.) flag_error(M.ctl, ERR_TURB, k, j, i, r_sa);
    else if (r_sa < 10.) {
      const double g_sa = r_sa + cw2 * (cr_pow(r_sa, 6., T) - r_sa);
      fw = g_sa * cr_pow(div_rn(1. + cw3_6, cr_pow(g_sa, 6., T) + cw3_6), (1. / 6.), T);
    }
  }
  const double brunt2 = brunt2_iface(M, k, j, i);
  const double brunt = sqrt_rn(fabs(brunt2));
  M.work0[x] = cb1 * S_tilda * nu;
  M.work1[x] = cw1 * fw * cr_pow(div_rn(nu, d_tilda), 2., T);
  M.work2[x] = dz_inv;
  M.work3[x] = brunt2 < 0. ? div_rn(nu * cr_exp(div_rn(-nu, nu_turb_limiter), T) * brunt2, brunt) : 0.;
}

// The wavefronts k + j + i = d of the in-place NU_TURB update: the three gradient terms from the
// neighbours (new at k-1, j-1, i-1; old at k+1, j+1, i+1), summed in the reference's order between
// the point's own terms.  One cluster of blocks per model, a cluster barrier between fronts: bounded by
// that chain of nk + nj + ni - 2 fronts, where a launch per front cost 5.5 us (210 launches a step at
// 128x64x20).  A thread keeps one (k, j) pair and walks along i with the fronts, so that a front waits
// only for the two new neighbours of other threads (read past L1, an L2 round trip), the arithmetic that
// needs them and the barrier: the rest -- old neighbours, which no front before the next but one changes,
// and the point's own terms -- is loaded a front ahead, its own last value is in a register.  Pairs beyond
// the cluster's threads take further sweeps over their share with everything loaded in the front.
constexpr int SA_THREADS = 128;
struct SaPoint { double north, east, above, w0, w1, w2, w3; };
__global__ void __launch_bounds__(SA_THREADS) k_sa_waves(DevModel M) {
  if (epic_member(M)) return;   // all blocks of a cluster are one member's
  const int nr = M.nj + 1, pairs = (M.nk - 1) * nr, ni = M.ni, n2 = (int)M.n2, row = M.iadim;
  const double c = 0.622 / (2. / 3.), floor_nu = 1.e-4 * M.kinvisc;   // cb2 / sigma
  double *NU = M.nu_turb;
  const int me = (int)(threadIdx.x * gridDim.x + blockIdx.x), all = (int)(gridDim.x * blockDim.x);   // fronts spread over the blocks
  auto load = [&](int x) {
    SaPoint p;
    p.north = NU[x + row]; p.east = NU[x + 1]; p.above = NU[x + n2];
    p.w0 = M.work0[x]; p.w1 = M.work1[x]; p.w2 = M.work2[x]; p.w3 = M.work3[x];
    return p;
  };
  auto update = [&](const SaPoint &p, int x, int jj, double nu, double west) {
    const double below = __ldcg(NU + x - n2), south = __ldcg(NU + x - row);
    const double g1 = half_of((p.east - west) * M.m[jj + 1]);
    const double g2 = half_of((p.north - nu) * M.n[jj + 2] + (nu - south) * M.n[jj]);
    const double g3 = (below - p.above) * p.w2;
    double dnudt = p.w0;
    dnudt += c * (g1 * g1);   // pow(g, 2.), the correctly rounded square
    dnudt += c * (g2 * g2);
    dnudt += c * (g3 * g3);
    dnudt -= p.w1;
    dnudt -= p.w3;
    const double v = dmaxr(floor_nu, nu + M.dt * dnudt);
    NU[x] = v;
    return v;
  };
  const bool mine = me < pairs;
  const int k0 = mine ? 1 + me / nr : 1, j0 = mine ? me - (k0 - 1) * nr : 0, x0 = M.at(k0, j0, 0);
  SaPoint next = {};
  double nu = 0., west = 0.;   // the pair's value at its next i, and the one just written before it
  if (mine) { next = load(x0 + 1); nu = NU[x0 + 1]; west = NU[x0]; }
  for (int d = 2; d <= M.nk - 1 + M.nj + ni; d++) {
    const int i = d - k0 - j0;
    if (mine && i >= 1 && i <= ni) {
      const SaPoint p = next;
      const double now = nu;
      if (i < ni) { next = load(x0 + i + 1); nu = p.east; }
      west = update(p, x0 + i, 2 * j0, now, west);
    }
    for (int q = me + all; q < pairs; q += all) {
      const int k = 1 + q / nr, j = q - (k - 1) * nr, iq = d - k - j;
      if (iq < 1 || iq > ni) continue;
      const int x = M.at(k, j, iq);
      update(load(x), x, 2 * j, __ldcg(NU + x), __ldcg(NU + x - 1));
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
}

// The solid-surface block (:2690-2704): NU_TURB(nk) = MAX(1e-4 kinvisc, NU_TURB(nk-1)) (the
// reference computes law_of_the_wall and invert_fv1 there first and then overwrites their result)
__global__ void k_sa_bottom(DevModel M) {
  if (epic_member(M)) return;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= (M.nj + 1) * M.ni) return;
  const int j = t / M.ni, i = 1 + t - j * M.ni;
  M.nu_turb[M.at(M.nk, j, i)] = dmaxr(nu_floor(M), M.nu_turb[M.at(M.nk - 1, j, i)]);
}

// bc_lateral of layers k0..k1, rows 0..nj+1 (src/single/s_epic_functions.c:39-87)
__global__ void k_pads(DevModel M, double *a, int k0, int k1) {
  if (epic_member(M, a)) return;
  const int nr = M.nj + 2;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= (k1 - k0 + 1) * nr) return;
  const int k = k0 + t / nr, j = t - (k - k0) * nr;
  const long long b = M.at(k, j, 0);
  a[b] = a[b + M.ni];
  a[b + M.ni + 1] = a[b + 1];
}

// restore_mass(NU_TURB_INDEX), epic_adjust.c:80-88: layers 0..nk+1, rows 0..nj, every column
__global__ void k_restore_nu(DevModel M) {
  if (epic_member(M)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned w = (unsigned)(M.nj + 1) * (unsigned)M.iadim;
  if (t >= w * (unsigned)(M.nk + 2)) return;
  const unsigned q = t / w;
  const long long x = M.at((int)q, 0, 0) + (t - q * w);
  M.nu_turb[x] = dmaxr(nu_floor(M), M.nu_turb[x]);
}

// ---------------------------------------------------------------------------------------------
// laplacian_h (:423-583) for the layers k0..nk of `var`, with DIFF_COEF = dc (nu_coef = 0) or
// 3/2 (kinvisc + NU_TURB) (nu_coef = 1); bf = the zonally filtered copy of var
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ double diff_coef(const DevModel &M, const double *dc, int nu_coef, long long x) {
  return nu_coef ? 3. / 2. * (M.kinvisc + M.nu_turb[x]) : dc[x];
}

// GH1 (the x-flux, rows 0..nj, with pads) and GH2 (the y-flux, rows 0..nj+1; 0 on the polar rows)
__global__ void k_lap_fluxes(DevModel M, const double *var, const double *bf, const double *dc, int nu_coef, int k0,
                             double *gh1, double *gh2) {
  if (epic_member(M, var, bf, dc, gh1, gh2)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 2);
  if (t >= (unsigned)(M.nk - k0 + 1) * nr * ni) return;
  const unsigned r = t / ni, q = r / nr;
  const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = k0 + (int)q;
  const long long x = M.at(k, j, i);
  if (j <= M.nj) {
    const double g1 = M.m[2 * j + 1] * (bf[x] - bf[x - 1]);
    write_with_pads(gh1, M, M.at(k, j, 0), i, g1 * (.5 * (diff_coef(M, dc, nu_coef, x) + diff_coef(M, dc, nu_coef, x - 1))));
  }
  double g2 = 0.;
  if (j >= 1 && j <= M.nj) {
    const long long xs = M.at(k, j - 1, i);
    g2 = M.n[2 * j] * (var[x] - var[xs]);
    g2 *= .5 * (diff_coef(M, dc, nu_coef, x) + diff_coef(M, dc, nu_coef, xs));
  }
  gh2[x] = g2;
}

// var += dt LPH, rows 0..nj (with pads), from the filtered GH1 and GH2
__global__ void k_lap_apply(DevModel M, double *var, int k0, const double *gh1, const double *gh2) {
  if (epic_member(M, var, gh1, gh2)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  if (t >= (unsigned)(M.nk - k0 + 1) * nr * ni) return;
  const unsigned r = t / ni, q = r / nr;
  const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = k0 + (int)q;
  const double m_2jp1 = M.m[2 * j + 1], n_2jp1 = M.n[2 * j + 1];
  const double m_2j_inv = (j == 0) ? 0. : div_rn(1., M.m[2 * j]);
  const double m_2jp2_inv = (j == M.nj) ? 0. : div_rn(1., M.m[2 * j + 2]);
  const long long x = M.at(k, j, i);
  const double lph = m_2jp1 * ((gh1[x + 1] - gh1[x]) + n_2jp1 * (gh2[M.at(k, j + 1, i)] * m_2jp2_inv - gh2[x] * m_2j_inv));
  write_with_pads(var, M, M.at(k, j, 0), i, var[x] + M.dt * lph);
}

// ---------------------------------------------------------------------------------------------
// The implicit vertical diffusions: scalar_vertical_diffusion (:1273-1488) of THETA and NU_TURB,
// uv_vertical_diffusion (:1940-2075) of U and V, each through crank_nicolson (epic_funcs_util.c:3643-3787)
// with tridiag(WITH_PIVOTING): band_decomp and band_back_sub for m1 = m2 = 1 (Numerical Recipes'
// bandec/banbks, :3130-3260) and one band_improve pass (:2994-3120, :3330-3400).
//
// A block takes 32 columns, one per lane, with every array in shared memory as [index][lane].  The
// heights, diffusivities, bands and the residual are pointwise in the levels, which the warps share;
// elimination (with row swaps) and back substitution are one warp's, their current rows in registers.
// One thread per column with its arrays in local memory took 682 us for NU_TURB (with its wall stress)
// and 176 us for each wind at 128x64x20: a chain of dependent quotients and local-memory round trips
// with two warps per SM.
//
// Arrays of n + 2 values a column (VD_ARRAYS of them): z, A and mu are indexed as crank_nicolson's; once
// the bands a, b, c, r stand, U0, U1, U2 and al (the decomposition) take the places of z, mu and the
// two stability arrays, and the answer that of A.
// ---------------------------------------------------------------------------------------------

enum { VD_THETA, VD_NU, VD_U, VD_V };
constexpr int VD_ARRAYS = 10, VD_THREADS = 256;

// stability_factor (:2309-2415) at the layers of column (j, i): s[K] = Ri[2K] as its slope limiter
// leaves it (K = 1..nk; the only entries the diffusions read).  The limiter runs over kk = 1..2nk in
// order, each step reading the entry the one before may have zeroed.
__device__ __forceinline__ void stability_ri(const DevModel &M, int j, int i, int kmin, double *s) {   // s[(K - kmin) * 32], K >= kmin
  const int nk = M.nk, x = M.at(0, j, i), n2 = (int)M.n2;
  const double max_ri = 100.;
  double ri = M.ri2[x + n2], cur = limit_range(-max_ri, ri, max_ri);   // kk = 1
  for (int k = 1; k <= nk; k++) {
    double nxt = limit_range(-max_ri, ri, max_ri);   // kk = 2k
    if (-(nxt - cur) > .9 * max_ri) nxt = 0.;
    if (k >= kmin) s[(k - kmin) * 32] = nxt;
    cur = nxt;
    const double below = M.ri2[x + min(k + 1, nk) * n2];
    nxt = limit_range(-max_ri, k == nk ? ri : .5 * (ri + below), max_ri);   // kk = 2k+1
    if (-(nxt - cur) > .9 * max_ri) nxt = 0.;
    cur = nxt;
    ri = below;
  }
}
__device__ __forceinline__ double stability_factor(double r) {
  return r > 0. ? div_rn(1., 1. + 10. * r * (1. + 8. * r)) : sqrt_rn(1. - 18. * r);
}

// forward elimination's row swaps and multipliers on b[0..n-1], then back substitution, of one column
__device__ __forceinline__ void vd_solve(int n, const double *U0, const double *U1, const double *U2, const double *al,
                                         unsigned long long swapped, double *b) {
  double cur = b[0];
  for (int k = 0; k < n - 1; k++) {
    double nxt = b[(k + 1) * 32];
    if ((swapped >> k) & 1) { const double t = cur; cur = nxt; nxt = t; }
    nxt -= al[k * 32] * cur;
    b[k * 32] = cur;
    cur = nxt;
  }
  double x1 = 0., x2 = 0.;
  for (int i = n - 1; i >= 0; i--) {
    double t = i == n - 1 ? cur : b[i * 32];
    if (i < n - 1) t -= U1[i * 32] * x1;
    if (i < n - 2) t -= U2[i * 32] * x2;
    t = div_rn(t, U0[i * 32]);
    b[i * 32] = t;
    x2 = x1;
    x1 = t;
  }
}

// M.turb_tau: the wall stresses (NU_TURB: WALL_H; U, V: their own)
__global__ void __launch_bounds__(VD_THREADS) k_vdiff(DevModel M, int what) {
  if (epic_member(M)) return;
  const double *tw = M.turb_tau;
  extern __shared__ double vd[];
  __shared__ int s_bad[32];
  __shared__ double s_dz[32];
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5), nw = VD_THREADS / 32;
  const int j0 = what == VD_V ? 1 : 0, nk = M.nk, ks = M.k_sigma, n2 = (int)M.n2;
  const int t = (int)blockIdx.x * 32 + lane;
  const bool live = t < (M.nj + 1 - j0) * M.ni;
  const int j = j0 + (live ? t / M.ni : 0), i = 1 + (live ? t % M.ni : 0);
  const int n = what == VD_THETA ? nk - ks + 2 : (what == VD_NU ? nk + 1 : nk - 1), S = 32 * (n + 2);
  double *z = vd + lane, *A = z + S, *mu = A + S, *a = mu + S, *b = a + S, *c = b + S, *r = c + S, *s0 = r + S, *s1 = s0 + S, *rho = s1 + S;
  double *U0 = z, *U1 = mu, *U2 = s0, *al = s1, *ans = A, *res = rho;
  const int col = M.at(0, j, i);
  const double gi = what == VD_V ? M.grav[2 * j] : M.grav[2 * j + 1];
  // the neighbouring column of the winds' stencil: (j, i-1) for U, (j-1, i) for V
  const int jn = what == VD_V ? j - 1 : j, in = what == VD_U ? i - 1 : i, coln = M.at(0, jn, in);
  const bool wind = what == VD_U || what == VD_V;
  double *F = what == VD_THETA ? M.theta : (what == VD_NU ? M.nu_turb : (what == VD_U ? M.u : M.v) + plane_offset(M, PL_UV));
  if (warp == 0) s_bad[lane] = n + 2;
  // the stability factors' Richardson numbers, from layer kmin on (THETA's diffusion uses ks-1..nk)
  const int kmin = what == VD_THETA ? ks - 1 : 1;
  if (live && M.stab && what != VD_NU && warp < (wind ? 2 : 1))
    stability_ri(M, warp == 0 ? j : jn, warp == 0 ? i : in, kmin, warp == 0 ? s0 : s1);
  __syncthreads();
  if (live) {
    auto gz = [&](int k) { return M.gz3[col + k * n2]; };
    auto gzm = [&](int k) { return .5 * (M.gz3[col + k * n2] + M.gz3[coln + k * n2]); };
    auto sf = [&](const double *s, int k) { return M.stab ? stability_factor(s[(k - kmin) * 32]) : 1.; };
    if (what == VD_THETA) {   // kay = nk - k + 1, k = nk..ks-2
      for (int kay = warp; kay <= n + 1; kay += nw) {
        const int k = nk - kay + 1;
        if (kay == 0) { A[0] = 1.e+20; z[0] = div_rn(gz(nk), gi); continue; }
        A[kay * 32] = M.theta[col + k * n2];
        z[kay * 32] = div_rn(gz(k), gi);
        if (kay <= n) mu[kay * 32] = sf(s0, k) * .5 * (M.dc_theta[col + k * n2] + M.dc_theta[col + (k - 1) * n2]);
      }
    } else if (what == VD_NU) {   // kay = nk - k + 1, k = nk..0
      const double sigma_inv = 3. / 2.;
      auto nu = [&](int k) { return M.nu_turb[col + k * n2]; };
      auto dee = [&](int k) { return sigma_inv * (M.kinvisc + .5 * (nu(k) + nu(k - 1))); };
      for (int kay = warp; kay <= n + 1; kay += nw) {
        const int k = nk - kay + 1;
        if (kay == 0) {
          const double z1 = div_rn(gz(nk), gi), z0 = div_rn(gz(nk) - (gz(nk - 1) - gz(nk)), gi), d = dee(nk);
          z[0] = z0;
          mu[0] = d;
          A[0] = nu(nk) - div_rn(tw[M.at2(j, i)] * (z1 - z0), d);
        } else if (kay == n + 1) {
          A[kay * 32] = 1.e+20;
          z[kay * 32] = div_rn(gz(0) + (gz(0) - gz(1)), gi);
        } else {
          A[kay * 32] = nu(k);
          z[kay * 32] = div_rn(gz(k), gi);
          if (k > 0) mu[kay * 32] = dee(k);
        }
      }
    } else {   // kay = nk - k, k = nk-1..1
      auto muk = [&](int k) {
        return M.dynvisc + .5 * (sf(s0, k) * M.rho2[col + k * n2] * .5 * (M.dc_uv[col + (k - 1) * n2] + M.dc_uv[col + k * n2]) +
                                 sf(s1, k) * M.rho2[coln + k * n2] * .5 * (M.dc_uv[coln + (k - 1) * n2] + M.dc_uv[coln + k * n2]));
      };
      for (int kay = warp; kay <= n + 1; kay += nw) {
        const int k = nk - kay;
        if (kay == 0) {
          const double z1 = div_rn(gzm(nk - 1), gi), z0 = div_rn(gzm(nk), gi), m = muk(nk - 1);
          z[0] = z0;
          mu[0] = m;
          A[0] = F[col + (nk - 1) * n2] - div_rn(tw[M.at2(j, i)] * (z1 - z0), m);
        } else if (kay == n + 1) {
          A[kay * 32] = 1.e+20;
          z[kay * 32] = div_rn(gzm(0), gi);
        } else {
          A[kay * 32] = F[col + k * n2];
          z[kay * 32] = div_rn(gzm(k), gi);
          rho[kay * 32] = .5 * (M.rho3[col + k * n2] + M.rho3[coln + k * n2]);
          mu[kay * 32] = muk(k);
        }
      }
    }
  }
  __syncthreads();
  // crank_nicolson: A[0] or A[n+1] above .99e20 marks a no-flux end; the first index whose height does
  // not increase ends the column with an error (the reference exits there)
  const bool flux0 = !(A[0] > .99e+20), fluxn = !(A[(n + 1) * 32] > .99e+20);
  const double dt = M.dt;
  if (live)
    for (int q = 1 + warp; q <= n + 1; q += nw) {
      const double dz = z[q * 32] - z[(q - 1) * 32];
      if (q >= (flux0 ? 1 : 2) && q <= (fluxn ? n + 1 : n) && z[q * 32] <= z[(q - 1) * 32]) atomicMin(&s_bad[lane], q);
      if (q > n) continue;
      const double c1 = q == 1 && !flux0 ? 0. : div_rn(mu[(q - 1) * 32], dz);
      const double c3 = q == n && !fluxn ? 0. : div_rn(mu[q * 32], z[(q + 1) * 32] - z[q * 32]);
      const double zz = z[(q + 1) * 32] - z[(q - 1) * 32];
      const double f = div_rn(dt, wind ? rho[q * 32] * zz : zz);
      a[(q - 1) * 32] = -c1 * f;
      b[(q - 1) * 32] = 1. + (c1 + c3) * f;
      c[(q - 1) * 32] = -c3 * f;
      const double m = A[q * 32] * (1. - (c1 + c3) * f);
      if (q == 1) r[0] = 2. * A[0] * c1 * f + m + A[64] * c3 * f;
      else if (q == n) r[(q - 1) * 32] = A[(q - 1) * 32] * c1 * f + m + 2. * A[(q + 1) * 32] * c3 * f;
      else r[(q - 1) * 32] = A[(q - 1) * 32] * c1 * f + m + A[(q + 1) * 32] * c3 * f;
    }
  __syncthreads();
  const int bad = s_bad[lane];
  if (warp == 0 && bad <= n + 1) s_dz[lane] = z[bad * 32] - z[(bad - 1) * 32];
  __syncwarp();
  unsigned long long swapped = 0;
  if (warp == 0 && live && bad > n + 1) {
    double p0 = b[0], p1 = c[0], p2 = 0.;
    for (int k = 0; k < n; k++) {
      double q0 = 0., q1 = 0., q2 = 0.;
      if (k + 1 < n) { q0 = a[(k + 1) * 32]; q1 = b[(k + 1) * 32]; q2 = k + 2 < n ? c[(k + 1) * 32] : 0.; }
      const bool sw = k + 1 < n && fabs(q0) > fabs(p0);
      if (sw) {
        swapped |= 1ull << k;
        double tt = p0; p0 = q0; q0 = tt;
        tt = p1; p1 = q1; q1 = tt;
        tt = p2; p2 = q2; q2 = tt;
      }
      if (p0 == 0.) p0 = 1.e-20;
      U0[k * 32] = p0;
      U1[k * 32] = p1;
      U2[k * 32] = p2;
      ans[(k + 1) * 32] = r[k * 32];
      if (k + 1 < n) {
        const double m = div_rn(q0, p0);
        al[k * 32] = m;
        p0 = q1 - m * p1;
        p1 = q2 - m * p2;
        p2 = 0.;
      }
    }
    vd_solve(n, U0, U1, U2, al, swapped, ans + 32);
  }
  __syncthreads();
  // band_improve: the residual of the original band in binary64, one correction
  if (live && bad > n + 1)
    for (int q = warp; q < n; q += nw) {
      double sdp = -r[q * 32];
      if (q > 0) sdp += a[q * 32] * ans[q * 32];
      sdp += b[q * 32] * ans[(q + 1) * 32];
      if (q < n - 1) sdp += c[q * 32] * ans[(q + 2) * 32];
      res[q * 32] = sdp;
    }
  __syncthreads();
  if (warp == 0 && live && bad > n + 1) vd_solve(n, U0, U1, U2, al, swapped, res);
  __syncthreads();
  if (!live) return;
  const int top = what == VD_THETA || what == VD_NU ? nk + 1 : nk;   // level = top - kay
  if (bad <= n + 1) {
    if (warp == 0) flag_error(M.ctl, ERR_TURB, top - bad, j, i, s_dz[lane]);
    return;
  }
  for (int kay = 1 + warp; kay <= n; kay += nw)
    write_with_pads(F, M, M.at(top - kay, j, 0), i, ans[kay * 32] - res[(kay - 1) * 32]);
}

// the wall stresses of all columns: WALL_U, WALL_V (tau_surface reads the neighbours' bottom winds,
// which the columns' solves then change) or WALL_H
__global__ void k_tau_wall(DevModel M, int index) {
  if (epic_member(M)) return;
  const int j0 = index == WALL_V ? 1 : 0;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= (M.nj + 1 - j0) * M.ni) return;
  const int j = j0 + t / M.ni, i = 1 + t - (j - j0) * M.ni;
  M.turb_tau[M.at2(j, i)] = tau_wall(M, index, j, i);
}

// ---------------------------------------------------------------------------------------------
// uv_horizontal_diffusion (:1571-1787).  work0 = COEFFD, work1 = H_RHO, work2 = UU, work3 = VV
// (layers 1..nk-1, zonally filtered); the stresses are recomputed where the updates read them.
// ---------------------------------------------------------------------------------------------

__global__ void k_uvh_coef(DevModel M) {
  if (epic_member(M)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned w = (unsigned)(M.nj + 1) * (unsigned)M.iadim;
  if (t >= w * (unsigned)(M.nk - 1)) return;
  const unsigned q = t / w;
  const long long x = M.at(1 + (int)q, 0, 0) + (t - q * w);
  M.work0[x] = M.dynvisc + M.rho3[x] * M.dc_uv[x];
  M.work1[x] = div_rn(M.h3[x], M.rho3[x]);
}

// TAU12 on the polar rows, per layer: vorticity(ON_SIGMATHETA, RELATIVE) there (epic_funcs_diag.c:
// 4279-4290, 4357-4379) times minus the row mean of COEFFD H_RHO, the sums in the reference's order.  One
// block per layer: the four rows staged in shared memory, a row summed per lane (one thread reading both
// rows of a pole from global memory took 43 us at 128x64x20).
__global__ void __launch_bounds__(128) k_uvh_poles(DevModel M) {
  if (epic_member(M)) return;
  extern __shared__ double rows[];   // [4][ni+1]: -UU(0), COEFFD H_RHO(0), UU(nj), COEFFD H_RHO(nj)
  __shared__ double sum[4];
  const int k = 1 + (int)blockIdx.x, ni = M.ni;
#pragma unroll 4
  for (int t = (int)threadIdx.x; t < 4 * ni; t += (int)blockDim.x) {
    const int r = t / ni, i = t - r * ni, x = M.at(k, (r & 2) ? M.nj : 0, i + 1);
    rows[r * (ni + 1) + i] = (r & 1) ? M.work0[x] * M.work1[x] : (r == 0 ? -M.work2[x] : M.work2[x]);
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const double *row = rows + threadIdx.x * (ni + 1);
    double s = 0.;
#pragma unroll 8
    for (int i = 0; i < ni; i++) s += row[i];
    sum[threadIdx.x] = s;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    const int north = (int)threadIdx.x;
    double ze = sum[2 * north], coeff = sum[2 * north + 1];
    if (north) ze *= M.mn[2 * (M.nj + 1)] / (M.m[2 * M.nj + 1] * (double)ni);
    else ze *= M.mn[0] / ((M.m[1]) * (double)ni);
    coeff /= ni;
    M.turb_pole[2 * k + north] = ze * -coeff;
  }
}

struct Stress { double t11, t22, t33; };

__device__ __forceinline__ Stress stress_h(const DevModel &M, int k, int j, int i) {
  if (i == 0) i = M.ni;   // bc_lateral
  const double *cd = M.work0, *hr = M.work1, *uu = M.work2, *vv = M.work3;
  auto U = [&](int jj, int ii) { return uu[M.at(k, jj, ii)]; };
  auto Vv = [&](int jj, int ii) { return vv[M.at(k, jj, ii)]; };
  auto H = [&](int jj, int ii) { return hr[M.at(k, jj, ii)]; };
  const int jj = 2 * j;
  const double rln_inv = div_rn(1., M.rln[jj + 1]), m_2jp1 = M.m[jj + 1], n_2jp2 = M.n[jj + 2], n_2jp1 = M.n[jj + 1], n_2j = M.n[jj];
  const double e11 = (U(j, i + 1) - U(j, i)) * m_2jp1 + .5 * (Vv(j, i) + Vv(j + 1, i)) * rln_inv * (M.rln[jj + 2] - M.rln[jj]) * n_2jp1;
  const double e22 = (Vv(j + 1, i) - Vv(j, i)) * n_2jp1;
  double coeff = div_rn(.5, H(j, i));
  double e33 = coeff * (U(j, i + 1) * (H(j, i + 1) - H(j, i)) * m_2jp1 + U(j, i) * (H(j, i) - H(j, i - 1)) * m_2jp1);
  if (Vv(j + 1, i) != 0.) e33 += coeff * Vv(j + 1, i) * (H(j + 1, i) - H(j, i)) * n_2jp2;
  if (Vv(j, i) != 0.) e33 += coeff * Vv(j, i) * (H(j, i) - H(j - 1, i)) * n_2j;
  coeff = H(j, i) * (2. / 3.) * cd[M.at(k, j, i)];
  Stress s;
  s.t11 = coeff * (2. * e11 - e22 - e33);
  s.t22 = coeff * (2. * e22 - e11 - e33);
  s.t33 = div_rn(coeff, H(j, i)) * (2. * e33 - e11 - e22);
  return s;
}

__device__ __forceinline__ double stress_12(const DevModel &M, int k, int j, int i) {
  if (j == 0) return M.turb_pole[2 * k];
  if (j == M.nj + 1) return M.turb_pole[2 * k + 1];
  if (i == 0) i = M.ni;   // bc_lateral
  const double *cd = M.work0, *hr = M.work1, *uu = M.work2, *vv = M.work3;
  auto c = [&](int jj, int ii) { return cd[M.at(k, jj, ii)] * hr[M.at(k, jj, ii)]; };
  const int jj = 2 * j;
  const double e12 = (vv[M.at(k, j, i)] - vv[M.at(k, j, i - 1)]) * M.m[jj] +
                     M.rln[jj] * (div_rn(uu[M.at(k, j, i)], M.rln[jj + 1]) - div_rn(uu[M.at(k, j - 1, i)], M.rln[jj - 1])) * M.n[jj];
  const double coeff = .25 * (c(j, i) + c(j, i - 1) + c(j - 1, i) + c(j - 1, i - 1));
  return coeff * e12;
}

__global__ void k_uvh_apply(DevModel M) {
  if (epic_member(M)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  if (t >= (unsigned)(M.nk - 1) * nr * ni) return;
  const unsigned r = t / ni, q = r / nr;
  const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = 1 + (int)q;
  const double *hr = M.work1;
  auto H = [&](int jj, int ii) { return hr[M.at(k, jj, ii == 0 ? M.ni : ii)]; };
  const long long tend = plane_offset(M, PL_UV_TEND);
  const Stress s = stress_h(M, k, j, i), sw = stress_h(M, k, j, i - 1);
  {
    const int jj = 2 * j;
    const double rln_inv = div_rn(1., M.rln[jj + 1]), m_2jp1 = M.m[jj + 1], n_2jp1 = M.n[jj + 1];
    const double h_inv = div_rn(2., M.hdry[M.at(k, j, i)] + M.hdry[M.at(k, j, i - 1)]);
    const double t12n = stress_12(M, k, j + 1, i), t12 = stress_12(M, k, j, i);
    const long long x = tend + M.at(k, j, i);
    M.dudt[x] += h_inv * (m_2jp1 * (s.t11 - sw.t11) +
                          n_2jp1 * rln_inv * (M.rln[jj + 2] * t12n - M.rln[jj] * t12 + .5 * (t12n + t12) * (M.rln[jj + 2] - M.rln[jj])) -
                          .5 * (s.t33 + sw.t33) * m_2jp1 * (H(j, i) - H(j, i - 1)));
  }
  if (j >= 1) {
    const Stress ss = stress_h(M, k, j - 1, i);
    const int jj = 2 * j;
    const double rln_inv = div_rn(1., M.rln[jj]), m_2j = M.m[jj], n_2j = M.n[jj];
    const double h_inv = div_rn(2., M.hdry[M.at(k, j, i)] + M.hdry[M.at(k, j - 1, i)]);
    const long long x = tend + M.at(k, j, i);
    M.dvdt[x] += h_inv * (m_2j * (stress_12(M, k, j, i) - stress_12(M, k, j, i - 1)) -
                          n_2j * rln_inv * (M.rln[jj + 1] * s.t22 - M.rln[jj - 1] * ss.t22 - .5 * (s.t11 + ss.t11) * (M.rln[jj + 1] - M.rln[jj - 1])) -
                          .5 * (s.t33 + ss.t33) * n_2j * (H(j, i) - H(j - 1, i)));
  }
}

// ---------------------------------------------------------------------------------------------
// set_diffusion_coef (:2171-2302), inside store_diag.  DIFFUSION_COEF_UV stays as it is above the
// bottom layer (the reference never sets it there).
// ---------------------------------------------------------------------------------------------

__global__ void k_dc_layers(DevModel M) {
  if (epic_member(M)) return;
  const int kend = M.gas_giant ? M.nk : M.nk - 1;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  if (t >= (unsigned)kend * nr * ni) return;
  const unsigned r = t / ni, q = r / nr;
  const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = 1 + (int)q;
  const long long x = M.at(k, j, i), row = M.at(k, j, 0);
  const double nu = M.nu_turb[x];
  double chi3 = div_rn(nu, M.kinvisc);
  chi3 *= chi3 * chi3;
  const double fv1 = div_rn(chi3, chi3 + SA_CV1_3);
  const double turb = fv1 * nu;
  const double v = limit_range(0., turb, M.turb_maxnu2[j]);
  write_with_pads(M.dc_theta, M, row, i, v);
  write_with_pads(M.dc_mass, M, row, i, v);
}

__global__ void k_dc_bottom(DevModel M) {
  if (epic_member(M)) return;
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (t >= (M.nj + 1) * M.ni) return;
  const int j = t / M.ni, i = 1 + t - j * M.ni;
  const int k = M.nk - 1;
  const double kin = kin_plane(M, PL_UV_DIS, k, j, i);
  const double u_tan = sqrt_rn(2. * kin);
  const double turb = law_of_the_wall(M, k, j, i, WALL_H, u_tan);
  const long long row = M.at(M.nk, j, 0);
  write_with_pads(M.dc_uv, M, row, i, limit_range(0., turb + M.kinvisc, M.turb_maxnu2[j]));
  const double v = limit_range(0., turb, M.turb_maxnu2[j]);
  write_with_pads(M.dc_theta, M, row, i, v);
  write_with_pads(M.dc_mass, M, row, i, v);
}

inline unsigned nblk(long long n, int th) { return (unsigned)((n + th - 1) / th); }

// cfl_dt (epic_funcs_diag.c:4884-5022): the minimum of each direction's limit over the grid, by
// an atomic minimum on the bits of the positive binary64 limits (their order is the integers');
// a minimum does not depend on the order of its operands, so the result is the reference's
__global__ void k_cfl(DevModel M, unsigned long long *lim) {
  if (epic_member(M, lim)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  double cx = DBL_MAX, cy = DBL_MAX, cz = DBL_MAX;
  if (t < (unsigned)M.nk * nr * ni) {
    const unsigned r = t / ni, q = r / nr;
    const int i = 1 + (int)(t - r * ni), j = (int)(r - q * nr), k = 1 + (int)q;
    const long long off = plane_offset(M, PL_UV);
    const double *U = M.u + off, *V = M.v + off;
    const double dz = M.dsgth[2 * k];
    double w = M.w3[M.at(k - 1, j, i)];
    if (w > 0.) cz = dminr(cz, dz / w);
    w = M.w3[M.at(k, j, i)];
    if (w < 0.) cz = dminr(cz, -dz / w);
    if (j >= 1) {
      const double dy = 1. / M.n[2 * j + 1];
      const double cs = sqrt(M.rgas * .5 * (M.t3[M.at(k, j, i)] + M.t3[M.at(k, j - 1, i)]) / (1. - M.kappa));
      double v = V[M.at(k, j + 1, i)] + cs;
      if (v > 0.) cy = dminr(cy, dy / v);
      v = V[M.at(k, j, i)] - cs;
      if (v < 0.) cy = dminr(cy, -dy / v);
    }
    if (fabs(M.lat[2 * j + 1]) <= M.lat0) {
      const double dx = 1. / M.m[2 * j + 1];
      const double cs = sqrt(M.rgas * .5 * (M.t3[M.at(k, j, i)] + M.t3[M.at(k, j, i - 1)]) / (1. - M.kappa));
      double u = U[M.at(k, j, i + 1)] + cs;
      if (u > 0.) cx = dminr(cx, dx / u);
      u = U[M.at(k, j, i)] - cs;
      if (u < 0.) cx = dminr(cx, -dx / u);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    cx = dminr(cx, __shfl_xor_sync(0xffffffffu, cx, o));
    cy = dminr(cy, __shfl_xor_sync(0xffffffffu, cy, o));
    cz = dminr(cz, __shfl_xor_sync(0xffffffffu, cz, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&lim[0], (unsigned long long)__double_as_longlong(cx));
    atomicMin(&lim[1], (unsigned long long)__double_as_longlong(cy));
    atomicMin(&lim[2], (unsigned long long)__double_as_longlong(cz));
  }
}

}  // namespace

int launch_cfl_dt(const DevModel &M, unsigned long long *lim, cudaStream_t s) {
  k_cfl<<<zg(nblk((long long)M.nk * (M.nj + 1) * M.ni, 128), M), 128, 0, s>>>(M, lim);
  return 0;
}

// ---- launchers ----

int launch_restore_nu(const DevModel &M, cudaStream_t s) {
  k_restore_nu<<<zg(nblk((long long)(M.nj + 1) * M.iadim * (M.nk + 2), 256), M), 256, 0, s>>>(M);
  return 0;
}

static int launch_pads(const DevModel &M, double *a, int k0, int k1, cudaStream_t s) {
  k_pads<<<zg(nblk((long long)(k1 - k0 + 1) * (M.nj + 2), 128), M), 128, 0, s>>>(M, a, k0, k1);
  return 0;
}

int launch_source_sink_turb(const DevModel &M, cudaStream_t s) {
  const long long cells = (long long)(M.nk - 1) * (M.nj + 1) * M.ni;
  k_sa_prep<<<zg(nblk(cells, 128), M), 128, 0, s>>>(M);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = zg(dim3((unsigned)M.sa_cluster), M);
  cfg.blockDim = dim3(SA_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)M.sa_cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_sa_waves, M);
  if (!M.gas_giant) k_sa_bottom<<<zg(nblk((long long)(M.nj + 1) * M.ni, 128), M), 128, 0, s>>>(M);
  return launch_pads(M, M.nu_turb, 0, M.nk + 1, s);
}

// laplacian_h of layers k0..nk of var, then var += dt LPH (scratch work0..2)
static int laplacian_step(const DevModel &M, double *var, const double *dc, int nu_coef, int k0, cudaStream_t s) {
  const int n = M.nk - k0 + 1;
  launch_filter_planes(M, var, PL_NONE, M.work0, k0, n, 0, s);   // zonal_filter(H2_INDEX) of a copy
  k_lap_fluxes<<<zg(nblk((long long)n * (M.nj + 2) * M.ni, 128), M), 128, 0, s>>>(M, var, M.work0, dc, nu_coef, k0, M.work1, M.work2);
  launch_filter_planes(M, M.work1, PL_NONE, M.work1, k0, n, 0, s);   // zonal_filter(U_INDEX) of GH1
  k_lap_apply<<<zg(nblk((long long)n * (M.nj + 1) * M.ni, 128), M), 128, 0, s>>>(M, var, k0, M.work1, M.work2);
  return 0;
}

int launch_theta_hdiff(const DevModel &M, cudaStream_t s, bool early) {
  laplacian_step(M, M.theta, M.dc_theta, 0, M.k_sigma - 1, s);
  return launch_set_p2etc(M, 1, s, early);
}
int launch_nu_hdiff(const DevModel &M, cudaStream_t s) {
  laplacian_step(M, M.nu_turb, nullptr, 1, 1, s);
  return launch_restore_nu(M, s);
}

static int launch_vdiff(const DevModel &M, int what, cudaStream_t s) {
  const int n = what == VD_THETA ? M.nk - M.k_sigma + 2 : (what == VD_NU ? M.nk + 1 : M.nk - 1);
  const long long cols = (long long)(M.nj + (what == VD_V ? 0 : 1)) * M.ni;
  k_vdiff<<<zg(nblk(cols, 32), M), VD_THREADS, (size_t)VD_ARRAYS * 32 * (n + 2) * sizeof(double), s>>>(M, what);
  return 0;
}
int launch_tau_wall_h(const DevModel &M, cudaStream_t s) {
  k_tau_wall<<<zg(nblk((long long)(M.nj + 1) * M.ni, 32), M), 32, 0, s>>>(M, WALL_H);
  return 0;
}

int launch_theta_vdiff(const DevModel &M, cudaStream_t s, bool early) {
  launch_vdiff(M, VD_THETA, s);
  return launch_set_p2etc(M, 1, s, early);
}
int launch_nu_vdiff(const DevModel &M, cudaStream_t s) {
  launch_vdiff(M, VD_NU, s);
  return launch_restore_nu(M, s);
}

int launch_uvh_coef(const DevModel &M, cudaStream_t s) {
  k_uvh_coef<<<zg(nblk((long long)(M.nj + 1) * M.iadim * (M.nk - 1), 256), M), 256, 0, s>>>(M);
  return 0;
}
int launch_uvh_filter(const DevModel &M, int which, cudaStream_t s) {
  switch (which) {
    case 0: return launch_filter_planes(M, M.work0, PL_NONE, M.work0, 1, M.nk - 1, 0, s);
    case 1: return launch_filter_planes(M, M.work1, PL_NONE, M.work1, 1, M.nk - 1, 0, s);
    case 2: return launch_filter_planes(M, M.u, PL_UV_DIS, M.work2, 1, M.nk - 1, 0, s);
    default: return launch_filter_planes(M, M.v, PL_UV_DIS, M.work3, 1, M.nk - 1, 1, s);
  }
}
int launch_uvh_apply(const DevModel &M, cudaStream_t s) {
  k_uvh_poles<<<zg(M.nk - 1, M), 128, (size_t)4 * (M.ni + 1) * sizeof(double), s>>>(M);
  k_uvh_apply<<<zg(nblk((long long)(M.nk - 1) * (M.nj + 1) * M.ni, 128), M), 128, 0, s>>>(M);
  return 0;
}

int launch_uv_vdiff(const DevModel &M, cudaStream_t s) {
  for (int comp = 0; comp < 2; comp++) {
    k_tau_wall<<<zg(nblk((long long)(M.nj + 1 - comp) * M.ni, 32), M), 32, 0, s>>>(M, comp == 0 ? WALL_U : WALL_V);
    launch_vdiff(M, comp == 0 ? VD_U : VD_V, s);
  }
  return 0;
}

// On the current device, whose own attributes these are: the most shared memory a launch takes (models of
// all sizes), and the blocks of the wavefront kernel's cluster -- 16 where the GPU can place them (a front of
// 1235 points at 128x64x20 is then a few per thread's SM), else the portable 8 -- into *cluster.  Whether it
// can is asked once per device.
int turb_kernels_init(int device, int *cluster) {
  static std::mutex mu;
  static std::map<int, bool> places16;
  const int big = (int)((size_t)VD_ARRAYS * 32 * (EPIC_TURB_MAX_NK + 3) * sizeof(double));
  const bool allowed = cudaFuncSetAttribute(k_sa_waves, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  {
    std::lock_guard<std::mutex> lock(mu);
    auto known = places16.find(device);
    if (known == places16.end()) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16);
      cfg.blockDim = dim3(SA_THREADS);
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 16;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int n = 0;
      known = places16.emplace(device, allowed && cudaOccupancyMaxActiveClusters(&n, k_sa_waves, &cfg) == cudaSuccess && n >= 1).first;
    }
    *cluster = allowed && known->second ? 16 : 8;
  }
  cudaGetLastError();
  return cudaFuncSetAttribute(k_vdiff, cudaFuncAttributeMaxDynamicSharedMemorySize, big) == cudaSuccess ? 0 : -1;
}

int launch_set_diffusion_coef(const DevModel &M, cudaStream_t s) {
  const int kend = M.gas_giant ? M.nk : M.nk - 1;
  k_dc_layers<<<zg(nblk((long long)kend * (M.nj + 1) * M.ni, 128), M), 128, 0, s>>>(M);
  if (!M.gas_giant) k_dc_bottom<<<zg(nblk((long long)(M.nj + 1) * M.ni, 64), M), 64, 0, s>>>(M);
  launch_pads(M, M.dc_uv, 0, M.nk + 1, s);
  launch_pads(M, M.dc_theta, 0, M.nk + 1, s);
  return launch_pads(M, M.dc_mass, 0, M.nk + 1, s);
}

}  // namespace epic

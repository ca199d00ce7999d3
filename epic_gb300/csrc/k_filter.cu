// High-latitude zonal filter kernels (the reference's zonal_filter, src/shared/epic_adjust.c:102-480).
//
// The reference filters one latitude row at a time: realft() forward, multiply wavenumber m by
// HIGH_LAT(J,m+1), realft() inverse and scale by 2/ni (epic_adjust.c:412-456), where realft and
// four1 are the Numerical Recipes in C (2nd ed., pp. 507, 513) real and complex radix-2 FFTs
// (epic_funcs_util.c:4023-4132).  Here a group of lanes of one warp owns one row and carries out the
// same arithmetic in parallel: every butterfly of a four1 stage and every iteration of realft's
// post-processing loop touches its own data, so they run concurrently; the twiddle factors,
// which NR builds by a recurrence, are computed once on the host with exactly that recurrence.
// Compiled without FMA contraction, each filtered row is bit-identical to the reference's.
#include "device_common.cuh"
#include "kernels.h"
#include "row_filter.cuh"
#include "epic_common.h"
#include "epic_gb300.h"

namespace epic {

// zonal_filter(index, plane, NULL, TWODIM) of planes k0..k0+nplanes-1, from src into dst
// (dst may equal src).  blockIdx.x = row j + 1, j in -1..nj+1; rows outside the filtered set are
// copied; rows 0..nj+1 get periodic pads (bc_lateral).
template <class R>
__global__ void k_filter_planes(DevModel M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, RowShape S) {
  if (epic_member(M, src, dst)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  src += plane_offset(M, src_sel);
  const int j = (int)blockIdx.x - 1, ni = M.ni;
  if (j > M.nj + 1) return;   // a member with fewer rows than the launch (batches of mixed sizes)
  const RowLane L = row_lane(S, k0, k0 + nplanes - 1);
  const int base = M.at(L.k, j, 0);
  const bool valid = vgrid ? (j >= 1 && j <= M.nj) : (j >= 0 && j <= M.nj);
  if (!(valid && row_is_filtered(M, j, vgrid))) {
    if (!L.live) return;
    const bool pads = j >= 0;
    for (int i = L.gl; i <= ni + 1; i += L.G) {
      if (pads && (i == 0 || i == ni + 1)) dst[base + i] = src[base + (i == 0 ? ni : 1)];
      else if (src != dst) dst[base + i] = src[base + i];
    }
    return;
  }
  const double *hl = (vgrid ? M.high_lat_pv : M.high_lat_h) + M.at2(j, 0);
  warm_filter<R>(M, hl);
  R *x = reinterpret_cast<R *>(smraw) + L.r * S.stride;
  const int lg = fft_log(ni);
  for (int e = L.gl; e < ni; e += L.G) x[fft_place(e, lg)] = L.live ? cv<R>(src[base + e + 1]) : R(0.);
  __syncwarp();
  filter_row<R>(M, reinterpret_cast<Cplx<R> *>(x), hl, L);
  if (!L.live) return;
  const R scale = filter_scale<R>(ni);
  for (int e = L.gl; e < ni; e += L.G) write_with_pads(dst, M, base, e + 1, to_d(x[e] * scale));
}


// Per-latitude var(gz) profile at the column of lowest bottom GZ, the first half of the
// THREEDIM branch of zonal_filter (epic_adjust.c:266-395).  One warp per row j: the lanes find
// the first column of minimum bottom GZ (the reference's strict-less scan) and fill the table;
// lane 0 fits the spline.  index: 0 = U, 1 = V, 2 = HDRY (log), 3 = THETA.
__global__ void k_varz_tables(DevModel M, const double *buff, int sel, int index, int kstart, int kend) {
  if (epic_member(M, buff)) return;
  buff += plane_offset(M, sel);
  const int jstart = index == 1 ? 1 : 0;
  const int lane = (int)(threadIdx.x & 31);
  const int j = jstart + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (j > M.nj) return;
  // the mixed forms filter (and so tabulate) only the filtered rows
  if (M.mixed && !row_is_filtered(M, j, index == 1)) return;
  const double *gz = M.gz;
  const int K = M.nk;
  int imin = 1 << 30;
  double gzmin = DBL_MAX;
  for (int i = 1 + lane; i <= M.ni; i += 32) {
    const double v = gz[M.at(K, j, i)];
    if (v < gzmin) { imin = i; gzmin = v; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, gzmin, o);
    const int oi = __shfl_xor_sync(0xffffffffu, imin, o);
    if (ov < gzmin || (ov == gzmin && oi < imin)) { gzmin = ov; imin = oi; }
  }
  const int i = imin == (1 << 30) ? 1 : imin;
  Trip *t = reinterpret_cast<Trip *>(M.ptable) + (long long)(j + 1) * (M.nk + 2);
  for (int k = kend - lane; k >= kstart; k -= 32) {
    const int kay = kend - k;
    double x;
    switch (index) {
      case 0: x = .5 * (gz[M.at(k, j, i)] + gz[M.at(k, j, i - 1)]); break;
      case 1: x = .5 * (gz[M.at(k, j, i)] + gz[M.at(k, j - 1, i)]); break;
      case 2: x = .5 * (gz[M.at(k, j, i)] + gz[M.at(k - 1, j, i)]); break;
      default: x = gz[M.at(k, j, i)]; break;
    }
    t[kay].x = x;
    t[kay].y = index == 2 ? xlog(M, buff[M.at(k, j, i)]) : buff[M.at(k, j, i)];
  }
  __syncwarp();
  // spline_pchip (epic_funcs_util.c:721-845): every slope uses only its two neighbouring
  // intervals, so the lanes compute them in parallel with the reference's expressions.
  const int n = kend - kstart + 1;
  bool bad = false;
  for (int q = 1 + lane; q < n; q += 32) bad |= t[q].x <= t[q - 1].x;
  if (__any_sync(0xffffffffu, bad)) {
    if (lane == 0) flag_error(M.ctl, ERR_PCHIP_X, kstart, j, i, t[0].x);
    return;
  }
  if (n == 2) {
    if (lane == 0) {
      const double del1 = div_rn(t[1].y - t[0].y, t[1].x - t[0].x);
      t[0].z = del1;
      t[1].z = del1;
    }
    return;
  }
  for (int q = lane; q < n; q += 32) {
    // the two intervals around point q (the first two for q = 0, the last two for q = n-1)
    const int m = q == 0 ? 1 : (q == n - 1 ? n - 2 : q);
    const double h1 = t[m].x - t[m - 1].x, h2 = t[m + 1].x - t[m].x;
    const double del1 = div_rn(t[m].y - t[m - 1].y, h1), del2 = div_rn(t[m + 1].y - t[m].y, h2);
    const double hsum = h1 + h2;
    double z;
    if (q == 0) {
      const double w1 = div_rn(h1 + hsum, hsum), w2 = div_rn(-h1, hsum);
      z = w1 * del1 + w2 * del2;
      if (pchst(z, del1) <= 0.0) z = 0.0;
      else if (pchst(del1, del2) < 0.0) {
        const double dmx = 3.0 * del1;
        if (fabs(dmx) < fabs(z)) z = dmx;
      }
    } else if (q == n - 1) {
      const double w1 = div_rn(-h2, hsum), w2 = div_rn(h2 + hsum, hsum);
      z = w1 * del1 + w2 * del2;
      if (pchst(z, del2) <= 0.0) z = 0.0;
      else if (pchst(del1, del2) < 0.0) {
        const double dmx = 3.0 * del2;
        if (fabs(dmx) < fabs(z)) z = dmx;
      }
    } else {
      z = 0.0;
      if (pchst(del1, del2) > 0.0) {
        const double hsumt3 = 3.0 * hsum;
        const double w1 = div_rn(hsum + h1, hsumt3), w2 = div_rn(hsum + h2, hsumt3);
        const double dmx = dmaxr(fabs(del1), fabs(del2)), dmn = dminr(fabs(del1), fabs(del2));
        z = div_rn(dmn, w1 * div_rn(del1, dmx) + w2 * div_rn(del2, dmx));
      }
    }
    t[q].z = z;
  }
}

// The mixed forms' profile: var(gz) to double-float accuracy (~48 bits) as the knot value plus the
// cubic's increment from the knot, evaluated in double-float on the distance gz - x_knot (gz and
// x_knot converted to double-floats on the integer pipe), with the cubic's coefficients computed
// in binary64 and split into double-floats; the deviation buff - var is formed in double-float
// and the filtered deviation added back to var in binary64 -- the field itself is never rounded
// to FP32, and the profile's own 48-bit rounding cancels between subtracting and adding it back.
// The profile has to be this accurate: out = var + F(buff - var) = buff - (I - F)(buff - var), so a
// rounding error of the profile that varies from column to column (an FP32 increment's does)
// passes the filter's high-wavenumber part (I - F) straight into THETA and HDRY on every filtered
// row, every step; with FP32 increments that was the largest single source of the mixed form's
// wind error after a simulated day (it halved the median member's U error to remove it).  HDRY is
// interpolated in log space: knot value exp(y) times exp(increment).  The knot values and the
// coefficients are tabulated once per row (varz_intervals_mixed); the interval is found in FP32
// (next to a knot either neighbouring cubic gives the same value, the pieces joining with their
// first derivative), the distance from its knot in double-float.
struct VarzInterval {
  float x, pad;
  float2 z0, c2, c3;   // double-float coefficients of the cubic in the distance from the knot
};
__device__ __forceinline__ float2 split_df(double v) {
  const dfl d = d2df(v);
  return make_float2(d.hi, d.lo);
}
__device__ __forceinline__ void varz_intervals_mixed(const Trip *t, int n, int index, double *knot, VarzInterval *iv) {
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    knot[q] = index == 2 ? ::exp(t[q].y) : t[q].y;
    VarzInterval v;
    v.x = d2f(t[q].x);
    v.pad = 0.f;
    v.z0 = split_df(t[q].z);
    v.c2 = v.c3 = make_float2(0.f, 0.f);
    if (q + 1 < n) {   // splint_pchip's cubic, epic_funcs_util.c:926-946
      const double h = t[q + 1].x - t[q].x;
      const double delta = div_rn(t[q + 1].y - t[q].y, h);
      const double del1 = div_rn(t[q].z - delta, h), del2 = div_rn(t[q + 1].z - delta, h);
      v.c3 = split_df(div_rn(del1 + del2, h));
      v.c2 = split_df(-(del1 + del1 + del2));
    }
    iv[q] = v;
  }
}
__device__ __forceinline__ dfl varz_profile_mixed(const Trip *t, const double *knot, const VarzInterval *iv, int n, int index,
                                                  dfl gzd, const float2 *exp2tab) {
  const float g = gzd.hi;
  int kay;
  if (g <= iv[0].x) kay = 0;
  else if (g >= iv[n - 1].x) kay = n - 2;
  else {
    int il = -1, iu = n;
    while (iu - il > 1) {
      const int im = (iu + il) >> 1;
      if (g >= iv[im].x) il = im; else iu = im;
    }
    kay = il;
  }
  // a NaN argument fails every comparison: keep the interval index inside the table
  kay = kay < 0 ? 0 : (kay > n - 2 ? n - 2 : kay);
  const VarzInterval v = iv[kay];
  const dfl xx = gzd - d2df(t[kay].x);
  const dfl inc = xx * (dfl(v.z0.x, v.z0.y) + xx * (dfl(v.c2.x, v.c2.y) + xx * dfl(v.c3.x, v.c3.y)));
  return index == 2 ? d2df(knot[kay]) * exp_df(inc, exp2tab) : d2df(knot[kay]) + inc;
}

// The FP64 form's profile of one latitude: the knots, and splint_pchip's cubic (epic_funcs_util.c:926-946)
// of every interval, whose coefficients depend on the interval alone -- computed once per block, not
// once per column.
struct VarzKnot { double x, y, z, c2, c3; };
__device__ __forceinline__ void varz_intervals(const Trip *t, int n, VarzKnot *kn) {
  for (int q = threadIdx.x; q < n; q += blockDim.x) {
    VarzKnot v = {t[q].x, t[q].y, t[q].z, 0., 0.};
    if (q + 1 < n) {
      const double h = t[q + 1].x - t[q].x;
      const double delta = div_rn(t[q + 1].y - t[q].y, h);
      const double del1 = div_rn(t[q].z - delta, h), del2 = div_rn(t[q + 1].z - delta, h);
      v.c3 = div_rn(del1 + del2, h);
      v.c2 = -(del1 + del1 + del2);
    }
    kn[q] = v;
  }
}
__device__ __forceinline__ double varz_profile(const VarzKnot *kn, int n, double g) {
  int kay;   // find_place_in_table (epic_funcs_util.c:2908-2967)
  if (fcmp(g, kn[0].x) <= 0) kay = 0;
  else if (fcmp(g, kn[n - 1].x) >= 0) kay = n - 2;
  else {
    int il = -1, iu = n;
    while (iu - il > 1) {
      const int im = (iu + il) >> 1;
      if (fcmp(g, kn[im].x) >= 0) il = im; else iu = im;
    }
    kay = il < 0 ? 0 : il;
  }
  const VarzKnot v = kn[kay];
  const double xx = g - v.x;
  return v.y + xx * (v.z + xx * (v.c2 + xx * v.c3));
}
// doubles of the block's table: knots and cubics (FP64), knot values and VarzInterval (mixed)
__host__ __device__ inline size_t varz_table_doubles(int nk, bool mixed) {
  return (size_t)(nk + 2) * (mixed ? 1 + sizeof(VarzInterval) / 8 : sizeof(VarzKnot) / 8) + (((nk + 2) & 1) ? 1 : 0);
}

// The rest of the THREEDIM zonal_filter: subtract var(gz), filter, add it back.
// blockIdx.x = row j - jstart, levels kstart.. by blockIdx.y.  Shared memory: the table, then per row
// the profile's values (binary64) and the deviation (the compute type).
template <class R>
__global__ void k_varz_filter_rows(DevModel M, double *buff, int sel, int index, int kstart, int kend, RowShape S) {
  if (epic_member(M, buff)) return;
  extern __shared__ __align__(16) double smd[];
  buff += plane_offset(M, sel);
  constexpr bool exact = std::is_same_v<R, double>;
  const int jstart = index == 1 ? 1 : 0, ni = M.ni;
  const int j = jstart + (int)blockIdx.x;
  if (j > M.nj) return;   // a member with fewer rows than the launch (batches of mixed sizes)
  const int vgrid = index == 1;
  const Trip *t = reinterpret_cast<const Trip *>(M.ptable) + (long long)(j + 1) * (M.nk + 2);
  const int n = kend - kstart + 1;
  const double *gz = M.gz;
  const bool filt = row_is_filtered(M, j, vgrid);
  // The mixed forms leave unfiltered rows untouched (their subtract-and-add-back is the identity
  // up to one rounding); the FP64 form repeats the reference's arithmetic on them.
  if (!filt && !exact) return;
  if (filt) warm_filter<R>(M, (vgrid ? M.high_lat_pv : M.high_lat_h) + M.at2(j, 0));
  VarzKnot *kn = reinterpret_cast<VarzKnot *>(smd);
  VarzInterval *iv = reinterpret_cast<VarzInterval *>(smd);
  double *knot = smd + (size_t)(M.nk + 2) * (sizeof(VarzInterval) / 8);
  if constexpr (exact) varz_intervals(t, n, kn);
  else varz_intervals_mixed(t, n, index, knot, iv);
  __syncthreads();
  const RowLane L = row_lane(S, kstart, kend);
  const int k = L.k, base = M.at(k, j, 0), lg = fft_log(ni);
  double *vz = smd + varz_table_doubles(M.nk, !exact) + (size_t)L.r * S.stride;
  R *x = reinterpret_cast<R *>(vz + ni);
  // the other value of the mean that gives the profile's argument: U, V and layer variables lie
  // half-way between GZ's points
  const int other = index == 0 ? -1 : (index == 1 ? -M.iadim : (index == 2 ? -(int)M.n2 : 0));
  for (int e = L.gl; e < ni; e += L.G) {
    const int p = base + e + 1;
    double v = 0.;
    R dev = R(0.);
    if (L.live) {
      if constexpr (exact) {
        const double g = other ? half_of(gz[p] + gz[p + other]) : gz[p];
        v = varz_profile(kn, n, g);
        if (index == 2) v = xexp(M, v);
        dev = buff[p] - v;
      } else {
        // the profile's argument, its value and the deviation in double-float (integer and FP32
        // pipes: this kernel had the FP64 unit half busy); the deviation is filtered in binary32 and
        // added back to the profile in binary64 below, the profile's own rounding cancelling
        const dfl g = other ? df_ldexp(d2df(gz[p]) + d2df(gz[p + other]), -1) : d2df(gz[p]);
        const dfl pv = varz_profile_mixed(t, knot, iv, n, index, g, M.exp2tab);
        v = df2d(pv);
        dev = (d2df(buff[p]) - pv).hi;
      }
    }
    vz[e] = v;
    x[row_place(filt, e, lg)] = dev;
  }
  __syncwarp();
  if (filt) filter_row<R>(M, reinterpret_cast<Cplx<R> *>(x), (vgrid ? M.high_lat_pv : M.high_lat_h) + M.at2(j, 0), L);
  if (!L.live) return;
  const R scale = filter_scale<R>(ni);
  // HDRY (index 2): restore_mass, which timestep() calls next (epic_timestep.c:212), on the new value
  for (int e = L.gl; e < ni; e += L.G) {
    const double v = to_d(filt ? x[e] * scale : x[e]) + vz[e];
    write_with_pads(buff, M, base, e + 1, index == 2 ? dmaxr(M.h_min[k], v) : v);
  }
}

// Row j of a zonal advection pass in shared memory: the zonally filtered copy that the fluxes come
// from, in order, a[0..ni-1] for i = 1..ni.
template <class R>
__device__ __forceinline__ void zonal_filtered_row(const DevModel &M, const double *buff, int base, int j, R *a, const RowLane &L) {
  const bool filt = row_is_filtered(M, j, 0);   // of the whole block
  const int ni = M.ni, lg = fft_log(ni);
#pragma unroll 4
  for (int e = L.gl; e < ni; e += L.G) a[row_place(filt, e, lg)] = L.live ? cv<R>(buff[base + e + 1]) : R(1.);
  __syncwarp();
  if (!filt) return;
  filter_row<R>(M, reinterpret_cast<Cplx<R> *>(a), M.high_lat_h + M.at2(j, 0), L);
  const R scale = filter_scale<R>(ni);
  for (int e = L.gl; e < ni; e += L.G) a[e] = a[e] * scale;
  __syncwarp();
}

// The last word on a cell of an advected field: HDRY (kind 1) takes restore_mass (epic_adjust.c:45-96),
// which advection() calls next (epic_flux.c:623); THETA (kind 3) loses OLD (UNITY - 1)
// (epic_flux.c:377-435), OLD being THETA before its advection (the vertical pass keeps it).
__device__ __forceinline__ double advected(const DevModel &M, int kind, int k, int x, double v) {
  if (kind == 1) return dmaxr(M.h_min[k], v);
  if (kind == 3) return v - M.old[x] * (M.unity[x] - 1.);
  return v;
}

// Zonal pass of hsu_advection (epic_flux.c:1316-1484), a row per lane group: the fluxes come from a
// zonally filtered copy of the row, the update goes to the unfiltered field.
// kind: 0 = interface variable (unity), 1 = HDRY (layer; u averaged to the layer),
// 2 = NU_TURB (interface variable with the floor NU_TURB_MIN), 3 = THETA (interface variable, then
// corrected by UNITY's advection, theta_corrected).
// Bound by latency on a small grid (a lane's few faces and cells one after another) and by the FP64 pipe
// on a large one: faces in pairs, four cells' loads before their stores.  A step of 64x32x10 389 -> 385 us,
// 12 mixed steps of 128x64x20 3.72 -> 3.70 ms, 8 fast ones of eight small runs 3.44 -> 3.41 ms.
// Shared arrays by i - 1: a (the filtered row), ff (the flux through the west face), ap (the
// predicted row); w (the velocity) by i, with the field's own pads.
template <class R>
__global__ void k_hsu_zonal(DevModel M, double *buff, int kind, int kstart, RowShape S) {
  if (epic_member(M, buff)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ni = M.ni;
  const int j = (int)blockIdx.x;
  if (j > M.nj) return;   // a member with fewer rows than the launch (batches of mixed sizes)
  const RowLane L = row_lane(S, kstart, M.nk);
  if (row_is_filtered(M, j, 0)) warm_filter<R>(M, M.high_lat_h + M.at2(j, 0));
  const int k = L.k, base = M.at(k, j, 0);
  R *a = reinterpret_cast<R *>(smraw) + L.r * S.stride, *ff = a + ni, *ap = ff + ni, *w = ap + ni;
  const R DT = cv<R>(M.dt);
  const R a_min = kind == 1 ? cv<R>(M.h_min[k]) : (kind == 2 ? cv<R>(1.e-3 * M.kinvisc) : R(0.));
  const double *U = M.u + (long long)M.ctl->it_uv * M.n3;
  const R n_inv = qdiv(R(1.), cv<R>(M.n[2 * j + 1]));
  const R mn1 = cv<R>(M.mn[2 * j + 1]);
#pragma unroll 4
  for (int i = L.gl; i <= ni + 1; i += L.G) {
    // u2d, with periodic pads for the layer average (bc_lateral(u2d))
    const int ii = kind == 1 ? (i == 0 ? ni : (i == ni + 1 ? 1 : i)) : i;
    R u2d = R(0.);
    if (L.live) u2d = kind == 1 ? half_of(cv<R>(U[M.at(k, j, ii)]) + cv<R>(U[M.at(k - 1, j, ii)])) : cv<R>(U[M.at(k, j, i)]);
    w[i] = u2d * n_inv;
  }
  zonal_filtered_row<R>(M, buff, base, j, a, L);
  const int mask = ni - 1;   // ni is a power of 2: rows wrap
  for (int e = L.gl; e < ni; e += L.G) ff[e] = hsu_upwind<R>(w[e + 1], a[e], a[(e - 1) & mask]);
  __syncwarp();
  unsigned top = 0;
  auto predict = [&] {
    for (int e = L.gl; e < ni; e += L.G) {
      const R p = a[e] + (ff[e] - ff[(e + 1) & mask]) * mn1 * DT;
      ap[e] = p;
      top = max(top, top_bits(p));
    }
  };
  predict();
  const bool odd = __any_sync(0xffffffffu, top >= NONFINITE_BITS<R>);   // in one of the warp's rows
  if (odd) {
    for (int e = L.gl; e < ni; e += L.G)
      if (hsu_upwind_tainted<R>(w[e + 1], a[e], a[(e - 1) & mask])) ff[e] = quiet_nan<R>();
    __syncwarp();
    predict();
  }
  __syncwarp();
  auto face = [&](int e) {
    const R v = w[e + 1];
    const bool neg = is_neg(v);   // from cell e west to e-1, else from e-1 east to e
    const int west = (e - 1) & mask, u = neg ? e : west, d = neg ? west : e, uu = (neg ? e + 1 : e - 2) & mask;
    const R au = a[u], ad = a[d], auu = a[uu];
    const R t = fabs((neg ? ad : auu) - twice_of(au) + (neg ? auu : ad)) + R(1.e-10);
    return hsu_face<R>(v, w[neg ? e + 2 : e], au, ad, ap[d], ap[u] - auu, t * t, a_min, a_min, mn1, DT);
  };
  for (int e = L.gl; e < ni; e += 2 * L.G) {   // two faces at once: each is a chain of ~15 dependent operations
    const int e1 = e + L.G;
    const R f0 = face(e), f1 = face(e1 & mask);
    ff[e] = f0;
    if (e1 < ni) ff[e1] = f1;
  }
  if (odd)
    for (int e = L.gl; e < ni; e += L.G) {
      const bool neg = is_neg(w[e + 1]);
      if (hsu_tainted<R>(neg, w[neg ? e + 2 : e], w[neg ? e : e + 2], a[(neg ? e - 2 : e + 1) & mask], ap[neg ? e : (e - 1) & mask])) ff[e] = quiet_nan<R>();
    }
  __syncwarp();
  if (!L.live) return;
  for (int e0 = L.gl; e0 < ni; e0 += 4 * L.G) {   // four cells' loads before the first store
    double v[4], off[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = e0 + q * L.G, x = base + e + 1;
      v[q] = off[q] = 0.;
      if (e >= ni) continue;
      v[q] = buff[x];
      if (kind == 3) off[q] = M.old[x] * (M.unity[x] - 1.);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int e = e0 + q * L.G;
      if (e >= ni) continue;
      double y = v[q] + to_d((ff[e] - ff[(e + 1) & mask]) * mn1 * DT);
      if (kind == 1) y = dmaxr(M.h_min[k], y);
      else if (kind == 3) y = y - off[q];
      write_with_pads(buff, M, base, e + 1, y);
    }
  }
}

// Zonal pass of akima_advection (epic_flux.c:1826-1932), a row per lane group: the fluxes come from a
// zonally filtered copy of the row, the update goes to the unfiltered field.
// kind: as k_hsu_zonal's (NU_TURB has no floor here).
// Shared arrays by i - 1: a (the filtered row), dl (the limited slopes), ff (the fluxes).
template <class R>
__global__ void k_akima_zonal(DevModel M, double *buff, int kind, int kstart, RowShape S) {
  if (epic_member(M, buff)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int ni = M.ni;
  const int j = (int)blockIdx.x;
  if (j > M.nj) return;   // a member with fewer rows than the launch (batches of mixed sizes)
  const RowLane L = row_lane(S, kstart, M.nk);
  if (row_is_filtered(M, j, 0)) warm_filter<R>(M, M.high_lat_h + M.at2(j, 0));
  const int k = L.k, base = M.at(k, j, 0), mask = ni - 1;
  R *a = reinterpret_cast<R *>(smraw) + L.r * S.stride, *dl = a + ni, *ff = dl + ni;
  const R DT = cv<R>(M.dt);
  const double *U = M.u + (long long)M.ctl->it_uv * M.n3;
  const R n_inv = qdiv(R(1.), cv<R>(M.n[2 * j + 1]));
  const R mn1 = cv<R>(M.mn[2 * j + 1]);
  zonal_filtered_row<R>(M, buff, base, j, a, L);
  for (int e = L.gl; e < ni; e += L.G) {
    const R d0 = a[e] - a[(e - 1) & mask], d1 = a[(e + 1) & mask] - a[e];
    const R tmp = d0 * d1;
    dl[e] = (tmp > R(0.)) ? qdiv(twice_of(tmp), d0 + d1) : R(0.);
  }
  __syncwarp();
  for (int e = L.gl; e < ni; e += L.G) {
    const R aval = half_of(a[e] + a[(e - 1) & mask]) - qdiv(dl[e] - dl[(e - 1) & mask], R(6.));
    R u2d = R(0.);
    if (L.live) {
      const int p = base + e + 1;
      u2d = kind == 1 ? half_of(cv<R>(U[p]) + cv<R>(U[p - (int)M.n2])) : cv<R>(U[p]);
    }
    ff[e] = u2d * aval * n_inv;
  }
  __syncwarp();
  if (!L.live) return;
  for (int e = L.gl; e < ni; e += L.G) {
    const double v = buff[base + e + 1] + to_d((ff[e] - ff[(e + 1) & mask]) * mn1 * DT);
    write_with_pads(buff, M, base, e + 1, advected(M, kind, k, base + e + 1, v));
  }
}

// The rows the tensor-core filter leaves alone (k_filter_planes_gemm filters the others): copied
// when dst is not src, periodic pads on rows 0..nj+1.  One warp per (row, plane).
__global__ void k_filter_rows_unfiltered(DevModel M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid) {
  if (epic_member(M, src, dst)) return;
  src += plane_offset(M, src_sel);
  const int lane = (int)(threadIdx.x & 31);
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int rows = M.nj + 3;
  if (w >= rows * nplanes) return;
  const int j = w % rows - 1, k = k0 + w / rows;
  const bool valid = vgrid ? (j >= 1 && j <= M.nj) : (j >= 0 && j <= M.nj);
  if (valid && row_is_filtered(M, j, vgrid)) return;
  const int base = M.at(k, j, 0);
  if (src != dst)
    for (int i = lane; i <= M.ni + 1; i += 32) dst[base + i] = src[base + i];
  __syncwarp();
  if (j >= 0 && lane == 0) {
    dst[base] = dst[base + M.ni];
    dst[base + M.ni + 1] = dst[base + 1];
  }
}

// ---- launchers ----

// The shape of a row kernel whose rows take `stride` values of `elem` bytes each: lanes a row as above;
// 128 threads a block (or the tuning table's choice, in whole warps: a warp's lanes all belong to rows that
// the block's shared memory holds), fewer where its rows would take more than 48 KB, so that several blocks
// share an SM.
static RowShape row_shape(const DevModel &M, int stride, size_t elem, unsigned &threads) {
  RowShape S;
  S.G = M.ni >= 128 ? 32 : (M.ni >= 64 ? 16 : 8);
  S.stride = stride;
  unsigned warps = M.tb[TB_ROW] > 0 ? ((unsigned)M.tb[TB_ROW] + 31u) / 32u : 4u;
  while (warps > 1 && warps * 32u / (unsigned)S.G * (unsigned)stride * elem > 48 * 1024) warps /= 2;
  threads = 32u * warps;
  S.rows = (int)threads / S.G;
  return S;
}
static size_t row_bytes(const RowShape &S, size_t elem) { return (size_t)S.rows * (size_t)S.stride * elem; }
static size_t relem(int fp32) { return fp32 ? sizeof(float) : sizeof(double); }

int launch_filter_rest(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s, int fp32) {
  if (nplanes <= 0 || !(fp32 && filter_gemm_usable(M))) return 0;
  // The rows the operator leaves alone are copied (and padded) by a light kernel of their own: done by
  // the operator's blocks, which fill an SM's shared memory each, they kept the filtered rows waiting (12
  // steps of 128x64x20 3.92 -> 4.07 ms).
  const long long warps = (long long)(M.nj + 3) * nplanes;
  k_filter_rows_unfiltered<<<zg(epic_blocks(32 * warps, 128), M), 128, 0, s>>>(M, src, src_sel, dst, k0, nplanes, vgrid);
  return 0;
}

int launch_filter_planes(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s,
                         int fp32, int shift, int filtered_rows_only) {
  if (nplanes <= 0) return 0;
  if (fp32 && filter_gemm_usable(M)) {
    if (!filtered_rows_only) launch_filter_rest(M, src, src_sel, dst, k0, nplanes, vgrid, s, fp32);
    return launch_filter_planes_gemm(M, src, src_sel, dst, k0, nplanes, vgrid, s, shift);
  }
  unsigned th;
  const RowShape S = row_shape(M, M.ni, relem(fp32), th);
  const dim3 grid(M.nj + 3, epic_blocks(nplanes, S.rows));
  EPIC_LAUNCH_R(fp32, k_filter_planes, grid, th, row_bytes(S, relem(fp32)), s, M, src, src_sel, dst, k0, nplanes, vgrid, S);
  return 0;
}

int launch_varz_filter(const DevModel &M, double *buff, int sel, int index, int kstart, int kend, cudaStream_t s) {
  const int jstart = index == 1 ? 1 : 0;
  const int nrows = M.nj - jstart + 1;
  k_varz_tables<<<zg(epic_blocks(32LL * nrows, 128), M), 128, 0, s>>>(M, buff, sel, index, kstart, kend);
  unsigned th;
  const RowShape S = row_shape(M, M.mixed ? M.ni + M.ni / 2 : 2 * M.ni, sizeof(double), th);
  const size_t smem = varz_table_doubles(M.nk, M.mixed) * sizeof(double) + row_bytes(S, sizeof(double));
  const dim3 grid(nrows, epic_blocks(kend - kstart + 1, S.rows));
  EPIC_LAUNCH_R(M.mixed, k_varz_filter_rows, grid, th, smem, s, M, buff, sel, index, kstart, kend, S);
  return 0;
}

int launch_akima_zonal(const DevModel &M, double *buff, int kind, int kstart, cudaStream_t s) {
  unsigned th;
  const RowShape S = row_shape(M, 3 * M.ni, relem(M.mixed), th);
  const dim3 grid(M.nj + 1, epic_blocks(M.nk - kstart + 1, S.rows));
  EPIC_LAUNCH_R(M.mixed, k_akima_zonal, grid, th, row_bytes(S, relem(M.mixed)), s, M, buff, kind, kstart, S);
  return 0;
}

int launch_hsu_zonal(const DevModel &M, double *buff, int kind, int kstart, cudaStream_t s) {
  unsigned th;
  const RowShape S = row_shape(M, 4 * M.ni + 2, relem(M.mixed), th);
  const dim3 grid(M.nj + 1, epic_blocks(M.nk - kstart + 1, S.rows));
  EPIC_LAUNCH_R(M.mixed, k_hsu_zonal, grid, th, row_bytes(S, relem(M.mixed)), s, M, buff, kind, kstart, S);
  return 0;
}

template <class R>
static void filter_attrs(int bytes) {
  cudaFuncSetAttribute(k_hsu_zonal<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_akima_zonal<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_varz_filter_rows<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(k_filter_planes<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Raised once to the most a launch takes (row_shape's 48 KB and the varz kernels' table), so models of
// different sizes in one process never lower the limit for one another.
int filter_kernels_init(int) {
  const size_t big = 48 * 1024 + varz_table_doubles(EPIC_MAX_NK, false) * sizeof(double);
  filter_attrs<double>((int)big);
  filter_attrs<float>((int)big);
  return 0;
}

size_t twiddle_doubles(int ni) { return 2 * nr_twiddle_pairs(ni); }

// Host: the twiddle factors four1 and realft generate by recurrence, in their order, with
// their arithmetic (epic_funcs_util.c:4047-4076, :4096-4120).  Compiled without contraction.
void fill_twiddles(int ni, double *tw) {
  const int N = ni / 2;
  const unsigned long n = (unsigned long)N << 1;
  double *out = tw;
  for (int isign = 1; isign >= -1; isign -= 2) {
    for (unsigned long mmax = 2; n > mmax; mmax <<= 1) {
      const double theta = isign * (2 * M_PI / mmax);
      double wtemp = sin(0.5 * theta);
      const double wpr = -2.0 * wtemp * wtemp;
      const double wpi = sin(theta);
      double wr = 1.0, wi = 0.0;
      for (unsigned long m = 1; m < mmax; m += 2) {
        *out++ = wr;
        *out++ = wi;
        wr = (wtemp = wr) * wpr - wi * wpi + wr;
        wi = wi * wpr + wtemp * wpi + wi;
      }
    }
  }
  for (int isign = 1; isign >= -1; isign -= 2) {
    double theta = M_PI / (double)((unsigned long)ni >> 1);
    if (isign != 1) theta = -theta;
    double wtemp = sin(0.5 * theta);
    const double wpr = -2.0 * wtemp * wtemp;
    const double wpi = sin(theta);
    double wr = 1.0 + wpr, wi = wpi;
    for (unsigned long i = 2; i <= ((unsigned long)ni >> 2); i++) {
      *out++ = wr;
      *out++ = wi;
      wr = (wtemp = wr) * wpr - wi * wpi + wr;
      wi = wi * wpr + wtemp * wpi + wi;
    }
  }
}

}  // namespace epic

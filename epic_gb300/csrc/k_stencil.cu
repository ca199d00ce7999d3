// Horizontal stencil kernels and the time update.  Each kernel restates the reference routine
// named in its comment; thread = one (k, j, i) cell unless stated otherwise.
#include "device_common.cuh"
#include "kernels.h"
#include "row_filter.cuh"
#include "epic_common.h"
#include "epic_gb300.h"

namespace epic {

// Cell index helpers for 3-D launches over k in [k0, k0+nk), j in [j0, j0+nj), i in 1..ni.
struct Cell { int k, j, i; };
// The index arithmetic is 32-bit unsigned (two divisions, remainders by multiply-subtract): a
// launch covers fewer than 2^31 cells of a member (epic_model_create bounds a field below 2^31
// elements), and 64-bit divisions cost as many instructions as the stencil's own loads.
__device__ __forceinline__ bool cell3(const DevModel &M, int k0, int nkk, int j0, int njj, Cell &c) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)njj;
  if (t >= (unsigned)nkk * nr * ni) return false;
  const unsigned r = t / ni, q = r / nr;
  c.i = 1 + (int)(t - r * ni);
  c.j = j0 + (int)(r - q * nr);
  c.k = k0 + (int)q;
  return true;
}
// (k, j, i) of cell t of the interior layers k = 1..nk-1, rows j = 0..nj (the wind updates)
__device__ __forceinline__ void cell_kji(const DevModel &M, unsigned t, int &k, int &j, int &i) {
  const unsigned ni = (unsigned)M.ni, nr = (unsigned)(M.nj + 1);
  const unsigned r = t / ni, q = r / nr;
  i = 1 + (int)(t - r * ni);
  j = (int)(r - q * nr);
  k = 1 + (int)q;
}
static inline unsigned cells_blocks(const DevModel &M, int nkk, int njj, int th) {
  return epic_blocks((long long)nkk * njj * M.ni, th);
}

template <class R>
__global__ void k_row_tables(DevModel M, R *out) {
  const int j = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (j > M.nj + 1) return;
  const bool h = j <= M.nj, v = j >= 1 && j <= M.nj;   // rows with an h point, v points off the poles
  auto inv = [&](const double *a, int jj) { return qdiv(R(1.), cv<R>(a[jj])); };
  R *t = out + j * RT_COUNT;
  const int jj = 2 * j;
  t[RT_NINV_H] = h ? inv(M.n, jj + 1) : R(0.);
  t[RT_MINV_V] = fabs(M.lat[jj]) == 90. ? R(0.) : inv(M.m, jj);
  t[RT_MINV_H] = h ? inv(M.m, jj + 1) : R(0.);
  t[RT_MNINV_H] = h ? inv(M.mn, jj + 1) : R(0.);
  t[RT_MNINV_V] = cv<R>(M.mn_inv[jj]);
  t[RT_MNPV] = v ? qdiv(R(.5), inv(M.mn, jj - 1) + inv(M.mn, jj + 1)) : R(0.);
  t[RT_GDX] = h ? qdiv(R(.5) * cv<R>(M.m[jj + 1]), cv<R>(M.grav[jj + 1])) : R(0.);
  t[RT_GDY] = qdiv(R(.5) * cv<R>(M.n[jj]), cv<R>(M.grav[jj]));
  t[RT_M_H] = h ? cv<R>(M.m[jj + 1]) : R(0.);
  t[RT_M_V] = cv<R>(M.m[jj]);
  t[RT_N_V] = cv<R>(M.n[jj]);
  t[RT_MN_H] = h ? cv<R>(M.mn[jj + 1]) : R(0.);
  t[RT_F_V] = cv<R>(M.f[jj]);
}

// d2dy2's coefficients times the viscosity coefficient of each order that uses them, once per model:
// the FP64 form's hyperviscosity is bound by the FP64 pipe (19 cycles a warp instruction and SM), and
// three of a point's products depend on its row alone.  The same products, so the same bits.
// 12 steps of 128x64x20 10.47 -> 10.23 ms, 3 of 256x128x32 15.2 -> 15.0 ms.
template <class R>
__global__ void k_visc_tables(DevModel M, R *out) {
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x), rows = M.nj + 2;
  if (t >= 24 * rows) return;
  const int v = t / (12 * rows), j = (t - v * 12 * rows) / 12, q = t % 12, order = 2 * (q / 3) + 2;
  const double c = order == 2 ? M.coef[2] : (order == 4 ? M.coef[4] : (order == 6 ? M.coef[6] : M.coef[8]));
  out[t] = j <= (v ? M.nj + 1 : M.nj) ? cv<R>(c) * cv<R>((v ? M.v_coef : M.h_coef)[3 * j + q % 3]) : R(0.);
}

// memset of DUDT, DVDT(it_uv_tend), epic_timestep.c:107-108
__global__ void k_zero_tend(DevModel M) {
  if (epic_member(M)) return;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= M.n3) return;
  const long long off = plane_offset(M, PL_UV_TEND);
  M.dudt[off + t] = 0.;
  M.dvdt[off + t] = 0.;
}

// ---------------------------------------------------------------------------------------------
// uv_core, epic_timestep.c:628-762, with get_kin (Suarez-Takacs blend for the Sadourney scheme,
// epic_funcs_diag.c:2694-2847) and the PV averages of include/epic_pv_schemes.h:48-61.
// ---------------------------------------------------------------------------------------------

// UH(j,i), j = 0..nj, of wind value u between h-points h0 = H(j,i) and hm = H(j,i-1)
template <class R>
__device__ __forceinline__ R uh_of(const DevModel &M, int j, R u, R h0, R hm) { return u * half_of(h0 + hm) * rt<R>(M, j, RT_NINV_H); }

// Kinetic energy per mass on the h grid, planes k = 1..nk-1, into work0 (with pads): kin_at up the rows,
// where a row's northern v terms are the next one's southern.
template <class R, int ROWS>
__global__ void k_uv_kin(DevModel M) {
  if (epic_member(M)) return;
  March s;
  if (!march<ROWS>(M, 1, M.nk - 1, 0, M.nj, s)) return;
  const int k = s.k, i = s.i, nj = M.nj;
  const long long off = plane_offset(M, PL_UV) + k * M.n2;
  const double *Uk = M.u + off, *Vk = M.v + off;
  auto u = [&](int j, int ii) { return cv<R>(Uk[M.at2(j, ii)]); };
  // v^2/mn of row j at the cell and of the mean of its neighbours
  auto vv = [&](int j, R &own, R &mean) {
    const R v0 = cv<R>(Vk[M.at2(j, i)]), vm = half_of(cv<R>(Vk[M.at2(j, i + 1)]) + cv<R>(Vk[M.at2(j, i - 1)])), w = rt<R>(M, j, RT_MNINV_V);
    own = v0 * v0 * w;
    mean = vm * vm * w;
  };
  R us_w = R(0.), us_e = R(0.), u_w = u(s.j0, i), u_e = u(s.j0, i + 1), vs, vsm;
  if (s.j0 > 0) { us_w = u(s.j0 - 1, i); us_e = u(s.j0 - 1, i + 1); }
  vv(s.j0, vs, vsm);
#pragma unroll
  for (int q = 0; q < ROWS; q++) {
    const int j = s.j0 + q;
    if (ROWS > 1 && j > s.j1) break;
    R un_w = R(0.), un_e = R(0.), vn, vnm;
    if (j < nj) { un_w = u(j + 1, i); un_e = u(j + 1, i + 1); }
    vv(j + 1, vn, vnm);
    const R mn1 = rt<R>(M, j, RT_MN_H);
    R kin = scale_down<2>(u_w * u_w + u_e * u_e + mn1 * (vs + vn));
    if (j != 0 && j != nj) {
      const R u2 = half_of(un_w + us_w), u4 = half_of(un_e + us_e);
      const R kin_s = scale_down<2>(u2 * u2 + u4 * u4 + mn1 * (vsm + vnm));
      kin = (R(5.) / R(6.)) * kin + (R(1.) / R(6.)) * kin_s;
    }
    write_with_pads(M.work0, M, M.at(k, j, 0), i, to_d(kin));
    us_w = u_w; us_e = u_e; u_w = un_w; u_e = un_e; vs = vn; vsm = vnm;
  }
}

// DVDT += (PV*UH terms + KIN(j-1)-KIN(j))*n, then the vertical advection of V, rows 1..nj.
template <class R, int ROWS>
__global__ void k_uv_core_v(DevModel M) {
  if (epic_member(M)) return;
  March s;
  if (!march<ROWS>(M, 1, M.nk - 1, 1, M.nj, s)) return;
  const int k = s.k, i = s.i, n2 = (int)M.n2, ie = i == M.ni ? 1 : i + 1;   // UH is periodic in i
  const long long off = plane_offset(M, PL_UV);
  const double *V = M.v + off, *Uk = M.u + off + k * M.n2, *Hk = M.h3 + k * M.n2;
  const double *PV = M.pv3 + k * M.n2, *KIN = M.work0 + k * M.n2, *W = M.w3 + k * M.n2;
  double *D = M.dvdt + plane_offset(M, PL_UV_TEND);
  auto pv = [&](int jj, int ii) { return cv<R>(PV[M.at2(jj, ii)]); };
  auto uh = [&](int jj, R &c, R &e) {   // UH(jj,i), UH(jj,i+1)
    const R hc = cv<R>(Hk[M.at2(jj, i)]);
    c = uh_of<R>(M, jj, cv<R>(Uk[M.at2(jj, i)]), hc, cv<R>(Hk[M.at2(jj, i - 1)]));
    // the row's last cell takes column 1, whose western neighbour is column 0
    e = uh_of<R>(M, jj, cv<R>(Uk[M.at2(jj, ie)]), cv<R>(Hk[M.at2(jj, ie)]), ie == 1 ? cv<R>(Hk[M.at2(jj, 0)]) : hc);
  };
  const int kk = 2 * k + 1;
  const R dsg = cv<R>(M.sgth[kk - 2]) - cv<R>(M.sgth[kk + 2]);
  R uhs_c, uhs_e, pc = pv(s.j0, i), pe = pv(s.j0, i + 1), ps_e = pv(s.j0 - 1, i + 1), ps = pv(s.j0 - 1, i) + pc;
  R kin_s = cv<R>(KIN[M.at2(s.j0 - 1, i)]), w_s = cv<R>(W[M.at2(s.j0 - 1, i)]);
  uh(s.j0 - 1, uhs_c, uhs_e);
#pragma unroll
  for (int q = 0; q < ROWS; q++) {
    const int j = s.j0 + q;
    if (ROWS > 1 && j > s.j1) break;
    const int x2 = M.at2(j, i), x = x2 + k * n2;
    const R pn = pv(j + 1, i), pn_e = pv(j + 1, i + 1), pp = pc + pe, pcn = pc + pn;
    const R ga = pp + pn_e, de = pcn + pe, al = ps + pe, be = pp + ps_e;
    R uh_c, uh_e;
    uh(j, uh_c, uh_e);
    const R kin = cv<R>(KIN[x2]), w = cv<R>(W[x2]);
    const R core = ((-ga * uh_e - de * uh_c - al * uhs_c - be * uhs_e) * (R(1.) / R(12.)) + kin_s - kin) * rt<R>(M, j, RT_N_V);
    double d = D[x] + to_d(core);
    d -= to_d(qdiv(half_of(w + w_s) * (cv<R>(V[x - n2]) - cv<R>(V[x + n2])), dsg));
    D[x] = d;
    ps = pcn; ps_e = pe; pc = pn; pe = pn_e; uhs_c = uh_c; uhs_e = uh_e; kin_s = kin; w_s = w;
  }
}

// DUDT += (PV*VH terms + KIN(i-1)-KIN(i))*m with the filtered KIN, then the vertical advection of U,
// rows 0..nj.
template <class R, int ROWS>
__global__ void k_uv_core_u(DevModel M) {
  if (epic_member(M)) return;
  March s;
  if (!march<ROWS>(M, 1, M.nk - 1, 0, M.nj, s)) return;
  const int k = s.k, i = s.i, n2 = (int)M.n2, nj = M.nj, iw = i == 1 ? M.ni : i - 1;   // VH is periodic in i
  const long long off = plane_offset(M, PL_UV);
  const double *U = M.u + off, *Vk = M.v + off + k * M.n2, *Hk = M.h3 + k * M.n2;
  const double *PV = M.pv3 + k * M.n2, *KIN = M.work0 + k * M.n2, *W = M.w3 + k * M.n2;
  double *D = M.dudt + plane_offset(M, PL_UV_TEND);
  auto pv = [&](int jj, int ii) { return cv<R>(PV[M.at2(jj, ii)]); };
  auto h = [&](int jj, int ii) { return cv<R>(Hk[M.at2(jj, ii)]); };
  // VH(jj,ii) on rows 1..nj between h-points hn = H(jj,ii) and hs = H(jj-1,ii); 0 at the poles
  auto vh = [&](int jj, int ii, R hn, R hs) { return cv<R>(Vk[M.at2(jj, ii)]) * half_of(hn + hs) * rt<R>(M, jj, RT_MINV_V); };
  const int kk = 2 * k + 1;
  const R dsg = cv<R>(M.sgth[kk - 2]) - cv<R>(M.sgth[kk + 2]);
  R pc = pv(s.j0, i), pw = pv(s.j0, i - 1), pe = pv(s.j0, i + 1), hc = h(s.j0, i), hw = h(s.j0, iw), vs_c = R(0.), vs_w = R(0.);
  if (s.j0 >= 1) {
    vs_c = vh(s.j0, i, hc, h(s.j0 - 1, i));
    vs_w = vh(s.j0, iw, hw, h(s.j0 - 1, iw));
  }
#pragma unroll
  for (int q = 0; q < ROWS; q++) {
    const int j = s.j0 + q;
    if (ROWS > 1 && j > s.j1) break;
    const int x2 = M.at2(j, i), x = x2 + k * n2;
    const R pn = pv(j + 1, i), pn_w = pv(j + 1, i - 1), pn_e = pv(j + 1, i + 1), pcn = pc + pn;
    const R al = pcn + pn_e, be = pn_w + pn + pc, ga = pw + pc + pn, de = pcn + pe;
    R vn_c = R(0.), vn_w = R(0.), hn = R(0.), hn_w = R(0.);
    if (j < nj) {
      hn = h(j + 1, i);
      hn_w = h(j + 1, iw);
      vn_c = vh(j + 1, i, hn, hc);
      vn_w = vh(j + 1, iw, hn_w, hw);
    }
    const R core = ((al * vn_c + be * vn_w + ga * vs_w + de * vs_c) * (R(1.) / R(12.)) + cv<R>(KIN[x2 - 1]) - cv<R>(KIN[x2])) *
                   rt<R>(M, j, RT_M_H);
    double d = D[x] + to_d(core);
    d -= to_d(qdiv(half_of(cv<R>(W[x2]) + cv<R>(W[x2 - 1])) * (cv<R>(U[x - n2]) - cv<R>(U[x + n2])), dsg));
    D[x] = d;
    pc = pn; pw = pn_w; pe = pn_e; hc = hn; hw = hn_w; vs_c = vn_c; vs_w = vn_w;
  }
}

// ---------------------------------------------------------------------------------------------
// uv_pgrad_finite_volume, epic_timestep.c:909-1273
// ---------------------------------------------------------------------------------------------

// Row sums in the reference's order (one addition after another) occupy the binary64 pipe for a
// whole warp instruction per addition whatever the number of active lanes, so the kernels that need
// them stage several rows in shared memory and sum one row per lane.  Rows lie ni+1 or ni+2
// values apart, which keeps the lanes on different banks or at most two on one.  ROW_SUM_SMEM bounds a block's rows.
constexpr size_t ROW_SUM_SMEM = 48 * 1024;
static __device__ __forceinline__ double row_sum(const double *row, int n) {
  double sum = 0.;
  if (n < 16) {
    for (int i = 0; i < n; i++) sum += row[i];
    return sum;
  }
  double b[8], c[8];   // n is a power of 2; the next eight values come while these are added
#pragma unroll
  for (int q = 0; q < 8; q++) b[q] = row[q];
  for (int i = 8; i < n; i += 8) {
#pragma unroll
    for (int q = 0; q < 8; q++) c[q] = row[i + q];
#pragma unroll
    for (int q = 0; q < 8; q++) sum += b[q], b[q] = c[q];
  }
#pragma unroll
  for (int q = 0; q < 8; q++) sum += b[q];
  return sum;
}
// levels per block of a kernel that sums `rows` rows of each, one per lane of a warp
// of which there are nk+1: no more than it takes to have a block per SM
static int row_sum_levels(const DevModel &M, int rows) {
  const int fit = (int)(ROW_SUM_SMEM / ((size_t)rows * (M.ni + 1) * sizeof(double)));
  const int want = (int)(((long long)(M.nk + 1) * (M.nbatch > 1 ? M.nbatch : 1) + M.sms - 1) / M.sms);
  int lv = fit > 32 / rows ? 32 / rows : fit;
  lv = lv > want ? want : lv;
  return lv < 1 ? 1 : lv;
}

// Pole boundary rows of GZ3 (zonal means of the adjacent row), epic_timestep.c:930-998.
// One block per lv levels, the two rows of each summed in the reference's order, a row per lane.
// With the rows read from global memory by one thread of a block per level it took 14 us at
// 128x64x20 (row_sum's comment).
__global__ void __launch_bounds__(256) k_gz_pole_rows(DevModel M, int lv) {
  if (epic_member(M)) return;
  extern __shared__ double rows[];   // [lv][2][ni+1]: rows 0 and nj of each level
  __shared__ double avg[32];
  const int ni = M.ni, k0 = (int)blockIdx.x * lv, nl = min(lv, M.nk + 1 - k0);
#pragma unroll 4
  for (int t = (int)threadIdx.x; t < 2 * nl * ni; t += (int)blockDim.x) {
    const int r = t / ni, i = t - r * ni;
    rows[r * (ni + 1) + i] = M.gz3[M.at(k0 + (r >> 1), (r & 1) ? M.nj : 0, i + 1)];
  }
  __syncthreads();
  if ((int)threadIdx.x < 2 * nl) avg[threadIdx.x] = row_sum(rows + (int)threadIdx.x * (ni + 1), ni) * inv_pow2(ni);
  __syncthreads();
  for (int t = (int)threadIdx.x; t < 2 * nl * (ni + 2); t += (int)blockDim.x) {
    const int r = t / (ni + 2), i = t - r * (ni + 2);
    const int x = M.at(k0 + (r >> 1), (r & 1) ? M.nj + 1 : -1, i);
    M.gz3[x] = avg[r];
    if (M.mixed) put_split(M.work1, x, avg[r]);
  }
}

// The finite-volume force is a sum of face integrals that is unchanged when every GZ3 (or every
// P2) of the stencil moves by one constant; the mixed form evaluates it in FP32 on
// GZ3 - GZ3(k,j,i) and P2 - P2(k,j,i), which keeps the FP32 products near the size of the
// differences the force is made of.  The differences are formed in FP32 from (hi, lo) splits of
// GZ3 and P2 (put_split: hi = float(x), lo = float(x - hi), in scratch work1 and work2, written by
// the kernels that computed the two fields) as (hi_x - hi_ref) + (lo_x - lo_ref): within a
// rounding or two of the FP64 difference, with no FP64 operation per stencil point.  The FP64
// form uses the values as they are.
// Double-float (dfl, the accurate mixed form) takes the same splits and forms the differences in
// double-float: the stencil's values then carry ~48 bits, and the face integrals' cancellation
// costs no accuracy that matters.
template <class R>
struct PgradRef {
  const DevModel &M;
  float2 zr, pr;
  __device__ __forceinline__ PgradRef(const DevModel &M_, int k, int j, int i) : M(M_) {
    if constexpr (!std::is_same_v<R, double>) {
      zr = reinterpret_cast<const float2 *>(M.work1)[M.at(k, j, i)];
      pr = reinterpret_cast<const float2 *>(M.work2)[M.at(k, j, i)];
    }
  }
  static __device__ __forceinline__ R diff(float2 v, float2 r) {
    if constexpr (std::is_same_v<R, float>) return (v.x - r.x) + (v.y - r.y);
    else return dfl(v.x, v.y) - dfl(r.x, r.y);
  }
  __device__ __forceinline__ R z(long long x) const {
    if constexpr (std::is_same_v<R, double>) return M.gz3[x];
    else return diff(reinterpret_cast<const float2 *>(M.work1)[x], zr);
  }
  __device__ __forceinline__ R p(long long x) const {
    if constexpr (std::is_same_v<R, double>) return M.p2[x];
    else return diff(reinterpret_cast<const float2 *>(M.work2)[x], pr);
  }
};
// Width of a u (v) control volume in longitude (latitude), radians, between the faces at
// half-levels ii-1 and ii+1: the FP64 form subtracts the two face coordinates in the compute
// type as the reference does; the mixed form subtracts in FP64 first (FP32 face coordinates
// of up to 2 pi would lose five digits to cancellation).
template <class R>
__device__ __forceinline__ R face_width(const double *deg, int iw, int ie) {
  if constexpr (std::is_same_v<R, double>) return deg[ie] * (M_PI / 180.) - deg[iw] * (M_PI / 180.);
  else return cv<R>((deg[ie] - deg[iw]) * (M_PI / 180.));
}

// Multiplication by a power of two, exact in every compute type: a double-float scales its two
// parts (two multiplications, where the general product takes seven operations).
struct Pow2 { float c; };
template <class R>
__device__ __forceinline__ R operator*(Pow2 s, R x) { return R(s.c) * x; }
__device__ __forceinline__ dfl operator*(Pow2 s, dfl x) { return dfl(s.c * x.hi, s.c * x.lo); }
__device__ __forceinline__ double operator*(Pow2 s, double x) { return s.c == .5f ? scale_down<1>(x) : (s.c == .25f ? scale_down<2>(x) : s.c * x); }

// The four quarter sums and two half sums of a face (lon_face, lat_face): in the FP64 form in
// the reference's order; the mixed forms share the pair each two of them have in common.
template <class R, class G>
__device__ __forceinline__ void face_sums(G gz, R &zb0, R &zb2, R &zt0, R &zt2, R &zb, R &zt) {
  if constexpr (std::is_same_v<R, double>) {
    zb0 = Pow2{.25f} * (gz(1, 1) + gz(1, 0) + gz(2, 1) + gz(2, 0));
    zb2 = Pow2{.25f} * (gz(1, 1) + gz(1, 2) + gz(2, 1) + gz(2, 2));
    zt0 = Pow2{.25f} * (gz(1, 1) + gz(1, 0) + gz(0, 1) + gz(0, 0));
    zt2 = Pow2{.25f} * (gz(1, 1) + gz(1, 2) + gz(0, 1) + gz(0, 2));
    zb = Pow2{.5f} * (gz(1, 1) + gz(2, 1));
    zt = Pow2{.5f} * (gz(1, 1) + gz(0, 1));
  } else {
    const R sb = gz(1, 1) + gz(2, 1), st = gz(1, 1) + gz(0, 1);
    zb0 = Pow2{.25f} * (sb + gz(1, 0) + gz(2, 0));
    zb2 = Pow2{.25f} * (sb + gz(1, 2) + gz(2, 2));
    zt0 = Pow2{.25f} * (st + gz(1, 0) + gz(0, 0));
    zt2 = Pow2{.25f} * (st + gz(1, 2) + gz(0, 2));
    zb = Pow2{.5f} * sb;
    zt = Pow2{.5f} * st;
  }
}

template <class R>
struct LonFace { R zbse, zbne, ztse, ztne, zbe, zte, pbe, pte, east; };

// East face of the u control volume at column i+c-1 (the quantities the reference carries
// from one i to the next).  z[a][b][c]: GZ3 at level k+a-1, row j+b-1, column i+c-1;
// p[a][c]: P2 at level k+a, row j, column i+c-1 (shifted by the reference values, §PgradRef).
template <class R>
__device__ __forceinline__ LonFace<R> lon_face(const DevModel &M, const R (&z)[3][3][2], const R (&p)[2][2], int c, int i) {
  auto gz = [&](int a, int b) { return z[a][b][c]; };
  LonFace<R> f;
  face_sums<R>(gz, f.zbse, f.zbne, f.ztse, f.ztne, f.zbe, f.zte);
  f.pbe = p[1][c];
  f.pte = p[0][c];
  const R a1 = f.ztne + f.ztse, b1 = f.ztne * f.ztse, a2 = f.zbne + f.zbse, b2 = f.zbne * f.zbse;
  const R terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
  const R terms2 = R(3.) * (a1 - a2);
  f.east = qdiv(-terms1 * (f.pbe - f.pte) + terms2 * (f.zte * f.pbe - f.zbe * f.pte), f.zte - f.zbe);
  return f;
}

// Rows shared by a block (ni divides the block: the launcher sizes the shared memory for it):
// each cell computes its east face once and takes its west face from the cell to its left --
// for i = 1 from the row's last cell, whose face at column ni equals the face at the periodic
// column 0 bit for bit (the fields' pad columns are copies).  The faces of one row then need one
// reference: the double-float form shifts by the row's value at i = 1 instead of each cell's own
// (its differences keep ~48 bits either way); the binary32 form keeps its per-cell reference and
// computes both faces.
template <class R>
__global__ void k_pgrad_lon(DevModel M) {
  if (epic_member(M)) return;
  Cell c;
  const bool share = !std::is_same_v<R, float> && (blockDim.x % (unsigned)M.ni) == 0u;
  const bool valid = cell3(M, 1, M.nk - 1, 0, M.nj + 1, c);
  if (!share && !valid) return;
  const int k = c.k, j = c.j, i = c.i;
  const R DLOGZ_TOL = R(1.e-2);
  LonFace<R> w, e;
  if (share) {
    extern __shared__ __align__(16) unsigned char pg_smem[];
    LonFace<R> *faces = reinterpret_cast<LonFace<R> *>(pg_smem);
    if (valid) {
      const PgradRef<R> ref(M, k, j, 1);
      R z[3][3][2], p[2][2];
#pragma unroll
      for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) z[a][b][1] = z[a][b][0] = ref.z(M.at(k + a - 1, j + b - 1, i));
#pragma unroll
      for (int a = 0; a < 2; a++) p[a][1] = p[a][0] = ref.p(M.at(k + a, j, i));
      e = lon_face<R>(M, z, p, 1, i);
      faces[threadIdx.x] = e;
    }
    __syncthreads();
    if (!valid) return;
    w = faces[i == 1 ? threadIdx.x + (unsigned)M.ni - 1u : threadIdx.x - 1u];
  } else {
    const PgradRef<R> ref(M, k, j, i);
    R z[3][3][2], p[2][2];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int b = 0; b < 3; b++)
#pragma unroll
        for (int q = 0; q < 2; q++) z[a][b][q] = ref.z(M.at(k + a - 1, j + b - 1, i + q - 1));
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int q = 0; q < 2; q++) p[a][q] = ref.p(M.at(k + a, j, i + q - 1));
    w = lon_face<R>(M, z, p, 0, i - 1);
    e = lon_face<R>(M, z, p, 1, i);
  }
  const R rho = Pow2{.5f} * (cv<R>(M.rho3[M.at(k, j, i)]) + cv<R>(M.rho3[M.at(k, j, i - 1)]));
  const R rlns = cv<R>(M.rln[2 * j]), rlnn = cv<R>(M.rln[2 * j + 2]);
  R a1 = e.ztne + e.ztse, a2 = w.ztne + w.ztse;
  R terms2 = R(3.) * (a1 - a2), top, bottom;
  if (fabs(qdiv(twice_of(e.zte - w.zte), e.zte + w.zte - e.zbe - w.zbe)) > DLOGZ_TOL) {
    const R b1 = e.ztne * e.ztse, b2 = w.ztne * w.ztse;
    const R terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
    top = qdiv(-terms1 * (w.pte - e.pte) + terms2 * (e.zte * w.pte - w.zte * e.pte), e.zte - w.zte);
  } else {
    top = Pow2{.5f} * (w.pte + e.pte) * terms2;
  }
  a1 = e.zbne + e.zbse;
  a2 = w.zbne + w.zbse;
  terms2 = R(3.) * (a1 - a2);
  if (fabs(qdiv(twice_of(e.zbe - w.zbe), e.zte + w.zte - e.zbe - w.zbe)) > DLOGZ_TOL) {
    const R b1 = e.zbne * e.zbse, b2 = w.zbne * w.zbse;
    const R terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
    bottom = qdiv(-terms1 * (w.pbe - e.pbe) + terms2 * (e.zbe * w.pbe - w.zbe * e.pbe), e.zbe - w.zbe);
  } else {
    bottom = Pow2{.5f} * (w.pbe + e.pbe) * terms2;
  }
  R pgflon = top - bottom + R(0.) - R(0.) + w.east - e.east;
  const R dzn = e.ztne - e.zbne + w.ztne - w.zbne;
  const R dzs = e.ztse - e.zbse + w.ztse - w.zbse;
  pgflon = qdiv(pgflon, face_width<R>(M.lon, 2 * i - 1, 2 * i + 1) * rho * (rlns * (dzs + Pow2{.5f} * dzn) + rlnn * (dzn + Pow2{.5f} * dzs)));
  const long long x = plane_offset(M, PL_UV_TEND) + M.at(k, j, i);
  M.dudt[x] = M.dudt[x] + to_d(pgflon);
}

template <class R>
struct LatFace { R zbnw, zbne, ztnw, ztne, zbn, ztn, pbn, ptn, north, rln; };

// North face of the v control volume at row j+b-1.  z[a][b][c]: GZ3 at level k+a-1, row j+b-1,
// column i+c-1; p[a][b][c]: P2 at level k+a, row j+b-1, column i+c-1 (shifted by the reference
// values).
template <class R>
__device__ __forceinline__ LatFace<R> lat_face(const DevModel &M, const R (&z)[3][2][3], const R (&p)[2][2][3], int b, int jrow) {
  auto gz = [&](int a, int c) { return z[a][b][c]; };
  LatFace<R> f;
  f.rln = cv<R>(M.rln[2 * jrow + 1]);
  face_sums<R>(gz, f.zbnw, f.zbne, f.ztnw, f.ztne, f.zbn, f.ztn);
  f.pbn = p[1][b][1];
  f.ptn = p[0][b][1];
  const R a1 = f.ztne + f.ztnw, b1 = f.ztne * f.ztnw, a2 = f.zbne + f.zbnw, b2 = f.zbne * f.zbnw;
  const R terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
  const R terms2 = R(3.) * (a1 - a2);
  f.north = qdiv(f.rln * (-terms1 * (f.pbn - f.ptn) + terms2 * (f.ztn * f.pbn - f.zbn * f.ptn)), f.ztn - f.zbn);
  return f;
}

// In the FP64 form each thread marches up ROWS rows, a row's north face being the next one's
// south; the mixed forms take one row (their differences are relative to the row's own cell).
template <class R, int ROWS>
__global__ void k_pgrad_lat(DevModel M) {
  if (epic_member(M)) return;
  static_assert(std::is_same_v<R, double> || ROWS == 1);
  March strip;
  if (!march<ROWS>(M, 1, M.nk - 1, 1, M.nj, strip)) return;
  const int k = strip.k, i = strip.i;
  const R DLOGZ_TOL = R(1.e-2);
  R z[3][2][3], p[2][2][3];
  LatFace<R> s, n;
#pragma unroll
  for (int q_ = 0; q_ < ROWS; q_++) {
  const int j = strip.j0 + q_;
  if (ROWS > 1 && j > strip.j1) break;
  const PgradRef<R> ref(M, k, j, i);
  const bool first = q_ == 0;
  auto load = [&](int b) {
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int q = 0; q < 3; q++) z[a][b][q] = ref.z(M.at(k + a - 1, j + b - 1, i + q - 1));
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int q = 0; q < 3; q++) p[a][b][q] = ref.p(M.at(k + a, j + b - 1, i + q - 1));
  };
  if (first) {
    load(0);
    s = lat_face<R>(M, z, p, 0, j - 1);
  } else {
    s = n;
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int q = 0; q < 3; q++) {
        z[a][0][q] = z[a][1][q];
        if (a < 2) p[a][0][q] = p[a][1][q];
      }
  }
  load(1);
  n = lat_face<R>(M, z, p, 1, j);
  // z(level k+a-1, row j+b-1, column i+q-1), pp(level k+a, row j+b-1, column i+q-1)
  auto gz = [&](int a, int b, int q) { return z[a][b][q]; };
  auto pp = [&](int a, int b, int q) { return p[a][b][q]; };
  const R rho = Pow2{.5f} * (cv<R>(M.rho3[M.at(k, j, i)]) + cv<R>(M.rho3[M.at(k, j - 1, i)]));
  const R rlt = cv<R>(M.rlt[2 * j]);
  const R rlns = s.rln, rlnn = n.rln;
  const R south = s.north, north = n.north;
  // s-face values carried over from row j-1: zbsw = zbnw(j-1), zbse = zbne(j-1), ...
  const R zbsw = s.zbnw, zbse = s.zbne, ztsw = s.ztnw, ztse = s.ztne;
  const R zbs = s.zbn, zts = s.ztn, pbs = s.pbn, pts = s.ptn;
  R a1, a2, b1, b2, b3, terms1, terms2;
  // levels: a = 0 (k-1), 1 (k), 2 (k+1); rows: b = 0 (j-1), 1 (j); columns: q = 0 (i-1), 1 (i), 2 (i+1)
  // the 8-point means are the means of the faces' quarter sums and the 4-point P means share their
  // centre-column pair (mixed forms; the FP64 form sums in the reference's order)
  R zbe, zte, pbe, pte, zbw, ztw, pbw, ptw;
  if constexpr (std::is_same_v<R, double>) {
    zbe = scale_down<3>(gz(1, 1, 1) + gz(1, 1, 2) + gz(1, 0, 1) + gz(1, 0, 2) + gz(2, 1, 1) + gz(2, 1, 2) + gz(2, 0, 1) + gz(2, 0, 2));
    zte = scale_down<3>(gz(0, 1, 1) + gz(0, 1, 2) + gz(0, 0, 1) + gz(0, 0, 2) + gz(1, 1, 1) + gz(1, 1, 2) + gz(1, 0, 1) + gz(1, 0, 2));
    pbe = Pow2{.25f} * (pp(1, 1, 1) + pp(1, 1, 2) + pp(1, 0, 1) + pp(1, 0, 2));
    pte = Pow2{.25f} * (pp(0, 1, 1) + pp(0, 1, 2) + pp(0, 0, 1) + pp(0, 0, 2));
    zbw = scale_down<3>(gz(1, 1, 1) + gz(1, 1, 0) + gz(1, 0, 1) + gz(1, 0, 0) + gz(2, 1, 1) + gz(2, 1, 0) + gz(2, 0, 1) + gz(2, 0, 0));
    ztw = scale_down<3>(gz(0, 1, 1) + gz(0, 1, 0) + gz(0, 0, 1) + gz(0, 0, 0) + gz(1, 1, 1) + gz(1, 1, 0) + gz(1, 0, 1) + gz(1, 0, 0));
    pbw = Pow2{.25f} * (pp(1, 1, 1) + pp(1, 1, 0) + pp(1, 0, 1) + pp(1, 0, 0));
    ptw = Pow2{.25f} * (pp(0, 1, 1) + pp(0, 1, 0) + pp(0, 0, 1) + pp(0, 0, 0));
  } else {
    zbe = Pow2{.5f} * (n.zbne + s.zbne);
    zte = Pow2{.5f} * (n.ztne + s.ztne);
    zbw = Pow2{.5f} * (n.zbnw + s.zbnw);
    ztw = Pow2{.5f} * (n.ztnw + s.ztnw);
    const R cb = pp(1, 1, 1) + pp(1, 0, 1), ct = pp(0, 1, 1) + pp(0, 0, 1);
    pbe = Pow2{.25f} * (cb + pp(1, 1, 2) + pp(1, 0, 2));
    pte = Pow2{.25f} * (ct + pp(0, 1, 2) + pp(0, 0, 2));
    pbw = Pow2{.25f} * (cb + pp(1, 1, 0) + pp(1, 0, 0));
    ptw = Pow2{.25f} * (ct + pp(0, 1, 0) + pp(0, 0, 0));
  }
  a1 = n.ztne + ztse; b1 = n.ztne * ztse; a2 = n.zbne + zbse; b2 = n.zbne * zbse;
  terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
  terms2 = R(3.) * (a1 - a2);
  const R east = qdiv(Pow2{.5f} * (rlns - rlnn) * (-terms1 * (pbe - pte) + terms2 * (zte * pbe - zbe * pte)), zte - zbe);
  a1 = n.ztnw + ztsw; b1 = n.ztnw * ztsw; a2 = n.zbnw + zbsw; b2 = n.zbnw * zbsw;
  terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
  terms2 = R(3.) * (a1 - a2);
  const R west = qdiv(Pow2{.5f} * (rlns - rlnn) * (-terms1 * (pbw - ptw) + terms2 * (ztw * pbw - zbw * ptw)), ztw - zbw);
  R top, bottom;
  a1 = n.ztne + n.ztnw; a2 = ztse + ztsw;
  terms2 = R(3.) * (a1 - a2);
  if (fabs(qdiv(twice_of(n.ztn - zts), n.ztn + zts - n.zbn - zbs)) > DLOGZ_TOL) {
    b1 = n.ztne * n.ztnw; b2 = ztse * ztsw; b3 = n.ztne * ztse + n.ztnw * ztsw;
    terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
    top = qdiv(Pow2{.5f} * ((n.ptn - pts) * ((rlnn + rlns) * terms1 + (rlnn - rlns) * (b1 + b2 - b3)) + (rlnn + rlns) * terms2 * (n.ztn * pts - zts * n.ptn)),
               n.ztn - zts);
  } else {
    top = Pow2{.25f} * (rlnn + rlns) * (pts + n.ptn) * terms2;
  }
  a1 = n.zbne + n.zbnw; a2 = zbse + zbsw;
  terms2 = R(3.) * (a1 - a2);
  if (fabs(qdiv(twice_of(n.zbn - zbs), n.ztn + zts - n.zbn - zbs)) > DLOGZ_TOL) {
    b1 = n.zbne * n.zbnw; b2 = zbse * zbsw; b3 = n.zbne * zbse + n.zbnw * zbsw;
    terms1 = a1 * a1 - b1 - (a2 * a2 - b2);
    bottom = qdiv(Pow2{.5f} * ((n.pbn - pbs) * ((rlnn + rlns) * terms1 + (rlnn - rlns) * (b1 + b2 - b3)) + (rlnn + rlns) * terms2 * (n.zbn * pbs - zbs * n.pbn)),
                  n.zbn - zbs);
  } else {
    bottom = Pow2{.25f} * (rlnn + rlns) * (pbs + n.pbn) * terms2;
  }
  R pgflat = top - bottom + south - (north + west + east);
  const R dzn = n.ztne - n.zbne + n.ztnw - n.zbnw;
  const R dzs = ztse - zbse + ztsw - zbsw;
  pgflat = qdiv(pgflat, face_width<R>(M.lat, 2 * j - 1, 2 * j + 1) * rho * rlt * (rlns * (dzs + Pow2{.5f} * dzn) + rlnn * (dzn + Pow2{.5f} * dzs)));
  const long long x = plane_offset(M, PL_UV_TEND) + M.at(k, j, i);
  M.dvdt[x] = M.dvdt[x] + to_d(pgflat);
  }
}

// ---------------------------------------------------------------------------------------------
// Meridional pass of hsu_advection, epic_flux.c:1060-1310.  kind: 0/1 interface (unity,
// THETA), 2 = HDRY (v averaged to the layer), 3 = NU_TURB (interface, floor NU_TURB_MIN).  Four launches over all planes k0..nk.
// ---------------------------------------------------------------------------------------------

// the velocity through the v point over its map factor; 0 outside the rows 0..nj+1
template <class R>
__device__ __forceinline__ R vm_at(const DevModel &M, const double *V, int kind, int k, int j, int i) {
  if (j < 0 || j > M.nj + 1) return R(0.);
  R v2d;
  if (kind == 2) v2d = (j >= 1 && j <= M.nj) ? half_of(cv<R>(V[M.at(k, j, i)]) + cv<R>(V[M.at(k - 1, j, i)])) : R(0.);
  else v2d = cv<R>(V[M.at(k, j, i)]);
  return v2d * rt<R>(M, j, RT_MINV_V);
}
template <class R>
__device__ __forceinline__ R hsu_floor(const DevModel &M, int kind, int k) {
  return kind == 2 ? cv<R>(M.h_min[k]) : (kind == 3 ? cv<R>(1.e-3 * M.kinvisc) : R(0.));
}
// The corrector flux through v row j (1..nj) by velocity w: the rows u and d are upstream and
// downstream of it, uu the row beyond u.  a, ap: the field and the predicted field by row.
template <class R, class FA, class FP>
__device__ __forceinline__ R hsu_merid_flux(const DevModel &M, R w, R w_up, int j, R a_min, R DT, FA a, FP ap) {
  const int nj = M.nj;
  const bool neg = is_neg(w);            // from row j south to j-1, else from j-1 north to j
  const int u = neg ? j : j - 1, d = neg ? j - 1 : j, uu = neg ? j + 1 : j - 2;
  const bool edge = neg ? u == nj : u == 0;
  const R au = a(u), ad = a(d), auu = edge ? R(0.) : a(uu);
  R t;
  if (edge) t = fabs(neg ? ad - au : -au + ad) + R(1.e-10);
  else t = fabs((neg ? ad : auu) - twice_of(au) + (neg ? auu : ad)) + R(1.e-10);
  return hsu_face<R>(w, w_up, au, ad, ap(d), edge ? R(0.) : ap(u) - auu, t * t, a_min, a_min, cv<R>(M.mn[2 * j]), DT);
}
// w_s, w_n: the velocities at rows j-1 and j+1
template <class R, class FA, class FP>
__device__ __forceinline__ bool hsu_merid_tainted(const DevModel &M, R w, R w_s, R w_n, int j, FA a, FP ap) {
  const bool neg = is_neg(w);
  const R a_dd = (neg ? j == 1 : j == M.nj) ? R(0.) : a(neg ? j - 2 : j + 1);
  return hsu_tainted<R>(neg, neg ? w_n : w_s, neg ? w_s : w_n, a_dd, ap(neg ? j : j - 1));
}

template <class R>
__global__ void k_hsu_merid_pred(DevModel M, const double *A, int kind, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 0, M.nj + 2, c)) return;   // rows 0..nj+1
  const double *V = M.v + plane_offset(M, PL_UV);
  R ff = R(0.);
  if (c.j >= 1 && c.j <= M.nj) {
    const R w = vm_at<R>(M, V, kind, c.k, c.j, c.i);
    const R north = cv<R>(A[M.at(c.k, c.j, c.i)]), south = cv<R>(A[M.at(c.k, c.j - 1, c.i)]);
    ff = hsu_upwind_tainted<R>(w, north, south) ? quiet_nan<R>() : hsu_upwind<R>(w, north, south);
  }
  write_with_pads(M.work1, M, M.at(c.k, c.j, 0), c.i, ff);
}

template <class R>
__global__ void k_hsu_merid_apred(DevModel M, const double *A, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 0, M.nj + 1, c)) return;
  const double *FF = M.work1;
  const long long x = M.at(c.k, c.j, c.i);
  const R da = (cv<R>(FF[x]) - cv<R>(FF[M.at(c.k, c.j + 1, c.i)])) * cv<R>(M.mn[2 * c.j + 1]) * cv<R>(M.dt);
  write_with_pads(M.work2, M, M.at(c.k, c.j, 0), c.i, A[x] + to_d(da));
}

template <class R>
__global__ void k_hsu_merid_corr(DevModel M, const double *A, int kind, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 0, M.nj + 2, c)) return;
  const int k = c.k, j = c.j, i = c.i, nj = M.nj;
  R ffv = R(0.);
  if (j >= 1 && j <= nj) {
    const double *V = M.v + plane_offset(M, PL_UV);
    const double *AP = M.work2;
    const R w = vm_at<R>(M, V, kind, k, j, i);
    const R w_s = vm_at<R>(M, V, kind, k, j - 1, i), w_n = vm_at<R>(M, V, kind, k, j + 1, i);
    auto a = [&](int jj) { return cv<R>(A[M.at(k, jj, i)]); };
    auto ap = [&](int jj) { return cv<R>(AP[M.at(k, jj, i)]); };
    ffv = hsu_merid_flux<R>(M, w, is_neg(w) ? w_n : w_s, j, hsu_floor<R>(M, kind, k), cv<R>(M.dt), a, ap);
    if (hsu_merid_tainted<R>(M, w, w_s, w_n, j, a, ap)) ffv = quiet_nan<R>();
  }
  write_with_pads(M.work3, M, M.at(k, j, 0), i, ffv);
}

template <class R>
__global__ void k_hsu_merid_update(DevModel M, double *A, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 0, M.nj + 1, c)) return;
  const double *FF = M.work3;
  const long long x = M.at(c.k, c.j, c.i);
  const R da = (cv<R>(FF[x]) - cv<R>(FF[M.at(c.k, c.j + 1, c.i)])) * cv<R>(M.mn[2 * c.j + 1]) * cv<R>(M.dt);
  write_with_pads(A, M, M.at(c.k, c.j, 0), c.i, A[x] + to_d(da));
}

// The four meridional passes fused: one thread per (k, i) marches j = 0..nj and keeps, in a
// sliding register window, the original field A at rows j-1..j+2 (A is updated in place behind
// the march), the velocity at rows j..j+2, the predictor fluxes FF at j+1, j+2, the
// predicted field AP at j, j+1 and the corrector flux FFV at j.  Every value is the same
// expression on the same operands as in the four passes (k_hsu_merid_pred/apred/corr/update),
// so the results are identical bit for bit, with no scratch traffic.  Row j+3's loads are issued
// at the top of iteration j, ahead of the arithmetic that does not need them.
template <class R>
__global__ void k_hsu_meridional(DevModel M, double *A, int kind, int k0) {
  if (epic_member(M, A)) return;
  const int i = 1 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int k = k0 + (int)blockIdx.y;
  if (i > M.ni) return;
  const int nj = M.nj;
  const double *V = M.v + plane_offset(M, PL_UV);
  const R DT = cv<R>(M.dt), a_min = hsu_floor<R>(M, kind, k);
  auto ld = [&](int jj) { return A[M.at(k, jj, i)]; };
  auto ff_of = [&](int jj, R w, R am1, R a0) { return (jj >= 1 && jj <= nj) ? (hsu_upwind_tainted<R>(w, a0, am1) ? quiet_nan<R>() : hsu_upwind<R>(w, a0, am1)) : R(0.); };
  auto ap_of = [&](int jj, double ad, R ff0, R ff1) { return cv<R>(ad + to_d((ff0 - ff1) * cv<R>(M.mn[2 * jj + 1]) * DT)); };
  // window at the top of iteration j
  R a_m1 = R(0.), a_0, a_1, a_2;   // A(j-1..j+2)
  double ad_0, ad_1, ad_2;         // A(j..j+2) in binary64
  R w_0, w_1, w_2;                 // velocity at j..j+2
  R ff_1, ff_2;                    // FF(j+1), FF(j+2)
  R ap_0, ap_1;                    // AP(j), AP(j+1)
  R ffv_0 = R(0.);                 // FFV(j); FFV(0) = 0
  ad_0 = ld(0); ad_1 = ld(1); ad_2 = ld(2);
  a_0 = cv<R>(ad_0); a_1 = cv<R>(ad_1); a_2 = cv<R>(ad_2);
  w_0 = vm_at<R>(M, V, kind, k, 0, i);
  w_1 = vm_at<R>(M, V, kind, k, 1, i);
  w_2 = vm_at<R>(M, V, kind, k, 2, i);
  {
    const R ff_0 = R(0.);   // FF(0): row 0 is outside 1..nj
    ff_1 = ff_of(1, w_1, a_0, a_1);
    ff_2 = ff_of(2, w_2, a_1, a_2);
    ap_0 = ap_of(0, ad_0, ff_0, ff_1);
    ap_1 = ap_of(1, ad_1, ff_1, ff_2);
  }
  for (int j = 0; j <= nj; j++) {
    // row j+3's inputs (rows beyond nj+1 do not exist and are not used)
    const int j3 = j + 3;
    double ad_3 = 0.;
    R w_3 = R(0.);
    if (j3 <= nj + 1) {
      ad_3 = ld(j3);
      w_3 = vm_at<R>(M, V, kind, k, j3, i);
    }
    // FFV(j+1): the corrector flux of row j+1 (k_hsu_merid_corr), its rows j-1..j+2 in the window
    R ffv_1 = R(0.);
    if (j + 1 <= nj) {
      auto a = [&](int jj) { return jj <= j ? (jj < j ? a_m1 : a_0) : (jj > j + 1 ? a_2 : a_1); };
      auto ap = [&](int jj) { return jj <= j ? ap_0 : ap_1; };
      ffv_1 = hsu_merid_flux<R>(M, w_1, is_neg(w_1) ? w_2 : w_0, j + 1, a_min, DT, a, ap);
      if (hsu_merid_tainted<R>(M, w_1, w_0, w_2, j + 1, a, ap)) ffv_1 = quiet_nan<R>();
    }
    // the update of row j (k_hsu_merid_update)
    const R da = (ffv_0 - ffv_1) * cv<R>(M.mn[2 * j + 1]) * cv<R>(M.dt);
    write_with_pads(A, M, M.at(k, j, 0), i, ad_0 + to_d(da));
    // advance the window to j+1: FF(j+3), AP(j+2)
    const R a_3 = cv<R>(ad_3);
    const R ff_3 = ff_of(j3, w_3, a_2, a_3);
    const R ap_2 = (j + 2 <= nj) ? ap_of(j + 2, ad_2, ff_2, ff_3) : R(0.);
    a_m1 = a_0; a_0 = a_1; a_1 = a_2; a_2 = a_3;
    ad_0 = ad_1; ad_1 = ad_2; ad_2 = ad_3;
    w_0 = w_1; w_1 = w_2; w_2 = w_3;
    ff_1 = ff_2; ff_2 = ff_3;
    ap_0 = ap_1; ap_1 = ap_2;
    ffv_0 = ffv_1;
  }
}

// The four passes in one kernel over tiles: a block takes TC neighbouring columns of one level, every
// row, with the field, the velocity, the fluxes and the predicted field in shared memory [row][column]
// and a barrier between the passes.  The same expressions on the same operands again.  On small and
// middle grids the four passes are four launches with too few warps each (27 us in all at 128x64x20 in
// the FP64 form), the march one thread a column in a chain of nj rows.
template <class R>
__global__ void __launch_bounds__(256) k_hsu_merid_tile(DevModel M, double *A, int kind, int k0, int TC) {
  if (epic_member(M, A)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nj = M.nj, tx = (int)threadIdx.x & (TC - 1), ty = (int)threadIdx.x / TC, ny = (int)blockDim.x / TC;
  const int i = (int)blockIdx.x * TC + tx + 1, k = k0 + (int)blockIdx.y;
  if ((int)blockIdx.x * TC >= M.ni) return;   // a member narrower than the launch
  const bool live = i <= M.ni;
  R *a = reinterpret_cast<R *>(smraw) + tx, *w = a + (nj + 2) * TC, *ff = w + (nj + 2) * TC, *ap = ff + (nj + 2) * TC;
  const double *V = M.v + plane_offset(M, PL_UV);
  const R DT = cv<R>(M.dt), a_min = hsu_floor<R>(M, kind, k);
  unsigned top = 0;
  for (int j = ty; j <= nj + 1; j += ny) {
    a[j * TC] = live && j <= nj ? cv<R>(A[M.at(k, j, i)]) : R(0.);
    const R v = live ? vm_at<R>(M, V, kind, k, j, i) : R(0.);
    w[j * TC] = v;
    top = max(top, top_bits(v));   // the poles' velocities are in no flux
  }
  __syncthreads();
  for (int j = ty; j <= nj + 1; j += ny)
    ff[j * TC] = j >= 1 && j <= nj ? hsu_upwind<R>(w[j * TC], a[j * TC], a[(j - 1) * TC]) : R(0.);
  __syncthreads();
  auto predict = [&] {
    if (live)
      for (int j = ty; j <= nj; j += ny) {
        const R p = cv<R>(A[M.at(k, j, i)] + to_d((ff[j * TC] - ff[(j + 1) * TC]) * cv<R>(M.mn[2 * j + 1]) * DT));
        ap[j * TC] = p;
        top = max(top, top_bits(p));
      }
  };
  predict();
  const bool odd = __syncthreads_or(top >= NONFINITE_BITS<R>);
  if (odd) {
    for (int j = 1 + ty; j <= nj; j += ny)
      if (hsu_upwind_tainted<R>(w[j * TC], a[j * TC], a[(j - 1) * TC])) ff[j * TC] = quiet_nan<R>();
    __syncthreads();
    predict();
    __syncthreads();
  }
  if (live)
    for (int j = 1 + ty; j <= nj; j += ny) {   // ff of rows 0 and nj+1 stays 0
      const R v = w[j * TC];
      ff[j * TC] = hsu_merid_flux<R>(M, v, w[(is_neg(v) ? j + 1 : j - 1) * TC], j, a_min, DT, [&](int jj) { return a[jj * TC]; },
                                     [&](int jj) { return ap[jj * TC]; });
    }
  if (odd && live)
    for (int j = 1 + ty; j <= nj; j += ny)
      if (hsu_merid_tainted<R>(M, w[j * TC], w[(j - 1) * TC], w[(j + 1) * TC], j, [&](int jj) { return a[jj * TC]; }, [&](int jj) { return ap[jj * TC]; }))
        ff[j * TC] = quiet_nan<R>();
  __syncthreads();
  if (live)
    for (int j = ty; j <= nj; j += ny) {
      const R da = (ff[j * TC] - ff[(j + 1) * TC]) * cv<R>(M.mn[2 * j + 1]) * cv<R>(M.dt);
      write_with_pads(A, M, M.at(k, j, 0), i, A[M.at(k, j, i)] + to_d(da));
    }
}

// ---------------------------------------------------------------------------------------------
// Meridional pass of akima_advection, epic_flux.c:1752-1820.  kind: 0/1 interface (unity,
// THETA; V of the interface), 2 = HDRY (V averaged to the layer).  Two launches over planes
// k0..nk: the fluxes FF (v rows 1..nj, into work3), then the update of rows 0..nj.
// ---------------------------------------------------------------------------------------------

template <class R>
__device__ __forceinline__ R akima_mean(R d0, R d1) {   // the dela of akima_advection
  const R tmp = d0 * d1;
  return (tmp > R(0.)) ? qdiv(twice_of(tmp), d0 + d1) : R(0.);
}

template <class R>
__global__ void k_akima_merid_flux(DevModel M, const double *A, int kind, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 1, M.nj, c)) return;   // v rows 1..nj
  const int k = c.k, j = c.j, i = c.i, nj = M.nj;
  auto a = [&](int jj) { return cv<R>(A[M.at(k, jj, i)]); };
  // deltaa(jj) = A(jj) - A(jj-1) on rows 1..nj, 0 elsewhere
  auto deltaa = [&](int jj) { return (jj < 1 || jj > nj) ? R(0.) : a(jj) - a(jj - 1); };
  const R dl_j = akima_mean<R>(deltaa(j), deltaa(j + 1));
  const R dl_jm = akima_mean<R>(deltaa(j - 1), deltaa(j));
  const double *V = M.v + plane_offset(M, PL_UV);
  const R v2d = kind == 2 ? half_of(cv<R>(V[M.at(k, j, i)]) + cv<R>(V[M.at(k - 1, j, i)])) : cv<R>(V[M.at(k, j, i)]);
  const R m_2j_inv = (fabs(M.lat[2 * j]) == 90.) ? R(0.) : qdiv(R(1.), cv<R>(M.m[2 * j]));
  const R aval = half_of(a(j) + a(j - 1)) - qdiv(dl_j - dl_jm, R(6.));
  write_with_pads(M.work3, M, M.at(k, j, 0), i, to_d(v2d * aval * m_2j_inv));
}

template <class R>
__global__ void k_akima_merid_update(DevModel M, double *A, int k0) {
  if (epic_member(M, A)) return;
  Cell c;
  if (!cell3(M, k0, M.nk - k0 + 1, 0, M.nj + 1, c)) return;   // rows 0..nj
  const int k = c.k, j = c.j, nj = M.nj;
  const double *FF = M.work3;
  auto ff = [&](int jj) { return (jj < 1 || jj > nj) ? R(0.) : cv<R>(FF[M.at(k, jj, c.i)]); };
  const long long x = M.at(k, j, c.i);
  const R da = (ff(j) - ff(j + 1)) * cv<R>(M.mn[2 * j + 1]) * cv<R>(M.dt);
  write_with_pads(A, M, M.at(k, j, 0), c.i, A[x] + to_d(da));
}

// ---------------------------------------------------------------------------------------------
// Hyperviscosity, epic_subgrid.c:590-1232
// ---------------------------------------------------------------------------------------------

// d2dy2 of planes k0..k1 of src into dst (coefficients per row from the init block, :1049-1141).
template <class R>
__global__ void k_d2dy2(DevModel M, const double *src, int src_sel, double *dst, int vgrid, int order, int k0, int nkk,
                        int of_state) {
  if (epic_member(M, src, dst)) return;
  Cell c;
  const int nrows = vgrid ? M.nj + 2 : M.nj + 1;   // v: j = 0..nj+1, h: j = 0..nj
  if (!cell3(M, k0, nkk, 0, nrows, c)) return;
  src += plane_offset(M, src_sel);
  const int k = c.k, j = c.j, i = c.i, nj = M.nj;
  const R *cf = visc_coef<R>(M, vgrid, order, j);   // the member's own (they depend on dt and dy0)
  const R a0 = cf[0], a1 = cf[1], a2 = cf[2];
  auto h = [&](int jj) { return cv<R>(src[M.at(k, jj, i)]); };
  R d;
  const int jlast = vgrid ? nj + 1 : nj;
  if (!std::is_same_v<R, double> && of_state) {
    // The mixed forms' second difference of a state field: the three coefficients sum to zero
    // (to ~1e-14 of the largest), so the stencil is a0 (h0 - h1) + a2 (h2 - h1) with the
    // differences taken in binary64 -- in binary32 the field's own rounding (1e-7 of its value,
    // 1e-4 of a neighbour difference) would enter the hyperviscous increment every step.
    const int m = j == 0 ? 1 : (j == jlast ? j - 1 : j);
    const double hm = src[M.at(k, m, i)];
    d = a0 * cv<R>(src[M.at(k, m - 1, i)] - hm) + a2 * cv<R>(src[M.at(k, m + 1, i)] - hm);
  } else if (j == 0) d = a0 * h(0) + a1 * h(1) + a2 * h(2);
  else if (j == jlast) d = a0 * h(j - 2) + a1 * h(j - 1) + a2 * h(j);
  else d = a0 * h(j - 1) + a1 * h(j) + a2 * h(j + 1);
  write_with_pads(dst, M, M.at(k, j, 0), i, d);
}

// The first two d2dy2 passes of meridional_hyperviscosity in one kernel: the first (of the state field;
// binary64 differences in the mixed forms as in k_d2dy2) into shared memory, the second from
// there into dst.  Block = TC columns of one layer k0 + blockIdx.y, every row; the values are
// those of two k_d2dy2 launches (the mixed forms' intermediate is a float either way), without the
// intermediate volume's write and read.
template <class R>
__global__ void __launch_bounds__(256) k_d2dy2_pair(DevModel M, const double *src, int src_sel, double *dst, int vgrid, int k0, int TC) {
  if (epic_member(M, src, dst)) return;
  constexpr bool exact = std::is_same_v<R, double>;
  extern __shared__ __align__(16) unsigned char smraw[];
  src += plane_offset(M, src_sel);
  const int tx = (int)threadIdx.x & (TC - 1), ty = (int)threadIdx.x / TC, ny = (int)blockDim.x / TC;
  R *d1 = reinterpret_cast<R *>(smraw) + tx;   // [row][column]
  const int i = (int)blockIdx.x * TC + tx + 1;
  const int k = k0 + (int)blockIdx.y;
  const int nj = M.nj, jlast = vgrid ? nj + 1 : nj;
  const bool live = i <= M.ni;
  for (int j = ty; j <= jlast; j += ny) {
    R d = R(0.);
    if (live) {
      const R *cf = visc_coef<R>(M, vgrid, 2, j);
      const R a0 = cf[0], a2 = cf[2];
      const int m = j == 0 ? 1 : (j == jlast ? j - 1 : j);
      const double hm = src[M.at(k, m, i)];
      if constexpr (exact) d = a0 * src[M.at(k, m - 1, i)] + cf[1] * hm + a2 * src[M.at(k, m + 1, i)];
      else d = a0 * cv<R>(src[M.at(k, m - 1, i)] - hm) + a2 * cv<R>(src[M.at(k, m + 1, i)] - hm);
    }
    d1[j * TC] = d;
  }
  __syncthreads();
  if (!live) return;
  for (int j = ty; j <= jlast; j += ny) {
    const R *cf = visc_coef<R>(M, vgrid, 4, j);
    const R a0 = cf[0], a1 = cf[1], a2 = cf[2];
    const int m = j == 0 ? 1 : (j == jlast ? j - 1 : j);
    const R d = a0 * d1[(m - 1) * TC] + a1 * d1[m * TC] + a2 * d1[(m + 1) * TC];
    write_with_pads(dst, M, M.at(k, j, 0), i, to_d(d));
  }
}

// A += dt*sign*D over the rows the reference updates (v: 1..nj, h: 0..nj).
template <class R>
__global__ void k_visc_apply(DevModel M, double *A, int sel, const double *D, int vgrid, double sign, int k0, int nkk) {
  if (epic_member(M, A, D)) return;
  Cell c;
  if (!cell3(M, k0, nkk, vgrid ? 1 : 0, vgrid ? M.nj : M.nj + 1, c)) return;
  A += plane_offset(M, sel);
  const long long x = M.at(c.k, c.j, c.i);
  write_with_pads(A, M, M.at(c.k, c.j, 0), c.i, A[x] + to_d(cv<R>(M.dt) * cv<R>(sign) * cv<R>(D[x])));
}

// One row of A (i = 1..ni and its periodic pads) with meridional_hyperviscosity's last order applied:
// a[i] = A + dt sign D (epic_subgrid.c:650-712), D the zonally filtered second difference.  filter: D is not
// filtered yet; the row is, in x (ni compute-type values), by the warp's 32 lanes.
template <class R>
__device__ __forceinline__ void visc_row(const DevModel &M, const double *A, const double *D, int base, int j, int vgrid, double sign, int filter,
                                         R *x, double *a, int lane) {
  const int ni = M.ni, lg = fft_log(ni);
  const bool filt = filter && row_is_filtered(M, j, vgrid);
  const R c = cv<R>(M.dt) * cv<R>(sign), scale = filter_scale<R>(ni);
  if (filt) {
    for (int e = lane; e < ni; e += 32) x[fft_place(e, lg)] = cv<R>(D[base + e + 1]);
    __syncwarp();
    const RowLane L = {lane, 32, 0, 0, true};
    filter_row<R>(M, reinterpret_cast<Cplx<R> *>(x), (vgrid ? M.high_lat_pv : M.high_lat_h) + M.at2(j, 0), L);
  }
  for (int e = lane; e < ni; e += 32) {
    const R d = filt ? x[e] * scale : cv<R>(D[base + e + 1]);
    const double v = A[base + e + 1] + to_d(c * d);
    a[e + 1] = v;
    if (e == 0) a[ni + 1] = v;
    if (e == ni - 1) a[0] = v;
  }
  __syncwarp();
}

// zonal_hyperviscosity, epic_subgrid.c:715-808, in the FP64 form: `rows` rows per block, a warp per
// row at a time; the row means, in the reference's order, by one warp with a row per lane (row_sum).
// Bound by those additions: with one lane of each row's warp summing it, 4 orders x ni additions a row
// held the binary64 pipe (71% busy) for 36 us a field at 128x64x20.  The meridional part's filter and
// last update come first (visc_row), on the row in shared memory: two launches and two passes fewer.
// A block with filtered rows alone took 24,000 cycles for them before its sums (12,000 each, 8,200 of them
// additions), beside blocks without any: the rows lie all over the latitudes, the mean is a product with a
// power of 2, and the coefficients are ready before the rows.  12 steps of 128x64x20 10.24 -> 10.10 ms, 8
// leapfrog steps of 64x47x13 3.14 -> 2.99 ms, 3 of 256x128x32 15.0 -> 14.8 ms.
__global__ void __launch_bounds__(256, 3) k_zonal_visc_rows(DevModel M, double *A, int sel, const double *D, double msign, int filter, int jbot,
                                                         int jhalf, int k0, int nkk, int restore, int rows) {
  if (epic_member(M, A, D)) return;
  extern __shared__ __align__(16) double vr[];
  if (filter) warm_filter<double>(M, nullptr);
  __shared__ double s_mean[32], s_dc[4][32];
  const int ni = M.ni, W = ni + 2, lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5);
  const int nr = M.nj - jbot + 1;
  // row r of block b is the member's row b + r nb, levels fastest: a block's rows lie all over the latitudes,
  // so every block has its share of the filtered ones
  const int total = nr * nkk, nb = (total + rows - 1) / rows;
  if ((int)blockIdx.x >= nb) return;   // a member with fewer rows than the launch
  const int nl = (total - (int)blockIdx.x + nb - 1) / nb;
  A += plane_offset(M, sel);
  double *a = vr, *h = a + rows * W, *d = h + rows * W;
  auto row_at = [&](int r, int &j, int &k) {
    const int at = (int)blockIdx.x + r * nb, q = at / nkk;
    j = jbot + q;
    k = k0 + at - q * nkk;
  };
  if ((int)threadIdx.x < nl) {   // the coefficients, while the rows come
    int j, k;
    row_at((int)threadIdx.x, j, k);
    const double mm = M.m[2 * j + jhalf];
    const bool taper = fabs(M.lat[2 * j + jhalf]) > M.lat0;
#pragma unroll
    for (int q = 0; q < 4; q++) s_dc[q][threadIdx.x] = taper ? M.coef[2 * q + 2] * M.m0 * M.m0 : M.coef[2 * q + 2] * mm * mm;
  }
  for (int r = w; r < nl; r += nw) {
    int j, k;
    row_at(r, j, k);
    visc_row<double>(M, A, D, M.at(k, j, 0), j, jhalf == 0, msign, filter, d + r * W, a + r * W, lane);
    for (int i = lane; i <= ni + 1; i += 32) h[r * W + i] = a[r * W + i];
  }
  __syncthreads();
  double sign = 1.;
  // fully unrolled so that M.coef[], M.nu[] are indexed by constants (M stays in registers)
#pragma unroll
  for (int itmp = 2; itmp <= 8; itmp += 2) {
    for (int r = w; r < nl; r += nw) {
      const double dc = s_dc[itmp / 2 - 1][r];
      const double *hr = h + r * W;
      for (int i = lane + 1; i <= ni; i += 32) d[r * W + i] = dc * (hr[i - 1] - twice_of(hr[i]) + hr[i + 1]);
    }
    __syncthreads();
    if ((int)threadIdx.x < nl) s_mean[threadIdx.x] = row_sum(d + (int)threadIdx.x * W + 1, ni) * inv_pow2(ni);
    __syncthreads();
    for (int r = w; r < nl; r += nw) {
      const double mean = s_mean[r];
      double *dr = d + r * W;
      for (int i = lane + 1; i <= ni; i += 32) {
        const double v = dr[i] - mean;
        dr[i] = v;
        if (i == 1) dr[ni + 1] = v;
        if (i == ni) dr[0] = v;
        if (M.nu[itmp] > 0.) a[r * W + i] += M.dt * sign * v;
      }
    }
    __syncwarp();
    sign = -sign;
    double rest = 0.;
#pragma unroll
    for (int q = itmp + 2; q <= 8; q += 2) rest += M.nu[q];
    if (!(rest > 0.)) break;
    double *t = h; h = d; d = t;   // swap roles
  }
  // restore (HDRY): restore_mass, which the hyperviscosity step calls next (epic_subgrid.c:240),
  // on the new row -- the same max per cell, one pass fewer
  for (int r = w; r < nl; r += nw) {
    int j, k;
    row_at(r, j, k);
    const int base = M.at(k, j, 0);
    for (int i = lane + 1; i <= ni; i += 32) {
      const double v = a[r * W + i];
      write_with_pads(A, M, base, i, restore ? dmaxr(M.h_min[k], v) : v);
    }
  }
}

// The same in the mixed forms: one warp per row (j, k), blockDim.x / 32 rows per block.  The updated
// row stays in FP64; the row mean is an FP32 warp reduction.
__global__ void __launch_bounds__(128, 8) k_zonal_visc_mixed(DevModel M, double *A, int sel, const double *D, double msign, int filter, int jbot, int jhalf, int k0, int restore) {
  if (epic_member(M, A, D)) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  if (filter) warm_filter<float>(M, nullptr);
  const int ni = M.ni, lane = (int)(threadIdx.x & 31), w = (int)(threadIdx.x >> 5), nw = (int)(blockDim.x >> 5);
  const int j = jbot + (int)blockIdx.x * nw + w;
  const int k = k0 + (int)blockIdx.y;
  if (j > M.nj) return;
  A += plane_offset(M, sel);
  const long long base = M.at(k, j, 0);
  const size_t row_bytes = (size_t)(ni + 2) * (sizeof(double) + 2 * sizeof(float));
  double *a = reinterpret_cast<double *>(smraw + w * row_bytes);
  float *hh = reinterpret_cast<float *>(a + (ni + 2)), *d = hh + (ni + 2);
  const unsigned full = 0xffffffffu;
  visc_row<float>(M, A, D, (int)base, j, jhalf == 0, msign, filter, d, a, lane);
  // the first second difference is of the field itself: its neighbour differences a(i+1) - a(i) in
  // binary64, one per point (k_d2dy2)
  for (int i = lane; i <= ni; i += 32) hh[i] = d2f(a[i + 1] - a[i]);
  __syncwarp();
  const bool taper = fabs(M.lat[2 * j + jhalf]) > M.lat0;
  const double mm = M.m[2 * j + jhalf];
  float sign = 1.f;
  // fully unrolled so that M.coef[], M.nu[] are indexed by constants (M stays in registers)
#pragma unroll
  for (int itmp = 2; itmp <= 8; itmp += 2) {
    const float dc = d2f(taper ? M.coef[itmp] * M.m0 * M.m0 : M.coef[itmp] * mm * mm);
    // the row sum of a periodic second difference vanishes but for rounding: FP32 suffices
    float fm = 0.f;
    for (int i = lane + 1; i <= ni; i += 32) {
      const float v = itmp == 2 ? dc * (hh[i] - hh[i - 1]) : dc * (hh[i - 1] - 2.f * hh[i] + hh[i + 1]);
      d[i] = v;
      fm += v;
    }
    for (int o = 16; o > 0; o >>= 1) fm += __shfl_xor_sync(full, fm, o);
    const float mean = fm / (float)ni;
    __syncwarp();
    for (int i = lane + 1; i <= ni; i += 32) {
      const float v = d[i] - mean;
      d[i] = v;
      if (i == 1) d[ni + 1] = v;
      if (i == ni) d[0] = v;
      if (M.nu[itmp] > 0.) a[i] += f2d(d2f(M.dt) * sign * v);
    }
    __syncwarp();
    sign = -sign;
    double rest = 0.;
#pragma unroll
    for (int q = itmp + 2; q <= 8; q += 2) rest += M.nu[q];
    if (!(rest > 0.)) break;
    float *t = hh; hh = d; d = t;   // swap roles
  }
  // restore (HDRY): restore_mass too (k_zonal_visc_rows)
  for (int i = lane + 1; i <= ni; i += 32) write_with_pads(A, M, base, i, restore ? dmaxr(M.h_min[k], a[i]) : a[i]);
}

// ---------------------------------------------------------------------------------------------
// divergence, vorticity, store_diag (epic_funcs_diag.c:3963-4445) and the Richardson number
// ---------------------------------------------------------------------------------------------

// DIV of (UU, VV) on planes k0.., rows 0..nj, divergence() :4064-4117
template <class R, int ROWS>
__global__ void k_divergence(DevModel M, const double *UU, const double *VV, int vsel, double *DI, int k0, int nkk) {
  if (epic_member(M, UU, VV, DI)) return;
  March s;
  if (!march<ROWS>(M, k0, nkk, 0, M.nj, s)) return;
  VV += plane_offset(M, vsel);
  const int k = s.k, i = s.i;
  auto vm = [&](int j) { return cv<R>(VV[M.at(k, j, i)]) * rt<R>(M, j, RT_MINV_V); };   // 0 at the poles
  R vs = vm(s.j0);
#pragma unroll
  for (int q = 0; q < ROWS; q++) {
    const int j = s.j0 + q;
    if (ROWS > 1 && j > s.j1) break;
    const int x = M.at(k, j, i);
    const R n_inv = rt<R>(M, j, RT_NINV_H), vn = vm(j + 1);
    write_with_pads(DI, M, x - i, i, to_d(rt<R>(M, j, RT_MN_H) * ((cv<R>(UU[x + 1]) * n_inv - cv<R>(UU[x]) * n_inv) + (vn - vs))));
    vs = vn;
  }
}

// Interior potential vorticity, vorticity(ON_SIGMATHETA, POTENTIAL) :4168-4186, planes 0..nk, rows 1..nj.
template <class R, int ROWS>
__global__ void k_pv_interior(DevModel M, const double *VV) {
  if (epic_member(M, VV)) return;
  March s;
  if (!march<ROWS>(M, 0, M.nk + 1, 1, M.nj, s)) return;
  const int k = s.k, i = s.i;
  const double *UU = M.u + plane_offset(M, PL_UV);
  auto um = [&](int j) { return cv<R>(UU[M.at(k, j, i)]) * rt<R>(M, j, RT_MINV_H); };
  auto hm = [&](int j) { return (cv<R>(M.h3[M.at(k, j, i)]) + cv<R>(M.h3[M.at(k, j, i - 1)])) * rt<R>(M, j, RT_MNINV_H); };
  R us = um(s.j0 - 1), hs = hm(s.j0 - 1);
#pragma unroll
  for (int q = 0; q < ROWS; q++) {
    const int j = s.j0 + q;
    if (ROWS > 1 && j > s.j1) break;
    const int x = M.at(k, j, i);
    const R un = um(j), hn = hm(j);
    const R ze = rt<R>(M, j, RT_M_V) * ((cv<R>(VV[x]) - cv<R>(VV[x - 1])) + rt<R>(M, j, RT_N_V) * (us - un));
    const R h_pv = (hn + hs) * rt<R>(M, j, RT_MNPV);
    write_with_pads(M.pv3, M, x - i, i, to_d(qdiv(ze + rt<R>(M, j, RT_F_V), h_pv)));
    us = un; hs = hn;
  }
}

// Polar potential vorticity from the circulation of the adjacent u row, :4279-4341.
// One block per lv planes: the four rows of each staged by every thread, then summed in the
// reference's order, a row per lane.  One thread summing a plane's four rows one after another took
// 27 us at 128x64x20.
__global__ void __launch_bounds__(256) k_pv_poles(DevModel M, int lv) {
  if (epic_member(M)) return;
  extern __shared__ double rows[];   // [lv][4][ni+1]: U(j=0), H(j=0), U(j=nj), H(j=nj) of each plane
  __shared__ double sum[32], pole[16];
  const int ni = M.ni, J = M.nj, k0 = (int)blockIdx.x * lv, nl = min(lv, M.nk + 1 - k0);
  const double *UU = M.u + plane_offset(M, PL_UV);
  const double *HH = M.h3;
#pragma unroll 4
  for (int t = (int)threadIdx.x; t < 4 * nl * ni; t += (int)blockDim.x) {
    const int r = t / ni, i = t - r * ni;
    const double v = ((r & 1) ? HH : UU)[M.at(k0 + (r >> 2), (r & 2) ? J : 0, i + 1)];
    rows[r * (ni + 1) + i] = (r & 3) == 0 ? -v : v;   // the south's circulation is the negated sum
  }
  __syncthreads();
  const int t = (int)threadIdx.x;
  if (t < 4 * nl) sum[t] = row_sum(rows + t * (ni + 1), ni);
  __syncthreads();
  if (t < 2 * nl) {
    const int north = t & 1;
    double ze = sum[2 * t], h = sum[2 * t + 1];
    ze *= north ? M.mn[2 * (J + 1)] / (M.m[2 * J + 1] * (double)(M.ni)) : M.mn[0] / ((M.m[1]) * (double)(M.ni));
    h *= inv_pow2(M.ni);
    pole[t] = (ze + (north ? M.f[2 * (J + 1)] : M.f[0])) / h;
  }
  __syncthreads();
  for (int q = (int)threadIdx.x; q < 2 * nl * (ni + 2); q += (int)blockDim.x) {
    const int r = q / (ni + 2), i = q - r * (ni + 2);
    M.pv3[M.at(k0 + (r >> 1), (r & 1) ? M.nj + 1 : 0, i)] = pole[r];
  }
}

// Richardson number in the layers, get_richardson/get_brunt2 (:2885-3156).  The V term of
// dvdz2 keeps the reference's sign slip (:3127-3128); only dudz2 decides the 1e6 branch.
template <class R>
__global__ void k_ri2(DevModel M) {
  if (epic_member(M)) return;
  Cell c;
  if (!cell3(M, 1, M.nk, 0, M.nj + 1, c)) return;
  const int k = c.k, j = c.j, i = c.i;
  const long long off = plane_offset(M, PL_UV);
  const double *U = M.u + off, *V = M.v + off;
  auto u = [&](int kk, int jj, int ii) { return cv<R>(U[M.at(kk, jj, ii)]); };
  auto v = [&](int kk, int jj, int ii) { return cv<R>(V[M.at(kk, jj, ii)]); };
  R dudz2 = half_of(u(k - 1, j, i) + u(k - 1, j, i + 1) - u(k, j, i) - u(k, j, i + 1));
  R dvdz2 = half_of(v(k - 1, j, i) + v(k - 1, j + 1, i) - v(k, j, i) + v(k, j + 1, i));
  dudz2 *= dudz2;
  dvdz2 *= dvdz2;
  R ri;
  if (RMath<R>::cmp(dudz2, R(0.)) != 0) {
    const long long x = M.at(k, j, i);
    const R pressure = cv<R>(M.p2[x]), temperature = cv<R>(M.t2[x]), density = cv<R>(M.rho2[x]);
    const R cp = R(1004.), mu = cv<R>(M.mu_dry);
    const R deltap = R(0.001) * pressure, deltaT = R(0.001) * temperature;
    auto dens = [&](R p, R t) { return qdiv(p * mu, R(8.314472e+3) * t); };   // return_density
    const R drho_dp_T = qdiv(dens(pressure + deltap, temperature) - dens(pressure - deltap, temperature), twice_of(deltap));
    const R drho_dT_p = qdiv(dens(pressure, temperature + deltaT) - dens(pressure, temperature - deltaT), twice_of(deltaT));
    const R Drho_Dp = qdiv(cv<R>(M.rho3[x]) - cv<R>(M.rho3[M.at(k - 1, j, i)]), cv<R>(M.p3[x]) - cv<R>(M.p3[M.at(k - 1, j, i)]));
    const R g = cv<R>(M.grav[2 * j + 1]);
    const R brunt2 = g * g * (Drho_Dp - drho_dp_T + qdiv(temperature, cp * density * density) * drho_dT_p * drho_dT_p);
    ri = qdiv(brunt2, dudz2 + dvdz2);
  } else {
    ri = R(1.e+6);
  }
  write_with_pads(M.ri2, M, M.at(k, j, 0), i, ri);
}

// divergence_damping apply step, epic_subgrid.c:1857-1881 (DIV from k_divergence in work2).
template <class R>
__global__ void k_divdamp_apply(DevModel M) {
  if (epic_member(M)) return;
  const double nudiv = M.nudiv;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned per = (unsigned)(M.nk - 1) * (unsigned)(M.nj + 1) * (unsigned)M.ni;
  if (t >= 2 * per) return;
  const int isv = t >= per;
  int i, j, k;
  cell_kji(M, isv ? t - per : t, k, j, i);
  const double *DIV = M.work2;
  const long long off = plane_offset(M, PL_UV_TEND);
  if (!isv) {
    const R coef = cv<R>((M.lat[2 * j + 1] > M.lat0) ? nudiv * M.m0 : nudiv * M.m[2 * j + 1]);
    const long long x = off + M.at(k, j, i);
    M.dudt[x] = M.dudt[x] + to_d(coef * (cv<R>(DIV[M.at(k, j, i)]) - cv<R>(DIV[M.at(k, j, i - 1)])));
  } else if (j >= 1) {
    const R coef = cv<R>(nudiv * M.n[2 * j]);
    const long long x = off + M.at(k, j, i);
    M.dvdt[x] = M.dvdt[x] + to_d(coef * (cv<R>(DIV[M.at(k, j, i)]) - cv<R>(DIV[M.at(k, j - 1, i)])));
  }
}

// ---------------------------------------------------------------------------------------------
// Time update: adams_bashforth_step / leapfrog_step (epic_timestep.c:406-615), the index
// rotation (:257-274) and timeplane_bookkeeping (epic_funcs_diag.c:7086-7124).
// ---------------------------------------------------------------------------------------------

__global__ void k_uv_decide(DevModel M) {
  if (epic_member(M)) return;
  Ctl *c = M.ctl;
  for (int w = 0; w < 2; w++) {
    const double *val = w == 0 ? M.u : M.v, *ten = w == 0 ? M.dudt : M.dvdt;
    const int jlo = w == 0 ? 0 : 1;
    const long long cell = M.at(1, jlo, 1);
    if (M.uv_scheme == EPIC_UV_AB3) {
      double *ab = c->ab[w];
      if (ten[(long long)c->it_minus2 * M.n3 + cell] == DBL_MAX) {
        if (ten[(long long)c->it_minus1 * M.n3 + cell] == DBL_MAX) { ab[0] = 1.; ab[1] = 0.; ab[2] = 0.; }
        else { ab[0] = 3. / 2.; ab[1] = -1. / 2.; ab[2] = 0.; }
      } else { ab[0] = 23. / 12.; ab[1] = -16. / 12.; ab[2] = 5. / 12.; }
      for (int q = 0; q < 3; q++) {
        const dfl d = d2df(ab[q]);
        c->abf[w][q] = make_float2(d.hi, d.lo);
      }
    } else {
      c->lf_first[w] = val[(long long)c->it_minus1 * M.n3 + cell] == DBL_MAX;
    }
  }
}

__global__ void k_uv_update(DevModel M) {
  if (epic_member(M)) return;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned per = (unsigned)(M.nk - 1) * (unsigned)(M.nj + 1) * (unsigned)M.ni;
  if (t >= 2 * per) return;
  const int w = t >= per;
  int i, j, k;
  cell_kji(M, w ? t - per : t, k, j, i);
  if (w == 1 && j == 0) return;   // v is updated for j = 1..nj
  const Ctl *c = M.ctl;
  double *val = w == 0 ? M.u : M.v;
  const double *ten = w == 0 ? M.dudt : M.dvdt;
  const long long x = M.at(k, j, i), base = M.at(k, j, 0);
  const double DT = M.dt;
  if (M.uv_scheme == EPIC_UV_AB3 && M.mixed) {
    // the mixed forms: the Adams-Bashforth sum in double-float on the integer and FP32 pipes
    // (~1e-14 of the increment) added to the binary64 wind -- one FP64 addition a point instead
    // of seven, which had put this kernel at the FP64 unit's rate
    // (a zero coefficient -- the first steps -- drops its term: the planes not yet written hold
    // the DBL_MAX marker, which has no binary32 part)
    const float2 *ab = c->abf[w];
    double *X = val + (long long)c->it_uv * M.n3;
    dfl s = dfl(ab[0].x, ab[0].y) * d2df(ten[(long long)c->it_zero * M.n3 + x]);
    if (ab[1].x != 0.f) s += dfl(ab[1].x, ab[1].y) * d2df(ten[(long long)c->it_minus1 * M.n3 + x]);
    if (ab[2].x != 0.f) s += dfl(ab[2].x, ab[2].y) * d2df(ten[(long long)c->it_minus2 * M.n3 + x]);
    write_with_pads(X, M, base, i, X[x] + df2d(dfl(d2f(M.dt), 0.f) * s));
  } else if (M.uv_scheme == EPIC_UV_AB3) {
    const double *ab = c->ab[w];
    double *X = val + (long long)c->it_uv * M.n3;
    const double v = X[x] + DT * (ab[0] * ten[(long long)c->it_zero * M.n3 + x] + ab[1] * ten[(long long)c->it_minus1 * M.n3 + x] +
                                  ab[2] * ten[(long long)c->it_minus2 * M.n3 + x]);
    write_with_pads(X, M, base, i, v);
  } else {
    double *X0 = val + (long long)c->it_zero * M.n3, *Xm1 = val + (long long)c->it_minus1 * M.n3;
    const double d = ten[(long long)c->it_uv_tend * M.n3 + x];
    if (c->lf_first[w]) {
      write_with_pads(Xm1, M, base, i, X0[x] + DT * d);
    } else {
      const double old_filtered = Xm1[x], present = X0[x];
      const double new_leap = old_filtered + 2. * DT * d;
      write_with_pads(Xm1, M, base, i, new_leap);
      write_with_pads(X0, M, base, i, present * (1. - 2. * 0.06) + 0.06 * (old_filtered + new_leap));
    }
  }
}

__global__ void k_uv_rotate(DevModel M) {
  if (epic_member(M)) return;
  Ctl *c = M.ctl;
  if (M.uv_scheme == EPIC_UV_AB3) {
    const int itmp = c->it_minus2;
    c->it_minus2 = c->it_minus1;
    c->it_minus1 = c->it_zero;
    c->it_zero = itmp;
    c->it_uv_tend = c->it_zero;   // it_uv and it_uv_dis stay 0: one plane (branches of the step read them meanwhile)
  } else {
    const int itmp = c->it_minus1;
    c->it_minus1 = c->it_zero;
    c->it_zero = itmp;
    c->it_uv = c->it_zero;
    c->it_uv_dis = (M.u[(long long)c->it_minus1 * M.n3 + M.at(1, 0, 1)] == DBL_MAX) ? c->it_zero : c->it_minus1;
    c->it_uv_tend = 0;
  }
  c->model_time += (long long)M.dt;
}

// End of a step: grid.itime += 1 (the driver loop, epic_main.c:424); a step that recorded a fatal
// error instead halts the model, as the reference's epic_error() ends the run in that step.
__global__ void k_itime_advance(DevModel M) {
  if (epic_member(M)) return;
  if (M.ctl->err_code != 0) M.ctl->halted = 1;
  else M.ctl->itime += 1;
}

// grid.itime as the caller's driver loop holds it (the drop-in: the driver advances it after each
// timestep() call, epic_main.c:424).  Runs on a halted model too.
__global__ void k_set_itime(DevModel M, long long itime) {
  epic_member(M);
  M.ctl->itime = itime;
}

// ---- launchers ----

int launch_zero_tend(const DevModel &M, cudaStream_t s) {
  k_zero_tend<<<zg(epic_blocks(M.n3, TB(M, TB_POINT)), M), TB(M, TB_POINT), 0, s>>>(M);
  return 0;
}

int launch_row_tables(const DevModel &M, cudaStream_t s) {
  const unsigned blocks = epic_blocks(M.nj + 2, 64);
  k_row_tables<double><<<blocks, 64, 0, s>>>(M, const_cast<double *>(M.rt64));
  k_row_tables<float><<<blocks, 64, 0, s>>>(M, const_cast<float *>(M.rt32));
  k_visc_tables<double><<<epic_blocks(24LL * (M.nj + 2), 128), 128, 0, s>>>(M, const_cast<double *>(M.vt64));
  k_visc_tables<float><<<epic_blocks(24LL * (M.nj + 2), 128), 128, 0, s>>>(M, const_cast<float *>(M.vt32));
  return 0;
}

int launch_uv_core(const DevModel &M, cudaStream_t s) {
  const int th = TB(M, TB_UV_CORE);
  EPIC_MARCH(M.mixed, k_uv_kin, M.nk - 1, M.nj + 1, th, s, M);
  EPIC_MARCH(M.mixed, k_uv_core_v, M.nk - 1, M.nj, th, s, M);
  // k_uv_kin wrote KIN on rows 0..nj with their pads
  launch_filter_planes(M, M.work0, PL_NONE, M.work0, 1, M.nk - 1, 0, s, M.mixed, 0, 1);
  EPIC_MARCH(M.mixed, k_uv_core_u, M.nk - 1, M.nj + 1, th, s, M);
  return 0;
}

int launch_pgrad_poles(const DevModel &M, cudaStream_t s) {
  const int lv = row_sum_levels(M, 2);
  k_gz_pole_rows<<<zg(epic_blocks(M.nk + 1, lv), M), 256, (size_t)2 * lv * (M.ni + 1) * sizeof(double), s>>>(M, lv);
  return 0;
}
// FP64 form: binary64; mixed: double-float on the splits; fast mixed: binary32 on the splits.
// k_pgrad_lon's face exchange wants whole rows in a block (one face per thread in shared memory); the
// FP64 form takes blocks of a row for it up to 512 columns.
int launch_pgrad_lon(const DevModel &M, cudaStream_t s) {
  int th = TB(M, TB_PGRAD);
  if (!M.mixed && M.ni > th && M.ni <= 512) th = M.ni;
  const dim3 grid = zg(cells_blocks(M, M.nk - 1, M.nj + 1, th), M);
  if (!M.mixed) k_pgrad_lon<double><<<grid, th, (size_t)th * sizeof(LonFace<double>), s>>>(M);
  else if (M.col64) k_pgrad_lon<dfl><<<grid, th, (size_t)th * sizeof(LonFace<dfl>), s>>>(M);
  else k_pgrad_lon<float><<<grid, th, 0, s>>>(M);
  return 0;
}
int launch_pgrad_lat(const DevModel &M, cudaStream_t s) {
  const int th = TB(M, TB_PGRAD);
  if (!M.mixed) {
    EPIC_MARCH_R(double, k_pgrad_lat, M.nk - 1, M.nj, th, s, M);
    return 0;
  }
  const dim3 grid = zg(dim3(epic_blocks((long long)(M.nk - 1) * M.ni, th), M.nj), M);
  if (M.col64) k_pgrad_lat<dfl, 1><<<grid, th, 0, s>>>(M);
  else k_pgrad_lat<float, 1><<<grid, th, 0, s>>>(M);
  return 0;
}

int launch_akima_meridional(const DevModel &M, double *buff, int kind, cudaStream_t s) {
  const int k0 = kind == 1 ? M.k_sigma - 1 : 1;
  const int nkk = M.nk - k0 + 1;
  const int th = TB(M, TB_HSU);
  EPIC_LAUNCH_R(M.mixed, k_akima_merid_flux, cells_blocks(M, nkk, M.nj, th), th, 0, s, M, buff, kind, k0);
  EPIC_LAUNCH_R(M.mixed, k_akima_merid_update, cells_blocks(M, nkk, M.nj + 1, th), th, 0, s, M, buff, k0);
  return 0;
}

// The meridional Hsu pass has three forms that give the same bits.  The tile (k_hsu_merid_tile) of 32, 16
// or 8 columns (64 bytes of a row) where its four arrays of nj+2 rows fit MERID_SMEM, as wide as leaves two
// blocks per SM; the march (k_hsu_meridional, one thread per (k, i, member) walking nj+1 rows) once those
// threads fill the GPU (large batches); else the four passes, whose threads cover every cell.  The
// tuning table's TB_HSU_MERID_VARIANT entry overrides the choice (HsuForm; tiles where they fit, else
// the four passes).
constexpr long long HSU_FUSED_MIN_THREADS = 65536;
constexpr size_t MERID_SMEM = 100 * 1024;   // two blocks per SM

// shared memory of one column of a tile: the field, the velocity, the fluxes and the predicted field
static size_t merid_column_bytes(const DevModel &M) { return (size_t)4 * (M.nj + 2) * (M.mixed ? sizeof(float) : sizeof(double)); }
// columns of a tile, 0 where 8 do not fit
static int merid_tile_columns(const DevModel &M, int nkk) {
  int TC = 32;
  while (TC > 8 && (long long)epic_blocks(M.ni, TC) * nkk * (M.nbatch > 1 ? M.nbatch : 1) < 2 * M.sms) TC /= 2;
  while (TC >= 8 && TC * merid_column_bytes(M) > MERID_SMEM) TC /= 2;
  return TC >= 8 ? TC : 0;
}
int hsu_meridional_form(const DevModel &M, int nkk) {
  const int entry = M.tb[TB_HSU_MERID_VARIANT];
  if (entry == HSU_MARCH || (entry == 0 && (long long)M.ni * nkk * (M.nbatch > 1 ? M.nbatch : 1) >= HSU_FUSED_MIN_THREADS)) return HSU_MARCH;
  return entry != HSU_PASSES && merid_tile_columns(M, nkk) ? HSU_TILES : HSU_PASSES;
}

int launch_hsu_meridional(const DevModel &M, double *buff, int kind, cudaStream_t s) {
  const int k0 = kind == 1 ? M.k_sigma - 1 : 1;
  const int nkk = M.nk - k0 + 1;
  const int th = TB(M, TB_HSU), form = hsu_meridional_form(M, nkk);
  if (form == HSU_MARCH) {
    EPIC_LAUNCH_R(M.mixed, k_hsu_meridional, dim3(epic_blocks(M.ni, th), nkk), th, 0, s, M, buff, kind, k0);
    return 0;
  }
  if (form == HSU_TILES) {
    const int TC = merid_tile_columns(M, nkk);
    EPIC_LAUNCH_R(M.mixed, k_hsu_merid_tile, dim3(epic_blocks(M.ni, TC), nkk), 256, TC * merid_column_bytes(M), s, M, buff, kind, k0, TC);
    return 0;
  }
  EPIC_LAUNCH_R(M.mixed, k_hsu_merid_pred, cells_blocks(M, nkk, M.nj + 2, th), th, 0, s, M, buff, kind, k0);
  EPIC_LAUNCH_R(M.mixed, k_hsu_merid_apred, cells_blocks(M, nkk, M.nj + 1, th), th, 0, s, M, buff, k0);
  EPIC_LAUNCH_R(M.mixed, k_hsu_merid_corr, cells_blocks(M, nkk, M.nj + 2, th), th, 0, s, M, buff, kind, k0);
  EPIC_LAUNCH_R(M.mixed, k_hsu_merid_update, cells_blocks(M, nkk, M.nj + 1, th), th, 0, s, M, buff, k0);
  return 0;
}

// index: 0 = U, 1 = V, 2 = HDRY, 3 = THETA
static void visc_krange(const DevModel &M, int index, int &k0, int &k1) {
  k0 = 1;
  k1 = M.nk;
  if (index == 0 || index == 1) k1 = M.nk - 1;
  if (index == 3) k0 = M.k_sigma - 1;
}

// meridional_hyperviscosity up to its last order's second difference, which is left in `last` (with its
// sign) for the zonal kernel to filter and apply
static void launch_meridional_hyperviscosity(const DevModel &M, int index, double *var, int sel, cudaStream_t s, double *&last, double &last_sign) {
  int k0, k1;
  visc_krange(M, index, k0, k1);
  const int nkk = k1 - k0 + 1;
  const int vgrid = index == 1;
  const int nrows = vgrid ? M.nj + 2 : M.nj + 1;
  // The first second-derivative reads the (possibly time-plane selected) field itself; later
  // ones ping-pong between two scratch volumes, as hh and d2dy2var do in the reference.
  double *cur_src = var;
  int src_sel = sel;
  double *bufs[2] = {M.work1, M.work2};
  int which = 0;
  double sign = 1.;
  // the first two passes in one kernel when nothing is applied between them
  const size_t pair_col = (size_t)nrows * (M.mixed ? sizeof(float) : sizeof(double));
  const long long strips = (long long)epic_blocks(M.ni, 16) * nkk * (M.nbatch > 1 ? M.nbatch : 1);
  const int pair_tc = 16 * pair_col <= 48 * 1024 && strips >= 2 * M.sms ? 16 : 8;
  const bool pair = !(M.nu[2] > 0.) && M.nu[4] + M.nu[6] + M.nu[8] > 0. && pair_tc * pair_col <= 48 * 1024;
  for (int itmp = 2; itmp <= 8; itmp += 2) {
    double *dst = bufs[which];
    if (pair && itmp == 2) {
      // the second pass's output goes where the unfused loop leaves it
      dst = bufs[1];
      EPIC_LAUNCH_R(M.mixed, k_d2dy2_pair, dim3(epic_blocks(M.ni, pair_tc), (unsigned)nkk), 256, pair_tc * pair_col, s, M, var, sel, dst,
                    vgrid, k0, pair_tc);
      itmp = 4;
      which = 1;
      sign = -sign;
    } else {
      EPIC_LAUNCH_R(M.mixed, k_d2dy2, cells_blocks(M, nkk, nrows, TB(M, TB_VISC)), TB(M, TB_VISC), 0, s, M, cur_src, src_sel, dst, vgrid, itmp, k0,
                    nkk, cur_src == var);
    }
    src_sel = PL_NONE;
    double rest = 0.;
    for (int q = itmp + 2; q <= 8; q += 2) rest += M.nu[q];
    if (!(rest > 0.)) {   // the last order, which is always applied
      last = dst;
      last_sign = sign;
      return;
    }
    if (M.nu[itmp] > 0.) {
      // k_d2dy2 / k_d2dy2_pair wrote every row of dst with its pads
      launch_filter_planes(M, dst, PL_NONE, dst, k0, nkk, vgrid, s, M.mixed, 0, 1);
      EPIC_LAUNCH_R(M.mixed, k_visc_apply, cells_blocks(M, nkk, vgrid ? M.nj : M.nj + 1, TB(M, TB_VISC)), TB(M, TB_VISC), 0, s, M, var, sel, dst, vgrid, sign, k0, nkk);
    }
    sign = -sign;
    cur_src = dst;
    which ^= 1;
  }
}

constexpr size_t VISC_ROWS_SMEM = 101 * 1024;   // two blocks per SM; 4 rows of EPIC_MAX_NI fit

// index 2 (HDRY) applies restore_mass as well (in the kernel, or alone without hyperviscosity)
int launch_hyperviscosity(const DevModel &M, int index, double *var, int sel, cudaStream_t s) {
  if (!(M.nu[4] + M.nu[6] + M.nu[8] > 0.)) return index == 2 ? launch_restore_mass(M, s) : 0;
  int k0, k1;
  visc_krange(M, index, k0, k1);
  double *D = nullptr, msign = 1.;
  launch_meridional_hyperviscosity(M, index, var, sel, s, D, msign);
  // the tensor cores filter whole planes; else the zonal kernel filters each row itself
  const int filter = !(M.mixed && filter_gemm_usable(M));
  if (!filter) launch_filter_planes(M, D, PL_NONE, D, k0, k1 - k0 + 1, index == 1, s, 1, 0, 1);
  const int jbot = index == 1 ? 1 : 0, jhalf = index == 1 ? 0 : 1;
  const int nrows = M.nj - jbot + 1, nkk = k1 - k0 + 1;
  if (!M.mixed) {
    // rows per block: a power of 2, the fewest that leave two blocks per SM or fewer (each order's
    // sums are one chain of ni additions per block), up to a warp's lanes and VISC_ROWS_SMEM
    const size_t row_bytes = (size_t)3 * (M.ni + 2) * sizeof(double);
    const long long total = (long long)nrows * nkk * (M.nbatch > 1 ? M.nbatch : 1);
    int rows = 4;
    while (rows < 32 && total > 2LL * M.sms * rows && 2 * rows * row_bytes <= VISC_ROWS_SMEM) rows *= 2;
    k_zonal_visc_rows<<<zg(epic_blocks((long long)nrows * nkk, rows), M), 256, rows * row_bytes, s>>>(M, var, sel, D, msign, filter, jbot,
                                                                                                     jhalf, k0, nkk, index == 2, rows);
    return 0;
  }
  const size_t row_bytes = (size_t)(M.ni + 2) * (sizeof(double) + 2 * sizeof(float));
  int rows = (int)((40 * 1024) / row_bytes);
  rows = rows < 1 ? 1 : (rows > 4 ? 4 : rows);
  dim3 grid((nrows + rows - 1) / rows, nkk);
  k_zonal_visc_mixed<<<zg(grid, M), 32 * rows, rows * row_bytes, s>>>(M, var, sel, D, msign, filter, jbot, jhalf, k0, index == 2);
  return 0;
}

// the largest dynamic shared memory of a launch, raised once for the process (models of all sizes)
int stencil_kernels_init() {
  if (cudaFuncSetAttribute(k_zonal_visc_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VISC_ROWS_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(k_hsu_merid_tile<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MERID_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(k_hsu_merid_tile<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MERID_SMEM) != cudaSuccess)
    return -1;
  return 0;
}

int launch_divergence_damping(const DevModel &M, cudaStream_t s) {
  if (M.nudiv == 0.) return 0;
  launch_filter_rest(M, M.u, PL_UV_DIS, M.work1, 1, M.nk - 1, 0, s, M.mixed);
  launch_filter_planes(M, M.u, PL_UV_DIS, M.work1, 1, M.nk - 1, 0, s, M.mixed, 0, 1);
  EPIC_MARCH(M.mixed, k_divergence, M.nk - 1, M.nj + 1, TB(M, TB_DIAG), s, M, M.work1, M.v, PL_UV_DIS, M.work2, 1, M.nk - 1);
  EPIC_LAUNCH_R(M.mixed, k_divdamp_apply, epic_blocks(2LL * (M.nk - 1) * (M.nj + 1) * M.ni, TB(M, TB_UPDATE)), TB(M, TB_UPDATE), 0, s, M);
  return 0;
}

int launch_uv_decide(const DevModel &M, cudaStream_t s) {
  k_uv_decide<<<zg(1, M), 1, 0, s>>>(M);
  return 0;
}
int launch_uv_update(const DevModel &M, cudaStream_t s) {
  k_uv_update<<<zg(epic_blocks(2LL * (M.nk - 1) * (M.nj + 1) * M.ni, TB(M, TB_UPDATE)), M), TB(M, TB_UPDATE), 0, s>>>(M);
  return 0;
}
int launch_uv_rotate(const DevModel &M, cudaStream_t s) {
  k_uv_rotate<<<zg(1, M), 1, 0, s>>>(M);
  return 0;
}

int launch_diag_filter_v(const DevModel &M, cudaStream_t s, cudaStream_t rest) {
  launch_filter_rest(M, M.v, PL_UV, M.work1, 0, M.nk + 1, 1, rest, M.mixed);
  return launch_filter_planes(M, M.v, PL_UV, M.work1, 0, M.nk + 1, 1, s, M.mixed, 0, 1);
}
int launch_diag_filter_u(const DevModel &M, cudaStream_t s, cudaStream_t rest) {
  launch_filter_rest(M, M.u, PL_UV, M.work2, 0, M.nk + 1, 0, rest, M.mixed);
  return launch_filter_planes(M, M.u, PL_UV, M.work2, 0, M.nk + 1, 0, s, M.mixed, 0, 1);
}
int launch_diag_pv(const DevModel &M, cudaStream_t s) {
  EPIC_MARCH(M.mixed, k_pv_interior, M.nk + 1, M.nj, TB(M, TB_DIAG), s, M, M.work1);
  return 0;
}
int launch_diag_pv_poles(const DevModel &M, cudaStream_t s) {
  const int lv = row_sum_levels(M, 4);
  k_pv_poles<<<zg(epic_blocks(M.nk + 1, lv), M), 256, (size_t)4 * lv * (M.ni + 1) * sizeof(double), s>>>(M, lv);
  return 0;
}
int launch_diag_div(const DevModel &M, cudaStream_t s) {
  EPIC_MARCH(M.mixed, k_divergence, M.nk + 1, M.nj + 1, TB(M, TB_DIAG), s, M, M.work2, M.v, PL_UV, M.div_uv3, 0, M.nk + 1);
  return 0;
}
int launch_diag_ri2(const DevModel &M, cudaStream_t s) {
  EPIC_LAUNCH_R(M.mixed, k_ri2, cells_blocks(M, M.nk, M.nj + 1, TB(M, TB_DIAG)), TB(M, TB_DIAG), 0, s, M);
  return 0;
}

int launch_itime_advance(const DevModel &M, cudaStream_t s) {
  k_itime_advance<<<zg(1, M), 1, 0, s>>>(M);
  return 0;
}

int launch_set_itime(const DevModel &M, long long itime, cudaStream_t s) {
  k_set_itime<<<zg(1, M), 1, 0, s>>>(M, itime);
  return 0;
}

}  // namespace epic

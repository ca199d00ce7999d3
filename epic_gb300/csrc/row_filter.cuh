// The zonal filter of one latitude row by a group of lanes of a warp (see k_filter.cu for the method and
// the reference's routines), shared by the kernels that work on whole rows.
#pragma once
#include "device_common.cuh"

namespace epic {

template <class R> struct __align__(2 * sizeof(R)) Cplx { R re, im; };

// Twiddle table layout (pairs), N = ni/2 complex points:
//   [0, N-1)              four1 isign=+1, stage with half h at offset h-1, entries p = 0..h-1
//   [N-1, 2N-2)           four1 isign=-1, same layout
//   [2N-2, 2N-2 + N/2-1)  realft forward post-processing, q = 1..N/2-1
//   [.., + N/2-1)         realft inverse pre-processing, q = 1..N/2-1
// The FP64 table holds the recurrence values of the reference; the mixed form reads the same
// values rounded to float.
__host__ __device__ inline size_t nr_twiddle_pairs(int ni) {
  const int N = ni / 2;
  return 2 * (size_t)(N - 1) + 2 * (size_t)(N / 2 - 1);
}

// ---- rows by lane groups ----
//
// A row belongs to G lanes of one warp (RowShape): 32, or fewer where a row has fewer butterflies, so
// that a warp instruction is full either way -- a binary64 one costs the pipe the same 19 clocks
// whatever the number of active lanes.  A block takes `rows` levels of one latitude row, so its rows
// are all filtered or all not and share what depends on the latitude; a row's passes are separated by
// __syncwarp alone.  With a block of two warps a row, its passes separated by block barriers and the
// twiddles copied to shared memory by each, the FP64 form's filters ran at 43-66% of the binary64 pipe
// with 3 warps resident per scheduler.
struct RowShape { int G, rows, stride; };   // lanes a row, rows a block, compute-type values a row in shared memory
struct RowLane {
  int gl, G, r, k;
  bool live;   // the row exists (the last block of a launch may have rows to spare)
};
__device__ __forceinline__ RowLane row_lane(const RowShape &S, int k0, int kend) {
  RowLane L;
  L.G = S.G;
  L.gl = (int)threadIdx.x & (S.G - 1);
  L.r = (int)threadIdx.x / S.G;
  const int k = k0 + (int)blockIdx.y * S.rows + L.r;
  L.live = k <= kend;
  L.k = L.live ? k : kend;
  return L;
}

template <class R> __device__ __forceinline__ const Cplx<R> *twiddle_table(const DevModel &M);
template <> __device__ __forceinline__ const Cplx<double> *twiddle_table<double>(const DevModel &M) { return reinterpret_cast<const Cplx<double> *>(M.tw); }
template <> __device__ __forceinline__ const Cplx<float> *twiddle_table<float>(const DevModel &M) { return reinterpret_cast<const Cplx<float> *>(M.twf); }

// The twiddles and a row's weights (if any) into L1, a cache line per lane of each warp, ahead of the
// stages that read them: each stage waits for its twiddles between two __syncwarp, an L2 round trip a
// stage for the first rows of an SM otherwise.  Plain loads whose values nobody waits for.
__device__ __forceinline__ void touch(const char *p, int bytes) {
  for (int b = 128 * ((int)threadIdx.x & 31); b < bytes; b += 128 * 32) {
    unsigned v;
    asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(p + b));
  }
}
template <class R>
__device__ __forceinline__ void warm_filter(const DevModel &M, const double *hl) {
  touch(reinterpret_cast<const char *>(twiddle_table<R>(M)), (int)(nr_twiddle_pairs(M.ni) * sizeof(Cplx<R>)));
  if (hl) touch(reinterpret_cast<const char *>(hl), (M.ni / 2 + 2) * 8);
}

// The place of row value e = i-1 among the N complex points in bit-reversed order, which
// filter_row takes its input in.
__device__ __forceinline__ int fft_place(int e, int lg) { return 2 * (int)(__brev((unsigned)(e >> 1)) >> (32 - lg)) + (e & 1); }
__device__ __forceinline__ int fft_log(int ni) { return 31 - __clz(ni / 2); }

// four1's Danielson-Lanczos stages on z (already bit-reversed); tw = this direction's table.  The
// first stage's only twiddle is (1, 0).
template <class R>
__device__ __forceinline__ void four1_stages(Cplx<R> *z, const Cplx<R> *tw, int N, const RowLane &L) {
  for (int b = L.gl; b < N / 2; b += L.G) {
    const Cplx<R> u = z[2 * b], v = z[2 * b + 1];
    z[2 * b] = {u.re + v.re, u.im + v.im};
    z[2 * b + 1] = {u.re - v.re, u.im - v.im};
  }
  __syncwarp();
  for (int h = 2; h < N; h <<= 1) {
    const Cplx<R> *wt = tw + (h - 1);
    for (int b = L.gl; b < N / 2; b += L.G) {
      const int p = b & (h - 1), i0 = 2 * (b - p) + p, j0 = i0 + h;
      const Cplx<R> w = wt[p], u = z[i0], v = z[j0];
      const R tempr = w.re * v.re - w.im * v.im;
      const R tempi = w.re * v.im + w.im * v.re;
      z[j0] = {u.re - tempr, u.im - tempi};
      z[i0] = {u.re + tempr, u.im + tempi};
    }
    __syncwarp();
  }
}

// Filter a row with weights h(I) = hl[I], I = 1..ni/2+1 (HIGH_LAT(J,I)): z holds the row's values in
// bit-reversed order (fft_place), on return the filtered row in order, to be multiplied by
// filter_scale.  Every lane of the warp must call this.  realft forward, the weights and realft
// inverse (epic_adjust.c:412-456) meet in one pass between the two four1 calls: both split loops and
// the weights act on the pair (q, N-q).  The reference's factors 1/2 (c1, c2, two per value) and 2/ni
// are powers of 2, which commute with every rounding in between (the values being far from the ends
// of the range), so they are left to the one final multiplication.
template <class R> __device__ __forceinline__ R filter_scale(int ni) { return cv<R>(.5 * inv_pow2(ni)); }
template <class R>
__device__ __forceinline__ void filter_row(const DevModel &M, Cplx<R> *z, const double *hl, const RowLane &L) {
  const int N = M.ni / 2, lg = fft_log(M.ni);
  const Cplx<R> *t4p = twiddle_table<R>(M), *t4m = t4p + (N - 1), *trp = t4p + 2 * (N - 1), *trm = trp + (N / 2 - 1);
  four1_stages(z, t4p, N, L);
  for (int q = L.gl; q < N / 2; q += L.G) {
    if (q == 0) {   // wavenumbers 0 and ni/2 share z[0]; ni/4 has no partner
      const Cplx<R> a = z[0], b = z[N / 2];
      const R s = (a.re + a.im) * cv<R>(hl[1]), d = (a.re - a.im) * cv<R>(hl[N + 1]);
      z[0] = {twice_of(s + d), twice_of(s - d)};
      const R h = R(4.) * cv<R>(hl[N / 2 + 1]);
      if (N > 1) z[N / 2] = {b.re * h, b.im * h};
      continue;
    }
    Cplx<R> a = z[q], b = z[N - q], w = trp[q - 1];
    R x = a.re + b.re, y = a.im - b.im, s = a.im + b.im, d = a.re - b.re;
    R ws = w.re * s, id = w.im * d, wd = w.re * d, is = w.im * s;
    const R hq = cv<R>(hl[q + 1]), hn = cv<R>(hl[N - q + 1]);
    a = {(x + ws + id) * hq, (y - wd + is) * hq};
    b = {(x - ws - id) * hn, (-y - wd + is) * hn};
    w = trm[q - 1];
    x = a.re + b.re; y = a.im - b.im; s = a.im + b.im; d = a.re - b.re;
    ws = w.re * s; id = w.im * d; wd = w.re * d; is = w.im * s;
    z[q] = {x - ws - id, y + wd - is};
    z[N - q] = {x + ws + id, -y + wd - is};
  }
  __syncwarp();
  for (int k = L.gl; k < N; k += L.G) {
    const int r = (int)(__brev((unsigned)k) >> (32 - lg));
    if (r > k) {
      const Cplx<R> t = z[k];
      z[k] = z[r];
      z[r] = t;
    }
  }
  __syncwarp();
  four1_stages(z, t4m, N, L);
}

__device__ __forceinline__ bool row_is_filtered(const DevModel &M, int j, int vgrid) {
  if (!M.filt_bands) return fabs(M.lat[vgrid ? 2 * j : 2 * j + 1]) >= M.lat0;
  return vgrid ? j <= M.filt_south_v || j >= M.filt_north_v : j <= M.filt_south_h || j >= M.filt_north_h;
}

// The place of row value e = i-1 for filter_row, or in order for a row that is not filtered.
__device__ __forceinline__ int row_place(bool filt, int e, int lg) { return filt ? fft_place(e, lg) : e; }

}  // namespace epic

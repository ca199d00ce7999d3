// The zonal filter of whole planes (zonal_filter TWODIM, src/shared/epic_adjust.c:412-456) as a
// dense filter-operator product on the fifth-generation tensor cores, for the mixed form
// (ni a multiple of 128).
//
// The reference filters one latitude row at a time: realft forward, wavenumber q scaled by
// HIGH_LAT(J,q+1), realft inverse, times 2/ni.  That is a circulant, symmetric operator:
// y(i) = sum_i' f_J((i - i') mod ni) x(i'), with
//     f_J(d) = (w_0 + (-1)^d w_{ni/2} + 2 sum_{q=1}^{ni/2-1} w_q cos(2 pi q d / ni)) / ni,
// w_q = HIGH_LAT(J, q+1).  For row J of every plane at once this is the product
//     D[m][n] = sum_k A[m][k] B[n][k],   A[m][k] = f_J((m0 + m - k) mod ni),  B[n][k] = x_n(k+1),
// in tiles of M = 128 output points, N columns and K = ni.  The columns are (member, plane) pairs:
// one CTA filters row J of up to 64 planes of several members of a batch at once (members that
// share the grid, so the operator), which is what amortises the operator's staging.  A CTA
// accumulates every 128-point tile of the row in its own tensor-memory columns, so it reads the
// whole input row before it writes any output (the filter may run in place).  Operands are staged
// in shared memory in the 128-byte-swizzled K-major layout (8-row atoms of 1024 bytes; the
// 16-byte chunk c of row r sits at chunk c ^ (r % 8)), multiplied by tcgen05.mma kind::tf32 issued
// by one thread into a 128 x N FP32 accumulator in tensor memory, and read back with tcgen05.ld.
// Three products per K step give FP32 accuracy from TF32 inputs ("3xTF32"): with a = a_hi + a_lo,
// a_hi = tf32(a), the sum a_hi b_hi + a_hi b_lo + a_lo b_hi misses only the a_lo b_lo term.
//
// The operator is circulant, so the 128 x 32 tile of output tile mt and K chunk kc depends on
// (128 mt - kc) mod ni alone: ni/32 distinct tiles per row.  They are built once per model on
// the host, already split into TF32 hi and lo parts, and kept in HBM for the filtered rows only
// (ni/32 x 32 KB per row); the TMA engine copies each step's pair into shared memory
// (cp.async.bulk.tensor with the 128-byte swizzle, completion counted on an mbarrier) while the
// threads convert and stage the planes' values.  At ni = 128 a row's four tiles stay in shared memory
// and a CTA takes several groups of columns in turn.
//
// What bounds it: latency on a single model (a few dozen CTAs, each a chain of load, convert, multiply,
// store), the staging and the plane traffic on a large batch, the products' shared-memory reads (5 KB
// each) on a long row.  So eight warps stage and store, one issues the products and one brings the
// operator tiles, all through mbarriers (no block barrier in the pipeline), with every tile of a short
// row and four chunks of plane values on their way at once.  With one thread for the tiles and the
// products, 950 cycles of tile requests came between every 760 of products; an epilogue that reads its
// row length and pointers again after each store takes twice as long.  A launch on 512x256 x 40 planes
// 105 -> 63 us, on 64 members of 128x64 x 20 planes 75 -> 55 us, on one such model 12.3 -> 11.3 us.
//
// With shift set, each row of each plane is filtered as x - x(1), and x(1) is added back to the
// output in binary64: the operator passes a constant unchanged (its wavenumber-0 weight is 1), so
// the result is the same while the FP32 rounding acts on the zonal variations only -- for the
// geopotential, ~1e-5 of its value.
//
// Every wait is bounded: a CTA whose operator copy or MMA completion does not arrive within the
// limit waits (bounded) for what it has in flight, records ERR_TIMEOUT in every member whose rows it
// leaves unwritten, frees its tensor memory and returns.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>
#include <cuda.h>
#include <cudaTypedefs.h>
#include "device_common.cuh"
#include "filter_pipeline.h"
#include "kernels.h"
#include "epic_common.h"
#include "epic_gb300.h"

namespace epic {

namespace {

constexpr int FG_M = 128;        // output points per tile (tensor-memory lanes)
constexpr int FG_KC = 32;        // K elements per staged chunk: one 128-byte swizzle row of FP32
constexpr int FG_NMAX = 64;      // columns per CTA ((member, plane) pairs), a multiple of 32
constexpr int FG_STAGE = 256;    // eight staging and epilogue warps: two per 32-lane quarter of tensor memory
constexpr int FG_WARPS = FG_STAGE / 32;
constexpr int FG_THREADS = FG_STAGE + 64;   // warp FG_WARPS issues the products, the next one the operator copies
constexpr int FG_GROUPS = 8;     // column groups a CTA takes in turn at most
#ifndef EPIC_FILTER_WAIT_LIMIT
#define EPIC_FILTER_WAIT_LIMIT (1u << 20)
#endif
constexpr unsigned FG_WAIT_LIMIT = EPIC_FILTER_WAIT_LIMIT;   // of the pipeline's waits (a test builds with 0)
constexpr unsigned FG_DRAIN_LIMIT = 1u << 20;                 // of the waits for what a CTA that gives up has in flight
constexpr unsigned FG_A_BYTES = FG_M * FG_KC * 4;   // one operator tile (hi or lo): 16 KB

// Byte offset of element (r, e), 0 <= e < 32, in a 128B-swizzled K-major tile of FP32 rows.
__device__ __forceinline__ unsigned sw128(int r, int e) {
  return (unsigned)((r >> 3) * 1024 + (r & 7) * 128 + ((((e >> 2) ^ (r & 7)) & 7) << 4) + (e & 3) * 4);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading-dimension byte offset
// (unused for swizzled K-major operands; 16 bytes), stride-dimension byte offset 1024 (between
// 8-row atoms), descriptor version 1, layout SWIZZLE_128B.
__device__ __forceinline__ uint64_t smem_desc(unsigned saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)(16 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Instruction descriptor for kind::tf32: D FP32, A and B TF32, both K-major, M = 128, N columns
// (a multiple of 16 up to 256).
__device__ __forceinline__ uint32_t idesc_tf32(int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(FG_M >> 4) << 24);
}

__device__ __forceinline__ float tf32_hi(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}

__device__ __forceinline__ void mma_tf32(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
}

// One operator tile (128 rows of 32 FP32) from the tensor map's row y into shared memory at
// dst (1024-byte aligned), counted on mbarrier mbar.  x is 0: the rows are exactly one 128-byte
// box wide, so the copy starts on the 16-byte boundary TMA requires.
__device__ __forceinline__ void tma_tile(unsigned dst, const void *map, int y, unsigned mbar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(0), "r"(y), "r"(mbar)
      : "memory");
}

// The operator's tensor map lies in global memory, written by a copy: before a block's first use of it, the
// accesses through the tensor-map proxy are ordered after that write.  Without it a map made at the address
// of an operator released earlier might be read as the old one, whose tiles have been freed.
__device__ __forceinline__ void acquire_tensor_map(const void *map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
}

// Bounded; gives up at once when another wait of the CTA has.
__device__ __forceinline__ bool mbar_wait(unsigned mbar, unsigned phase, volatile int *fail, unsigned limit = FG_WAIT_LIMIT) {
  for (unsigned it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (done) return true;
    if (*fail) return false;
  }
  *fail = 1;
  return false;
}
__device__ __forceinline__ void mbar_arrive(unsigned mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mma_commit(unsigned mbar) {   // arrives once the products issued so far are done
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

}  // namespace

// blockIdx.x = row j + 1, j in -1..nj+1.  The columns of a launch lie in `units` groups: group u is
// plane chunk u % nch (pc planes) of G members from q0 = (u / nch) G; column n = g pc + p is plane
// k0 + chunk pc + p of member q0 + g, N = G pc rounded up to 32 (idle columns stay zero).
// blockIdx.y / msplit = the first group of a CTA, which takes every gs-th from there; msplit CTAs (a
// cluster) share a row's 128-point output tiles.  Rows outside the filtered set return at once
// (k_filter_rows_unfiltered copies them).  A member the batch has halted keeps its planes
// untouched.  G > 1, and several groups per CTA, only when the members share the launch's geometry and
// operator (fop_shared).
//
// Steps t count (group, K chunk c, output tile) in order.  The issuing thread waits for step t's
// operator tiles and chunk, issues the products and commits them to the buffers they read; the copying
// thread refills a buffer once the products that read it are done; with `resident` (ni = 128, one tile
// per chunk) the
// four buffers are filled once.  The staging threads keep FG_BUFS chunks of their columns' values in
// registers ahead of the one they convert, across groups.  In place, the CTAs of a cluster have all read
// a row before any writes it.
__global__ void __launch_bounds__(FG_THREADS, 1) k_filter_planes_gemm(DevModel M, const double *src, int src_sel, double *dst, int k0,
                                                                      int nplanes, int vgrid, int shift, int pc, int G, int N, int msplit,
                                                                      int units, int gs, int resident) {
  extern __shared__ __align__(16) unsigned char fg_raw[];
  // operator tiles landed / read (per buffer), plane chunk staged / read (per buffer), accumulator
  // complete / read out, every product done (a CTA that gave up)
  __shared__ __align__(8) uint64_t bars[4 * FG_BUFS + 3];
  __shared__ uint32_t tmem_base;
  __shared__ volatile int fail;
  __shared__ int s_written[FG_GROUPS];                  // staging warps that have written their share of a group
  __shared__ const double *s_src[FG_GROUPS][FG_NMAX];   // each column's row (i = 0), null when idle
  __shared__ double *s_dst[FG_GROUPS][FG_NMAX];
  __shared__ double s_x1[FG_GROUPS][FG_NMAX];           // the subtracted value of each column's row (shift), else 0
  const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int j = (int)blockIdx.x - 1;
  const int nch = (nplanes + pc - 1) / pc;
  const int u0 = (int)blockIdx.y / msplit, msi = (int)blockIdx.y - u0 * msplit;
  const int members = M.batch ? M.nbatch : 1;
  // geometry: a one-member CTA takes its member's own (batches of mixed sizes); the members of
  // a larger group share the launch's
  const DevModel &Mg = M.batch ? M.batch[(u0 / nch) * G] : M;
  const DevModel &opm = M.fop_shared ? M : Mg;
  const int ni = Mg.ni, mtiles = ni / FG_M, nchunks = ni / FG_KC, ntiles = ni / FG_KC;
  // this CTA's output tiles (a member narrower than the launch may leave some CTAs without one)
  const int mts = mtiles >= msplit ? mtiles / msplit : 1, mt0 = msi * mts;
  if (mt0 >= mtiles) return;
  if (j > Mg.nj + 1) return;   // a member with fewer rows than the launch
  const int slot = opm.fop_slot[vgrid * (Mg.nj + 3) + j + 1];
  if (slot < 0) return;
  const int ngroups = (units - u0 + gs - 1) / gs;   // of this CTA, at most FG_GROUPS

  // FG_BUFS operator buffers of A_hi, A_lo (128 x 32 FP32 each), then FG_BUFS plane buffers of B_hi,
  // B_lo (N x 32 each); the swizzle atoms need a 1024-byte aligned base
  const unsigned b_bytes = (unsigned)N * FG_KC * 4;
  unsigned char *fg_smem = fg_raw + ((1024u - ((unsigned)__cvta_generic_to_shared(fg_raw) & 1023u)) & 1023u);
  const unsigned a_s = (unsigned)__cvta_generic_to_shared(fg_smem), b_off = FG_BUFS * 2 * FG_A_BYTES;
  const unsigned bars_s = (unsigned)__cvta_generic_to_shared(&bars[0]);
  const unsigned a_full = bars_s, a_free = bars_s + 8 * FG_BUFS, b_full = a_free + 8 * FG_BUFS, b_free = b_full + 8 * FG_BUFS;
  const unsigned acc_full = b_free + 8 * FG_BUFS, acc_free = acc_full + 8, drained = acc_free + 8;
  const uint32_t tcols = (uint32_t)(mts * N) <= 32 ? 32u : 1u << (32 - __clz(mts * N - 1));   // a power of 2 >= 32
  // step t's operator tiles, for offset (128 mt - kc) mod ni, hi then lo
  const void *const fop = opm.fop_map;
  const unsigned fop_y = (unsigned)(slot * ntiles * 2 * FG_M);
  auto load_a = [&](int buf, int c, int mt) {
    const int tt = (((mt0 + mt) * FG_M - c * FG_KC) & (ni - 1)) / FG_KC, y = (int)fop_y + tt * 2 * FG_M;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a_full + 8 * buf), "r"(2 * FG_A_BYTES) : "memory");
    tma_tile(a_s + buf * 2 * FG_A_BYTES, fop, y, a_full + 8 * buf);
    tma_tile(a_s + buf * 2 * FG_A_BYTES + FG_A_BYTES, fop, y + FG_M, a_full + 8 * buf);
  };
  // the copying thread's next load: group lg, chunk lc, output tile lmt; a resident operator is loaded once
  const int steps = ngroups * nchunks * mts, loads = resident ? nchunks : steps;
  int issued = 0, lc = 0, lmt = 0;
  auto load_next = [&]() {
    load_a(issued % FG_BUFS, lc, lmt);
    issued++;
    if (++lmt == mts) {
      lmt = 0;
      if (++lc == nchunks) lc = 0;
    }
  };
  if (tid < FG_GROUPS) s_written[tid] = 0;
  if (tid == FG_STAGE + 32) {
    fail = 0;
    for (int q = 0; q < FG_BUFS; q++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a_full + 8 * q));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a_free + 8 * q));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_full + 8 * q), "r"(FG_WARPS));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_free + 8 * q));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(acc_full));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(acc_free), "r"(FG_WARPS));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(drained));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncwarp();
  if (warp == FG_WARPS) {
    const unsigned dst_s = (unsigned)__cvta_generic_to_shared(&tmem_base);
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_s), "r"(tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  for (int t = tid; t < ngroups * N; t += FG_THREADS) {
    const int gi = t / N, n = t - gi * N, u = u0 + gi * gs;
    const int g = n / pc, plane = (u % nch) * pc + n - g * pc, q = (u / nch) * G + g;
    const double *sp = nullptr;
    double *dp = nullptr;
    if (g < G && q < members && plane < nplanes) {
      const DevModel &mq = M.batch ? M.batch[q] : M;
      if (!mq.ctl->halted) {
        const int row = Mg.at(k0 + plane, j, 0);
        sp = member_ptr(M, mq, src) + plane_offset(mq, src_sel) + row;
        dp = member_ptr(M, mq, dst) + row;
      }
    }
    s_src[gi][n] = sp;
    s_dst[gi][n] = dp;
    s_x1[gi][n] = shift && sp ? sp[1] : 0.;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t dtmem = tmem_base;

  if (warp >= FG_WARPS) {
    if (warp == FG_WARPS && lane == 0) {
      const uint32_t idesc = idesc_tf32(N);
      // every operand lies below 2^18 bytes: a descriptor moves by its address / 16
      const uint64_t a_desc = smem_desc(a_s), b_desc = smem_desc(a_s + b_off);
      const uint64_t b_lo = b_bytes >> 4;
      constexpr uint64_t A_LO = FG_A_BYTES >> 4;
      bool ok = true;
      int t = 0, n = 0;
      for (int gi = 0; gi < ngroups && ok; gi++) {
        if (gi > 0) {   // the accumulator read out
          ok = mbar_wait(acc_free, (unsigned)((gi - 1) & 1), &fail);
          asm volatile("tcgen05.fence::after_thread_sync;");
        }
        for (int c = 0; c < nchunks && ok; c++, n++) {   // chunks in order
          const int bb = n % FG_BUFS;
          const uint64_t b = b_desc + (uint64_t)bb * 2 * b_lo;
          ok = mbar_wait(b_full + 8 * bb, (unsigned)((n / FG_BUFS) & 1), &fail);
          for (int mt = 0; mt < mts && ok; mt++, t++) {
            const int ab = t % FG_BUFS;
            ok = mbar_wait(a_full + 8 * ab, resident ? 0u : (unsigned)((t / FG_BUFS) & 1), &fail);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint64_t a = a_desc + (uint64_t)ab * 2 * A_LO;
            const uint32_t d_mt = dtmem + (uint32_t)(mt * N);
#pragma unroll
            for (int ks = 0; ks < FG_KC / 8; ks++) {   // K = 8 TF32 (32 bytes) per instruction
              mma_tf32(d_mt, a + 2 * ks, b + 2 * ks, idesc, ks > 0 ? 1u : (uint32_t)(c > 0));
              mma_tf32(d_mt, a + 2 * ks, b + b_lo + 2 * ks, idesc, 1u);
              mma_tf32(d_mt, a + A_LO + 2 * ks, b + 2 * ks, idesc, 1u);
            }
            if (fg_signals_operator(t, loads)) mma_commit(a_free + 8 * ab);
          }
          if (ok && fg_signals_chunk(n, ngroups * nchunks)) mma_commit(b_free + 8 * bb);
        }
        if (ok) mma_commit(acc_full);
      }
    } else if (warp > FG_WARPS && lane == 0) {
      acquire_tensor_map(fop);
      while (issued < loads && issued < FG_BUFS) load_next();
      while (issued < loads && mbar_wait(a_free + 8 * (issued % FG_BUFS), (unsigned)((issued / FG_BUFS - 1) & 1), &fail)) load_next();
      // the copies in flight are waited for (bounded by the limit) whether or not their steps are reached,
      // so that nothing writes this CTA's shared memory after it is released
      for (int q = issued > FG_BUFS ? issued - FG_BUFS : 0; q < issued; q++) {
        int none = 0;
        mbar_wait(a_full + 8 * (q % FG_BUFS), (unsigned)((q / FG_BUFS) & 1), &none, FG_DRAIN_LIMIT);
      }
    }
    __syncwarp();
    if (msplit > 1)
      for (int gi = 0; gi < ngroups; gi++) {   // the staging threads' cluster barriers
        asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      }
  } else {
    // B[n][e] = x_n(kc + e + 1) - x1_n, zero in idle columns: thread tid converts 4 neighbouring values of
    // column tid/8 and, for N = 64, of column 32 + tid/8, in every chunk (a column per warp, whole rows of 256
    // bytes a load, is slower: four times the stores and row pointers, 64 members 71 -> 80 us a launch)
    constexpr int BQ = FG_NMAX * FG_KC / 4 / FG_STAGE;   // 2
    const int nq = N * (FG_KC / 4) / FG_STAGE, e0 = 4 * (tid % (FG_KC / 4)), lg_nchunks = 31 - __clz(nchunks);
    const int total = ngroups * nchunks;
    double breg[FG_BUFS][BQ][4];
    auto load_b = [&](int n, double (&bn)[BQ][4]) {
      const int gi = n >> lg_nchunks, kc = (n & (nchunks - 1)) * FG_KC;
#pragma unroll
      for (int u = 0; u < BQ; u++) {
        if (u >= nq) break;
        const int col = tid / (FG_KC / 4) + u * (FG_STAGE / (FG_KC / 4));
        const double *row = s_src[gi][col];
#pragma unroll
        for (int v = 0; v < 4; v++) bn[u][v] = row ? row[kc + e0 + 1 + v] : 0.;
      }
    };
#pragma unroll
    for (int q = 0; q < FG_BUFS; q++)
      if (q < total) load_b(q, breg[q]);
    auto epilogue = [&](int gi) {
      __syncwarp();
      if (msplit > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");   // this CTA has read its row
      const bool done = mbar_wait(acc_full, (unsigned)(gi & 1), &fail);
      asm volatile("tcgen05.fence::after_thread_sync;");
      __syncwarp();
      if (msplit > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      if (__all_sync(0xffffffffu, done)) {
        for (int mt = 0; mt < mts; mt++)
          for (int cg = (warp >> 2) * 16; cg < N; cg += 32) {
            __syncwarp();
            // warp w reads tensor-memory lanes 32 (w % 4)..+31: output point 128 mt + 32 (w % 4) + lane, columns cg..cg+15
            uint32_t r[16];
            const uint32_t taddr = dtmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(mt * N + cg);
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                  "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
            double *row[16];   // read before the stores, which might overlap anything
#pragma unroll
            for (int n = 0; n < 16; n++) row[n] = s_dst[gi][cg + n];
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int i = (mt0 + mt) * FG_M + (warp & 3) * 32 + lane + 1;
            const int pad = i == ni ? 0 : (i == 1 ? ni + 1 : i);   // ni is at least FG_M
#pragma unroll
            for (int n = 0; n < 16; n++) {
              if (!row[n]) continue;
              double y = f2d(__uint_as_float(r[n]));
              if (shift) y += s_x1[gi][cg + n];
              row[n][i] = y;
              if (pad != i) row[n][pad] = y;
            }
          }
        if (lane == 0) atomicAdd(&s_written[gi], 1);
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_free);
    };
    for (int n0 = 0; n0 < total; n0 += FG_BUFS) {
#pragma unroll
      for (int q = 0; q < FG_BUFS; q++) {   // chunk n in buffer q
        const int n = n0 + q;
        if (n >= total) break;
        if (n >= FG_BUFS) mbar_wait(b_free + 8 * q, (unsigned)((n / FG_BUFS - 1) & 1), &fail);
        unsigned char *bh = fg_smem + b_off + q * 2 * b_bytes, *bl = bh + b_bytes;
        const int gi = n >> lg_nchunks;
#pragma unroll
        for (int u = 0; u < BQ; u++) {
          if (u >= nq) break;
          const int col = tid / (FG_KC / 4) + u * (FG_STAGE / (FG_KC / 4));
          const double x1 = s_x1[gi][col];
          float4 b4;
          if (shift)
            b4 = make_float4(d2f(breg[q][u][0] - x1), d2f(breg[q][u][1] - x1), d2f(breg[q][u][2] - x1), d2f(breg[q][u][3] - x1));
          else b4 = make_float4(d2f(breg[q][u][0]), d2f(breg[q][u][1]), d2f(breg[q][u][2]), d2f(breg[q][u][3]));
          const float4 hv = make_float4(tf32_hi(b4.x), tf32_hi(b4.y), tf32_hi(b4.z), tf32_hi(b4.w));
          const unsigned off = sw128(col, e0);
          *reinterpret_cast<float4 *>(bh + off) = hv;
          *reinterpret_cast<float4 *>(bl + off) = make_float4(b4.x - hv.x, b4.y - hv.y, b4.z - hv.z, b4.w - hv.w);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(b_full + 8 * q);
        if (n + FG_BUFS < total) load_b(n + FG_BUFS, breg[q]);
        if (n + 1 == (gi + 1) * nchunks) epilogue(gi);
      }
    }
  }
  // every wait of the other threads is over, and every signal and product was waited for (the last group's
  // products in its epilogue) -- unless a wait gave up: then the issuing thread waits (bounded) for all it
  // has issued, so that nothing arrives in the shared or tensor memory of a CTA that has gone
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (fail) {
    if (tid == FG_STAGE) {
      int none = 0;
      mma_commit(drained);
      mbar_wait(drained, 0u, &none, FG_DRAIN_LIMIT);
    }
    // every member with a row that this CTA has not written, or not whole
    for (int t = tid; t < ngroups * G; t += FG_THREADS) {
      const int gi = t / G, u = u0 + gi * gs, q = (u / nch) * G + t - gi * G;
      if (s_written[gi] < FG_WARPS && q < members) flag_error(M.batch ? M.batch[q].ctl : M.ctl, ERR_TIMEOUT, k0 + (u % nch) * pc, j, 0, 0.);
    }
    __syncthreads();
  }
  if (warp == FG_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(dtmem), "r"(tcols));
}

// dynamic shared memory of a CTA with N columns: operator buffers, plane buffers, the alignment slack of
// the swizzle atoms
size_t filter_gemm_smem_bytes(int n) { return 1024 + (size_t)FG_BUFS * 2 * (FG_A_BYTES + (size_t)n * FG_KC * 4); }

bool filter_gemm_usable(const DevModel &M) { return M.fop_map && M.ni % FG_M == 0 && M.ni <= 8 * FG_M; }

// Columns per CTA: up to 64.  Planes beyond that split into chunks; members of one operator fill the
// rest of the columns.  The accumulators of a CTA's output tiles take mts x N <= 512 tensor-memory columns.
int launch_filter_planes_gemm(const DevModel &M, const double *src, int src_sel, double *dst, int k0, int nplanes, int vgrid, cudaStream_t s,
                              int shift) {
  const int members = M.batch ? M.nbatch : 1;
  const int pc = nplanes < FG_NMAX ? nplanes : FG_NMAX;
  const int nch = (nplanes + pc - 1) / pc;
  int G = M.fop_shared ? FG_NMAX / pc : 1;
  if (G > members) G = members;
  const int N = ((G * pc + 31) / 32) * 32;
  const int units = nch * ((members + G - 1) / G);
  const int sms = M.sms, mtiles = M.ni / FG_M, rows = (M.nj + 3) / 2;   // about half the rows are filtered
  // one CTA per SM (its buffers fill the shared memory).  Few units: a cluster of CTAs shares a row's
  // output tiles (each tile's sums are unchanged) as long as they are all resident at once: a second
  // round pays the setup, the first loads and the staging of the whole row again (512x256 x 40 planes:
  // one round of 129 CTAs 70 us, two of 258 half as long each 87 us, before the epilogue above).
  int msplit = 1;
  while (2 * msplit <= mtiles && (long long)rows * units * msplit * 2 <= sms) msplit *= 2;
  // many units, and the row's operator in the four buffers: a CTA takes several groups
  const int resident = M.ni == FG_KC * FG_BUFS && (M.fop_shared || !M.batch);
  int gs = units;
  if (resident) {
    gs = sms / rows > 1 ? sms / rows : 1;
    if (gs > units) gs = units;
    if ((units + gs - 1) / gs > FG_GROUPS) gs = (units + FG_GROUPS - 1) / FG_GROUPS;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(M.nj + 3), (unsigned)(gs * msplit), 1u);
  cfg.blockDim = dim3(FG_THREADS);
  cfg.dynamicSmemBytes = filter_gemm_smem_bytes(N);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = (unsigned)msplit;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_filter_planes_gemm, M, src, src_sel, dst, k0, nplanes, vgrid, shift, pc, G, N, msplit, units, gs, resident) ==
                 cudaSuccess
             ? 0
             : -1;
}

int filter_gemm_init(int) {
  return cudaFuncSetAttribute(k_filter_planes_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)filter_gemm_smem_bytes(FG_NMAX)) ==
                 cudaSuccess
             ? 0
             : -1;
}

// Host: the circulant kernel f_J(d) of every row (h rows from HIGH_LAT_H, v rows from
// HIGH_LAT_PV), rows indexed J+1 = 0..nj+2, rounded to FP32.
void fill_filter_kernels(int ni, int nj, const double *hl_h, const double *hl_pv, long long iadim, float *fh, float *fv) {
  const int N = ni / 2;
  std::vector<double> cs(ni);
  for (int mq = 0; mq < ni; mq++) cs[mq] = cos(2. * M_PI * mq / ni);
  for (int g = 0; g < 2; g++) {
    const double *hl = g ? hl_pv : hl_h;
    float *out = g ? fv : fh;
    for (int row = 0; row < nj + 3; row++) {
      const double *w = hl + (long long)row * iadim;   // w[I], I = 1..N+1
      for (int d = 0; d < ni; d++) {
        double f = w[1] + ((d & 1) ? -w[N + 1] : w[N + 1]);
        for (int q = 1; q < N; q++) f += 2. * w[q + 1] * cs[(long long)q * d % ni];
        out[(long long)row * ni + d] = (float)(f / ni);
      }
    }
  }
}

namespace {

// cvt.rna.tf32.f32 on the host: round to nearest (ties away from zero) to 10 fraction bits, the
// 13 bits below cleared
float tf32_rna(float x) {
  uint32_t u;
  std::memcpy(&u, &x, 4);
  if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0x1000u) & 0xffffe000u;
  float r;
  std::memcpy(&r, &u, 4);
  return r;
}

// which rows the filter changes: |lat| >= lat0 among the h rows j = 0..nj and the v rows 1..nj
// (row_is_filtered); slot[g (nj+3) + j+1], g = 0 for h rows and 1 for v rows
int filter_slots(const epic_grid &g, std::vector<int> &slot) {
  slot.assign(2 * (size_t)(g.nj + 3), -1);
  int n = 0;
  for (int gr = 0; gr < 2; gr++)
    for (int j = gr ? 1 : 0; j <= g.nj; j++)
      if (std::fabs(g.lat[gr ? 2 * j : 2 * j + 1]) >= g.lat0) slot[(size_t)gr * (g.nj + 3) + j + 1] = n++;
  return n;
}

}  // namespace

bool filter_operator_wanted(const epic_grid &g, int precision) {
  return precision != EPIC_PREC_FP64 && g.ni % FG_M == 0 && g.ni <= 8 * FG_M;
}

// Device bytes of a model's operator allocation: the tiles (ni/32 x 2 x 16 KB per filtered row),
// the slot table and the tensor map, with the alignments TMA wants.
size_t filter_operator_bytes(const epic_grid &g) {
  std::vector<int> slot;
  const int n = filter_slots(g, slot);
  return (size_t)n * (g.ni / FG_KC) * 2 * FG_A_BYTES + 1024 + ((slot.size() * sizeof(int) + 255) / 256) * 256 + 256;
}

// Host: the operator tiles of the filtered rows.  For slot s (row J of the h or v grid), tile t
// (offset 32 t) and part h (0: the TF32 part hi = tf32(f), 1: the rest f - hi), row m and column e
// hold the two parts of f_J((32 t + m - e) mod ni), f_J the row's circulant kernel rounded to FP32
// (fill_filter_kernels); the rows of 32 FP32 are stored one after another, tile (s, t, h) at row
// ((s ni/32 + t) 2 + h) 128.  They are copied into one device allocation with the slot table and
// the TMA tensor map that describes them (2-D: 32 FP32 per row, boxes of 32 x 128 with the
// 128-byte swizzle of the kernel's operand layout).  hash identifies the operator (equal hashes:
// the same tiles): models of one grid on one device share one allocation (released by
// filter_operator_release when its last model goes), and a batch of them filters with member 0's.
namespace {
// Operators are shared between the models of one grid on one device: a process-wide table of the
// allocations, keyed by device and hash, counted by the models that use them.
struct OperatorCopy {
  int device;
  uint64_t hash;
  void *base;
  const void *map;
  const int *slot;
  int users;
};
std::mutex g_op_mu;
std::vector<OperatorCopy> g_ops;
}  // namespace

void filter_operator_release(void *mem) {
  if (!mem) return;
  std::lock_guard<std::mutex> lock(g_op_mu);
  for (size_t q = 0; q < g_ops.size(); q++)
    if (g_ops[q].base == mem) {
      if (--g_ops[q].users == 0) {
        cudaFree(g_ops[q].base);
        g_ops.erase(g_ops.begin() + (long)q);
      }
      return;
    }
}

int filter_operator_create(const epic_grid &g, const double *hl_h, const double *hl_pv, long long iadim, cudaStream_t s, DevModel &d,
                           void **mem, uint64_t *hash, const char **why) {
  *mem = nullptr;
  const int ni = g.ni, ntiles = ni / FG_KC;
  std::vector<int> slot;
  const int nslots = filter_slots(g, slot);
  std::vector<float> fh((size_t)(g.nj + 3) * ni), fv((size_t)(g.nj + 3) * ni);
  fill_filter_kernels(ni, g.nj, hl_h, hl_pv, iadim, fh.data(), fv.data());
  uint64_t hs = 1469598103934665603ull;   // FNV-1a over everything the tiles are made of
  auto mix = [&](const void *p, size_t n) {
    const unsigned char *c = static_cast<const unsigned char *>(p);
    for (size_t q = 0; q < n; q++) hs = (hs ^ c[q]) * 1099511628211ull;
  };
  mix(&ni, sizeof ni);
  mix(slot.data(), slot.size() * sizeof(int));
  mix(fh.data(), fh.size() * sizeof(float));
  mix(fv.data(), fv.size() * sizeof(float));
  *hash = hs;
  int device = -1;
  cudaGetDevice(&device);
  std::lock_guard<std::mutex> lock(g_op_mu);
  for (auto &c : g_ops)
    if (c.device == device && c.hash == hs) {   // a model of the same grid made it already
      c.users++;
      d.fop_map = c.map;
      d.fop_slot = c.slot;
      *mem = c.base;
      return 0;
    }
  const size_t tile_floats = (size_t)FG_M * FG_KC;
  std::vector<float> tiles((size_t)(nslots > 0 ? nslots : 1) * ntiles * 2 * tile_floats, 0.f);
  for (int gr = 0; gr < 2; gr++)
    for (int r = 0; r < g.nj + 3; r++) {
      const int sl = slot[(size_t)gr * (g.nj + 3) + r];
      if (sl < 0) continue;
      const float *f = (gr ? fv.data() : fh.data()) + (size_t)r * ni;
      for (int t = 0; t < ntiles; t++) {
        float *hi = tiles.data() + (((size_t)sl * ntiles + t) * 2) * tile_floats, *lo = hi + tile_floats;
        for (int m = 0; m < FG_M; m++)
          for (int e = 0; e < FG_KC; e++) {
            const float a = f[(FG_KC * t + m - e + 2 * ni) & (ni - 1)], h = tf32_rna(a);
            hi[m * FG_KC + e] = h;
            lo[m * FG_KC + e] = a - h;
          }
      }
    }
  const size_t tile_bytes = tiles.size() * sizeof(float), slot_bytes = ((slot.size() * sizeof(int) + 255) / 256) * 256;
  char *base = nullptr;
  if (cudaMalloc(&base, tile_bytes + 1024 + slot_bytes + 256) != cudaSuccess) {
    *why = "cudaMalloc of the filter operator tiles failed";
    return -1;
  }
  char *tiles_d = base + ((1024 - ((uintptr_t)base & 1023)) & 1023);   // cudaMalloc gives 256-byte alignment
  int *slot_d = reinterpret_cast<int *>(tiles_d + tile_bytes);
  CUtensorMap *map_d = reinterpret_cast<CUtensorMap *>(reinterpret_cast<char *>(slot_d) + slot_bytes);

  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      cudaFree(base);
      *why = "cuTensorMapEncodeTiled not available from the driver";
      return -1;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  CUtensorMap map;
  std::memset(&map, 0, sizeof map);
  const cuuint64_t gdim[2] = {(cuuint64_t)FG_KC, (cuuint64_t)(tiles.size() / FG_KC)};
  const cuuint64_t gstride[1] = {(cuuint64_t)FG_KC * sizeof(float)};
  const cuuint32_t box[2] = {(cuuint32_t)FG_KC, (cuuint32_t)FG_M}, estride[2] = {1, 1};
  if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, tiles_d, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
    cudaFree(base);
    *why = "cuTensorMapEncodeTiled rejected the filter operator's layout";
    return -1;
  }
  cudaError_t e = cudaMemcpyAsync(tiles_d, tiles.data(), tile_bytes, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(slot_d, slot.data(), slot.size() * sizeof(int), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(map_d, &map, sizeof map, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // the host vectors go out of scope
  if (e != cudaSuccess) {
    cudaFree(base);
    *why = "copy of the filter operator failed";
    return -1;
  }
  d.fop_map = map_d;
  d.fop_slot = slot_d;
  *mem = base;
  g_ops.push_back({device, hs, base, map_d, slot_d, 1});
  return 0;
}

}  // namespace epic

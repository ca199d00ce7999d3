// Which steps of the tensor-core filter's pipeline (k_filter_gemm.cu) signal a buffer as read.  Step t
// multiplies the operator tiles in buffer t % BUFS and plane chunk n the values in buffer n % BUFS; the
// signal is asynchronous, so one is sent only where a later load of the buffer waits for it: a signal that
// nobody waits for could arrive when the CTA has gone, in the shared memory of the SM's next one.
#pragma once

#ifdef __CUDACC__
#define EPIC_HD __host__ __device__
#else
#define EPIC_HD
#endif

namespace epic {

constexpr int FG_BUFS = 4;   // operator tile pairs and chunks of plane values in shared memory, each

// loads: operator tile pairs that the CTA brings, one per step, or once per buffer (a resident operator)
EPIC_HD inline bool fg_signals_operator(int t, int loads) { return t + FG_BUFS < loads; }
EPIC_HD inline bool fg_signals_chunk(int n, int chunks) { return n + FG_BUFS < chunks; }

}  // namespace epic

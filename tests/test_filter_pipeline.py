"""The tensor-core filter's buffers (epic_gb300/csrc/filter_pipeline.h): every asynchronous signal that a
buffer has been read is waited for by the load that follows in that buffer, and every such load has its
signal, for the step counts of all row lengths, column groups and clusters."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "epic_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "filter_pipeline.h"
using namespace epic;
// signals of each buffer against the loads that wait for one (every load but a buffer's first)
static int check(int steps, int loads, bool (*signals)(int, int)) {
  int sent[FG_BUFS] = {0}, waited[FG_BUFS] = {0}, bad = 0;
  for (int t = 0; t < steps; t++) sent[t % FG_BUFS] += signals(t, loads);
  for (int l = FG_BUFS; l < loads; l++) waited[l % FG_BUFS]++;
  for (int q = 0; q < FG_BUFS; q++) bad += sent[q] != waited[q];
  return bad;
}
int main() {
  int bad = 0;
  for (int ni = 128; ni <= 1024; ni *= 2)
    for (int groups = 1; groups <= 8; groups++)
      for (int mts = 1; mts <= ni / 128; mts *= 2) {
        const int chunks = groups * (ni / 32), steps = chunks * mts, resident = ni == 32 * FG_BUFS;
        bad += check(steps, steps, fg_signals_operator) + check(chunks, chunks, fg_signals_chunk);
        if (resident) bad += check(steps, ni / 32, fg_signals_operator);   // the operator is loaded once
      }
  printf("%d\n", bad);
  return bad != 0;
}
"""


def test_every_signal_is_waited_for(tmp_path):
    src, exe = tmp_path / "pipeline.cpp", str(tmp_path / "pipeline")
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    kernel = open(os.path.join(CSRC, "k_filter_gemm.cu")).read()
    # the kernel's signals to the buffers are sent under these conditions alone
    for bar, rule in (("a_free", "fg_signals_operator("), ("b_free", "fg_signals_chunk(")):
        sent = [line for line in kernel.splitlines() if f"mma_commit({bar}" in line]
        assert sent and all(rule in line for line in sent), sent

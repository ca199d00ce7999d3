"""A wait of the tensor-core filter that runs out: the kernel returns, and every member whose rows were
not written reports it (not only the first of the thread block's members).  The library is linked with the
filter built for a wait limit of 0, so that no wait succeeds."""
import os
import shutil
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..")

PROGRAM = """
import sys
import epic_gb300
from epic_gb300 import Batch, EPIC_PREC_MIXED, EpicError, HSConfig, Model, hs_setup
epic_gb300.load_library(sys.argv[1])
for members in (1, 14):
    models = []
    for q in range(members):
        ga, f = hs_setup(HSConfig(ni=128, nj=16, nk=5, dt=60, seed=q))
        m = Model(ga, EPIC_PREC_MIXED)
        m.upload(f)
        models.append(m)
    b = Batch(models)
    b.run(1)
    silent = []
    for q, m in enumerate(models):
        try:
            m.sync()
            silent.append(q)
        except EpicError as e:
            assert "not signalled in time" in str(e), e
    assert not silent, silent
    b.close()
"""


def test_every_member_reports(gpu, tmp_path):
    from epic_gb300 import build
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    obj, so = str(tmp_path / "k_filter_gemm.o"), str(tmp_path / "libepic_limit.so")
    subprocess.run([nvcc, *build._flags(), "-DEPIC_FILTER_WAIT_LIMIT=0u", "-c", os.path.join(build.SRC, "k_filter_gemm.cu"), "-o", obj], check=True)
    others = [os.path.join(build.OUT, os.path.basename(s) + ".o") for s in build.SOURCES if s != "k_filter_gemm.cu"]
    subprocess.run([nvcc, build.ARCH, "-shared", "-cudart", "static", "-o", so, obj, *others], check=True)
    r = subprocess.run([sys.executable, "-c", PROGRAM, so], cwd=ROOT, env=dict(os.environ, PYTHONPATH=ROOT), capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr

"""Copies that a launch on another stream could overtake: the library's streams are non-blocking, so what
a kernel reads is on the device before the call that made it returns (host code over a stand-in for the
CUDA runtime; no GPU is needed)."""
import pytest

from epic_gb300 import Batch, EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, hs_setup
from host_library import host_library, host_library_file  # noqa: F401


@pytest.mark.parametrize("form,shapes", [(EPIC_PREC_FP64, [(16, 8), (16, 8), (32, 16)]), (EPIC_PREC_MIXED, [(128, 8), (128, 8)])])
def test_batch_descriptions_arrive_before_launches(host_library, form, shapes):
    models = []
    for q, (ni, nj) in enumerate(shapes):
        ga, f = hs_setup(HSConfig(ni=ni, nj=nj, nk=4, dt=60, seed=q))
        m = Model(ga, form)
        m.upload(f)
        m.timestep(EPIC_SYNC_DIAGS_ONLY)
        models.append(m)
    b = Batch(models)
    assert host_library.fake_unordered_writes(b.stream) == 0
    b.run(2)
    assert host_library.fake_unordered_writes(b.stream) == 0
    b.close()
    for m in models:
        m.close()

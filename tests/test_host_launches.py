"""What the library launches, by its host code over a stand-in for the CUDA runtime (no GPU is needed)."""
import pytest

from epic_gb300 import EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, TUNE_GROUPS, hs_setup
from host_library import host_library, host_library_file, launches  # noqa: F401

ROW_KERNELS = ("k_varz_filter_rows", "k_hsu_zonal", "k_filter_planes")


def _model(ni, nj, nk, form=EPIC_PREC_FP64, **kw):
    ga, f = hs_setup(HSConfig(ni=ni, nj=nj, nk=nk, dt=60, **kw))
    m = Model(ga, form)
    m.upload(f)
    return m


@pytest.mark.parametrize("threads", [48, 96, 250, 16, 1])
@pytest.mark.parametrize("ni,form", [(16, EPIC_PREC_FP64), (64, EPIC_PREC_MIXED), (512, EPIC_PREC_FP64)])
def test_row_kernels_take_whole_warps(host_library, ni, form, threads):
    """A row belongs to lanes of one warp and a block's shared memory holds the rows of its warps: a tuning
    table's entry that is no multiple of 32 (or that halves to one) must not leave lanes without a row."""
    m = _model(ni, 8, 4, form)
    m.set_tuning([0] * 8 + [threads] + [0] * (TUNE_GROUPS - 9))
    host_library.fake_reset_counts()
    m.timestep(EPIC_SYNC_DIAGS_ONLY)
    m.timestep()
    for k in ROW_KERNELS:
        n, _, th, _, _ = launches(host_library, k)
        assert n and th >= 32 and th % 32 == 0, (k, n, th)
    m.close()

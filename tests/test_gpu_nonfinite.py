"""Advection of a field with an infinity or a NaN in it, in the FP64 form: what a bad cell reaches is what it
reaches in the restatement (the reference multiplies the downwind side's terms by a zero velocity, which
keeps a NaN a NaN), bit for bit in every finite cell."""
import numpy as np
import pytest

from epic_gb300 import EPIC_PROFILE_N2, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, TUNE_HSU_MERID_VARIANT, hs_setup
from oracle_lib import Port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
# rows in and out of the zonal filter, the pole rows, the first, middle and last levels
@pytest.mark.parametrize("field,k,j", [("theta", 9, 8), ("theta", 10, 1), ("hdry", 1, 8), ("hdry", 6, 9), ("hdry", 10, 0), ("u", 6, 8), ("v", 6, 8),
                                       ("w3", 6, 7)])
@pytest.mark.parametrize("form", [1, 2, 3])
def test_advection(gpu, field, k, j, value, form):
    ga, f = hs_setup(HSConfig(ni=32, nj=16, nk=10, dt=300, seed=3, state="jet", profile=EPIC_PROFILE_N2))
    port = Port(ga, cr_libm=True)
    port.upload(f)
    port.timestep(EPIC_SYNC_DIAGS_ONLY)
    port.run(3)
    f = port.download()
    f.arrays[field][..., k, j + 1, 12] = value
    port.upload(f)
    port.stage(6)
    want = port.download()
    m = Model(ga)
    m.set_tuning([0] * TUNE_HSU_MERID_VARIANT + [form])
    m.upload(f)
    m.run_stage(6)
    got = m.download()
    for n in ("hdry", "theta", "p3"):
        a, b = got.arrays[n], want.arrays[n]
        assert np.array_equal(a, b, equal_nan=True), (n, int((~((a == b) | (np.isnan(a) & np.isnan(b)))).sum()), int(np.isnan(b).sum()))

"""The turbulence closure's column solves and wavefronts at the ends of their range: the most and the
fewest levels, a last tile with columns to spare, more (level, row) pairs than a cluster has threads, the
stability factor on and off; every stage equals the correctly rounded restatement bit for bit."""
import pytest

from epic_gb300 import EPIC_PROFILE_N2, HSConfig
from test_gpu_parity import _stage_by_stage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,nk", [(8, 9, 5), (16, 13, 64), (16, 67, 40), (64, 9, 11)])
@pytest.mark.parametrize("stab", [0, 1])
def test_turbulence_columns(gpu, ni, nj, nk, stab):
    _stage_by_stage(HSConfig(ni=ni, nj=nj, nk=nk, dt=20, seed=nk, state="jet", profile=EPIC_PROFILE_N2, turbulence=True,
                             stability_factor=stab, nu4=0.5 * min(1., 2. * nj / ni)**4))

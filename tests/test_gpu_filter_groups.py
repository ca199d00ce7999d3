"""The tensor-core filter gives the same bits however a launch divides its work: a single model (a
cluster of CTAs shares each row's output tiles) and a member of a batch (several column groups per
CTA, or whole rows per CTA), for one to eight 128-point output tiles per row and for more planes than a
CTA has columns."""
import numpy as np
import pytest

from epic_gb300 import Batch, EPIC_PREC_MIXED, EPIC_PROFILE_N2, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, hs_setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,nk,members", [(128, 64, 20, 14), (256, 12, 70, 3), (512, 20, 7, 30), (1024, 24, 5, 20)])
def test_members_equal_single_models(gpu, ni, nj, nk, members):
    grids = [hs_setup(HSConfig(ni=ni, nj=nj, nk=nk, dt=max(1, 600 // ni), seed=q, state="jet", profile=EPIC_PROFILE_N2,
                               nu4=0.5 * min(1., 2. * nj / ni)**4)) for q in range(members)]
    models = [Model(ga, EPIC_PREC_MIXED) for ga, _ in grids]
    b = Batch(models)
    b.upload([f for _, f in grids])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(2)
    b.sync()
    for q in (0, members - 1):
        single = Model(grids[q][0], EPIC_PREC_MIXED)
        single.upload(grids[q][1])
        single.timestep(EPIC_SYNC_DIAGS_ONLY)
        single.run(2)
        want, got = single.download(), models[q].download()
        for n in want.arrays:
            assert np.array_equal(want.arrays[n], got.arrays[n]), f"member {q}: {n}"

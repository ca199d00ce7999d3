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


def test_operators_made_where_others_were_released(gpu):
    """Operators of different grids made and released in turn: 128x64 and 256x64 have the same number of
    filtered rows, so that one's tensor map may come to lie where the other's was.  Every pass gives the
    first one's bits."""
    grids = [hs_setup(HSConfig(ni=ni, nj=64, nk=5, dt=60, seed=ni, nu4=0.03)) for ni in (128, 256)]
    want = {}
    for turn in range(5):
        for q, (ga, f) in enumerate(grids):
            m = Model(ga, EPIC_PREC_MIXED)
            m.upload(f)
            m.timestep(EPIC_SYNC_DIAGS_ONLY)
            m.run(2)
            got = m.download()
            m.close()   # the last model of the grid: its operator goes
            w = want.setdefault(q, got)
            for n in w.arrays:
                assert np.array_equal(w.arrays[n], got.arrays[n]), (turn, q, n)

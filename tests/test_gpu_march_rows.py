"""Kernels whose launch shape follows the amount of work give the same bits in every shape: a single
model (one row a thread, 512-thread column tiles, filter operators shared by a cluster) against a member
of a batch large enough for two or four rows a thread and 256-thread tiles, with row counts that leave
every remainder."""
import numpy as np
import pytest

from epic_gb300 import Batch, EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, hs_setup

pytestmark = pytest.mark.gpu
SMS = 152


@pytest.mark.parametrize("form", [EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST])
@pytest.mark.parametrize("ni,nj,members,rows", [(64, 31, 3, 1), (64, 30, 9, 2), (64, 33, 8, 2), (64, 32, 16, 4), (64, 34, 14, 4), (256, 9, 12, 4)])
def test_batch_member_equals_single_model(gpu, form, ni, nj, members, rows):
    nk = 11
    cells = ni * nk * (nj + 1) * members
    assert rows == (4 if cells >= 4 * SMS * 512 else 2 if cells >= 2 * SMS * 512 else 1)
    # hyperviscosity stable at the shorter of the two spacings (the oracle stops on 256 x 9 with the default)
    a = 2. * nj / ni
    nu = dict(nu4=0.5 * a**4) if a < 0.9 else dict()
    grids = [hs_setup(HSConfig(ni=ni, nj=nj, nk=nk, dt=60, seed=q, **nu)) for q in range(members)]
    models = [Model(ga, form) for ga, _ in grids]
    b = Batch(models)
    b.upload([f for _, f in grids])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(2)
    b.sync()
    for q in (0, members - 1):
        alone = Model(grids[q][0], form)
        alone.upload(grids[q][1])
        alone.timestep(EPIC_SYNC_DIAGS_ONLY)
        alone.run(2)
        x, y = models[q].download(), alone.download()
        for n in x.arrays:
            assert np.array_equal(x.arrays[n], y.arrays[n]), f"member {q}: {n} differs"

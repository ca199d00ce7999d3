"""A captured step runs as concurrent branches (Model.run, Batch.run); a step enqueued directly runs
its kernels one after another (Model.timestep).  Both give the same bits for every array, in every
form, time and advection scheme, with the optional physics, and in a batch of mixed sizes."""
import ctypes as C

import numpy as np
import pytest

from epic_gb300 import (Batch, EPIC_ADV_AKIMA, EPIC_ADV_HSU, EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST, EPIC_PROFILE_N2,
                        EPIC_SYNC_DIAGS_ONLY, EPIC_UV_AB3, EPIC_UV_LEAPFROG, HSConfig, Model, TUNE_HSU_MERID_VARIANT, hs_setup)

pytestmark = pytest.mark.gpu
JET = dict(state="jet", profile=EPIC_PROFILE_N2)


def _serial(ga, f, form, steps):
    m = Model(ga, form)
    m.upload(f)
    m.timestep(EPIC_SYNC_DIAGS_ONLY)
    for q in range(steps):
        m.timestep()
        assert m.lib.epic_model_set_itime(m._h, C.c_int64(f.struct.itime + q + 1)) == 0
    return m.download()


def _same(a, b, what):
    for n in a.arrays:
        assert np.array_equal(a.arrays[n], b.arrays[n]), f"{what}: {n} differs"


@pytest.mark.parametrize("form", [EPIC_PREC_FP64, EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST])
@pytest.mark.parametrize("shape", [(16, 9, 5), (64, 31, 13), (128, 64, 20)])
@pytest.mark.parametrize("extra", [dict(), dict(uv_scheme=EPIC_UV_LEAPFROG, advection_scheme=EPIC_ADV_AKIMA, nudiv=0.5),
                                   dict(gas_giant=True, x_h2=0.864, x_he=0.136, nu6=0.2, **JET), dict(turbulence=True, **JET)])
def test_branches_equal_the_serial_step(gpu, form, shape, extra):
    if extra.get("turbulence") and form != EPIC_PREC_FP64:
        pytest.skip("the turbulence closure is in the FP64 form only")
    cfg = HSConfig(ni=shape[0], nj=shape[1], nk=shape[2], dt=60, seed=5, **extra)
    ga, f = hs_setup(cfg)
    want = _serial(ga, f, form, 4)
    m = Model(ga, form)
    m.upload(f)
    m.timestep(EPIC_SYNC_DIAGS_ONLY)
    m.run(4)
    _same(m.download(), want, "run")


@pytest.mark.parametrize("form", [EPIC_PREC_FP64, EPIC_PREC_MIXED])
@pytest.mark.parametrize("turbulence", [False, True])
def test_branches_in_a_mixed_size_batch(gpu, form, turbulence):
    if turbulence and form != EPIC_PREC_FP64:
        pytest.skip("the turbulence closure is in the FP64 form only")
    grids = [hs_setup(HSConfig(ni=ni, nj=nj, nk=11, dt=60, seed=q, turbulence=turbulence, **JET))
             for q, (ni, nj) in enumerate([(32, 17), (64, 32), (32, 40)])]
    want = [_serial(ga, f, form, 3) for ga, f in grids]
    models = [Model(ga, form) for ga, _ in grids]
    b = Batch(models)
    b.upload([f for _, f in grids])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(3)
    b.sync()
    for m, w in zip(models, want):
        _same(m.download(), w, "batch")


# the meridional pass as four launches, whose scratch UNITY, HDRY and THETA take one after another
@pytest.mark.parametrize("form,extra", [(EPIC_PREC_FP64, dict()), (EPIC_PREC_MIXED, dict()), (EPIC_PREC_FP64, dict(turbulence=True, **JET))])
@pytest.mark.parametrize("sizes", [[(64, 31)], [(32, 17), (64, 32), (32, 40)]])
def test_branches_with_four_meridional_passes(gpu, form, extra, sizes):
    grids = [hs_setup(HSConfig(ni=ni, nj=nj, nk=13, dt=60, seed=q, **extra)) for q, (ni, nj) in enumerate(sizes)]
    want = [_serial(ga, f, form, 3) for ga, f in grids]
    models = [Model(ga, form) for ga, _ in grids]
    b = Batch(models)
    b.set_tuning([0] * TUNE_HSU_MERID_VARIANT + [2])
    b.upload([f for _, f in grids])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(3)
    b.sync()
    for m, w in zip(models, want):
        _same(m.download(), w, "four passes")

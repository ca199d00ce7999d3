"""Kernels that work on whole latitude rows (the zonal filter, the 3-D filter, the zonal advection pass,
zonal hyperviscosity, the polar row sums), the column kernels beside them and the meridional passes, in
the FP64 form at the ends of their range of row lengths: every stage equals the correctly rounded
restatement bit for bit."""
import ctypes as C

import numpy as np
import pytest

from epic_gb300 import (Batch, EPIC_ADV_AKIMA, EPIC_ADV_HSU, EPIC_PROFILE_N2, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, TUNE_HSU_MERID_VARIANT,
                        hs_setup)
from oracle_lib import Port
from test_gpu_parity import STEP_STAGES, _spin_up, _stage_by_stage

pytestmark = pytest.mark.gpu


# the shortest and longest rows, levels that do and do not fill the
# last block, more rows than a block sums at once (at ni = 1024 the C library rounds one of the filter's weights,
# made on the host, otherwise than the correctly rounded functions)
@pytest.mark.parametrize("ni,nj,nk", [(4, 7, 5), (8, 9, 6), (16, 40, 9), (32, 12, 17), (64, 33, 21), (128, 9, 8), (256, 12, 5), (512, 8, 5)])
@pytest.mark.parametrize("adv", [EPIC_ADV_HSU, EPIC_ADV_AKIMA])
def test_rows(gpu, ni, nj, nk, adv):
    a = min(1., 2. * nj / ni)   # hyperviscosity stable at the shorter of the two spacings
    _stage_by_stage(HSConfig(ni=ni, nj=nj, nk=nk, dt=max(1, 600 // ni), seed=ni + nk, advection_scheme=adv, nu4=0.5 * a**4,
                             nu6=0.05 * a**6, nu8=0.02 * a**8, state="jet", profile=EPIC_PROFILE_N2, turbulence=ni == 32))


# the meridional Hsu pass's forms (tiles of 32, 16 and 8 columns, the march, the four passes) on the last
# and first number of rows of each
@pytest.mark.parametrize("form,nj", [(0, 98), (0, 99), (0, 198), (0, 199), (0, 399), (1, 198), (1, 199), (1, 799)])
def test_meridional_forms(gpu, form, nj):
    ga, f = hs_setup(HSConfig(ni=16, nj=nj, nk=4, dt=5, seed=nj, state="jet", profile=EPIC_PROFILE_N2))
    got = []
    for variant in (0, 1, 2):
        m = Model(ga, form)
        m.set_tuning([0] * TUNE_HSU_MERID_VARIANT + [variant])
        m.upload(f)
        m.timestep(EPIC_SYNC_DIAGS_ONLY)
        m.run(2)
        got.append(m.download())
    for n in ("hdry", "theta", "p3", "u"):
        for g in got[1:]:
            assert np.array_equal(got[0].arrays[n], g.arrays[n]), n


# block sizes of the row kernels that are no multiple of a warp, or halve to one where a row's values fill
# a block's share of shared memory
@pytest.mark.parametrize("form,ni", [(0, 512), (0, 16), (1, 64)])
def test_row_block_sizes(gpu, form, ni):
    ga, f = hs_setup(HSConfig(ni=ni, nj=8, nk=5, dt=max(1, 600 // ni), seed=ni, nu4=0.5 * min(1., 16. / ni)**4))
    got = []
    for threads in (0, 1, 48, 96, 250):
        m = Model(ga, form)
        m.set_tuning([0] * 8 + [threads])
        m.upload(f)
        m.timestep(EPIC_SYNC_DIAGS_ONLY)
        m.run(2)
        got.append(m.download())
    for n in got[0].arrays:
        for g in got[1:]:
            assert np.array_equal(got[0].arrays[n], g.arrays[n]), n


# the meridional pass's tiles asked for by the tuning table (where they do not fit, the four passes), as a
# single model and as an autotuned batch
@pytest.mark.parametrize("form,ni,nj", [(0, 16, 30), (1, 64, 30), (0, 16, 400), (1, 16, 800)])
def test_meridional_tiles_by_table(gpu, form, ni, nj):
    ga, f = hs_setup(HSConfig(ni=ni, nj=nj, nk=4, dt=5, seed=nj, state="jet", profile=EPIC_PROFILE_N2))
    got = []
    for variant in (0, 3, 2):
        m = Model(ga, form)
        m.set_tuning([0] * TUNE_HSU_MERID_VARIANT + [variant])
        m.upload(f)
        m.timestep(EPIC_SYNC_DIAGS_ONLY)
        m.run(2)
        got.append(m.download())
    models = [Model(ga, form) for _ in range(2)]
    b = Batch(models)
    b.upload([f, f])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    assert b.autotune(trial_steps=1)[TUNE_HSU_MERID_VARIANT] in (1, 2, 3)
    b.upload([f, f])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(2)
    got.append(b.download([f.copy(), f.copy()])[1])
    for n in got[0].arrays:
        for g in got[1:]:
            assert np.array_equal(got[0].arrays[n], g.arrays[n]), n


# The longest rows (one row a block, no shared faces in the longitude gradient).  One filter weight, made on
# the host, is rounded otherwise by the C library than in the restatement: 2^-52 of one wavenumber's amplitude, so
# stages that filter agree to 1e-12 of a field's largest value (a few thousand such roundings) and the others in
# every bit; members of a batch and the captured step agree with the single model and the serial step in
# every bit.
@pytest.mark.parametrize("adv", [EPIC_ADV_HSU, EPIC_ADV_AKIMA])
def test_longest_rows(gpu, adv):
    a = 2. * 9 / 1024
    kw = dict(ni=1024, nj=9, nk=6, dt=1, advection_scheme=adv, nu4=0.5 * a**4, nu6=0.05 * a**6, nu8=0.02 * a**8, state="jet", profile=EPIC_PROFILE_N2)
    cfg = HSConfig(seed=2, **kw)
    ga, f = _spin_up(cfg, 4)
    port, model = Port(ga, cr_libm=True), Model(ga)
    port.upload(f)
    model.upload(f)
    for st in STEP_STAGES:
        port.stage(st)
        model.run_stage(st)
        got, want = model.download(), port.download()
        for n in want.arrays:
            x, y = got.arrays[n], want.arrays[n]
            if st in (0, 1, 2, 4, 7, 11, 12, 14, 17):   # no zonal filter in them
                assert np.array_equal(x, y), (st, n)
            else:
                ok = np.abs(y) < 1e300   # the time planes not written yet hold the largest double
                assert np.array_equal(x[~ok], y[~ok]) and np.abs(x[ok] - y[ok]).max() <= 1e-12 * np.abs(y[ok]).max(), (st, n)
        model.upload(want)
    grids = [(ga, f)] + [hs_setup(HSConfig(seed=q, **kw)) for q in (5, 6)]
    models = [Model(g) for g, _ in grids]
    b = Batch(models)
    b.upload([h for _, h in grids])
    b.timestep(EPIC_SYNC_DIAGS_ONLY)
    b.run(2)
    b.sync()
    for m, (g, h) in zip(models, grids):
        captured, serial = Model(g), Model(g)
        for one in (captured, serial):
            one.upload(h)
            one.timestep(EPIC_SYNC_DIAGS_ONLY)
        captured.run(2)
        for q in range(2):
            serial.timestep()
            assert serial.lib.epic_model_set_itime(serial._h, C.c_int64(h.struct.itime + q + 1)) == 0
        x, y, z = m.download(), captured.download(), serial.download()
        for n in x.arrays:
            assert np.array_equal(x.arrays[n], y.arrays[n]) and np.array_equal(x.arrays[n], z.arrays[n]), n

"""The serving loop (epic_gb300/serving.py): runs of different shapes admitted by an HBM budget
and advanced in per-shape-class batches give each run the bits it gets alone."""
import numpy as np
import pytest

from epic_gb300 import EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST, EPIC_PROFILE_N2, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, hs_setup, model_bytes
from epic_gb300.serving import RunRequest, RunServer, latency_summary

pytestmark = pytest.mark.gpu


def _requests():
    shapes = [(32, 16, 10), (64, 32, 10), (32, 16, 10), (64, 32, 20), (32, 16, 10), (64, 32, 10)]
    steps = [9, 20, 33, 12, 17, 5]
    return [RunRequest(q, HSConfig(ni=a, nj=b, nk=c, dt=300, seed=50 + q), steps[q], arrival=0.002 * q,
                       kf_scale=1.0 + 0.03 * (q - 2)) for q, (a, b, c) in enumerate(shapes)]


def test_serving_results_equal_alone(gpu):
    reqs = _requests()
    # a budget that holds about three of these runs at a time, so admission has to wait
    need = [model_bytes(hs_setup(r.cfg)[0], EPIC_PREC_MIXED) for r in reqs]
    budget = sum(sorted(need)[-3:])
    mix = RunServer(hbm_budget=budget, precision=EPIC_PREC_MIXED, round_steps=4, keep_fields=True).serve(reqs)
    assert [r.rid for r in mix] == list(range(len(reqs)))
    for r, q in zip(mix, reqs):
        alone = RunServer(hbm_budget=budget, precision=EPIC_PREC_MIXED, round_steps=64, keep_fields=True).serve(
            [RunRequest(q.rid, q.cfg, q.steps, 0.0, q.kf_scale)])[0]
        for k in r.fields.arrays:
            assert np.array_equal(r.fields.arrays[k], alone.fields.arrays[k]), (q.rid, k)
        assert r.fields.struct.itime == q.steps
    s = latency_summary(mix)
    assert s["p99_s"] >= s["p50_s"] > 0 and s["aggregate_cell_steps_per_s"] > 0


def test_serving_rejects_oversized_request(gpu):
    q = RunRequest(0, HSConfig(ni=64, nj=32, nk=10, dt=300), 3)
    with pytest.raises(ValueError, match="budget"):
        RunServer(hbm_budget=1 << 20).serve([q])


# sizes whose filters run on the tensor cores, in clusters and with shared operators, beside small grids;
# jets beside resting columns in one launch class
STREAM = [((256, 128, 10), 60, True), ((128, 64, 10), 240, False), ((256, 128, 10), 60, True), ((64, 32, 32), 300, False),
          ((256, 128, 10), 120, False), ((128, 64, 20), 60, True), ((512, 256, 10), 60, True), ((256, 128, 10), 60, True),
          ((64, 32, 10), 60, True), ((128, 64, 32), 90, False), ((512, 256, 10), 60, False), ((128, 64, 10), 60, True),
          ((64, 32, 10), 60, True), ((128, 64, 20), 120, False), ((256, 128, 10), 120, False), ((128, 64, 32), 60, True)]


@pytest.mark.parametrize("form", [EPIC_PREC_MIXED, EPIC_PREC_MIXED_FAST])
def test_serving_stream_of_tensor_core_sizes(gpu, form):
    """Runs join and leave classes whose batches are re-formed while other classes' are in flight, twice
    over (so that operators, pools and batch descriptions are released and made again): every result
    equals the run alone."""
    rng = np.random.default_rng(11)
    reqs = []
    for q, ((ni, nj, nk), dt, jet) in enumerate(STREAM):
        kw = dict(state="jet", profile=EPIC_PROFILE_N2) if jet else {}
        reqs.append(RunRequest(q, HSConfig(ni=ni, nj=nj, nk=nk, dt=dt, seed=300 + q, **kw), int(rng.integers(12, 49)), 0.01 * q,
                               1.0 + 0.02 * (q % 5 - 2)))
    alone = []
    for r in reqs:
        ga, f = hs_setup(r.cfg)
        ga.struct.hs_kf *= r.kf_scale
        m = Model(ga, form)
        m.upload(f)
        m.timestep(EPIC_SYNC_DIAGS_ONLY)
        m.run(r.steps)
        m.sync()
        alone.append(m.download())
        m.close()
    for _ in range(2):
        got = RunServer(hbm_budget=40 << 30, precision=form, round_steps=4, keep_fields=True).serve(reqs)
        for r, w in zip(got, alone):
            assert r.error is None, (r.rid, r.error)
            for k in w.arrays:
                assert np.array_equal(r.fields.arrays[k], w.arrays[k]), (r.rid, r.shape, k)

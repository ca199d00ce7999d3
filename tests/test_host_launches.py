"""What the library launches, by its host code over a stand-in for the CUDA runtime (no GPU is needed)."""
import pytest

from epic_gb300 import Batch, EPIC_PREC_FP64, EPIC_UV_LEAPFROG, EPIC_PREC_MIXED, EPIC_SYNC_DIAGS_ONLY, HSConfig, Model, TUNE_GROUPS, TUNE_HSU_MERID_VARIANT, hs_setup, model_bytes
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


@pytest.mark.parametrize("sms,rows", [(152, 1), (76, 2), (38, 4)])
def test_launch_rules_follow_the_device(host_library, sms, rows):
    """As many rows a thread as leave 512 threads per SM of the model's own device: 90112 cells."""
    host_library.fake_device(1, sms, 1)
    host_library.cudaSetDevice(1)
    m = _model(64, 63, 23)
    host_library.fake_reset_counts()
    m.timestep()
    assert launches(host_library, "k_uv_kin")[4] == -(-64 // rows)
    m.close()
    host_library.cudaSetDevice(0)


@pytest.mark.parametrize("ni,nj,form,members", [(64, 32, EPIC_PREC_MIXED, 2), (32, 16, EPIC_PREC_FP64, 8)])
def test_autotuner_times_the_replayed_step(host_library, ni, nj, form, members):
    """The tuner's trial steps are replays of the captured step, as Batch.run's are, and every form of the
    meridional pass is among its candidates: the stand-in's clock counts kernels, of which the tiles take
    one a field where the march or the passes are no fewer."""
    models = [_model(ni, nj, 5, form, seed=q) for q in range(members)]
    b = Batch(models)
    host_library.fake_reset_counts()
    table = b.autotune(trial_steps=2)
    assert host_library.fake_direct_launches() == 0
    assert host_library.fake_graph_launches() >= 3 * (9 * 4 + 3)   # a warm-up and two timed steps per candidate
    assert table[TUNE_HSU_MERID_VARIANT] == 3 and table[:8] == [128] * 8
    host_library.fake_reset_counts()
    b.run(1)
    assert launches(host_library, "k_hsu_merid_tile")[0] == 3 and launches(host_library, "k_hsu_merid_pred")[0] == 0
    b.close()


@pytest.mark.parametrize("clusters", [1, 0])
def test_wavefront_cluster_on_every_device(host_library, clusters):
    """The wavefront kernel's cluster of 16 blocks needs an attribute that belongs to a device: a model of
    the closure on the second device of a process launches it as one on the first does, and a device that
    cannot place 16 takes 8 beside one that can."""
    host_library.fake_device(1, 152, clusters)
    for device, want in ((0, 16), (1, 16 if clusters else 8), (0, 16), (1, 16 if clusters else 8)):
        assert host_library.cudaSetDevice(device) == 0
        m = _model(16, 8, 4, turbulence=True)
        host_library.fake_reset_counts()
        m.timestep()
        n, cluster, _, gx, _ = launches(host_library, "k_sa_waves")
        assert (n, cluster, gx) == (1, want, want)
        m.close()
    host_library.cudaSetDevice(0)


@pytest.mark.parametrize("kw,volumes", [(dict(), 28 + 8), (dict(uv_scheme=EPIC_UV_LEAPFROG), 26 + 8), (dict(turbulence=True), 28 + 8 + 4)])
@pytest.mark.parametrize("shape", [(64, 32, 20), (256, 128, 32)])
def test_device_bytes_of_a_model(cuda_lib, shape, kw, volumes):
    """A model takes its state, eight scratch volumes (gz, unity, old, work0..3, lp3; whatever the branches of
    a step) and tables of less than a volume: what a serving budget was reckoned with."""
    ni, nj, nk = shape
    volume = 8 * (ni + 2) * (nj + 3) * (nk + 2)
    got = model_bytes(hs_setup(HSConfig(ni=ni, nj=nj, nk=nk, dt=60, **kw))[0], EPIC_PREC_FP64)
    assert volumes * volume < got < (volumes + 1) * volume


@pytest.mark.parametrize("streams", [0, 1, 2])
def test_step_is_captured_without_side_streams(host_library, streams):
    """Where the branches' streams cannot be made the step is still captured, on its one stream."""
    m = _model(16, 8, 4)
    host_library.fake_streams_left(streams)
    host_library.fake_reset_counts()
    m.run(3)
    assert host_library.fake_graph_launches() == 3 and host_library.fake_direct_launches() == 0
    m.close()

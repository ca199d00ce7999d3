"""Performance cases: the runs a user of epic_gb300 makes, from one drop-in step to an ensemble.

A case is one grid (or a batch of grids) with its precision form, schemes and physics, and what is
done with it in one pass:

    forecast   upload an initial state, synchronise its diagnostics, advance `steps` steps, download
               the state: the driver's run between two saves (Model) or an ensemble's (Batch)
    diagnose   upload a state, synchronise its diagnostics, download them (SYNC_DIAGS_ONLY)
    step_host  end-to-end steps on a state that lives in host memory: the reference-side timestep()
               wrapper (Model.step_host), or the pipelined ensemble step that moves the prognostic
               arrays (Batch.step_host); the state advances from pass to pass

Host arrays are pinned.  A single run's outputs are its winds, most recent wind tendencies and every
other state array; an ensemble's are its arrays with all members' values at once.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from epic_gb300 import (Batch, EPIC_ADV_AKIMA, EPIC_ADV_HSU, EPIC_IO_STATE, EPIC_PREC_FP64, EPIC_PREC_MIXED,
                        EPIC_PREC_MIXED_FAST, EPIC_PROFILE_HS_EQ, EPIC_PROFILE_N2, EPIC_SYNC_DIAGS_ONLY, EPIC_UV_AB3,
                        EPIC_UV_LEAPFROG, Fields, HSConfig, Model, TURB_FIELDS, hs_setup)
from epic_gb300.abi import FIELD_NAMES_3D

FORMS = {"fp64": EPIC_PREC_FP64, "mixed": EPIC_PREC_MIXED, "fast": EPIC_PREC_MIXED_FAST}

# the state is the Held-Suarez column at rest ("hs"), the balanced zonal jets ("jet"), the jets over
# the gas-giant lower boundary ("jetgg") and that with hydrogen-helium thermodynamics ("jetggh2")
_DEFAULTS = dict(do="forecast", form="fp64", ni=128, nj=64, nk=20, dt=300, steps=1, members=1, state="hs", leapfrog=False,
                 akima=False, damping=False, turbulence=False, mixed_sizes=False)


def _case(name=None, **kw):
    c = dict(_DEFAULTS)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one call of the reference-side timestep() wrapper on the smallest production grid: latency
        _case("dropin_step_fp64_64x32x10", do="step_host", ni=64, nj=32, nk=10, dt=100),
        # an hour of the drop-in form on the everyday grid
        _case("hour_fp64_128x64x20", steps=12),
        # zonal jets at the finer resolution, between two saves
        _case("jets_fp64_256x128x32", ni=256, nj=128, nk=32, dt=60, steps=3, state="jet"),
        # the gas-giant path, rows and layers that divide by nothing
        _case("gasgiant_h2_fp64_128x91x27", ni=128, nj=91, nk=27, dt=60, steps=4, state="jetggh2"),
        # the turbulence closure on the jets
        _case("turbulence_fp64_128x64x20", steps=4, state="jet", turbulence=True),
        # the other time and advection schemes with divergence damping, odd sizes
        _case("leapfrog_akima_fp64_64x47x13", ni=64, nj=47, nk=13, dt=120, steps=8, leapfrog=True, akima=True, damping=True),
        # an hour of one grid in the mixed form
        _case("hour_mixed_128x64x20", form="mixed", steps=12),
        # the largest single grid
        _case("large_mixed_512x256x40", form="mixed", ni=512, nj=256, nk=40, dt=60, steps=4),
        # the headline ensemble: 64 members in one batch
        _case("ensemble64_mixed_128x64x20", form="mixed", steps=6, members=64),
        # an ensemble whose state lives on the host, stepped through the pipelined call
        _case("host_ensemble16_mixed_128x64x20", do="step_host", form="mixed", dt=60, steps=4, members=16),
        # what a serving loop batches: runs of one launch class and different sizes, fast form
        _case("serving_batch_fast_64x32x20", form="fast", ni=64, nj=32, nk=20, dt=120, steps=8, members=8, mixed_sizes=True),
        # diagnostics of a given state (a restart, or fields wanted without a step)
        _case("diagnose_mixed_256x128x32", do="diagnose", form="mixed", ni=256, nj=128, nk=32, dt=60, state="jet"),
    ]


# rough cell-steps/s a form reaches once the GPU is full: keeps drawn cases below the largest listed one
_RATE = {"fp64": 6.0e7, "mixed": 7.0e8, "fast": 8.0e8}
_MOST_S = 0.05


def draw(rng):
    while True:
        form = rng.choice(("fp64", "fp64", "mixed", "mixed", "fast"))
        ni = rng.choice((16, 32, 64, 64, 128, 128, 256, 512))
        nj = max(6, int(round(ni * 2.0 ** rng.uniform(-1.3, -0.6))))
        nk = int(round(5 * 2.0 ** rng.uniform(0.0, 3.0)))
        members = 1 if rng.random() < 0.6 else int(round(2.0 ** rng.uniform(1.0, 6.0)))
        turbulence = form == "fp64" and rng.random() < 0.2
        state = rng.choice(("hs", "hs", "jet", "jetgg", "jetggh2"))
        do = rng.choice(("forecast", "forecast", "forecast", "diagnose")) if members == 1 else "forecast"
        steps = 1 if do == "diagnose" else int(round(2.0 ** rng.uniform(0.0, 4.0)))
        cells = ni * nj * nk * members
        if cells > 64 * 128 * 64 * 20 or cells * (steps + 1) / _RATE[form] * (2.5 if turbulence else 1.0) > _MOST_S:
            continue
        return _case(do=do, form=form, ni=ni, nj=nj, nk=nk, dt=min(300, 9600 // max(ni, 2 * nj)), steps=steps, members=members,
                     state=state, leapfrog=rng.random() < 0.25, akima=rng.random() < 0.25, damping=rng.random() < 0.25,
                     turbulence=turbulence, mixed_sizes=members > 1 and rng.random() < 0.3)


def _sizes(case):
    """(ni, nj) of each member; with mixed sizes they alternate between the case's grid, one of half
    the rows (odd) and one of half the resolution (of the same zonal-filter path)."""
    ni, nj, n = case["ni"], case["nj"], case["members"]
    if not case["mixed_sizes"]:
        return [(ni, nj)] * n
    half = ni // 2 if ni // 2 >= 16 and (ni % 128 != 0) == (ni // 2 % 128 != 0) else ni
    return [((ni, nj), (ni, max(5, nj // 2 | 1)), (half, max(5, nj // 2)))[q % 3] for q in range(n)]


def _config(case, ni, nj, seed):
    jet = case["state"] != "hs"
    h2 = dict(x_h2=0.864, x_he=0.136) if case["state"].endswith("h2") else {}
    return HSConfig(ni=ni, nj=nj, nk=case["nk"], dt=case["dt"], seed=seed,
                    uv_scheme=EPIC_UV_LEAPFROG if case["leapfrog"] else EPIC_UV_AB3,
                    advection_scheme=EPIC_ADV_AKIMA if case["akima"] else EPIC_ADV_HSU, nudiv=0.5 if case["damping"] else 0.0,
                    profile=EPIC_PROFILE_N2 if jet else EPIC_PROFILE_HS_EQ, state="jet" if jet else "hs",
                    gas_giant=case["state"].startswith("jetgg"), turbulence=case["turbulence"], **h2)


def _grids(case, seed):
    """(grid, initial state) of each member, as a program has them before it starts a run: its own
    noise (or jets), and in an ensemble a drag rate within 10% of the reference's."""
    rng = np.random.default_rng(seed)
    out = []
    for ni, nj in _sizes(case):
        ga, f = hs_setup(_config(case, ni, nj, int(rng.integers(1 << 30))))
        if case["members"] > 1:
            ga.struct.hs_kf *= 1.0 + float(rng.uniform(-0.1, 0.1))
        out.append((ga, f))
    return out


class _Store:
    """Host arrays of members of one size, an ensemble's storage: one pinned block holds each member's
    state arrays back to back (a state then moves with one copy each way)."""

    def __init__(self, like, count):
        def zeros(shape):
            return torch.zeros((count,) + shape, dtype=torch.float64, pin_memory=True).numpy()

        packed = ["u", "v", "dudt", "dvdt"] + FIELD_NAMES_3D
        planes = {n: like.arrays[n].shape[0] if n in packed[:4] else 1 for n in packed}
        block, off = zeros((sum(planes.values()),) + like.layout.shape3), 0
        self.arrays = {}
        for n in packed:
            self.arrays[n] = block[:, off:off + planes[n]] if n in packed[:4] else block[:, off]
            off += planes[n]
        self.arrays.update({n: zeros(a.shape) for n, a in like.arrays.items() if n not in planes})
        self.fields = []
        for q in range(count):
            f = Fields(like.layout.ni, like.layout.nj, like.layout.nk, like.uv_scheme, turbulence=like.turbulence)
            for n in self.arrays:
                f.arrays[n] = self.arrays[n][q]
                setattr(f.struct, n, self.arrays[n][q].ctypes.data_as(C.POINTER(C.c_double)))
            f._block = None
            self.fields.append(f)

    def fill(self, fields):
        for f, g in zip(self.fields, fields):
            for n in self.arrays:
                f.arrays[n][...] = g.arrays[n]
            for n in ("it_zero", "it_minus1", "it_minus2", "itime", "model_time"):
                setattr(f.struct, n, getattr(g.struct, n))


def prepare(case, seed):
    form = FORMS[case["form"]]
    grids = _grids(case, seed)
    models = [Model(ga, form) for ga, _ in grids]
    state = {"do": case["do"], "steps": case["steps"], "grids": [ga for ga, _ in grids], "models": models}
    if case["members"] == 1:
        state["host"] = grids[0][1].copy(pinned=True)
        state["out"] = grids[0][1].copy(pinned=True)
        if case["do"] == "step_host":   # a run in progress: its diagnostics belong to its state
            m = models[0]
            m.upload(state["host"])
            m.timestep(EPIC_SYNC_DIAGS_ONLY)
            m.download(state["host"])
        return state
    state["batch"] = Batch(models)
    # members of one size share their storage
    state["in_stores"], state["out_stores"] = [], []
    order_in, order_out = [None] * len(grids), [None] * len(grids)
    for key in sorted({(f.layout.ni, f.layout.nj) for _, f in grids}):
        at = [q for q, (_, f) in enumerate(grids) if (f.layout.ni, f.layout.nj) == key]
        for stores, order in ((state["in_stores"], order_in), (state["out_stores"], order_out)):
            if case["do"] == "step_host" and stores is state["out_stores"]:
                continue
            s = _Store(grids[at[0]][1], len(at))
            s.fill([grids[q][1] for q in at])
            stores.append(s)
            for q, f in zip(at, s.fields):
                order[q] = f
    state["host"], state["out"] = order_in, order_out
    if case["do"] == "step_host":
        b = state["batch"]
        b.upload(state["host"])
        b.timestep(EPIC_SYNC_DIAGS_ONLY)
        b.sync()
        b.download(state["host"])
    return state


def _single_outputs(f):
    out = {"u": f.wind("u"), "v": f.wind("v"), "dudt": f.tendency("dudt"), "dvdt": f.tendency("dvdt")}
    out.update({n: f.arrays[n] for n in FIELD_NAMES_3D if n != "u_spinup"})
    out["gz_surface"] = f.gz_surface
    if f.turbulence:
        out.update({n: f.arrays[n] for n in TURB_FIELDS})
    return out


def _ensemble_outputs(stores, names):
    """Each array of all members of a size at once; of the wind arrays the current planes (every
    member has made the same number of steps, so their time-plane indices agree)."""
    out = []
    for s in stores:
        f, got = s.fields[0], {}
        wind = 0 if f.uv_scheme == EPIC_UV_AB3 else f.struct.it_zero
        tend = f.struct.it_minus1 if f.uv_scheme == EPIC_UV_AB3 else 0
        for n in names:
            a = s.arrays[n]
            got[n] = a[:, wind] if n in ("u", "v") else a[:, tend] if n in ("dudt", "dvdt") else a
        out.append(got)
    return out


def run(state):
    n = state["steps"]
    if "batch" in state:
        b = state["batch"]
        if state["do"] == "step_host":
            b.step_host(state["host"], nsteps=n, groups=8, io=EPIC_IO_STATE)
            return _ensemble_outputs(state["in_stores"], ["u", "v", "dudt", "dvdt", "hdry", "theta"])
        b.upload(state["host"])
        b.timestep(EPIC_SYNC_DIAGS_ONLY)
        b.run(n)
        b.download(state["out"])
        names = ["u", "v", "dudt", "dvdt", "hdry", "theta", "p3", "t3", "rho3", "gz3", "heat3", "pv3", "div_uv3", "w3"]
        return _ensemble_outputs(state["out_stores"], names)
    m = state["models"][0]
    if state["do"] == "step_host":
        m.step_host(state["host"], n)
        return _single_outputs(state["host"])
    m.upload(state["host"])
    m.timestep(EPIC_SYNC_DIAGS_ONLY)
    if state["do"] == "forecast":
        m.run(n)
    m.download(state["out"])
    out = _single_outputs(state["out"])
    if state["do"] == "diagnose":   # what the call computes from the state
        for k in ("u", "v", "dudt", "dvdt", "gz_surface"):
            del out[k]
    return out


def work(case):
    """Bytes: a state's arrays in and out of the device once, and per step the compulsory traffic of
    the prognostic variables (u, v, hdry, theta and two older tendency planes of each wind read; u, v,
    hdry, theta and the new tendencies written).  Flops: about 1500 operations a cell and step and 500
    a cell for the diagnostics (transcendentals counted as 20), estimated from the reference's loops."""
    nbytes = flops = 0.0
    for ni, nj in _sizes(case):
        cells, n3 = ni * nj * case["nk"], (ni + 2) * (nj + 3) * (case["nk"] + 2)
        planes = 10 if case["do"] == "step_host" and case["members"] > 1 else 28 + (4 if case["turbulence"] else 0)
        steps = 0 if case["do"] == "diagnose" else case["steps"]
        moves = steps if case["do"] == "step_host" and case["members"] > 1 else 1
        nbytes += 2 * 8 * planes * n3 * moves + 14 * 8 * cells * steps
        flops += 1500.0 * cells * steps + (0.0 if case["do"] == "step_host" else 500.0 * cells)
    return {"bytes": nbytes, "flops": flops}


# ---- the diagnostics of a state in binary64 numpy, from the model's equations ----

def exact(case, seed):
    """The diagnostics of an ideal-gas state over terrain.  A run of whole steps has no such value
    here: the step is some twenty coupled routines, and its binary64 form is itself compared bit for
    bit with a restatement of the reference in the tests."""
    if case["do"] != "diagnose" or case["state"] not in ("hs", "jet") or case["turbulence"]:
        return None
    (ga, f), = _grids(case, seed)
    g, L = ga.struct, f.layout
    ni, nj, nk, ks = L.ni, L.nj, L.nk, int(g.k_sigma)
    sg, ds = ga.sigmatheta, ga.dsgth
    lay = slice(1, nk + 1)                       # K = 1..nk
    rows = slice(1, nj + 2)                      # J = 0..nj
    jh, jv = 2 * np.arange(nj + 1) + 1, 2 * np.arange(nj + 2)
    grav = ga.g[jh][:, None]
    coeff = 1.0 / (1.0 - np.exp(-g.hybrid_alpha * (1.0 - g.sigma_sigma)))

    def theta_of(level, sigma):
        gs = np.where(sigma <= g.sigma_sigma, 0.0, np.where(sigma >= 1.0, 1.0, coeff * (1.0 - np.exp(-g.hybrid_alpha * (sigma - g.sigma_sigma)))))
        fs = (1.0 - gs) * (g.zeta0 + sigma * (g.zeta1 - g.zeta0))
        with np.errstate(divide="ignore", invalid="ignore"):
            return (level - fs) / gs

    hdry, theta = f.hdry[:, rows].copy(), f.theta[:, rows].copy()
    p3 = f.p3[:, rows].copy()
    for k in range(1, nk + 1):
        p3[k] = p3[k - 1] + ds[2 * k] * grav * hdry[k]
    top, bot = p3[0].copy(), p3[nk].copy()
    for k in range(ks - 1, nk):
        p3[k] = bot * np.exp((sg[2 * k + 1] - g.zeta0) / (g.zeta1 - g.zeta0) * np.log(top / bot))
    hl = np.zeros_like(p3)
    for k in range(1, nk + 1):
        hl[k] = (p3[k] - p3[k - 1]) / (grav * ds[2 * k])
        hdry[k] = np.maximum(ga.h_min[k], hl[k])
    lt = np.log(top / bot)
    for k in range(0, ks - 1):
        theta[k] = theta_of(sg[2 * k + 1], np.log(p3[k] / bot) / lt)
    k1 = g.kappa + 1.0
    p2, h3, theta2 = np.zeros_like(p3), np.zeros_like(p3), f.theta2[:, rows].copy()
    for k in range(1, nk + 1):
        p2[k] = ((p3[k] ** k1 - p3[k - 1] ** k1) / (k1 * (p3[k] - p3[k - 1]))) ** (1.0 / g.kappa)
        h3[k] = hl[nk] if k == nk else (ds[2 * k] * hl[k] + ds[2 * k + 2] * hl[k + 1]) / (ds[2 * k] + ds[2 * k + 2])
    p2[0] = p3[0] * p3[0] / p2[1]
    h3[0] = h3[1]
    for k in range(1, ks - 1):
        theta2[k] = theta_of(sg[2 * k], np.log(p2[k] / bot) / lt)
    theta2[ks - 1] = 0.5 * (theta[ks - 1] + theta[ks - 2])
    for k in range(ks, nk + 1):   # linear in sigmatheta between the interfaces around the layer
        x0, x1 = sg[2 * k + 1], sg[2 * k - 1]
        theta2[k] = theta[k] + (theta[k - 1] - theta[k]) * (sg[2 * k] - x0) / (x1 - x0)
    theta2[0] = sg[0]
    mu_over_r = (1.0 / (g.rgas / 8.314472e3)) / 8.314472e3
    t3 = theta * (p3 / g.press0) ** g.kappa
    t2 = np.zeros_like(t3)
    t2[lay] = theta2[lay] * (p2[lay] / g.press0) ** g.kappa
    with np.errstate(divide="ignore", invalid="ignore"):
        rho3, rho2 = p3 * mu_over_r / t3, p2 * mu_over_r / t2
        exner3 = g.cp * t3 / theta
        rho2[0] = rho3[0] * rho3[0] / rho2[1]
    t2[0] = t3[0]
    gz = np.zeros_like(p3)
    gz[nk] = g.topo_scale * f.gz_surface[rows]
    dl = np.zeros_like(p3)
    dl[lay] = np.log(p3[1:nk + 1] / p3[0:nk])
    for k in range(nk, 0, -1):
        if k == nk or k == 1:
            gz[k - 1] = gz[k] + (p3[k] + p3[k - 1]) / (rho3[k] + rho3[k - 1]) * dl[k]
            continue
        a, b, c = dl[k + 1], dl[k], dl[k - 1]    # the cubic through four levels, integrated over the middle one
        ba, cb = b + a, c + b
        cba = c + ba
        q0, q1, q2, q3 = (p3[m] / rho3[m] for m in (k + 1, k, k - 1, k - 2))
        gz[k - 1] = gz[k] - (q0 * (b ** 3 * (cb + c)) / (a * ba * cba) + q1 * (b * (b * (b + 2 * (a - cb)) - 6 * a * cb)) / (a * cb)
                             + q2 * (b * (b * (b + 2 * (c - ba)) - 6 * ba * c)) / (ba * c)
                             + q3 * (b ** 3 * (a + ba)) / (cba * cb * c)) / 12.0
    mont = gz + g.cpr * g.rgas * t3

    # the zonal filter poleward of lat0: Fourier amplitudes scaled by min(1, r / sin^2(k dlon / 2))
    deg = np.pi / 180.0
    lat0 = g.lat0 * deg
    rln0 = g.re / np.sqrt(1.0 + (g.rp / g.re * np.tan(lat0)) ** 2)
    rlt0 = rln0 / (np.cos(lat0) * (np.sin(lat0) ** 2 + (g.re / g.rp * np.cos(lat0)) ** 2))
    m0, n0 = 1.0 / (rln0 * g.dln * deg), 1.0 / (rlt0 * g.dlt * deg)

    def zonal_filter(a, jj):
        spec = np.fft.rfft(a[..., 1:ni + 1], axis=-1)
        wave = np.arange(1, ni // 2 + 1)
        for q, h in enumerate(jj):
            if abs(ga.lat[h]) >= g.lat0:
                r = ga.mn[h] / (ga.m[h] * ga.n[h]) * ((ga.n[h] / n0) / (ga.m[h] / m0)) ** 2
                spec[..., q, 1:] *= np.minimum(1.0, r * np.sin(wave * g.dln * deg / 2.0) ** -2.0)
        out = np.fft.irfft(spec, n=ni, axis=-1)
        return np.concatenate((out[..., -1:], out, out[..., :1]), axis=-1)

    kk = slice(0, nk + 1)
    u, v = f.wind("u")[kk, 1:nj + 2], f.wind("v")[kk, 1:nj + 3]   # v rows J = 0..nj+1, zero at the poles
    fu = zonal_filter(u, jh)
    m, n, mn = ga.m, ga.n, ga.mn
    inv_m = np.zeros(nj + 2)
    inv_m[1:nj + 1] = 1.0 / m[jv[1:nj + 1]]
    vm = v * inv_m[:, None]
    div = np.zeros_like(p3)
    div[kk, :, 1:ni + 1] = mn[jh][:, None] * ((fu[..., 2:] - fu[..., 1:-1]) / n[jh][:, None] + (vm[:, 1:, 1:ni + 1] - vm[:, :-1, 1:ni + 1]))
    fv = zonal_filter(f.wind("v")[kk, 2:nj + 2], jv[1:nj + 1])    # J = 1..nj
    um = u / m[jh][:, None]
    j = jv[1:nj + 1]
    ze = m[j][:, None] * ((fv[..., 1:ni + 1] - fv[..., 0:ni]) + n[j][:, None] * (um[:, :-1, 1:ni + 1] - um[:, 1:, 1:ni + 1]))
    area = 1.0 / mn[jh]
    hk = h3[kk]
    hs = (hk[..., 1:ni + 1] + hk[..., 0:ni]) * area[:, None]
    hpv = (hs[:, 1:] + hs[:, :-1]) * (0.5 / (area[1:] + area[:-1]))[:, None]
    pv = np.zeros((nk + 2, nj + 3, ni + 2))
    pv[kk, 2:nj + 2, 1:ni + 1] = (ze + ga.f[j][:, None]) / hpv
    pv[kk, 1, 1:ni + 1] = ((-u[:, 0, 1:ni + 1].sum(-1) * mn[0] / (m[1] * ni) + ga.f[0]) / hk[:, 0, 1:ni + 1].mean(-1))[:, None]
    pv[kk, nj + 2, 1:ni + 1] = ((u[:, nj, 1:ni + 1].sum(-1) * mn[2 * nj + 2] / (m[2 * nj + 1] * ni) + ga.f[2 * nj + 2])
                                / hk[:, nj, 1:ni + 1].mean(-1))[:, None]

    # Newtonian cooling of Held and Suarez (1994)
    ka, kw = 1.0 / (40 * 86400.0), 1.0 / (4 * 86400.0)
    cl = np.cos(ga.lat[jh] * deg)[:, None]
    heat = np.zeros_like(p3)
    if g.newt_cool_on:
        p = p3[lay]
        amp = np.maximum(0.0, (p / p3[nk] - 0.7) / 0.3)
        teq = np.maximum(200.0, (315.0 - 60.0 * (1.0 - cl * cl) - 10.0 * np.log(p / 1e5) * cl * cl) * (p / 1e5) ** g.kappa)
        heat[lay] = -1004.0 * (ka + (kw - ka) * cl ** 4 * amp) * (t3[lay] - teq)

    def whole(a, like):
        """On the stored array: rows J = 0..nj and their periodic columns computed, the rest as it was."""
        out = like.copy()
        out[kk, rows] = a[kk]
        return out

    def wrap(a):
        a[..., 0], a[..., ni + 1] = a[..., ni], a[..., 1]
        return a

    out = {n: None for n in FIELD_NAMES_3D if n != "u_spinup"}
    hdry[0] = f.hdry[0, rows]
    for name, a in (("hdry", hdry), ("theta", theta), ("p3", p3), ("h3", h3), ("p2", p2), ("theta2", theta2), ("t2", t2), ("t3", t3),
                    ("rho2", rho2), ("rho3", rho3), ("exner3", exner3), ("gz3", gz), ("mont3", mont),
                    ("heat3", wrap(heat)), ("div_uv3", wrap(div))):
        out[name] = whole(a, f.arrays[name])
    full = f.pv3.copy()
    full[kk, 1:nj + 3] = wrap(pv)[kk, 1:nj + 3]
    out["pv3"] = full
    return out

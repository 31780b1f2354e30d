"""The work a user of this framework has it do, as cases that can be timed.

The path is one 2DDI time step after another: a host binds its module arrays
once (``adc_gpu_bind``), steps the model with ``adc_run`` (many steps per
call), ``adc_timestep`` (one per call) or the four phase calls a Fortran host
has in place of its own subroutines, and copies the state back at output
times (``adc_sync_to_host``).  Beside it stand the ITPACK ``jcg`` drop-in on
host arrays, the batched ensemble and the learned initial guess with its
training on the device.

A case names the mesh by its kind and its two node counts, the entry point
(``call``), the number of time steps of one pass, and the options in use.
``prepare`` builds the module arrays of that mesh with an initial state and
a forcing drawn from the seed and binds them; ``run`` is one output
interval: the steps, then the state back on the host.  Passes on one state
continue its simulation.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from adcirc_b200 import _lib, ensemble, learned, meshgen, model

# state a host writes at an output or hotstart step
OUTPUTS = ("eta1", "eta2", "etas", "uu2", "vv2", "qx2", "qy2", "h1", "h2", "tk", "totalarea",
           "alphal", "wsx2", "wsy2", "pr2", "nodecode", "nnodecode", "noff", "mju")
PRECISIONS = {"fp64": _lib.ADC_PREC_FP64, "mixed": _lib.ADC_PREC_MIXED}


def listed():
    return [
        # a small linear tide model stepped by a Fortran host through the four
        # phase calls (the quarter-annular harbour of the tests): all latency
        dict(name="harbour_phases", mesh="harbour", nx=21, ny=31, call="phases", steps=8,
             precision="fp64"),
        # the wetting and drying beach of the parity tests, many steps a call
        dict(name="beach_run", mesh="beach", nx=41, ny=13, call="run", steps=200, precision="fp64"),
        # the tidal channel of the bench specification, 4,961 nodes, fully wet
        dict(name="channel_run", mesh="channel", nx=121, ny=41, call="run", steps=240,
             precision="fp64"),
        # the channel with a river and a storm, one call per time step as a
        # host does that has its own per-step work (coupling, station output)
        dict(name="channel_river_step", mesh="river", nx=121, ny=41, call="step", steps=40,
             precision="fp64"),
        # the channel with an internal barrier (levee) and a fort.19 series on
        # the open boundary: barrier overflow and series forcing
        dict(name="levee_run", mesh="levee", nx=121, ny=41, call="run", steps=120,
             precision="fp64"),
        # a county-size surge model: storm, tides, wetting and drying
        dict(name="shelf_25k_run", mesh="shelf", nx=157, ny=159, call="run", steps=200,
             precision="fp64"),
        # the FP32 assembly / matrix / momentum option on a mid-size mesh
        dict(name="shelf_100k_mixed", mesh="shelf", nx=313, ny=321, call="run", steps=200,
             precision="mixed"),
        # the learned initial guess being trained beside the solver: network
        # forward, backward, Adam, and the solves it learns from
        dict(name="shelf_50k_train", mesh="shelf", nx=229, ny=221, call="train", steps=30,
             precision="fp64"),
        # forecast ensemble: members of uneven size stepped together
        dict(name="ensemble_6", mesh="shelf", nx=199, ny=201, call="ensemble", steps=60, members=6,
             precision="fp64"),
        # the ITPACK drop-in on host arrays, one GWCE solve
        dict(name="jcg_90k", mesh="shelf", nx=299, ny=307, call="jcg", steps=1, noalloc=False,
             precision="fp64"),
        # a basin-scale surge model, one call per time step
        dict(name="shelf_250k_step", mesh="shelf", nx=499, ny=503, call="step", steps=60,
             precision="fp64"),
        # the size of the headline benchmark, state out every ten minutes of
        # simulated time at DT = 1 s (half of that here)
        dict(name="shelf_600k_run", mesh="shelf", nx=775, ny=773, call="run", steps=300,
             precision="fp64"),
    ]


def draw(rng):
    """A case of the same ranges: any entry point, sizes spread over the
    logarithm of the node count, odd shapes among them."""
    call = rng.choice(["phases", "run", "run", "run", "step", "step", "jcg", "ensemble", "train"])
    mesh = "shelf"
    if call in ("run", "step", "phases") and rng.random() < 0.4:
        mesh = rng.choice(["harbour", "beach", "channel", "river", "levee"])
    if mesh == "shelf":
        top = {"run": 500e3, "step": 300e3, "phases": 60e3, "jcg": 120e3, "ensemble": 40e3,
               "train": 60e3}[call]
        n = math.exp(rng.uniform(math.log(2500.0), math.log(top)))
        aspect = rng.uniform(0.7, 1.4)
        nx = max(40, int(math.sqrt(n * aspect)))
        ny = max(40, int(n / nx) + rng.randrange(3))
    elif mesh == "harbour":
        nx, ny = rng.randrange(11, 60), rng.randrange(16, 80)
    elif mesh == "beach":
        nx, ny = rng.randrange(31, 90), rng.randrange(9, 40)
    else:
        nx, ny = 121, 41
    case = dict(mesh=mesh, nx=nx, ny=ny, call=call, precision="fp64",
                steps={"run": rng.randrange(60, 240), "step": rng.randrange(20, 60),
                       "phases": rng.randrange(4, 12), "jcg": 1, "ensemble": rng.randrange(20, 60),
                       "train": rng.randrange(10, 30)}[call])
    if call == "run" and mesh == "shelf" and rng.random() < 0.25:
        case["precision"] = "mixed"
    if call == "ensemble":
        case["members"] = rng.randrange(2, 7)
    if call == "jcg":
        # the variant without allocations holds its staging in 32 MiB
        case["noalloc"] = nx * ny < 80000 and rng.random() < 0.5
    return case


# ------------------------------------------------------------------ meshes

def _hilbert(i, j, order):
    """Distance along the Hilbert curve of order `order` (2^order a side)."""
    d = np.zeros_like(i)
    i, j = i.copy(), j.copy()
    s = 1 << (order - 1)
    while s > 0:
        ri, rj = ((i & s) > 0).astype(np.int64), ((j & s) > 0).astype(np.int64)
        d += s * s * ((3 * ri) ^ rj)
        flip = (rj == 0) & (ri == 1)
        i, j = np.where(flip, s - 1 - i, i), np.where(flip, s - 1 - j, j)
        i, j = np.where(rj == 0, j, i), np.where(rj == 0, i, j)
        s >>= 1
    return d


_raw = {}


def _shelf_mesh(nx, ny):
    """A coastal shelf of 200 x 160 km with nx x ny nodes: rows graded to the
    coast, interior nodes jittered, diagonals at random (4 to 8 neighbours),
    nodes along a Hilbert curve; 60 m at the shelf break, 0 m at a winding
    coast, land to +3 m, half a metre of bottom roughness.  Open boundary:
    the south edge, the other sides are land."""
    if (nx, ny) in _raw:
        return _raw[nx, ny]
    rng = np.random.default_rng(1000003 * nx + ny)
    lx, ly = 200e3, 160e3
    t = np.linspace(0.0, 1.0, ny)
    ys = ly * (t + 0.12 * np.sin(2.0 * math.pi * (t - 0.04)) / (2.0 * math.pi) * 2.0)
    ys = (ys - ys[0]) * (ly / (ys[-1] - ys[0]))
    xs = np.linspace(0.0, lx, nx)
    X, Y = np.meshgrid(xs, ys, indexing="ij")
    hx, hy = lx / (nx - 1), np.gradient(ys)[None, :]
    inner = np.zeros((nx, ny))
    inner[1:-1, 1:-1] = 0.2
    X = X + inner * hx * rng.uniform(-1.0, 1.0, (nx, ny))
    Y = Y + inner * hy * rng.uniform(-1.0, 1.0, (nx, ny))
    coast = 0.8 * ly + 5e3 * np.sin(2.0 * math.pi * X / 61e3) + 2e3 * np.sin(2.0 * math.pi * X / 17e3)
    s = coast - Y
    depth = np.where(s > 0, 60.0 * np.sqrt(np.clip(s / 100e3, 0.0, 1.2)), 3.0 * np.clip(s / 20e3, -1.0, 0.0))
    rough = (0.5 * np.sin(2.0 * math.pi * X / 7.3e3 + 0.4) * np.sin(2.0 * math.pi * Y / 5.1e3)
             * np.clip(1.0 - np.abs(s) / 40e3, 0.0, 1.0))
    depth = depth + rough
    nid = np.arange(nx * ny).reshape(nx, ny)
    a, b, c, d = nid[:-1, :-1], nid[1:, :-1], nid[1:, 1:], nid[:-1, 1:]
    up = rng.random(a.shape) < 0.5
    t1 = np.where(up[..., None], np.stack([a, b, c], -1), np.stack([a, b, d], -1)).reshape(-1, 3)
    t2 = np.where(up[..., None], np.stack([a, c, d], -1), np.stack([b, c, d], -1)).reshape(-1, 3)
    nm = np.concatenate([t1, t2])
    I, J = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    perm = np.argsort(_hilbert(I.ravel(), J.ravel(), max(nx, ny).bit_length()), kind="stable")
    inv = np.empty_like(perm)
    inv[perm] = np.arange(perm.size)
    nm = inv[nm]
    nm = nm[np.lexsort((nm.max(axis=1), nm.min(axis=1)))]
    nid = inv[nid]
    land = np.concatenate([nid[-1, :], nid[-2::-1, -1], nid[0, -2::-1]])   # SE, NE, NW, SW corners
    raw = meshgen.RawMesh("shelf", X.ravel()[perm], Y.ravel()[perm], depth.ravel()[perm], nm,
                          nid[::-1, 0].copy(), [(0, land)], {"lx": lx, "ly": ly})
    while len(_raw) >= 8:   # the members of one ensemble
        _raw.pop(next(iter(_raw)))
    _raw[nx, ny] = raw
    return raw


def _bumps(x, y, rng, amp):
    """A smooth random field of about `amp`, a few waves across the domain."""
    lx, ly = x.max() - x.min(), y.max() - y.min()
    f = np.zeros_like(x)
    for _ in range(4):
        kx, ky = rng.uniform(0.5, 3.0, 2)
        f += np.cos(2.0 * math.pi * (kx * (x - x.min()) / lx + ky * (y - y.min()) / ly)
                    + rng.uniform(0.0, 2.0 * math.pi))
    return 0.5 * amp * f


def _shelf_case(nx, ny, rng):
    """The surge settings of the framework (model.surge_case: hybrid friction,
    slope limiter, TAU0 = -1, M2 + K1) on the shelf, half an hour of ramp, a
    sloping initial sea and a Holland vortex that crosses the coast."""
    raw = _shelf_mesh(nx, ny)
    c = model.surge_case(raw=raw, vortex=False, nws=8, tide_scale=float(rng.uniform(0.5, 1.5)))
    eta0 = _bumps(raw.x, raw.y, rng, 0.3)
    _start_from(c, eta0)
    c.schedule = model.Schedule(dt=c.params["dt"], dramp=0.02, dramp_mete=0.02)
    heading, speed = float(90.0 + rng.uniform(-30.0, 30.0)), float(rng.uniform(3.0, 8.0))
    c.vortex = model.straight_track(float(rng.uniform(60e3, 140e3)) + 0.5, 40e3 + 0.5, heading, speed,
                                    float(rng.uniform(920.0, 980.0)), float(rng.uniform(20.0, 60.0)),
                                    1.3, hours=72.0)
    return c


def _start_from(c, eta0):
    """Cold start (cstart.F) of a built case from the elevations eta0."""
    a, p, n = c.arrays, c.params, _lib.ptr
    a["eta1"][:] = 0.0
    a["eta2"][:] = eta0
    for k in ("nodecode", "nnodecode", "mju"):
        a[k][:] = 0
    a["noff"][:] = 1
    a["totalarea"][:] = 0.0
    rc = _lib.load().adc_coldstart(
        c.sizes["np"], c.sizes["ne"], p["nolifa"], p["h0"], n(a["dp"], _lib.dp_), n(a["nm"], _lib.ip_),
        n(a["areas"], _lib.dp_), n(a["eta1"], _lib.dp_), n(a["eta2"], _lib.dp_),
        n(a["nnodecode"], _lib.ip_), n(a["nodecode"], _lib.ip_), n(a["noff"], _lib.ip_),
        n(a["mju"], _lib.ip_), n(a["totalarea"], _lib.dp_))
    if rc != 0:
        raise RuntimeError(f"adc_coldstart: {rc}")


def _case(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"]])
    amp = float(rng.uniform(0.3, 0.6))
    # no advective terms where the tests run the same mesh for days
    linear = dict(ifnlct=0, ifnlcat=0)
    if case["mesh"] == "shelf":
        return _shelf_case(case["nx"], case["ny"], rng)
    if case["mesh"] == "harbour":
        c = model.quarter_annulus_case(nr=case["nx"], nth=case["ny"], amp=amp)
        _start_from(c, _bumps(c.arrays["x"], c.arrays["y"], rng, 0.05))
        return c
    if case["mesh"] == "beach":
        raw = meshgen.beach_mesh(case["nx"], case["ny"])
        tides = [(2.0 * math.pi / 10800.0, 0.0, 1.0, np.full(raw.open_nodes.size, amp),
                  np.zeros(raw.open_nodes.size))]
        sched = model.Schedule(dt=2.0, reftim=0.25 * 10800.0 / 86400.0, nramp=0)
        c = model.build_case(raw, model.default_params(2.0, **linear), sched, tides)
        _start_from(c, _bumps(raw.x, raw.y, rng, 0.05))
        return c
    if case["mesh"] == "channel":
        c = model.channel_case(amp=amp, **linear)
    elif case["mesh"] == "river":
        c = model.channel_case(amp=amp, vortex=True, river=float(rng.uniform(0.3, 1.0)), **linear)
        c.vortex = model.straight_track(30.3e3, 3.7e3, float(rng.uniform(60.0, 100.0)), 0.2,
                                        float(rng.uniform(960.0, 985.0)), 8.0, 1.3, hours=96.0,
                                        interval_h=6.0)
    else:
        c = model.channel_case(amp=amp, levee=float(rng.uniform(0.1, 0.2)), elev_series=600.0,
                               series_hours=96.0, **linear)
        ser = c.elev_series
        c.elev_series = model.Series(ser.interval, ser.values - ser.values[:1]
                                     - 0.1 * np.arange(ser.values.shape[0])[:, None] * ser.interval / 3600.0)
    eta0 = _bumps(c.arrays["x"], c.arrays["y"], rng, 0.1)
    if case["mesh"] == "levee":   # high water against the levee, the polder behind it dry
        eta0 = np.where(c.arrays["x"] <= 30e3, 0.2 + 0.3 * eta0, -1.0)
    _start_from(c, eta0)
    return c


# ----------------------------------------------------------------- systems

def _gwce_system(case, seed):
    """One GWCE system in the arrays gwce.F hands to jcg: COEF(NP,MNEI) of
    consistent mass and gravity terms, its NeiTab, a load vector and the
    guess of the previous step (a few percent off)."""
    rng = np.random.default_rng([seed, 7])
    c = _case(case, seed)
    a, n, mnei = c.arrays, c.sizes["np"], c.sizes["mnei"]
    nm = a["nm"].astype(np.int64) - 1                       # (NE, 3)
    area2, fx, fy = a["areas"], a["fdxe"], a["fdye"]        # (NE,), (3, NE)
    dt, g = c.params["dt"], c.params["g"]
    depth = np.maximum(a["dp"] + a["eta2"], 0.05)[nm].mean(axis=1)
    tau0 = a["tau0var"][nm].mean(axis=1)
    mass = 0.5 * area2 * (1.0 / dt + 0.5 * tau0) / dt / 12.0
    grav = c.params["a00"] * g * depth / (2.0 * area2)
    coef = np.zeros((n, mnei), order="F")
    pos = a["csr_position"].astype(np.int64)
    for k in range(3):
        np.add.at(coef[:, 0], nm[:, k], 2.0 * mass + grav * (fx[k] ** 2 + fy[k] ** 2))
        for slot, l in enumerate([(k + 1) % 3, (k + 2) % 3] if k != 1 else [0, 2]):
            l = [[1, 2], [0, 2], [0, 1]][k][slot]
            np.add.at(coef, (nm[:, k], pos[:, k, slot] - 1), mass + grav * (fx[k] * fx[l] + fy[k] * fy[l]))
    x = 1e-3 * _bumps(a["x"], a["y"], rng, 1.0)
    rhs = _ell_times(coef, a["neitab"], x)
    u0 = x * (1.0 + 0.03 * np.cos(7.0 * np.arange(n) / n))
    return coef, a["neitab"], rhs, u0, c


def _ell_times(coef, neitab, x):
    idx = np.maximum(neitab.astype(np.int64) - 1, 0)
    return np.einsum("ij,ij->i", coef, np.where(neitab > 0, x[idx], 0.0))


class _Jcg:
    def __init__(self, case, seed):
        self.lib = _lib.load()
        self.coef, neitab, self.rhs0, self.u0, _ = _gwce_system(case, seed)
        self.jcoef = np.asfortranarray(neitab, np.int32)
        self.n, self.mnei = self.coef.shape
        self.rhs, self.u = self.rhs0.copy(), self.u0.copy()
        self.itmax = 200
        self.nw = 4 * self.n + 4 * self.itmax
        self.wksp, self.iwksp = np.zeros(self.nw), np.zeros(3 * self.n, np.int32)
        self.iparm, self.rparm = np.zeros(12, np.int32), np.zeros(12)
        self.call = self.lib.adc_jcg_noalloc if case["noalloc"] else self.lib.adc_jcg
        self.lib.adc_jcg_reset()


# ------------------------------------------------------------- the contract

def prepare(case, seed):
    call = case["call"]
    if call == "jcg":
        return {"call": call, "jcg": _Jcg(case, seed)}
    prec = PRECISIONS[case["precision"]]
    st = {"call": call, "steps": case["steps"], "it": 1}
    if call == "ensemble":
        members = []
        for k in range(case["members"]):
            shrink = 0.35 ** (k / max(1, case["members"] - 1))   # uneven sizes, a factor of about 8
            members.append(_case(dict(case, nx=max(40, int(case["nx"] * shrink)),
                                      ny=max(40, int(case["ny"] * shrink))), seed + 1000 * k))
        st["ens"] = ensemble.Ensemble(members, prec=prec)
        return st
    c = _case(case, seed)
    st["gm"] = model.GpuModel(c, prec=prec)
    if call == "train":
        p = learned.init_params(np.array([0.0, 0.0, 0.0, 0.0, 20.0, 0.8, 0.0, 0.0, 0.0]),
                                np.array([0.3, 1e-3, 0.5, 0.5, 20.0, 0.4, 0.1, 1e-3, 1e-3]), 1e-4,
                                seed=seed)
        v = learned.layer_views(p)
        v["w_out"][:] = np.random.default_rng(seed).normal(0.0, 0.1, learned.H)
        st["gm"].set_predictor(p)
        st["gm"].predictor_train(True, 1e-3)
    return st


def _state(c):
    return {k: c.arrays[k] for k in OUTPUTS}


def run(st):
    call = st["call"]
    if call == "jcg":
        j = st["jcg"]
        j.rhs[:], j.u[:] = j.rhs0, j.u0
        i, d = _lib.ip_, _lib.dp_
        j.lib.adc_dfault(_lib.ptr(j.iparm, i), _lib.ptr(j.rparm, d))
        j.iparm[0], j.rparm[0] = j.itmax, 1e-10
        ier = C.c_int(0)
        j.call(C.byref(C.c_int(j.n)), C.byref(C.c_int(j.n)), C.byref(C.c_int(j.mnei)),
               _lib.ptr(j.jcoef, i), _lib.ptr(j.coef, d), _lib.ptr(j.rhs, d), _lib.ptr(j.u, d),
               _lib.ptr(j.iwksp, i), C.byref(C.c_int(j.nw)), _lib.ptr(j.wksp, d),
               _lib.ptr(j.iparm, i), _lib.ptr(j.rparm, d), C.byref(ier))
        return {"u": j.u, "coef": j.coef, "rhs": j.rhs, "numitr": int(j.iparm[0]), "ier": ier.value}
    n = st["steps"]
    if call == "ensemble":
        e = st["ens"]
        numitr, _ = e.run(n)
        out = {"numitr": numitr}
        for k, m in enumerate(e.models):
            m.sync_to_host()
            a = m.case.arrays
            out[f"m{k}"] = {f: a[f] for f in ("eta2", "etas", "uu2", "vv2", "nodecode", "noff")}
        return out
    gm, it = st["gm"], st["it"]
    st["it"] = it + n
    if call in ("run", "train"):
        numitr, _ = gm.run(it, n)
    elif call == "step":
        numitr = np.array([gm.step(it + k).numitr for k in range(n)], np.int32)
    else:
        numitr = np.zeros(n, np.int32)
        lib, o = gm.lib, _lib.AdcStepOut()
        for k in range(n):
            s = C.byref(gm.case.schedule.step(it + k))
            rc = lib.adc_shift_friction(gm.h, s) or lib.adc_gwce_new(gm.h, s, C.byref(o))
            numitr[k] = o.numitr
            rc = rc or lib.adc_wetdry(gm.h, s, C.byref(o)) or lib.adc_momentum(gm.h, s)
            if rc != 0:
                raise RuntimeError(f"step {it + k}: status {rc}")
    gm.sync_to_host()
    out = dict(_state(gm.case), numitr=numitr)
    if call == "train":
        out["predictor"] = gm.get_predictor()
        out["loss"] = gm.predictor_stats()[0]
    return out


def work(case):
    """Per node and time step: the state read and written once (25 and 20
    doubles), two elements of geometry and flags (80 B each), seven matrix
    entries written and read (8 B); 1,300 FP64 operations (two elements'
    GWCE, momentum and wet/dry terms, 15 JCG iterations).  A pass also
    writes the state out, once.  A lone solve reads and writes COEF and reads
    JCOEF and three vectors."""
    n = float(case["nx"] * case["ny"])
    if case["call"] == "jcg":
        return {"bytes": n * (8 * 20 + 4 * 10 + 8 * 4), "flops": n * 15 * 26}
    if case["call"] == "ensemble":
        m = case["members"]
        n = n * sum(0.35 ** (2.0 * k / max(1, m - 1)) for k in range(m))
    per, flops = 8.0 * 45 + 2 * 80.0 + 8.0 * 14, 1300.0
    if case["call"] == "train":
        # three message-passing layers forward and backward: activations of
        # 64 BF16 read and written, 3 x 2 x 128 x 64 products a layer
        per, flops = per + 3 * 6 * 128.0, flops + 3 * 6 * 128 * 64.0
    return {"bytes": n * (case["steps"] * per + 8.0 * 40), "flops": n * case["steps"] * flops}


def exact(case, seed):
    """The solution of a lone GWCE system (conjugate gradients in 64 bits to
    rounding); COEF and the load vector come back as they were.  A time
    marching run has no value of that kind."""
    if case["call"] != "jcg":
        return None
    coef, neitab, b, x0, _ = _gwce_system(case, seed)
    idx = torch.from_numpy(np.maximum(neitab.astype(np.int64) - 1, 0))
    A = torch.from_numpy(np.where(neitab > 0, coef, 0.0))
    mul = lambda v: (A * v[idx]).sum(dim=1)
    b, x, d = torch.from_numpy(b), torch.from_numpy(x0.copy()), A[:, 0]
    r = b - mul(x)
    z = r / d
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(200):
        q = mul(p)
        alpha = rz / torch.dot(p, q)
        x = x + alpha * p
        r = r - alpha * q
        if float(r.norm()) <= 1e-16 * float(b.norm()):
            break
        z = r / d
        new = torch.dot(r, z)
        p, rz = z + (new / rz) * p, new
    return {"u": x.numpy(), "coef": coef, "rhs": b.numpy(), "numitr": None, "ier": None}

"""Performance cases of the framework: whole calls as a user's program makes them.

A pass is one piece of work from the model arrays in host memory (page-locked,
as a program that cares for speed keeps them) to the results in host memory:

- ``shot``: one plan is created, run for its steps, read and closed -- the
  reference program's main(), and the inner loop of a survey;
- ``batch``: several shots in one batch, sharing a model or each its own;
- ``serve``: a burst of requests to a server that is already up.

``exact`` restates the time loop (staggered-grid elastic update with C-PML,
receivers, source) in float64 torch operations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ela3d_gb300 as ela

RICKER, GAUSS_DERIV = ela.STF_RICKER, ela.STF_GAUSS_DERIV


# ------------------------------------------------------------------ cases --
def _shot(name, nx, ny, nz, npml, steps, **kw):
    c = {"kind": "shot", "nx": nx, "ny": ny, "nz": nz, "npml": npml, "steps": steps, "fp64": False,
         "explosive": False, "clean": False, "model": "dome", "sampgat": 1, "energy_every": 0, "snap_every": 0,
         "snap_last": 3}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # (a shot returns its seismograms, source trace and, unless said
        # otherwise, the three velocity snapshots the reference writes)
        # the smallest grids of a request stream: two half-steps of a few
        # microseconds each, so latency and waits between blocks count
        _shot("shot_64", 64, 64, 64, 10, 400),
        # the reference's CPU-sized cube, the whole named shot
        _shot("cube_101", 101, 101, 101, 10, 1000, model="homogeneous"),
        # the same cube in the FP64 build, which checks FP32 results
        _shot("cube_101_fp64", 101, 101, 101, 10, 150, model="homogeneous", fp64=True),
        # an FP64 re-run of a heterogeneous shot with the other source kind
        _shot("fp64_explosive_160", 160, 128, 144, 12, 50, fp64=True, explosive=True),
        # the headline shot: layered dome, 201-receiver line
        _shot("anticline_256", 256, 256, 256, 16, 300, snap_last=1),
        # the reference program's own use: the five-medium 201^3 model, its
        # explosive source, samples every second step
        _shot("explosive_201", 201, 201, 201, 10, 200, model="matlab", explosive=True, sampgat=2),
        # a survey box of no convenient size, textbook profiles
        _shot("ragged_150", 150, 211, 93, 13, 400, clean=True),
        # a run that is watched: energy check every 20 steps, a vz snapshot
        # every 100
        _shot("monitored_192", 192, 160, 176, 14, 200, energy_every=20, snap_every=100, snap_last=0),
        # a grid far beyond the L2, its model generated on the device
        _shot("large_640", 640, 512, 384, 16, 30, model="device", snap_last=0),
        # shots of one survey: one model, many source positions
        {"name": "batch_shared_192", "kind": "batch", "shots": 8, "shared": True, "lo": 192, "hi": 192, "npml": 16,
         "steps": 60, "grids": 0},
        # independent shots of every size (edges are multiples of 16)
        {"name": "batch_uneven", "kind": "batch", "shots": 10, "shared": False, "lo": 64, "hi": 320, "npml": 0,
         "steps": 80, "grids": 1},
        # a burst of requests with lognormal edges
        {"name": "serve_16", "kind": "serve", "requests": 16, "lo": 64, "hi": 256, "steps": 100, "grids": 2},
    ]


_COST = 5.1e9   # cell-updates of the largest listed pass (256^3, 300 steps)


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["shot"] * 7 + ["fp64", "fp64", "batch", "batch", "serve"])
    if kind == "batch":
        if rng.random() < 0.5:
            n = 16 * rng.randint(6, 13)
            return {"kind": "batch", "shots": rng.randint(4, 10), "shared": True, "lo": n, "hi": n,
                    "npml": rng.randint(10, 20), "steps": rng.randint(40, 60), "grids": 0}
        return {"kind": "batch", "shots": rng.randint(6, 12), "shared": False, "lo": 64, "hi": 256, "npml": 0,
                "steps": rng.randint(50, 80), "grids": rng.randint(10, 10 ** 6)}
    if kind == "serve":
        return {"kind": "serve", "requests": rng.randint(8, 20), "lo": 64, "hi": 256, "steps": rng.randint(60, 100),
                "grids": rng.randint(10, 10 ** 6)}
    fp64 = kind == "fp64"
    nx, ny, nz = (_edge(rng, 64, 180 if fp64 else 400) for _ in range(3))
    cells = nx * ny * nz
    # the FP64 build runs about a fifteenth of the FP32 rate
    steps = int(min(600 if not fp64 else 150, (_COST if not fp64 else _COST / 16) / cells))
    kw = {"fp64": fp64, "explosive": rng.random() < 0.35, "clean": rng.random() < 0.3, "sampgat": rng.choice([1, 1, 2, 4]),
          "model": rng.choice(["dome", "dome", "homogeneous", "device"])}
    if not fp64 and rng.random() < 0.2:
        kw["energy_every"] = rng.choice([10, 20, 50])
    kw["snap_last"] = 3 if cells < 4e6 else rng.choice([0, 1, 3])
    return _shot(None, nx, ny, nz, rng.randint(8, 20), max(20, steps), **kw)


# ----------------------------------------------------------------- inputs --
def _dome_spec(rng, nx, ny, nz, seed, layers=None, perturb=0.02):
    """Layered dome in the form of the device generator's model spec: cp
    increasing with depth, cs = cp / ratio, rho = 310 cp^0.25."""
    n = int(rng.integers(3, 7)) if layers is None else layers
    cps = np.sort(rng.uniform(1800.0, 4500.0, n))
    return {"kind": 1, "nlayers": n, "cp": [float(v) for v in cps],
            "cs_ratio": [float(v) for v in rng.uniform(1.6, 2.0, n)],
            "depth": [float(v) for v in np.sort(rng.uniform(0.15, 0.9, n - 1)) * nz] + [1e9],
            "dome_amp": float(rng.uniform(0.05, 0.2)) * nz, "dome_sigma": float(rng.uniform(0.15, 0.35)) * min(nx, ny),
            "dome_xc": (nx - 1) / 2.0, "dome_yc": (ny - 1) / 2.0, "rho_coef": 310.0, "rho_pow": 0.25,
            "perturb": perturb, "seed": seed}


def _lsr(z, n):
    """Logical right shift of int64 tensors."""
    return (z >> n) & ((1 << (64 - n)) - 1)


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def _hash_uniform(seed, cell, stream):
    """SplitMix64 of (seed, cell) as a uniform in [0, 1), the noise of the device generator."""
    z = (cell * 2 + (stream + 1)) * _i64(0x9E3779B97F4A7C15) + _i64(seed)
    z = (z ^ _lsr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _lsr(z, 27)) * _i64(0x94D049BB133111EB)
    z = z ^ _lsr(z, 31)
    return _lsr(z, 11).double() / 9007199254740992.0


def _dome_model(spec, nx, ny, nz):
    """The dome as float32 tensors on the GPU, [nz, ny, nx]."""
    x = torch.arange(nx, dtype=torch.float64, device="cuda")[None, None, :]
    y = torch.arange(ny, dtype=torch.float64, device="cuda")[None, :, None]
    k = torch.arange(nz, dtype=torch.float64, device="cuda")[:, None, None]
    r2 = (x - spec["dome_xc"]) ** 2 + (y - spec["dome_yc"]) ** 2
    dome = spec["dome_amp"] * torch.exp(-r2 / (2.0 * spec["dome_sigma"] ** 2))
    layer = torch.zeros((nz, ny, nx), dtype=torch.int64, device="cuda")
    for d in spec["depth"]:
        layer += k >= d - dome
    layer.clamp_(max=spec["nlayers"] - 1)
    cpl = torch.tensor(spec["cp"], dtype=torch.float64, device="cuda")
    ratio = torch.tensor(spec["cs_ratio"], dtype=torch.float64, device="cuda")
    cp, cs, rho = cpl[layer], (cpl / ratio)[layer], (spec["rho_coef"] * cpl ** spec["rho_pow"])[layer]
    if spec["perturb"] > 0:
        cell = torch.arange(nx * ny * nz, device="cuda").reshape(nz, ny, nx)
        cp = cp * (1.0 + spec["perturb"] * (2.0 * _hash_uniform(spec["seed"], cell, 0) - 1.0))
        rho = rho * (1.0 + spec["perturb"] * (2.0 * _hash_uniform(spec["seed"], cell, 1) - 1.0))
    return cp.float(), cs.float(), rho.float()


def _matlab_model(nx, ny, nz):
    """The five-medium anticline at any size (depths scale with nz / 201)."""
    sc = nz / 201.0
    X = torch.linspace(0.0, math.pi, nx, dtype=torch.float64, device="cuda")[None, None, :]
    Y = torch.linspace(0.0, math.pi, ny, dtype=torch.float64, device="cuda")[None, :, None]
    Z = (((torch.sin(X) + torch.sin(Y)) / 2.0 - 0.5) / 0.5).clamp(min=0.0)
    k = torch.arange(1, nz + 1, dtype=torch.float64, device="cuda")[:, None, None]
    m = torch.ones((nz, ny, nx), dtype=torch.int64, device="cuda")
    m[(k > 121 * sc - 100 * sc * Z)] = 2
    third = k > 161 * sc - 100 * sc * Z
    m[third] = 3
    m[third & (k < 80 * sc)] = 4
    m[k > 201 * sc - 100 * sc * Z] = 5
    media = torch.tensor([[0, 0, 0], [3000, 1700, 2800], [3600, 1400, 2300], [3000, 1700, 2800],
                          [3600, 1700, 2800], [3650, 1500, 2450]], dtype=torch.float32, device="cuda")
    return media[:, 0][m], media[:, 1][m], media[:, 2][m]


def _line(xs, nx, y, z):
    """Receivers along x through (xs, y, z), at most 201 and inside the grid."""
    n = min(201, nx)
    x0 = min(max(xs - n // 2, 0), nx - n)
    x = np.arange(x0, x0 + n, dtype=np.int32)
    return np.stack([x, np.full_like(x, y), np.full_like(x, z)], axis=1)


def _shot_inputs(case, seed):
    """(ShotParams, model kind, spec or tensors) of one shot case."""
    rng = np.random.default_rng(seed)
    nx, ny, nz, npml = case["nx"], case["ny"], case["nz"], case["npml"]
    spec = None
    if case["model"] == "homogeneous":
        cp = float(np.float32(3300.0 * (1.0 + 0.02 * rng.uniform(-1, 1))))
        model = tuple(torch.full((nz, ny, nx), v, dtype=torch.float32, device="cuda")
                      for v in (cp, cp / 1.732, 2800.0))
        cmax = cp
    elif case["model"] == "matlab":
        model, cmax = _matlab_model(nx, ny, nz), 3650.0
    else:
        spec = _dome_spec(rng, nx, ny, nz, seed)
        model = None if case["model"] == "device" else _dome_model(spec, nx, ny, nz)
        cmax = max(spec["cp"]) * 1.02
    # half the CFL limit; the source's period spans the first third of the run
    dt = 0.5 * 10.0 / (cmax * math.sqrt(3.0))
    f0 = min(35.0, max(8.0, 3.0 / (case["steps"] * dt)))
    sx = int(rng.integers(npml + 2, nx - npml - 2))
    sy = int(rng.integers(npml + 2, ny - npml - 2))
    sz = min(npml + 3, nz - 2)
    p = ela.ShotParams(
        nx=nx, ny=ny, nz=nz, nstep=case["steps"], dx=10.0, dy=10.0, dz=10.0, dt=dt, npml=npml,
        pml_mode=ela.PML_CLEAN if case["clean"] else ela.PML_COMPAT, f0=f0, t0=1.2 / f0, factor=1e7,
        stf=GAUSS_DERIV if case["explosive"] else RICKER,
        src_kind=ela.SRC_EXPLOSIVE if case["explosive"] else ela.SRC_FORCE, src=(sx, sy, sz),
        angle_force=30.0 if case["explosive"] else 0.0, sampgat=case["sampgat"], rec=_line(sx, nx, sy, sz),
        precision=ela.FP64 if case["fp64"] else ela.FP32, it_output=case["snap_every"],
        energy_every=case["energy_every"])
    return p, model, spec


def _many_grids(case):
    """[(nx, ny, nz, npml, steps)] of a batch or a burst of requests."""
    rng = np.random.default_rng(case["grids"])
    out = []
    for _ in range(case["shots"] if case["kind"] == "batch" else case["requests"]):
        if case["kind"] == "serve":
            n = [int(min(max(round(rng.lognormal(math.log(128.0), 0.45)), case["lo"]), case["hi"])) for _ in range(3)]
        elif case["shared"]:
            n = [case["lo"]] * 3
        else:
            n = [16 * int(rng.integers(case["lo"] // 16, case["hi"] // 16 + 1)) for _ in range(3)]
        npml = case.get("npml") or min(int(rng.integers(10, 21)), (min(n) - 10) // 2)
        # shots of other sizes run for other numbers of steps
        steps = case["steps"] if case.get("shared") else int(case["steps"] * rng.uniform(0.8, 1.2))
        out.append((*n, npml, steps))
    return out


def _many_inputs(case, seed):
    """[(ShotParams, model tensors)] of a batch or a burst of requests."""
    rng = np.random.default_rng(seed)
    out, model = [], None
    for i, (nx, ny, nz, npml, steps) in enumerate(_many_grids(case)):
        if model is None or not case.get("shared"):
            spec = _dome_spec(rng, nx, ny, nz, seed + i)
            model, cmax = _dome_model(spec, nx, ny, nz), max(spec["cp"]) * 1.02
        dt = 0.5 * 10.0 / (cmax * math.sqrt(3.0))
        f0 = min(35.0, max(8.0, 3.0 / (steps * dt)))
        sx = int(rng.integers(npml + 2, nx - npml - 2))
        sy = int(rng.integers(npml + 2, ny - npml - 2))
        p = ela.ShotParams(nx=nx, ny=ny, nz=nz, nstep=steps, dt=dt, npml=npml, f0=f0, t0=1.2 / f0,
                           src=(sx, sy, npml + 3), rec=_line(sx, nx, sy, npml + 3))
        out.append((p, model))
    return out


def _host(model):
    """Page-locked numpy copies of the model tensors."""
    out = []
    for t in model:
        a = ela.pinned_empty(tuple(t.shape))
        torch.from_numpy(a).copy_(t)
        out.append(a)
    return out


def prepare(case, seed):
    if case["kind"] == "shot":
        p, model, spec = _shot_inputs(case, seed)
        device_model = case["model"] == "device"
        return {"case": case, "p": p, "spec": spec if device_model else None,
                "model": None if device_model else _host(model)}
    shots, seen = [], {}
    for p, model in _many_inputs(case, seed):
        if id(model) not in seen:
            seen[id(model)] = (model, _host(model))
        shots.append((p, *seen[id(model)][1]))
    state = {"case": case, "shots": shots}
    if case["kind"] == "serve":
        state["server"] = ela.Server(hbm_budget_bytes=16 << 30)
    return state


# ------------------------------------------------------------------- run --
def _last(case):
    """Velocity components a shot returns after its last step: none, vz, or all."""
    return {0: (), 1: (ela.VZ,), 3: (ela.VX, ela.VY, ela.VZ)}[case["snap_last"]]


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        with ela.Batch(state["shots"]) as b:
            b.run(max(p.nstep for p, *_ in state["shots"]))
            return [b.seismograms(i) for i in range(len(state["shots"]))]
    if case["kind"] == "serve":
        srv = state["server"]
        tickets = [srv.submit(*s) for s in state["shots"]]
        out = []
        for t in tickets:
            srv.wait(t)
            out.append(srv.read(t))
            srv.release(t)
        return out
    p = state["p"]
    plan = ela.Plan.from_model(p, state["spec"]) if state["spec"] else ela.Plan(p, *state["model"])
    with plan:
        out, fp64 = [], case["fp64"]
        if case["snap_every"]:
            for _ in range(p.nstep // case["snap_every"]):
                plan.run(case["snap_every"])
                out.append(plan.field(ela.VZ, fp64=fp64))
            plan.run(p.nstep % case["snap_every"])
        else:
            plan.run(p.nstep)
        out.append(plan.seismograms(fp64=fp64))
        out.append(plan.source_trace(fp64=fp64))
        out.extend(plan.field(c, fp64=fp64) for c in _last(case))
        if case["energy_every"]:
            out.append(plan.energy())
    return out


# ------------------------------------------------------------------ work --
def _shot_work(nx, ny, nz, npml, steps, word):
    """A time step streams the nine fields and the C-PML memory variables (12
    per direction of a cell inside a layer: read and written) once, and reads
    the model; about 130 operations a cell and 10 a layer direction."""
    cells = nx * ny * nz
    pml = sum(min(1.0, 2.0 * npml / n) for n in (nx, ny, nz))
    return np.array([cells * steps * word * (2 * 9 + 3 + 12 * pml), cells * steps * (130.0 + 30.0 * pml)])


def work(case):
    if case["kind"] == "shot":
        w = _shot_work(case["nx"], case["ny"], case["nz"], case["npml"], case["steps"], 8 if case["fp64"] else 4)
    else:
        w = sum(_shot_work(*g, 4) for g in _many_grids(case))
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ----------------------------------------------------------------- exact --
def _profiles(p):
    """Per axis (a, b, 1/K, a_half, b_half, 1/K_half) in float64."""
    out = []
    compat = p.pml_mode == ela.PML_COMPAT
    amax = math.pi * p.f0 if p.alpha_max < 0 else p.alpha_max
    for axis, (n, d) in enumerate(((p.nx, p.dx), (p.ny, p.dy), (p.nz, p.dz))):
        thick = p.npml * d
        norm = p.npml * p.dy if compat and axis == 2 else thick
        d0 = -(p.npower + 1.0) * p.vpml * math.log(p.rcoef) / (2.0 * thick)
        omax = (n - 1) * d - thick
        prof = np.zeros((6, n))
        for i in range(n):
            for half in (0, 1):
                D, K, al = 0.0, 1.0, 0.0
                pos = d * i + (d / 2.0 if half else 0.0)
                lo = thick - pos
                if compat and axis == 2 and half:
                    lo = p.npml * p.dy - (p.dy * (p.ny - 1) + p.dy / 2.0)
                top = thick if compat and axis == 2 and not half else norm
                for depth, nrm in ((lo, norm), (pos - omax, top)):
                    if depth >= 0.0:
                        x = depth / nrm
                        D = d0 * x ** p.npower
                        K = 1.0 + (p.k_max - 1.0) * x ** p.npower
                        al = amax * (1.0 - x) + 0.1 * amax
                if not compat or axis == 0:
                    al = max(al, 0.0)
                b = math.exp(-(D / K + al) * p.dt)
                a = D * (b - 1.0) / (K * (D + K * al)) if abs(D) > 1e-6 else 0.0
                if compat and axis == 0 and half:
                    a = 0.0
                prof[3 * half:3 * half + 3, i] = (a, b, 1.0 / K)
        out.append(torch.tensor(prof, device="cuda"))
    return out


def _source(p, it):
    a = math.pi ** 2 * p.f0 ** 2
    tau = (it - 1) * p.dt - p.t0
    g = math.exp(-a * tau * tau)
    if p.stf == GAUSS_DERIV:
        return -p.factor * 2.0 * a * tau * g
    return p.factor * (1.0 - 2.0 * a * tau * tau) * g


class _Layers:
    """Memory variables of one derivative: only the cells at both ends of its axis carry any."""

    def __init__(self, p, axis, half, shape, prof):
        dim = 2 - axis
        w, n = p.npml + 1, shape[dim]
        self.parts = []
        for lo in (0, n - w):
            s = list(shape)
            s[dim] = w
            view = [1, 1, 1]
            view[dim] = w
            coef = [prof[axis][3 * half + q, lo:lo + w].reshape(view) for q in range(3)]
            self.parts.append((dim, lo, w, coef, torch.zeros(s, dtype=torch.float64, device="cuda")))

    def apply(self, d):
        for dim, lo, w, (a, b, ik), psi in self.parts:
            s = d.narrow(dim, lo, w)
            psi.mul_(b).addcmul_(a.expand_as(s), s)
            s.mul_(ik).add_(psi)
        return d


def _simulate(p, model, steps, snaps):
    """The time loop in float64; returns (seismograms, source trace, fields
    after the steps in `snaps`, the nine final fields)."""
    cp, cs, rho = (t.double() for t in model)
    shape = cp.shape
    prof = _profiles(p)

    def shifted(t, dim, by):
        """t at index + by, zero outside the grid."""
        n, out = t.shape[dim], torch.zeros_like(t)
        if by > 0:
            out.narrow(dim, 0, n - 1).copy_(t.narrow(dim, 1, n - 1))
        else:
            out.narrow(dim, 1, n - 1).copy_(t.narrow(dim, 0, n - 1))
        return out

    Z, Y, X = 0, 1, 2
    up = {X: 1.0 / p.dx, Y: 1.0 / p.dy, Z: 1.0 / p.dz}

    def mean_mu(d1, by1, d2, by2):
        s = (shifted(cs, d1, by1) + shifted(cs, d2, by2)) / 2.0
        return (shifted(rho, d1, by1) + shifted(rho, d2, by2)) / 2.0 * s * s * p.dt

    l2m = rho * cp * cp * p.dt
    lam = l2m - 2.0 * rho * cs * cs * p.dt
    mu_xy, mu_xz, mu_yz = mean_mu(X, -1, Y, 1), mean_mu(X, -1, Z, 1), mean_mu(Y, 1, Z, 1)
    buoy = [p.dt / ((rho + shifted(rho, d, by)) / 2.0) for d, by in ((X, -1), (Y, 1), (Z, 1))]

    def region(x, y, z):
        """0/1 mask of the cells an update covers, as one factor per axis."""
        m = torch.ones(shape, dtype=torch.float64, device="cuda")
        for dim, (lo, hi), n in ((X, x, p.nx), (Y, y, p.ny), (Z, z, p.nz)):
            m.narrow(dim, 0, lo).zero_()
            m.narrow(dim, n - hi, hi).zero_()
        return m

    normal = region((0, 1), (1, 0), (1, 0))
    l2m *= normal
    lam *= normal
    del normal
    mu_xy *= region((1, 0), (0, 1), (0, 0))
    mu_xz *= region((1, 0), (0, 0), (0, 0))
    mu_yz *= region((0, 0), (0, 1), (0, 0))
    for b, r in zip(buoy, (((1, 0), (1, 0), (1, 0)), ((0, 1), (0, 1), (1, 0)), ((0, 1), (1, 0), (0, 1)))):
        b *= region(*r)
    vx, vy, vz, sxx, syy, szz, sxy, sxz, syz = (torch.zeros(shape, dtype=torch.float64, device="cuda")
                                                for _ in range(9))
    # (axis, half node) of the nine derivatives of each half-step
    mem = {}

    def diff(t, dim, by, key):
        d = torch.zeros_like(t)
        n = t.shape[dim]
        hi, lo = t.narrow(dim, 1, n - 1), t.narrow(dim, 0, n - 1)
        if by > 0:   # t[i+1] - t[i]: half nodes; beyond the grid the field is zero
            torch.sub(hi, lo, out=d.narrow(dim, 0, n - 1))
            d.narrow(dim, n - 1, 1).sub_(t.narrow(dim, n - 1, 1))
        else:
            torch.sub(hi, lo, out=d.narrow(dim, 1, n - 1))
            d.narrow(dim, 0, 1).add_(t.narrow(dim, 0, 1))
        d *= up[dim]
        if key not in mem:
            mem[key] = _Layers(p, 2 - dim, 1 if by > 0 else 0, shape, prof)
        return mem[key].apply(d)

    rec = torch.tensor(np.asarray(p.rec), dtype=torch.int64, device="cuda")
    nsamp = p.nstep // p.sampgat
    seis = torch.zeros((rec.shape[0], 3, nsamp), dtype=torch.float64, device="cuda")
    trace = torch.zeros((3, p.nstep + 1), dtype=torch.float64, device="cuda")
    sx, sy, sz = p.src
    at = (sz, sy, sx)
    taken = []
    ang = p.angle_force * math.pi / 180.0
    # (only vz is forced: rho averaged as in its update, zero above the last plane)
    r0, r1 = float(rho[at]), float(rho[sz + 1, sy, sx]) if sz + 1 < p.nz else 0.0
    force_scale = p.dt / ((r0 + r1) / 2.0)
    expl_scale = p.dt * float(rho[at] * cp[at] * cp[at])
    for it in range(1, steps + 1):
        ex, ey, ez = diff(vx, X, 1, "exx"), diff(vy, Y, -1, "eyy"), diff(vz, Z, -1, "ezz")
        sxx.addcmul_(l2m, ex).addcmul_(lam, ey + ez)
        syy.addcmul_(lam, ex + ez).addcmul_(l2m, ey)
        szz.addcmul_(lam, ex + ey).addcmul_(l2m, ez)
        sxy.addcmul_(mu_xy, diff(vy, X, -1, "yx").add_(diff(vx, Y, 1, "xy")))
        sxz.addcmul_(mu_xz, diff(vz, X, -1, "zx").add_(diff(vx, Z, 1, "xz")))
        syz.addcmul_(mu_yz, diff(vz, Y, 1, "zy").add_(diff(vy, Z, 1, "yz")))
        vx.addcmul_(buoy[0], diff(sxx, X, -1, "sxx").add_(diff(sxy, Y, -1, "sxy_y")).add_(diff(sxz, Z, -1, "sxz_z")))
        vy.addcmul_(buoy[1], diff(sxy, X, 1, "sxy_x").add_(diff(syy, Y, 1, "syy")).add_(diff(syz, Z, -1, "syz_z")))
        vz.addcmul_(buoy[2], diff(sxz, X, 1, "sxz_x").add_(diff(syz, Y, -1, "syz_y")).add_(diff(szz, Z, 1, "szz")))
        if it % p.sampgat == 0 and it // p.sampgat <= nsamp:
            q = it // p.sampgat - 1
            for c, v in enumerate((vx, vy, vz)):
                seis[:, c, q] = v[rec[:, 2], rec[:, 1], rec[:, 0]]
        s = _source(p, it)
        if p.src_kind == ela.SRC_EXPLOSIVE:
            for c, (f, w) in enumerate(((sxx, math.sin(ang)), (syy, math.sin(ang)), (szz, math.cos(ang)))):
                f[at] += w * s * expl_scale
                trace[c, it] = f[at]
        else:
            vz[at] += s * force_scale
            for c, f in enumerate((vx, vy, vz)):
                trace[c, it] = f[at]
        if it in snaps:
            taken.append(vz.clone())
    return seis, trace, taken, (vx, vy, vz, sxx, syy, szz, sxy, sxz, syz), (cp, cs, rho)


def _energy(p, fields, model):
    vx, vy, vz, sxx, syy, szz, sxy, sxz, syz = fields
    cp, cs, rho = model
    mu = rho * cs * cs
    lam = rho * cp * cp - 2.0 * mu
    e = 0.5 * rho * (vx * vx + vy * vy + vz * vz)
    tr = sxx + syy + szz
    ss = sxx * sxx + syy * syy + szz * szz + 2.0 * (sxy * sxy + sxz * sxz + syz * syz)
    e = e + ss / (4.0 * mu) - lam / (4.0 * mu * (3.0 * lam + 2.0 * mu)) * tr * tr
    return float(e.sum()) * p.dx * p.dy * p.dz


def exact(case, seed):
    if case["kind"] != "shot":
        return [_simulate(p, model, p.nstep, ())[0].cpu().numpy() for p, model in _many_inputs(case, seed)]
    p, model, spec = _shot_inputs(case, seed)
    if model is None:
        model = _dome_model(spec, p.nx, p.ny, p.nz)
    every = case["snap_every"]
    snaps = set(range(every, p.nstep + 1, every)) if every else ()
    seis, trace, taken, fields, dmodel = _simulate(p, model, p.nstep, snaps)
    out = [t.cpu().numpy() for t in taken] + [seis.cpu().numpy(), trace.cpu().numpy()]
    out.extend(fields[c].cpu().numpy() for c in _last(case))
    if case["energy_every"]:
        out.append(_energy(p, fields, dmodel))
    return out

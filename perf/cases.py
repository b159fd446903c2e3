"""Performance cases: the work a user of this framework has it do.

A case is a plain dict; ``prepare`` writes its run directory (seeded terrain,
medium and sources), creates the session and gives it a developed wavefield,
``run`` is one pass through the public entry points, ``exact`` is the same
run in FP64 written in plain torch.  Kinds:

* ``cg``        CGFDM (MacCormack + RK4, PML) time steps, FP32 storage
* ``cg16``      the same with FP16-delta storage
* ``sc``        ME-AWENO (WENO5 + TVD-RK3, sponge) time steps
* ``batch``     several CGFDM shots of uneven sizes advanced together
* ``gradient``  seismogram misfit and its gradient through the adjoint
* ``whole``     a complete run: directory on disk -> traces on the host

A pass of the stepping kinds goes on from where the last one stopped, as a
run does between two looks at its traces; ``room`` is how many passes a
session has steps for.
"""

from __future__ import annotations

import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(ROOT, "cgfdm3d-eqr-sc_b200"), os.path.join(os.getcwd(), "cgfdm3d-eqr-sc_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

from cgfdm import Batch, Session, autograd, cases, configs  # noqa: E402

H = 3            # halo cells on each side


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest models: a parity or teaching grid, where launches and latency count
        dict(name="cg_small", kind="cg", nx=64, ny=60, nz=48, nPML=8, hills=True, source="couple", steps=96,
             room=400, stations=8, field=False),
        # the homogeneous half-space of the framework's CPU-runnable configuration, with a look at the whole field
        dict(name="cg_halfspace", kind="cg", nx=128, ny=128, nz=96, nPML=12, hills=False, source="couple", steps=192,
             room=60, stations=16, field=True),
        # a site model of no convenient size: ragged tiles in every direction
        dict(name="cg_ragged", kind="cg", nx=213, ny=151, nz=117, nPML=10, hills=True, source="ricker", steps=48,
             room=120, stations=32, field=False),
        # the headline workload: curvilinear terrain, finite fault, 400 stations
        dict(name="cg_terrain_fault", kind="cg", nx=400, ny=400, nz=200, nPML=12, hills=True, source="fault",
             steps=24, room=60, stations=400, field=False),
        # FP16-delta storage, the option for models that do not fit otherwise
        dict(name="cg_fp16", kind="cg16", nx=192, ny=184, nz=112, nPML=12, hills=True, source="couple", steps=24,
             room=120, stations=32, field=False),
        # a shot catalogue: twelve models of uneven sizes in one launch per stage
        dict(name="cg_batch", kind="batch", shots=12, low=64, high=256, sizes=5, nPML=12, steps=16, room=60,
             stations=32),
        # full-waveform inversion: one shot's misfit and gradient for new medium parameters
        dict(name="cg_gradient", kind="gradient", nx=144, ny=136, nz=104, nPML=12, hills=True, source="ricker",
             steps=64, every=22, stations=48),
        # the ME-AWENO scheme: a small model
        dict(name="sc_small", kind="sc", nx=72, ny=64, nz=56, hills=True, source="couple", steps=48, room=200,
             stations=8, field=True),
        # a ragged basin model
        dict(name="sc_ragged", kind="sc", nx=181, ny=203, nz=97, hills=True, source="ricker", steps=16, room=120,
             stations=32, field=False),
        # the basin workload at the depth and aspect of its configuration
        dict(name="sc_basin", kind="sc", nx=384, ny=384, nz=192, hills=True, source="ricker", steps=8, room=60,
             stations=100, field=False),
        # the program a user of the reference runs: directory in, traces and peak velocities out
        dict(name="cg_whole_run", kind="whole", nx=160, ny=152, nz=100, nPML=12, hills=True, source="fault",
             steps=256, stations=64),
    ]


def draw(rng):
    """One more case of the same ranges: sizes log-uniform and mostly odd, cost no more than the largest listed."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cg", "cg", "cg", "sc", "sc", "cg16", "batch", "gradient", "whole"])
    if kind == "batch":
        return dict(kind=kind, shots=rng.randint(3, 12), low=64, high=rng.randint(120, 256), sizes=rng.randint(0, 999),
                    nPML=12, steps=8 * rng.randint(1, 2), room=60, stations=rng.randint(8, 32))
    top = {"cg": (400, 200), "sc": (320, 192), "cg16": (260, 128), "gradient": (144, 104), "whole": (200, 120)}[kind]
    c = dict(kind=kind, nx=size(60, top[0]), ny=size(60, top[0]), nz=size(48, top[1]), hills=rng.random() < 0.8,
             source=rng.choice(["couple", "ricker", "fault"]), stations=rng.randint(8, 64))
    points = c["nx"] * c["ny"] * c["nz"]
    if kind != "sc":
        c["nPML"] = rng.randint(6, 14)
    if kind == "gradient":
        c.update(source=rng.choice(["couple", "ricker"]), steps=rng.randint(48, 64), every=rng.randint(16, 48))
    elif kind == "whole":
        c.update(steps=rng.randint(128, 256))
    else:
        n = 8 if kind == "sc" else 24
        n = max(n, min(96, int(n * 4e6 / points))) // 8 * 8 + rng.choice([0, 0, 3])
        c.update(steps=n, room=max(60, min(400, int(3e9 / (points * n)))), field=points < 4e5 and rng.random() < 0.5)
    return c


def work(case):
    """Bytes: per point and step the state read and written and the 12 metric and medium fields read, per
    absorbing-layer point the auxiliary state read and written.  Flops: the scheme's arithmetic."""
    if case["kind"] == "batch":
        return {k: sum(work(c)[k] for c in _shots(case)) for k in ("bytes", "flops")}
    n = float(case["nx"] * case["ny"] * case["nz"])
    s = case["steps"]
    if case["kind"] == "sc":
        return {"bytes": 4.0 * (9 + 13 + 9) * n * s, "flops": 19.4e3 * n * s}
    p = case["nPML"]
    faces = p * (2.0 * case["ny"] * case["nz"] + 2.0 * case["nx"] * case["nz"] + case["nx"] * case["ny"])
    w = {"bytes": 4.0 * (30 * n + 18 * faces) * s, "flops": 2.2e3 * n * s}
    # the gradient: the forward run and the transposed steps, which also read the forward's right-hand sides
    return {"bytes": 3 * w["bytes"], "flops": 2.5 * w["flops"]} if case["kind"] == "gradient" else w


def tolerance(case):
    """About four times what the separately rounded build of the library differs by from the default one."""
    fp32 = {"rel": 3e-6, "max": 1e-4}
    return {"cg": fp32, "batch": fp32, "whole": fp32, "gradient": {"rel": 4e-6, "max": 4e-4},
            "cg16": {"rel": 3e-4, "max": 1e-2}, "sc": {"rel": 1.2e-5, "max": 2e-3}}[case["kind"]]


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _shots(case):
    """The shots of a batch: uneven sizes from the case's own numbers."""
    r = random.Random(case["sizes"])
    lo, hi = case["low"], case["high"]
    return [dict(kind="cg", nx=r.randint(lo, hi), ny=r.randint(lo, hi), nz=r.randint(lo, max(lo, hi // 2)),
                 nPML=case["nPML"], hills=r.random() < 0.8, source="couple", steps=case["steps"], room=case["room"],
                 stations=case["stations"], field=False) for _ in range(case["shots"])]


def _total_steps(case):
    return case["steps"] * case.get("room", 1) + (PRERUN if case["kind"] == "cg16" else 0)


PRERUN = 128     # FP16 storage starts from rest: steps before the first pass


def _terrain(case, rng):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if not case["hills"]:
        return None
    t = configs.gaussian_hills(nx, ny, DH, rng, hrange=(50.0, 0.05 * nz * DH), wrange=(1500.0, 6000.0))
    return t


DH = 100.0


def _z(case, terrain):
    """Heights of the padded grid's points, float32, by the library's terrain-following (or flat) convention."""
    nz = case["nz"]
    K = (np.arange(nz + 2 * H) - H).astype(np.float32)
    if terrain is None:
        z = (K + np.float32(1)) * np.float32(DH) - np.float32(nz * DH)
        return np.broadcast_to(z[:, None, None], (nz + 2 * H, case["ny"] + 2 * H, case["nx"] + 2 * H))
    return configs._coords_z(terrain, nz, DH)


def _waves(shape, fields, rng, dev, short=9.0, long=40.0, n=5):
    """A sum of n plane waves per field, wavelengths short..long cells, float32 [fields] + shape, of unit variance."""
    z, y, x = (torch.arange(s, device=dev, dtype=torch.float32) for s in shape)
    out = torch.zeros((fields,) + shape, device=dev)
    for _ in range(n):
        v = rng.standard_normal(3)
        k = v / np.linalg.norm(v) * 2 * math.pi / rng.uniform(short, long)
        ph = (z * float(k[0]))[:, None, None] + (y * float(k[1]))[None, :, None] + (x * float(k[2]))[None, None, :]
        c, s = torch.cos(ph), torch.sin(ph)
        for f in range(fields):
            a, b = rng.standard_normal(2) / math.sqrt(n)
            out[f] += float(a) * c + float(b) * s
    return out


def _medium(case, z, rng, dev):
    """(Vs, Vp, rho) [nzp][nyp][nxp][3]: layers by depth with smooth +-3 % perturbations, Vp 4500 -> 7000 m/s
    (a low-velocity top layer of 2600 m/s for the ME-AWENO models), Vs = Vp / 1.73, Gardner density."""
    zt = torch.tensor(np.ascontiguousarray(z), device=dev)
    depth = zt[-H - 1].max() - zt
    total = case["nz"] * DH
    vp = torch.full_like(zt, 7000.0)
    tops = np.sort(rng.uniform(0.1, 0.9, 3)) * total
    for d, v in zip(reversed(tops), (6200.0, 5400.0, 2600.0 if case["kind"] == "sc" else 4500.0)):
        vp = torch.where(depth < float(d), torch.full_like(vp, v), vp)
    vp = vp * (1.0 + 0.03 * torch.tanh(_waves(tuple(zt.shape), 1, rng, dev)[0]))
    return torch.stack([vp / 1.73, vp, 310.0 * vp.pow(0.25)], -1)


def _field(case, med, rng, dev):
    """A developed wavefield [nzp][nyp][nxp][9] fading out in the absorbing layers: velocities of about 0.05 m/s and
    the stresses that go with them (for ME-AWENO momentum and strain)."""
    shape = tuple(med.shape[:3])
    w = _waves(shape, 9, rng, dev)
    if case["kind"] == "sc":
        w[:3] *= 0.05 * 2700.0
        w[3:] *= 0.05 / 5000.0
    else:
        w[:3] *= 0.05
        w[3:] *= 0.05 * 2700.0 * 5000.0
    edge = case.get("nPML", 20)
    for ax, n in enumerate(shape):
        i = torch.arange(n, device=dev, dtype=torch.float32)
        low = (i - H + 1).clamp(min=0)
        d = low if ax == 0 else torch.minimum(low, (n - H - i).clamp(min=0))
        t = torch.sin((d / (edge + 4.0)).clamp(max=1.0) * (math.pi / 2)) ** 2
        if ax == 0 and case["kind"] != "sc":
            t[n - H:] = 0        # the CGFDM halo above the surface is never written
        w *= t.view([1] + [-1 if a == ax else 1 for a in range(3)])
    return w.permute(1, 2, 3, 0).contiguous()


def _fault(case, z, rng, dt):
    """Sub-faults of a planar rupture around the middle of the model, at cell centres: (points for the source file,
    their cells and parameters)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    total = _total_steps(case)
    nt = int(math.ceil((total + 2) * dt / 0.02)) + 4
    t = np.arange(nt) * 0.02
    nl, nw = max(4, nx // 10), max(4, nz // 10)
    pts, cells = [], []
    for a in range(nl):
        for b in range(nw):
            i, j = nx // 2 + 2 * (a - nl // 2), ny // 2 + (a - nl // 2)
            k = nz - 6 - 2 * b
            # the cell of x is the integer part of x / DH + 1/2, cut towards zero
            x, y = (v if v >= 0 else v - 1 for v in (i - nx // 2, j - ny // 2))
            lon, lat = cases.aeqd_inv(100.0, 30.0, x * DH, y * DH)
            dz = float(z[H + 1, H + j, H + i]) - float(z[H, H + j, H + i])
            tr = 0.004 * math.hypot(a - nl / 2, b - nw / 2)
            rise = 0.4
            rate = (rng.uniform(0.5, 1.5) * 0.004 * np.clip(1 - np.abs(t - tr - rise / 2) / (rise / 2), 0, None)
                    * 2 / rise).astype(np.float32)
            rake = float(rng.uniform(60, 120))
            pts.append(cases.FaultPoint(lon, lat, -(nz - 1 - k) * dz, 4e4, 30.0, 60.0, np.full(nt, rake, np.float32),
                                        rate))
            # a flat grid's surface lies one cell above where its depths are measured from
            cells.append((i, j, k if case["hills"] else k - 1))
    pts.append(cases.FaultPoint(100.0, 30.0, 0.0, 1.0, 30.0, 60.0, np.zeros(nt, np.float32),
                                np.zeros(nt, np.float32)))
    return pts, cells, nt


def _inputs(case, seed):
    """All a run directory needs, from the seed alone."""
    rng = np.random.default_rng([int(seed), 17])
    dev = _device()
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    terrain = _terrain(case, rng)
    z = _z(case, terrain)
    med = _medium(case, z, rng, dev)
    vp_max = float(med[..., 1].max())
    dt = float(np.float32(cases.cfl_dt(DH, vp_max, 0.4)))
    pos = (int(rng.integers(nx // 3, 2 * nx // 3)), int(rng.integers(ny // 3, 2 * ny // 3)),
           nz - 1 - int(rng.integers(8, 16)))
    # stations at the surface and in boreholes; near the source where the run starts from rest
    e = 4
    lo, hi = [e, e, e], [nx - e, ny - e, nz - e]
    if case["kind"] not in ("cg", "sc"):
        at = (nx // 2, ny // 2) if case["source"] == "fault" else pos
        for a in range(2):
            lo[a], hi[a] = max(e, at[a] - 20), min(hi[a], at[a] + 20)
        lo[2] = nz - 30
    st = [(int(rng.integers(lo[0], hi[0])), int(rng.integers(lo[1], hi[1])),
           nz - 1 if n % 2 == 0 else int(rng.integers(lo[2], hi[2]))) for n in range(case["stations"])]
    c = cases.Case(NX=nx, NY=ny, NZ=nz, DH=DH, DT=dt, steps=_total_steps(case), nPML=case.get("nPML", 12), layers=(),
                   stations=st, extra={"mediumFile": "medium.bin", "useMedium": 1})
    if terrain is not None:
        c.extra["terrainFile"] = "terrain.bin"
    cells = None
    if case["source"] == "fault":
        c.fault_dt = 0.02
        c.fault, cells, _ = _fault(case, z, rng, dt)
    elif case["source"] == "couple":
        c.double_couple = dict(X=pos[0], Y=pos[1], Z=pos[2], strike=float(rng.uniform(0, 360)),
                               dip=float(rng.uniform(20, 90)), rake=float(rng.uniform(-180, 180)), Mw=8.0,
                               duration=0.5)
    else:
        c.ricker_point = pos + (2.0,)
    return dict(case=c, terrain=terrain, z=z, med=med, dt=dt, pos=pos, cells=cells, rng=rng, dev=dev)


def _write(case, inp, directory):
    cases.write_case(inp["case"], directory, scheme="SCFDM" if case["kind"] == "sc" else "CGFDM")
    inp["med"].cpu().numpy().tofile(os.path.join(directory, "medium.bin"))
    if inp["terrain"] is not None:
        inp["terrain"].tofile(os.path.join(directory, "terrain.bin"))


def _session(case, seed):
    inp = _inputs(case, seed)
    with tempfile.TemporaryDirectory() as d:
        _write(case, inp, d)
        s = Session(d, options='{"storage": "fp16"}' if case["kind"] == "cg16" else None)
    if case["kind"] == "cg16":
        s.run(PRERUN)
    elif case["kind"] in ("cg", "sc"):
        s.set_wavefield(_field(case, inp["med"], inp["rng"], inp["dev"]).cpu().numpy())
    return s, inp


def _observed(case, rng, dt):
    """Recorded traces to fit: a wavelet per station and component."""
    t = np.arange(case["steps"]) * dt
    obs = np.zeros((case["stations"], case["steps"], 3), np.float32)
    for s in range(case["stations"]):
        for c in range(3):
            obs[s, :, c] = rng.standard_normal() * cases.ricker(t, rng.uniform(3, 6), rng.uniform(0.3, 0.9) * t[-1])
    return obs * 1e-9     # the explosive source's moment is 1e9 N m


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ss = [_session(c, seed * 100 + n)[0] for n, c in enumerate(_shots(case))]
        return {"case": case, "sessions": ss, "batch": Batch(ss)}
    if kind == "whole":
        d = tempfile.TemporaryDirectory()
        _write(case, _inputs(case, seed), d.name)
        return {"case": case, "dir": d}
    s, inp = _session(case, seed)
    if kind == "gradient":
        m = [inp["med"][H:-H, H:-H, H:-H, c].contiguous().requires_grad_() for c in (1, 0, 2)]
        return {"case": case, "session": s, "medium": m,
                "observed": torch.from_numpy(_observed(case, inp["rng"], inp["dt"]))}
    return {"case": case, "session": s}


def _products(s, field=False):
    """What a run leaves behind: the traces and the peak ground velocities (and the field)."""
    st = s.stations()
    out = {"velocity": st[:, :, :3], "stress": st[:, :, 3:], "pgv": s.pgv()}
    if field:
        w = s.wavefield()
        out["first"], out["second"] = w[..., :3], w[..., 3:]
    return out


def run(state):
    case = state["case"]
    kind, n = case["kind"], case["steps"]
    if kind == "batch":
        if state["sessions"][0].info.steps_done + n > state["sessions"][0].info.NT:
            raise RuntimeError("the batch has no steps left: more room is needed")
        state["batch"].run(n)
        return [_products(s) for s in state["sessions"]]
    if kind == "whole":
        with Session(state["dir"].name) as s:
            s.run(s.info.NT)
            return _products(s)
    s = state["session"]
    if kind == "gradient":
        vp, vs, rho = state["medium"]
        J = autograd.misfit(vp, vs, rho, s, state["observed"], case["every"])
        g = torch.autograd.grad(J, (vp, vs, rho))
        return {"misfit": J.detach(), "vp": g[0], "vs": g[1], "rho": g[2]}
    if s.info.steps_done + n > s.info.NT:
        raise RuntimeError("the session has no steps left: more room is needed")
    s.run(n)
    return _products(s, case["field"])


# ------------------------------------------------------- the run in FP64
F32 = np.float32
AF = [float(F32(v)) for v in (-0.30874, -0.6326, 1.2330, -0.3334, 0.04168)]
CF = [float(F32(v)) for v in (-1.16666667, 1.33333333, -0.16666667)]
ALPHA = [0.5, 0.5, 1.0]
BETA = [float(F32(v)) for v in (0.16666667, 0.33333333, 0.33333333, 0.16666667)]
SIGNS = [(-1, -1, -1), (1, 1, -1), (1, 1, 1), (-1, -1, 1), (-1, 1, -1), (1, -1, -1), (1, -1, 1), (-1, 1, 1)]
PI32 = float(F32(3.141592657))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_forward(c, seed * 100 + n)[0] for n, c in enumerate(_shots(case))]
    if kind == "gradient":
        return _gradient64(case, seed)
    out, _ = _forward(case, seed)
    return out


def _coords(inp, dev):
    z = torch.tensor(np.ascontiguousarray(inp["z"]), device=dev)
    c = inp["case"]
    ax = []
    for n, centre in ((c.NX, c.NX // 2), (c.NY, c.NY // 2)):
        i = (torch.arange(n + 2 * H, device=dev) - H).float()
        ax.append(i * F32(DH) - float(F32(centre) * F32(DH)))
    x = ax[0][None, None, :].expand_as(z)
    y = ax[1][None, :, None].expand_as(z)
    return x, y, z


def _cut(a, axis, o, low=H, high=H):
    """The interior of a padded array, shifted by o cells along axis (0 x, 1 y, 2 z)."""
    for ax in range(3):
        d, s = 2 - ax, o if ax == axis else 0
        a = a.narrow(d + a.dim() - 3, low + s, a.shape[d + a.dim() - 3] - low - high)
    return a


def _diff(a, axis, fb, scale):
    """One-sided 5-point difference of the interior of a padded array."""
    r = AF[0] * _cut(a, axis, -fb)
    for m in range(1, 5):
        r = r + AF[m] * _cut(a, axis, (m - 1) * fb)
    return r * (fb * scale)


def _metric_cg(inp, dev):
    """The nine metric terms and the Jacobian over the interior, evaluated and rounded in FP32 as the model is."""
    rdh = float(F32(1.0 / DH))
    af = [torch.tensor(v, device=dev, dtype=torch.float32) for v in AF]

    def d(a, axis):
        def one(fb):
            r = af[0] * _cut(a, axis, -fb)
            for m in range(1, 5):
                r = r + af[m] * _cut(a, axis, (m - 1) * fb)
            return (r * fb) * rdh
        return (one(1) + one(-1)) * 0.5

    xyz = _coords(inp, dev)
    (xa, xb, xc), (ya, yb, yc), (za, zb, zc) = [[d(a, ax) for ax in range(3)] for a in xyz]
    jac = xa * yb * zc + xb * yc * za + xc * ya * zb - xc * yb * za - xb * ya * zc - xa * zb * yc
    inv = 1.0 / jac

    def cof(p, q, r, s):
        return ((p * q - r * s) * inv).double()

    m = [cof(yb, zc, yc, zb), cof(xc, zb, xb, zc), cof(xb, yc, xc, yb),
         cof(yc, za, ya, zc), cof(xa, zc, xc, za), cof(xc, ya, xa, yc),
         cof(ya, zb, yb, za), cof(xb, za, xa, zb), cof(xa, yb, xb, ya)]
    return m, jac.double()


def _layers(n, npml, top, dev):
    """(alpha, beta, d) of the absorbing profile along one axis, interior points."""
    L = DH * (npml - 1)
    R = 10.0 ** (-(math.log10(npml) - 1.0) / math.log10(2.0) - 3.0)
    d0 = -3.0 * 6000.0 / (2.0 * L) * math.log(R)
    ls = torch.full((n,), -1.0, dtype=torch.float64, device=dev)
    i = torch.arange(npml, dtype=torch.float64, device=dev) * DH
    ls[:npml] = i.flip(0)
    if top:
        ls[n - npml:] = i
    on = ls >= 0
    al = torch.where(on, PI32 * 0.5 * (1 - ls / L), torch.zeros_like(ls))
    be = torch.where(on, 1 + 2 * (ls / L) ** 2, torch.ones_like(ls))
    d = torch.where(on, d0 * (ls / L) ** 2, torch.zeros_like(ls))
    return al, 1 / be, d / be


def _along(v, axis):
    return v.view([-1 if 2 - axis == d else 1 for d in range(3)])


def _dir_rhs(m, d, mu, lam, buo):
    dv = m[0] * d[0] + m[1] * d[1] + m[2] * d[2]
    return [(m[0] * d[3] + m[1] * d[6] + m[2] * d[7]) * buo, (m[0] * d[6] + m[1] * d[4] + m[2] * d[8]) * buo,
            (m[0] * d[7] + m[1] * d[8] + m[2] * d[5]) * buo] + _dir_stress(m, d, mu, lam, dv)


def _dir_stress(m, d, mu, lam, dv=None):
    dv = m[0] * d[0] + m[1] * d[1] + m[2] * d[2] if dv is None else dv
    return [dv * lam + 2 * mu * m[c] * d[c] for c in range(3)] + [
        (m[1] * d[0] + m[0] * d[1]) * mu, (m[2] * d[0] + m[0] * d[2]) * mu, (m[2] * d[1] + m[1] * d[2]) * mu]


def _surface_matrices(m, mu, lam):
    """Vzeta = RX Vxi + RY Veta of a traction-free surface; m, mu, lam of the surface layer."""
    xi, et, zt = (torch.stack(m[3 * r:3 * r + 3], -1) for r in range(3))
    mu, lam = mu[..., None, None], lam[..., None, None]
    eye = torch.eye(3, dtype=torch.float64, device=mu.device)

    def block(a):      # traction on the surface normal zt of a velocity gradient along a
        s = (zt * a).sum(-1)[..., None, None]
        return lam * zt[..., :, None] * a[..., None, :] + mu * (zt[..., None, :] * a[..., :, None] + s * eye)

    # the diagonal carries 2 lambda + mu in place of lambda + 2 mu, as the scheme's matrices do
    def chi(a):
        b = block(a)
        return b + torch.diag_embed((lam[..., 0] - mu[..., 0]) * zt * a)

    inv = torch.linalg.inv(chi(zt))
    return -inv @ chi(xi), -inv @ chi(et)


class _Cg:
    """One CGFDM model in FP64: the RK4 step of the interior state and the absorbing layers' auxiliaries."""

    def __init__(self, case, inp, med=None, metric=None):
        dev = self.dev = inp["dev"]
        self.nP = case["nPML"]
        self.rdh, self.dt = float(F32(1.0 / DH)), float(F32(inp["dt"]))
        self.m, self.jac = _metric_cg(inp, dev) if metric is None else metric
        med = [_cut(inp["med"][..., c], 0, 0).double() for c in range(3)] if med is None else med
        vs, vp, rho = med
        self.mu = rho * vs * vs
        self.lam = rho * (vp * vp - 2 * vs * vs)
        self.buo = 1 / rho
        nz, ny, nx = self.jac.shape
        self.prof = [_layers(n, self.nP, top, dev) for n, top in ((nx, True), (ny, True), (nz, False))]
        self.RX, self.RY = _surface_matrices([a[-1] for a in self.m], self.mu[-1], self.lam[-1])

    def faces(self):
        """(direction, layer's low index, its length) in the order of the auxiliaries."""
        nz, ny, nx = self.jac.shape
        return [(0, 0), (1, 0), (2, 0), (0, nx - self.nP), (1, ny - self.nP)]

    def rest(self):
        return torch.zeros((9,) + tuple(self.jac.shape), dtype=torch.float64, device=self.dev)

    def aux_rest(self):
        shape, out = list(self.jac.shape), []
        for d, _ in self.faces():
            s = list(shape)
            s[2 - d] = self.nP
            out.append(torch.zeros([9] + s, dtype=torch.float64, device=self.dev))
        return out

    def rhs(self, W, aux, fb):
        """(DT dW/dt, DT daux/dt) of the interior state W [9][nz][ny][nx]."""
        pad = torch.nn.functional.pad(W, (H,) * 6)
        mu, lam, buo, dt = self.mu, self.lam, self.buo, self.dt
        h, top_v, haux = None, [], [None] * 5
        extra = []
        for d in range(3):
            m = self.m[3 * d:3 * d + 3]
            al, be, dd = self.prof[d]
            raw = [_diff(pad[f], d, fb[d], self.rdh) for f in range(9)]
            if d < 2:
                top_v.append([raw[c][-3:] * _along(be, d) for c in range(3)])
            c = _dir_rhs(m, [r * _along(be, d) for r in raw], mu, lam, buo)
            h = c if h is None else [a + b for a, b in zip(h, c)]
            for n, (dn, lo) in enumerate(self.faces()):
                if dn != d:
                    continue

                def cut(a):
                    return a.narrow(2 - d, lo, self.nP)

                dv = _along(dd[lo:lo + self.nP], d)
                dr = [cut(r) * dv for r in raw]
                r = _dir_rhs([cut(a) for a in m], dr, cut(mu), cut(lam), cut(buo))
                if d < 2:
                    M = (self.RX if d == 0 else self.RY).narrow(1 - d, lo, self.nP)
                    vz = [sum(M[..., a, b] * dr[b][-1] for b in range(3)) for a in range(3)]
                    t = _dir_stress([cut(a)[-1] for a in self.m[6:9]], vz, cut(mu)[-1], cut(lam)[-1])
                    r = r[:3] + [torch.cat([r[3 + f][:-1], (r[3 + f][-1] + t[f])[None]]) for f in range(6)]
                ad = _along((dd + al)[lo:lo + self.nP], d)
                haux[n] = torch.stack([(r[f] - ad * aux[n][f]) * dt for f in range(9)])
                b = _along(be[lo:lo + self.nP], d)
                size = W.shape[3 - d]
                p = [0, 0] * d + [lo, size - lo - self.nP]
                extra.append(torch.nn.functional.pad(-b * aux[n] * dt, p))
        top = self.surface(pad, top_v, fb)
        h = torch.stack([torch.cat([h[f][:-3], top[f]]) for f in range(9)]) * dt
        for e in extra:
            h = h + e
        return h, haux

    def surface(self, pad, vel, fb):
        """The top three layers: the traction image and the one-sided vertical derivatives of the velocity."""
        mu, lam = self.mu[-3:], self.lam[-3:]
        lx = []
        T = [pad[3], pad[6], pad[7]], [pad[6], pad[4], pad[8]], [pad[7], pad[8], pad[5]]
        for d in range(3):
            m = [torch.nn.functional.pad(a * self.jac, (H,) * 6) for a in self.m[3 * d:3 * d + 3]]
            if d < 2:
                lo = pad.shape[1] - 2 * H - 3
                cutz = [a[lo:] for a in m]
                J = [sum(cutz[b] * T[a][b][lo:] for b in range(3)) for a in range(3)]
                lx.append([_diff(j, d, fb[d], self.rdh) * _along(self.prof[d][1], d) for j in J])
            else:
                lo = pad.shape[1] - 2 * H - 6
                J = [sum(m[b][lo:lo + 8] * T[a][b][lo:lo + 8] for b in range(3)) for a in range(3)]   # below the surface
                J = [torch.cat([j, torch.zeros_like(j[:1]), -j.flip(0)[:3]]) for j in J]
                lx.append([_diff(j, 2, fb[2], self.rdh)[-3:] for j in J])
        bj = self.buo[-3:] / self.jac[-3:]
        out = [bj * (lx[0][c] + lx[1][c] + lx[2][c]) for c in range(3)]
        v = [pad[c][:, H:-H, H:-H] for c in range(3)]
        f3, s = fb[2], pad.shape[1] - H - 1
        vz = []
        for c in range(3):
            w = v[c]
            third = f3 * (CF[0] * w[s - 2] + CF[1] * w[s - 2 + f3] + CF[2] * w[s - 2 + 2 * f3]) * self.rdh
            second = f3 * (w[s - 1 + f3] - w[s - 1]) * self.rdh
            first = sum(self.RX[..., c, b] * vel[0][b][-1] + self.RY[..., c, b] * vel[1][b][-1] for b in range(3))
            vz.append(torch.stack([third, second, first]))
        parts = [_dir_stress([a[-3:] for a in self.m[3 * d:3 * d + 3]], x, mu, lam)
                 for d, x in ((0, vel[0]), (1, vel[1]), (2, vz))]
        return out + [a + b + c for a, b, c in zip(*parts)]

    def step(self, W, aux, it):
        fb = SIGNS[it % 8]
        m, ma, w, wa = W, aux, W, aux
        for s in range(4):
            h, ha = self.rhs(w, wa, fb)
            fb = tuple(-v for v in fb)
            t = (m if s == 0 else t) + BETA[s] * h                                             # noqa: F821
            ta = [(a if s == 0 else b) + BETA[s] * c for a, b, c in zip(ma, ma if s == 0 else ta, ha)]  # noqa: F821
            if s < 3:
                w = m + ALPHA[s] * h
                wa = [a + ALPHA[s] * c for a, c in zip(ma, ha)]
        return t, ta


def _gauss_weights():
    i = np.arange(-3, 4)
    g = np.exp(-(i / 1.5) ** 2) / (1.5 * 1.772453850905516)
    return torch.tensor(g[:, None, None] * g[None, :, None] * g[None, None, :] / 0.998125703461425)


def _mechanism(strike, dip, rake):
    """(Mxx, Myy, Mzz, Mxy, Mxz, Myz) of a unit double couple."""
    s, d, r = (math.radians(v) for v in (strike, dip, rake))
    a = math.sin(d) * math.cos(r)
    m11 = -(a * math.sin(2 * s) + math.sin(2 * d) * math.sin(r) * math.sin(s) ** 2)
    m22 = a * math.sin(2 * s) - math.sin(2 * d) * math.sin(r) * math.cos(s) ** 2
    m12 = a * math.cos(2 * s) + 0.5 * math.sin(2 * d) * math.sin(r) * math.sin(2 * s)
    m13 = -(math.cos(d) * math.cos(r) * math.cos(s) + math.cos(2 * d) * math.sin(r) * math.sin(s))
    m23 = -(math.cos(d) * math.cos(r) * math.sin(s) - math.cos(2 * d) * math.sin(r) * math.cos(s))
    return [m22, m11, -(m11 + m22), m12, -m23, -m13]


def _source(case, inp, mu, lam, jac, sc):
    """f(W, it): the source's stress (or strain) added to the interior state at the start of step it.  mu, lam, jac
    over the interior."""
    c, dt, dev = inp["case"], float(F32(inp["dt"])), inp["dev"]
    vol = DH ** 3

    def strain(s, mu, lam):
        tr = s[0] + s[1] + s[2]
        den = 2 * mu * mu + 3 * lam * mu
        e = [((lam + mu) * s[a] - 0.5 * lam * (tr - s[a])) / den for a in range(3)]
        return e + [s[5] / mu, s[4] / mu, s[3] / mu]

    if case["source"] == "fault":
        cells = torch.tensor(inp["cells"], device=dev)
        i, j, k = cells[:, 0], cells[:, 1], cells[:, 2]
        pts = c.fault[:-1]
        mt = torch.tensor([_mechanism(p.strike, p.dip, float(p.rake[0])) for p in pts], device=dev,
                          dtype=torch.float64).T
        rate = torch.tensor(np.stack([p.rate for p in pts]), device=dev, dtype=torch.float64)
        scale = mu[k, j, i] / (jac[k, j, i] * vol) * pts[0].area

        def add(W, it):
            t = it * dt
            n = int(F32(F32(it) * F32(dt)) / F32(c.fault_dt))
            w = (t - n * float(F32(c.fault_dt))) / float(F32(c.fault_dt))
            r = (rate[:, n] + (rate[:, n + 1] - rate[:, n]) * w) * scale
            s = [mt[a] * r for a in range(6)]
            if sc:
                s = strain(s, mu[k, j, i], lam[k, j, i])
            W = W.clone()
            for a in range(6):
                W[3 + a].index_put_((k, j, i), -s[a] * dt, accumulate=True)
            return W
        return add
    X, Y, Z = inp["pos"]
    g = _gauss_weights().to(dev)
    box = (slice(Z - 3, Z + 4), slice(Y - 3, Y + 4), slice(X - 3, X + 4))
    j0 = jac[Z, Y, X]

    def add(W, it):
        t = it * dt
        if case["source"] == "ricker":
            fc = c.ricker_point[3]
            r = PI32 * fc * (t - 1.0 / fc)
            s = r * (3 - 2 * r * r) * math.exp(-r * r) * math.sqrt(PI32) * 0.5 * fc * PI32 * 1e9
            v = -s * g / (j0 * vol) * dt
            if sc:
                v = v / (3 * lam[box] + 2 * mu[box])
            parts = [v, v, v]
        else:
            q = c.double_couple
            td = t - (q["duration"] / 2 + 1)
            s = math.exp(-td * td / q["duration"] ** 2) / (math.sqrt(PI32) * q["duration"])
            v = s * g / (j0 * vol) * 1.5 * 10.0 ** (q["Mw"] + 6) * dt
            parts = [m * v for m in _mechanism(q["strike"], q["dip"], q["rake"])]
            if sc:
                parts = strain(parts, mu[box], lam[box])
        W = W.clone()
        for a, p in enumerate(parts):
            W[(3 + a,) + box] += p
        return W
    return add


def _record(case, inp):
    st = np.array(inp["case"].stations)
    n = _total_steps(case)
    return st, np.zeros((len(st), n, 9)), torch.zeros((case["ny"], case["nx"], 2), dtype=torch.float64,
                                                      device=inp["dev"])


def _peak(pgv, v):
    h = (v[0] ** 2 + v[1] ** 2).sqrt()
    return torch.maximum(pgv, torch.stack([h, (v[0] ** 2 + v[1] ** 2 + v[2] ** 2).sqrt()], -1))


def _forward(case, seed):
    with torch.no_grad():
        inp = _inputs(case, seed)
        return (_forward_sc if case["kind"] == "sc" else _forward_cg)(case, inp), None


def _forward_cg(case, inp):
    M = _Cg(case, inp)
    W, aux = M.rest(), M.aux_rest()
    steps = case["steps"]
    if case["kind"] == "cg16":
        steps += PRERUN
    elif case["kind"] == "cg":
        w = _field(case, inp["med"], inp["rng"], inp["dev"]).permute(3, 0, 1, 2)
        W = _cut(w, 0, 0).double()
    src = _source(case, inp, M.mu, M.lam, M.jac, False)
    st, traces, pgv = _record(case, inp)
    s = [torch.tensor(st[:, a], device=M.dev) for a in range(3)]
    rows = []
    for it in range(steps):
        W, aux = M.step(src(W, it), aux, it)
        rows.append(W[:, s[2], s[1], s[0]].T)
        pgv = _peak(pgv, W[:3, -1])
    traces[:, :steps] = torch.stack(rows, 1).cpu().numpy()
    out = {"velocity": traces[:, :, :3], "stress": traces[:, :, 3:], "pgv": pgv}
    if case.get("field"):
        w = torch.nn.functional.pad(W, (H,) * 6).permute(1, 2, 3, 0)
        out["first"], out["second"] = w[..., :3], w[..., 3:]
    return out


def _gradient64(case, seed):
    """The gradient by automatic differentiation of the FP64 run, a step at a time from kept states."""
    from torch.utils.checkpoint import checkpoint

    if case["nx"] * case["ny"] * case["nz"] * case["steps"] > 1.4e8:
        return None         # well over 20 s
    inp = _inputs(case, seed)
    dev = inp["dev"]
    metric = _metric_cg(inp, dev)
    med = [_cut(inp["med"][..., c], 0, 0).double().requires_grad_() for c in range(3)]
    obs = torch.tensor(_observed(case, inp["rng"], inp["dt"]), device=dev, dtype=torch.float64)
    st = np.array(inp["case"].stations)
    s = [torch.tensor(st[:, a], device=dev) for a in range(3)]
    n_aux = 5

    def step(it, vs, vp, rho, W, *aux):
        M = _Cg(case, inp, (vs, vp, rho), metric)
        src = _source(case, inp, M.mu, M.lam, M.jac, False)
        W, aux = M.step(src(W, it), list(aux), it)
        return (W,) + tuple(aux)

    M = _Cg(case, inp, None, metric)
    state = (M.rest(),) + tuple(M.aux_rest())
    del M
    J = 0.0
    for it in range(case["steps"]):
        state = checkpoint(step, it, *med, *state, use_reentrant=False)
        v = state[0][:3, s[2], s[1], s[0]].T
        J = J + 0.5 * ((v - obs[:, it]) ** 2).sum()
    assert len(state) == 1 + n_aux
    gvs, gvp, grho = torch.autograd.grad(J, med)
    p = case["nPML"]
    keep = torch.zeros_like(gvs)
    keep[p:, p:-p, p:-p] = 1
    return {"misfit": J.detach(), "vp": gvp * keep, "vs": gvs * keep, "rho": grho * keep}


# ------------------------------------------------- ME-AWENO in FP64
def _weno(a, b, c, d, e):
    """Left state of the face between c and d from five cells."""
    b1 = (10 * c * c - 31 * c * d + 25 * d * d + 11 * c * e - 19 * d * e + 4 * e * e) / 3
    b2 = (4 * b * b - 13 * b * c + 13 * c * c + 5 * b * d - 13 * c * d + 4 * d * d) / 3
    b3 = (4 * a * a - 19 * a * b + 25 * b * b + 11 * a * c - 31 * b * c + 10 * c * c) / 3
    w1, w2, w3 = 0.3125 / (b1 + 1e-6) ** 2, 0.625 / (b2 + 1e-6) ** 2, 0.0625 / (b3 + 1e-6) ** 2
    return (w1 * (0.375 * c + 0.75 * d - 0.125 * e) + w2 * (-0.125 * b + 0.75 * c + 0.375 * d)
            + w3 * (0.375 * a - 1.25 * b + 1.875 * c)) / (w1 + w2 + w3)


def _flux(n, lam, mu, buo, u):
    tr = lam * (u[3] + u[4] + u[5])
    return [-(n[0] * (tr + 2 * mu * u[3]) + mu * (n[1] * u[8] + n[2] * u[7])),
            -(n[1] * (tr + 2 * mu * u[4]) + mu * (n[0] * u[8] + n[2] * u[6])),
            -(n[2] * (tr + 2 * mu * u[5]) + mu * (n[0] * u[7] + n[1] * u[6])),
            -buo * n[0] * u[0], -buo * n[1] * u[1], -buo * n[2] * u[2],
            -buo * (n[1] * u[2] + n[2] * u[1]), -buo * (n[0] * u[2] + n[2] * u[0]), -buo * (n[0] * u[1] + n[1] * u[0])]


def _forward_sc(case, inp):
    dev, dt, rdh = inp["dev"], float(F32(inp["dt"])), float(F32(1.0 / DH))
    xyz = _coords(inp, dev)
    shape = xyz[2].shape

    def central(a, axis):
        r = torch.zeros(shape, dtype=torch.float32, device=dev)
        dim = 2 - axis
        n = a.shape[dim]
        r.narrow(dim, 1, n - 2).copy_(((a.narrow(dim, 2, n - 2) - a.narrow(dim, 0, n - 2)).double() * 0.5 * rdh).float())
        return r.double()

    c = [[central(a, ax) for a in xyz] for ax in range(3)]          # c[axis][component]

    def cross(p, q):
        return [p[(a + 1) % 3] * q[(a + 2) % 3] - p[(a + 2) % 3] * q[(a + 1) % 3] for a in range(3)]

    met = [[v.float().double() for v in cross(c[(d + 1) % 3], c[(d + 2) % 3])] for d in range(3)]
    jac = sum(c[0][a] * met[0][a] for a in range(3)).float().double()
    ring = torch.nn.functional.pad(torch.ones([n - 4 for n in shape], dtype=torch.float64, device=dev), (2,) * 6)
    met = [[v * ring for v in row] for row in met]     # the model's metric is zero in its two outermost layers
    vs, vp, rho = (inp["med"][..., a].double() for a in range(3))
    mu = (rho * vs * vs).float().double()
    lam = (rho * (vp * vp - 2 * vs * vs)).float().double()
    buo = (1 / rho).float().double()
    alpha = float(inp["med"][..., 1].max())
    W = _field(case, inp["med"], inp["rng"], dev).permute(3, 0, 1, 2).double().contiguous()
    inner = (slice(None),) + (slice(H, -H),) * 3
    cell = inner[1:]
    coef = (dt * rdh / jac)[cell]
    nz = case["nz"]
    damp = torch.ones(tuple(coef.shape), dtype=torch.float64, device=dev)
    G = np.exp(-(0.015 * np.arange(21)) ** 2)
    for axis, n, high in ((0, case["nx"], True), (1, case["ny"], True), (2, nz, False)):
        f = np.ones(n)
        i = np.arange(n)
        f[i <= 20] *= G[20 - i[i <= 20]]
        if high:
            f[i >= n - 20] *= G[20 - (n - i[i >= n - 20])]
        damp = damp * _along(torch.tensor(f, device=dev), axis)

    def sweep(W, axis):
        """-DT dF/dx over the interior: Lax-Friedrichs fluxes of the faces between WENO states, corrected."""
        dim = 2 - axis

        def sh(a, o, extra=0):
            for ax in range(3):
                d = 2 - ax
                if ax == axis:
                    a = a.narrow(d, H + o, a.shape[d] - 2 * H + extra)
                else:
                    a = a.narrow(d, H, a.shape[d] - 2 * H)
            return a

        # faces m + 1/2 for m = H - 1 .. n - 1 of the padded axis; zero beyond
        n = W.shape[1 + dim] - 2 * H
        uL = [_weno(*(sh(W[v], o - 1, 1) for o in (-2, -1, 0, 1, 2))) for v in range(9)]
        uR = [_weno(*(sh(W[v], o, 1) for o in (2, 1, 0, -1, -2))) for v in range(9)]
        nrm = [sh(a, -1, 1) for a in met[axis]]
        la, mm, bb = sh(lam, -1, 1), sh(mu, -1, 1), sh(buo, -1, 1)
        fL, fR = _flux(nrm, la, mm, bb, uL), _flux(nrm, la, mm, bb, uR)
        F = [0.5 * (a + b - alpha * (r - l)) for a, b, r, l in zip(fL, fR, uR, uL)]
        pad = [0, 0] * axis + [2, 2]
        out = []
        for v in range(9):
            E = torch.nn.functional.pad(F[v], pad)                      # faces p - 5/2 .. p + 5/2
            f = [E.narrow(dim, t, n) for t in range(6)]

            def corrected(b):
                return (f[b] - (-f[b - 2] + 16 * f[b - 1] - 30 * f[b] + 16 * f[b + 1] - f[b + 2]) / 288
                        + 7 / 5760 * (f[b - 2] - 4 * f[b - 1] + 6 * f[b] - 4 * f[b + 1] + f[b + 2]))
            out.append(-(corrected(3) - corrected(2)) * coef)
        # the top three layers correct with point fluxes
        k0 = nz - 3
        if axis < 2:
            cutW = [a[H + k0:H + nz] for a in W]
            cn = [a[H + k0:H + nz] for a in met[axis]]
            cl, cm, cb = lam[H + k0:H + nz], mu[H + k0:H + nz], buo[H + k0:H + nz]
            hu = _flux(cn, cl, cm, cb, cutW)
            other = 2 - (1 - axis)

            def at(a, o):
                a = a.narrow(other, H, a.shape[other] - 2 * H)
                return a.narrow(dim, H + o, a.shape[dim] - 2 * H)
        else:
            hu = _flux(*([a[k0:] for a in met[2]],), lam[k0:], mu[k0:], buo[k0:], [a[k0:] for a in W])

            def at(a, o):
                return a[:, H:-H, H:-H].narrow(0, H + o, 3)
        for v in range(9):
            g = [at(hu[v], o) for o in range(-3, 4)]
            f = F[v].narrow(dim, 1, n), F[v].narrow(dim, 0, n)
            f = [x[-3:] for x in f]

            def o2(b):
                return (-5 * g[b] + 39 * g[b + 1] - 34 * g[b + 2] - 34 * g[b + 3] + 39 * g[b + 4] - 5 * g[b + 5]) / 48

            def o4(b):
                return 0.5 * (g[b] - 3 * g[b + 1] + 2 * g[b + 2] + 2 * g[b + 3] - 3 * g[b + 4] + g[b + 5])

            A = f[0] - o2(1) / 24 + 7 / 5760 * o4(1)
            B = f[1] - o2(0) / 24 + 7 / 5760 * o4(0)
            out[v] = torch.cat([out[v][:-3], coef[-3:] * -(A - B)])
        return out

    def rhs(W):
        h = sweep(W, 0)
        for axis in (1, 2):
            h = [a + b for a, b in zip(h, sweep(W, axis))]
        return torch.stack(h)

    top = (slice(None), H + nz - 1, slice(H, -H), slice(H, -H))
    t = top[1:]

    def surface(W):
        """The characteristic free surface in the basis of the surface normal and the two tangents."""
        nrm = torch.stack([met[2][a][t] / jac[t] for a in range(3)], -1)
        t1, t2 = (torch.stack([c[d][a][t] for a in range(3)], -1) for d in (0, 1))
        B = torch.stack([v / v.norm(dim=-1, keepdim=True) for v in (nrm, t1, t2)], -1)
        R = torch.linalg.inv(B)
        u = W[top]
        la, mm, bb = lam[t], mu[t], buo[t]
        ro, cs, cp = 1 / bb, (mm * bb).sqrt(), ((la + 2 * mm) * bb).sqrt()
        tr = la * (u[3] + u[4] + u[5])
        S = torch.stack([tr + 2 * mm * u[3], mm * u[8], mm * u[7], mm * u[8], tr + 2 * mm * u[4], mm * u[6],
                         mm * u[7], mm * u[6], tr + 2 * mm * u[5]], -1).view(tuple(tr.shape) + (3, 3))
        v = (R @ torch.stack([u[0] * bb, u[1] * bb, u[2] * bb], -1)[..., None])[..., 0]
        T = R @ S @ R.transpose(-1, -2)
        ratio = la / (la + 2 * mm)
        v = torch.stack([v[..., 0] - T[..., 0, 0] / (cp * ro), v[..., 1] - T[..., 0, 1] / (cs * ro),
                         v[..., 2] - T[..., 0, 2] / (cs * ro)], -1)
        T2 = T.clone()
        T2[..., 1, 1] -= T[..., 0, 0] * ratio
        T2[..., 2, 2] -= T[..., 0, 0] * ratio
        T2[..., 0, :] = 0
        T2[..., :, 0] = 0
        S = B @ T2 @ B.transpose(-1, -2)
        v = (B @ v[..., None])[..., 0]
        tr = S[..., 0, 0] + S[..., 1, 1] + S[..., 2, 2]
        comp = 1 / (2 * mm * (3 * la + 2 * mm))
        e = [(2 * (la + mm) * S[..., d, d] - la * (tr - S[..., d, d])) * comp for d in range(3)]
        W = W.clone()
        W[top] = torch.stack([v[..., 0] * ro, v[..., 1] * ro, v[..., 2] * ro] + e
                             + [S[..., 1, 2] / mm, S[..., 0, 2] / mm, S[..., 0, 1] / mm])
        for k in range(H + nz, H + nz + H):
            w = W[:, :, H:-H, H:-H]
            W[:, k, H:-H, H:-H] = 4 * w[:, k - 1] - 6 * w[:, k - 2] + 4 * w[:, k - 3] - w[:, k - 4]
        return W

    li, mi, bi = lam[cell], mu[cell], buo[cell]
    src = _source(case, inp, mi, li, jac[cell], True)
    st, traces, pgv = _record(case, inp)
    s = [torch.tensor(st[:, a], device=dev) for a in range(3)]
    rows = []
    for it in range(case["steps"]):
        W = W.clone()
        W[inner] = src(W[inner], it)
        m = W
        for stage, (p, q) in enumerate(((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3))):
            h = rhs(W)
            W = W.clone()
            W[inner] = p * m[inner] + q * (W[inner] + h)
        W = surface(W)
        W[inner] = W[inner] * damp
        u = W[inner][:, s[2], s[1], s[0]]
        la, mm, bb = (a[s[2], s[1], s[0]] for a in (li, mi, bi))
        tr = la * (u[3] + u[4] + u[5])
        rows.append(torch.stack([u[0] * bb, u[1] * bb, u[2] * bb, tr + 2 * mm * u[3], tr + 2 * mm * u[4],
                                 tr + 2 * mm * u[5], mm * u[8], mm * u[7], mm * u[6]], -1))
        pgv = _peak(pgv, W[inner][:3, -1] * bi[-1])
    traces[:, :case["steps"]] = torch.stack(rows, 1).cpu().numpy()
    out = {"velocity": traces[:, :, :3], "stress": traces[:, :, 3:], "pgv": pgv}
    if case.get("field"):
        w = W.permute(1, 2, 3, 0)
        out["first"], out["second"] = w[..., :3], w[..., 3:]
    return out

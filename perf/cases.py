"""The work that a user of cfdwavemaker_gb300 has it do, as cases that can be timed.

A CFD solver loads one wave model (``waveinput.dat``) and then asks it for
kinematics: one point at a time from a legacy host code, a boundary's faces from
host arrays, a whole field on the device, the z = 0 sums at many points, an s-grid
ring that it advances and queries, or the learned update of that ring.  Each case is
one such use through the public entry points; sizes are those of the repository's
benchmark, tests and configurations, made ragged where a user's would be.

The wave model is the process's own (one per process, as in the reference), so a
case fixes the sea and the seed makes the points, the start time of the ring or the
channel fields.  The irregular-sea and s-grid values are FP32 sums that the C ABI
hands out in FP64; the cases that ask for them give them to the caller in the single
precision in which such a solver keeps its fields.

``exact`` restates what is computed in plain FP64 torch / numpy.
"""
from __future__ import annotations

import ctypes as C
import math
import os

import numpy as np
import torch

import cfdwavemaker_gb300 as cw
from cfdwavemaker_gb300 import seastate as ss

DEV = "cuda" if torch.cuda.is_available() else "cpu"
G = 9.81
RHO = 1025.0
MTHETA = 20.0                     # mean direction of every wave, degrees
PI_IRR = 3.1415926535897          # the truncated pi of the irregular-sea code
NLEV = 16                         # levels of the shipped learned-update weights
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(cw.__file__)), "data", "surrogate_nl16.bin")


def listed():
    return [
        # a host code without batching: u, v, w and eta of one point, call by call
        # (long-crested design sea, 128 components)
        {"name": "scalar_calls", "kind": "scalar", "nfreq": 128, "ndir": 1},
        # a boundary patch of a CPU solver: host arrays in and out, short-crested sea
        {"name": "boundary_host", "kind": "host", "n": 5003, "nfreq": 64, "ndir": 4},
        # initialising a field on the device: eta, u, v, w and the pressure
        {"name": "field_points", "kind": "points", "n": 65536, "nfreq": 128, "ndir": 1},
        # the same with the Smit s-coordinate theory
        {"name": "field_smit", "kind": "smit", "n": 16411, "nfreq": 24, "ndir": 5},
        # second-order sums at z = 0 of a fully spread sea, precision form
        {"name": "precision_form", "kind": "qform", "n": 100003, "nfreq": 256, "ndir": 16},
        # one ring update of the standard s-grid (default column form)
        {"name": "sgrid_update", "kind": "update", "nx": 256, "ny": 256, "nl": 16, "nfreq": 64, "ndir": 16,
         "pressure": False},
        # a small s-grid with the dynamic pressure on the ring
        {"name": "sgrid_pressure", "kind": "update", "nx": 47, "ny": 38, "nl": 12, "nfreq": 64, "ndir": 5,
         "pressure": True},
        # cell-centre queries against the standard ring
        {"name": "sgrid_query", "kind": "query", "n": 1000003, "nx": 256, "ny": 256, "nl": 16, "nfreq": 64,
         "ndir": 16},
        # velocities of a regular wave over a whole mesh
        {"name": "regular_field", "kind": "regular", "n": 4000037, "theory": "stream", "order": 24, "height": 8.0,
         "period": 12.0, "depth": 20.0},
        # the learned update: the network alone over the standard grid ...
        {"name": "network_forward", "kind": "forward", "b": 1, "h": 264, "w": 264},
        # ... a training step's loss and gradient on patches ...
        {"name": "network_gradient", "kind": "gradient", "b": 8, "h": 72, "w": 72},
        # ... and a predicted and checked ring update as wave_force_update runs it
        {"name": "learned_update", "kind": "learned", "nx": 256, "ny": 256, "nfreq": 64, "ndir": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scalar", "host", "points", "smit", "qform", "update", "query", "regular", "forward",
                       "gradient", "learned"])
    c = {"kind": kind}
    if kind == "scalar":
        c.update(nfreq=_log(rng, 16, 256), ndir=rng.choice([1, 2, 3]))
    elif kind == "host":
        c.update(n=_log(rng, 2, 40000), nfreq=_log(rng, 24, 96), ndir=rng.choice([1, 2, 3, 4]))
    elif kind == "points":
        c.update(n=_log(rng, 300, 65536), nfreq=_log(rng, 24, 128), ndir=rng.choice([1, 2]))
        if c["nfreq"] * c["ndir"] > 128:
            c["n"] = max(300, c["n"] // 4)
    elif kind == "smit":
        c.update(n=_log(rng, 200, 16411), nfreq=_log(rng, 12, 24), ndir=rng.choice([1, 3, 5]))
    elif kind == "qform":
        c.update(n=_log(rng, 1000, 70000), nfreq=_log(rng, 40, 256), ndir=rng.choice([4, 8, 12, 16]))
    elif kind == "update":
        c.update(nx=_log(rng, 16, 128), ny=_log(rng, 16, 128), nl=rng.choice([8, 10, 12, 16]),
                 nfreq=_log(rng, 24, 96), ndir=rng.choice([1, 3, 5, 8, 10]), pressure=rng.random() < 0.4)
    elif kind == "query":
        c.update(n=_log(rng, 1000, 1000000), nx=_log(rng, 24, 256), ny=_log(rng, 24, 256),
                 nl=rng.choice([8, 12, 16]), nfreq=_log(rng, 24, 64), ndir=rng.choice([1, 4, 8, 16]))
    elif kind == "regular":
        c.update(n=_log(rng, 1000, 4000000), depth=round(rng.uniform(18.0, 40.0), 3),
                 height=round(rng.uniform(2.0, 7.0), 3), period=round(rng.uniform(9.0, 13.0), 3))
        c.update(theory="stream", order=rng.randint(8, 24)) if rng.random() < 0.7 else c.update(theory="stokes",
                                                                                                order=5)
    elif kind == "forward":
        c.update(b=rng.choice([1, 2]), h=_log(rng, 24, 186), w=_log(rng, 24, 186))
    elif kind == "gradient":
        c.update(b=rng.choice([1, 2, 4, 8]), h=_log(rng, 24, 72), w=_log(rng, 24, 72))
    else:
        c.update(nx=_log(rng, 32, 200), ny=_log(rng, 32, 200), nfreq=_log(rng, 24, 64), ndir=rng.choice([4, 8, 16]))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
DEPTH = 100.0                     # of the short-crested seas
GRID_DT, LEARN_DT = 0.5, 0.1
SPACING = 1000.0 / 255.0          # of the standard 256 x 256 grid over 1 km


def _sea(case):
    """Component columns and depth: the long-crested 128-component design sea's
    parameters for one direction, the short-crested sea's otherwise."""
    nf, nd = case["nfreq"], case["ndir"]
    if nd == 1:
        return ss.irregular_components(4.0, 10.0, 3.3, nf, 0.3, 2.0, 50.0, 12345), 50.0
    return ss.irregular_components(6.0, 12.0, 2.0, nf, 0.25, 1.6, DEPTH, 2024, ndir=nd, spreading_s=10.0), DEPTH


def _grid(case, t0):
    nx, ny = case["nx"], case["ny"]
    return {"bounds": (0.0, SPACING * (nx - 1), 0.0, SPACING * (ny - 1)), "nx": nx, "ny": ny,
            "nl": case.get("nl", NLEV), "t0": t0, "dt": LEARN_DT if case["kind"] == "learned" else GRID_DT,
            "stretch": (0.7, 1.5)}


def _t0(case, seed):
    """The ring's start time (a query case keeps one ring for all its points)."""
    return 12.0 if case["kind"] == "query" else float(np.random.default_rng(seed).uniform(5.0, 60.0))


_wm = cw.CFDwavemaker()
_loaded = [None]                  # text of the loaded model
_qform = [None]                   # text of the model whose precision form is built
_stream = [None]


def _ok(rc):
    if rc != 0:
        raise RuntimeError("cfdwavemaker_gb300: %d %s" % (rc, cw.last_error()))


def _load(text, again=False):
    if again or _loaded[0] != text:
        _loaded[0] = _qform[0] = None
        _ok(_wm.initialize_text(text))
        _loaded[0] = text


def _use_stream(on):
    """A device user's stream for the device-pointer calls; none for the host calls."""
    if on and _stream[0] is None:
        _stream[0] = torch.cuda.Stream()
    cw.load().cfdwm_set_stream(C.c_void_p(_stream[0].cuda_stream) if on else None)


def _points(case, seed):
    """x, y, z, t of a point case, host FP64: a patch of the sea from the seabed to
    above the crests, a few wave periods."""
    kind = case["kind"]
    n = 1 if kind == "scalar" else case["n"]
    rng = np.random.default_rng(seed)
    if kind == "qform":
        return rng.uniform(0, 1000, n), rng.uniform(0, 1000, n), np.zeros(n), rng.uniform(0, 100, n)
    if kind == "query":
        g = _grid(case, _t0(case, seed))
        return (rng.uniform(0, g["bounds"][1], n), rng.uniform(0, g["bounds"][3], n), rng.uniform(-DEPTH, 6.0, n),
                np.full(n, g["t0"] + rng.uniform(0.0, GRID_DT)))
    if kind == "regular":
        x, z = rng.uniform(0, 300, n), rng.uniform(-case["depth"], 0.7 * case["height"], n)
        return x, rng.uniform(-50, 50, n), z, rng.uniform(0, 2 * case["period"], n)
    depth = 50.0 if case["ndir"] == 1 else DEPTH
    t = np.full(n, rng.uniform(0, 60)) if kind == "host" else rng.uniform(0, 60, n)
    return rng.uniform(0, 500, n), rng.uniform(-100, 100, n), rng.uniform(-depth, 4.0, n), t


def _channels(case, seed, which):
    """Smooth unit-variance channel planes as the network meets them (which 0: its
    inputs, 1: its targets)."""
    b, h, w = case["b"], case["h"], case["w"]
    ch = 8 * NLEV if which == 0 else 1 + 3 * NLEV
    if which:
        h, w = h - 8, w - 8
    gen = torch.Generator(device=DEV).manual_seed(2 * seed + which)
    f = torch.randn(b, ch, h // 4 + 2, w // 4 + 2, generator=gen, device=DEV)
    f = torch.nn.functional.interpolate(f, size=(h, w), mode="bilinear", align_corners=True)
    return (f * (1.4 if which == 0 else 0.5)).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    L = cw.load()
    s = {"kind": kind, "lib": L}
    if kind in ("forward", "gradient"):
        _use_stream(kind == "forward")
        _ok(L.cfdwm_surrogate_load(WEIGHTS.encode()))
        s["dims"] = (case["b"], case["h"], case["w"])
        s["x"] = _channels(case, seed, 0)
        if kind == "forward":
            s["y"] = torch.zeros(case["b"], 1 + 3 * NLEV, case["h"] - 8, case["w"] - 8, device=DEV)
        else:
            s["t"] = _channels(case, seed, 1)
            s["grad"] = torch.zeros(L.cfdwm_surrogate_nparams(), device=DEV)
        return s
    if kind == "regular":
        _load(ss.write_regular(None, case["theory"], case["height"], case["depth"], period=case["period"],
                               order=case["order"], mtheta=MTHETA, rho=RHO))
    else:
        comps, depth = _sea(case)
        grid = _grid(case, _t0(case, seed)) if kind in ("update", "query", "learned") else None
        # a ring case starts from its own freshly filled ring
        _load(ss.write_irregular(None, comps, depth, extrap=2, rho=RHO, mtheta=MTHETA, lsgrid=grid,
                                 vertical_theory="smit" if kind == "smit" else None),
              again=kind in ("update", "learned"))
    if kind in ("update", "learned"):
        _use_stream(True)
        if kind == "learned":
            _ok(L.cfdwm_surrogate_load(WEIGHTS.encode()))
        elif case["pressure"]:
            _wm.sgrid_pressure(True)
        s["dt"] = LEARN_DT if kind == "learned" else GRID_DT
        nxy, nl = case["nx"] * case["ny"], case.get("nl", NLEV)
        s["nx"] = case["nx"]
        s["eta"] = torch.zeros(nxy, device=DEV)
        s["vel"] = torch.zeros(4 if case.get("pressure") else 3, nxy * nl, device=DEV)
        return s
    p = _points(case, seed)
    if kind in ("scalar", "host"):
        _use_stream(False)
        s["p"] = tuple(float(a[0]) for a in p) if kind == "scalar" else p
        return s
    _use_stream(True)
    n = s["n"] = p[0].size
    s["p"] = [torch.as_tensor(a, device=DEV) for a in p]
    if kind == "qform":
        if _qform[0] != _loaded[0]:
            _ok(L.cfdwm_qform_build(1))
            _qform[0] = _loaded[0]
        s["out"] = torch.zeros(n, 4, device=DEV)
    elif kind == "query":
        s["out"] = torch.zeros(n, 4, device=DEV, dtype=torch.float64)
    else:
        s["out"] = torch.zeros(3 if kind == "regular" else 5, n, device=DEV, dtype=torch.float64)
    return s


def run(s):
    kind, L = s["kind"], s["lib"]
    if kind == "scalar":
        x, y, z, t = s["p"]
        return [np.float32(v) for v in _wm.velocity(x, y, z, t)] + [np.float32(_wm.surface_elevation(x, y, t))]
    if kind == "host":
        x, y, z, t = s["p"]
        kin = _wm.kinematics_batch(x, y, z, t).astype(np.float32)
        return [kin[:, q] for q in range(4)] + [_wm.dynamic_pressure_batch(x, y, z, t).astype(np.float32)]
    if kind == "forward":
        _ok(L.cfdwm_surrogate_forward(cw._ptr(s["x"]), *s["dims"], cw._ptr(s["y"])))
        return s["y"]
    if kind == "gradient":
        loss = C.c_double(0.0)
        _ok(L.cfdwm_surrogate_loss_grad(cw._ptr(s["x"]), cw._ptr(s["t"]), *s["dims"], C.byref(loss),
                                        cw._ptr(s["grad"])))
        return [np.float32(loss.value), s["grad"]]
    if kind in ("update", "learned"):
        t0, _ = _wm.sgrid_state()
        if kind == "update":
            _wm.force_update(t0 + 1.5 * s["dt"])
        else:
            _ok(L.cfdwm_surrogate_step(1, 0.2, 64, None, None))
        _ok(L.cfdwm_sgrid_block_export(0, 0, s["nx"], cw._ptr(s["eta"])))
        for f in range(s["vel"].shape[0]):
            _ok(L.cfdwm_sgrid_block_export(1 + f, 0, s["nx"], cw._ptr(s["vel"][f])))
        return [s["eta"], *s["vel"]]
    x, y, z, t = (cw._ptr(a) for a in s["p"])
    n, out = s["n"], s["out"]
    if kind == "qform":
        _ok(L.cfdwm_qform_eval(x, y, t, n, 1, cw._ptr(out)))
        return list(out.unbind(1))
    if kind == "query":
        _ok(L.wave_Kinematics_batch(x, y, z, t, n, cw._ptr(out)))
    elif kind == "regular":
        _ok(L.wave_VeloXYZ_batch(x, y, z, t, n, cw._ptr(out[0]), cw._ptr(out[1]), cw._ptr(out[2])))
        return list(out)
    else:
        _ok(L.wave_SurfElev_batch(x, y, t, n, cw._ptr(out[0])))
        _ok(L.wave_VeloXYZ_batch(x, y, z, t, n, cw._ptr(out[1]), cw._ptr(out[2]), cw._ptr(out[3])))
        _ok(L.wave_DynPres_batch(x, y, z, t, n, cw._ptr(out[4])))
    with torch.cuda.stream(_stream[0]):
        return list(out.float().unbind(1 if kind == "query" else 0))


def work(case):
    """Bytes: inputs and outputs once (and the tables and ring that have to be read).
    Operations: a multiply-add of the sums is two; the depth profile of a component
    or pair counts four, its phase terms six."""
    kind = case["kind"]
    N = case.get("nfreq", 0) * case.get("ndir", 1)
    pairs = N * (N + 1) // 2
    if kind == "scalar":
        return {"bytes": 3 * 48 * pairs + 8 * pairs + 4 * 64, "flops": 3 * 24 * pairs + 6 * pairs}
    if kind == "host":
        n = case["n"]
        return {"bytes": 72 * n + 56 * pairs, "flops": n * (36.0 * pairs + 40 * N)}
    if kind == "points":
        n = case["n"]
        return {"bytes": 72 * n + 56 * pairs, "flops": n * (36.0 * pairs + 40 * N)}
    if kind == "smit":
        n = case["n"]
        return {"bytes": 72 * n + 72 * pairs, "flops": n * (60.0 * pairs + 40 * N)}
    if kind == "qform":
        # four fields, a cosine and a sine half each, over the upper triangle
        return {"bytes": 40.0 * case["n"] + 32.0 * pairs, "flops": 16.0 * pairs * case["n"]}
    if kind in ("update", "learned"):
        nodes = case["nx"] * case["ny"] * case.get("nl", NLEV)
        nf = 4 if case.get("pressure") else 3
        if kind == "learned":
            return {"bytes": 4.0 * nodes * (3 * 11 + 8), "flops": nodes * N * 24.0 + _net_flops(
                1, case["nx"] + 8, case["ny"] + 8)}
        # the slot, its gradients, the first order per node and the second-order
        # forms of a column in as few depth functions as hold FP32 accuracy (12)
        return {"bytes": 4.0 * nodes * nf * 11,
                "flops": nodes * N * 4.0 * nf + case["nx"] * case["ny"] * (2 + 2 * nf * 12) * 2.0 * pairs}
    if kind == "query":
        nodes = case["nx"] * case["ny"] * case["nl"]
        return {"bytes": 64.0 * case["n"] + min(160.0 * nodes, 1280.0 * case["n"]), "flops": 800.0 * case["n"]}
    if kind == "regular":
        return {"bytes": 56.0 * case["n"], "flops": case["n"] * (16.0 * case["order"] + 60)}
    x = 4.0 * case["b"] * 8 * NLEV * case["h"] * case["w"]
    y = 4.0 * case["b"] * (1 + 3 * NLEV) * (case["h"] - 8) * (case["w"] - 8)
    f = _net_flops(case["b"], case["h"], case["w"])
    return {"bytes": x + y, "flops": f} if kind == "forward" else {"bytes": x + y, "flops": 3.0 * f}


def _net_flops(b, h, w):
    ch, tot = [8 * NLEV, 32, 32, 32, 1 + 3 * NLEV], 0.0
    for l in range(4):
        tot += 18.0 * ch[l] * ch[l + 1] * (h - 2 * l - 2) * (w - 2 * l - 2)
    return b * tot


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        return _exact_net(case, seed)
    if kind == "regular":
        return _exact_regular(case, seed) if case["theory"] == "stream" else None
    if kind == "query":
        return None               # a spline through a ring that only the library fills
    if kind == "learned":
        return _exact_learned(case, seed)
    sea = _Sea64(*_sea(case))
    if kind == "qform":
        x, y, _, t = (torch.as_tensor(a, device=DEV) for a in _points(case, seed))
        return _forms64(sea, x, y, t)
    if kind == "update":
        N, nodes = case["nfreq"] * case["ndir"], case["nx"] * case["ny"] * case["nl"]
        return _exact_update(case, seed, sea, nodes * N * N < 4e10)
    x, y, z, t = (torch.as_tensor(a, device=DEV) for a in _points(case, seed))
    rows = []
    step = max(1, int(4e7) // (sea.n * (sea.n + 1) // 2))
    for b in range(0, x.numel(), step):
        q = slice(b, b + step)
        rows.append((sea.smit if kind == "smit" else sea.point)(x[q], y[q], z[q], t[q]))
    r = torch.cat(rows, 1)                                   # eta, u, v, w, p
    if kind == "scalar":
        return [r[1, 0], r[2, 0], r[3, 0], r[0, 0]]
    return list(r)


class _Sea64:
    """Second-order Sharma-Dean sums of a sea in FP64 (all ramps 1, x = y = 0 origin)."""

    def __init__(self, comps, depth):
        self.h = depth
        o, A, k, ph, th = (torch.as_tensor(np.asarray(comps[q]), device=DEV) for q in
                           ("omega", "A", "k", "phase", "theta"))
        self.o, self.A, self.k, self.ph, self.n = o, A, k, ph, o.numel()
        th = th + MTHETA * PI_IRR / 180.0
        self.ct, self.st = torch.cos(th), torch.sin(th)
        self.kx, self.ky = k * self.ct, k * self.st
        # all pairs i < m and the diagonal, as vectors
        i, m = torch.triu_indices(self.n, self.n, device=DEV)
        self.i, self.m, d = i, m, i == m
        self.diag = d
        h, g = depth, G
        R = k * torch.tanh(k * h)
        S = torch.sqrt(R)
        kk, gam = k[i] * k[m], self.ct[i] * self.ct[m] + self.st[i] * self.st[m]
        self.kdot = kk * gam
        self.kp = torch.where(d, 2 * k[i], torch.sqrt((k[i] ** 2 + k[m] ** 2 + 2 * kk * gam).clamp(min=0)))
        self.km = torch.where(d, 0 * kk, torch.sqrt((k[i] ** 2 + k[m] ** 2 - 2 * kk * gam).clamp(min=0)))
        sp, sm = S[i] + S[m], S[i] - S[m]
        Rp = R[i] * R[m]
        ui, um = k[i] ** 2 - R[i] ** 2, k[m] ** 2 - R[m] ** 2
        Dp = (2 * sp ** 2 * (kk * gam - Rp) + sp * (S[i] * um + S[m] * ui)) / (sp ** 2 - self.kp * torch.tanh(
            self.kp * h))
        Dn = 6 * R[i] * ui / (2 * R[i] - k[i] * torch.tanh(2 * k[i] * h))
        self.hm = (k[i] != k[m]) & ~d
        den = torch.where(self.hm, sm ** 2 - self.km * torch.tanh(self.km * h), torch.ones_like(kk))
        Dm = torch.where(self.hm, (2 * sm ** 2 * (kk * gam + Rp) + sm * (S[m] * ui - S[i] * um)) / den, 0 * kk)
        ag = A * g / o
        one = torch.ones_like(kk)
        self.op, self.om = o[i] + o[m], o[i] - o[m]
        # potential amplitudes of the sum and difference terms
        self.P = torch.where(d, 0.25 * ag[i] ** 2 * Dn, 0.5 * ag[i] * ag[m] * Dp) / self.op
        self.M = torch.where(self.hm, 0.5 * ag[i] * ag[m] * Dm / torch.where(self.hm, self.om, one), 0 * kk)
        ap = (Dp - (kk * gam - Rp)) / torch.sqrt(Rp) + R[i] + R[m]
        an = (Dn - ui) / R[i] + 2 * R[i]
        am = torch.where(self.hm, (Dm - (kk * gam + Rp)) / torch.sqrt(Rp) + R[i] + R[m], 0 * kk)
        self.ap, self.am, self.an = torch.where(d, an, ap), am, an
        self.hp = (k[i] + k[m]) <= k.max()                   # the pair cache's sum pairs (diagonal: 2 k)
        self.Ep = torch.where(d, 0.25 * A[i] ** 2 * an, 0.5 * A[i] * A[m] * ap) * self.hp
        self.Em = 0.5 * A[i] * A[m] * am

    @staticmethod
    def prof(k, z, h):
        """cosh(k (z + h)) / cosh(k h) and sinh(k (z + h)) / cosh(k h)."""
        q = 1 / (1 + torch.exp(-2 * k * h))
        e, y = torch.exp(k * z), torch.exp(-k * (z + 2 * h))
        return q * (e + y), q * (e - y)

    def phasors(self, x, y, t):
        f = self.kx * x[:, None] + self.ky * y[:, None] - self.o * t[:, None] + self.ph
        return torch.cos(f), torch.sin(f)

    def trig(self, c, s):
        i, m = self.i, self.m
        cc, sn, sc, cs = c[:, i] * c[:, m], s[:, i] * s[:, m], s[:, i] * c[:, m], c[:, i] * s[:, m]
        return cc - sn, cc + sn, sc + cs, sc - cs

    def eta2(self, cp, cm):
        return cp @ self.Ep + cm @ self.Em

    def first(self, c, s, z):
        """u1, v1, w1, dp1 [n points] at z [n points], and the profiles."""
        F, H = self.prof(self.k, z[:, None], self.h)
        a = self.A * G * self.k / self.o
        return torch.stack([(F * c) @ (a * self.ct), (F * c) @ (a * self.st), (H * s) @ a,
                            (F * c) @ (self.A * RHO * G)]), F, H

    def taylor(self, c, s):
        a = self.A * self.o * self.k
        return torch.stack([c @ (a * self.ct), c @ (a * self.st), s @ (a / torch.tanh(self.k * self.h)),
                            c @ (self.A * RHO * G * self.k)])

    def second(self, trig, z, F, H, cache):
        """u2, v2, w2, dp2; cache: the pair cache's terms only (s-grid), else all pairs."""
        i, m, d = self.i, self.m, self.diag
        cp, cm, sp, sm = trig
        Fp, Hp = self.prof(self.kp, z[:, None], self.h)
        Fm, Hm = self.prof(self.km, z[:, None], self.h)
        keep = (self.hp | d) if cache else torch.ones_like(d)
        P = self.P * keep
        a, b = cp * Fp, cm * Fm
        out = [a @ (P * (self.kx[i] + self.kx[m])) + b @ (self.M * (self.kx[i] - self.kx[m])),
               a @ (P * (self.ky[i] + self.ky[m])) + b @ (self.M * (self.ky[i] - self.ky[m])),
               (sp * Hp) @ (P * self.kp) + (sm * Hm) @ (self.M * self.km)]
        p = a @ (P * self.op) + b @ (self.M * self.om)
        # the phase-free products of the first-order profiles, as the reference adds them
        w = torch.where(d, 0 * P, (keep if cache else torch.ones_like(d)).double()) * G * G / (self.o[i] * self.o[m])
        p = p - (F[:, i] * F[:, m]) @ (w * self.kdot) + (H[:, i] * H[:, m]) @ (w * self.k[i] * self.k[m])
        p = p - F @ (2 * G * G * (self.kx + self.ky) / self.o) + H @ (2 * G * G * self.k / self.o)
        return torch.stack(out + [RHO * p])

    def point(self, x, y, z, t):
        c, s = self.phasors(x, y, t)
        tr = self.trig(c, s)
        z = z.clamp(min=-self.h)
        z0, za = z.clamp(max=0.0), z.clamp(min=0.0)
        u1, F, H = self.first(c, s, z0)
        v = u1 + self.second(tr, z0, F, H, False) + self.taylor(c, s) * za
        return torch.cat([(c @ self.A + self.eta2(tr[0], tr[1]))[None], v])

    def smit(self, x, y, z, t):
        i, m, d, h, g, A, o = self.i, self.m, self.diag, self.h, G, self.A, self.o
        c, s = self.phasors(x, y, t)
        cp, cm, sp, sm = self.trig(c, s)
        eta = c @ A + self.eta2(cp, cm)
        zz = z.clamp(min=-h)
        D = h + eta
        zs, s1 = h * (h + zz) / D - h, ((h + zz) / D)[:, None]
        u1, F, H = self.first(c, s, zs)
        hp, hm = (self.hp | d).double(), self.hm.double()
        AA = torch.where(d, 0.5 * A[i] ** 2, A[i] * A[m])
        q = torch.where(d, 3 * o[i] ** 2, o[i] ** 2 + o[m] ** 2 + o[i] * o[m])
        Hp = -g / self.op * (self.ap / 2 - q / (2 * g) + g * self.kdot / (2 * o[i] * o[m])) * AA * hp
        om = torch.where(self.hm, self.om, torch.ones_like(self.om))
        Hm = -g / om * (self.am / 2 - (o[i] ** 2 + o[m] ** 2 - o[i] * o[m]) / (2 * g) +
                        g * self.kdot / (2 * o[i] * o[m])) * AA * hm
        Hm = Hm * (self.om.abs() > 1e-12)
        Fp, Sp = self.prof(self.kp, zs[:, None], h)
        Fm, Sm = self.prof(self.km, zs[:, None], h)
        kw = self.k / o
        a, b = kw * H, kw * self.k * h * F
        a1, a2, b1, b2 = a[:, i], a[:, m], b[:, i], b[:, m]
        bc, bm = -Hp * cp * Fp, -Hm * cm * Fm
        bs = Hp * self.kp * Sp * sp + Hm * self.km * Sm * sm
        half = torch.where(d, 0.25 * A[i] ** 2, A[i] * A[m]) * g
        gp, gm = half * hp, half * hm
        kxp, kxm, kyp, kym = (self.kx[i] + self.kx[m], self.kx[i] - self.kx[m], self.ky[i] + self.ky[m],
                              self.ky[i] - self.ky[m])
        u2 = bc @ kxp + bm @ kxm + ((s1 * (a1 + a2) * cp) @ (gp * kxp) + (s1 * (a1 - a2) * cm) @ (gm * kxm))
        v2 = bc @ kyp + bm @ kym
        w2 = -bs.sum(1)
        dphi = -h * bs.sum(1) + (((a1 + a2) + s1 * (b1 + b2)) * sp) @ gp + (((a1 - a2) + s1 * (b1 - b2)) * sm) @ gm
        w = RHO * g * g * self.kdot / (o[i] * o[m]) * AA
        ff, hh = F[:, i] * F[:, m], H[:, i] * H[:, m]
        p2 = RHO * (bc @ self.op + bm @ self.om) - ((ff - hh) * cp) @ (w * hp) - ((ff + hh) * cm) @ (w * hm)
        ex = -s @ (A * self.k * self.ct)
        ps = (H * s) @ (A * g * self.k / o) * h
        u2 = u2 - (h + zz) / D ** 2 * ex * (ps + dphi)
        v = (u1 + torch.stack([u2, v2, w2, p2])) * (z <= eta)
        return torch.cat([eta[None], v])


def _forms64(sea, x, y, t, eta_only=False):
    """eta2 (and u2, v2, w2) of the pair cache at z = 0."""
    n, N, i, m = x.numel(), sea.n, sea.i, sea.m
    keep = sea.hp | sea.diag

    def mat(v):
        W = torch.zeros(N, N, dtype=torch.float64, device=DEV)
        W[i, m] = v
        return W

    P, M = sea.P * keep, sea.M
    coef = [(sea.Ep, sea.Em)]
    coef += [(P * (k[i] + k[m]), M * (k[i] - k[m])) for k in (sea.kx, sea.ky)]
    coef += [(P * sea.kp * torch.tanh(sea.kp * sea.h), M * sea.km * torch.tanh(sea.km * sea.h))]
    # columns in blocks: of an upper triangle only the rows before the block's end
    coef = coef[:1] if eta_only else coef
    W = [(mat(p + q), mat(q - p) if f < 3 else mat(p - q)) for f, (p, q) in enumerate(coef)]
    out = torch.zeros(n, len(W), dtype=torch.float64, device=DEV)
    for b in range(0, n, 16384):
        q = slice(b, b + 16384)
        c, s = sea.phasors(x[q], y[q], t[q])
        for m0 in range(0, N, 256):
            m1 = min(N, m0 + 256)
            for f in range(len(W)):
                A, B = W[f][0][:m1, m0:m1], W[f][1][:m1, m0:m1]
                if f < 3:
                    out[q, f] += ((c[:, :m1] @ A) * c[:, m0:m1] + (s[:, :m1] @ B) * s[:, m0:m1]).sum(1)
                else:
                    out[q, f] += ((s[:, :m1] @ A) * c[:, m0:m1] + (c[:, :m1] @ B) * s[:, m0:m1]).sum(1)
    return list(out.unbind(1))


def _levels(grid, depth, eta):
    """Heights [n][nl] of the stretched levels under the elevation eta [n]."""
    nl = grid["nl"]
    a, b = grid["stretch"]
    sig = [-(max(math.tan(-(m / max(1, nl - 1) - 1.0) * a), 0.0) ** b) / math.tan(a) ** b for m in range(nl)]
    return eta[:, None] + torch.tensor(sig, dtype=torch.float64, device=DEV) * (depth + eta[:, None])


def _columns(case, halo=0):
    i = torch.arange(-halo, case["nx"] + halo, device=DEV, dtype=torch.float64) * SPACING
    j = torch.arange(-halo, case["ny"] + halo, device=DEV, dtype=torch.float64) * SPACING
    X, Y = torch.meshgrid(i, j, indexing="ij")
    return X.reshape(-1), Y.reshape(-1)


def _exact_update(case, seed, sea, levels):
    """The newest slot after one update; without `levels` (too many pairs) its
    elevation alone."""
    grid = _grid(case, _t0(case, seed))
    t = grid["t0"] + 3 * GRID_DT
    X, Y = _columns(case)
    nl, nf = case["nl"], 4 if case["pressure"] else 3
    if not levels:
        T = torch.full_like(X, t)
        eta1 = torch.cat([sea.phasors(X[b:b + 8192], Y[b:b + 8192], T[b:b + 8192])[0] @ sea.A
                          for b in range(0, X.numel(), 8192)])
        return [eta1 + _forms64(sea, X, Y, T, True)[0]] + [None] * nf
    etas, vel = [], []
    step = max(1, int(2e7) // (sea.n * (sea.n + 1) // 2))
    for b in range(0, X.numel(), step):
        x, y = X[b:b + step], Y[b:b + step]
        c, s = sea.phasors(x, y, torch.full_like(x, t))
        tr = sea.trig(c, s)
        eta = c @ sea.A + sea.eta2(tr[0], tr[1])
        etas.append(eta)
        z = _levels(grid, sea.h, eta)
        ty = sea.taylor(c, s)
        lev = []
        for l in range(nl):
            z0, za = z[:, l].clamp(max=0.0), z[:, l].clamp(min=0.0)
            u1, F, H = sea.first(c, s, z0)
            lev.append((u1 + sea.second(tr, z0, F, H, True) + ty * za)[:nf])
        vel.append(torch.stack(lev, 2))           # [nf][columns][nl]
    return [torch.cat(etas), *torch.cat(vel, 1).reshape(nf, -1)]


def _exact_regular(case, seed):
    """Stream-function wave (Rienecker and Fenton): Newton's method in wave-number
    units on kd, c, mean speed, q, r, the surface heights and the coefficients."""
    N, H, T, d = case["order"], case["height"], case["period"], case["depth"]
    jj = np.arange(1, N + 1)
    cj = np.cos(np.outer(np.arange(N + 1), jj) * np.pi / N)
    sj = np.sin(np.outer(np.arange(N + 1), jj) * np.pi / N)

    def eqs(z, H):
        K, c, U, q, r = z[:5]
        Y, B = z[5:N + 6], z[N + 6:]
        arg = np.outer(K + Y, jj)
        q_ = 1 / (1 + np.exp(-2 * jj * K))
        ch = (np.exp(arg - jj * K) + np.exp(-arg - jj * K)) * q_
        sh = (np.exp(arg - jj * K) - np.exp(-arg - jj * K)) * q_
        psi = (sh * cj) @ B - U * Y - q
        ber = 0.5 * ((-U + (ch * cj) @ (jj * B)) ** 2 + ((sh * sj) @ (jj * B)) ** 2) + Y - r
        head = [c * T * math.sqrt(G * K / d) - 2 * np.pi, c - U, Y[0] + Y[N] + 2 * Y[1:N].sum(),
                Y[0] - Y[N] - K * H / d]
        return np.concatenate([head, psi, ber])

    w = 2 * np.pi / T
    k = float(ss.dispersion_k(np.array([w]), d)[0])
    z = None
    for part in (0.2, 0.4, 0.6, 0.8, 1.0):
        kH = k * H * part
        if z is None:
            c = math.sqrt(math.tanh(k * d))
            z = np.concatenate([[k * d, c, c, 0.0, 0.5 * c * c], 0.5 * kH * np.cos(np.arange(N + 1) * np.pi / N),
                                [0.5 * kH / c], np.zeros(N - 1)])
        for _ in range(40):
            r0 = eqs(z, H * part)
            J = np.empty((z.size, z.size))
            for e in range(z.size):
                zz, hh = z.copy(), 1e-6 * max(1e-2, abs(z[e]))
                zz[e] += hh
                zm = z.copy()
                zm[e] -= hh
                J[:, e] = (eqs(zz, H * part) - eqs(zm, H * part)) / (2 * hh)
            dz = np.linalg.solve(J, -r0)
            z = z + dz
            if np.abs(dz).sum() < 1e-12:
                break
    K, c, U = z[:3]
    k = K / d
    sg = math.sqrt(G / k)
    x, y, zz, t = (torch.as_tensor(a, device=DEV) for a in _points(case, seed))
    th = MTHETA * math.pi / 180.0
    ph = k * (math.cos(th) * x + math.sin(th) * y - c * sg * t)
    ky = k * (zz.clamp(min=-d) + d)
    su, sw = torch.zeros_like(x), torch.zeros_like(x)
    for j in range(1, N + 1):
        q = 1 / (1 + math.exp(-2 * j * K))
        a, b = torch.exp(j * (ky - K)) * q, torch.exp(-j * (ky + K)) * q
        su += sg * j * z[N + 5 + j] * (a + b) * torch.cos(j * ph)
        sw += sg * j * z[N + 5 + j] * (a - b) * torch.sin(j * ph)
    u = (c - U) * sg + su
    return [math.cos(th) * u, math.sin(th) * u, sw]


def _net(nl=NLEV):
    """The shipped weights: BF16 kernels and FP32 biases, in FP64."""
    raw = open(WEIGHTS, "rb").read()
    w = torch.as_tensor(np.frombuffer(raw, np.float32, offset=24).copy(), device=DEV)
    ch, o, W, b = [8 * nl, 32, 32, 32, 1 + 3 * nl], 0, [], []
    for l in range(4):
        n = ch[l + 1] * ch[l] * 9
        W.append(w[o:o + n].bfloat16().double().reshape(ch[l + 1], ch[l], 3, 3))
        o += n
    for l in range(4):
        b.append(w[o:o + ch[l + 1]].double())
        o += ch[l + 1]
    return W, b


def _conv(x, w, b):
    """Valid 3 x 3 convolution as nine matrix products."""
    B, _, H, Wd = x.shape
    y = b[None, :, None, None].expand(B, -1, H - 2, Wd - 2)
    for dy in range(3):
        for dx in range(3):
            y = y + torch.einsum("oc,bchw->bohw", w[:, :, dy, dx], x[:, :, dy:dy + H - 2, dx:dx + Wd - 2])
    return y


def _forward64(x, W, b):
    for l in range(4):
        x = _conv(x, W[l], b[l])
        if l < 3:
            x = x * torch.sigmoid(x)
    return x


def _exact_net(case, seed):
    W, b = _net()
    x = _channels(case, seed, 0).double()
    if case["kind"] == "forward":
        return _forward64(x, W, b)
    for p in W + b:
        p.requires_grad_(True)
    y = _forward64(x, W, b)
    wt = torch.ones(1 + 3 * NLEV, dtype=torch.float64, device=DEV)
    wt[0] = NLEV
    d = y - _channels(case, seed, 1).double()
    loss = (wt[None, :, None, None] * d * d).sum() / (d.shape[0] * d.shape[2] * d.shape[3] * wt.sum())
    loss.backward()
    return [float(loss), torch.cat([p.grad.reshape(-1) for p in W + b])]


def _exact_learned(case, seed):
    sea = _Sea64(*_sea(case))
    grid = _grid(case, _t0(case, seed))
    t = grid["t0"] + 3 * LEARN_DT
    X, Y = _columns(case, 4)
    a2 = sea.A ** 2
    sig = math.sqrt(0.5 * float(a2.sum()))
    om, km = float((a2 * sea.o).sum() / a2.sum()), float((a2 * sea.k).sum() / a2.sum())
    a = sea.A * G * sea.k / sea.o
    cc = torch.stack([a * sea.ct, a * sea.st, sea.A], 1)
    feats, bases, etas = [], [], []
    for b in range(0, X.numel(), 1024):
        x, y = X[b:b + 1024], Y[b:b + 1024]
        c, s = sea.phasors(x, y, torch.full_like(x, t))
        e1 = c @ sea.A
        z = _levels(grid, sea.h, e1)
        z0, za = z.clamp(max=0.0), z.clamp(min=0.0)
        F, H = sea.prof(sea.k, z0[:, :, None], sea.h)             # [n][nl][N]
        uc, us = (F * c[:, None]) @ cc, (F * s[:, None]) @ cc     # u, v, p: in phase, quadrature
        wc, wq = (H * s[:, None]) @ a, -(H * c[:, None]) @ a
        f = torch.stack([uc[..., 0], us[..., 0], uc[..., 1], us[..., 1], wc, wq, uc[..., 2], us[..., 2]], 2)
        f[:, :, :6] /= sig * om
        f[:, :, 6:] /= sig
        ty = sea.taylor(c, s)
        feats.append(f.reshape(f.shape[0], -1))
        bases.append(torch.stack([uc[..., 0] + ty[0][:, None] * za, uc[..., 1] + ty[1][:, None] * za,
                                  wc + ty[2][:, None] * za]))
        etas.append(e1)
    nxh, nyh = case["nx"] + 8, case["ny"] + 8
    feat = torch.cat(feats).T.reshape(1, 8 * NLEV, nxh, nyh)
    W, b = _net()
    y = _forward64(feat, W, b)[0].reshape(1 + 3 * NLEV, -1)       # [49][nx ny]
    inner = lambda v: v.reshape(*v.shape[:-1], nxh, nyh)[..., 4:-4, 4:-4].reshape(*v.shape[:-1], -1)  # noqa: E731
    eta = inner(torch.cat(etas)) + y[0] * km * sig * sig
    base = inner(torch.cat(bases, 1).permute(0, 2, 1))            # [3][nl][nx ny]
    vel = base + y[1:].reshape(3, NLEV, -1) * km * sig * sig * om
    return [eta, *vel.permute(0, 2, 1).reshape(3, -1)]

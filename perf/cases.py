"""The work that users of the framework have it do, as timed cases.

Each case is one call of a solver's public interface (``step`` of the flat,
Kerr-Schild, log-spherical, cylindrical and staggered field solvers and of a
batch of log-spherical runs) or one training step of the warm-start network,
over sizes, options and precisions that the drivers, tests and the benchmark
of this repository use.  ``exact`` restates every one of them in plain torch
in 64 bits.

Field arrays are (d2, d1, d0) with the guard points, in the order
Ex Ey Ez Bx By Bz P.
"""
import math
import random

import torch

# LSRK(5,4) coefficients of the collocated solvers
RK_A = (0.0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257)
RK_B = (0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681)
RK_C = (0.0, 0.1496590219993, 0.3704009573644, 0.6222557631345, 0.9582821306784)

BATCH_GRIDS = ((512, 256), (768, 384), (1024, 512), (2048, 1024))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: a driver's loop that advances a 32^3 box (the
        # size of the quick runs and tests) one step per call
        _flat("flat_box_32_call", (32, 32, 32), steps=1),
        # the Alfven-packet size, a few steps per call as between diagnostics
        _flat("flat_box_128", (128, 128, 128), steps=4),
        # the benchmark's grid, one step
        _flat("flat_box_512", (512, 512, 512), steps=1),
        # a rotating star with an absorbing layer on an odd grid (rows of an
        # odd length): the rotator runs of the warm-start study
        _flat("flat_star_191", (191, 191, 191), steps=2, star=True),
        # the FP64 run that single-precision results are judged by
        _flat("flat_box_160_f64", (160, 144, 128), steps=1, f64=True),
        # a ragged box in the other semantics (the reference's GPU build)
        _flat("flat_box_ragged_gpu", (250, 187, 122), steps=2, semantics="gpu"),
        # the Kerr-Schild Wald problem at its configured size
        {"name": "gr_wald_256", "kind": "gr", "n0": 256, "n1": 256, "n2": 256, "half": 20.0,
         "pml": 16, "steps": 1},
        # the log-spherical pulsar at the largest grid of its configuration
        {"name": "sph_2048x1024", "kind": "sph", "n0": 2048, "n1": 1024, "steps": 4},
        # uneven log-spherical runs advanced together
        {"name": "sph_batch_8", "kind": "batch", "runs": 8, "grids": "0 1 2 3 2 1 0 1", "steps": 4},
        # the cylindrical pulsar of the benchmark
        {"name": "cyl_1024x2048", "kind": "cyl", "n0": 1024, "n1": 2048, "steps": 4},
        # the staggered solver's plane-wave box, ordinary size
        {"name": "yee_box_256", "kind": "yee", "n0": 256, "n1": 256, "n2": 256, "steps": 2},
        # one training step of the warm-start network, the benchmark's batch
        {"name": "unet_train_8x64", "kind": "unet", "samples": 8, "side": 64},
    ]


def _flat(name, n, steps, star=False, f64=False, semantics="cpu", arithmetic="reference"):
    return {"name": name, "kind": "flat", "n0": n[0], "n1": n[1], "n2": n[2], "steps": steps,
            "star": star, "f64": f64, "semantics": semantics, "arithmetic": arithmetic}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("flat", "flat", "flat", "flat", "gr", "sph", "batch", "cyl", "yee", "unet"))
    if kind == "flat":
        f64 = rng.random() < 0.2
        star = rng.random() < 0.3
        side = _log_int(rng, 24, 200 if f64 else 400)
        # axes within a factor of two of one another, of any parity
        n = [max(20, int(side * rng.uniform(0.7, 1.25))) for _ in range(3)]
        if star:
            n = [max(40, side)] * 3
        semantics = rng.choice(("cpu", "cpu", "gpu"))
        arithmetic = "fast" if semantics == "cpu" and rng.random() < 0.25 else "reference"
        c = _flat("", n, rng.randint(1, 4) if side < 200 else 1, star, f64, semantics, arithmetic)
    elif kind == "gr":
        side = _log_int(rng, 40, 240)
        n = [max(40, int(side * rng.uniform(0.8, 1.05))) for _ in range(3)]
        c = {"kind": "gr", "n0": n[0], "n1": n[1], "n2": n[2], "half": 20.0 if side > 100 else 8.0,
             "pml": 6 if side < 100 else 12, "steps": rng.randint(1, 2)}
    elif kind == "sph":
        side = _log_int(rng, 64, 1024)
        c = {"kind": "sph", "n0": int(2 * side * rng.uniform(0.8, 1.0)), "n1": side,
             "steps": rng.randint(1, 4)}
    elif kind == "batch":
        runs = rng.randint(2, 8)
        c = {"kind": "batch", "runs": runs, "steps": rng.randint(1, 4),
             "grids": " ".join(str(rng.randint(0, 2)) for _ in range(runs))}
    elif kind == "cyl":
        side = _log_int(rng, 64, 1024)
        c = {"kind": "cyl", "n0": side, "n1": int(2 * side * rng.uniform(0.8, 1.0)),
             "steps": rng.randint(1, 4)}
    elif kind == "yee":
        side = _log_int(rng, 24, 320)
        n = [max(20, int(side * rng.uniform(0.7, 1.2))) for _ in range(3)]
        c = {"kind": "yee", "n0": n[0], "n1": n[1], "n2": n[2], "steps": rng.randint(1, 3)}
    else:
        c = {"kind": "unet", "samples": rng.randint(1, 8), "side": 2 * rng.randint(8, 32)}
    c.pop("name", None)
    return c


# ------------------------------------------------- parameters of the cases

def _middle(n, d):
    """Distance of the first of n points from an origin midway between two."""
    return (n // 2 + 0.5) * d


def _settings(case, seed, run=0):
    """The simulation parameters of a case as a plain dict (the fields of
    SimParams that differ from its defaults, and what exact needs)."""
    rng = random.Random(7919 * seed + run)
    kind = case["kind"]
    s = {"semantics": "cpu", "arithmetic": "reference", "f64": False, "steps": case.get("steps", 1),
         "use_edotb_damping": True, "damp_gamma": 0.2, "ch2": 1.0, "tau": 2.0, "KOeps": 0.5,
         "problem": 0, "pml": [0, 0, 0], "pmllen": 1, "sigpml": 0.1, "sizes": None}
    if kind == "flat":
        n = [case["n0"], case["n1"], case["n2"]]
        s.update(N=n, guard=[3, 3, 3], semantics=case["semantics"], arithmetic=case["arithmetic"],
                 f64=case["f64"])
        if case["star"]:
            # an oblique rotator in a box with an absorbing layer, 12 cells to
            # the star's radius; the half-cell shift keeps points off the origin
            d = 4.0 / 12.0
            incl = math.radians(rng.uniform(10.0, 80.0))
            s.update(lower=[-_middle(m, d) for m in n], size=[d * m for m in n], periodic=[False] * 3,
                     pml=[max(4, n[0] // 16)] * 3, pmllen=max(1, n[0] // 32), problem=1,
                     radius=4.0 + 0.013, omega=rng.uniform(0.03, 0.06), b0=1.0,
                     p1=math.sin(incl), p2=0.0, p3=math.cos(incl), dt=0.4 * d)
        else:
            h = 1.0 / max(n)
            s.update(lower=[0.0] * 3, size=[h * m for m in n], periodic=[True] * 3, dt=0.5 * h)
    elif kind == "gr":
        n = [case["n0"], case["n1"], case["n2"]]
        d = 2 * case["half"] / max(n)
        s.update(N=n, guard=[3, 3, 3], lower=[-_middle(m, d) for m in n],
                 size=[d * m for m in n], periodic=[False] * 3, pml=[case["pml"]] * 3,
                 pmllen=max(1, case["pml"] // 2), a=rng.uniform(0.85, 0.95), dt=0.3 * d)
    elif kind in ("sph", "batch"):
        if kind == "batch":
            nr, nth = BATCH_GRIDS[int(case["grids"].split()[run])]
        else:
            nr, nth = case["n0"], case["n1"]
        length = math.log(100.0)
        s.update(N=[nr, nth, 1], guard=[4, 4, 0], lower=[0.0] * 3, size=[length, math.pi, 1.0],
                 periodic=[False] * 3, pml=[8, 0, 0], pmllen=8, problem=1, radius=1.0,
                 omega=1.0 / rng.uniform(3.0, 10.0), b0=1.0, dt=0.3 * length / nr)
    elif kind == "cyl":
        nr, nz = case["n0"], case["n1"]
        rmax = 64.0 * nr / 1024.0 if nr >= 256 else 16.0
        dz = 2 * rmax / nz
        s.update(N=[nr, nz, 1], guard=[3, 3, 0], lower=[0.0, -_middle(nz, dz), 0.0],
                 size=[rmax, 2 * rmax, 1.0], periodic=[False] * 3, pml=[8, 8, 0], pmllen=4,
                 problem=1, radius=rmax / 16.0 + 0.003, omega=rng.uniform(0.04, 0.06), b0=1.0,
                 dt=0.4 * min(rmax / nr, dz))
    elif kind == "yee":
        n = [case["n0"], case["n1"], case["n2"]]
        h = 1.0 / max(n)
        s.update(N=n, guard=[2, 2, 2], lower=[0.0] * 3, size=[h * m for m in n],
                 periodic=[True] * 3, dt=0.5 * h)
    s["dims"] = [s["N"][a] + 2 * s["guard"][a] for a in range(3)]
    s["delta"] = [s["size"][a] / s["N"][a] for a in range(3)]
    s["tiny"] = 1e-11 if s["f64"] else 1e-7
    return s


def _axis(s, a, shift=0.0):
    n = torch.arange(s["dims"][a], dtype=torch.float64, device=_device())
    return s["lower"][a] + s["delta"][a] * (n - s["guard"][a] + shift)


class _Waves:
    """A sum of plane waves with whole numbers of wavelengths per box."""

    def __init__(self, rng, s, amplitude, count=6, top=4):
        self.modes = []
        for _ in range(count):
            n = [rng.randint(-top, top) for _ in range(3)]
            if n[0] == 0:
                n[0] = 1
            k = [2 * math.pi * n[a] / s["size"][a] for a in range(3)]
            self.modes.append((k, rng.uniform(0, 2 * math.pi), rng.uniform(0.5, 1.0)))
        total = math.sqrt(sum(m[2] ** 2 for m in self.modes) / 2)
        self.modes = [(k, p, w * amplitude / total) for k, p, w in self.modes]

    def at(self, x, y, z):
        out = torch.zeros(torch.broadcast_shapes(x.shape, y.shape, z.shape), dtype=torch.float64,
                          device=x.device)
        for k, phase, w in self.modes:
            out += w * torch.sin(k[0] * x + k[1] * y + (k[2] * z + phase))
        return out


def _start(case, seed, run=0):
    """Start fields: a background field of the problem with waves on it, an
    E below |B|, and a P of the size that the cleaning keeps it at."""
    s = _settings(case, seed, run)
    dtype = torch.float64 if s["f64"] else torch.float32
    rng = random.Random(104729 * seed + 31 * run + 1)
    kind = case["kind"]
    amp = 0.2 if kind in ("flat", "yee") and not s["problem"] else 0.03
    db = [_Waves(rng, s, amp) for _ in range(3)]
    de = [_Waves(rng, s, 0.1) for _ in range(3)]
    dp = _Waves(rng, s, 0.01)
    d0, d1, d2 = s["dims"]
    f = [torch.empty((d2, d1, d0), dtype=dtype, device=_device()) for _ in range(7)]
    x = _axis(s, 0)[None, None, :]
    y = _axis(s, 1)[None, :, None]
    zs = _axis(s, 2)[:, None, None]
    for k0 in range(0, d2, 16):
        z = zs[k0:k0 + 16]
        if kind == "gr":
            back, scale = [0.0, 0.0, 1.0 / _cks(s, x, y, z)["sg"]], 1.0
        elif kind in ("sph", "batch"):
            r = torch.exp(x)
            scale = 1.0 / r ** 4
            back = [2.0 * torch.cos(y) * scale, torch.sin(y) * scale, 0.0]
        elif kind == "cyl":
            r = torch.sqrt(x * x + y * y)
            scale = s["radius"] ** 3 / torch.clamp(r, min=0.4 * s["radius"]) ** 3
            back = [3.0 * x * y / r ** 2 * scale, (3.0 * y * y / r ** 2 - 1.0) * scale, 0.0]
        elif s["problem"]:
            r = torch.sqrt(x * x + y * y + z * z)
            scale = 1.0 / r ** 3
            back = [c * s["b0"] for c in _dipole(s, x, y, z, 0.0)]
        else:
            back, scale = [1.0, 0.0, 0.0], 1.0
        w = [db[c].at(x, y, z) for c in range(3)]
        if kind in ("sph", "batch", "cyl"):
            # a component that vanishes on the axis keeps vanishing there
            zero = torch.sin(y) if kind != "cyl" else x / (x.abs() + s["radius"])
            odd = (1, 2) if kind != "cyl" else (0, 2)
        B = [back[c] + scale * w[c] * (zero if kind in ("sph", "batch", "cyl") and c in odd else 1.0)
             for c in range(3)]
        E = [scale * de[c].at(x, y, z) for c in range(3)]
        if kind in ("sph", "batch", "cyl"):
            E = [E[c] * zero * 0.5 for c in range(3)]
        for c in range(3):
            f[c][k0:k0 + 16] = E[c]
            f[3 + c][k0:k0 + 16] = B[c]
        f[6][k0:k0 + 16] = scale * dp.at(x, y, z)
    return s, f


# ------------------------------------------------- what a program has in hand

class _Buffer:
    """One of the library's device arrays as torch sees it; keeps the fields
    that own it."""

    def __init__(self, data, fid, f64):
        self.owner = data
        ptr, shape = data.dev_ptr(fid), data.shape
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8" if f64 else "<f4",
                                         "data": (int(ptr), False), "version": 3, "strides": None}


class _Solver:
    """An environment, its fields on the device and a solver, as a driver
    sets them up."""

    def __init__(self, cls, s, fields):
        import numpy as np

        from coffee_b200.config import SimParams
        from coffee_b200.solver import SimData, SimEnvironment

        p = SimParams()
        for name in ("N", "guard", "lower", "size", "pml", "pmllen", "sigpml", "problem", "radius",
                     "omega", "b0", "p1", "p2", "p3", "a", "dt", "use_edotb_damping", "damp_gamma",
                     "ch2", "tau", "KOeps"):
            if name in s:
                setattr(p, name, s[name])
        p.periodic_boundary = s["periodic"]
        self.env = SimEnvironment(p)
        self.data = SimData(self.env, np.float64 if s["f64"] else np.float32)
        self.views = [torch.as_tensor(_Buffer(self.data, k, s["f64"]), device="cuda")
                      for k in range(7)]
        for v, f in zip(self.views, fields):
            v.copy_(f)
        torch.cuda.synchronize()
        self.solver = cls(self.data, self.env, **({"semantics": s["semantics"]}
                                                  if cls.__name__ == "FieldSolverEZ" else {}))
        if s["arithmetic"] != "reference":
            self.solver.set_arithmetic(s["arithmetic"])
        self.time, self.dt = 0.0, s["dt"]


def prepare(case, seed):
    from coffee_b200 import solver as S

    kind = case["kind"]
    if kind == "unet":
        return _prepare_unet(case, seed)
    if kind == "batch":
        runs = []
        for m in range(case["runs"]):
            s, f = _start(case, seed, m)
            runs.append(_Solver(S.FieldSolverEZSpherical, s, f))
        return {"kind": kind, "runs": runs, "batch": S.SphBatch([r.solver for r in runs]),
                "steps": case["steps"]}
    cls = {"flat": S.FieldSolverEZ, "gr": S.FieldSolverGrEZ, "sph": S.FieldSolverEZSpherical,
           "cyl": S.FieldSolverEZCylindrical, "yee": S.FieldSolver}[kind]
    s, f = _start(case, seed)
    return {"kind": kind, "run": _Solver(cls, s, f), "steps": case["steps"]}


def run(state):
    kind = state["kind"]
    if kind == "unet":
        net = state["net"]
        out = net.forward(state["x"])
        loss, dout = net.loss(out, state["target"], state["mask"])
        net.backward(dout)
        net.step(state["lr"])
        return {"out": out, "loss": loss, "gw": [L.gw for L in net.layers],
                "gb": [L.gb for L in net.layers]}
    if kind == "batch":
        state["batch"].step(state["steps"])
        return [r.views for r in state["runs"]]
    r = state["run"]
    if state["steps"] == 1:
        r.solver.evolve_fields(r.time)
    else:
        r.solver.step(r.time, state["steps"])
    r.time += state["steps"] * r.dt
    return r.views[:6] if kind == "yee" else r.views


def work(case):
    """Each field read once and written once in a call; the operations of
    every step."""
    kind = case["kind"]
    if kind == "unet":
        full = case["samples"] * case["side"] ** 3
        macs = 27 * (16 * 16 * 3 + 48 * 16 + (16 * 32 + 32 * 32) / 8)
        # forward, input gradient (not of the first layer) and weight gradient
        return {"bytes": full * (16 * 2 + 16 * 4 + 4 + 16 * 4),
                "flops": 2.0 * full * (3 * macs - 27 * 16 * 16)}
    if kind == "batch":
        pts = sum(BATCH_GRIDS[int(g)][0] * BATCH_GRIDS[int(g)][1] for g in case["grids"].split())
    else:
        pts = case["n0"] * case["n1"] * case.get("n2", 1)
    size = 8 if case.get("f64") else 4
    # per point and step: five stages of derivatives, current, update and
    # clamps, and the dissipation pass (staggered: three substeps)
    flops = {"flat": 5 * 260 + 280, "gr": 5 * 520 + 500, "sph": 5 * 270 + 230, "batch": 5 * 270 + 230,
             "cyl": 5 * 220 + 200, "yee": 3 * 330}[kind]
    fields = 6 if kind == "yee" else 7
    return {"bytes": 2.0 * fields * size * pts, "flops": float(flops) * pts * case["steps"]}


def tolerance(case):
    """About four times the largest distance from `exact` over the listed and
    sixty drawn cases.  Rounding shows most where a field is the small
    difference of large ones: P and B_phi beside the axis, the few points
    around the dipole's and the ring's singularity (which a tighter
    Kerr-Schild box resolves better)."""
    kind = case["kind"]
    if kind == "unet":
        return {"rel": 2e-2}
    if case.get("f64"):
        return {"rel": 1e-13 if case["star"] else 5e-15}
    if kind == "flat":
        return {"rel": 3e-5 if case["star"] else 8e-6}
    if kind == "gr":
        return {"rel": 5e-5 if case["half"] > 10.0 else 3e-3}
    return {"rel": {"sph": 3e-4, "batch": 3e-4, "cyl": 4e-4, "yee": 2e-6}[kind]}


# ----------------------------------------------------- 64-bit restatements

def exact(case, seed):
    kind = case["kind"]
    if kind == "unet":
        return _exact_unet(case, seed)
    if kind == "batch":
        out = []
        for m in range(case["runs"]):
            s, f = _start(case, seed, m)
            out.append(_sph_steps(s, [a.double() for a in f]))
        return out
    s, f = _start(case, seed)
    f = [a.double() for a in f]
    step = {"flat": _flat_steps, "gr": _gr_steps, "sph": _sph_steps, "cyl": _cyl_steps,
            "yee": _yee_steps}[kind]
    out = step(s, f)
    return out[:6] if kind == "yee" else out


def _box(s, ax=None, off=0, k0=None, k1=None):
    """Slices of the update box (planes k0..k1 of it), shifted by `off` along
    axis `ax`."""
    sl = []
    for a in (2, 1, 0):
        lo, hi = s["guard"][a], s["dims"][a] - s["guard"][a]
        if a == 2 and k0 is not None:
            lo, hi = k0, k1
        o = off if a == ax else 0
        sl.append(slice(lo + o, hi + o))
    return tuple(sl)


def _d4(s, f, ax, k0=None, k1=None, w=None):
    """4th-order first difference of f (times the weight w) in the box."""
    def g(off):
        b = _box(s, ax, off, k0, k1)
        return f[b] if w is None else f[b] * w[b]
    return (g(-2) - 8.0 * g(-1) + 8.0 * g(1) - g(2)) / (12.0 * s["delta"][ax])


def _d6(s, f, ax, k0=None, k1=None, w=None):
    out = 0.0
    for off, c in zip(range(-3, 4), (1.0, -6.0, 15.0, -20.0, 15.0, -6.0, 1.0)):
        b = _box(s, ax, off, k0, k1)
        out = out + c * (f[b] if w is None else f[b] * w[b])
    return out


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]


def _wrap(s, fields):
    """Guard points of the periodic axes."""
    for f in fields:
        for a in range(3):
            if not s["periodic"][a]:
                continue
            g, n, d = s["guard"][a], s["N"][a], 2 - a
            f.narrow(d, 0, g).copy_(f.narrow(d, n, g))
            f.narrow(d, n + g, g).copy_(f.narrow(d, g, g))


def _clamp(s, E, B, lower=lambda v: v, floor_e=0.0):
    """E.B = 0, then |E| <= |B|, with the metric's lowering of an index."""
    B2 = torch.clamp(_dot(B, lower(B)), min=s["tiny"])
    q = _dot(E, lower(B)) / B2
    E = [E[c] - q * B[c] for c in range(3)]
    E2 = torch.clamp(_dot(E, lower(E)), min=floor_e)
    top = _dot(B, lower(B)) if floor_e else B2
    f = torch.where(E2 > top, torch.sqrt(top / torch.clamp(E2, min=1e-300)), torch.ones_like(E2))
    return [e * f for e in E]


def _shape(r, r0, width):
    return 0.5 * (1.0 - torch.tanh((r - r0) / width))


def _relax(sig, u, un, tiny):
    """Relaxation towards the start-of-step value where sig > tiny."""
    on = sig > tiny
    sg = torch.where(on, sig, torch.ones_like(sig))
    e = torch.exp(-sg)
    return torch.where(on, e * un + (1.0 - e) / sg * (u - un), u)


def _layer_sigma(s, pos, scale, axes=(0, 1, 2)):
    sig = 0.0
    for a in axes:
        hi = s["lower"][a] + s["size"][a] - s["pml"][a] * s["delta"][a]
        lo = s["lower"][a] + s["pml"][a] * s["delta"][a]
        q = torch.clamp(torch.maximum(pos[a] - hi, lo - pos[a]), min=0.0) / scale[a]
        sig = sig + s["sigpml"] * q ** 3
    return sig


# flat collocated solver

def _dipole(s, x, y, z, phase):
    c, sn = math.cos(phase), math.sin(phase)
    p = [s["p1"] * c - s["p2"] * sn, s["p1"] * sn + s["p2"] * c, s["p3"]]
    r2 = x * x + y * y + z * z
    pr = p[0] * x + p[1] * y + p[2] * z
    den = r2 ** 1.5 + s["tiny"]
    return [(3.0 * v * pr / (r2 + s["tiny"]) - m) / den for v, m in ((x, p[0]), (y, p[1]), (z, p[2]))]


def _flat_star(s, E, B, pos, t):
    """The rotating star: blends B and E towards the rotating dipole and
    -v x B near the surface."""
    x, y, z = pos
    r2 = torch.clamp(x * x + y * y + z * z, min=s["tiny"])
    r = torch.sqrt(r2)
    R, d = s["radius"], s["delta"][0]
    near = r < (1.5 if s["semantics"] == "cpu" else 2.0) * R
    bn = [s["b0"] * c for c in _dipole(s, x, y, z, s["omega"] * t)]
    p = (x, y, z)

    def blend(new, old, s_r, s_t):
        rn, ro = _dot(new, p) / r2, _dot(old, p) / r2
        return [rn * p[c] * s_r + ro * p[c] * (1 - s_r) + (new[c] - rn * p[c]) * s_t +
                (old[c] - ro * p[c]) * (1 - s_t) for c in range(3)]

    w = _shape(r, R - 4.0 * d, 0.5 * d)
    nb = blend(bn, B, w, w)
    v = [-s["omega"] * y, s["omega"] * x]
    en = [-v[1] * nb[2], v[0] * nb[2], -v[0] * nb[1] + v[1] * nb[0]]
    ne = blend(en, E, _shape(r, R, 0.25 * d), _shape(r, R, 0.5 * d))
    inside = r < 0.5 * R
    nb = [torch.where(inside, bn[c], nb[c]) for c in range(3)]
    ne = [torch.where(inside, en[c], ne[c]) for c in range(3)]
    return ([torch.where(near, ne[c], E[c]) for c in range(3)],
            [torch.where(near, nb[c], B[c]) for c in range(3)])


def _flat_steps(s, U):
    cpu = s["semantics"] == "cpu"
    dt, tau, tiny, dev = s["dt"], s["tau"], s["tiny"], U[0].device
    box = _box(s)
    X, Y, Z = (_axis(s, a) for a in range(3))
    lanes = 8 if s["f64"] else 16
    lane = ((torch.arange(s["N"][0], device=dev)) % lanes).double()
    planes = range(s["guard"][2], s["dims"][2] - s["guard"][2], 32)
    end = s["dims"][2] - s["guard"][2]
    dU = [torch.zeros_like(U[0][box]) for _ in range(7)]
    layer = any(m > 0 for m in s["pml"])
    x, y = X[box[2]][None, None, :], Y[box[1]][None, :, None]
    t = 0.0

    def boundary(E, B, P, z, tb, sl, un):
        if s["problem"]:
            E, B = _flat_star(s, E, B, (x, y, z), tb)
        if un is not None and layer:
            d = s["delta"]
            sig = _layer_sigma(s, (x, y, z), [s["pmllen"] * (d[a] if cpu else d[0]) for a in range(3)])
            E = [_relax(sig, E[c], un[c][sl], tiny) for c in range(3)]
            if cpu:
                bg = [s["b0"] * c for c in _dipole(s, x, y, z, 0.0)]
                on = sig > tiny
                sg = torch.where(on, sig, torch.ones_like(sig))
                e = torch.exp(-sg)
                B = [torch.where(on, bg[c] + e * (un[3 + c][sl] - bg[c]) + (1 - e) / sg *
                                 (B[c] - un[3 + c][sl]), B[c]) for c in range(3)]
            else:
                B = [_relax(sig, B[c], un[3 + c][sl], tiny) for c in range(3)]
                P = _relax(sig, P, un[6][sl], tiny)
        return E, B, P

    for _ in range(s["steps"]):
        Un = [u.clone() for u in U] if layer else None
        for i in range(5):
            new = [u.clone() for u in U]
            for k0 in planes:
                k1 = min(k0 + 32, end)
                sl = _box(s, None, 0, k0, k1)
                own = (slice(k0 - s["guard"][2], k1 - s["guard"][2]),)
                z = Z[k0:k1][:, None, None]

                def d(c, a):
                    return _d4(s, U[c], a, k0, k1)
                rotE = [d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)]
                rotB = [d(5, 1) - d(4, 2), d(3, 2) - d(5, 0), d(4, 0) - d(3, 1)]
                divE, divB = d(0, 0) + d(1, 1) + d(2, 2), d(3, 0) + d(4, 1) + d(5, 2)
                E, B, P = [u[sl] for u in U[:3]], [u[sl] for u in U[3:6]], U[6][sl]
                B2 = torch.clamp(_dot(B, B), min=tiny)
                chi, EB = B2 - _dot(E, E), _dot(E, B)
                E02 = 0.5 * (torch.sqrt(chi * chi + 4.0 * EB * EB) - chi) + B2
                Jp = (_dot(B, rotB) - _dot(E, rotE) + EB * s["damp_gamma"] / dt) / B2
                C = _cross(E, B)
                J = [divE / E02 * C[c] + Jp * B[c] for c in range(3)]
                gP = [d(6, a) for a in range(3)]
                if cpu:
                    # y and z are those of the point plus its SIMD lane's cells
                    rt = torch.sqrt(x ** 2 + (y + (lane * s["delta"][1])[None, None, :]) ** 2 +
                                    (z + (lane * s["delta"][2])[None, None, :]) ** 2)
                    gP = [g * _shape(rt, 3.0, 0.5) for g in gP]
                rhs = [dt * (rotB[c] - J[c]) for c in range(3)]
                rhs += [-dt * (rotE[c] + gP[c]) for c in range(3)]
                rhs.append(-P / tau - dt * s["ch2"] * divB)
                nu = []
                for c in range(7):
                    dU[c][own] = RK_A[i] * dU[c][own] + rhs[c]
                    nu.append(U[c][sl] + RK_B[i] * dU[c][own])
                En, Bn, Pn = _clamp(s, nu[:3], nu[3:6]), nu[3:6], nu[6]
                En, Bn, Pn = boundary(En, Bn, Pn, z, t + RK_C[i] * dt, sl, Un if i == 4 else None)
                for c in range(3):
                    new[c][sl], new[3 + c][sl] = En[c], Bn[c]
                new[6][sl] = Pn
            _wrap(s, new)
            U = new
        new = [u.clone() for u in U]
        for k0 in planes:
            k1 = min(k0 + 32, end)
            sl = _box(s, None, 0, k0, k1)
            nu = []
            for c in range(7):
                v = U[c][sl]
                if c < 6 or not cpu:
                    v = v + s["KOeps"] / 64.0 * sum(_d6(s, U[c], a, k0, k1) for a in range(3))
                nu.append(v)
            En, Bn, Pn = boundary(_clamp(s, nu[:3], nu[3:6]), nu[3:6], nu[6],
                                  Z[k0:k1][:, None, None], t + dt, sl, None)
            for c in range(3):
                new[c][sl], new[3 + c][sl] = En[c], Bn[c]
            new[6][sl] = Pn
        _wrap(s, new)
        U = new
        t += dt
    return U


# Kerr-Schild solver

def _cks(s, x, y, z):
    """Kerr-Schild r, lapse, shift, sqrt(gamma) and the 3-metric."""
    a, tiny = s["a"], s["tiny"]
    q = x * x + y * y + z * z - a * a
    r = torch.sqrt(0.5 * (q + torch.sqrt(torch.clamp(q * q + 4.0 * (a * z) ** 2, min=tiny))))
    den = torch.clamp(r ** 4 + a * a * z * z, min=tiny)
    H = 2.0 * r ** 3 / den
    l = [(r * x + a * y) / (r * r + a * a), (r * y - a * x) / (r * r + a * a), z / r]
    m = {"r": r, "l": l, "H": H, "sg": torch.sqrt(1.0 + H), "alpha": 1.0 / torch.sqrt(1.0 + H)}
    m["beta"] = [H / (1.0 + H) * v for v in l]
    return m


def _cks_lower(m, v):
    q = m["H"] * _dot(m["l"], v)
    return [v[c] + q * m["l"][c] for c in range(3)]


def _cks_raise(m, v):
    q = m["H"] / (1.0 + m["H"]) * _dot(m["l"], v)
    return [v[c] - q * m["l"][c] for c in range(3)]


def _gr_steps(s, U):
    dt, tiny = s["dt"], s["tiny"]
    box = _box(s)
    X, Y, Z = _axis(s, 0)[None, None, :], _axis(s, 1)[None, :, None], _axis(s, 2)[:, None, None]
    M = _cks(s, X, Y, Z)
    m = {k: ([c[box] for c in v] if isinstance(v, list) else v[box]) for k, v in M.items()}
    pos = (X[..., box[2]], Y[:, box[1]], Z[box[0]])
    dU = [torch.zeros_like(U[0][box]) for _ in range(7)]
    sg, r, shape = m["sg"], m["r"], _shape(m["r"], 5.0, 1.0)
    rh = 1.0 + math.sqrt(1.0 - s["a"] ** 2)
    outer = _layer_sigma(s, pos, [s["pmllen"] * s["delta"][0]] * 3)
    inner = s["sigpml"] * dt * torch.clamp((0.7 * rh - r) / (0.2 * rh), min=0.0) ** 3

    def lower(v):
        return _cks_lower(m, v)

    def put(U, vals):
        new = [u.clone() for u in U]
        for c in range(7):
            new[c][box] = vals[c]
        return new

    for _ in range(s["steps"]):
        Un = [u[box] for u in U]
        for i in range(5):
            D, B = U[:3], U[3:6]
            Dl, Bl = _cks_lower(M, D), _cks_lower(M, B)
            bB, bD = _cross(M["beta"], B), _cross(M["beta"], D)
            E = [M["alpha"] * Dl[c] + M["sg"] * bB[c] for c in range(3)]
            H = [M["alpha"] * Bl[c] - M["sg"] * bD[c] for c in range(3)]

            def curl(f):
                return [(_d4(s, f[2], 1) - _d4(s, f[1], 2)) / sg, (_d4(s, f[0], 2) - _d4(s, f[2], 0)) / sg,
                        (_d4(s, f[1], 0) - _d4(s, f[0], 1)) / sg]

            def div(f):
                return sum(_d4(s, f[a], a, w=M["sg"].expand_as(f[a])) for a in range(3)) / sg
            rotE, rotH, divD, divB = curl(E), curl(H), div(D), div(B)
            d, b, P = [u[box] for u in D], [u[box] for u in B], U[6][box]
            dl, bl, e = lower(d), lower(b), [u[box] for u in E]
            B2 = torch.clamp(_dot(b, bl), min=tiny)
            Jp = _dot(bl, rotH) - _dot(dl, rotE)
            C = _cross(e, bl)
            J = [(divD * C[c] / sg + Jp * b[c]) / B2 for c in range(3)]
            Pd = [_d4(s, U[6], a) for a in range(3)]
            Pu = _cks_raise(m, Pd)
            rhs = [dt * (rotH[c] - J[c]) for c in range(3)]
            rhs += [dt * (-rotE[c] + (-m["alpha"] * Pu[c] + m["beta"][c] * divB) * shape)
                    for c in range(3)]
            rhs.append(dt * (-m["alpha"] * divB + _dot(m["beta"], Pd)) - m["alpha"] * P / s["tau"])
            nu = []
            for c in range(7):
                dU[c] = RK_A[i] * dU[c] + rhs[c]
                nu.append(U[c][box] + RK_B[i] * dU[c])
            nu[:3] = _clamp(s, nu[:3], nu[3:6], lower, tiny)
            if i == 4:
                for c in range(6):
                    v = _relax(outer, nu[c], Un[c], tiny)
                    v = _relax(inner, v, Un[c], tiny)
                    nu[c] = torch.where(r < 0.01 * rh, torch.zeros_like(v), v)
            U = put(U, nu)
        nu = [u[box] + s["KOeps"] / 64.0 * sum(_d6(s, u, a) for a in range(3)) for u in U]
        nu[:3] = _clamp(s, nu[:3], nu[3:6], lower, tiny)
        U = put(U, nu)
    return U


# log-spherical solver (x = ln r, y = theta)

def _sph_steps(s, U):
    dt, tiny = s["dt"], s["tiny"]
    box = _box(s)
    r, th = torch.exp(_axis(s, 0))[None, None, :], _axis(s, 1)[None, :, None]
    sn = torch.sin(th)
    g11, g33 = (r * r).expand_as(U[0]), (r * sn) ** 2
    sq = r ** 3 * sn.abs()
    rb, sb, thb = r[..., box[2]], sn[:, box[1]], th[:, box[1]]
    a11, a33 = rb * rb, (rb * sb) ** 2
    sg = torch.clamp(rb ** 3 * sb.abs(), min=tiny)
    dU = [torch.zeros_like(U[0][box]) for _ in range(7)]
    xh = s["lower"][0] + s["size"][0] - s["pml"][0] * s["delta"][0]
    sig = s["sigpml"] * torch.clamp((rb - math.exp(xh)) / s["pmllen"], min=0.0) ** 3
    sig = sig.expand_as(dU[0])
    g, d1 = s["guard"][1], s["dims"][1]

    def lower(v):
        return [a11 * v[0], a11 * v[1], a33 * v[2]]

    def axis(U):
        i = slice(s["guard"][0], s["dims"][0] - s["guard"][0])
        for j, inw in ((g, 1), (d1 - g, -1)):
            for c in range(7):
                U[c][:, j, i] = U[c][:, j + inw, i] if c in (0, 3, 6) else 0.0
            for n in range(1, 4):
                for c, par in enumerate((1, -1, -1, 1, -1, -1)):
                    U[c][:, j - inw * n, i] = par * U[c][:, j + inw * n, i]

    def star(E, B):
        R, d = s["radius"], s["delta"][0]
        bn = [s["b0"] * 2.0 * torch.cos(thb) / rb ** 3, s["b0"] * sb / rb ** 3]
        v = s["omega"] * rb * sb
        en = [v * bn[1], -v * bn[0]]
        surf = ((rb - R).abs() < 0.5 * d).expand_as(E[0])
        inside = (~surf & (rb < R - tiny)).expand_as(E[0])
        both, zero = surf | inside, torch.zeros_like(E[0])
        w = torch.where
        B = [w(both, bn[0] / rb, B[0]), w(inside, bn[1] / rb, B[1]), w(inside, zero, B[2])]
        E = [w(inside, en[0] / rb, E[0]), w(both, en[1] / rb, E[1]), w(both, zero, E[2])]
        return E, B

    def put(U, vals):
        new = [u.clone() for u in U]
        for c in range(7):
            new[c][box] = vals[c]
        axis(new)
        return new

    U = [u.clone() for u in U]
    axis(U)
    for _ in range(s["steps"]):
        Un = [u[box] for u in U]
        for i in range(5):
            def dx(f, w):
                return _d4(s, f, 0, w=w.expand_as(f))

            def dy(f, w):
                return _d4(s, f, 1, w=w.expand_as(f))

            def curl(f):
                return [dy(f[2], g33) / sg, -dx(f[2], g33) / sg, (dx(f[1], g11) - dy(f[0], g11)) / sg]

            def div(f):
                return (dx(f[0], sq) + dy(f[1], sq)) / sg
            rotE, rotB, divE, divB = curl(U[:3]), curl(U[3:6]), div(U[:3]), div(U[3:6])
            E, B, P = [u[box] for u in U[:3]], [u[box] for u in U[3:6]], U[6][box]
            el, bl = lower(E), lower(B)
            B2 = torch.clamp(_dot(B, bl), min=tiny)
            chi, EB = B2 - _dot(E, el), _dot(E, bl)
            E02 = 0.5 * (torch.sqrt(chi * chi + 4.0 * EB * EB) - chi) + B2
            Jp = (_dot(bl, rotB) - _dot(el, rotE) + s["damp_gamma"] / dt * EB) / B2
            C = _cross(el, bl)
            J = [divE / sg / E02 * C[c] + Jp * B[c] for c in range(3)]
            rhs = [dt * (rotB[c] - J[c]) for c in range(3)]
            rhs += [-dt * (rotE[0] + _d4(s, U[6], 0) / a11), -dt * (rotE[1] + _d4(s, U[6], 1) / a11),
                    -dt * rotE[2], -dt * s["ch2"] * divB - P / s["tau"]]
            nu = []
            for c in range(7):
                dU[c] = RK_A[i] * dU[c] + rhs[c]
                nu.append(U[c][box] + RK_B[i] * dU[c])
            nu[:3] = _clamp(s, nu[:3], nu[3:6], lower)
            nu[:3], nu[3:6] = star(nu[:3], nu[3:6])
            if i == 4:
                nu[:6] = [_relax(sig, nu[c], Un[c], tiny) for c in range(6)]
            U = put(U, nu)
        w = sq.expand_as(U[0])
        nu = [u[box] + s["KOeps"] / 64.0 * (_d6(s, u, 0, w=w) + _d6(s, u, 1, w=w)) / sg for u in U]
        nu[:3] = _clamp(s, nu[:3], nu[3:6], lower)
        nu[:3], nu[3:6] = star(nu[:3], nu[3:6])
        U = put(U, nu)
    return U


# cylindrical solver (x = R, y = z; components R, z, phi)

def _cyl_steps(s, U):
    dt, tiny = s["dt"], s["tiny"]
    box = _box(s)
    h, g = s["delta"][0], s["guard"][0]
    Rf = _axis(s, 0)[None, None, :].expand_as(U[0])
    R, z = Rf[box][:, :1], _axis(s, 1)[None, :, None][:, box[1]]
    on_axis = R.abs() < 0.25 * h
    Rd = torch.where(R.abs() < tiny, torch.full_like(R, tiny), R)
    dU = [torch.zeros_like(U[0][box]) for _ in range(7)]
    r2 = torch.clamp(R * R + z * z, min=tiny)
    r = torch.sqrt(r2)
    xh = s["lower"][0] + s["size"][0] - s["pml"][0] * h
    sig = s["sigpml"] * torch.clamp((R - xh) / (s["pmllen"] * h), min=0.0) ** 3
    sig = sig + _layer_sigma(s, (R, z), [s["pmllen"] * h] * 2, axes=(1,))
    sig = sig.expand_as(dU[0])

    def clamp(v):
        # components (R, z, phi): the products do not see the handedness
        return _clamp(s, v[:3], v[3:6])

    def star(v):
        rad = s["radius"]
        m = s["b0"] * rad ** 3
        bn = [m * 3.0 * R * z / r2 / (r ** 3 + tiny), m * (3.0 * z * z / r2 - 1.0) / (r ** 3 + tiny), 0.0]
        near, inside = (r < 2.0 * rad).expand_as(v[0]), (r < 0.5 * rad).expand_as(v[0])

        def blend(new, old, s_r, s_t):
            rn, ro = (new[0] * R + new[1] * z) / r2, (old[0] * R + old[1] * z) / r2
            return [rn * p * s_r + ro * p * (1 - s_r) + (new[c] - rn * p) * s_t +
                    (old[c] - ro * p) * (1 - s_t) for c, p in ((0, R), (1, z))]
        w = _shape(r, rad - 4.0 * h, 0.5 * h)
        nb = blend(bn, v[3:6], w, w) + [v[5] * (1 - w)]
        en = [-s["omega"] * R * v[4], s["omega"] * R * v[3], 0.0]
        w1, w2 = _shape(r, rad, 0.25 * h), _shape(r, rad, 0.5 * h)
        ne = blend(en, v[:3], w1, w2) + [v[2] * (1 - w2)]
        out = []
        for c, (core, rim) in enumerate(zip(en + bn, ne + nb)):
            core = core if torch.is_tensor(core) else torch.zeros_like(v[c])
            out.append(torch.where(near, torch.where(inside, core, rim), v[c]))
        return out + [v[6]]

    def put(U, v, un):
        new = [u.clone() for u in U]
        v = [a.clone() for a in v]
        parity = (-1, 1, -1, -1, 1, -1, 1)
        for c in range(7):
            for n in range(1, 4):  # the columns beyond the axis mirror those inside
                new[c][:, box[1], g - n] = parity[c] * v[c][:, :, n]
            v[c][:, :, 0] = v[c][:, :, 1] if parity[c] > 0 else 0.0
        v = star(v)
        if un is not None:
            v = [_relax(sig, v[c], un[c], tiny) for c in range(6)] + [v[6]]
        for c in range(7):
            new[c][box] = v[c]
        return new

    for _ in range(s["steps"]):
        Un = [u[box] for u in U]
        for i in range(5):
            def drr(f):
                return torch.where(on_axis, 2.0 * _d4(s, f, 0), _d4(s, f, 0, w=Rf) / Rd)

            def curl(f):
                return [-_d4(s, f[2], 1), drr(f[2]), _d4(s, f[0], 1) - _d4(s, f[1], 0)]

            def div(f):
                return drr(f[0]) + _d4(s, f[1], 1)
            rotE, rotB, divE, divB = curl(U[:3]), curl(U[3:6]), div(U[:3]), div(U[3:6])
            E, B, P = [u[box] for u in U[:3]], [u[box] for u in U[3:6]], U[6][box]
            B2 = torch.clamp(_dot(B, B), min=tiny)
            Jp = _dot(B, rotB) - _dot(E, rotE)
            C = [E[2] * B[1] - E[1] * B[2], E[0] * B[2] - E[2] * B[0], E[1] * B[0] - E[0] * B[1]]
            J = [(divE * C[c] + Jp * B[c]) / B2 for c in range(3)]
            rhs = [dt * (rotB[c] - J[c]) for c in range(3)]
            rhs += [-dt * (rotE[0] + _d4(s, U[6], 0)), -dt * (rotE[1] + _d4(s, U[6], 1)), -dt * rotE[2],
                    -dt * s["ch2"] * divB - P / s["tau"]]
            nu = []
            for c in range(7):
                dU[c] = RK_A[i] * dU[c] + rhs[c]
                nu.append(U[c][box] + RK_B[i] * dU[c])
            nu[:3] = clamp(nu)
            U = put(U, nu, Un if i == 4 else None)
        nu = [u[box] + s["KOeps"] / 64.0 * (_d6(s, u, 0) + _d6(s, u, 1)) for u in U]
        nu[:3] = clamp(nu)
        U = put(U, nu, None)
    return U


# staggered solver

EDGE = ((1, 0, 0), (0, 1, 0), (0, 0, 1))  # half-cell offsets of E_x, E_y, E_z
FACE = ((0, 1, 1), (1, 0, 1), (1, 1, 0))  # and of B_x, B_y, B_z
VERTEX = (0, 0, 0)


def _shift(f, a, n):
    """f at the point n cells up along axis a (values that wrap around are
    guard points that nothing reads)."""
    return torch.roll(f, -n, 2 - a)


def _interp(f, at, to):
    """Mean of f's values around the position `to` along every axis where it
    is half a cell off."""
    for a in range(3):
        if at[a] != to[a]:
            f = 0.5 * (f + _shift(f, a, -1 if at[a] else 1))
    return f


def _yee_steps(s, U):
    dt, tiny = s["dt"], s["tiny"]
    box = _box(s)
    E, B = [u.clone() for u in U[:3]], [u.clone() for u in U[3:6]]

    def d(f, a, n):  # forward (1) or backward (-1) difference
        return n * (_shift(f, a, n) - f) / s["delta"][a]

    def curl(f, n):
        return [d(f[2], 1, n) - d(f[1], 2, n), d(f[0], 2, n) - d(f[2], 0, n),
                d(f[1], 0, n) - d(f[0], 1, n)]
    for _ in range(s["steps"]):
        En, Bn = [e.clone() for e in E], [b.clone() for b in B]
        for sub, (c1, c2, c3) in enumerate(((1.0, 0.0, 1.0), (0.75, 0.25, 0.25),
                                            (1 / 3.0, 2 / 3.0, 2 / 3.0))):
            rho = torch.zeros_like(E[0])
            rho[box] = sum(d(E[a], a, -1) for a in range(3))[box]
            cE, cB = curl(E, 1), curl(B, -1)
            Es, Bs = [e.clone() for e in E], [b.clone() for b in B]
            for c in range(3):
                e = [_interp(E[a], EDGE[a], EDGE[c]) for a in range(3)]
                b = [_interp(B[a], FACE[a], EDGE[c]) for a in range(3)]
                J = _interp(rho, VERTEX, EDGE[c]) * _cross(e, b)[c] / (_dot(b, b) + tiny)
                Es[c][box] = (c1 * En[c] + c2 * E[c] + c3 * dt * (cB[c] - J))[box]
                Bs[c][box] = (c1 * Bn[c] + c2 * B[c] - c3 * dt * cE[c])[box]
            E = [e.clone() for e in Es]
            for c in range(3):
                e = [_interp(Es[a], EDGE[a], EDGE[c]) for a in range(3)]
                b = [_interp(Bs[a], FACE[a], EDGE[c]) for a in range(3)]
                e2, b2 = _dot(e, e) + tiny, _dot(b, b) + tiny
                v = Es[c]
                if sub == 2:
                    v = v - _dot(e, b) * b[c] / b2
                v = torch.where(e2 > b2, torch.sqrt(b2 / e2) * v, v)
                E[c][box] = v[box]
            B = Bs
            _wrap(s, E + B)
    return E + B + [U[6]]


# ----------------------------------------------------- the warm-start network

UNET = ((16, 16), (16, 16), (16, 32), (32, 32), (48, 16), (16, 16))  # channels in, out


def _unet_inputs(case, seed):
    """Weights, a batch of samples, their targets and the mask of trained
    points (those outside a star in the middle of the box)."""
    gen = torch.Generator().manual_seed(1000003 + seed)
    dev, n, m = _device(), case["samples"], case["side"]
    w = [(torch.randn(k, 27, c, generator=gen) * math.sqrt(2.0 / (27 * c))).to(dev) for c, k in UNET]
    b = [(0.05 * torch.randn(k, generator=gen)).to(dev) for _, k in UNET]
    gpu = torch.Generator(device=dev).manual_seed(2000003 + seed)
    u = torch.linspace(-1.0, 1.0, m, device=dev)
    z, y, x = torch.meshgrid(u, u, u, indexing="ij")
    basis = torch.stack([x, y, z, torch.sin(3 * x), torch.cos(3 * y), torch.sin(3 * z), x * y, y * z], -1)
    mix = torch.randn(n, 8, 32, generator=gpu, device=dev)
    smooth = torch.einsum("zyxi,nic->nzyxc", basis, mix)
    inputs = (smooth[..., :16] + 0.1 * torch.randn(n, m, m, m, 16, generator=gpu, device=dev))
    target = torch.tanh(smooth[..., 16:]).contiguous()
    mask = (x * x + y * y + z * z > 0.1).float().expand(n, m, m, m).contiguous()
    return w, b, inputs.to(torch.bfloat16).contiguous(), target, mask


def _prepare_unet(case, seed):
    from coffee_b200.surrogate import UNet

    w, b, x, target, mask = _unet_inputs(case, seed)
    net = UNet(seed=0)
    for L, wi, bi in zip(net.layers, w, b):
        L.w.copy_(wi)
        L.b.copy_(bi)
        L.refresh()
    return {"kind": "unet", "net": net, "x": x, "target": target, "mask": mask, "lr": 2e-3}


def _exact_unet(case, seed):
    import torch.nn.functional as F

    w, b, x, target, mask = _unet_inputs(case, seed)
    W = [wi.double().reshape(k, 3, 3, 3, c).permute(0, 4, 1, 2, 3).contiguous().requires_grad_()
         for wi, (c, k) in zip(w, UNET)]
    bias = [bi.double().requires_grad_() for bi in b]
    count = float(mask.double().sum()) * 16
    total, outs = 0.0, []
    for n in range(case["samples"]):
        def conv(i, v):
            return F.conv3d(v, W[i], bias[i], padding=1)

        def leaky(v):
            return F.leaky_relu(v, 0.1)
        v = x[n].double().permute(3, 0, 1, 2)[None]
        a2 = leaky(conv(1, leaky(conv(0, v))))
        a4 = leaky(conv(3, leaky(conv(2, F.avg_pool3d(a2, 2)))))
        up = F.interpolate(a4, scale_factor=2, mode="nearest")
        out = conv(5, leaky(conv(4, torch.cat([up, a2], 1))))[0].permute(1, 2, 3, 0)
        loss = ((out - target[n].double()) ** 2 * mask[n][..., None].double()).sum() / count
        loss.backward()
        total = total + loss.detach()
        outs.append(out.detach())
    gw = [g.grad.permute(0, 2, 3, 4, 1).reshape(g.shape[0], 27, g.shape[1]) for g in W]
    return {"out": torch.stack(outs), "loss": total, "gw": gw, "gb": [g.grad for g in bias]}

"""Timed workloads of the point-vortex backend, called through its public entry points.

A case is a dict of plain values; its "kind" says which call is timed:

    rk4         a state goes up, a run of RK4 steps is made on the device, the state comes back
    dopri5      the same with adaptive DOPRI5 steps, each followed by the close-dipole events
    evaluate    velocities of host arrays (VelocityKernel.evaluate)
    range       velocities of a range of targets of host arrays (one rank's share of a population)
    velocity    velocities of the device-resident state
    invariants  the conserved quantities of the device-resident state (one diagnostics row)
    rows        one trajectory frame as text
    ensemble    a batch of uneven simulations: admitted, advanced to a step budget, read, released

Populations are seeded: uniform positions where the call meets close pairs in earnest, and a jittered
lattice (a population whose close pairs are gone) where a fixed step or a wall needs it.
"""
import math

import numpy as np
import torch

from pointvortex_b200 import (DeviceDipoleManager, DiskKernel, InfinitePlaneKernel,
                              PeriodicBoxKernel, VelocityField, VortexSystem)
from pointvortex_b200 import _lib
from pointvortex_b200.batch import Batch, geometry_params

TWO_PI = 2.0 * math.pi
PRECISION = {"fp64": _lib.PRECISION_FP64, "fp32c": _lib.PRECISION_FP32C}


def listed():
    return [
        # the smallest: a thousand vortices in the plane between two output times, 100 RK4 steps
        dict(name="plane_rk4_n1024", kind="rk4", geometry="infinite", n=1024, precision="fp64",
             core=0.0, layers=8, dt=1e-4, steps=100),
        # a few hundred vortices in a disk, adaptive, an odd size: launches and latency
        dict(name="disk_dopri5_n301", kind="dopri5", geometry="disk", n=301, precision="fp64",
             core=0.0, layers=8, dt=2e-3, rtol=1e-9, atol=1e-12, distance=1e-3, steps=8),
        # the everyday run: a doubly periodic box, adaptive, with dipole events
        dict(name="periodic_dopri5_n4096", kind="dopri5", geometry="periodic", n=4096,
             precision="fp64", core=0.0, layers=8, dt=3e-6, rtol=1e-9, atol=1e-12, distance=1e-3,
             steps=8),
        # a large disk under a fixed step
        dict(name="disk_rk4_n16384", kind="rk4", geometry="disk", n=16384, precision="fp64",
             core=0.0, layers=8, dt=1e-5, steps=2),
        # the drop-in call of a host program that keeps its own state, odd size, with a core radius
        dict(name="plane_evaluate_n8191", kind="evaluate", geometry="infinite", n=8191,
             precision="fp64", core=1e-3, layers=8),
        # one of four ranks' targets of a periodic population
        dict(name="periodic_range_n12000", kind="range", geometry="periodic", n=12000,
             precision="fp64", core=0.0, layers=8, begin=3000, end=6001),
        # large populations on the device, one evaluation: plane (ragged size) and box (the largest)
        dict(name="plane_velocity_n50001", kind="velocity", geometry="infinite", n=50001,
             precision="fp64", core=0.0, layers=8),
        dict(name="periodic_velocity_n65536", kind="velocity", geometry="periodic", n=65536,
             precision="fp64", core=0.0, layers=8),
        # the FP32-compensated form in an adaptive run
        dict(name="periodic_fp32c_dopri5_n16384", kind="dopri5", geometry="periodic", n=16384,
             precision="fp32c", core=0.0, layers=8, dt=8e-7, rtol=1e-6, atol=1e-9, distance=1e-4,
             steps=4),
        # an ensemble of uneven sizes and mixed geometry
        dict(name="ensemble_s96", kind="ensemble", sims=96, smallest=64, largest=4096,
             precision="fp64", dt=1e-3, rtol=1e-8, atol=1e-10, steps=3),
        # diagnostics of a large periodic population
        dict(name="periodic_invariants_n16384", kind="invariants", geometry="periodic", n=16384,
             precision="fp64", core=0.0, layers=8),
        # a trajectory frame
        dict(name="trajectory_rows_n16384", kind="rows", geometry="disk", n=16384,
             precision="fp64", core=0.0, layers=8),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rk4", "dopri5", "dopri5", "evaluate", "range", "velocity", "velocity",
                       "ensemble", "invariants", "rows"])
    if kind == "ensemble":
        c = dict(kind=kind, sims=rng.randint(16, 96), smallest=rng.randint(48, 128),
                 largest=_log_uniform(rng, 600, 4096),
                 precision=rng.choice(["fp64", "fp64", "fp32c"]), dt=1e-3, rtol=1e-8,
                 atol=1e-10, steps=rng.randint(2, 4))
        if c["precision"] == "fp32c":  # tolerances that FP32 terms can meet, a bounded step
            c.update(dt=1e-5, dtmax=1e-5, rtol=1e-5, atol=1e-7)
        return c
    geometry = rng.choice(["infinite", "periodic", "periodic", "disk"])
    c = dict(kind=kind, geometry=geometry, precision="fp64",
             core=rng.choice([0.0, 0.0, 1e-3]) if geometry == "infinite" else 0.0,
             layers=rng.choice([8, 8, 8, 8, 16, 4]) if geometry == "periodic" else 8)
    if kind == "rk4":
        c.update(n=_log_uniform(rng, 64, 16384), dt=1e-5, steps=rng.randint(1, 20),
                 precision=rng.choice(["fp64", "fp64", "fp32c"]))
        if c["precision"] == "fp32c":
            c["dt"] = 2e-6
        if c["n"] > 4000:
            c["steps"] = 1 + c["steps"] % 4
    elif kind == "dopri5":
        c.update(n=_log_uniform(rng, 128, 16384), steps=rng.randint(2, 8), distance=1e-3,
                 rtol=1e-9, atol=1e-12, precision=rng.choice(["fp64", "fp64", "fp32c"]))
        # a first step that the controller has to shorten once or a few times
        c["dt"] = (0.6 / c["n"] if geometry == "disk"
                   else (5.0 if geometry == "infinite" else 50.0) / c["n"] ** 2)
        if c["precision"] == "fp32c":  # tolerances that FP32 terms can meet, a bounded step
            c.update(n=_log_uniform(rng, 2048, 16384), dt=2e-6, dtmax=2e-6, rtol=1e-6, atol=1e-9,
                     distance=1e-4)
        if c["n"] > 4000:
            c["steps"] = 2 + c["steps"] % 3
    elif kind in ("evaluate", "range"):
        c.update(n=_log_uniform(rng, 256, 24000))
        if kind == "range":
            ranks = rng.randint(2, 8)
            rank = rng.randrange(ranks)
            c.update(begin=c["n"] * rank // ranks, end=c["n"] * (rank + 1) // ranks)
    elif kind == "velocity":
        c.update(n=_log_uniform(rng, 512, 60000))
    elif kind == "invariants":
        c.update(n=_log_uniform(rng, 256, 20000))
    else:
        c.update(n=_log_uniform(rng, 256, 40000))
    return c


# -- inputs --------------------------------------------------------------------------------------
def _circulations(n, rng, geometry):
    if geometry != "disk" and n % 2 == 0:
        g = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
        rng.shuffle(g)
        return g
    g = rng.standard_normal(n)
    if geometry == "periodic":
        g -= g.mean()
    return g


def _population(geometry, n, rng, spaced):
    """(x, y, circulation) in [-1, 1]^2, the 2 pi box or the unit disk. spaced: no close pairs."""
    g = _circulations(n, rng, geometry)
    if geometry == "disk":
        if spaced:  # a sunflower spiral, jittered by a fifth of its spacing
            i = rng.permutation(n) + 0.5
            r, th = 0.9 * np.sqrt(i / n), i * (math.pi * (3.0 - math.sqrt(5.0)))
            h = 0.18 * math.sqrt(math.pi / n)
            return (r * np.cos(th) + rng.uniform(-h, h, n), r * np.sin(th) + rng.uniform(-h, h, n), g)
        r, th = 0.95 * np.sqrt(rng.random(n)), TWO_PI * rng.random(n)
        return r * np.cos(th), r * np.sin(th), g
    half = math.pi if geometry == "periodic" else 1.0
    if spaced:  # a square lattice, jittered by a fifth of its spacing
        side = math.isqrt(n - 1) + 1
        h = 2.0 * half / side
        cell = rng.permutation(side * side)[:n]
        x = -half + (cell % side + 0.5 + rng.uniform(-0.2, 0.2, n)) * h
        y = -half + (cell // side + 0.5 + rng.uniform(-0.2, 0.2, n)) * h
        return x, y, g
    return rng.uniform(-half, half, n), rng.uniform(-half, half, n), g


def _state(case, seed):
    rng = np.random.default_rng([seed, case["n"]])
    spaced = case["kind"] == "rk4" or (case["kind"] == "dopri5" and case["geometry"] == "disk")
    return _population(case["geometry"], case["n"], rng, spaced)


def _members(case, seed):
    """The ensemble's simulations: geometry in turn, sizes log-uniform and even (by the case alone)."""
    sizes = np.random.default_rng([case["sims"], case["smallest"], case["largest"]])
    rng = np.random.default_rng([seed, 11])
    members = []
    for k in range(case["sims"]):
        n = int(math.exp(sizes.uniform(math.log(case["smallest"]), math.log(case["largest"]))))
        n += n % 2
        geometry = ("infinite", "periodic", "disk")[k % 3]
        members.append((geometry, _population(geometry, n, rng, geometry == "disk")))
    return members


def _kernel(case):
    kw = dict(precision=PRECISION[case["precision"]])
    if case["geometry"] == "infinite":
        return InfinitePlaneKernel(case["core"], **kw)
    if case["geometry"] == "periodic":
        return PeriodicBoxKernel(TWO_PI, TWO_PI, case["layers"], **kw)
    return DiskKernel(1.0, **kw)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = _members(case, seed)
        total = sum(st[0].size for _, st in members)
        return dict(case=case, members=members,
                    params=[geometry_params(g, precision=case["precision"]) for g, _ in members],
                    batch=Batch(total + 256 * (len(members) + 1), len(members),
                                max_steps=case["steps"], partial_factor=40))
    x, y, g = _state(case, seed)
    s = dict(case=case, kernel=_kernel(case), system=VortexSystem(x, y, g))
    if case["kind"] == "dopri5":
        s["dipoles"] = DeviceDipoleManager(s["kernel"], removal=True, distance=case["distance"])
    if case["kind"] in ("velocity", "invariants"):
        s["kernel"].uploadDeviceState(s["system"])
    if case["kind"] == "rows":
        # a population in an order of the seed's: every frame has the same number of bytes
        order = np.random.default_rng(seed).permutation(x.size)
        x, y, g = (a[order] for a in _state(case, 0))
        u, v = 30.0 * np.random.default_rng(5).standard_normal((2, x.size))[:, order]
        s.update(system=VortexSystem(x, y, g), velocity=VelocityField(u, v))
    return s


# -- one pass ------------------------------------------------------------------------------------
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "ensemble":
        return _run_ensemble(state)
    k, system = state["kernel"], state["system"]
    if kind == "rk4":
        k.uploadDeviceState(system)
        k.rk4Advance(c["dt"], c["steps"])
        after = VortexSystem(system.x, system.y, system.circulation)
        k.downloadDeviceState(after)
        return [after.x, after.y]
    if kind == "dopri5":
        # the step sizes and the error estimate are the integrator's own: they show in the state and
        # in the rejections (the estimate itself is a difference of nearly equal numbers)
        k.uploadDeviceState(system)
        dt, rejected, events = c["dt"], 0, 0
        for _ in range(c["steps"]):
            r = k.deviceDopri5Step(dt, c["atol"], c["rtol"], 1e-12,
                                   c.get("dtmax", 0.1))
            dt = r.suggestedTimeStep
            rejected += r.rejectedSteps
            events += state["dipoles"].process()
        after = k.downloadDeviceSystem()
        out = np.zeros((3, system.size()))  # events make the population smaller
        out[:, :after.size()] = after.x, after.y, after.circulation
        return [out[0], out[1], out[2], rejected, events]
    if kind == "evaluate":
        f = k.evaluate(system)
        return [f.x, f.y]
    if kind == "range":
        f = k.evaluateRange(system.x, system.y, system.circulation, None, c["begin"], c["end"])
        return [f.x, f.y]
    if kind == "velocity":
        f = k.evaluateDeviceState()
        return [f.x, f.y]
    if kind == "invariants":
        i = k.stateInvariants()
        return np.array([i.circulation, i.linearImpulseX, i.linearImpulseY, i.angularImpulse,
                         i.hamiltonian])
    text = k.formatTrajectoryHost(0.37, 17, system, state["velocity"])
    return np.frombuffer(text, dtype=np.uint8)


def _run_ensemble(state):
    c, b = state["case"], state["batch"]
    ids = [b.add(p, *st, 1.0, dt=c["dt"], atol=c["atol"], rtol=c["rtol"], dtmax=c.get("dtmax", 0.1))
           for p, (_, st) in zip(state["params"], state["members"])]
    b.run()
    xs, ys, accepted, rejected = [], [], [], []
    for sid in ids:
        info = b.info(sid)
        x, y = b.result(sid)
        xs.append(x)
        ys.append(y)
        accepted.append(info.acceptedSteps)
        rejected.append(info.rejectedSteps)
    for sid in ids:
        b.release(sid)
    return [np.concatenate(xs), np.concatenate(ys), np.array(accepted), np.array(rejected)]


# -- what a pass cannot do without ---------------------------------------------------------------
# Operations of one ordered pair (fused multiply-add two, a division or a function one): the plane 11;
# the disk 33 with its image; the box 50, half of a doubly periodic term that serves both vortices.
FLOPS = {"infinite": 11.0, "disk": 33.0, "periodic": 50.0}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        lo, hi = math.log(case["smallest"]), math.log(case["largest"])
        mean_n = (math.exp(hi) - math.exp(lo)) / (hi - lo)
        mean_n2 = (math.exp(2 * hi) - math.exp(2 * lo)) / (2 * (hi - lo))
        evals = 6.0 * case["steps"] + 1.0
        mean_flops = sum(FLOPS.values()) / 3.0
        return {"bytes": 40.0 * case["sims"] * mean_n,
                "flops": evals * case["sims"] * mean_n2 * mean_flops}
    n, f = float(case["n"]), FLOPS[case["geometry"]]
    if kind == "rk4":
        return {"bytes": 40.0 * n, "flops": 4.0 * case["steps"] * n * n * f}
    if kind == "dopri5":
        return {"bytes": 48.0 * n, "flops": (6.0 * case["steps"] + 1.0) * n * n * f}
    if kind == "range":
        targets = float(case["end"] - case["begin"])
        return {"bytes": 24.0 * n + 16.0 * targets, "flops": targets * n * f}
    if kind in ("evaluate", "velocity"):
        return {"bytes": 40.0 * n, "flops": n * n * f}
    if kind == "invariants":
        return {"bytes": 24.0 * n, "flops": 0.5 * n * n * f}
    return {"bytes": 40.0 * n + 127.0 * n, "flops": 0.0}


# -- the reference formulas in 64 bits -----------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _wrap(d):
    return d - TWO_PI * torch.round(d / TWO_PI)


def _velocity(case, x, y, g, begin=0, end=None):
    """Velocities of targets [begin, end): the reference's sums, term by term."""
    n = x.numel()
    end = n if end is None else end
    geometry, layers = case["geometry"], case.get("layers", 8)
    eps2 = case.get("core", 0.0) ** 2
    us, vs = [], []
    rows = max(1, min(end - begin, (1 << 25) // max(n, 1)))
    for t0 in range(begin, end, rows):
        t1 = min(t0 + rows, end)
        dx, dy = x[t0:t1, None] - x[None, :], y[t0:t1, None] - y[None, :]
        own = torch.zeros_like(dx, dtype=torch.bool)
        own[torch.arange(t1 - t0, device=x.device), torch.arange(t0, t1, device=x.device)] = True
        if geometry == "periodic":
            dx, dy = _wrap(dx), _wrap(dy)
            sx2, sy2 = torch.sin(0.5 * dx) ** 2, torch.sin(0.5 * dy) ** 2
            su, sv = torch.zeros_like(dx), torch.zeros_like(dx)
            for m in range(-min(layers, 6), min(layers, 6) + 1):
                for total, d, s2 in ((su, dx, sy2), (sv, dy, sx2)):
                    a = d - TWO_PI * m
                    term = 0.5 / (torch.sinh(0.5 * a) ** 2 + s2)
                    term = torch.where(a.abs() > 40.0, 0.0, term)
                    total += torch.where(own, 0.0, term)
            c = (0.5 / TWO_PI) * g
            u = -((torch.sin(dy) * su) @ c)
            v = (torch.sin(dx) * sv) @ c
        else:
            c = g / TWO_PI
            inv = torch.where(own, 0.0, 1.0 / (dx * dx + dy * dy + eps2))
            u = -((dy * inv) @ c)
            v = (dx * inv) @ c
            if geometry == "disk":
                tx, ty = x[t0:t1, None], y[t0:t1, None]
                a = 1.0 - (tx * x[None, :] + ty * y[None, :])
                b = ty * x[None, :] - tx * y[None, :]
                den = a * a + b * b
                u += ((b * x[None, :] - a * y[None, :]) / den) @ c
                v += ((a * x[None, :] + b * y[None, :]) / den) @ c
        us.append(u)
        vs.append(v)
    return torch.cat(us), torch.cat(vs)


_A = [[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
      [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
      [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
      [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_B4 = [5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40]


def _dopri5(case, x, y, g, steps, distance=None):
    """(x, y, g, accepted, rejected, events) after `steps` accepted steps from case["dt"], fewer
    when a stage leaves the disk."""
    dt, k0, rejected, events = case["dt"], None, 0, 0
    for accepted in range(steps):
        while True:
            ks = [k0 if k0 is not None else _velocity(case, x, y, g)]
            for s in range(1, 7):
                px = x + dt * sum(a * k[0] for a, k in zip(_A[s], ks))
                py = y + dt * sum(a * k[1] for a, k in zip(_A[s], ks))
                if case["geometry"] == "disk" and float((px * px + py * py).max()) >= 1.0:
                    return x, y, g, accepted, rejected, events
                ks.append(_velocity(case, px, py, g))
            err = 0.0
            for at, new, part in ((x, px, 0), (y, py, 1)):
                e = dt * sum((b5 - b4) * k[part] for b5, b4, k in zip(_A[6] + [0.0], _B4, ks))
                scale = case["atol"] + case["rtol"] * torch.maximum(at.abs(), new.abs())
                err = max(err, float((e.abs() / scale).max()))
            factor = 5.0 if err == 0.0 else min(5.0, max(0.2, 0.9 * err ** -0.2))
            suggested = min(case.get("dtmax", 0.1), max(1e-12, dt * factor))
            if err <= 1.0:
                break
            rejected += 1
            k0 = ks[0]
            dt = max(1e-12, min(suggested, 0.9 * dt))
        x, y, k0, dt = px, py, ks[6], suggested
        if distance is not None:
            keep, found = _without_dipoles(case, x, y, g, distance)
            if found:
                x, y, g, k0 = x[keep], y[keep], g[keep], None
                events += found
    return x, y, g, steps, rejected, events


def _without_dipoles(case, x, y, g, distance):
    """(indices kept, events): opposite pairs closer than distance, and in the disk vortices
    closer than it to their image, closest first, each vortex once."""
    n, found = x.numel(), []
    rows = max(1, (1 << 25) // n)
    for t0 in range(0, n, rows):
        dx, dy = x[t0:t0 + rows, None] - x[None, :], y[t0:t0 + rows, None] - y[None, :]
        if case["geometry"] == "periodic":
            dx, dy = _wrap(dx), _wrap(dy)
        d2 = dx * dx + dy * dy
        hit = (d2 < distance * distance) & (g[t0:t0 + rows, None] * g[None, :] < 0.0)
        for i, j in hit.nonzero().tolist():
            if t0 + i < j:
                found.append((float(d2[i, j]), t0 + i, j))
    if case["geometry"] == "disk":
        r2 = x * x + y * y
        i2 = ((1.0 - r2) / torch.sqrt(r2)) ** 2
        found += [(float(i2[i]), i, n) for (i,) in (i2 < distance * distance).nonzero().tolist()]
    gone, events = set(), 0
    for _, i, j in sorted(found):
        if i not in gone and j not in gone:
            gone.update(k for k in (i, j) if k < n)
            events += 1
    keep = torch.tensor([i for i in range(n) if i not in gone], device=x.device)
    return keep, events


def _invariants(case, x, y, g):
    energy, n, layers = 0.0, x.numel(), case["layers"]
    rows = max(1, (1 << 25) // n)
    for t0 in range(0, n, rows):
        t1 = min(t0 + rows, n)
        dx, dy = x[t0:t1, None] - x[None, :], y[t0:t1, None] - y[None, :]
        later = torch.arange(n, device=x.device)[None, :] > torch.arange(t0, t1, device=x.device)[:, None]
        if case["geometry"] == "periodic":
            dx, dy = _wrap(dx), _wrap(dy)
            s2 = torch.sin(0.5 * dy) ** 2
            term = -dx * dx / TWO_PI
            for m in range(-layers, layers + 1):
                # log(2 (sinh^2 h + s2)) - log cosh(2 pi m) with sinh^2 h = e^(2|h|) (1 - e^(-2|h|))^2 / 4
                h = (0.5 * (dx - TWO_PI * m)).abs()
                q = torch.exp(-2.0 * h)
                a = TWO_PI * abs(m)
                log_cosh = a + math.log1p(math.exp(-2.0 * a)) - math.log(2.0)
                term = term + 2.0 * h + torch.log(0.5 * (1.0 - q) ** 2 + 2.0 * s2 * q) - log_cosh
        elif case["geometry"] == "infinite":
            term = torch.log(dx * dx + dy * dy + case["core"] ** 2)
        else:
            dot = x[t0:t1, None] * x[None, :] + y[t0:t1, None] * y[None, :]
            cross = y[t0:t1, None] * x[None, :] - x[t0:t1, None] * y[None, :]
            term = torch.log((dx * dx + dy * dy) / ((1.0 - dot) ** 2 + cross * cross))
        energy += float((torch.where(later, term, 0.0) * (g[t0:t1, None] * g[None, :])).sum())
    if case["geometry"] == "disk":
        energy += float(-(g * g * torch.log(1.0 - (x * x + y * y))).sum())
    moments = [math.fsum(v.tolist()) for v in (g, g * x, g * y, g * (x * x + y * y))]
    return np.array(moments + [-energy / (2.0 * TWO_PI)])


def exact(case, seed):
    def up(*arrays):
        return [torch.from_numpy(np.ascontiguousarray(a)).to(_device()) for a in arrays]

    kind = case["kind"]
    if kind == "rows":
        return None  # text: the bytes themselves
    if kind == "ensemble":
        xs, ys, accepted, rejected = [], [], [], []
        for geometry, st in _members(case, seed):
            sub = dict(case, geometry=geometry, core=0.0, layers=8)
            x, y, _, a, r, _ = _dopri5(sub, *up(*st), case["steps"])
            xs.append(x)
            ys.append(y)
            accepted.append(a)
            rejected.append(r)
        return [torch.cat(xs), torch.cat(ys), np.array(accepted), np.array(rejected)]
    x, y, g = up(*_state(case, seed))
    if kind == "rk4":
        dt = case["dt"]
        for _ in range(case["steps"]):
            a = _velocity(case, x, y, g)
            b = _velocity(case, x + 0.5 * dt * a[0], y + 0.5 * dt * a[1], g)
            c = _velocity(case, x + 0.5 * dt * b[0], y + 0.5 * dt * b[1], g)
            d = _velocity(case, x + dt * c[0], y + dt * c[1], g)
            x = x + dt * (a[0] + 2.0 * b[0] + 2.0 * c[0] + d[0]) / 6.0
            y = y + dt * (a[1] + 2.0 * b[1] + 2.0 * c[1] + d[1]) / 6.0
        return [x, y]
    if kind == "dopri5":
        out = torch.zeros((3, x.numel()), dtype=torch.float64)
        *after, _, rejected, events = _dopri5(case, x, y, g, case["steps"], case["distance"])
        for row, a in zip(out, after):
            row[:a.numel()] = a.cpu()
        return [out[0], out[1], out[2], rejected, events]
    if kind == "range":
        u, v = torch.zeros_like(x), torch.zeros_like(x)
        u[case["begin"]:case["end"]], v[case["begin"]:case["end"]] = _velocity(
            case, x, y, g, case["begin"], case["end"])
        return [u, v]
    if kind == "invariants":
        return _invariants(case, x, y, g)
    return list(_velocity(case, x, y, g))

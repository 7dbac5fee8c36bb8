"""DOPRI5 steps of small FP64 populations in one cooperative launch: bit for bit the launch sequence's
(which runs with per-launch profiling on) -- accepted and rejected attempts, the cached derivative,
evaluation counts, dipole events, errors and the state they leave -- and the exit of its grid
barrier's bounded wait."""
import numpy as np
import pytest

import pointvortex_b200 as pv
from pointvortex_b200 import ics

pytestmark = pytest.mark.gpu


def make(name):
    if name == "periodic":
        return pv.PeriodicBoxKernel(2.0, 2.0, 8)
    if name == "periodic_m3":
        return pv.PeriodicBoxKernel(2.0, 2.0, 3)
    return pv.DiskKernel(1.0) if name == "disk" else pv.InfinitePlaneKernel(0.0)


def state(name, n):
    x, y, g = (ics.disk(n, 9 + n, 1.0, 0.8) if name == "disk"
               else ics.infinite_plane(n + n % 2, 9 + n))
    if name != "disk":
        x, y, g = x[:n], y[:n], np.random.default_rng(n).standard_normal(n)
        g -= g.mean()
    return x, y, g


def run(name, n, profiling, dt, steps, distance=None, **solve):
    k = make(name)
    k.setProfiling(profiling)
    # dipole events keep the box neutral only with equal strengths
    x, y, g = ics.periodic_box(n, 9 + n, 2.0) if distance else state(name, n)
    k.uploadDeviceState(pv.VortexSystem(x, y, g))
    manager = pv.DeviceDipoleManager(k, removal=True, distance=distance) if distance else None
    out, error = [], None
    try:
        for _ in range(steps):
            r = k.deviceDopri5Step(dt, solve.get("atol", 1e-12), solve.get("rtol", 1e-9),
                                   solve.get("dtmin", 1e-12), 0.1)
            out.append((r.acceptedTimeStep, r.suggestedTimeStep, r.normalizedError,
                        r.rejectedSteps, manager.process() if manager else 0))
            dt = r.suggestedTimeStep
    except (RuntimeError, ValueError) as exc:
        error = (type(exc), str(exc))
    s = k.downloadDeviceSystem()
    return out, error, k.evaluationCount, s.x, s.y, s.circulation


def same(a, b):
    assert a[:3] == b[:3]
    assert all(np.array_equal(p, q) for p, q in zip(a[3:], b[3:]))


@pytest.mark.parametrize("name", ["infinite", "periodic", "periodic_m3", "disk"])
@pytest.mark.parametrize("n", [1, 2, 31, 64, 147, 149, 301, 743, 1024, 2047])
def test_equals_the_launch_sequence(name, n):
    dt = 1e-2 / n if name == "disk" else 2.0 / n ** 2  # shortened by the controller at first
    a, b = (run(name, n, profiling, dt, 5) for profiling in (False, True))
    same(a, b)


def test_with_dipole_events():
    a, b = (run("periodic", 600, profiling, 1e-5, 4, distance=5e-3) for profiling in (False, True))
    same(a, b)
    assert a[1] is None
    assert sum(r[4] for r in a[0]) > 0  # some pairs were removed


@pytest.mark.parametrize("solve", [dict(atol=1e-300, rtol=0.0, dtmin=1e-300),   # rejection cap
                                   dict(atol=1e-15, rtol=0.0, dtmin=1e-3)])     # the dt floor
def test_failures_leave_the_state(solve):
    a, b = (run("infinite", 50, profiling, 0.1, 1, **solve) for profiling in (False, True))
    same(a, b)
    assert a[1] == (RuntimeError, "adaptive integrator could not satisfy tolerance")
    assert np.array_equal(a[3], state("infinite", 50)[0])


def test_a_stage_outside_the_disk():
    """A first step so long that a stage leaves the disk: the same error on both routes, the state
    unchanged, and a shorter step works afterwards."""
    results = []
    for profiling in (False, True):
        k = pv.DiskKernel(1.0)
        k.setProfiling(profiling)
        x, y, g = ics.disk(300, 4, 1.0, 0.9)
        k.uploadDeviceState(pv.VortexSystem(x, y, g))
        with pytest.raises(ValueError, match="vortex lies on or outside the disk"):
            k.deviceDopri5Step(0.5, 1e-12, 1e-9, 1e-12, 1.0)
        s = k.downloadDeviceSystem()
        assert np.array_equal(s.x, x) and np.array_equal(s.y, y)
        r = k.deviceDopri5Step(1e-7, 1e-12, 1e-9, 1e-12, 1.0)
        s = k.downloadDeviceSystem()
        results.append((r.acceptedTimeStep, r.normalizedError, s.x.tobytes(), s.y.tobytes()))
    assert results[0] == results[1]


def test_barrier_timeout_leaves_the_state():
    x, y, g = ics.infinite_plane(1024, 33)
    fresh = pv.InfinitePlaneKernel(0.0)
    fresh.uploadDeviceState(pv.VortexSystem(x, y, g))
    fresh.deviceDopri5Step(1e-6, 1e-12, 1e-9, 1e-12, 0.1)
    want = fresh.downloadDeviceSystem()
    k = pv.InfinitePlaneKernel(0.0)
    timeouts = 0
    for _ in range(8):
        k.uploadDeviceState(pv.VortexSystem(x, y, g))
        k.setWaitLimits(barrier_polls=0)
        try:
            k.deviceDopri5Step(1e-6, 1e-12, 1e-9, 1e-12, 0.1)
        except RuntimeError as exc:
            assert "a bounded device wait timed out" in str(exc)
            timeouts += 1
            s = k.downloadDeviceSystem()
            assert np.array_equal(s.x, x) and np.array_equal(s.y, y)
    assert timeouts >= 1
    k.setWaitLimits()
    k.uploadDeviceState(pv.VortexSystem(x, y, g))
    k.deviceDopri5Step(1e-6, 1e-12, 1e-9, 1e-12, 0.1)
    s = k.downloadDeviceSystem()
    assert np.array_equal(s.x, want.x) and np.array_equal(s.y, want.y)

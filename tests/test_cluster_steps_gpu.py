"""Small populations' steps in one cluster against the same steps on the whole grid, which a context with
a barrier limit of its own takes: bit for bit, at the edges of the rule (a thread for each target and
chunk, half of them in the box), with fewer vortices than CTAs, over rejections, and with the errors
that a step can end with."""
import numpy as np
import pytest

from pointvortex_b200 import ics
from pointvortex_b200.kernel import DiskKernel, InfinitePlaneKernel, PeriodicBoxKernel, VortexSystem

pytestmark = pytest.mark.gpu
GRID_LIMIT = (1 << 24) + 1  # the default is 2^24 polls


def pair(geometry, n):
    made = []
    for grid in (False, True):
        if geometry == "infinite":
            k, s = InfinitePlaneKernel(0.0), ics.infinite_plane(n, 7)
        elif geometry == "disk":
            k, s = DiskKernel(1.0), ics.disk(n, 7, 1.0, 0.8, gaussian=False)
        else:
            layers = 8 if geometry == "periodic" else 4
            k, s = PeriodicBoxKernel(2.0, 2.0, layers), ics.periodic_box(n, 7)
        if grid:
            k.setWaitLimits(barrier_polls=GRID_LIMIT)
        k.uploadDeviceState(VortexSystem(*s))
        made.append(k)
    return made


def same(a, b):
    a, b = a.downloadDeviceSystem(), b.downloadDeviceSystem()
    return np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y)


@pytest.mark.parametrize("geometry", ["infinite", "disk", "periodic", "series"])
@pytest.mark.parametrize("n", [2, 14, 16, 18, 48, 50, 128, 208, 210, 224, 226, 302, 304, 320, 322])
def test_steps_are_the_grid_s(geometry, n):
    a, b = pair(geometry, n)
    for k in (a, b):
        k.rk4Advance(1e-6, 5)
        k.deviceRk4Step(1e-6)
    assert same(a, b)
    da = db = 1e-3
    for _ in range(4):
        ra = a.deviceDopri5Step(da, 1e-10, 1e-8, 1e-13, 0.1)
        rb = b.deviceDopri5Step(db, 1e-10, 1e-8, 1e-13, 0.1)
        assert ra == rb
        da, db = ra.suggestedTimeStep, rb.suggestedTimeStep
        assert same(a, b)


@pytest.mark.parametrize("step", ["rk4", "dopri5"])
def test_errors_are_the_grid_s(step):
    """A coincident pair (reported by the evaluation) and a stage that leaves the disk."""
    for make, state in ((lambda: InfinitePlaneKernel(0.0), ics.infinite_plane(100, 3)),
                        (lambda: DiskKernel(1.0), ics.disk(100, 3, 1.0, 0.8, gaussian=False))):
        x, y, g = (np.array(v) for v in state)
        if make().__class__ is InfinitePlaneKernel:
            x[3], y[3], dt = x[90], y[90], 1e-4
        else:
            dt = 1e3
        said = []
        for grid in (False, True):
            k = make()
            if grid:
                k.setWaitLimits(barrier_polls=GRID_LIMIT)
            k.uploadDeviceState(VortexSystem(x, y, g))
            with pytest.raises((RuntimeError, ValueError)) as e:
                if step == "rk4":
                    k.rk4Advance(dt, 3)
                else:
                    k.deviceDopri5Step(dt, 1e-10, 1e-8, 1e-13, 1e4)
            out = k.downloadDeviceSystem()
            assert np.array_equal(out.x, x) and np.array_equal(out.y, y)
            said.append(str(e.value))
        assert said[0] == said[1]

"""Disks of any radius whose square is a number: the once-per-unordered-pair form, which works with the fourth
power of the radius, serves radii of 2^-200 to 2^200 and leaves the others to the ordered kernel and to
ordered work items. Radii are powers of two, by which every position scales without rounding; velocities go
with 1 / radius, so that they agree with those of the unit disk to the parity tolerance, 1e-12 of their
scale, and steps that scale with the square of the radius to the rounding of three of them, 1e-14 of the
radius."""
import numpy as np
import pytest

import pointvortex_b200 as pv
from conftest import normalized_error
from pointvortex_b200 import ics
from pointvortex_b200.batch import Batch, geometry_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power,symmetric", [(-300, 0), (-201, 0), (-200, 1), (200, 1), (201, 0), (300, 0)])
def test_device_state_and_host_evaluation(power, symmetric):
    n, r = 4100, 2.0 ** power
    x, y, g = ics.disk(n, 5, 1.0, 0.9)
    one = pv.DiskKernel(1.0).evaluateRange(x, y, g, None, 0, n - 1)  # the ordered kernel
    k = pv.DiskKernel(r)
    k.uploadDeviceState(pv.VortexSystem(r * x, r * y, g))
    assert k.statePlan()["symmetric"] == symmetric
    for f in (k.evaluateDeviceState(), k.evaluate(r * x, r * y, g)):
        error = normalized_error((f.x * r)[:-1], (f.y * r)[:-1], one.x[:-1], one.y[:-1])
        assert error.max() <= 1e-12


def solve(radii, n=600, steps=3):
    b = Batch(len(radii) * (n + 256), len(radii), max_steps=steps, partial_factor=64)
    x, y, g = ics.disk(n, 7, 1.0, 0.8, gaussian=False)
    ids = []
    for r in radii:
        dt = 1e-6 * r * r
        ids.append(b.add(geometry_params("disk", disk_radius=r), r * x, r * y, g, 1e3 * dt, dt=dt,
                         atol=1e-10 * r, rtol=1e-8, dtmin=1e-6 * dt, dtmax=dt))
    b.run()
    out = [(b.info(i), b.result(i)) for i in ids]
    b.close()
    return out


def test_batch_members():
    powers = (-140, 0, 140, -210, 210)
    (_, (x1, y1)), = solve([1.0])
    for p, (info, (x, y)) in zip(powers, solve([2.0 ** p for p in powers])):
        assert info.state == "budget" and info.acceptedSteps == 3, (p, info)
        assert info.targetsPerThread == (0 if abs(p) <= 200 else 2), (p, info)
        assert np.max(np.hypot(x * 2.0 ** -p - x1, y * 2.0 ** -p - y1)) <= 1e-14, p

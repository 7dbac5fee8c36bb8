"""The FP64 disk once per unordered pair (the device state from N = 4096: one, two and four targets
per lane) against the ordered kernel and the oracle: whole and ragged last blocks, vortices up to
0.999 of the radius, an off-size radius, the reference's error for a coincident pair, and
repeatability. Both forms round each term a few times, so the velocity parity tolerance (1e-12)
applies. (Nearer the wall it cannot: the reference's own 1 - t.s loses 2^-53 / (1 - |s|^2 / R^2) of
the image term, for any order of evaluation.)"""
import numpy as np
import pytest

import pointvortex_b200 as pv
from conftest import normalized_error
from oracle.pyoracle import Geometry
from pointvortex_b200 import ics

pytestmark = pytest.mark.gpu


def loaded(x, y, g, radius=1.0):
    k = pv.DiskKernel(radius)
    k.uploadDeviceState(pv.VortexSystem(x, y, g))
    return k


@pytest.mark.parametrize("n,targets", [(4096, 1), (4127, 1), (8191, 1), (8192, 2), (8250, 2),
                                       (16384, 4), (16500, 4)])
def test_against_ordered_and_oracle(port, n, targets):
    radius = 2.5 if n % 2 else 1.0
    x, y, g = ics.disk(n, 60 + n, radius, 0.999)
    x[0], y[0] = 0.0, 0.0                                   # at the centre: no image velocity
    k = loaded(x, y, g, radius)
    plan = k.statePlan()
    assert plan["symmetric"] and plan["symmetric_targets"] == targets
    f = k.evaluateDeviceState()
    small = pv.DiskKernel(radius)
    for t0, t1 in ((0, 40), (n // 2, n // 2 + 40), (n - 40, n)):
        o = small.evaluateRange(x, y, g, None, t0, t1)      # the ordered kernel
        u, v = port.evaluate_range(Geometry("disk", disk_radius=radius), x, y, g, t0, t1)
        rms = np.sqrt(np.mean(f.x ** 2 + f.y ** 2))
        for a, b in ((o.x[t0:t1], o.y[t0:t1]), (u, v)):
            scale = np.maximum(np.hypot(a, b), rms)
            assert np.max(np.hypot(f.x[t0:t1] - a, f.y[t0:t1] - b) / scale) <= 1e-12
    again = k.evaluateDeviceState()
    assert np.array_equal(f.x, again.x) and np.array_equal(f.y, again.y)


@pytest.mark.parametrize("i,j", [(7, 4090), (64, 65)])
def test_coincident_pair_is_the_reference_error(port, i, j):
    x, y, g = ics.disk(4100, 5, 1.0, 0.9)
    x[i], y[i] = x[j], y[j]
    with pytest.raises(RuntimeError, match="coincident vortices in disk"):
        loaded(x, y, g).evaluateDeviceState()


def test_smaller_populations_use_the_ordered_kernel():
    x, y, g = ics.disk(4095, 2, 1.0, 0.9)
    assert not loaded(x, y, g).statePlan()["symmetric"]

"""Host evaluations of all targets go once per unordered pair where the device state does: next to the
smallest such populations, odd sizes, outside the box and with contexts that change their size; against the
ordered kernel (which a range of one target less takes), within the parity tolerance of 1e-12 of the
velocity's scale, and equal to the device state's velocities bit for bit."""
import numpy as np
import pytest

from pointvortex_b200 import ics
from pointvortex_b200.kernel import DiskKernel, InfinitePlaneKernel, PeriodicBoxKernel, VortexSystem

pytestmark = pytest.mark.gpu


def case(geometry, n):
    if geometry == "periodic":
        x, y, g = ics.periodic_box(n + n % 2, 5)
        x, y, g = x[:n], y[:n], g[:n] - g[:n].mean()
        x[::5] += 4.0
        return PeriodicBoxKernel(2.0, 2.0, 8), (x, y, g)
    if geometry == "disk":
        return DiskKernel(1.0), ics.disk(n, 5, 1.0, 0.8, gaussian=False)
    return InfinitePlaneKernel(0.0), ics.infinite_plane(n, 5)


@pytest.mark.parametrize("geometry,sizes", [("periodic", (2047, 2048, 2049, 5001, 2050)),
                                            ("disk", (4095, 4096, 4097, 9001, 4100)),
                                            ("infinite", (16383, 16384, 16385, 20001))])
def test_against_ranges_and_the_device_state(geometry, sizes):
    kernel, _ = case(geometry, 64)
    for n in sizes:
        fresh, (x, y, g) = case(geometry, n)
        f = kernel.evaluate(x, y, g)
        part = fresh.evaluateRange(x, y, g, None, 0, n - 1)  # arrays of n, the last entry left alone
        scale = np.sqrt(np.mean(f.x ** 2 + f.y ** 2))
        size = np.maximum(np.hypot(f.x, f.y), scale)
        assert np.max((np.hypot(f.x - part.x, f.y - part.y) / size)[:-1]) <= 1e-12, n
        whole = fresh.evaluateRange(x, y, g, None, 0, n)
        assert np.array_equal(whole.x, f.x) and np.array_equal(whole.y, f.y)
        if n >= sizes[1]:
            fresh.uploadDeviceState(VortexSystem(x, y, g))
            assert fresh.statePlan()["symmetric"]
            s = fresh.evaluateDeviceState()
            assert np.array_equal(s.x, f.x) and np.array_equal(s.y, f.y)


@pytest.mark.parametrize("geometry,n", [("periodic", 4096), ("disk", 5000), ("infinite", 16500)])
def test_coincident_pair(geometry, n):
    kernel, (x, y, g) = case(geometry, n)
    x[7], y[7] = x[n - 9], y[n - 9]
    with pytest.raises(RuntimeError, match="coincident"):
        kernel.evaluate(x, y, g)

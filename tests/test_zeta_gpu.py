"""The rational periodic pair term on the GPU where its route or its reduction changes: image counts
and box lengths on both sides of the rule, displacements across the seams, positions outside the box,
and the symmetric kernels' tiles, against the oracle (per-vortex velocity error <= 1e-12)."""
import numpy as np
import pytest

import pointvortex_b200 as pv
from conftest import normalized_error
from oracle.pyoracle import Geometry
from pointvortex_b200 import ics

pytestmark = pytest.mark.gpu


def check(port, length, layers, x, y, g, device_state=False):
    k = pv.PeriodicBoxKernel(length, length, layers)
    if device_state:
        k.uploadDeviceState(pv.VortexSystem(x, y, g))
        f = k.evaluateDeviceState()
    else:
        f = k.evaluate(x, y, g)
    geo = Geometry("periodic", box_length_x=length, box_length_y=length, image_layers=layers)
    u, v = port.evaluate(geo, x, y, g)
    assert normalized_error(f.x, f.y, u, v).max() <= 1e-12


@pytest.mark.parametrize("layers", [5, 6, 7])
@pytest.mark.parametrize("length", [1.0 / 70000.0, 1.0 / 65536.0, 1e-3, 2 * np.pi, 65536.0, 7e4])
def test_routes(port, layers, length):
    x, y, g = ics.periodic_box(130, 3, length)
    check(port, length, layers, x, y, g)


@pytest.mark.parametrize("device_state", [False, True])
def test_seams_and_far_positions(port, device_state):
    """Vortices on the seams, close pairs across them, and a third of the population shifted by
    whole boxes."""
    length = 2.0
    x, y, g = ics.periodic_box(2082 if device_state else 258, 5, length)
    x[:4] = [-1.0, 1.0 - 1e-7, -1.0 + 2e-7, np.nextafter(1.0, 0.0)]
    y[:4] = [0.3, 0.3, 0.3 + 1e-7, -0.9]
    y[4:6], x[4:6] = [-1.0, np.nextafter(1.0, 0.0) - 1e-6], 0.125
    x[::3] += 6.0
    y[1::3] -= 4.0
    check(port, length, 8, x, y, g, device_state)


@pytest.mark.parametrize("n", [2048, 2079, 2112])
@pytest.mark.parametrize("targets", [0, 2])
def test_symmetric_tiles(port, n, targets):
    """Whole and ragged last tiles of the one- and two-target forms."""
    from pointvortex_b200 import autotune
    x, y, _ = ics.periodic_box(n + n % 2, 7 + n, 2.0)
    x, y = x[:n], y[:n]
    g = np.random.default_rng(n).standard_normal(n)
    g -= g.mean()
    saved = autotune.get_symmetric_entry(1, 0, 11)
    try:
        autotune.set_symmetric_entry(1, 0, 11, 2, 0, targets)
        check(port, 2.0, 8, x, y, g, device_state=True)
    finally:
        autotune.set_symmetric_entry(1, 0, 11, *saved)


@pytest.mark.parametrize("layers", [5, 6, 64])
@pytest.mark.parametrize("length", [1.0 / 65536.0, 2.0, 7e4])
@pytest.mark.parametrize("n", [2, 128, 130, 386])
def test_hamiltonian_routes(port, layers, length, n):
    """The sigma form and the image product on both sides of the rule, tiles whole and ragged,
    positions outside the box; the Hamiltonian's parity tolerance (1e-12 of its terms' scale)."""
    x, y, g = ics.periodic_box(n, 11 + n, length)
    x[::3] += 3 * length
    k = pv.PeriodicBoxKernel(length, length, layers)
    got = k.invariants(pv.VortexSystem(x, y, g)).hamiltonian
    geo = Geometry("periodic", box_length_x=length, box_length_y=length, image_layers=layers)
    want = port.invariants(geo, x, y, g)[4]
    assert abs(got - want) <= 1e-12 * max(abs(want), 1.0)

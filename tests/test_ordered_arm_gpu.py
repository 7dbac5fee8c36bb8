"""The once-per-unordered-pair forms of the device state against the ordered-pair kernel at every target.
A host evaluation of all targets takes the same form as the device state, so the ordered side is a range
of all targets but the last, and a range of that one: a range of fewer targets than vortices always runs
the ordered kernel. Both agree to the parity tolerance, 1e-12 of the velocity's scale."""
import numpy as np
import pytest

import pointvortex_b200 as pv
from conftest import normalized_error
from pointvortex_b200 import autotune, ics

pytestmark = pytest.mark.gpu

L = 2 * np.pi


def ordered(k, x, y, g):
    n = x.size
    most = k.evaluateRange(x, y, g, None, 0, n - 1)
    last = k.evaluateRange(x, y, g, None, n - 1, n)
    return (np.append(most.x[:n - 1], last.x[n - 1]), np.append(most.y[:n - 1], last.y[n - 1]))


def check(k, state, symmetric_targets=None):
    k.uploadDeviceState(pv.VortexSystem(*state))
    plan = k.statePlan()
    assert plan["symmetric"]
    assert symmetric_targets is None or plan["symmetric_targets"] == symmetric_targets
    f = k.evaluateDeviceState()
    u, v = ordered(k, *state)
    assert normalized_error(f.x, f.y, u, v).max() <= 1e-12
    return f, u, v


@pytest.mark.parametrize("layers", [8, 3])
@pytest.mark.parametrize("n,entry", [(2050, (2, 0, 0)), (3000, (2, 0, 0)), (4100, (2, 0, 0)),
                                     (4136, (2, 0, 2)), (8192, (2, 0, 0)), (8250, (2, 7, 0)),
                                     (8250, (2, 8, 0)), (24000, (2, 0, 0)), (24000, (2, 0, 2))])
def test_box(n, layers, entry):
    bucket = n.bit_length() - 1
    saved = autotune.get_symmetric_entry(1, 0, bucket)
    try:
        autotune.set_symmetric_entry(1, 0, bucket, *entry)
        f, u, v = check(pv.PeriodicBoxKernel(L, L, layers), ics.periodic_box(n, 31 + n, L),
                        entry[2] or 1)
    finally:
        autotune.set_symmetric_entry(1, 0, bucket, *saved)
    # the two are different kernels: their sums are rounded differently somewhere
    assert not np.array_equal(f.x, u)


@pytest.mark.parametrize("core", [0.0, 1e-3])
@pytest.mark.parametrize("n,targets", [(16390, 4), (20001, 4), (33000, 8), (40000, 8), (40000, 4)])
def test_plane(n, targets, core):
    bucket = n.bit_length() - 1
    saved = autotune.get_symmetric_entry(0, 0, bucket)
    try:
        autotune.set_symmetric_entry(0, 0, bucket, 2, 0, targets)
        f, u, v = check(pv.InfinitePlaneKernel(core), ics.infinite_plane(n, 17), targets)
    finally:
        autotune.set_symmetric_entry(0, 0, bucket, *saved)
    assert not np.array_equal(f.x, u)


@pytest.mark.parametrize("n,targets", [(4097, 1), (9001, 2), (16500, 4), (24003, 4)])
def test_disk(n, targets):
    f, u, v = check(pv.DiskKernel(1.0), ics.disk(n, 5, 1.0, 0.95), targets)
    assert not np.array_equal(f.x, u)

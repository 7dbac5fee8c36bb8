"""Pinned staging of host transfers: growth past the buffer, a context's first (direct) transfers,
transfers beyond the staging limit, uploads back to back while an earlier one may be in flight, and
batch admissions that wrap the staging or need several pieces. Copies are exact: every comparison is
bit for bit, against the arrays themselves or against a fresh context's first call."""
import numpy as np
import pytest

from pointvortex_b200 import ics
from pointvortex_b200.batch import Batch, geometry_params
from pointvortex_b200.kernel import InfinitePlaneKernel, VortexSystem

pytestmark = pytest.mark.gpu


def system(n, seed):
    rng = np.random.default_rng(seed)
    return VortexSystem(rng.standard_normal(n), rng.standard_normal(n), rng.standard_normal(n))


def same(a, b):
    return all(np.array_equal(getattr(a, k), getattr(b, k)) for k in ("x", "y", "circulation"))


def used(kernel):
    """The kernel after the 64 transfers that a context makes directly."""
    a = system(2, 1)
    for _ in range(32):
        kernel.uploadDeviceState(a)
        kernel.downloadDeviceState(a)
    return kernel


# 2^20 + 1 vortices: four arrays of 8 MB, just past 32 MB; then back into the staging
@pytest.mark.parametrize("sizes", [(5, 1, 4096, 2048, 4097, 1), (3, 3, 3, (1 << 20) + 1, 7, 1 << 20)])
@pytest.mark.parametrize("staged", [False, True])
def test_state_round_trips(sizes, staged):
    k = InfinitePlaneKernel(0.0)
    if staged:
        used(k)
    for i, n in enumerate(sizes):
        a = system(n, i)
        k.uploadDeviceState(a)
        x = a.x.copy()
        a.x[:] = 7.0  # the caller's arrays are free once the call returns
        out = k.downloadDeviceSystem()
        a.x[:] = x
        assert same(out, a), n
        k.uploadDeviceState(system(n, 100 + i))  # and again without a download between
        b = system(n, 200 + i)
        k.uploadDeviceState(b)
        assert same(k.downloadDeviceSystem(), b), n


def test_later_calls_equal_a_context_s_first():
    k = used(InfinitePlaneKernel(0.0))
    for i, n in enumerate((2, 300, 8191, 33, 300)):
        s = system(n, i)
        first = InfinitePlaneKernel(0.0)
        a, b = k.evaluate(s.x, s.y, s.circulation), first.evaluate(s.x, s.y, s.circulation)
        assert np.array_equal(a.x, b.x) and np.array_equal(a.y, b.y), n
        assert k.invariants(s) == first.invariants(s)
        assert (k.formatTrajectoryHost(0.5, 3, s, a) ==
                InfinitePlaneKernel(0.0).formatTrajectoryHost(0.5, 3, s, a))


# 256 KB of staging hold some 10,900 vortices: several members take two pieces or more, the rest wrap
def test_batch_admissions_wrap_the_staging():
    sizes = [60001, 1, 20000, 20000, 20000, 257, 43690, 100]
    b = Batch(sum(sizes) + 256 * len(sizes), len(sizes), max_steps=1)
    states = [ics.disk(n, 3 + n, 1.0, 0.8, gaussian=False) if n > 1 else
              (np.array([0.1]), np.array([0.2]), np.array([1.0])) for n in sizes]
    ids = [b.add(geometry_params("disk"), *s, 0.0, dt=1e-6) for s in states]  # t_end 0: done as admitted
    b.run()
    for i, (x, y, _) in zip(ids, states):
        xr, yr = b.result(i)
        assert np.array_equal(xr, x) and np.array_equal(yr, y), len(x)
    b.close()

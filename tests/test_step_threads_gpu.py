"""Contexts of different host threads step independently: small populations of unlike sizes, whose steps
are launches of one kernel with unlike amounts of shared memory, at the same time. (Where a launch sets that
kernel's limit to its own amount, some one in twenty thousand finds it lowered by another thread's and fails.)
Without an error, and bit for bit what each gives by itself. N = 64 and 300 in the plane step in one cluster, 400 and 2047 on the
whole grid."""
import threading

import numpy as np
import pytest

import pointvortex_b200 as pv
from pointvortex_b200 import ics

pytestmark = pytest.mark.gpu


def run(n, method, count):
    k = pv.InfinitePlaneKernel(1e-3)
    k.uploadDeviceState(pv.VortexSystem(*ics.infinite_plane(n, 5)))
    for _ in range(count):
        if method == "rk4":
            k.deviceRk4Step(1e-6)
        else:
            k.deviceDopri5Step(1e-6, 1e-10, 1e-8, 1e-12, 1e-6)
    s = k.downloadDeviceSystem()
    k.close()
    return s.x, s.y


@pytest.mark.parametrize("method", ["rk4", "dopri5"])
@pytest.mark.parametrize("sizes,count", [((64, 300), 1500), ((400, 2047) * 4, 4000)])
def test_threads_step_contexts_of_unlike_sizes(sizes, count, method):
    alone = {n: run(n, method, count) for n in set(sizes)}
    together, errors = [], []

    def drive(n):
        try:
            together.append((n, run(n, method, count)))
        except Exception as exc:  # reported by the main thread
            errors.append((n, exc))

    threads = [threading.Thread(target=drive, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for n, (x, y) in together:
        assert np.array_equal(x, alone[n][0]) and np.array_equal(y, alone[n][1]), n

"""The batch's once-per-unordered-pair items of FP64 plane members (from 128 to 4096 vortices, four targets
per lane) at the edges of their rule and of their 128-blocks: alone as in the mix, bit for bit, and
against the same members on ordered items, which a batch-table entry asks for. Two evaluations differ by the
parity tolerance, 1e-12 of the velocity; steps of at most 1e-4 at speeds up to 1e2 move that to 1e-14 a
step, which close pairs amplify by a factor of a few: 1e-11 over three steps. The controller takes its next step
from the -1/5 power of an error estimate that is a difference of nearly equal sums, so the two reach times
that differ by up to 1e-6 of themselves, and their positions by that times the speed."""
import numpy as np
import pytest

from pointvortex_b200 import autotune, ics
from pointvortex_b200.batch import Batch, geometry_params

pytestmark = pytest.mark.gpu
SIZES = (126, 128, 129, 255, 257, 640, 1023, 1025, 2047, 4096, 4097)


def solve(sizes):
    b = Batch(sum(n + 256 for n in sizes), len(sizes), max_steps=3, partial_factor=64)
    ids = [b.add(geometry_params("infinite"), *ics.infinite_plane(n, 3 + n), 1.0, dt=1e-6, atol=1e-10,
                 rtol=1e-8, dtmax=1e-4) for n in sizes]
    b.run()
    out = [(b.info(i), b.result(i)) for i in ids]
    b.close()
    return out


def test_alone_in_the_mix_and_against_ordered_items():
    for n in SIZES:
        autotune.set_batch_entry(0, 0, n.bit_length() - 1, 0)
    for n, (info, (x, y)) in zip(SIZES, solve(SIZES)):
        pairs = 128 <= n <= 4096
        assert (info.targetsPerThread == 0) == pairs, (n, info)
        (alone, (xa, ya)), = solve([n])
        assert alone.acceptedSteps == info.acceptedSteps
        assert np.array_equal(x, xa) and np.array_equal(y, ya), n
        try:
            autotune.set_batch_entry(0, 0, n.bit_length() - 1, 4)
            (ordered, (xo, yo)), = solve([n])
        finally:
            autotune.set_batch_entry(0, 0, n.bit_length() - 1, 0)
        assert ordered.targetsPerThread == 4
        assert ordered.acceptedSteps == info.acceptedSteps and ordered.state == info.state
        late = abs(info.time - ordered.time)
        assert late <= 1e-6 * info.time
        x0, y0, _ = ics.infinite_plane(n, 3 + n)
        speed = np.max(np.hypot(x - x0, y - y0)) / info.time
        assert np.max(np.hypot(x - xo, y - yo)) <= 1e-11 + 1.1 * late * speed, n

"""The batch's once-per-unordered-pair items of smaller FP64 members (box and disk, 128 to 4096
vortices) at the edges of their rule and of their 128-blocks: results alone equal results in the mix
bit for bit, and agree with the same members on ordered items (a batch-table entry asks for those)
after a few accepted steps. Two evaluations differ by the parity tolerance, 1e-12 of the velocity;
steps of at most 1e-4 at speeds up to 1e2 move that to 1e-14 a step, which close pairs amplify by a
factor of a few: 1e-11 over three steps."""
import numpy as np
import pytest

from pointvortex_b200 import autotune, ics
from pointvortex_b200.batch import Batch, geometry_params

pytestmark = pytest.mark.gpu

MEMBERS = [(g, n) for g in ("periodic", "disk") for n in (126, 128, 130, 256, 1022, 2046, 4096, 4098)]


def state(boundary, n):
    if boundary == "periodic":
        return ics.periodic_box(n, 3 + n)
    x, y, g = ics.disk(n, 3 + n, 1.0, 0.8, gaussian=False)
    return x, y, g


def solve(members):
    b = Batch(sum(n + 256 for _, n in members), len(members), max_steps=3, partial_factor=64)
    ids = [b.add(geometry_params(g), *state(g, n), 1.0, dt=1e-6, atol=1e-10, rtol=1e-8, dtmax=1e-4)
           for g, n in members]
    b.run()
    out = [(b.info(i), b.result(i)) for i in ids]
    b.close()
    return out


@pytest.fixture
def no_entries():
    """The batch table without entries for the members' sizes (pv_get_batch_tuning reports the
    default where there is none, so a test that puts back what it read leaves an entry)."""
    for g, n in MEMBERS:
        autotune.set_batch_entry(autotune.GEOMETRIES[g], 0, n.bit_length() - 1, 0)


def test_alone_in_the_mix_and_against_ordered_items(no_entries):
    mixed = solve(MEMBERS)
    for (g, n), (info, (x, y)) in zip(MEMBERS, mixed):
        pairs = n >= 128 and (n <= 4096 or g == "periodic")
        assert (info.targetsPerThread == 0) == pairs, (g, n, info)
        (alone, (xa, ya)), = solve([(g, n)])
        assert alone.acceptedSteps == info.acceptedSteps
        assert np.array_equal(x, xa) and np.array_equal(y, ya), (g, n)
        if pairs and n < 2048 or (g == "disk" and pairs):
            key = (autotune.GEOMETRIES[g], 0, n.bit_length() - 1)
            try:
                autotune.set_batch_entry(*key, 1)
                (ordered, (xo, yo)), = solve([(g, n)])
            finally:
                autotune.set_batch_entry(*key, 0)
            assert ordered.targetsPerThread == 1
            assert ordered.acceptedSteps == info.acceptedSteps and ordered.state == info.state
            assert np.max(np.hypot(x - xo, y - yo)) <= 1e-11, (g, n)

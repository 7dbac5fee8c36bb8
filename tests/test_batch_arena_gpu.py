"""A batch as large as the device's memory allows with the partial-sum room that its caller asked for, but not
with the room of small members' once-per-unordered-pair items beside it: it is made all the same, and such
members take ordered items, with the bits that a table entry asking for those gives."""
import numpy as np
import pytest
import torch

from pointvortex_b200 import autotune, ics
from pointvortex_b200.batch import Batch, geometry_params

pytestmark = pytest.mark.gpu

MEMBERS = [("infinite", 300, 4), ("periodic", 256, 1), ("disk", 4096, 2)]  # and their default targets


def solve(batch):
    ids = []
    for geometry, n, _ in MEMBERS:
        st = (ics.periodic_box(n, 3) if geometry == "periodic" else
              ics.disk(n, 3, 1.0, 0.8) if geometry == "disk" else ics.infinite_plane(n, 3))
        ids.append(batch.add(geometry_params(geometry), *st, 1.0, dt=1e-6, dtmax=1e-4))
    batch.run()
    out = [(batch.info(i), batch.result(i)) for i in ids]
    batch.close()
    return out


def test_a_batch_near_the_memory_limit():
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    vortices = int(0.7 * free / 432)  # with 512 bytes a vortex more: 1.5 times the free memory
    large = solve(Batch(vortices, 8, max_steps=3))
    for geometry, n, t in MEMBERS:
        autotune.set_batch_entry(autotune.GEOMETRIES[geometry], 0, n.bit_length() - 1, t)
    small = solve(Batch(20000, 8, max_steps=3))
    for (geometry, n, t), (a, (xa, ya)), (b, (xb, yb)) in zip(MEMBERS, large, small):
        assert a.state == b.state == "budget" and a.targetsPerThread == b.targetsPerThread == t
        assert np.array_equal(xa, xb) and np.array_equal(ya, yb), (geometry, n)

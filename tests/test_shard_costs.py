"""The replicas' partition balances the time that a batch takes: with the measured milliseconds of an attempt
(FP64, full batches, by geometry and population), no rank of a mixed ensemble takes five percent longer than
the mean, beyond the longest-processing-time rule's own slack of one simulation."""
import numpy as np
import pytest

from pointvortex_b200.shard import partition, simulation_cost

# attempts of 256, 64, 16 and 4 simulations of these populations
SIZES = {512: 256, 1024: 64, 2048: 16, 4096: 4}
ATTEMPT_MS = {"infinite": (0.494, 0.411, 0.381, 0.398), "disk": (0.775, 0.681, 0.630, 0.645),
              "periodic": (1.222, 1.072, 1.006, 0.992)}
MS = {(g, n): ms / SIZES[n] for g, row in ATTEMPT_MS.items() for n, ms in zip(SIZES, row)}


@pytest.mark.parametrize("world", [2, 4, 8])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_ranks_take_equal_times(world, seed):
    rng = np.random.default_rng(seed)
    keys = list(MS)
    specs = [keys[k] for k in rng.choice(len(keys), 64, p=[1 / 12] * 12)]
    owner = partition([simulation_cost(*s) for s in specs], world)
    loads = np.zeros(world)
    for s, r in zip(specs, owner):
        loads[r] += MS[s]
    assert loads.max() <= 1.05 * loads.mean() + max(MS.values()) / 2

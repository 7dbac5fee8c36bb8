"""FP64 batch members in a box that does not take the rational pair term: fewer than six image layers, or a
side outside that term's range. From 2048 vortices they take the once-per-unordered-pair items with one
target per lane. At the edges of their 128-blocks: alone as in the mix, bit for bit; against the same
members on ordered items (mode 1 of the symmetric form's table asks for those); and against the oracle's
steps.

Three steps of 1e-7 in the units of a box of side 2 pi (which the controller accepts at once and its
largest step holds there): two evaluations differ by the parity tolerance, 1e-12 of a velocity, which at
speeds up to 1e3 moves a position by 3e-16, and a step's addition rounds it by 2e-16 in each of the two
runs: 1e-14 of that box."""
import numpy as np
import pytest

from oracle.pyoracle import Geometry
from pointvortex_b200 import autotune, ics
from pointvortex_b200.batch import Batch, geometry_params

pytestmark = pytest.mark.gpu

TWO_PI = 2.0 * np.pi
STEPS, DT = 3, 1e-7
MEMBERS = [(layers, length, n) for layers, length in ((1, TWO_PI), (3, TWO_PI), (5, TWO_PI), (8, 7e4))
           for n in (2048, 2050, 4098)]


def solve(members, steps=STEPS):
    b = Batch(sum(n + 256 for _, _, n in members), len(members), max_steps=steps, partial_factor=64)
    ids = []
    for layers, length, n in members:
        unit = length / TWO_PI
        dt = DT * unit * unit  # speeds go with 1 / length
        ids.append(b.add(geometry_params("periodic", box_length=length, image_layers=layers),
                         *ics.periodic_box(n, 3 + n, length), 1e3 * dt, dt=dt, atol=1e-10 * unit,
                         rtol=1e-8, dtmin=1e-6 * dt, dtmax=dt))
    b.run()
    out = [(b.info(i), b.result(i)) for i in ids]
    b.close()
    return out


@pytest.fixture
def ordered_items():
    """Makes the members' admissions take ordered items; puts the table back afterwards."""
    keys = sorted({n.bit_length() - 1 for _, _, n in MEMBERS})
    saved = {b: autotune.get_symmetric_entry(1, 0, b) for b in keys}

    def ordered():
        for b in keys:
            autotune.set_symmetric_entry(1, 0, b, 1, 0, 0)

    yield ordered
    for b, entry in saved.items():
        autotune.set_symmetric_entry(1, 0, b, *entry)


def test_alone_in_the_mix_and_against_ordered_items(ordered_items):
    mixed = solve(MEMBERS)
    for member, (info, (x, y)) in zip(MEMBERS, mixed):
        assert info.state == "budget" and info.acceptedSteps == STEPS, (member, info)
        assert info.targetsPerThread == 0 and info.rejectedSteps == 0, (member, info)
        (_, (xa, ya)), = solve([member])
        assert np.array_equal(x, xa) and np.array_equal(y, ya), member
    ordered_items()
    for member, (info, (x, y)), (other, (xo, yo)) in zip(MEMBERS, mixed, solve(MEMBERS)):
        assert other.targetsPerThread > 0 and other.time == info.time, (member, other)
        error = np.max(np.hypot(x - xo, y - yo))
        assert error <= 1e-14 * member[1] / TWO_PI, (member, error)


@pytest.mark.parametrize("layers,n", [(1, 2050), (5, 2048)])
def test_matches_the_oracle(port, layers, n):
    (info, (x, y)), = solve([(layers, TWO_PI, n)], 1)
    assert info.targetsPerThread == 0 and info.acceptedSteps == 1
    geo = Geometry("periodic", box_length_x=TWO_PI, box_length_y=TWO_PI, image_layers=layers,
                   absolute_tolerance=1e-10, relative_tolerance=1e-8, minimum_time_step=1e-6 * DT,
                   maximum_time_step=DT)
    xr, yr, g = ics.periodic_box(n, 3 + n, TWO_PI)
    xr, yr, r = port.stepper(geo, n).dopri5_step(xr, yr, g, DT)
    assert r[0] == DT
    assert np.max(np.hypot(x - xr, y - yr)) <= 1e-14

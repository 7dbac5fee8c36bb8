"""The Hamiltonian's loops with the table logarithm: sizes around the 128-tiles, two vortices whose
squared distance is next to 1 (where the logarithm vanishes), and arguments that send a thread to the
general loop (subnormal and overflowing squares, coincident vortices in the last tile), against sums in
80-bit arithmetic.

Bound a pair: the argument's roundings are at most 3 (plane) or 16 (disk: products and differences of
numbers up to 1 against a denominator of at least 0.13) units of 2^-53 and move the logarithm by as much;
the logarithm and its products add 3 units of 2^-53 of |log|. The final sums are compensated: one more
unit of the result."""
import numpy as np
import pytest

from pointvortex_b200.kernel import DiskKernel, InfinitePlaneKernel, VortexSystem

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53
LD = np.longdouble


def check(kernel, x, y, g, radius=None):
    x, y, g = (np.asarray(a, dtype=float) for a in (x, y, g))
    X, Y, G = x.astype(LD), y.astype(LD), g.astype(LD)
    dx, dy = X[:, None] - X[None, :], Y[:, None] - Y[None, :]
    arg = dx * dx + dy * dy
    roundings = 3
    if radius:
        roundings = 16
        r2 = LD(radius) ** 2
        dot = X[:, None] * X[None, :] + Y[:, None] * Y[None, :]
        cross = Y[:, None] * X[None, :] - X[:, None] * Y[None, :]
        arg = arg * r2 / ((r2 - dot) ** 2 + cross ** 2)
    i, j = np.triu_indices(x.size, 1)
    w, l = G[i] * G[j], np.log(arg[i, j])
    total = np.sum(w * l)
    bound = np.sum(abs(w) * (roundings + 3 * abs(l))) * EPS
    if radius:
        own = np.log((r2 - X * X - Y * Y) / LD(radius))
        total -= np.sum(G * G * own)
        bound += np.sum(G * G * (roundings + 3 * abs(own))) * EPS
    want = -total / (4 * LD(np.pi))
    got = kernel.invariants(VortexSystem(x, y, g)).hamiltonian
    assert abs(LD(got) - want) <= bound / (4 * np.pi) + 2 * EPS * abs(want), (got, want)


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 257])
@pytest.mark.parametrize("radius", [None, 1.0])
def test_tiles(n, radius):
    rng = np.random.default_rng(n)
    r, t = 0.8 * np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n)
    k = DiskKernel(radius) if radius else InfinitePlaneKernel(0.0)
    check(k, r * np.cos(t), r * np.sin(t), rng.standard_normal(n), radius)


@pytest.mark.parametrize("d", [1.0, 1 + 2.0 ** -52, 1 - 2.0 ** -53, 1 + 1e-9, 1 - 1e-9, 0.999, 1.002])
def test_next_to_one(d):
    check(InfinitePlaneKernel(0.0), [0.0, d], [0.0, 0.0], [1.0, 2.0])


@pytest.mark.parametrize("d", [1e-160, 3e-155, 1e-150, 1e153])
def test_range_of_the_argument(d):
    """1e-160 and 3e-155 have subnormal squares (1e-320 keeps three digits: its own rounding is the
    argument's, taken from the computed square)."""
    rng = np.random.default_rng(3)
    x = np.concatenate([rng.random(200), [0.0, d]])
    y = np.concatenate([rng.random(200), [0.0, 0.0]])
    g = rng.standard_normal(202)
    k = InfinitePlaneKernel(0.0)
    got = k.invariants(VortexSystem(x, y, g)).hamiltonian
    X, Y, G = x.astype(LD), y.astype(LD), g.astype(LD)
    i, j = np.triu_indices(202, 1)
    arg = (X[i] - X[j]) ** 2 + (Y[i] - Y[j]) ** 2
    arg[-1] = LD(d * d)
    w, l = G[i] * G[j], np.log(arg)
    want = -np.sum(w * l) / (4 * LD(np.pi))
    assert abs(LD(got) - want) <= (np.sum(abs(w) * (3 + 3 * abs(l))) / (4 * np.pi) + 2 * abs(want)) * EPS


@pytest.mark.parametrize("kernel", [lambda: InfinitePlaneKernel(0.0), lambda: DiskKernel(1.0)])
def test_coincident_pair_in_the_last_tile(kernel):
    rng = np.random.default_rng(4)
    x, y = 0.5 * rng.random(300), 0.5 * rng.random(300)
    x[299], y[299] = x[290], y[290]
    with pytest.raises(RuntimeError, match="coincident"):
        kernel().invariants(VortexSystem(x, y, np.ones(300)))


@pytest.mark.parametrize("n", [31, 33, 63, 65, 97, 160, 2047, 2048, 2049, 4096, 4097])
@pytest.mark.parametrize("radius", [None, 1.0])
def test_shared_tiles(n, radius):
    """The shares of a tile's sources that four blocks take up to 2048 vortices
    and two up to 4096, whole, ragged and empty."""
    test_tiles(n, radius)

"""Row blocks of the text formatter at their edges: sizes around the 128 rows of a block, rows of
every length (so that a block's text starts at every offset within a word), and the longest values.
Byte for byte against rows written with "%.17g"."""
import numpy as np
import pytest

from pointvortex_b200.kernel import InfinitePlaneKernel, VelocityField, VortexSystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 383, 16385, 131073])
def test_frames(n):
    rng = np.random.default_rng(n)
    cols = rng.standard_normal((5, n)) * 10.0 ** rng.integers(-3, 4, (5, n))
    cols[:, ::7] = np.round(cols[:, ::7])
    cols[:, ::5] *= 10.0 ** rng.integers(-300, 290)
    cols[:, 0] = -1.2345678901234567e-308
    cols[3, n // 2] = -2.2250738585072014e-308
    x, y, g, u, v = cols
    k = InfinitePlaneKernel(0.0)
    text = k.formatTrajectoryHost(-1.2345678901234567e-300, 12345678901234567890, VortexSystem(x, y, g),
                                  VelocityField(u, v))
    want = "".join("%.17g,%d,%d,%.17g,%.17g,%.17g,%.17g,%.17g\n" %
                   (-1.2345678901234567e-300, 12345678901234567890, i, *cols[:, i]) for i in range(n))
    assert text.decode() == want
    k.uploadDeviceState(VortexSystem(x, y, g))
    block = "".join("%.17g %.17g %.17g\n" % (x[i], y[i], g[i]) for i in range(n))
    assert k.formatCheckpointVortices().decode() == block

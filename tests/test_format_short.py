"""The two-word path of the formatter (pointvortex_b200/csrc/pv_format.cuh, 5^s with 0 <= s <= 27)
at its edges, compiled for the host: both sides of the sizes where it hands over to the long numbers,
exact ties (m / 4 and m / 8 with odd m end in a 5 after 17 digits), shifts by a whole word, and
trailing zeros in every form. Text is compared byte for byte with a correctly rounded "%.17g"."""
import numpy as np
import pytest

from test_format import fmt_many, harness  # noqa: F401


def values(kind):
    rng = np.random.default_rng(11)
    odd = (rng.integers(2 ** 51, 2 ** 52, 20_000) * 2 + 1).astype(np.float64)
    if kind == "ties":
        return np.concatenate([odd / 4, odd / 8, odd / 16, odd / 2, odd])
    if kind == "decades":  # s = 16 - k from 30 down to -2, with both neighbours of each power of ten
        p = np.array([float(f"{d}e{k}") for k in range(-14, 19) for d in (1, 2, 5, 9.5, 9.999999999999999)])
        return np.concatenate([p, np.nextafter(p, 0), np.nextafter(p, np.inf)])
    if kind == "binades":
        m = np.concatenate([[1.0, 1.5, 2.0 - 2.0 ** -52], 1.0 + rng.random(40)])
        return np.ldexp(m[:, None], np.arange(-45, 62)[None, :]).ravel()
    if kind == "zeros":  # few digits: zeros to cut before and after the point
        return np.array([d * 10.0 ** k for d in (1, 7, 10, 12, 120, 1001) for k in range(-12, 18)])
    return rng.standard_normal(60_000) * 10.0 ** rng.integers(-14, 19, 60_000)


@pytest.mark.parametrize("kind", ["ties", "decades", "binades", "zeros", "random"])
def test_two_word_path(harness, kind):  # noqa: F811
    v = values(kind)
    v = np.concatenate([v, -v])
    want = ["%.17g" % float(x) for x in v]
    assert fmt_many(harness, v) == want


def test_counts(harness):  # noqa: F811
    import ctypes
    buf = ctypes.create_string_buffer(32)
    for p in range(20):
        for v in (10 ** p - 1, 10 ** p, 10 ** p + 1, 2 ** 32 - 1, 2 ** 32, 2 ** 64 - 1):
            harness.pvf_format_u64(v, buf)
            assert buf.value.decode() == str(v)

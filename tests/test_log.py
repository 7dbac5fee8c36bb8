"""The pair energies' logarithm (pointvortex_b200/csrc/pv_log.cuh) compiled for the host, against a
50-digit logarithm: every table point, both edges of every interval, the neighbourhood of 1, and the
whole range of exponents.

Bound: the sum k log 2 + T is exact and T is good to 0.01 units; the last addition rounds by half a
unit; the tail is rounded by half a unit of its own, at most the result's (next to 1, where |T| is
twice the largest tail; where T = 0 the tail is the result and nothing is added); the polynomial and its
roundings, 2^-8 of the tail, stay below 0.05: 1.1 units."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("log") / "liblog_harness.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-mfma", "-shared", "-fPIC", "-o", str(out),
                    os.path.join(HERE, "native", "log_harness.cpp")], check=True)
    f = ctypes.CDLL(str(out)).pvl_log_many
    f.restype = ctypes.c_size_t
    f.argtypes = [ctypes.POINTER(ctypes.c_double), ctypes.c_size_t, ctypes.POINTER(ctypes.c_double)]
    return f


def logs(lib, v):
    v = np.ascontiguousarray(v, dtype=np.float64)
    out = np.zeros_like(v)
    p = ctypes.POINTER(ctypes.c_double)
    return lib(v.ctypes.data_as(p), v.size, out.ctypes.data_as(p)), out


def values(kind):
    rng = np.random.default_rng(5)
    if kind == "points":
        m = 1.0 + np.arange(129) / 128
        edges = 1.0 + (np.arange(128) + 0.5) / 128
        v = np.concatenate([m, edges, np.nextafter(edges, 0), np.nextafter(m, 0), np.nextafter(m, 3)])
        return np.concatenate([v, v / 2, v * 8, v * 2.0 ** -30])
    if kind == "near 1":
        d = 2.0 ** -np.arange(1.0, 53.0)
        return np.concatenate([1 + d, 1 - d / 2, 1 + d * rng.random(52), 1 - d * rng.random(52), [1.0]])
    if kind == "exponents":
        return np.ldexp(1.0 + rng.random(2046), np.arange(-1022, 1024))
    return np.exp(rng.normal(0, 2, 20_000))


@pytest.mark.parametrize("kind", ["points", "near 1", "exponents", "random"])
def test_against_50_digits(lib, kind):
    v = values(kind)
    refused, got = logs(lib, v)
    assert refused == 0
    mpmath.mp.dps = 50
    for x, y in zip(v, got):
        want = mpmath.log(mpmath.mpf(float(x)))
        if want == 0:
            assert y == 0.0
            continue
        ulp = np.spacing(abs(float(want)))
        assert abs(mpmath.mpf(float(y)) - want) <= 1.1 * ulp, (x, y)


def test_refuses_what_is_not_positive_and_normal(lib):
    v = [0.0, -0.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072009e-308, -1e-310]
    assert logs(lib, v)[0] == len(v)
    assert logs(lib, [2.2250738585072014e-308, 1.7976931348623157e308])[0] == 0

"""The word of the small steps' grid barrier (pointvortex_b200/csrc/pv_barrier.cuh) compiled for the host: a
barrier opens at its last arrival and not before, from the launch on and where the count of arrivals passes
2^40 (148 CTAs meet four times an RK4 step: a launch of two thousand million steps gets there), and errors
and breaks show at their own barrier only."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
M64 = (1 << 64) - 1


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("barrier") / "libbarrier_harness.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(out),
                    os.path.join(HERE, "native", "barrier_harness.cpp")], check=True)
    f = ctypes.CDLL(str(out))
    u64, u32 = ctypes.c_ulonglong, ctypes.c_uint
    for name, res, args in (("arrival", u64, [ctypes.c_int, u32]), ("arrivals", u64, [u32]),
                            ("open", ctypes.c_int, [u64, u64]), ("errors", ctypes.c_int, [u64, u32]),
                            ("broken", u64, [u32]), ("max_ctas", u32, [])):
        fn = getattr(f, "pvl_" + name)
        fn.restype, fn.argtypes = res, args
    return f


@pytest.mark.parametrize("ctas", [1, 2, 16, 148, 2047])
@pytest.mark.parametrize("done", [0, (1 << 40) // 3, (1 << 40) - 2047 * 2, (1 << 40) - 1, 1 << 40, (1 << 41) + 5])
def test_opens_at_the_last_arrival(lib, ctas, done):
    """done: barriers' arrivals already counted, rounded to whole barriers."""
    assert ctas <= lib.pvl_max_ctas()
    rounds = done // ctas
    word = open_at = 0
    for bit in reversed(range(64)):  # rounds * arrivals, by doubling, with the carries of additions
        word = (word + word) & M64
        open_at = (open_at + open_at) & M64
        if rounds >> bit & 1:
            word = (word + lib.pvl_arrivals(ctas)) & M64
            open_at = (open_at + lib.pvl_arrivals(ctas)) & M64
    assert lib.pvl_open(word, open_at)
    for r in range(4):
        parity = (rounds + r + 1) & 1
        before = open_at
        open_at = (open_at + lib.pvl_arrivals(ctas)) & M64
        for c in range(ctas):
            assert not lib.pvl_open(word, open_at)
            word = (word + lib.pvl_arrival(0, parity)) & M64
        assert lib.pvl_open(word, open_at)
        assert lib.pvl_open(word, before)  # a poller that is one barrier behind
        assert not lib.pvl_errors(word, 0) and not lib.pvl_errors(word, 1)


@pytest.mark.parametrize("parity", [0, 1])
def test_errors_and_breaks_keep_to_their_barrier(lib, parity):
    ctas = lib.pvl_max_ctas()
    word = 0
    for c in range(ctas):  # every CTA met one
        assert not lib.pvl_open(word, lib.pvl_arrivals(ctas))
        word = (word + lib.pvl_arrival(1, parity)) & M64
        assert lib.pvl_errors(word, parity) and not lib.pvl_errors(word, parity ^ 1)
        assert not word & (lib.pvl_broken(0) | lib.pvl_broken(1))
    assert lib.pvl_open(word, lib.pvl_arrivals(ctas))
    broken = word | lib.pvl_broken(parity)
    assert broken != word and not broken & lib.pvl_broken(parity ^ 1)
    assert lib.pvl_open(broken, lib.pvl_arrivals(ctas))
    assert not lib.pvl_open(broken, 2 * lib.pvl_arrivals(ctas))

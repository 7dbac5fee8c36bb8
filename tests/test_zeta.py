"""The periodic box's rational pair term, evaluated on the CPU with the header's coefficients
(csrc/pv_geometry.cuh, ZetaPair): both components against the reference's truncated image sums
(src/compute.cpp:234-240) in extended precision, over the whole box -- seams, corners and close pairs
among the points.

Tolerance: the coefficients are good to 6.6e-18 of zeta's part F/z of the term, and its double
evaluation here (no fused multiply-adds: at most about 16 roundings on the longest path, of which
those of the two polynomials count fully) stays below 16 * 2^-53 = 1.8e-15 of |F/z|; the linear part
pi conj(z)/L^2 is at most of F/z's own size in the box. |F/z| <= |K| + |z|/L with K the term itself."""
import pathlib
import re

import numpy as np

HEADER = pathlib.Path(__file__).resolve().parent.parent / "pointvortex_b200" / "csrc" / "pv_geometry.cuh"
LD = np.longdouble
PI = LD("3.14159265358979323846264338327950288")


def _coefficients(name):
    body = re.search(rf"{name}\[\d\] = \{{([^}}]+)\}}", HEADER.read_text()).group(1)
    return [LD(c.strip()) for c in body.split(",")]


def _scaled(length):
    """The host's scaling: units of L/2, times L/pi, a monic denominator."""
    p, q = _coefficients("kZetaP"), _coefficients("kZetaQ")
    unit4 = (LD(2) / LD(length)) ** 4
    lead = q[3] * unit4 ** 3
    return ([float(c * unit4 ** k * LD(length) / PI / lead) for k, c in enumerate(p)],
            [float(c * unit4 ** k / lead) for k, c in enumerate(q[:3])])


def _term(x, y, length):
    zp, zq = _scaled(length)
    yy = y * y
    a, r, b = x * x - yy, x * x + yy, x * y
    r2 = r * r
    n = r2 * r2
    wr, wi = r2 - 8.0 * (b * b), 4.0 * (a * b)
    tr = wr + wr
    p4 = tr * zp[5] + zp[4]
    p3 = tr * p4 + (zp[3] - n * zp[5])
    p2 = tr * p3 + (zp[2] - n * p4)
    p1 = tr * p2 + (zp[1] - n * p3)
    pr, pi = wr * p1 + (zp[0] - n * p2), wi * p1
    q2 = tr + zq[2]
    q1 = tr * q2 + (zq[1] - n)
    qr, qi = wr * q1 + (zq[0] - n * q2), wi * q1
    dr, di = x * qr - y * qi, x * qi + y * qr
    den = dr * dr + di * di
    return (pr * di - pi * dr) / den - y / length, (pr * dr + pi * di) / den - x / length


def _reference(x, y, length, layers=8):
    hx, hy = (2 * PI / LD(length)) * x.astype(LD), (2 * PI / LD(length)) * y.astype(LD)
    su, sv = np.zeros_like(hx), np.zeros_like(hx)
    for m in range(-layers, layers + 1):
        ax, ay = hx - 2 * PI * m, hy - 2 * PI * m
        near_x, near_y = abs(ax) <= 40, abs(ay) <= 40
        su += np.where(near_x, LD(0.5) / (np.sinh(np.where(near_x, ax, 1) / 2) ** 2 + np.sin(hy / 2) ** 2), 0)
        sv += np.where(near_y, LD(0.5) / (np.sinh(np.where(near_y, ay, 1) / 2) ** 2 + np.sin(hx / 2) ** 2), 0)
    return np.sin(hy) * su, np.sin(hx) * sv


def _points(length):
    rng = np.random.default_rng(3)
    half = 0.5 * length
    x, y = rng.uniform(-half, half, 4000), rng.uniform(-half, half, 4000)
    x[:400] = half * np.sign(x[:400])              # seams and corners
    y[200:600] = half * np.sign(y[200:600])
    x[600:1200] *= 10.0 ** rng.uniform(-8, 0, 600)  # close pairs
    y[600:1200] *= 10.0 ** rng.uniform(-8, 0, 600)
    return x, y


def test_rational_term_matches_the_image_sums():
    for length in (2 * np.pi, 2.0, 1.0 / 65536.0, 65536.0, 0.3):
        x, y = _points(length)
        ku, kv = _term(x, y, length)
        ru, rv = _reference(x, y, length)
        scale = np.hypot(ru, rv) + np.hypot(x, y) / length
        assert np.max(np.hypot(ku - ru, kv - rv) / scale) <= 16 * 2.0 ** -53, length


def test_exchange_negates_the_term_exactly():
    x, y = _points(2 * np.pi)
    a, b = _term(x, y, 2 * np.pi), _term(-x, -y, 2 * np.pi)
    assert np.array_equal(a[0], -b[0]) and np.array_equal(a[1], -b[1])


def test_energy_matches_the_image_logarithms():
    """box_energy against the reference's sum (src/compute.cpp:186-196), both in extended precision:
    what is checked are the coefficients, good to 8.8e-19 of sigma and rounded to double, so within
    2 * 2^-53 per coefficient's share (below 1.2 in sum) of the logarithm."""
    s = _coefficients("kZetaS")
    e0 = LD(re.search(r"kEnergyConstant = ([-0-9.]+);", HEADER.read_text()).group(1))
    for length in (2 * np.pi, 0.3):
        x, y = _points(length)
        x, y = x.astype(LD), y.astype(LD)
        w = ((x + 1j * y) * 2 / LD(length)) ** 4
        poly = sum(LD(c) * w ** k for k, c in enumerate(s))
        r = x * x + y * y
        got = e0 + 2 * np.log(2 * PI / LD(length)) - PI * r / LD(length) ** 2 + np.log(r * abs(poly) ** 2)
        hx, hy = 2 * PI / LD(length) * x, 2 * PI / LD(length) * y
        want = -hx * hx / (2 * PI) + np.log(2 * (np.sinh(hx / 2) ** 2 + np.sin(hy / 2) ** 2))
        for m in range(1, 9):
            a = 2 * PI * m
            # (cosh(x - a) - cos y)(cosh(x + a) - cos y) / cosh^2 a
            want += np.log((np.cosh(hx) / np.cosh(a) - np.cos(hy)) ** 2 + (np.tanh(a) * np.sin(hy)) ** 2)
        assert np.max(np.abs(got - want)) <= 4 * 2.0 ** -53

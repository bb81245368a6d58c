"""The FP64 form's fixed-point pair arithmetic (mdg_fixed.cuh), built for the host, against exact rational arithmetic.

Bounds, from the formats: a position is exact to 2^-55 modulo 8; r^2 is off by
the float rounding of its cross products (at most four roundings of
2 sum |d| 2^-29, that is 2^-49 r) plus 2^-56; the force factor follows with its
slope 96 y^5 + 336 y^8 in r^2 (y = r^-2), 48 y^4 2^-58 from the cut of y^3 and
2^-51 from the last units; the products add 2^-53 of the force and 2^-51.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
RC = 2.5


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed") / "fixed.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixed_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def _p(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def test_positions_exact_modulo_8(lib):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-8, 400, 500), rng.uniform(-1, 1, 300), [0.0, 8.0, -8.0, 4.0, 3.9999999999999996, 1e-300, 0.25, -0.25]])
    out = np.zeros((len(x), 2))
    lib.fixed_positions(_p(x), len(x), _p(out))
    for v, (hi, lo) in zip(x, out):
        d = (Fraction(float(v)) - Fraction(float(hi)) - Fraction(float(lo))) % 8
        d = min(d, 8 - d)
        assert d <= (0 if abs(v) >= 0.25 else Fraction(1, 2 ** 55)), v


def _exact(qi, qj, c2x8):
    d = [Fraction(float(b)) - Fraction(float(a)) for a, b in zip(qi, qj)]
    r2 = sum(v * v for v in d)
    y = 1 / r2
    df = 24 * y ** 4 - 48 * y ** 7 + Fraction(c2x8)
    return [df * v for v in d], r2


@pytest.mark.parametrize("lo,hi", [(0.92, 0.95), (0.95, 1.0), (1.0, 1.122), (1.122, 1.5), (1.5, 2.0), (2.0, 2.5)])
def test_pair_force_against_exact_arithmetic(lib, lo, hi):
    s2 = 1.0 / RC ** 2
    c2x8 = 8.0 * (6.0 * s2 ** 7 - 3.0 * s2 ** 4)
    rng = np.random.default_rng(int(1000 * lo))
    n = 400
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    qi = rng.uniform(0, 200, (n, 3))
    qj = qi + u * rng.uniform(lo, hi, (n, 1))
    f, r2 = np.zeros((n, 3)), np.zeros(n)
    lib.fixed_forces(_p(qi), _p(qj), n, ctypes.c_double(c2x8), _p(f), _p(r2))
    worst = np.zeros(2)
    for k in range(n):
        ex, er2 = _exact(qi[k], qj[k], c2x8)
        r, y = float(er2) ** 0.5, 1.0 / float(er2)
        dr2 = 2.0 ** -49 * r + 2.0 ** -56
        assert abs(float(Fraction(float(r2[k])) - er2)) <= dr2 + float(er2) * 2.0 ** -53
        ddf = (96 * y ** 5 + 336 * y ** 8) * dr2 + 48 * y ** 4 * 2.0 ** -58 + 2.0 ** -51
        size = max(abs(float(v)) for v in ex)
        err = max(abs(float(Fraction(float(a)) - b)) for a, b in zip(f[k], ex))
        assert err <= r * ddf + 2.0 ** -53 * size + 2.0 ** -51
        # the double expression on the same inputs
        d = qj[k] - qi[k]
        q2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        inv = 1.0 / q2
        i6 = inv * inv * inv
        g = ((i6 * inv) * (24.0 - 48.0 * i6) + c2x8) * d
        worst += [err ** 2, max(abs(float(Fraction(float(a)) - b)) for a, b in zip(g, ex)) ** 2]
    # no less exact than the double expression where the pair force matters (above 2^-51 absolute)
    assert worst[0] <= worst[1] + n * 2.0 ** -102

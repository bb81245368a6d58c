"""The fixed-point pair force of far pairs (mdg_fixed.cuh), built for the host, against exact arithmetic.

The force factor and the sums have fixed units, so a pair's error does not
shrink with its force: the bound of test_fixed.py by itself, without a comparison
with the double expression, whose error is relative and smaller from 2 sigma on.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("far") / "far.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixed_check.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("rc,lo,hi", [(2.5, 1.5, 2.0), (2.5, 2.0, 2.3), (2.5, 2.3, 2.5), (3.5, 2.5, 3.0), (3.5, 3.0, 3.5)])
def test_far_pairs(lib, rc, lo, hi):
    s2 = 1.0 / rc ** 2
    c2x8 = 8.0 * (6.0 * s2 ** 7 - 3.0 * s2 ** 4)
    rng = np.random.default_rng(int(1000 * lo))
    n = 600
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    qi = rng.uniform(0, 200, (n, 3))
    qj = qi + u * rng.uniform(lo, hi, (n, 1))
    f, r2 = np.zeros((n, 3)), np.zeros(n)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    lib.fixed_forces(p(qi), p(qj), n, ctypes.c_double(c2x8), p(f), p(r2))
    for k in range(n):
        d = [Fraction(float(b)) - Fraction(float(a)) for a, b in zip(qi[k], qj[k])]
        er2 = sum(v * v for v in d)
        ey = 1 / er2
        df = 24 * ey ** 4 - 48 * ey ** 7 + Fraction(c2x8)
        r, y = float(er2) ** 0.5, float(ey)
        dr2 = 2.0 ** -49 * r + 2.0 ** -56
        ddf = (96 * y ** 5 + 336 * y ** 8) * dr2 + 48 * y ** 4 * 2.0 ** -58 + 2.0 ** -51
        size = max(abs(float(df * v)) for v in d)
        err = max(abs(float(Fraction(float(a)) - df * v)) for a, v in zip(f[k], d))
        assert err <= r * ddf + 2.0 ** -53 * size + 2.0 ** -51

"""r^2 of pairs across the box's faces in fixed point (mdg_fixed.cuh), built for the host, against exact arithmetic.

Three rests add up in such a pair's separation: its own, the partner's and the
box side's, up to 0.75 units of 2^-28 an axis.  Bound: each rest is off by 2^-27
units, the two sums by 2^-26 and 2^-25, together less than 2^-24 (2^-52 sigma,
2 sum |d| of it in r^2); the cross products are rounded four times, relative
2^-24 of 2 sum |d| 0.75 2^-28, that is 6 sum |d| 2^-52; so sum |d| 2^-49, and 2^-54
for the rests' own squares and the last unit.
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
    so = str(tmp_path_factory.mktemp("faces") / "faces.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", os.path.join(HERE, "fixed_faces_check.cpp"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def _with_rest(x, rest):
    """The multiple of 2^-29 next to x, plus `rest` of them."""
    return (np.floor(x * 2.0 ** 29) + rest) * 2.0 ** -29


# the longest separations of the single box and the batch (3.6), the adjoint and the observers without a handle (3.9), and shorter
@pytest.mark.parametrize("r", [1.0, 2.5, 3.0, 3.2, 3.4, 3.6, 3.89])
@pytest.mark.parametrize("rest", [0.49, 0.3, "any"])
def test_corner_pairs(lib, r, rest):
    rng = np.random.default_rng(int(1000 * r))
    n = 400
    L = rng.uniform(8.0, 200.0, (n, 3))
    s = rng.choice([-1, 1], (n, 3))
    # particles near opposite faces, so that qj + s L - qi has length r along a direction near a corner's
    u = np.abs(rng.normal(1.0, 0.2, (n, 3)))
    u /= np.linalg.norm(u, axis=1)[:, None]
    d = s * u * r * rng.uniform(0.97, 1.0, (n, 1))
    part = rng.uniform(0.0, 1.0, (n, 3))
    qi = np.where(s > 0, L - part * np.abs(d), part * np.abs(d))
    qj = qi + d - s * L
    if rest != "any":  # every rest as far out as it gets, all with the same sign in the separation
        e = rng.uniform(0.98, 1.0, (3, n, 3)) * rest
        L, qi, qj = _with_rest(L, s * e[0]), _with_rest(qi, -e[1]), _with_rest(qj, e[2])
    out = np.zeros((n, 2))
    pd, pi = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    si = np.ascontiguousarray(s, dtype=np.int32)
    lib.fixed_image_r2(qi.ctypes.data_as(pd), qj.ctypes.data_as(pd), si.ctypes.data_as(pi), L.ctypes.data_as(pd), n,
                       out.ctypes.data_as(pd))
    for k in range(n):
        sep = [Fraction(float(qj[k, c])) + int(s[k, c]) * Fraction(float(L[k, c])) - Fraction(float(qi[k, c])) for c in range(3)]
        exact = sum(v * v for v in sep)
        got = (Fraction(int(out[k, 0])) * 2 ** 32 + int(out[k, 1])) / Fraction(2) ** 58
        bound = sum(abs(v) for v in sep) * Fraction(1, 2 ** 49) + Fraction(1, 2 ** 54)
        assert abs(got - exact) <= bound, (k, float(got - exact), float(bound))

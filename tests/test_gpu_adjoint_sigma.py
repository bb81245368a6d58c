"""The adjoint's fixed-point sums at the ends of the sigma range that takes them, against its double form.

The same trajectory with a margin whose search length leaves the fixed-point
range: J to 1e-13, gradients to 1e-11, as test_gpu_fixed.py's cases at sigma near 1.
"""
import numpy as np
import pytest

from tests.helpers import liquid_like

pytestmark = pytest.mark.gpu


def _both(q, p, L, cutoff, margins, **kw):
    from mdacp_gb300.adjoint import Adjoint
    out = []
    for margin in margins:
        a = Adjoint(L, len(q), cutoff=cutoff, margin=margin, **kw)
        out.append((a.forward(q, p),) + a.backward())
    return out


@pytest.mark.parametrize("objective", ["pe", "pressure"])
@pytest.mark.parametrize("sigma,cutoff", [(0.8, 2.3), (1.5, 1.7), (1.8, 1.5), (1.8, 1.02)])
def test_liquid_at_the_ends_of_the_range(sigma, cutoff, objective):
    q, p, L = liquid_like(0.7 / sigma ** 3, 5, amp=0.08 * sigma, temperature=0.7, seed=7)
    q[11] = np.mod(q[10] + [0.85 * sigma, 0.0, 0.0], L)
    (j0, dq0, dp0, de0, ds0), (j1, dq1, dp1, de1, ds1) = _both(q, p, L, cutoff, (0.4, 1.2), steps=13, checkpoint_every=5, dt=0.001,
                                                              epsilon=1.2, sigma=sigma, objective=objective)
    assert abs(j0 - j1) <= 1e-13 * abs(j1)
    assert np.linalg.norm(dq0 - dq1) <= 1e-11 * np.linalg.norm(dq1)
    assert np.linalg.norm(dp0 - dp1) <= 1e-11 * np.linalg.norm(dp1)
    assert abs(de0 - de1) <= 1e-11 * abs(de1) and abs(ds0 - ds1) <= 1e-11 * abs(ds1)


@pytest.mark.parametrize("count", [6, 8, 12, 40])
@pytest.mark.parametrize("sigma", [1.0, 1.8])
def test_crowded_row_of_the_pressure_gradient(sigma, count):
    # `count` partners at 0.93 sigma on one side of a particle: an eighth of the pressure's slope is 166 a pair, at sigma 1.8
    # 279 with the separation, past the integer sums' 2^11 from 8 partners on; a step too short to move anything
    rng = np.random.default_rng(count)
    u = np.array([1.0, 0.0, 0.0]) + 0.02 * rng.normal(size=(count, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    q = np.concatenate([[[5.0, 5.0, 5.0]], np.array([5.0, 5.0, 5.0]) + 0.93 * sigma * u, [[11.0, 11.0, 11.0]]])
    L = np.full(3, 12.0)
    (_, dq0, *_), (_, dq1, *_) = _both(q, np.zeros_like(q), L, 1.5, (0.4, 1.2) if sigma > 1.5 else (0.4, 1.3), steps=1,
                                       checkpoint_every=1, dt=1e-18, sigma=sigma, objective="pressure")
    assert np.linalg.norm(dq0[0] - dq1[0]) <= 1e-11 * np.linalg.norm(dq1[0])

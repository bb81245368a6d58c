"""mdg_observe_noalloc over its forms (fixed-point pair sums, double ones outside their range) against all pairs in float64."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(q, p, L, rc):
    import torch
    from mdacp_gb300 import native
    pad = np.zeros((len(q), 1))
    qd, pd = (torch.from_numpy(np.hstack([x, pad])).cuda() for x in (q, p))
    out = torch.zeros(3, dtype=torch.float64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    assert native.load().mdg_observe_noalloc(ptr(qd), ptr(pd), len(q), (ctypes.c_double * 3)(*L), rc, ptr(out), None) == 0
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _expected(q, p, L, rc):
    """The three sums and the sums of the terms' sizes."""
    d = q[:, None] - q[None]
    d -= L * np.rint(d / L)
    r2 = (d ** 2).sum(-1)[np.triu_indices(len(q), 1)]
    r2 = r2[r2 <= rc * rc]
    s2 = 1.0 / (rc * rc)
    c2 = 6.0 * s2 ** 7 - 3.0 * s2 ** 4
    c0 = -s2 ** 6 + s2 ** 3 - c2 / s2
    terms = [0.5 * p ** 2, 4.0 * (r2 ** -6 - r2 ** -3 + c2 * r2 + c0), (24.0 * r2 ** -3 - 48.0 * r2 ** -6 + 8.0 * c2 * r2) / 3.0]
    return np.array([t.sum() for t in terms]), np.array([np.abs(t).sum() for t in terms])


# 3.9 and beyond, and below 1.0: the double sums; the boxes hold from 2 cells a side up, the particle
# counts from 1 up and more than 32 a cell; positions unwrapped by whole boxes
@pytest.mark.parametrize("rc,cells,n", [(2.5, 2.05, 1), (2.5, 2.05, 37), (2.5, 2.9, 300), (2.5, 4.3, 1200), (1.0, 6.4, 700),
                                        (0.97, 6.4, 700), (3.89, 2.2, 900), (3.95, 2.2, 900), (2.5, 9.1, 2500)])
def test_forms(rc, cells, n):
    rng = np.random.default_rng(int(100 * rc) + n)
    L = np.array([1.0, 1.01, 1.03]) * cells * rc
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    q = (grid[rng.permutation(len(grid))[:n]] + 0.5 + rng.uniform(-0.2, 0.2, (n, 3))) / side * L
    if n > 30:
        q[1] = q[0] + [0.86, 0.0, 0.0]  # a close pair
    p = rng.normal(size=(n, 3))
    want, size = _expected(q, p, L, rc)
    # 2^-50 a term and the rounding of the sums
    assert np.all(np.abs(_call(q, p, L, rc) - want) <= 1e-12 * size + 1e-15 * n)
    shifted = q + L * rng.integers(-1, 2, (n, 3))
    assert np.all(np.abs(_call(shifted, p, L, rc) - want) <= 1e-11 * size + 1e-14 * n)


def test_not_a_number_shows_in_the_sums():
    rng = np.random.default_rng(1)
    L = np.full(3, 12.0)
    q, p = rng.random((200, 3)) * L, np.zeros((200, 3))
    q[17, 1] = np.nan
    out = _call(q, p, L, 2.5)
    assert np.isnan(out[1]) and np.isnan(out[2])

"""mdg_observe_noalloc in nearly empty boxes (a thread per particle below 0.16 particles a cell) against all pairs in float64.

Both sides of the line, cell counts that are and are not a multiple of the scan's
eight, one and several of its rounds (8,192 cells); tolerances as test_gpu_noalloc_forms.py.
"""
import numpy as np
import pytest

from tests.test_gpu_noalloc_forms import _call, _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,n", [(9, 110), (9, 120), (10, 159), (10, 161), (21, 700), (21, 1600), (20, 1000)])
def test_line_between_the_forms(cells, n):
    rc = 2.5
    rng = np.random.default_rng(n)
    L = np.array([1.0, 1.01, 1.03]) * (cells + 0.2) * rc
    # groups of up to 4 within reach of one another, the rest far apart
    side = int(np.ceil((n / 4) ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    base = (grid + 0.5) / side * L
    near = np.array([[0.0, 0.0, 0.0], [1.1, 0.0, 0.0], [0.0, 1.05, 0.2], [0.3, 0.4, 1.3]])
    q = (base[:, None] + near[None] + rng.uniform(-0.04, 0.04, (len(base), 4, 3))).reshape(-1, 3)[:n]
    q = np.mod(q - 0.3, L)
    p = rng.normal(size=(n, 3))
    want, size = _expected(q, p, L, rc)
    assert np.all(np.abs(_call(q, p, L, rc) - want) <= 1e-12 * size + 1e-15 * n)

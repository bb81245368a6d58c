"""The pair list against the oracle where the build's warp per cell changes its work: cells of more than 32 particles, more
than 512 candidates, at most 8, 16 or 32 home particles, empty cells, and boxes of so few cells that two warps share one.
"""
import numpy as np
import pytest

from oracle import port
from tests.helpers import directed_pair_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,n,clumped", [(3, 40, False), (3, 900, False), (3, 2400, False), (7, 2500, False), (5, 3000, True),
                                             (15, 9000, False), (15, 40000, False), (16, 6000, True)])
def test_pair_list_of_a_cell_per_warp(cells, n, clumped):
    from mdacp_gb300.manager import MDManager
    rng = np.random.default_rng(cells * n)
    L = np.full(3, cells * 2.02)
    q = rng.random((n, 3)) * L
    if clumped:  # most particles in a corner, across the faces
        k = n // 2
        q[:k] = np.mod(rng.normal(0.0, 1.0, (k, 3)), L)
    q = np.minimum(q, np.nextafter(L, 0.0))
    ref = port.System(q, np.zeros_like(q), L, rc=1.8, margin=0.2)
    ref.make_pairlist()
    want = directed_pair_keys(ref.pairs(), n, half=True)
    m = MDManager(L, capacity=n, cutoff=1.8, margin=0.2, precision="mixed")
    m.set_state(q, np.zeros_like(q))
    m.make_pairlist()
    assert np.array_equal(directed_pair_keys(m.pairs(), n, half=False), want)

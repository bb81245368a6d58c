"""The list build of boxes with few particles a cell (one thread per particle) against the oracle's pair set.

Boxes on both sides of the line (six particles a cell, 16,000 cells), empty
cells, two cells along a side, particles on the faces, and rows that outgrow their capacity.
"""
import numpy as np
import pytest

from oracle import port
from tests.helpers import directed_pair_keys, wrap

pytestmark = pytest.mark.gpu

RC, MARGIN = 2.5, 0.5


def _gas(n, box, seed, clump=0):
    rng = np.random.default_rng(seed)
    q = rng.uniform(0.0, 1.0, (n, 3)) * box
    if clump:  # a dense region among the empty cells
        q[:clump] = wrap(rng.uniform(0.0, 4.0, (clump, 3)) - 2.0, box)
    q[-6:-3] = 0.0                      # on the lower faces
    q[-6:-3] += rng.uniform(0.0, 1e-9, (3, 3))
    q[-3:] = np.nextafter(box, 0.0)     # and just below the upper ones
    q[-1] += np.array([-1.0, -1.5, 0.0])
    return q


def _check(q, box, precision="fp64", **kw):
    from mdacp_gb300.manager import MDManager
    m = MDManager(box, capacity=len(q), cutoff=RC, margin=MARGIN, precision=precision, **kw)
    m.set_state(q, np.zeros_like(q))
    m.make_pairlist()
    ref = port.System(q, np.zeros_like(q), box, rc=RC, margin=MARGIN)
    ref.make_pairlist()
    n = len(q)
    assert np.array_equal(directed_pair_keys(m.pairs(), n, half=False), directed_pair_keys(ref.pairs(), n, half=True))
    return m.stats()


# cells: 27,000 in a cube, 16,128 and 15,872 just about the line, 18,000 with two along one side
@pytest.mark.parametrize("cells", [(30, 30, 30), (32, 28, 18), (32, 31, 16), (150, 60, 2)])
@pytest.mark.parametrize("per_cell", [0.05, 0.9, 5.8, 6.2])
def test_pair_set(cells, per_cell):
    box = np.array(cells) * 3.01
    st = _check(_gas(int(per_cell * np.prod(cells)), box, int(10 * per_cell), clump=100), box)
    assert st["cells"] == cells


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_overflow_in_a_gas(precision):
    box = np.array([30, 30, 30]) * 3.01
    st = _check(_gas(20001, box, 3, clump=400), box, precision, list_capacity=16)
    assert st["list_capacity"] >= st["max_neighbours"] > 16

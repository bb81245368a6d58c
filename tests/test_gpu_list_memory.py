"""Neighbour lists that do not fit the GPU's memory: an error on every call, no access to rows that are not there, and use afterwards.

A clump needs rows of a few thousand entries at a capacity (or beside so many
particles) that they would take over 300 GB.
"""
import ctypes

import numpy as np
import pytest

from tests.helpers import liquid_like

pytestmark = pytest.mark.gpu


def _clump(n, L):
    # n particles within a tenth of sigma: rows of n - 1
    return 0.5 * L + np.random.default_rng(1).uniform(-0.05, 0.05, (n, 3))


@pytest.mark.parametrize("precision,graphs", [("fp64", 1), ("fp64", 2), ("mixed", 1), ("mixed", 0)])
def test_single_box(precision, graphs):
    from mdacp_gb300 import native
    from mdacp_gb300.manager import MDManager
    q, p, L = liquid_like(0.7, 6, amp=0.05, seed=2)
    c = _clump(2600, L)
    m = MDManager(L, capacity=40000000, cutoff=2.5, margin=0.5, precision=precision, use_graphs=graphs)
    for _ in range(2):
        m.set_state(c, np.zeros_like(c))
        for call in (m.make_pairlist, m.observe_raw, m.forces, lambda: (m.calculate(3), m.synchronize())):
            with pytest.raises(native.MDGError, match="neighbour list"):
                call()
    m.set_state(q, p)
    m.calculate(20)
    small = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.5, precision=precision, use_graphs=graphs)
    small.set_state(q, p)
    small.calculate(20)
    assert np.array_equal(np.concatenate(m.state()), np.concatenate(small.state()))


@pytest.mark.parametrize("flat", [False, True])
def test_batch(flat):
    # a clump in one box, many particles in the others: every box's rows have the longest one's capacity
    from mdacp_gb300 import native
    from mdacp_gb300.batch import Batch
    q, p, L = liquid_like(0.7, 16, amp=0.05, seed=3)
    c = _clump(3000, L)
    boxes = [(q, p, L)] * 1300 + [(c, np.zeros_like(c), L)]
    b = Batch(boxes, cutoff=2.5, margin=0.4, precision="mixed", list_capacity=96)
    b.set_shape(256, 1, 2)
    b.set_flat(flat)
    for call in (b.observe_raw, lambda: b.calculate(3), b.observe_raw):
        with pytest.raises(native.MDGError, match="neighbour list"):
            call()
    ordinary = [(q, p, L)] * 1300 + [(q[:3000], p[:3000], L)]
    q4, p4 = (np.concatenate([np.hstack([x[k], np.zeros((len(x[k]), 1))]) for x in ordinary]) for k in (0, 1))
    dp = ctypes.POINTER(ctypes.c_double)
    b._ck(b.lib.mdg_batch_set_state(b._h, q4.ctypes.data_as(dp), p4.ctypes.data_as(dp)))
    b.calculate(5)
    sums = b.observe_raw()
    one = Batch([ordinary[0], ordinary[-1]], cutoff=2.5, margin=0.4, precision="mixed")
    one.set_shape(256, 1, 2)
    one.set_flat(flat)
    one.calculate(5)
    np.testing.assert_allclose(sums[[0, 1299, 1300]], one.observe_raw()[[0, 0, 1]], rtol=1e-12)

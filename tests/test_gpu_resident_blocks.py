"""The resident kernel beside other handles with steps outstanding: narrow launches, or graphs for larger mixed boxes.

On 152 SMs: at least 128 particles a block, 256 threads from 9,729 to 38,912 particles; from there
graphs beside two other handles, from 152,001 beside one.  The particles' arithmetic does
not depend on any of it: bit for bit as plain step launches.
"""
import threading

import numpy as np
import pytest

from tests.helpers import liquid_like
from tests.test_gpu_resident import _run

pytestmark = pytest.mark.gpu


def _box(n, seed):
    cells = int(np.ceil((n / 4) ** (1 / 3)))
    q, p, L = liquid_like(0.8, cells, amp=0.08, temperature=1.4, seed=seed)
    return q[:n].copy(), p[:n] - p[:n].mean(axis=0), L


def _outstanding(count):
    """Handles of 500 particles with steps that nobody has asked for yet."""
    from mdacp_gb300.manager import MDManager
    q, p, L = _box(500, 1)
    out = []
    for _ in range(count):
        m = MDManager(L, capacity=500, cutoff=2.5, margin=0.3, precision="mixed")
        m.set_state(q, p)
        m.calculate(20)
        out.append(m)
    return out


@pytest.mark.parametrize("precision,thermostat,n,others", [
    ("mixed", "nve", 500, 1), ("mixed", "langevin", 4001, 2), ("mixed_plain", "nve", 9728, 1), ("mixed", "nve", 9729, 3),
    ("mixed_plain", "langevin", 19457, 1), ("mixed", "langevin", 38912, 1), ("mixed_plain", "nve", 38913, 1),
    ("mixed", "nve", 38913, 2), ("mixed", "langevin", 152001, 1)])
def test_beside_other_handles(precision, thermostat, n, others):
    q, p, L = _box(n, n)
    kw = dict(precision=precision, thermostat=thermostat, dt=0.004)
    steps = 50 if n < 50000 else 25
    s0, _, st0 = _run(q, p, L, [steps], False, **kw)
    beside = _outstanding(others)
    s1, _, st1 = _run(q, p, L, [7, steps - 7], True, **kw)
    assert st0["rebuilds"] > 1 and st0["prunes"] > st0["rebuilds"]
    for key in ("steps", "rebuilds", "prunes", "inner_pairs", "listed_pairs", "max_neighbours"):
        assert st0[key] == st1[key], key
    assert np.array_equal(s0, s1)
    for m in beside:
        m.synchronize()


@pytest.mark.parametrize("n,others,graphs", [(4000, 3, False), (38912, 3, False), (38913, 1, False), (38913, 2, True),
                                             (152000, 1, False), (152001, 1, True), (152001, 0, False)])
def test_way_taken(n, others, graphs):
    # launches of ten steps after the first: one kernel, or two a step and ten a rebuild
    from mdacp_gb300.manager import MDManager
    q, p, L = _box(n, n)
    m = MDManager(L, capacity=n, cutoff=2.5, margin=0.3, precision="mixed", dt=0.002)
    m.set_state(q, p)
    m.calculate(1)
    m.synchronize()
    beside = _outstanding(others)
    before = m.stats()
    m.calculate(10)
    m.synchronize()
    after = m.stats()
    launches, rebuilds = after["kernel_launches"] - before["kernel_launches"], after["rebuilds"] - before["rebuilds"]
    assert launches == (20 + 10 * rebuilds if graphs else 1)
    # confirmed, replaced or destroyed: no longer beside it
    for k, b in enumerate(beside):
        if k == 0:
            b.synchronize()
        elif k == 1:
            b.set_state(*_box(500, 2)[:2])
        else:
            b.close()
    before = m.stats()["kernel_launches"]
    m.calculate(10)
    m.synchronize()
    assert m.stats()["kernel_launches"] - before == 1


def test_several_handles_at_once():
    # from one thread each
    sizes = [864, 4000, 9000, 12000, 864, 20000, 45000]
    boxes = [_box(n, n + k) for k, n in enumerate(sizes)]
    alone = [_run(q, p, L, [60], False, precision="mixed", dt=0.004)[0] for q, p, L in boxes]
    got = [None] * len(boxes)

    def work(k):
        q, p, L = boxes[k]
        got[k] = _run(q, p, L, [20] * 3, True, precision="mixed", dt=0.004)[0]

    for _ in range(2):
        ts = [threading.Thread(target=work, args=(k,)) for k in range(len(boxes))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for a, g in zip(alone, got):
            assert np.array_equal(a, g)

"""Blocks of the mixed resident kernel: sizes where their number changes, and launches of several handles side by side.

On 152 SMs: 32 particles a block up to 2,432, 64 to 4,864 (with the lists by a warp per cell),
as many as fall to it to 6,080, and at least 96 from there.  The particles' arithmetic does not depend on any of it: bit for bit as
plain step launches.
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


@pytest.mark.parametrize("precision,thermostat,n", [
    ("mixed", "nve", 2432), ("mixed", "langevin", 2433), ("mixed_plain", "nve", 4864), ("mixed", "nve", 4865),
    ("mixed", "nve", 6080), ("mixed_plain", "nve", 6081),
    ("mixed_plain", "langevin", 7296), ("mixed", "langevin", 7297), ("mixed_plain", "nve", 9729), ("mixed", "nve", 14593)])
def test_block_sizes(precision, thermostat, n):
    q, p, L = _box(n, n)
    kw = dict(precision=precision, thermostat=thermostat, dt=0.004)
    s0, _, st0 = _run(q, p, L, [50], False, **kw)
    s1, _, st1 = _run(q, p, L, [7, 43], True, **kw)
    assert st0["rebuilds"] > 2 and st0["prunes"] > st0["rebuilds"]
    for key in ("steps", "rebuilds", "prunes", "inner_pairs", "listed_pairs", "max_neighbours"):
        assert st0[key] == st1[key], key
    assert np.array_equal(s0, s1)


def test_several_handles_at_once():
    # launches that share the SMs out, from one thread each
    sizes = [864, 4000, 4500, 7000, 864, 20000]
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

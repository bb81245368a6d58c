"""Steps by graphs (use_graphs = 2) where a small box would otherwise take the resident kernel, and lanes per particle.

The SWITCH graph and plain launches run the same kernels, decided by the
prelude or by the kernels themselves: bit for bit.  Lane counts of the
FP64 form's kernels outside the resident kernel change at 2,432, 9,728 and 38,912
particles: forces, observers and steps against the oracle.
"""
import numpy as np
import pytest

from tests.helpers import liquid_like
from tests.test_gpu_fixed import _check
from tests.test_gpu_resident import _run

pytestmark = pytest.mark.gpu


def _box(n, density=0.8):
    cells = int(np.ceil((n / 4) ** (1 / 3)))
    q, p, L = liquid_like(density, cells, amp=0.08, temperature=1.4, seed=n)
    return q[:n].copy(), p[:n] - p[:n].mean(axis=0), L


@pytest.mark.parametrize("thermostat", ["nve", "langevin", "nosehoover"])
@pytest.mark.parametrize("precision,n", [("fp64", 1500), ("fp64", 10001), ("mixed", 4001), ("mixed_plain", 20000)])
def test_graphs_match_plain_launches(precision, n, thermostat):
    q, p, L = _box(n)
    kw = dict(precision=precision, thermostat=thermostat, dt=0.004)
    s0, o0, st0 = _run(q, p, L, [60], 0, **kw)
    s2, o2, st2 = _run(q, p, L, [1] * 5 + [2, 53], 2, **kw)
    assert st0["rebuilds"] > 2 and st0["prunes"] > st0["rebuilds"]
    for key in ("steps", "rebuilds", "prunes", "inner_pairs", "listed_pairs", "max_neighbours"):
        assert st0[key] == st2[key], key
    assert np.array_equal(s0, s2) and np.array_equal(o0, o2)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_graphs_recover_from_overflow_and_report_bad_states(precision):
    from mdacp_gb300 import native
    from mdacp_gb300.manager import MDManager
    q, p, L = _box(2048)
    ref = _run(q, p, L, [30], 0, precision=precision, dt=0.004)[0]
    m = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.3, precision=precision, dt=0.004, list_capacity=32, use_graphs=2)
    m.set_state(q, p)
    m.calculate(30)
    assert np.array_equal(np.concatenate(m.state()), ref)
    bad = p.copy()
    bad[3] = np.nan
    m.set_state(q, bad)
    with pytest.raises(native.MDGError):
        m.calculate(20)
        m.synchronize()
    m.set_state(q, p)
    m.calculate(30)
    assert np.array_equal(np.concatenate(m.state()), ref)


@pytest.mark.parametrize("graphs", [0, 1, 2])
def test_launches_of_the_three_ways(graphs):
    # ten steps: ten graph steps of two kernels (and the rebuilds'), one resident launch, or every kernel of every step
    q, p, L = _box(864)
    from mdacp_gb300.manager import MDManager
    m = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.3, precision="mixed", use_graphs=graphs)
    m.set_state(q, p)
    m.make_pairlist()
    before = m.stats()
    m.calculate(10)
    m.synchronize()
    after = m.stats()
    launches, rebuilds = after["kernel_launches"] - before["kernel_launches"], after["rebuilds"] - before["rebuilds"]
    assert launches == {0: 110, 1: 1, 2: 20 + 10 * rebuilds}[graphs]


@pytest.mark.parametrize("graphs", [0, 1, 2])
@pytest.mark.parametrize("n", [2431, 2432, 9727, 9728, 38911, 38912])
def test_lane_boundaries(n, graphs):
    q, p, L = _box(n, 0.7)
    _check(q, p, L, steps=10 if n < 20000 else 2, use_graphs=graphs)

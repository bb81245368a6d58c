"""The resident step kernel of small boxes (one cooperative launch per mdg_calculate call) against plain step launches.

The particles' arithmetic is the same, so the mixed forms agree bit for bit
through rebuilds and re-selections, however the steps are split into calls;
FP64 sums the rows' lowest parts over other lanes (2^-54 of a force) and
Nose-Hoover the kinetic energy over other blocks: 1e-12 relative after 60 steps.
"""
import numpy as np
import pytest

from tests.helpers import liquid_like

pytestmark = pytest.mark.gpu


def _run(q, p, L, calls, use_graphs, **kw):
    from mdacp_gb300.manager import MDManager
    m = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.3, use_graphs=use_graphs, gamma=1.0, **kw)
    m.set_state(q, p)
    for k in calls:
        m.calculate(k)
    return np.concatenate(m.state()), m.observe_raw(), m.stats()


# particle counts on both sides of the lane counts and of one pass of 512 or 1,024 threads on 152 SMs
@pytest.mark.parametrize("precision,thermostat,n", [
    ("mixed", "nve", 500), ("mixed", "langevin", 4001), ("mixed_plain", "nve", 77825), ("mixed", "nve", 155649),
    ("mixed_plain", "langevin", 999), ("mixed", "nosehoover", 6000), ("fp64", "nve", 500), ("fp64", "nve", 2433),
    ("fp64", "langevin", 9000), ("fp64", "nosehoover", 20001), ("fp64", "nve", 77824)])
def test_resident_matches_plain_launches(precision, thermostat, n):
    cells = int(np.ceil((n / 4) ** (1 / 3)))
    q, p, L = liquid_like(0.8, cells, amp=0.08, temperature=1.4, seed=n)
    q, p = q[:n].copy(), p[:n] - p[:n].mean(axis=0)
    kw = dict(precision=precision, thermostat=thermostat, dt=0.004)
    steps = 60 if n < 50000 else 25
    s0, o0, st0 = _run(q, p, L, [steps], False, **kw)
    s1, o1, st1 = _run(q, p, L, [1] * 7 + [steps - 7], True, **kw)
    assert st0["rebuilds"] > 2 and st0["prunes"] > st0["rebuilds"]
    for key in ("steps", "rebuilds", "prunes", "inner_pairs", "listed_pairs", "max_neighbours"):
        assert st0[key] == st1[key], key
    if precision != "fp64" and thermostat != "nosehoover":
        assert np.array_equal(s0, s1)
    else:
        np.testing.assert_allclose(s1, s0, rtol=1e-12, atol=1e-12 * np.abs(s0).max())
    np.testing.assert_allclose(o1, o0, rtol=1e-11)


def test_two_boxes_in_turn_on_two_handles():
    # two resident launches outstanding on two streams: each as it runs alone
    from mdacp_gb300.manager import MDManager
    boxes = [liquid_like(0.7, c, amp=0.05, seed=c) for c in (8, 11)]
    alone = [_run(q, p, L, [40], True, precision="mixed")[0] for q, p, L in boxes]
    ms = []
    for q, p, L in boxes:
        m = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.3, precision="mixed")
        m.set_state(q, p)
        ms.append(m)
    for _ in range(40):
        for m in ms:
            m.calculate(1)
    for m, a in zip(ms, alone):
        assert np.array_equal(np.concatenate(m.state()), a)


def test_overflow_and_bad_state_in_the_resident_kernel():
    from mdacp_gb300 import native
    from mdacp_gb300.manager import MDManager
    q, p, L = liquid_like(0.8, 8, amp=0.08, seed=4)
    ref = _run(q, p, L, [30], False, precision="mixed", dt=0.004)[0]
    m = MDManager(L, capacity=len(q), cutoff=2.5, margin=0.3, precision="mixed", dt=0.004, list_capacity=32)
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

"""The FP64 form on fixed-point pair arithmetic: the calls and states where it changes path, against the oracle.

Lanes per particle change with the particle count (12,288 and 65,536); a pair
closer than r^2 = 0.8425 and a row whose sums may overflow take the double
expression; a particle that leaves the modulus's guard sends the step there;
a cut-off below one sigma or a search length near 4 keeps the double kernel.
Forces: |dF_i| <= 1e-12 max(|F_i|, sum |f_ij|), as the parity tests.
"""
import numpy as np
import pytest

from oracle import port
from tests.helpers import liquid_like, pair_force_abs_sum

pytestmark = pytest.mark.gpu


def _manager(L, n, **kw):
    from mdacp_gb300.manager import MDManager
    kw.setdefault("cutoff", 2.5)
    kw.setdefault("margin", 0.5)
    return MDManager(L, capacity=n, **kw)


def _check(q, p, L, steps=20, **kw):
    ref = port.System(q, p, L, rc=kw.get("cutoff", 2.5), margin=kw.get("margin", 0.5), dt=kw.get("dt", 0.001),
                      rebuild_policy=port.REBUILD_HALFMARGIN)
    ref.make_pairlist()
    fr = ref.forces()
    scale = np.maximum(np.linalg.norm(fr, axis=1), pair_force_abs_sum(q, L, ref.pairs(), kw.get("cutoff", 2.5)))
    m = _manager(L, len(q), **kw)
    m.set_state(q, p)
    f = m.forces()
    assert np.all(np.linalg.norm(f - fr, axis=1) <= 1e-12 * scale + 1e-14)
    obs = m.observe_raw()
    np.testing.assert_allclose(obs, ref.observe_raw(), rtol=1e-12)
    if steps:
        ref.calculate(steps)
        m.calculate(steps)
        np.testing.assert_allclose(m.observe_raw(), ref.observe_raw(), rtol=1e-10)
    return m


# particle counts on both sides of the lane thresholds and of block edges
@pytest.mark.parametrize("n", [500, 1001, 12287, 12288, 65535, 65537])
def test_lane_counts(n):
    cells = int(np.ceil((n / 4) ** (1 / 3)))
    q, p, L = liquid_like(0.7, cells, amp=0.08, seed=n)
    q, p = q[:n].copy(), p[:n] - p[:n].mean(axis=0)
    _check(q, p, L, steps=10 if n < 20000 else 2)


# 3.4 + 0.3 fits the modulus, 3.5 + 0.3 does not; a cut-off of 1.12 does, 0.9 does not
@pytest.mark.parametrize("cutoff,margin", [(3.0, 0.3), (3.2, 0.3), (3.5, 0.3), (1.12, 0.3), (0.9, 0.3)])
def test_cutoffs_on_both_paths(cutoff, margin):
    q, p, L = liquid_like(0.6, 7, amp=0.05, seed=3)
    m = _manager(L, len(q), cutoff=cutoff, margin=margin)
    m.set_state(q, p)
    ref = port.System(q, p, L, rc=cutoff, margin=margin, rebuild_policy=port.REBUILD_HALFMARGIN)
    ref.make_pairlist()
    fr = ref.forces()
    assert np.abs(m.forces() - fr).max() <= 1e-12 * max(np.abs(fr).max(), 1.0)
    m.calculate(30)
    ref.calculate(30)
    np.testing.assert_allclose(m.observe_raw(), ref.observe_raw(), rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("r", [0.7, 0.9, 0.9178, 0.918, 0.93, 1.0])
def test_close_pairs(r):
    # pairs at distance r along different directions, across a face of the box too
    L = np.array([14.0, 13.0, 12.0])
    d = np.array([[1, 0, 0], [0, 1, 0], [0, 0, 1], [1, 1, 1], [-1, 2, 0.5]], dtype=float)
    d /= np.linalg.norm(d, axis=1)[:, None]
    base = np.array([[13.8, 3, 3], [3, 12.9, 3], [3, 3, 0.1], [7, 7, 7], [10, 3, 8]])
    q = np.mod(np.concatenate([base, base + r * d]), L)
    _check(q, np.zeros_like(q), L, steps=0)


def test_row_sums_beyond_the_integer_range():
    # 40 partners crowded at 0.93 on one side of a particle: the sum of their forces passes 2^11
    rng = np.random.default_rng(5)
    u = np.array([1.0, 0.0, 0.0]) + 0.02 * rng.normal(size=(40, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    q = np.concatenate([[[5.0, 5.0, 5.0]], np.array([5.0, 5.0, 5.0]) + 0.93 * u, rng.uniform(8, 10, (5, 3))])
    L = np.array([12.0, 12.0, 12.0])
    m = _manager(L, len(q), list_capacity=64)
    m.set_state(q, np.zeros_like(q))
    ref = port.System(q, np.zeros_like(q), L, rc=2.5, margin=0.5)
    ref.make_pairlist()
    fr = ref.forces()[0]
    assert np.abs(fr).max() > 2.0 ** 11
    np.testing.assert_allclose(m.forces()[0], fr, rtol=1e-12, atol=1e-9)


@pytest.mark.parametrize("speed", [300.0, 900.0, 3200.0])
def test_fast_particle_leaves_the_guard(speed):
    # one particle that crosses 0.3, 0.9 or 3.2 sigma a step: guard, rebuild every step, modulus
    q, p, L = liquid_like(0.3, 5, amp=0.05, seed=9)
    p[7] = [speed, -0.6 * speed, 0.3 * speed]
    m = _manager(L, len(q))
    m.set_state(q, p)
    ref = port.System(q, p, L, rc=2.5, margin=0.5, rebuild_policy=port.REBUILD_HALFMARGIN)
    ref.make_pairlist()
    m.make_pairlist()
    for _ in range(2):
        m.calculate(1)
        ref.calculate(1)
    qm, pm = m.state()
    qr, pr = ref.state()[:2]
    np.testing.assert_allclose(pm, pr[:, :3], rtol=1e-9, atol=1e-9 * speed)


def test_lanes_and_graphs_do_not_change_the_trajectory():
    # the same steps through graphs and plain launches: bit for bit
    q, p, L = liquid_like(0.8, 12, seed=2)
    out = []
    for graphs in (True, False):
        m = _manager(L, len(q), use_graphs=graphs)
        m.set_state(q, p)
        m.calculate(60)
        out.append(np.concatenate(m.state()))
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("shape,flat", [((128, 1, 2), False), ((256, 2, 1), False), ((256, 1, 2), True)])
def test_batch_paths_match_the_single_box(shape, flat):
    # an ordinary box, one with a pair at 0.8 and one with a fast particle: each as MDManager runs it alone
    from mdacp_gb300.batch import Batch
    boxes = []
    for k in range(3):
        q, p, L = liquid_like(0.4, 5, amp=0.05, seed=20 + k)
        if k == 1:
            q[11] = np.mod(q[10] + [0.8, 0.0, 0.0], L)
        if k == 2:
            p[7] = [700.0, -200.0, 90.0]
        boxes.append((q, p, L))
    b = Batch(boxes, cutoff=2.5, margin=0.5, dt=0.001)
    b.set_shape(*shape)
    b.set_flat(flat)
    b.calculate(2)
    sums, states = b.observe_raw(), b.state()
    for k, (q, p, L) in enumerate(boxes):
        m = _manager(L, len(q))
        m.set_state(q, p)
        m.calculate(2)
        np.testing.assert_allclose(states[k][1], m.state()[1], rtol=1e-9, atol=1e-9 * np.abs(p).max())
        np.testing.assert_allclose(sums[k], m.observe_raw(), rtol=1e-9)


@pytest.mark.parametrize("objective,epsilon,sigma,seed", [("pe", 1.0, 1.0, 1), ("pressure", 1.0, 1.0, 2), ("pe", 1.3, 1.07, 3),
                                                          ("pressure", 0.7, 0.93, 4)])
def test_adjoint_in_fixed_point(objective, epsilon, sigma, seed):
    # 500 atoms, one pair at 0.85 sigma, an uneven last segment: margin 0.4 takes the
    # fixed-point sums, margin 1.2 (search length + margin above 3.9) the double ones
    from mdacp_gb300.adjoint import Adjoint
    q, p, L = liquid_like(0.7, 5, amp=0.08, temperature=0.7, seed=seed)
    q[11] = np.mod(q[10] + [0.85 * sigma, 0.0, 0.0], L)
    out = []
    for margin in (0.4, 1.2):
        a = Adjoint(L, len(q), steps=13, checkpoint_every=5, dt=0.001, cutoff=2.3, margin=margin, epsilon=epsilon, sigma=sigma,
                    objective=objective)
        J = a.forward(q, p)
        out.append((J,) + a.backward())
    (j0, dq0, dp0, de0, ds0), (j1, dq1, dp1, de1, ds1) = out
    assert abs(j0 - j1) <= 1e-13 * abs(j1)
    assert np.linalg.norm(dq0 - dq1) <= 1e-11 * np.linalg.norm(dq1)
    assert np.linalg.norm(dp0 - dp1) <= 1e-11 * np.linalg.norm(dp1)
    assert abs(de0 - de1) <= 1e-11 * abs(de1) and abs(ds0 - ds1) <= 1e-11 * abs(ds1)


def test_adjoint_list_of_many_particles():
    # 8,788 atoms: a lane's candidates no longer fit its mask words
    from mdacp_gb300.adjoint import Adjoint
    q, p, L = liquid_like(0.7, 13, amp=0.05, temperature=0.7, seed=5)
    a = Adjoint(L, len(q), steps=3, checkpoint_every=2, dt=0.001, cutoff=2.5, margin=0.4)
    m = _manager(L, len(q), margin=0.4)
    m.set_state(q, p)
    u = []
    for _ in range(3):
        m.calculate(1)
        u.append(m.observe_raw()[1] / len(q))
    assert abs(a.forward(q, p) - np.mean(u)) <= 1e-12 * abs(np.mean(u))

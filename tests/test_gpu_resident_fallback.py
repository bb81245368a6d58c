"""The resident step kernel where the fixed-point form falls back to the double row walk, over many steps of one launch.

Rows and positions are rewritten between the grid barriers of the launch, so
the fallback must read them as ordinary data.  Against plain step launches,
whose fallback is the same arithmetic: 1e-11 relative (rounding of the other
lanes' sums, 150 steps of a solid or 30 of a gas).
"""
import numpy as np
import pytest

from tests.helpers import liquid_like

pytestmark = pytest.mark.gpu


def _compare(q, p, L, calls, **kw):
    from mdacp_gb300.manager import MDManager
    out = []
    for graphs in (False, True):
        m = MDManager(L, capacity=len(q), use_graphs=graphs, gamma=1.0, **kw)
        m.set_state(q, p)
        for k in calls:
            m.calculate(k)
        out.append((np.concatenate(m.state()), m.stats()))
    (s0, st0), (s1, st1) = out
    for key in ("steps", "rebuilds", "prunes", "inner_pairs", "listed_pairs", "max_neighbours"):
        assert st0[key] == st1[key], key
    np.testing.assert_allclose(s1, s0, rtol=1e-11, atol=1e-11 * np.abs(s0).max())
    return st0


@pytest.mark.parametrize("thermostat", ["nve", "langevin", "nosehoover"])
@pytest.mark.parametrize("cells", [6, 8, 14])
def test_rows_too_long_for_the_integer_sums(cells, thermostat):
    # more than 243 entries: 7 n - 1700 is above any sum of force factors, so every row is walked in double
    q, p, L = liquid_like(1.35, cells, amp=0.02, temperature=4.0, seed=cells)
    st = _compare(q, p, L, [150], cutoff=3.55, margin=0.15, dt=0.0005, precision="fp64", thermostat=thermostat, temperature=4.0)
    assert st["inner_pairs"] > 250 * len(q) and st["rebuilds"] > 1 and st["prunes"] > st["rebuilds"]


@pytest.mark.parametrize("thermostat", ["nve", "nosehoover"])
def test_particle_outside_the_guard_every_step(thermostat):
    # 1.2 sigma a step along a channel of a sparse lattice: its first half-drift already leaves the guard (0.484)
    q, p, L = liquid_like(0.05, 5, amp=0.05, seed=9)
    a = L[0] / 5
    q = np.concatenate([q, [[0.1, 0.25 * a, 0.25 * a]]])
    p = np.concatenate([p, [[1200.0, 0.0, 0.0]]])
    st = _compare(q, p, L, [30], cutoff=2.5, margin=0.5, dt=0.001, precision="fp64", thermostat=thermostat,
                  temperature=float(np.mean(p ** 2)))
    assert st["rebuilds"] >= 30

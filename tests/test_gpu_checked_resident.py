"""The bounds-checked build (libmdg_check.so) through the resident kernel, the step graphs and plain launches.

As test_gpu_checked.py: the checks must never fire on valid runs, and the three
ways give the same mixed trajectories bit for bit (FP64 to the rounding of the
lanes' sums, 1e-11).
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = r'''
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from mdacp_gb300 import native
from mdacp_gb300.manager import MDManager
from tests.helpers import liquid_like
lib = native.load()
assert lib._name.endswith("libmdg_check.so"), lib._name

def run(q, p, L, graphs, steps, **kw):
    m = MDManager(L, capacity=len(q), use_graphs=graphs, gamma=1.0, **kw)
    m.set_state(q, p)
    m.calculate(steps)
    s = np.concatenate(m.state())
    return s, m.stats()["kernel_launches"]

ordinary = dict(cutoff=2.5, margin=0.3, dt=0.004)
dense = dict(cutoff=3.55, margin=0.15, dt=0.0005)  # rows too long for the integer sums
cases = [(0.8, 6, 1.4, "mixed", "nve", 60, ordinary), (0.8, 14, 1.4, "mixed_plain", "langevin", 40, ordinary),
         (0.3, 22, 1.4, "mixed", "langevin", 40, ordinary), (0.8, 6, 1.4, "fp64", "nve", 60, ordinary),
         (0.5, 16, 1.4, "fp64", "nosehoover", 40, ordinary), (1.35, 6, 4.0, "fp64", "nve", 60, dense),
         (0.8, 8, 1.4, "mixed", "nve", 40, dict(ordinary, list_capacity=32))]
for density, cells, T, precision, thermostat, steps, kw in cases:
    q, p, L = liquid_like(density, cells, amp=0.02 if T > 2 else 0.08, temperature=T, seed=cells)
    out = [run(q, p, L, g, steps, precision=precision, thermostat=thermostat, temperature=T, **kw) for g in (0, 1, 2)]
    assert out[1][1] < out[2][1] < out[0][1]  # the resident kernel was taken
    for s, _ in out[1:]:
        if precision == "fp64":
            np.testing.assert_allclose(s, out[0][0], rtol=1e-11, atol=1e-11 * np.abs(s).max())
        else:
            assert np.array_equal(s, out[0][0])
print("checked cases ok")
'''


def test_checked_build_in_the_resident_kernel():
    from mdacp_gb300 import build
    build.build(check=True)
    r = subprocess.run([sys.executable, "-c", CASES, ROOT], env=dict(os.environ, MDG_LIBRARY="check"),
                       capture_output=True, text=True, timeout=1200, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert "checked cases ok" in r.stdout

"""Gradients over checkpoint segments longer than the window of steps whose forces and derivatives are held.

55,296 particles: 121 steps fit the fixed-point form's window, 303 the double form's.  One segment
of 130 steps in fixed point (two windows) against the double form (one), and segments of
exactly one window and of one step more; J to 1e-13, gradients to 1e-11, as test_gpu_fixed.py.
"""
import numpy as np
import pytest

from tests.helpers import liquid_like

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("objective,every", [("pe", 121), ("pe", 122), ("pressure", 130)])
def test_segments_beyond_the_window(objective, every):
    from mdacp_gb300.adjoint import Adjoint
    q, p, L = liquid_like(0.7, 24, amp=0.05, temperature=0.7, seed=3)
    assert (1 << 30) // (160 * len(q)) == 121 and (1 << 30) // (64 * len(q)) == 303
    out = []
    for margin in (0.4, 1.2):
        a = Adjoint(L, len(q), steps=130, checkpoint_every=every, dt=0.0002, cutoff=2.3, margin=margin, objective=objective)
        out.append((a.forward(q, p),) + a.backward())
        if margin == 0.4:  # and the same again from the captured passes
            again = (a.forward(q, p),) + a.backward()
            assert again[0] == out[0][0] and all(np.array_equal(x, y) for x, y in zip(again[1:], out[0][1:]))
        a.close()
    (j0, dq0, dp0, de0, ds0), (j1, dq1, dp1, de1, ds1) = out
    assert abs(j0 - j1) <= 1e-13 * abs(j1)
    assert np.linalg.norm(dq0 - dq1) <= 1e-11 * np.linalg.norm(dq1)
    assert np.linalg.norm(dp0 - dp1) <= 1e-11 * np.linalg.norm(dp1)
    assert abs(de0 - de1) <= 1e-11 * abs(de1) and abs(ds0 - ds1) <= 1e-11 * abs(ds1)


def test_memory_of_a_long_segment():
    # 20,000 steps of 4,000 particles between checkpoints: 96 bytes a particle and step, and a window of 1 GB
    import torch
    from mdacp_gb300.adjoint import Adjoint
    q, p, L = liquid_like(0.7, 10, amp=0.05, seed=4)
    torch.cuda.init()
    free0 = torch.cuda.mem_get_info()[0]
    a = Adjoint(L, len(q), steps=20000, checkpoint_every=20000, dt=0.0002, margin=0.5)
    used = free0 - torch.cuda.mem_get_info()[0]
    assert used < 96 * 4000 * 20000 + 1.3 * 2 ** 30
    a.close()

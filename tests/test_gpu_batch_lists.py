"""Readers of a batch's pair lists at states that have none yet, and errors in both layouts of the step.

A pool that had to grow holds rows only of the boxes that were still behind;
a new, replaced or restored state has none.  mdg_batch_observe walks rows, so it
must build them first.  FP64 against the oracle run on each box alone
(1e-10, as the batch parity tests), the mixed forms against a pool that is large enough.
"""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_batch import DT, MARGIN, RC, _oracle_obs

pytestmark = pytest.mark.gpu

LAYOUTS = [((256, 1, 2), False), ((128, 2, 2), False), ((256, 1, 4), True)]


def _replicas(nbox, seed, rho):
    from mdacp_gb300.batch import make_replicas
    return make_replicas(nbox, seed=seed, n_range=(500, 1500), rho_range=rho)


def _batch(boxes, shape, flat, **kw):
    from mdacp_gb300.batch import Batch
    b = Batch(boxes, cutoff=RC, margin=MARGIN, dt=DT, **kw)
    b.set_shape(*shape)
    b.set_flat(flat)
    return b


def _set(b, boxes):
    q4, p4 = np.zeros((b.offsets[-1], 4)), np.zeros((b.offsets[-1], 4))
    for k, (q, p, _) in enumerate(boxes):
        q4[b.offsets[k]:b.offsets[k + 1], :3] = q
        p4[b.offsets[k]:b.offsets[k + 1], :3] = p
    dp = ctypes.POINTER(ctypes.c_double)
    b._ck(b.lib.mdg_batch_set_state(b._h, q4.ctypes.data_as(dp), p4.ctypes.data_as(dp)))


def _uneven():
    # rows of 72 entries hold the lists of the dilute boxes (at most 55), not those of the dense one (about 90)
    return _replicas(5, 31, (0.3, 0.4)) + _replicas(1, 32, (0.85, 0.9))


@pytest.mark.parametrize("shape,flat", LAYOUTS)
def test_observe_after_some_boxes_overflowed(shape, flat):
    boxes = _uneven()
    b = _batch(boxes, shape, flat, list_capacity=72)
    done = 0
    for steps in (41, 20):
        b.calculate(steps)
        done += steps
        np.testing.assert_allclose(b.observe_raw(), _oracle_obs(boxes, done), rtol=1e-10, atol=1e-10)
    assert b.stats()["list_capacity"] > 72


@pytest.mark.parametrize("precision", ["mixed", "mixed_plain"])
@pytest.mark.parametrize("shape,flat", LAYOUTS)
def test_overflow_of_some_boxes_in_the_mixed_forms(shape, flat, precision):
    # the same states bit for bit as with rows that are long enough; the sums of up to 1,500 row sums
    # of at most 10^3, added in another order
    boxes, runs = _uneven(), []
    for cap in (72, 160):
        b = _batch(boxes, shape, flat, precision=precision, list_capacity=cap)
        b.calculate(41)
        state = np.concatenate([np.concatenate(x) for x in b.state()])  # an observation that builds lists wraps positions
        runs.append((b.observe_raw(), state))
    assert np.array_equal(runs[0][1], runs[1][1])
    np.testing.assert_allclose(runs[0][0], runs[1][0], rtol=1e-12, atol=1e-9)


@pytest.mark.parametrize("shape,flat", LAYOUTS)
def test_observe_ahead_of_the_first_step(shape, flat):
    # after creation, with rows too short for any box, after a replaced state and after the autotuner; then the steps as ever
    boxes, other = _replicas(3, 33, (0.3, 0.8)), _replicas(3, 33, (0.3, 0.8))
    other = [(q[::-1].copy(), p[::-1].copy(), L) for q, p, L in other]
    for cap in (0, 8):
        b = _batch(boxes, shape, flat, list_capacity=cap)
        np.testing.assert_allclose(b.observe_raw(), _oracle_obs(boxes, 0), rtol=1e-10)
        b.calculate(30)
        np.testing.assert_allclose(b.observe_raw(), _oracle_obs(boxes, 30), rtol=1e-10, atol=1e-10)
        _set(b, other)
        np.testing.assert_allclose(b.observe_raw(), _oracle_obs(other, 0), rtol=1e-10)
    b.tune(trial_steps=3)
    np.testing.assert_allclose(b.observe_raw(), _oracle_obs(other, 0), rtol=1e-10)
    b.calculate(30)
    np.testing.assert_allclose(b.observe_raw(), _oracle_obs(other, 30), rtol=1e-10, atol=1e-10)


def test_observing_first_changes_no_step():
    # the list that an observation built is built again by the first step, from the same positions
    boxes = _replicas(4, 34, (0.3, 0.8))
    states = []
    for first in (False, True):
        b = _batch(boxes, (256, 1, 4), True, precision="mixed")
        if first:
            b.observe_raw()
        b.calculate(60)
        states.append(np.concatenate([np.concatenate(x) for x in b.state()]))
    assert np.array_equal(*states)


@pytest.mark.parametrize("shape,flat", LAYOUTS)
def test_bad_coordinate_names_its_box(shape, flat):
    # the error, on the first step and later; a new state runs
    from mdacp_gb300 import native
    boxes = _replicas(4, 35, (0.3, 0.8))
    bad = list(boxes)
    p = boxes[2][1].copy()
    p[17] = np.nan
    bad[2] = (boxes[2][0], p, boxes[2][2])
    q = boxes[1][0].copy()
    q[3, 0] += 5.0 * boxes[1][2][0]
    far = list(boxes)
    far[1] = (q, boxes[1][1], boxes[1][2])
    b = _batch(bad, shape, flat)
    with pytest.raises(native.MDGError, match="box 2: bad coordinate"):
        b.calculate(20)
    _set(b, far)
    with pytest.raises(native.MDGError, match="box 1: bad coordinate"):
        b.calculate(20)
    with pytest.raises(native.MDGError, match="box 1: bad coordinate"):
        b.observe_raw()
    _set(b, boxes)
    b.calculate(20)
    np.testing.assert_allclose(b.observe_raw(), _oracle_obs(boxes, 20), rtol=1e-10, atol=1e-10)


def test_no_state_is_refused():
    from mdacp_gb300 import batch, native
    lib = batch._lib()
    prm = batch.BatchParams()
    lib.mdg_batch_params_default(ctypes.byref(prm))
    n = (ctypes.c_int32 * 1)(500)
    L = (ctypes.c_double * 3)(9.0, 9.0, 9.0)
    h = ctypes.c_void_p()
    native.check(lib.mdg_batch_create(ctypes.byref(prm), 1, n, L, ctypes.byref(h)))
    out = (ctypes.c_double * 3)()
    t = ctypes.c_int32()
    assert lib.mdg_batch_observe(h, out) == 5
    assert lib.mdg_batch_calculate(h, 1) == 5 and lib.mdg_batch_calculate(h, 0) == 0
    assert lib.mdg_batch_get_state(h, None, None) == 5
    assert lib.mdg_batch_tune(h, 3, ctypes.byref(t), ctypes.byref(t), ctypes.byref(t)) == 5
    lib.mdg_batch_destroy(h)

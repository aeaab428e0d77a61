"""Scalars that a call reads and overwrites: what the device sees is the value before the call, whatever way it gets there."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import core, runtime

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where,change", [("cpu", "decay"), ("cpu", "sign"), ("gpu", "sign")])
@pytest.mark.parametrize("host_argument", [True, False])
def test_a_learning_rate_that_changes(rt, where, change, host_argument):
    """(p, p - lr * g), (lr, lr / 2 or -lr), eager, captured and replayed; powers of two, so every product is exact and only
    the additions to p round, in the same way here and there."""
    device = core.Device(where, 0)
    lr = cgt.shared(np.array(1.0, "f4"), device=device)
    half = cgt.shared(np.array(0.5, "f4"), device=device)
    p = cgt.shared(np.zeros((33, 5), "f4"), fixed_shape_mask="all")
    g = cgt.matrix("g", fixed_shape=(33, 5))
    f = cgt.function([g], [], updates=[(p, p - lr * g), (lr, lr * half if change == "decay" else -lr)])
    (want, rate) = (np.zeros((33, 5), "f4"), np.float32(1.0))
    for step in range(12):
        v = np.random.RandomState(step).randn(33, 5).astype("f4")
        f(v if host_argument else runtime.device_array(v))
        want = want - rate * v
        rate = rate * np.float32(0.5 if change == "decay" else -1.0)
        assert np.array_equal(p.op.get_value(), want), step
        assert lr.op.get_value() == rate, step


def test_a_large_host_variable(rt):
    """A host array above the size at which the copy engine takes over, read on the device, with other values every call."""
    n = 100000
    table = cgt.shared(np.zeros((n,), "f4"), device=core.Device("cpu", 0), fixed_shape_mask="all")
    f = cgt.function([], [table * 2.0])
    for step in range(6):
        v = np.random.RandomState(step).randn(n).astype("f4")
        table.op.set_value(v)
        assert np.array_equal(f()[0], v * 2), step


@pytest.mark.parametrize("rows,move", [(1, 1), (3, 2)])
def test_a_cursor_that_moves(rt, rows, move):
    """x[k:k+rows] with k a host variable that the call moves on: the slice is taken where k was before the call."""
    k = cgt.shared(np.array(0, "i8"), device=core.Device("cpu", 0))
    x = cgt.matrix("x", fixed_shape=(40, 5))
    f = cgt.function([x], [x[k:k + rows] * 2.0], updates=[(k, k + move)])
    a = np.arange(200, dtype="f4").reshape(40, 5)
    v = runtime.device_array(a)
    for step in range(12):
        assert np.array_equal(f(v)[0], 2 * a[step * move:step * move + rows]), step

"""Arguments into and results out of a compiled function, around the sizes where another way of copying takes over."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import runtime

pytestmark = pytest.mark.gpu

KB = 1 << 8  # floats


@pytest.mark.parametrize("n", [1, 5, 16 * KB, 16 * KB + 3, 256 * KB, 256 * KB + 1, 1024 * KB - 1, 1024 * KB, 2600 * KB + 7])
def test_arguments_and_results_of_every_size(rt, n):
    """Doubling and negation are exact: results have to match to the bit on the first (eager), captured and replayed
    runs, whether the argument is a new host array, the same one with other values, pinned, or on the device."""
    x = cgt.vector("x")
    f = cgt.function([x], [x * 2.0, -x, x.reshape([cgt.size(x, 0), 1])])
    rs = np.random.RandomState(n)
    pinned = runtime.pinned_empty((n,), "f4")
    kept = rs.randn(n).astype("f4")
    for run in range(9):
        a = rs.randn(n).astype("f4")
        if run % 4 == 1:
            kept[:] = a
            arg = kept
        elif run % 4 == 2:
            pinned[:] = a
            arg = pinned
        elif run % 4 == 3:
            arg = runtime.device_array(a)
        else:
            arg = a
        twice, neg, view = f(arg)
        assert np.array_equal(twice, a * 2) and np.array_equal(neg, -a) and np.array_equal(view, a[:, None]), run


def test_more_arguments_and_results_than_one_copy_kernel_takes(rt):
    xs = [cgt.vector("x%d" % i) for i in range(40)]
    f = cgt.function(xs, [x + 1.0 for x in xs])
    rs = np.random.RandomState(0)
    for _ in range(4):
        vals = [rs.randn(3 + i).astype("f4") for i in range(40)]
        for (v, got) in zip(vals, f(*vals)):
            assert np.array_equal(got, v + np.float32(1))

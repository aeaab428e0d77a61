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


@pytest.mark.parametrize("n", [6, 300 * KB])
def test_an_argument_that_is_handed_back(rt, n):
    """The result is the array of this call: also when another array of the same shape was there when the step's graph was
    captured, and when the result is a view of the argument."""
    x = cgt.vector("x", fixed_shape=(n,))
    f = cgt.function([x], [x, x * 2.0, x.reshape([2, n // 2])])
    rs = np.random.RandomState(0)
    vals = [rs.randn(n).astype("f4") for _ in range(3)]
    on_device = [runtime.device_array(v) for v in vals]
    for i in [0, 0, 0, 0, 0, 1, 1, 2, 0, 1, 2, 2]:
        (same, twice, view) = f(on_device[i])
        assert np.array_equal(twice, vals[i] * 2) and np.array_equal(same, vals[i]) and np.array_equal(view, vals[i].reshape(2, -1)), i
    for i in [0, 1, 2, 0]:
        assert np.array_equal(f(vals[i])[0], vals[i])


@pytest.mark.parametrize("sizes", [(2, 2), (2, 3, 1), (40,), (70, 2)])
def test_large_host_arrays_in_one_call(rt, sizes):
    """Arrays above a megabyte share the pinned staging memory, above 32 MB in several stretches: the second one finds the
    first one's copies still under way. Doubling is exact."""
    MB = 1 << 18  # floats
    xs = [cgt.vector("x%d" % i) for i in range(len(sizes))]
    f = cgt.function(xs, [cgt.sum(x * 2.0) if i else x * 2.0 for (i, x) in enumerate(xs)])
    rs = np.random.RandomState(1)
    for run in range(4):
        vals = [rs.randint(-8, 8, size=n * MB + 5).astype("f4") for n in sizes]
        got = f(*vals)
        assert np.array_equal(got[0], vals[0] * 2), run
        for (v, g) in zip(vals[1:], got[1:]):   # whole numbers, every partial sum below 2^24: exact in any order
            assert g == 2 * v.astype("f8").sum(), run

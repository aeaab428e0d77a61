"""What a step reads of a variable that it also overwrites: the compiled instruction list, executed on numpy arrays
(tests/host_run.py), against the oracle, which evaluates everything before it updates anything. Both evaluate an operation
by the same function, so results are the same bits unless a comment says otherwise."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import core, nn
from oracle import cpu_backend
from tests.host_run import HostRun


def _var(rs, *shape):
    return cgt.shared((rs.randn(*shape) * 0.3).astype("f4"), fixed_shape_mask="all")


def _same_as_oracle(inputs, outputs, updates, steps=4, exact=True):
    run, oracle = HostRun(inputs, outputs, updates), cpu_backend.function(inputs, outputs, updates=updates)
    for step in range(steps):
        rs = np.random.RandomState(step)
        args = [(rs.randn(*x.get_fixed_shape()) * 0.3).astype("f4") for x in inputs]
        pairs = list(zip(run(*args), oracle(*args))) + [(run.value(v), oracle.get_value(v)) for (v, _new) in updates]
        for (i, (got, want)) in enumerate(pairs):
            if exact:
                assert np.array_equal(got, want), (step, i)
            else:   # the sums are added up in another order: at most n * eps of the sum of their terms, all positive here
                np.testing.assert_allclose(got, want, rtol=2000 * np.finfo("f4").eps)
    return run


def _copies(run):
    return sum(isinstance(op, core.ElwiseUnary) and op.opname == "cast_to_f4" for op in run.ops())


OPTIMIZERS = {"sgd": dict(learning_rate=0.1), "momentum": dict(learning_rate=0.1), "nesterov_momentum": dict(learning_rate=0.1), "adagrad": {},
              "rmsprop": {}, "adadelta": {}, "adam": {}}


@pytest.mark.parametrize("merge", [True, False])
@pytest.mark.parametrize("name", sorted(OPTIMIZERS))
def test_optimizers(name, merge):
    rs = np.random.RandomState(0)
    x = cgt.matrix("x", fixed_shape=(32, 24))
    (W, b, V) = (_var(rs, 24, 40), _var(rs, 1, 40), _var(rs, 40, 10))
    loss = cgt.square(cgt.tanh(cgt.broadcast("+", x.dot(W), b, "xx,1x")).dot(V)).sum() / 32.0
    with cgt.scoped_update_config(merge_parameter_updates=merge):
        run = _same_as_oracle([x], [loss], getattr(nn, name)(loss, [W, b, V], **OPTIMIZERS[name]))
    assert not _copies(run)


def test_a_shared_operation_on_overwritten_variables_runs_once():
    rs = np.random.RandomState(0)
    (a, b, p) = (_var(rs, 33, 5), _var(rs, 33, 5), _var(rs, 33, 5))
    s = 0.1 * (a + b)
    _same_as_oracle([], [], [(a, a - s), (b, b - s)])
    s = 0.1 * (a + cgt.tanh(p * 0.5))   # only tanh(p / 2) may be repeated, and p is not overwritten
    _same_as_oracle([], [], [(a, a - s), (b, b - s)])


def test_a_gradient_that_two_parameters_share_is_one_launch():
    rs = np.random.RandomState(0)
    g = cgt.matrix("g", fixed_shape=(33, 5))
    (a, b) = (_var(rs, 33, 5), _var(rs, 33, 5))
    step = 0.1 * cgt.tanh(g)
    run = _same_as_oracle([g], [], [(a, a - step), (b, b - step)])
    assert [op.k for op in run.ops() if isinstance(op, core.MultiFusedElwise)] == [2]


def test_factorisation():
    """X ~ U.V by gradient steps: each factor's gradient is a product with the other's old value."""
    rs = np.random.RandomState(0)
    X = cgt.matrix("X", fixed_shape=(64, 48))
    (U, V) = (_var(rs, 64, 32), _var(rs, 32, 48))
    loss = cgt.square(X - U.dot(V)).sum()
    run = _same_as_oracle([X], [loss], nn.sgd(loss, [U, V], 0.01))
    assert not _copies(run)
    # X - U.V and one of the updates carry their chains; the other's product has to run before the first update
    assert sum(isinstance(op, core.Mul22Chain) for op in run.ops()) == 2


def test_a_product_with_the_old_value_runs_before_the_update():
    rs = np.random.RandomState(0)
    A = cgt.matrix("A", fixed_shape=(64, 64))
    (v, p) = (_var(rs, 64, 64), _var(rs, 64, 64))
    new = 0.9 * v - 0.1 * cgt.tanh(v)
    _same_as_oracle([A], [], [(v, new), (p, p - 0.5 * A.dot(v) + new)])
    _same_as_oracle([A], [v.dot(A) - new], [(v, new)])


@pytest.mark.parametrize("view", ["itself", "slice", "reshape"])
def test_a_chain_does_not_overwrite_what_its_product_multiplies(view):
    rs = np.random.RandomState(0)
    W = _var(rs, 64, 64)
    A = cgt.matrix("A", fixed_shape=(64, 16 if view == "slice" else 64))
    part = {"itself": W, "slice": W[16:32], "reshape": W.reshape([32, 128]).reshape([64, 64])}[view]
    _same_as_oracle([A], [], [(W, cgt.tanh(A.dot(part)))])
    _same_as_oracle([A], [], [(W, W - 0.1 * A.dot(part))])


def test_merged_updates_do_not_read_each_others_variables():
    """Every kind of order between updates of one form: p reads v before it changes, d as well, q reads w's new value."""
    rs = np.random.RandomState(0)
    g = cgt.matrix("g", fixed_shape=(33, 5))
    (v, p, d) = (_var(rs, 33, 5), _var(rs, 33, 5), _var(rs, 33, 5))
    _same_as_oracle([g], [], [(p, p - 0.1 * v), (v, v - 0.1 * g)])
    _same_as_oracle([g], [], [(v, v - 0.1 * g), (p, p - 0.1 * v)])
    s = 0.1 * v
    _same_as_oracle([g], [], [(p, p - s), (d, d - s), (v, v - 0.2 * g)])
    new = v - 0.1 * g
    _same_as_oracle([g], [], [(v, new), (p, p - 0.1 * new), (d, d - 0.1 * g)])
    h = cgt.matrix("h", fixed_shape=(5, 33))
    (t, u) = (_var(rs, 5, 33), _var(rs, 33, 5))   # through views of each other
    _same_as_oracle([h], [], [(u, u - 0.1 * t.reshape([33, 5])), (t, t - 0.1 * h)])
    run = _same_as_oracle([g], [], [(x, x - 0.1 * g) for x in (v, p, d)])
    assert [op.k for op in run.ops() if isinstance(op, core.MultiFusedElwise)] == [3]


def test_norms_of_an_old_and_a_new_value():
    rs = np.random.RandomState(0)
    B = cgt.matrix("B", fixed_shape=(33, 5))
    (U, V, W) = (_var(rs, 33, 5), _var(rs, 40, 7), _var(rs, 1, 9))
    new = U - 0.1 * cgt.tanh(U - B)
    run = _same_as_oracle([B], [cgt.square(x).sum() * 1.0 for x in (U, V, new, W)], [(U, new), (V, V * 0.9)], exact=False)
    assert [len(op.ndims) for op in run.ops() if isinstance(op, core.SumSquares)] == [3]   # all but the new value's


@pytest.mark.parametrize("fuse", [True, False])
def test_what_needs_old_and_new_value(fuse):
    """v and its new value meet in one operation, or in one chain after fusion; updates that need each other's variable."""
    rs = np.random.RandomState(0)
    (v, p, n) = (_var(rs, 33, 5), _var(rs, 33, 5), _var(rs, 12, 5))
    new = 0.9 * v - 0.1 * cgt.tanh(v)
    with cgt.scoped_update_config(fuse_elementwise=fuse):
        _same_as_oracle([], [cgt.square(v * new)], [(v, new), (p, p - v * new)])
        _same_as_oracle([], [], [(v, new), (p, p - 0.5 * v + new)])
        _same_as_oracle([], [cgt.concatenate([v[0:9], new], axis=0) * 2.0], [(v, new)])
        _same_as_oracle([], [], [(v, v - p), (p, p - v)])
        _same_as_oracle([], [], [(v, v - p), (p, p + cgt.concatenate([n, v[3:24]], axis=0)), (n, n * v[0:12])])


def test_updates_that_read_their_variable_elsewhere():
    rs = np.random.RandomState(0)
    x = cgt.matrix("x", fixed_shape=(1, 40))
    A = cgt.matrix("A", fixed_shape=(40, 40))
    (W, last) = (_var(rs, 8, 40), _var(rs, 40, 40))
    _same_as_oracle([x], [], [(W, cgt.concatenate([x, W[0:7]], axis=0))])          # the last eight rows
    _same_as_oracle([A], [], [(last, last.dot(A)), (W, W.dot(A))])
    _same_as_oracle([A], [], [(last, last.T)])
    _same_as_oracle([x], [], [(W, W - cgt.repeat(W[0:1], 8, axis=0))])
    _same_as_oracle([], [], [(W, nn.softmax(W))], exact=False)


def test_ordinary_steps_take_no_copies():
    """The copies are for steps that have no other order: none of the configurations and optimizers has them."""
    from cgt_b200 import compilation, configs
    small = {"mlp": dict(batch=8), "cifar": dict(batch=2), "wide": dict(batch=2), "lstm": dict(seq_len=4, batch=4), "vae": dict(batch=5)}
    for (name, kw) in small.items():
        cfg = configs.BUILDERS[name](**kw)
        eg = compilation.execution_graph(cfg.inputs, [cfg.loss] + list(cfg.extra_outputs), cfg.updates, [])[0]
        assert not any(isinstance(getattr(i, "op", None), core.ElwiseUnary) and i.op.opname == "cast_to_f4" for i in eg.instrs), name


def test_a_slice_that_is_handed_out_keeps_its_old_value():
    rs = np.random.RandomState(0)
    W = _var(rs, 8, 40)
    run = _same_as_oracle([], [W[2:5], W[0:3].reshape([12, 10])], [(W, W * 0.9)])
    assert not any(isinstance(op, core.LeadingSlice) for op in run.ops())
    run = _same_as_oracle([], [cgt.tanh(W[2:5])], [(W, W * 0.9)])
    assert any(isinstance(op, core.LeadingSlice) for op in run.ops())


@pytest.mark.parametrize("delay", [True, False])
def test_host_arithmetic_behind_the_device_work(delay):
    """Steps scaled by several norms that the host works out, a host variable that the host overwrites, and the order of
    what reads and writes it: the same bits wherever the host's instructions stand, and one stretch of them when delayed."""
    from cgt_b200 import compilation
    rs = np.random.RandomState(0)
    x = cgt.matrix("x", fixed_shape=(33, 5))
    (a, b, p) = (_var(rs, 33, 5), _var(rs, 33, 5), _var(rs, 33, 5))
    lr = cgt.shared(np.array(0.25, "f4"), device=core.Device("cpu", 0))
    with cgt.scoped_update_config(delay_host_arithmetic=delay, fuse_square_sums=False):
        norms = [cgt.sqrt(cgt.square(v * x).sum()) for v in (a, b, p)]
        scale = lr / (norms[0] + norms[1] * norms[2])
        run = _same_as_oracle([x], [norms[1] * 2.0, lr * 1.0 + norms[0]],
                              [(a, a - scale * x), (b, b - norms[0] * lr * x), (p, p - x), (lr, lr * 0.5 + 0.0 * norms[2])])
    instrs = [i for i in run.eg.instrs if isinstance(i, compilation.ReturnByRef) and not i.once and not isinstance(i.op, core.Constant)]
    downloads = [i for i in instrs if isinstance(i.op, core.Transport) and i.write_loc.devtype == "cpu"]
    roots = [k for (k, i) in enumerate(instrs) if getattr(i.op, "opname", "") == "sqrt"]
    assert len(downloads) == 3 and len(roots) == 3
    (first, last) = (min(roots), max(instrs.index(d) for d in downloads))
    assert (first > last) == delay


def test_one_value_for_several_variables_and_views_as_values():
    rs = np.random.RandomState(0)
    (a, b, c) = (_var(rs, 6, 6), _var(rs, 6, 6), _var(rs, 6, 6))
    x = cgt.matrix("x", fixed_shape=(6, 6))
    y = cgt.matrix("y", fixed_shape=(4, 9))
    new = a + x * b
    _same_as_oracle([x], [c - new], [(a, new), (b, new), (c, new)])
    _same_as_oracle([y], [a * 2.0], [(a, cgt.tanh(y).reshape([6, 6]))])
    _same_as_oracle([], [a * 2.0, b * 3.0], [(a, cgt.concatenate([b, b], axis=0)[3:9]), (b, b - a)])

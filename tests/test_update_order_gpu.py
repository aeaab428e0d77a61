"""Steps that read what they overwrite, on the device: eager, captured and replayed calls against the oracle."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import nn
from oracle import cpu_backend

pytestmark = pytest.mark.gpu


def _var(rs, *shape):
    return cgt.shared((rs.randn(*shape) * 0.3).astype("f4"), fixed_shape_mask="all")


def _factorisation(rs):
    X = cgt.matrix("X", fixed_shape=(64, 48))
    (U, V) = (_var(rs, 64, 32), _var(rs, 32, 48))
    loss = cgt.square(X - U.dot(V)).sum()
    return [X], [loss], nn.sgd(loss, [U, V], 0.002)


def _old_and_new(rs):
    A = cgt.matrix("A", fixed_shape=(64, 64))
    (v, p) = (_var(rs, 64, 64), _var(rs, 64, 64))
    new = 0.9 * v - 0.1 * cgt.tanh(v)
    return [A], [cgt.square(v).sum() * 1.0, cgt.square(new).sum() * 1.0, v * new], [(v, new), (p, p - 0.05 * A.dot(v) + 0.1 * new - 0.5 * v)]


def _own_rows(rs):
    A = cgt.matrix("A", fixed_shape=(64, 16))
    x = cgt.matrix("x", fixed_shape=(1, 40))
    (W, last) = (_var(rs, 64, 64), _var(rs, 8, 40))
    return [A, x], [], [(W, W - 0.1 * A.dot(W[16:32])), (last, cgt.concatenate([x, last[0:7]], axis=0))]


def _views_and_shared_values(rs):
    x = cgt.matrix("x", fixed_shape=(64, 40))
    (a, b, c, d) = (_var(rs, 64, 40), _var(rs, 64, 40), _var(rs, 40, 64), _var(rs, 16, 40))
    new = 0.5 * a + x * b
    return [x], [cgt.tanh(c), d * 2.0], [(a, new), (b, new), (c, cgt.tanh(x + a).reshape([40, 64])), (d, cgt.tanh(x)[8:24])]


def _each_other(rs):
    g = cgt.matrix("g", fixed_shape=(333, 50))
    (v, p, d) = (_var(rs, 333, 50), _var(rs, 333, 50), _var(rs, 333, 50))
    s = 0.1 * v
    return [g], [], [(p, p - s), (d, d - s), (v, v - 0.2 * g)]


def _optimizer(name):
    def build(rs):
        x = cgt.matrix("x", fixed_shape=(32, 24))
        (W, b, V) = (_var(rs, 24, 40), _var(rs, 1, 40), _var(rs, 40, 10))
        loss = cgt.square(cgt.tanh(cgt.broadcast("+", x.dot(W), b, "xx,1x")).dot(V)).sum() / 32.0
        return [x], [loss], getattr(nn, name)(loss, [W, b, V], learning_rate=0.05)
    return build


@pytest.mark.parametrize("build", [_factorisation, _old_and_new, _own_rows, _views_and_shared_values, _each_other, _optimizer("momentum"), _optimizer("nesterov_momentum"),
                                   _optimizer("rmsprop"), _optimizer("adadelta")])
def test_against_the_oracle(rt, build):
    (inputs, outputs, updates) = build(np.random.RandomState(0))
    oracle, f = cpu_backend.function(inputs, outputs, updates=updates), cgt.function(inputs, outputs, updates=updates)
    steps, K = 6, 64
    for step in range(steps):
        rs = np.random.RandomState(step)
        args = [(rs.randn(*x.get_fixed_shape()) * 0.3).astype("f4") for x in inputs]
        pairs = list(zip(f(*args), oracle(*args))) + [(v.op.get_value(), oracle.get_value(v)) for (v, _new) in updates]
        for (i, (got, want)) in enumerate(pairs):
            # sums of at most K terms in another order, carried on through the steps; 8 for what cancels
            assert np.linalg.norm(got - want) <= 8 * K * steps * np.finfo("f4").eps * max(np.linalg.norm(want), 1e-3), (step, i)

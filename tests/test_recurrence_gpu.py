"""The steps of an unrolled recurrent network as one launch (compilation.fuse_recurrences) against a launch per product
and chain: edges of the rows per cluster, of the units per block and of the K groups; networks that must not be grouped."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import configs, core, nn

pytestmark = pytest.mark.gpu


def _recurrences(f):
    return [i.op for i in f.eg.instrs if isinstance(getattr(i, "op", None), core.Recurrence)]


def _both_ways(build, calls):
    out = {}
    for on in (False, True):
        with cgt.scoped_update_config(fuse_recurrences=on):
            (f, variables, batch) = build()
        assert on or not _recurrences(f)
        # eager, captured and replayed runs with other inputs each
        got = [np.asarray(v).copy() for i in range(calls) for v in f(*batch(np.random.RandomState(i)))]
        out[on] = (got + [v.op.get_value().copy() for v in variables], _recurrences(f))
    return out


def _close(out, K, T):
    """Rounding errors of random sign grow as the root of their number, K per sum and T sums in a row; 8 for their spread
    and for the few sums that cancel."""
    bound = 8 * np.sqrt(K * T) * np.finfo("f4").eps
    for (a, b) in zip(out[False][0], out[True][0]):
        assert np.linalg.norm(a.astype("f8") - b) <= bound * max(np.linalg.norm(a), 1e-3)


@pytest.mark.parametrize("T,B,V,H,L", [(7, 64, 65, 128, 2), (8, 1, 30, 32, 1), (7, 64, 40, 32, 1), (7, 33, 47, 90, 1), (9, 17, 31, 50, 2),
                                       (8, 129, 35, 64, 1), (7, 7, 33, 101, 1), (7, 31, 30, 129, 1), (50, 8, 30, 100, 1)])
def test_lstm_training_step(rt, T, B, V, H, L):
    def build():
        cfg = configs.build_lstm(vocab=V, hidden=H, n_layers=L, seq_len=T, batch=B)
        return cfg.compile(), [v for (v, _new) in cfg.updates], cfg.batch_fn
    out = _both_ways(build, 4)
    (got, recs) = out[True]
    assert recs and all(r.steps >= core.Recurrence.LEAST for r in recs)
    _close(out, 4 * H, T)


def _cells(T, B, H, feedback):
    """An unrolled cell h' = sigmoid(z[:, :H]) * tanh(z[:, H:]) + h with z = (x.W + b) + (h.U + c); with feedback x
    depends on h by another way than U."""
    def build():
        rs = np.random.RandomState(0)
        shared = lambda *shape: cgt.shared((rs.randn(*shape) * 0.2).astype("f4"), fixed_shape_mask="all")
        (W, U, V) = (shared(24, 2 * H), shared(H, 2 * H), shared(H, 24))
        (b, c) = (shared(1, 2 * H), shared(1, 2 * H))
        x = cgt.tensor3("x", fixed_shape=(T, B, 24))
        h = cgt.tanh(x[0].dot(cgt.constant((rs.randn(24, H) * 0.2).astype("f4"))))
        hs = []
        for t in range(T):
            xt = x[t] + cgt.tanh(h.dot(V)) if feedback else x[t]
            z = cgt.broadcast("+", xt.dot(W), b, "xx,1x") + cgt.broadcast("+", h.dot(U), c, "xx,1x")
            h = cgt.sigmoid(z[:, 0:H]) * cgt.tanh(z[:, H:2 * H]) + h * 0.9
            hs.append(h)
        loss = cgt.add_multi([cgt.square(k).sum() for k in hs]) / (T * B)
        params = [W, U, b, c] + ([V] if feedback else [])
        f = cgt.function([x], [loss, hs[-1], hs[T // 2]], updates=[(p, p - 0.01 * g) for (p, g) in zip(params, cgt.grad(loss, params))])
        return f, params, lambda r: [r.randn(T, B, 24).astype("f4")]
    return build


@pytest.mark.parametrize("B,H", [(40, 48), (64, 128), (70, 33)])
def test_cell_with_results_handed_out(rt, B, H):
    out = _both_ways(_cells(8, B, H, False), 4)
    assert out[True][1]
    _close(out, 2 * H, 8)


def test_feedback_by_another_way_is_not_grouped(rt):
    out = _both_ways(_cells(9, 40, 48, True), 4)
    _close(out, 96, 9)


@pytest.mark.parametrize("dtype", ["f4", "f8"])
def test_column_sums_over_a_cluster_of_blocks(rt, dtype):
    """[R, K] over R: rows around those at which two, four and eight blocks share a column, with and without a remainder."""
    from cgt_b200 import runtime
    rs = np.random.RandomState(5)
    for (R, K) in [(255, 33), (256, 1), (257, 70), (511, 32), (512, 31), (513, 512), (1023, 40), (1024, 64), (1025, 129), (2048, 2400), (3200, 512), (4096, 5)]:
        a = rs.randn(R, K).astype(dtype)
        with cgt.scoped_update_config(precision="single" if dtype == "f4" else "double"):
            x = cgt.matrix("x")
            f = cgt.function([x], [cgt.sum(x, axis=0), cgt.max(x, axis=0)])
        (total, top) = f(runtime.device_array(a))
        # any order of R additions is off by at most R * eps * sum |a|
        assert (np.abs(total.reshape(-1) - a.astype("f8").sum(0)) <= R * np.finfo(dtype).eps * np.abs(a).sum(0)).all(), (R, K)
        assert np.array_equal(top.reshape(-1), a.max(0))


def test_sums_of_squares_of_many_arrays(rt):
    """Every remainder of the 16-byte loads, one element, ragged views, more arrays than one launch takes."""
    shapes = [(1, 1), (3, 1), (1, 5), (65, 512), (7, 4096), (1, 4097), (128, 33), (1024, 1024)] + [(i + 1, 3) for i in range(30)]
    xs = [cgt.matrix("x%d" % i, fixed_shape=s) for (i, s) in enumerate(shapes)]
    for on in (False, True):
        with cgt.scoped_update_config(fuse_square_sums=on):
            f = cgt.function(xs, [cgt.square(x).sum() * 1.0 for x in xs])
        assert any(isinstance(getattr(i, "op", None), core.SumSquares) for i in f.eg.instrs) == on
        for call in range(3):
            vals = [np.random.RandomState(call).randn(*s).astype("f4") for s in shapes]
            for (v, got) in zip(vals, f(*vals)):
                want = np.square(v.astype("f8")).sum()
                assert abs(got - want) <= v.size * np.finfo("f4").eps * want

"""FMA products (csrc/gemm_tile.cu): edges of the tiles, of the K slices and of the splits; the output-stage program."""
import numpy as np
import pytest

import cgt_b200 as cgt
from cgt_b200 import runtime
from tests.gpu_util import Dev, call

pytestmark = pytest.mark.gpu

SHAPES = [
    # (M, N, K): one element, ragged tiles, exact tiles, K below / at / above a slice, few rows, long K over several clusters
    (1, 1, 1), (31, 33, 65), (32, 32, 64), (33, 97, 63), (64, 64, 128), (65, 130, 257), (129, 31, 31), (1, 257, 784), (5, 70, 130),
    (8, 33, 2048), (9, 20, 39200), (20, 9, 8191), (200, 300, 5), (700, 600, 100), (60, 60, 0),
]


@pytest.mark.parametrize("dtype", ["f4", "f8"])
@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_tile_products(rt, dtype, tA, tB):
    rs = np.random.RandomState(3)
    eps = np.finfo(dtype).eps
    for (M, N, K) in SHAPES:
        A = rs.randn(*((K, M) if tA else (M, K))).astype(dtype)
        B = rs.randn(*((N, K) if tB else (K, N))).astype(dtype)
        dA, dB, dC = Dev(A), Dev(B), Dev(np.full((M, N), 7, dtype))
        lda, ldb = max(A.shape[1], 1), max(B.shape[1], 1)
        if dtype == "f4":
            call("cgtb_sgemm", tA, tB, M, N, K, dA.ptr, lda, dB.ptr, ldb, dC.ptr, N, 6)
        else:
            call("cgtb_dgemm", tA, tB, M, N, K, dA.ptr, lda, dB.ptr, ldb, dC.ptr, N)
        a, b = (A.T if tA else A).astype("f8"), (B.T if tB else B).astype("f8")
        # any order of K additions of rounded products is off by at most K * eps * sum |a||b|; float64 is checked against
        # another float64 product, which is off by as much itself
        bound = 2 * (K + 2) * eps * (np.abs(a) @ np.abs(b)) + 1e-30
        assert (np.abs(dC.get() - a @ b) <= bound).all(), (M, N, K)


@pytest.mark.parametrize("B,xdim,hidden", [(1, 70, 33), (7, 64, 300), (33, 129, 65), (128, 784, 256), (300, 40, 500)])
def test_chains_in_the_output_stage_change_no_bit(rt, B, xdim, hidden):
    """x.W + b, tanh, its derivative, the gradients and p - lr * dW: with the chains run by the products and as kernels of
    their own, losses and parameters are the same bits (every kernel that carries a chain occurs in these sizes)."""
    results = {}
    rs = np.random.RandomState(B)
    xs = rs.rand(B, xdim).astype("f4")
    for on in (False, True):
        with cgt.scoped_update_config(fuse_product_chains=on):
            x = cgt.matrix("x", fixed_shape=(B, xdim))
            r2 = np.random.RandomState(1)
            W = cgt.shared((r2.randn(xdim, hidden) * 0.1).astype("f4"), fixed_shape_mask="all")
            b = cgt.shared(r2.randn(1, hidden).astype("f4"), fixed_shape_mask="all")
            V = cgt.shared((r2.randn(hidden, hidden) * 0.1).astype("f4"), fixed_shape_mask="all")
            h = cgt.tanh(cgt.broadcast("+", x.dot(W), b, "xx,1x"))
            loss = cgt.square(cgt.tanh(h.dot(V))).sum() / B
            grads = cgt.grad(loss, [W, b, V])
            f = cgt.function([x], [loss, h], updates=[(p, p - 0.1 * g) for (p, g) in zip([W, b, V], grads)])
        n = sum("op:Mul22Chain" in repr(i) for i in f.eg.instrs)
        assert (n > 0) == on
        results[on] = [np.asarray(v).copy() for _ in range(4) for v in f(xs)] + [p.op.get_value() for p in (W, b, V)]
    for (p, q) in zip(results[False], results[True]):
        assert np.array_equal(p, q)


@pytest.mark.parametrize("P,M,N,K", [(64, 64, 64, 64), (512, 64, 64, 64), (16, 256, 256, 128), (128, 256, 256, 256), (70, 100, 100, 1000)])
def test_batched_products_are_plain_float32(rt, P, M, N, K):
    """A chain of K rounded additions of random terms is off by u * sqrt(K / 6) (2-norm, u = 2^-24), half as much again for
    its spread; the TF32 split of the tensor-core kernels is off by more. Long batches and short ones alike."""
    rs = np.random.RandomState(0)
    (A, B) = (rs.randn(P, M, K).astype("f4"), rs.randn(P, K, N).astype("f4"))
    (dA, dB, dC) = (Dev(A), Dev(B), Dev(np.zeros((P, M, N), "f4")))
    call("cgtb_sgemm_batched", 0, 0, P, M, N, K, dA.ptr, K, M * K, dB.ptr, N, K * N, dC.ptr, N, M * N, 0)
    want = A.astype("f8") @ B.astype("f8")
    assert np.linalg.norm(dC.get() - want) <= 1.5 * 2.0 ** -24 * np.sqrt(K / 6.0) * np.linalg.norm(want)

"""Products summed over a batch (strideC = 0) and column sums of a batch, against one call per matrix."""
import math

import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from parallelreverseautodiff_b200.graph import Graph
from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,n,k,batch", [(3, 5, 7, 2), (84, 24, 56, 4), (300, 70, 33, 9), (2048, 128, 256, 4), (40, 64, 16384, 5)])
@pytest.mark.parametrize("beta", [0.0, 1.0])
def test_sum_over_batch(engine, dtype, m, n, k, batch, beta):
    r = rng(m + n)
    A, B = r.standard_normal((batch * m, k)).astype(dtype), r.standard_normal((batch * k, n)).astype(dtype)
    C0 = r.standard_normal((m, n)).astype(dtype)
    dA, dB, one, sep = engine.upload(A), engine.upload(B), engine.upload(C0), engine.upload(C0)
    engine.gemm(dA.view((m, k)), dB.view((k, n)), one, batch=batch, strideA=m * k, strideB=k * n, strideC=0, beta=beta)
    for b in range(batch):
        engine.gemm(dA.view((m, k), b * m * k), dB.view((k, n), b * k * n), sep, beta=1.0 if b else beta)
    want = sum(A[b * m:(b + 1) * m].astype(np.float64) @ B[b * k:(b + 1) * k].astype(np.float64) for b in range(batch)) + beta * C0
    tol = (3e-6 if dtype == np.float32 else 1e-14) * batch * np.sqrt(k)
    np.testing.assert_allclose(one.numpy(), want, rtol=0, atol=tol * 4)
    if dtype == np.float64 and m * n * k * batch < 1 << 24:     # the same kernels, and sums in double either way
        np.testing.assert_array_equal(one.numpy(), sep.numpy())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("rows,cols,batch", [(1, 1, 1), (84, 56, 4), (512, 33, 3), (513, 40, 4), (2048, 256, 4), (700, 70000, 2), (100000, 3, 2)])
def test_column_sums_of_a_batch(engine, dtype, rows, cols, batch):
    x = rng(rows).standard_normal((batch, rows, cols)).astype(dtype)
    out = engine.empty((batch, cols), dtype)
    engine.column_sums(engine.upload(x.reshape(-1, cols)), out, rows, batch, 0.125)
    np.testing.assert_allclose(out.numpy(), 0.125 * x.astype(np.float64).sum(1), rtol=1e-6 if dtype == np.float32 else 1e-12, atol=1e-9)


@pytest.mark.parametrize("dtype,m,n,k", [(np.float32, 20, 30, 40), (np.float64, 20, 30, 40), (np.float64, 512, 256, 512)])
def test_a_recorded_sum_without_scratch(dtype, m, n, k):
    """A recording cannot grow scratch: the sum then goes product by product."""
    batch, r = 4, rng(m)
    A, B = r.standard_normal((batch, m, k)).astype(dtype), r.standard_normal((batch, k, n)).astype(dtype)
    with E.Engine(0) as eng:
        a, b, out = eng.upload(A.reshape(-1, k)), eng.upload(B.reshape(-1, n)), eng.zeros((m, n), dtype)
        seq = eng.record(lambda: eng.gemm(a.view((m, k)), b.view((k, n)), out, batch=batch, strideA=m * k, strideB=k * n, strideC=0))
        seq.launch()
        want = np.einsum("bmk,bkn->mn", A.astype(np.float64), B.astype(np.float64))
        np.testing.assert_allclose(out.numpy(), want, rtol=0, atol=(1e-5 if dtype == np.float32 else 1e-13) * batch * np.sqrt(k))
        seq.close()
        for x in (a, b, out):
            x.free()


def test_a_recorded_backward_with_the_scratch_of_single_products():
    """Packing a float Backward's gradient once takes twice the scratch of one product: a recording that has only that much goes
    product by product, with the same values."""
    n, r = 512, rng(9)
    up = [r.standard_normal((n, n)).astype(np.float32) for _ in range(3)]
    with E.Engine(0) as eng:
        A, B, dC = (eng.upload(x) for x in up)
        want_a, _ = eng.matmul_backward(A, B, dC, need_dB=False)
        _, want_b = eng.matmul_backward(A, B, dC, need_dA=False)
        dA, dB = eng.zeros((n, n), np.float32), eng.zeros((n, n), np.float32)
        seq = eng.record(lambda: eng.matmul_backward(A, B, dC, dA=dA, dB=dB))
        seq.launch()
        np.testing.assert_array_equal(dA.numpy(), want_a.numpy())
        np.testing.assert_array_equal(dB.numpy(), want_b.numpy())
        seq.close()
        for x in (A, B, dC, want_a, want_b, dA, dB):
            x.free()


def test_partial_products_count_as_scratch():
    """The products of a sum over a batch wait in scratch, which the device's facts include."""
    n, batch = 100, 4
    with E.Engine(0) as eng:
        a, out = eng.zeros((batch * n, n), np.float32), eng.empty((n, n), np.float32)
        before = eng.device_info()["scratch_bytes"]
        eng.gemm(a.view((n, n)), a.view((n, n)), out, batch=batch, strideA=n * n, strideB=n * n, strideC=0)
        assert eng.device_info()["scratch_bytes"] - before >= batch * n * n * 4
        a.free()
        out.free()


@pytest.mark.parametrize("rows,where", [(n, "operation") for n in (5, 20, 45, 64, 100, 200, 512)] + [(n, "graph") for n in (5, 20, 45, 64, 100)])
def test_column_sums_lose_no_more_than_eight_chains(engine, rows, where):
    """Column sums in double, on average over many columns as close to the exact sum as eight chains (row r in chain r mod 8) that
    are added one after the other: the separate kernel's order in its first form."""
    cols = 600 if where == "operation" else 96
    x = rng(rows).standard_normal((rows, cols))
    chains = np.zeros((8, cols))
    for r in range(rows):
        chains[r % 8] += x[r]
    eight = np.zeros(cols)
    for c in chains:
        eight += c
    if where == "operation":
        got = engine.add_broadcast_backward(engine.upload(x)).numpy()[0]
    else:
        g = Graph(engine, np.float64)
        d = engine.zeros((1, cols), np.float64)
        y = g.input(engine.zeros((rows, cols), np.float64))
        for _ in range(40):                              # enough operations for a plan
            y = g.node("MatrixMultiplyScalarOperation", [y], scalar=1.0)
        out = g.node("MatrixAddBroadcastingOperation", [y, g.weight(engine.zeros((1, cols), np.float64), d)])
        g.forward()
        n0 = engine.launch_count()
        g.backward(out, engine.upload(x))
        assert engine.launch_count() - n0 == 1
        got = d.numpy()[0]
        g.close()
    exact = np.array([math.fsum(c) for c in x.T])
    rms = lambda a: np.sqrt(np.mean((a - exact) ** 2))  # noqa: E731
    assert rms(got) <= 1.1 * rms(eight) + 1e-17          # (a tenth: the scatter of the mean over the columns)

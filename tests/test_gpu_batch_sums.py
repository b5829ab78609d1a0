"""Products summed over a batch (strideC = 0) and column sums of a batch, against one call per matrix."""
import numpy as np
import pytest

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

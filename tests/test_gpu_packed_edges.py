"""Packing of matrices that fill their last tiles only in part, with column sums, and the LayerNorm passes that pack."""
import numpy as np
import pytest

import oracle as O
from parallelreverseautodiff_b200 import engine as E
from util import assert_close, rng

pytestmark = pytest.mark.gpu
f = np.float32
BOTH = E.PACK_ROWS | E.PACK_COLS
SHAPES = [(1, 4), (129, 96), (300, 132), (2560, 96), (1000, 288), (8193, 384), (384, 128), (257, 130)]


def _absprod(a, b):
    return np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)


def _check_products(engine, P, X, r, what):
    """X Y and X^T Z through the packed X, in both orientations."""
    m, n = X.shape
    Y, Z = r.standard_normal((n, 40)).astype(f), r.standard_normal((m, 24)).astype(f)
    PY = engine.packed(n, 40, E.PACK_COLS, 0, 128).pack(engine.upload(Y))
    PZ = engine.packed(m, 24, E.PACK_COLS, 0, 128).pack(engine.upload(Z))
    a, b = engine.empty((m, 40), f), engine.empty((n, 24), f)
    engine.gemm_packed(P, E.PACK_ROWS, PY, E.PACK_COLS, a)
    engine.gemm_packed(P, E.PACK_COLS, PZ, E.PACK_COLS, b)
    assert_close(a.numpy(), O.matmul_forward(X, Y), _absprod(X, Y), f"{what} by rows")
    assert_close(b.numpy(), O.matmul_forward(np.ascontiguousarray(X.T), Z), _absprod(X.T, Z), f"{what} by columns")


@pytest.mark.parametrize("block", [128, 256])
@pytest.mark.parametrize("shape", SHAPES)
def test_column_sums_and_ragged_tiles(engine, shape, block):
    m, n = shape
    r = rng(m + n)
    X, S = r.standard_normal(shape).astype(f), r.standard_normal(shape).astype(f)
    sums = engine.empty((n,), f)
    P = engine.packed(m, n, BOTH, 128, block).column_sums(sums).pack(engine.upload(X))
    np.testing.assert_allclose(sums.numpy(), X.astype(np.float64).sum(0), rtol=1e-6, atol=1e-6)
    if block == 128:
        _check_products(engine, P, X, r, f"{shape}")
    dev = engine.upload(S), engine.upload(X)
    copy, ref = engine.empty(shape, f), engine.act_backward(E.ACT_GELU, *dev)
    P.act_backward(E.ACT_GELU, *dev, copy)
    np.testing.assert_array_equal(copy.numpy(), ref.numpy())
    np.testing.assert_allclose(sums.numpy(), ref.numpy().astype(np.float64).sum(0), rtol=1e-6, atol=1e-6)
    sums = engine.zeros((n,), f)
    P.column_sums(sums).column_sums(None).pack(dev[0])
    assert not sums.numpy().any()


@pytest.mark.parametrize("shape", [(1, 4), (129, 96), (1024, 128), (1000, 100), (127, 64)])
def test_layernorm_packs(engine, shape):
    m, n = shape
    r = rng(m)
    X, D, R = (r.standard_normal(shape).astype(f) for _ in range(3))
    x, d, res = engine.upload(X), engine.upload(D), engine.upload(R)
    mu, sd, tot, dx = engine.empty((m,), f), engine.empty((m,), f), engine.empty(shape, f), engine.empty(shape, f)
    sums = engine.empty((n,), f)
    P = engine.packed(m, n, BOTH, 128, 128).column_sums(sums)
    for src, kw in ((X, {}), (X + R, dict(residual=res, sum_out=tot))):
        ref, mr, sr = O.layernorm_forward(src)
        P.layernorm(x, mu, sd, **kw)
        if kw:
            np.testing.assert_array_equal(tot.numpy(), src)
        assert_close(mu.numpy(), np.asarray(mr).reshape(m), 1.0, "mean")
        assert_close(sd.numpy(), np.asarray(sr).reshape(m), 1.0, "sigma")
        np.testing.assert_allclose(sums.numpy(), ref.astype(np.float64).sum(0), rtol=1e-4, atol=1e-5 * m)
        if m > 1:
            _check_products(engine, P, ref, r, f"LayerNorm {shape}")
    P.layernorm_backward(tot, mu, sd, d, res, dx)
    want = R + engine.layernorm_backward(tot, mu, sd, d).numpy()
    np.testing.assert_array_equal(dx.numpy(), want)
    np.testing.assert_array_equal(engine.layernorm_backward_add(tot, mu, sd, d, res).numpy(), want)
    np.testing.assert_allclose(sums.numpy(), want.astype(np.float64).sum(0), rtol=1e-5, atol=1e-5 * m)
    _check_products(engine, P, want, r, f"LayerNorm.Backward {shape}")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(5, 7), (33, 64), (3, 1)])
def test_layernorm_backward_add(engine, dtype, shape):
    r = rng(9)
    X, D, R = (r.standard_normal(shape).astype(dtype) for _ in range(3))
    y, mu, sd = engine.layernorm_forward(engine.upload(X))
    got = engine.layernorm_backward_add(engine.upload(X), mu, sd, engine.upload(D), engine.upload(R))
    want = R + engine.layernorm_backward(engine.upload(X), mu, sd, engine.upload(D)).numpy()
    np.testing.assert_array_equal(got.numpy(), want)

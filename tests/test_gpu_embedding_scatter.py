"""Ordered scatter-add where rows collect no, one, a warp's worth and many hits, against the sequential loop, bit for bit."""
import numpy as np
import pytest

import oracle as O
from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,vocab,dim,hot", [(1, 1, 1, 0), (31, 3, 5, 0), (32, 1, 8, 0), (33, 1, 8, 0), (1000, 17, 12, 500), (3000, 700, 33, 1500),
                                             (5000, 9, 1030, 0), (70000, 50, 4, 40000), (140000, 3, 6, 0), (2000, 20000, 64, 100), (100, 131000, 4, 0), (72, 131000, 4, 0)])
def test_scatter_in_input_order(engine, dtype, n, vocab, dim, hot):
    r = rng(n + vocab)
    idx = r.integers(0, vocab, n)
    idx[r.permutation(n)[:hot]] = vocab // 2
    col = idx.astype(dtype).reshape(n, 1)
    dOut = (r.standard_normal((n, dim)) * 10.0 ** r.integers(-3, 4, (n, 1))).astype(dtype)
    W = r.standard_normal((vocab, dim)).astype(dtype)
    i, d = engine.upload(col), engine.upload(dOut)
    np.testing.assert_array_equal(engine.embedding_backward(i, d, vocab).numpy(), O.embedding_backward(col, dOut, vocab))
    np.testing.assert_array_equal(engine.embedding_forward(i, engine.upload(W)).numpy(), O.embedding_forward(col, W))

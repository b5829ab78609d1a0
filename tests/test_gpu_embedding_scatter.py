"""Ordered scatter-add where rows collect no, one, a warp's worth and many hits, against the sequential loop, bit for bit."""
import time

import numpy as np
import pytest

import oracle as O
from parallelreverseautodiff_b200._lib import PradError, check
from parallelreverseautodiff_b200.engine import dtype_code
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


@pytest.mark.parametrize("dtype,dim", [(np.float32, 20), (np.float64, 3)])
@pytest.mark.parametrize("n,vocab", [(2500, 511), (2500, 512), (2500, 513), (3000, 7681), (3000, 8192), (3000, 8193), (40000, 91072), (40000, 91073)])
def test_scatter_at_the_edges_of_the_grouping(engine, dtype, dim, n, vocab):
    """Row counts on both sides of a segment, of sixteen of them and of what one launch groups; rows of 0, 1, 4, 5, 32, 33 and many
    hits at both ends of the table; a table that does not start at a 16-byte boundary."""
    r = rng(n + vocab + dim)
    idx = r.integers(0, vocab, n)
    at = 0
    for row, hits in ((0, 33), (vocab - 1, 32), (1, 5), (vocab - 2, 4), (2, 1), (vocab // 2, 700)):
        idx[at:at + hits] = row
        at += hits
    idx = r.permutation(idx)
    col = idx.astype(dtype).reshape(n, 1)
    dOut = (r.standard_normal((n, dim)) * 10.0 ** r.integers(-3, 4, (n, 1))).astype(dtype)
    expected = O.embedding_backward(col, dOut, vocab)
    i, d = engine.upload(col), engine.upload(dOut)
    np.testing.assert_array_equal(engine.embedding_backward(i, d, vocab).numpy(), expected)
    room = engine.upload(np.full((1, vocab * dim + 1), np.nan, dtype))
    odd = room.view((vocab, dim), 1)
    engine.embedding_backward(i, d, vocab, out=odd)
    np.testing.assert_array_equal(odd.numpy(), expected)


def test_bad_indices_are_told_apart_from_the_calls_after_them(engine):
    W, d = engine.upload(np.ones((5, 4), np.float32)), engine.upload(np.ones((3, 4), np.float32))
    good, bad = (engine.upload(np.array(v, np.float32).reshape(3, 1)) for v in ([0, 4, 4], [1, 5, 2]))
    for _ in range(3):
        with pytest.raises(PradError):
            engine.embedding_forward(bad, W)
        assert engine.embedding_forward(good, W).numpy().sum() == 12
        with pytest.raises(PradError):
            engine.embedding_backward(bad, d, 5)
        np.testing.assert_array_equal(engine.embedding_backward(good, d, 5).numpy()[:, 0], [1, 0, 0, 0, 2])


@pytest.mark.parametrize("dtype,dim", [(np.float32, 1), (np.float32, 33), (np.float32, 132), (np.float32, 260), (np.float64, 18), (np.float64, 67)])
@pytest.mark.parametrize("n,vocab", [(9000, 60), (60000, 500), (60000, 2500), (140000, 700), (140000, 540), (530000, 3000)])
def test_rows_of_many_and_of_very_many_hits(engine, dtype, dim, n, vocab):
    """Most rows beyond what a warp orders: lists of 33, 255, 256, 257, 2048 and 2049 hits beside those of the calls' own lengths, over one
    segment of rows, over several, and in calls that are too large for one launch, where a list runs over several windows."""
    r = rng(n + vocab + dim)
    idx = r.integers(0, vocab, n)
    at = 0
    for row, hits in ((0, 33), (vocab - 1, 256), (1, 257), (vocab - 2, 255), (2, 2048), (vocab // 2, 2049)):
        idx[idx == row] = (vocab - 3) - row % 7
        idx[at:at + hits] = row
        at += hits
    idx = r.permutation(idx)
    col = idx.astype(dtype).reshape(n, 1)
    dOut = (r.standard_normal((n, dim)) * 10.0 ** r.integers(-3, 4, (n, 1))).astype(dtype)
    got = engine.embedding_backward(engine.upload(col), engine.upload(dOut), vocab).numpy()
    np.testing.assert_array_equal(got, O.embedding_backward(col, dOut, vocab))


def test_rows_of_many_hits_cost_what_their_data_costs(engine):
    """The same rows of dOut, added up over 50000 rows of about 21 hits and over 25000 of about 42: two ways through the sums, the same
    bytes.  (A search per task that grew with the number of such rows made the second one 60 times as slow.)"""
    n, dim = 1 << 20, 64
    dOut = engine.zeros((n, dim), np.float32)
    times = []
    for vocab in (50000, 25000):
        idx = engine.upload(rng(vocab).integers(0, vocab, (n, 1)).astype(np.float32))
        out = engine.empty((vocab, dim), np.float32)
        best = 1e9
        for _ in range(4):
            engine.sync()
            t = time.perf_counter()
            engine.embedding_backward(idx, dOut, vocab, out=out)
            engine.sync()
            best = min(best, time.perf_counter() - t)
        times.append(best)
    assert times[1] < 10 * times[0], times


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_gather_of_one_column_in_the_place_of_its_indices(engine, dtype):
    """A row is written after its own index has been read, so a one-column gather may replace its indices.  The table's values are no
    indices: whoever looked at them there would find rows outside the table."""
    n, vocab = 1 << 20, 1000
    idx = rng(3).integers(0, vocab, (n, 1))
    W = -1.0 - np.arange(vocab, dtype=dtype).reshape(vocab, 1)
    table = engine.upload(W)
    for _ in range(5):
        m = engine.upload(idx.astype(dtype))
        check(engine.lib.prad_embedding_forward(engine.ctx, dtype_code(dtype), m.ptr, table.ptr, m.ptr, n, vocab, 1))
        np.testing.assert_array_equal(m.numpy(), W[idx[:, 0]])

"""Mean and deviation of a gradient from one pass: sizes at the edges of a CTA's share, values far from zero, unaligned tensors."""
import numpy as np
import pytest

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 511, 512, 513), (1023, 1024, 1025, 5000), (300001, 7), (2100000, 2049)])
@pytest.mark.parametrize("mean", [0.0, 1000.0])
def test_limits_against_64_bits(engine, dtype, sizes, mean):
    """A clipped value is 1 + |z|, z = (g - mean) / sigma over the tensor.  Mean and sigma are rounded to the matrix type once, which
    moves z by at most u |mean| / sigma and 2 u |z| (u: the type's rounding); |z| stays below 8 here."""
    r = rng(sum(sizes))
    host = [(mean + 3.0 * r.standard_normal((1, n))).astype(dtype) for n in sizes]
    room = engine.upload(np.zeros((1, sum(sizes) + len(sizes)), dtype))
    dev, at = [], 0
    for g in host:                                  # every tensor one element further: aligned and not
        dev.append(room.view(g.shape, at))
        engine.copy(dev[-1], engine.upload(g))
        at += g.size + 1
    engine.clip_reference(dev, 1e6, 1e-30)
    u = np.finfo(dtype).eps
    for g, d in zip(host, dev):
        x = g.astype(np.float64)
        got = d.numpy().astype(np.float64)
        sigma = x.std()
        if g.size == 1:                             # sigma 0: no limit
            np.testing.assert_array_equal(got, x)
            continue
        limit = 1 + np.abs((x - x.mean()) / sigma)
        expected = np.clip(x, -limit, limit)
        assert np.abs(got - expected).max() <= 4 * u * (abs(mean) / sigma + 8 * 8 + np.abs(x).max() / sigma)

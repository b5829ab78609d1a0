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


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("beside", [0, 40000, 3000000])
@pytest.mark.parametrize("spread", [1, 2, 3])
def test_limits_where_the_deviations_are_rounding(engine, dtype, spread, beside):
    """Gradients of one value repeated (spread 1), or of neighbouring numbers of the type: c + k units in the last place, k < spread.  The
    mean is a number of the type near them, c + j units, so sigma and z are those of the small whole numbers k - j, up to the five
    roundings of sigma (conversion, quotient, root) and of the limit.  Sigma 0 (all equal to the mean) sets no limit.  That holds for
    one CTA and for several, alone or beside a large tensor, which changes how many a tensor gets."""
    u, clip = np.finfo(dtype).eps, dtype(4)
    for n in (600, 700, 931, 1000, 1500, 3000, 8113, 17689, 70001):
        r = rng(n)
        unit = u * 4                                # of numbers in [4, 8)
        ks = [r.integers(0, spread, n) if spread > 1 else np.zeros(n, int) for _ in range(6)]
        host = [(dtype(r.uniform(4.1, 7.9)) + (k * unit).astype(dtype)).reshape(1, n) for k in ks]
        dev = [engine.upload(g) for g in host]
        large = [engine.upload(r.standard_normal((1, beside)).astype(dtype))] if beside else []
        engine.clip_reference(dev + large, float(clip), 1e-30)
        for g, d, k in zip(host, dev, ks):
            got, low = d.numpy().astype(np.float64)[0], g.min().astype(np.float64)
            k = np.rint((g[0].astype(np.float64) - low) / unit)
            errors = []
            for j in range(-16, 17):
                sigma = np.sqrt(np.mean((k - j) ** 2))
                limit = np.minimum(4.0, 1 + np.abs(k - j) / sigma) if sigma else np.inf
                errors.append(np.abs(got - np.minimum(g[0].astype(np.float64), limit)).max())
            assert min(errors) <= 8 * u * 4, (n, min(errors))

"""Tile shapes of the SIMT product: edges of every tile size, remainders of k against the stages, rows that do not start at
a 16-byte boundary, and both products of a Backward in one launch -- bit for bit the oracle's sequential loops."""
import numpy as np
import pytest

import oracle as O
from parallelreverseautodiff_b200 import engine as E
from util import rng

pytestmark = pytest.mark.gpu

# from one 16 x 16 tile to several 128 x 128 tiles per SM (float)
SHAPES = [(1, 1, 17), (15, 33, 16), (16, 16, 16), (17, 31, 18), (40, 129, 50), (97, 160, 96), (260, 784, 100), (513, 66, 513),
          (130, 40, 520), (700, 33, 702), (1030, 9, 1027), (2050, 7, 2049)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("M,K,N", SHAPES)
def test_products_equal_the_sequential_loops(engine, dtype, M, K, N):
    r = rng(M + K + N)
    A, B, dC = (r.standard_normal(s).astype(dtype) for s in ((M, K), (K, N), (M, N)))
    saved = r.standard_normal((M, K)).astype(dtype)
    a, b, dc, sv = (engine.upload(x) for x in (A, B, dC, saved))
    np.testing.assert_array_equal(engine.matmul_forward(a, b).numpy(), O.matmul_forward(A, B))
    dA, dB = O.matmul_backward(A, B, dC)
    gA, gB = engine.matmul_backward(a, b, dc)
    np.testing.assert_array_equal(gA.numpy(), dA)
    np.testing.assert_array_equal(gB.numpy(), dB)
    hA, hB = engine.matmul_backward(a, b, dc, act_below=E.ACT_LEAKY_RELU, saved_below=sv, act_alpha=0.01, dB=gB, accumulate_dB=True)
    np.testing.assert_array_equal(hA.numpy(), O.leaky_relu_backward(saved, dA, 0.01))
    np.testing.assert_array_equal(hB.numpy(), dB + dB)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
def test_pitches_and_epilogues(engine, dtype, pad):
    M, K, N = 75, 101, 53
    r = rng(pad)
    A, B = r.standard_normal((M, K + pad)).astype(dtype), r.standard_normal((K, N + pad)).astype(dtype)
    bias = r.standard_normal((1, N)).astype(dtype)
    ref = O.matmul_forward(np.ascontiguousarray(A[:, :K]), np.ascontiguousarray(B[:, :N]))
    out = engine.zeros((M, N + pad), dtype)
    engine.gemm(engine.upload(A), engine.upload(B), out, M=M, N=N, K=K, lda=K + pad, ldb=N + pad, ldc=N + pad)
    np.testing.assert_array_equal(out.numpy()[:, :N], ref)
    assert not out.numpy()[:, N:].any()
    a, b = engine.upload(np.ascontiguousarray(A[:, :K])), engine.upload(np.ascontiguousarray(B[:, :N]))
    z = engine.empty((M, N), dtype)
    y = engine.matmul_forward(a, b, bias=engine.upload(bias), Z_out=z, act=E.ACT_LEAKY_RELU, act_alpha=0.01)
    np.testing.assert_array_equal(z.numpy(), ref + bias)
    np.testing.assert_array_equal(y.numpy(), O.leaky_relu_forward(ref + bias, 0.01))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("M,K,N", [(512, 32, 512), (512, 33, 512), (512, 48, 508), (510, 49, 510), (184, 80, 1008), (1000, 271, 96), (1000, 273, 96),
                                   (256, 512, 512), (256, 764, 512), (256, 784, 512)])
def test_ways_to_copy_small_tiles(engine, dtype, M, K, N):
    """32 x 32 tiles on both sides of the rules for their copies: the last stage of k half full or fuller, aligned rows or not, up to four
    tiles an SM and more."""
    test_products_equal_the_sequential_loops(engine, dtype, M, K, N)

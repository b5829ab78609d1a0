"""Products of packed operands at output widths whose tiles are narrower than 256 columns, with bias, beta and k slices:
against pairs of CTAs (whose tiles are always 256 wide) bit for bit, and sliced contractions against double."""
import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from util import rng

pytestmark = pytest.mark.gpu
f = np.float32


@pytest.mark.parametrize("n", [1, 31, 32, 33, 96, 127, 130, 160, 255, 257, 288, 300, 384, 510, 520, 1040])
@pytest.mark.parametrize("m,k", [(129, 96), (2000, 160), (385, 40)])
def test_narrow_tiles(engine, m, n, k):
    r = rng(m + n + k)
    X, Y = r.standard_normal((m, k)).astype(f), r.standard_normal((k, n)).astype(f)
    bias, C0 = engine.upload(r.standard_normal((1, n)).astype(f)), r.standard_normal((m, n)).astype(f)
    PX = engine.packed(m, k, E.PACK_ROWS, 128).pack(engine.upload(X))
    PY = engine.packed(k, n, E.PACK_COLS, 0, 128).pack(engine.upload(Y))
    outs = []
    for mode in ("0", "2"):
        engine.set_option("tc_pair", mode)
        got = [engine.upload(C0) for _ in range(3)]
        engine.gemm_packed(PX, E.PACK_ROWS, PY, E.PACK_COLS, got[0])
        engine.gemm_packed(PX, E.PACK_ROWS, PY, E.PACK_COLS, got[1], bias=bias)
        engine.gemm_packed(PX, E.PACK_ROWS, PY, E.PACK_COLS, got[2], alpha=0.5, beta=1.0, bias=bias)
        outs.append([g.numpy() for g in got])
    engine.set_option("tc_pair", "1")          # the default
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    want = X.astype(np.float64) @ Y
    np.testing.assert_allclose(outs[0][0], want, rtol=0, atol=2e-5 * np.sqrt(k))


@pytest.mark.parametrize("m,n", [(96, 96), (96, 288), (384, 96), (130, 31), (64, 2048)])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_many_slices(engine, m, n, beta):
    r, k = rng(m * n), 160 * 1024 + 32
    X, Y, C0 = (r.standard_normal(s).astype(f) for s in ((k, m), (k, n), (m, n)))
    PX = engine.packed(k, m, E.PACK_COLS, 0, 128).pack(engine.upload(X))
    PY = engine.packed(k, n, E.PACK_COLS, 0, 128).pack(engine.upload(Y))
    out = engine.upload(C0)
    engine.gemm_packed(PX, E.PACK_COLS, PY, E.PACK_COLS, out, alpha=0.25, beta=beta)
    want = 0.25 * (X.astype(np.float64).T @ Y) + beta * C0
    np.testing.assert_allclose(out.numpy(), want, rtol=0, atol=2e-6 * np.sqrt(k))


@pytest.mark.parametrize("m,k,n", [(1000, 520, 300), (4097, 130, 258), (640, 511, 515)])
@pytest.mark.parametrize("act", [E.ACT_NONE, E.ACT_GELU, E.ACT_LEAKY_RELU, E.ACT_TANH])
def test_backward_of_a_large_float_product(engine, m, k, n, act):
    """Both gradients from one packing of dC: the bits of one product at a time, in one call with the activation or after it."""
    r = rng(m + n)
    A, B, dOut, saved = (engine.upload(r.standard_normal(s).astype(f)) for s in ((m, k), (k, n), (m, n), (m, n)))
    dC = engine.act_backward(act, saved, dOut, 0.1) if act != E.ACT_NONE else dOut
    dA1, _ = engine.matmul_backward(None, B, dC, need_dB=False)
    _, dB1 = engine.matmul_backward(A, None, dC, need_dA=False)
    dA2, dB2 = engine.matmul_backward(A, B, dC)
    dP3, dA3, dB3 = engine.matmul_act_backward(A, B, dOut, act, saved, 0.1)
    np.testing.assert_array_equal(dP3.numpy(), dC.numpy())
    for got, want in ((dA2, dA1), (dB2, dB1), (dA3, dA1), (dB3, dB1)):
        np.testing.assert_array_equal(got.numpy(), want.numpy())
    acc = engine.upload(np.ones((k, n), f))
    dA4 = engine.matmul_backward(A, B, dC, dB=acc, accumulate_dB=True, dB_scale=0.5, act_below=E.ACT_LEAKY_RELU,
                                 saved_below=A, act_alpha=0.1)[0]
    np.testing.assert_array_equal(dA4.numpy(), engine.act_backward(E.ACT_LEAKY_RELU, A, dA1, 0.1).numpy())
    np.testing.assert_allclose(acc.numpy(), 1 + 0.5 * dB1.numpy(), rtol=0, atol=1e-5 * np.abs(dB1.numpy()).max())

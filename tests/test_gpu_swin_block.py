"""SwinBlock below and above the size from which its activations are kept as packed operands only: several backwards of one
forward, products chosen anew in between, operands that do not start at 16 bytes."""
import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from parallelreverseautodiff_b200.networks import SwinBlock
from util import rng

pytestmark = pytest.mark.gpu

DIM, HEADS, WINDOW = 128, 4, 16
TOKENS = (512, 8192)          # 8192 * 128 * 128 = 2^27 multiply-adds: packed


def _block(engine):
    r, d = rng(7), DIM
    blk = SwinBlock(engine, np.float32, d, HEADS, WINDOW)
    he = lambda a, b: (r.standard_normal((a, b)) * np.sqrt(2.0 / a)).astype(np.float32)  # noqa: E731
    bias = lambda n: (r.standard_normal((1, n)) * 0.1).astype(np.float32)  # noqa: E731
    blk.set_parameters({"Wqkv": he(d, 3 * d), "bqkv": bias(3 * d), "Wproj": he(d, d), "bproj": bias(d),
                        "W1": he(d, 4 * d), "b1": bias(4 * d), "W2": he(4 * d, d), "b2": bias(d)})
    return blk


def _data(T, seed):
    return rng(seed).standard_normal((T, DIM)).astype(np.float32)


def _results(blk, dx):
    return {"d_x": dx.numpy(), **{k: m.numpy() for k, m in blk.g.items()}}


def _once(engine, x, d_out):
    blk = _block(engine)
    blk.forward(engine.upload(x))
    return _results(blk, blk.backward(engine.upload(d_out)))


def _close(a, b):
    """Two evaluations whose products are both good to about 2e-6 of their result, eight products deep."""
    for k in a:
        assert np.linalg.norm((a[k] - b[k]).astype(np.float64)) <= 5e-5 * np.linalg.norm(b[k].astype(np.float64)), k


@pytest.mark.parametrize("T", TOKENS)
def test_every_backward_of_a_forward_is_the_same(engine, T):
    x, grads = _data(T, 1), [_data(T, 2), _data(T, 3)]
    want = [_once(engine, x, d) for d in grads]
    blk = _block(engine)
    blk.forward(engine.upload(x))
    for k in (0, 1, 0):
        got = _results(blk, blk.backward(engine.upload(grads[k])))
        for name in got:
            np.testing.assert_array_equal(got[name], want[k][name], err_msg=name)


@pytest.mark.parametrize("T", TOKENS)
@pytest.mark.parametrize("first,then", [("auto", "simt"), ("simt", "auto")])
def test_products_chosen_anew_between_forward_and_backward(engine, T, first, then):
    x, d_out = _data(T, 1), _data(T, 2)
    want = _once(engine, x, d_out)
    blk = _block(engine)
    try:
        engine.set_option("gemm_f32", first)
        blk.forward(engine.upload(x))
        engine.set_option("gemm_f32", then)
        for _ in range(2):
            _close(_results(blk, blk.backward(engine.upload(d_out))), want)
    finally:
        engine.set_option("gemm_f32", "auto")


@pytest.mark.parametrize("T", TOKENS)
@pytest.mark.parametrize("x_off,d_off", [(1, 0), (0, 1), (2, 3)])
def test_operands_off_a_16_byte_boundary(engine, T, x_off, d_off):
    x, d_out = _data(T, 1), _data(T, 2)
    want = _once(engine, x, d_out)

    def shifted(a, off):
        whole = engine.upload(np.concatenate([np.zeros(off, np.float32), a.ravel()]))
        return whole, whole.view(a.shape, off)

    blk = _block(engine)
    keep_x, xv = shifted(x, x_off)
    keep_d, dv = shifted(d_out, d_off)
    blk.forward(xv)
    _close(_results(blk, blk.backward(dv)), want)

"""Fused windowed attention, forward and Backward, against numpy in double, at window sizes around every tile size."""
import numpy as np
import pytest

from util import assert_close, rms, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ws", [1, 4, 9, 16, 17, 33, 36, 41, 49, 56, 57, 64])
@pytest.mark.parametrize("heads,hd", [(1, 16), (3, 32), (2, 64)])
def test_window_attention(engine, ws, heads, hd):
    f, r, nw = np.float32, rng(ws + hd), 5
    d, T, scale = heads * hd, 5 * ws, 1 / np.sqrt(hd)
    qkv, d_out = r.standard_normal((T, 3 * d)).astype(f), r.standard_normal((T, d)).astype(f)
    split = lambda m, o: m[:, o:o + d].astype(np.float64).reshape(nw, ws, heads, hd).transpose(0, 2, 1, 3)  # noqa: E731
    merge = lambda m: m.transpose(0, 2, 1, 3).reshape(T, d)  # noqa: E731
    Q, K, V, dO = split(qkv, 0), split(qkv, d), split(qkv, 2 * d), split(d_out, 0)
    S = scale * Q @ K.transpose(0, 1, 3, 2)
    P = np.exp(S - S.max(-1, keepdims=True))
    P /= P.sum(-1, keepdims=True)
    dP = dO @ V.transpose(0, 1, 3, 2)
    dS = P * (dP - (dP * P).sum(-1, keepdims=True))
    ref = np.concatenate([merge(scale * dS @ K), merge(scale * dS.transpose(0, 1, 3, 2) @ Q), merge(P.transpose(0, 1, 3, 2) @ dO)], 1)
    q = engine.upload(qkv)
    p, o, dq = engine.empty((nw * heads * ws, ws), f), engine.empty((T, d), f), engine.empty((T, 3 * d), f)
    engine.window_attention_forward(q, p, o, nw, ws, heads, hd, scale)
    engine.window_attention_backward(q, p, engine.upload(d_out), dq, nw, ws, heads, hd, scale)
    assert_close(p.numpy(), P.reshape(-1, ws).astype(f), 0.5, "window attention P")
    assert_close(o.numpy(), merge(P @ V).astype(f), 1.0, "window attention out")
    assert_close(dq.numpy(), ref.astype(f), 2 * rms(ref) + 0.1, "window attention d_qkv")

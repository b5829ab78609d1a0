"""Both products of a MatrixMultiplyOperation.Backward in one call: the values of the two calls one after the other, also where
a result takes the place of a matrix that the other product reads."""
import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from util import rng

pytestmark = pytest.mark.gpu


# bit-exact products, FP64 tensor cores, packed float products
@pytest.mark.parametrize("dtype,m,k,n", [(np.float32, 65, 48, 130), (np.float64, 33, 70, 40), (np.float64, 512, 512, 512),
                                         (np.float32, 512, 512, 640)])
@pytest.mark.parametrize("place", ["dB over B", "dA over A", "dB over the saved tensor", "apart"])
@pytest.mark.parametrize("recorded", [False, True])
def test_results_in_the_place_of_operands(engine, dtype, m, k, n, place, recorded):
    if place == "dB over the saved tensor" and n > m:
        m, n = n, m
    r = rng(m + k)
    up = lambda *s: r.standard_normal(s).astype(dtype)  # noqa: E731
    a, b, dc, saved = up(m, k), up(k, n), up(m, n), up(m, k)
    A, B, dC, S = (engine.upload(x) for x in (a, b, dc, saved))
    want_a, _ = engine.matmul_backward(A, B, dC, need_dB=False, act_below=E.ACT_TANH, saved_below=S)
    _, want_b = engine.matmul_backward(want_a if place == "dA over A" else A, B, dC, need_dA=False)
    want_a, want_b = want_a.numpy(), want_b.numpy()
    dA = A if place == "dA over A" else engine.empty((m, k), dtype)
    dB = {"dB over B": B, "dB over the saved tensor": S.view((k, n))}.get(place)
    dB = dB or engine.empty((k, n), dtype)
    run = lambda: engine.matmul_backward(A, B, dC, dA=dA, dB=dB, act_below=E.ACT_TANH, saved_below=S)  # noqa: E731
    if recorded:
        seq = engine.record(run)
        seq.launch()
        seq.close()
    else:
        run()
    if place == "apart":                  # one launch may use other slices of k than two: the same within the sums' rounding
        eps = np.finfo(dtype).eps * (1 if dtype == np.float64 else 4)      # packed operands carry 22 bits
        for got, want, terms in ((dA.numpy(), want_a, np.abs(dc) @ np.abs(b.T)), (dB.numpy(), want_b, np.abs(a.T) @ np.abs(dc))):
            assert (np.abs(got - want) <= 8 * eps * terms).all()
    else:
        np.testing.assert_array_equal(dA.numpy(), want_a)
        np.testing.assert_array_equal(dB.numpy(), want_b)

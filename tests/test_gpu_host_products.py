"""Products handed over as host arrays at sizes whose contraction is cut into slices: the same as on device matrices."""
import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,m,k,n", [(np.float64, 4096, 256, 128), (np.float32, 8192, 128, 128)])
def test_host_backward_equals_device_backward(engine, dtype, m, k, n):
    r = rng(m)
    A, B = r.standard_normal((m, k)).astype(dtype), r.standard_normal((k, n)).astype(dtype)
    dOut, saved = r.standard_normal((m, n)).astype(dtype), r.standard_normal((m, n)).astype(dtype)
    hP, hA, hB = engine.matmul_act_backward_host(A, B, dOut, E.ACT_TANH, saved, 0.0)
    dP = engine.act_backward(E.ACT_TANH, engine.upload(saved), engine.upload(dOut))
    dA, dB = engine.matmul_backward(engine.upload(A), engine.upload(B), dP)
    np.testing.assert_array_equal(hP, dP.numpy())
    np.testing.assert_array_equal(hA, dA.numpy())
    np.testing.assert_array_equal(hB, dB.numpy())

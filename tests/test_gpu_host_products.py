"""Products handed over as host arrays at sizes whose contraction is cut into slices: the same as on device matrices."""
import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,m,k,n", [(np.float64, 4096, 256, 128), (np.float32, 8192, 128, 128),
                                           (np.float64, 512, 512, 512), (np.float64, 70, 4000, 520), (np.float64, 1024, 512, 256)])
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
    tol = 1e-13 if dtype == np.float64 else 2e-5
    for got, want in ((hA, hP.astype(np.float64) @ B.T), (hB, A.astype(np.float64).T @ hP)):
        np.testing.assert_allclose(got, want, rtol=0, atol=tol * np.abs(want).max())


def test_host_steps_repeat_and_follow_changes(engine):
    """train_step_host replays its launches from the second equal step on: changed slopes, batch sizes, learning rates and
    options take effect, and every step equals the separate calls bit for bit."""
    from parallelreverseautodiff_b200.networks import FeedForwardNetwork
    r = rng(5)
    sizes, nets = [12, 20, 9], []
    for _ in range(2):
        net = FeedForwardNetwork(engine, np.float64, sizes)
        net.set_weights([rng(1).standard_normal((12, 20)), rng(2).standard_normal((20, 9))], [np.zeros((1, 20)), np.zeros((1, 9))])
        nets.append(net)
    a, b = nets
    for step in range(12):
        rows = 7 if step in (5, 6) else 16
        if step == 8:
            a.Parameters.LeakyReLUAlpha = b.Parameters.LeakyReLUAlpha = 0.3
        a.Parameters.AdamIteration = b.Parameters.AdamIteration = step + 1
        a.Parameters.LearningRate = b.Parameters.LearningRate = 1e-3 / (step + 1)
        x, t = r.standard_normal((rows, 12)), r.standard_normal((rows, 9))
        la = a.train_step_host(x, t)
        b._ensure_buffers(rows)
        engine.upload(x, out=b.A[0])
        engine.upload(t, out=b.target)
        b.forward()
        lb = float(b.loss_value().numpy()[0, 0])
        b.backward()
        b.clip_and_optimize()
        assert la == lb, step
        np.testing.assert_array_equal(a.dX.numpy(), b.dX.numpy())
        for p, q in zip(a.params, b.params):
            np.testing.assert_array_equal(p.numpy(), q.numpy())


def test_host_steps_of_alternating_batch_sizes(engine):
    """Epochs of full batches and a rest: the recordings of both sizes serve every epoch, with the values of the separate calls;
    other sizes in between, and the device's calls, change nothing."""
    from parallelreverseautodiff_b200.networks import FeedForwardNetwork
    r = rng(6)
    sizes, nets = [12, 20, 9], []
    for _ in range(2):
        net = FeedForwardNetwork(engine, np.float32, sizes, loss="mse")
        net.set_weights([rng(1).standard_normal((12, 20)), rng(2).standard_normal((20, 9))], [np.zeros((1, 20)), np.zeros((1, 9))])
        nets.append(net)
    a, b = nets
    recordings = {}
    for epoch in range(4):
        for rows in [16, 16, 16, 5, 5] + ([3] if epoch == 1 else []):
            x, t = r.standard_normal((rows, 12)).astype(np.float32), r.standard_normal((rows, 9)).astype(np.float32)
            la = a.train_step_host(x, t)
            recordings[epoch, rows] = a._host_sequence
            b._ensure_buffers(rows)
            engine.upload(x, out=b.A[0])
            engine.upload(t, out=b.target)
            b.forward()
            lb = float(b.loss_value().numpy()[0, 0])
            b.backward()
            b.clip_and_optimize()
            assert la == lb, (epoch, rows)
            np.testing.assert_array_equal(a.dX.numpy(), b.dX.numpy())
            for p, q in zip(a.params, b.params):
                np.testing.assert_array_equal(p.numpy(), q.numpy())
    assert recordings[0, 16] is not None and recordings[1, 16] is recordings[0, 16] and recordings[1, 5] is recordings[0, 5]
    assert recordings[2, 16] is not None and recordings[3, 16] is recordings[2, 16] and recordings[3, 5] is recordings[2, 5]


def test_host_steps_call_replaced_methods_every_time(engine):
    """A program's own forward, loss or backward runs in every step, not only in the one that would be recorded."""
    from parallelreverseautodiff_b200.networks import FeedForwardNetwork

    class Counting(FeedForwardNetwork):
        calls = 0

        def forward(self, *a, **k):
            self.calls += 1
            return super().forward(*a, **k)

    own = Counting(engine, np.float32, [6, 5, 4], loss="mse")
    plain = FeedForwardNetwork(engine, np.float32, [6, 5, 4], loss="mse")
    seen = []
    backward = plain.backward
    plain.backward = lambda *a, **k: (seen.append(1), backward(*a, **k))[1]
    x, t = rng(1).standard_normal((8, 6)).astype(np.float32), rng(2).standard_normal((8, 4)).astype(np.float32)
    for _ in range(5):
        own.train_step_host(x, t)
        plain.train_step_host(x, t)
    assert own.calls == 5 and len(seen) == 5

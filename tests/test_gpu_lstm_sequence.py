"""prad_lstm_forward / prad_lstm_backward (all time steps in one launch) against the operations one by one, bit for bit:
hidden sizes on both sides of every tile and cluster size, batches of one to several tiles and turns."""
import multiprocessing

import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from parallelreverseautodiff_b200.networks import LstmNetwork
from util import rng

pytestmark = pytest.mark.gpu

ACT = {"i": E.ACT_SIGMOID, "f": E.ACT_SIGMOID, "g": E.ACT_TANH, "o": E.ACT_SIGMOID}


def _forward_by_operation(net, x, y):
    """The time loop of the forward with one library call per managed operation."""
    e, T, B, nh, G = net.eng, net.T, net.B, net.n_h, net.GATES
    e.upload(x.reshape(T * B, -1), out=net.X)
    e.upload(y.reshape(T * B, -1), out=net.Y)
    e.zero_(net.Hprev)
    st = net._step
    for g in G:
        e.gemm(net.X, net.W[g], net.pre[g], transB=True)
    for t in range(T):
        for g in G:
            p = st(net.pre[g], t)
            if t > 0:
                e.gemm(st(net.Hprev, t), net.U[g], p, transB=True, beta=1.0)
            e.add_broadcast_forward(p, net.b[g], out=p)
            e.act_forward(ACT[g], p, out=st(net.gate[g], t))
        e.hadamard_forward(st(net.gate["i"], t), st(net.gate["g"], t), out=st(net.IG, t))
        if t > 0:
            e.hadamard_forward(st(net.gate["f"], t), st(net.C, t - 1), out=st(net.FC, t))
        else:
            e.zero_(st(net.FC, t))
        e.add_forward(st(net.FC, t), st(net.IG, t), out=st(net.C, t))
        e.act_forward(E.ACT_TANH, st(net.C, t), out=st(net.tanhC, t))
        e.hadamard_forward(st(net.gate["o"], t), st(net.tanhC, t), out=st(net.H, t))
        if t + 1 < T:
            e.copy(st(net.Hprev, t + 1), st(net.H, t))


def _backward_by_step(net):
    """The time loop of the backward with one cell call and one product per gate and step."""
    e, T, B, nh, G, st = net.eng, net.T, net.B, net.n_h, net.GATES, net._step
    rec, dc_next = [], None
    for t in range(T - 1, -1, -1):
        dc_prev = e.empty((B, nh), net.dtype) if t > 0 else None
        e.lstm_cell_backward(st(net.H, t), st(net.Y, t), 2.0 / nh, rec, dc_next, [st(net.gate[g], t) for g in G], st(net.tanhC, t),
                             st(net.C, t - 1) if t > 0 else None, [st(net.dpre[g], t) for g in G], dc_prev)
        dc_next = dc_prev
        rec = [e.empty((B, nh), net.dtype) for _ in G]
        for g, m in zip(G, rec):
            e.gemm(st(net.dpre[g], t), net.U[g], m)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nh,B,T", [(1, 1, 1), (7, 2, 3), (8, 3, 2), (9, 5, 4), (56, 7, 5), (64, 33, 3), (65, 1, 3), (100, 9, 3),
                                    (129, 18, 3), (192, 4, 3), (193, 31, 2), (256, 32, 4), (256, 70, 2), (257, 3, 3)])
def test_sequence_equals_the_operations(engine, dtype, nh, B, T):
    r = rng(nh * 100 + B)
    n_in = 5
    x, y = r.standard_normal((T, B, n_in)).astype(dtype), r.standard_normal((T, B, nh)).astype(dtype)
    par = [{g: (r.standard_normal(s) * c).astype(dtype) for g in LstmNetwork.GATES}
           for s, c in (((nh, n_in), 0.4), ((nh, nh), 1 / np.sqrt(nh)), ((nh,), 0.1))]
    a, b = (LstmNetwork(engine, dtype, n_in, nh, T, B, fused_cell=f) for f in (True, False))
    for net in (a, b):
        net.set_parameters(*par)
    a.forward(x, y)
    _forward_by_operation(b, x, y)
    for name in ("C", "tanhC", "H", "Hprev", "FC", "IG"):
        np.testing.assert_array_equal(getattr(a, name).numpy(), getattr(b, name).numpy(), err_msg=name)
    for g in a.GATES:
        np.testing.assert_array_equal(a.pre[g].numpy(), b.pre[g].numpy(), err_msg="pre " + g)
        np.testing.assert_array_equal(a.gate[g].numpy(), b.gate[g].numpy(), err_msg="gate " + g)
    a.backward()
    _backward_by_step(b)
    for g in a.GATES:
        np.testing.assert_array_equal(a.dpre[g].numpy(), b.dpre[g].numpy(), err_msg="dpre " + g)


def _take_turns(dtype, sizes):
    """Steps of networks of these sizes one after another; a later step of a network repeats its first one."""
    T, B, n_in = 3, 33, 5
    with E.Engine(0) as engine:
        nets, first = {}, {}
        for nh in sizes:
            r = rng(nh)
            x, y = r.standard_normal((T, B, n_in)).astype(dtype), r.standard_normal((T, B, nh)).astype(dtype)
            if nh not in nets:
                nets[nh] = LstmNetwork(engine, dtype, n_in, nh, T, B)
                nets[nh].set_parameters(*[{g: (r.standard_normal(s) * 0.2).astype(dtype) for g in LstmNetwork.GATES}
                                          for s in ((nh, n_in), (nh, nh), (nh,))])
            net = nets[nh]
            n0 = engine.launch_count()
            net.forward(x, y)
            net.backward()
            got = [net.H.numpy(), net.dX.numpy()] + [net.dU[g].numpy() for g in net.GATES]
            launches = engine.launch_count() - n0
            if nh in first:
                assert launches == first[nh][1]
                for a, b in zip(got, first[nh][0]):
                    np.testing.assert_array_equal(a, b)
            first.setdefault(nh, (got, launches))
        del nets, net


@pytest.mark.parametrize("dtype,sizes", [("float64", (128, 64, 128)), ("float32", (128, 64, 128)), ("float64", (192, 96, 192))])
def test_networks_of_different_sizes_take_turns(dtype, sizes):
    """One kernel serves several cluster sizes: a small network between two steps of a large one changes nothing.  In a process
    of its own, whose first launches of these kernels are the ones here."""
    p = multiprocessing.get_context("spawn").Process(target=_take_turns, args=(np.dtype(dtype), sizes))
    p.start()
    p.join(120)
    assert p.exitcode == 0

"""Graph walks as one kernel against one launch per operation: every operation type, shared and deep values, fan-in beyond
eight, pieces at the edges of 256 elements and of the product tiles, gradient destinations in one buffer."""
import ctypes as C

import numpy as np
import pytest

from parallelreverseautodiff_b200 import engine as E
from parallelreverseautodiff_b200.graph import Graph
from util import rng

pytestmark = pytest.mark.gpu


def _network(g, eng, dt, rows, cols, inner, r, store):
    """A graph that uses every node type; `store` keeps (weight, gradient) matrices."""
    up = lambda *s: eng.upload((r.standard_normal(s) * 0.5).astype(dt))  # noqa: E731

    def weight(*s):
        m, d = up(*s), eng.zeros(s, dt)
        store.append(d)
        return g.weight(m, d)

    x = g.input(up(rows, inner))
    h = g.node("MatrixMultiplyOperation", [x, weight(inner, cols)])
    h = g.node("MatrixAddBroadcastingOperation", [h, weight(1, cols)])
    parts = []
    for op in ("LeakyReLUOperation", "SigmoidOperation", "TanhOperation", "GELUOperation", "ReLUOperation", "AmplifiedSigmoidOperation",
               "SoftmaxOperation", "LayerNormalizationOperation", "SineSoftmaxOperation"):
        parts.append(g.node(op, [h], scalar=0.01))
    had = g.node("HadamardProductOperation", [parts[0], parts[1]])
    s3 = g.node("MatrixAddThreeOperation", [had, parts[2], parts[3]])
    s3 = g.node("MatrixAddOperation", [s3, parts[4]])
    s3 = g.node("MatrixMultiplyScalarOperation", [s3], scalar=0.7)
    for p in parts[5:]:
        s3 = g.node("MatrixAddOperation", [s3, p])
    t = g.node("MatrixTransposeOperation", [s3])
    q = g.node("MatrixMultiplyOperation", [t, s3])               # cols x cols
    w = weight(cols, cols)
    outs = [g.node("MatrixMultiplyOperation", [q, w]), g.node("HadamardProductOperation", [q, w])]
    return g.node("MatrixAddOperation", outs), outs[0]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows,cols,inner", [(1, 1, 1), (3, 5, 2), (16, 16, 300), (17, 31, 9), (64, 8, 64), (65, 33, 40), (100, 1, 7)])
def test_plan_equals_separate_launches(engine, dtype, rows, cols, inner):
    results = []
    for plan in ("1", "0"):
        r = rng(rows * 10 + cols)
        engine.set_option("graph_plan", plan)
        try:
            store = []
            g = Graph(engine, dtype)
            end, mid = _network(g, engine, dtype, rows, cols, inner, r, store)
            d = engine.upload(r.standard_normal((cols, cols)).astype(dtype))
            got, launches = [], []
            for _ in range(2):                        # the second pass adds to the destinations
                n0 = engine.launch_count()
                g.forward()
                g.backward(end, d)
                launches.append(engine.launch_count() - n0)
                got += [g.data(end).numpy(), g.gradient(mid).numpy()] + [s.numpy() for s in store]
            assert g.consumers(mid) == 1
            results.append((got, launches))
            g.close()
        finally:
            engine.set_option("graph_plan", "1")
    (a, la), (b, lb) = results
    assert la == [2, 2] and lb[0] > 40
    tol = dict(rtol=1e-12, atol=1e-12) if dtype == np.float64 else dict(rtol=1e-5, atol=1e-5)   # (row and column sums)
    for x, y in zip(a, b):
        np.testing.assert_allclose(x, y, **tol)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_products_sums_and_elementwise_chains_are_the_same_bits(engine, dtype):
    """Shared weights over many uses (fan-in and += chains longer than eight), one flat gradient buffer, changing start gradients."""
    n, uses = 37, 11
    results = []
    for plan in ("1", "0"):
        r = rng(3)
        engine.set_option("graph_plan", plan)
        try:
            flat = engine.zeros((2 * n * n,), dtype)
            wm = engine.upload((r.standard_normal((n, n)) * 0.3).astype(dtype))
            g = Graph(engine, dtype)
            h = x = g.input(engine.upload(r.standard_normal((n, n)).astype(dtype)))
            hs = []
            for k in range(uses):
                w = g.weight(wm, flat.view((n, n), (k % 2) * n * n))
                h = g.node("TanhOperation", [g.node("MatrixMultiplyOperation", [w, h])])
                hs.append(g.node("HadamardProductOperation", [h, x]))
            total = hs[0]
            for k in hs[1:]:
                total = g.node("MatrixAddOperation", [total, k])
            starts = [engine.upload(r.standard_normal((n, n)).astype(dtype)) for _ in range(6)]
            got = []
            for d in starts + starts[:2]:
                g.forward()
                g.backward(total, d)
                got += [g.data(total).numpy(), g.gradient(x).numpy(), flat.numpy()]
            results.append(got)
            g.close()
        finally:
            engine.set_option("graph_plan", "1")
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_a_recorded_walk_survives_the_growth_of_its_graph(engine, dtype):
    """A recording of the forward keeps running the plan it was made with after nodes were added and the graph planned anew."""
    n, r = 24, rng(8)
    x = engine.upload(r.standard_normal((n, n)).astype(dtype))
    g = Graph(engine, dtype)
    w, h = g.input(engine.upload((r.standard_normal((n, n)) * 0.3).astype(dtype))), g.input(x)

    def layer(h):
        m = g.node("MatrixMultiplyOperation", [w, h])
        return g.node("MatrixAddOperation", [h, g.node("HadamardProductOperation", [g.node("TanhOperation", [m]), g.node("SigmoidOperation", [m])])])

    for _ in range(6):
        h = layer(h)
    g.forward()
    seq = engine.record(g.forward)
    assert seq.launches == 1
    end = h
    for _ in range(4):
        h = layer(h)
        g.forward()
    junk = [engine.zeros((n, n), dtype) for _ in range(64)]            # whatever was freed is in use again
    want = []
    for k in range(3):
        engine.upload((rng(20 + k).standard_normal((n, n))).astype(dtype), out=x)
        g.forward()
        want.append((g.data(end).numpy(), g.data(h).numpy()))
    for k in range(3):
        engine.upload((rng(20 + k).standard_normal((n, n))).astype(dtype), out=x)
        seq.launch()
        np.testing.assert_array_equal(g.data(end).numpy(), want[k][0])
        np.testing.assert_array_equal(g.data(h).numpy(), want[-1][1])  # the new nodes are not part of the recording
    assert not any(m.numpy().any() for m in junk)
    seq.close()
    g.close()


def _backward_from(g, starts, gradients):
    E.check(g.eng.lib.prad_graph_backward_multi(g.h, (C.c_int * len(starts))(*starts), E.Engine._ptr_list(gradients), len(starts)))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_one_plan_serves_every_start_gradient(engine, dtype):
    """A program gets new loss gradients from every pass: the plan of the first pass runs them too, and says whose gradient is whose."""
    n, steps = 24, 5
    r = rng(5)
    up = lambda: engine.upload((r.standard_normal((n, n)) * 0.3).astype(dtype))  # noqa: E731
    g = Graph(engine, dtype)
    dw = engine.zeros((n, n), dtype)
    w, h = g.weight(up(), dw), g.input(up())
    starts = []
    for _ in range(steps):
        h = g.node("TanhOperation", [g.node("MatrixMultiplyOperation", [w, h])])
        starts.append(g.node("MatrixAddOperation", [h, g.node("MatrixTransposeOperation", [h])]))
    g.forward()
    sets = [[up() for _ in starts] for _ in range(7)]
    sets.append([sets[0][0]] * steps)                        # one gradient for all
    flat = engine.upload(r.standard_normal((steps * n * n + 1,)).astype(dtype))
    sets.append([flat.view((n, n), 1 + k * n * n) for k in range(steps)])      # off a 16-byte boundary
    sets.append([flat.view((n, n), k * 3 * n) for k in range(steps)])         # overlapping
    want = []
    for d in sets:
        engine.set_option("graph_plan", "0")
        try:
            engine.zero_(dw)
            _backward_from(g, starts, d)
            want.append([g.gradient(h).numpy(), g.gradient(starts[0]).numpy(), dw.numpy()])
        finally:
            engine.set_option("graph_plan", "1")
    _backward_from(g, starts, sets[0])
    for d, expected in zip(sets, want):
        for recorded in (True, False):                       # a recording uses a plan that is there, but cannot make one
            engine.zero_(dw)
            if recorded:
                seq = engine.record(lambda: _backward_from(g, starts, d))
                assert seq.launches == 1
                seq.launch()
            else:
                n0 = engine.launch_count()
                _backward_from(g, starts, d)
                assert engine.launch_count() - n0 == 1
            for a, b in zip([g.gradient(h).numpy(), g.gradient(starts[0]).numpy(), dw.numpy()], expected):
                np.testing.assert_array_equal(a, b)
            assert g.gradient(starts[0]).ptr == d[0].ptr     # nothing else flows into it
            if recorded:
                seq.close()
    g.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("starts", [3, 70])
def test_start_gradients_that_the_walk_itself_writes(engine, dtype, starts):
    """A start gradient in memory that Backward writes (a gradient destination, a gradient of the last pass) is read in turn; and
    more start values than fit the kernel's short table."""
    n = 8
    results = []
    for plan in ("1", "0"):
        r = rng(11)
        up = lambda: engine.upload((r.standard_normal((n, n)) * 0.3).astype(dtype))  # noqa: E731
        engine.set_option("graph_plan", plan)
        try:
            g = Graph(engine, dtype)
            dw = engine.zeros((n, n), dtype)
            w, x = g.weight(up(), dw), g.input(up())
            h, ends = x, []
            for _ in range(starts):
                h = g.node("SigmoidOperation", [g.node("MatrixMultiplyOperation", [w, h])])
                ends.append(g.node("MatrixAddOperation", [g.node("MatrixMultiplyScalarOperation", [h], scalar=0.5), h]))
            g.forward()
            d = [up() for _ in ends]
            got = []
            n0 = engine.launch_count()
            _backward_from(g, ends, d)
            if plan == "1":
                assert engine.launch_count() - n0 == 1
            got += [dw.numpy(), g.gradient(x).numpy()]
            for last in (dw, g.gradient(x), g.gradient(w), g.gradient(ends[0])):
                _backward_from(g, ends, d[:-1] + [last])
                got += [dw.numpy(), g.gradient(x).numpy()]
            results.append(got)
            g.close()
        finally:
            engine.set_option("graph_plan", "1")
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)


def test_plans_of_many_sets_of_start_values(engine):
    """Sets of start values beyond those whose plans are kept run one launch per operation; the kept ones stay."""
    n, r = 8, rng(12)
    up = lambda: engine.upload((r.standard_normal((n, n)) * 0.3).astype(np.float32))  # noqa: E731
    g = Graph(engine, np.float32)
    w, h = g.input(up()), g.input(up())
    for _ in range(6):
        h = g.node("SigmoidOperation", [g.node("MatrixMultiplyOperation", [w, h])])
    ends = [g.node("TanhOperation", [h]) for _ in range(20)]
    g.forward()
    d = up()
    launches = []
    for _ in range(3):
        for end in ends:
            n0 = engine.launch_count()
            g.backward(end, d)
            launches.append(engine.launch_count() - n0)
    assert launches[:16] == [1] * 16 and min(launches[16:20]) > 6
    assert launches[20:40] == launches[:20] == launches[40:]
    g.close()


# units, columns, inputs, steps, and how many of a step's three products (of the inputs, twice of the state) the forward program takes
# along, in double and in float
FUSED = [(5, 1, 3, 2, 3, 3), (13, 7, 9, 3, 3, 3), (16, 8, 64, 6, 3, 3), (64, 8, 65, 2, 3, 3), (96, 4, 96, 7, 3, 3), (24, 21, 12, 4, 3, 3),
         (16, 32, 7, 3, 3, 3), (15, 33, 7, 3, 0, 0),              # columns: the last that fit, the first that do not
         (64, 32, 33, 2, 3, 3), (65, 32, 7, 2, 0, 0),             # outputs
         (16, 32, 64, 2, 3, 3), (16, 32, 65, 2, 2, 3), (16, 32, 129, 2, 2, 2),      # the second operand
         (230, 2, 230, 2, 3, 3), (230, 2, 600, 2, 0, 3),          # k in two parts, in double and in float
         (220, 2, 230, 2, 0, 3), (400, 1, 500, 2, 0, 0)]          # two parts for too few pieces; many parts


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("units,cols,inner,steps,in_double,in_float", FUSED)
def test_products_inside_programs_are_the_same_bits(engine, dtype, units, cols, inner, steps, in_double, in_float):
    """Cells whose products are taken along by the programs that read them, forward and backward, and cells beyond every limit of
    that: column counts that divide a piece and that do not, more k than shared memory has room for, gradients of shared weights added
    up over the steps."""
    results, launches = [], []
    for plan in ("1", "0"):
        r = rng(units + cols + inner)
        up = lambda *s: engine.upload((r.standard_normal(s) * 0.4).astype(dtype))  # noqa: E731
        engine.set_option("graph_plan", plan)
        try:
            g = Graph(engine, dtype)
            grads, w = [], {}
            for name, shape in (("We", (units, inner)), ("Wa", (units, units)), ("Wb", (units, units)), ("b", (units, cols))):
                grads.append(engine.zeros(shape, dtype))
                w[name] = (up(*shape), grads[-1])
            h, outs = g.input(up(units, cols)), []
            for _ in range(steps):
                x = g.node("MatrixMultiplyOperation", [g.weight(*w["We"]), g.input(up(inner, cols))])
                a = g.node("MatrixAddThreeOperation", [x, g.node("MatrixMultiplyOperation", [g.weight(*w["Wa"]), h]), g.weight(*w["b"])])
                c = g.node("SigmoidOperation", [g.node("MatrixMultiplyOperation", [g.weight(*w["Wb"]), h])])
                h = g.node("HadamardProductOperation", [g.node("TanhOperation", [a]), c])
                outs.append(g.node("MatrixAddOperation", [h, x]))
            got = []
            for k in range(2):
                n0 = engine.launch_count()
                g.forward()
                launches.append(engine.launch_count() - n0)
                got += [g.data(o).numpy() for o in outs]
                g.backward(outs[-1 - k], up(units, cols))
                got += [d.numpy() for d in grads]
            results.append(got)
            forward, backward = g.plan_products()
            expected = in_double if dtype == np.float64 else in_float
            assert forward == (plan == "1") * steps * expected
            # (no plan for the backward of a weight beyond 65536 values)
            assert backward == 0 if plan == "0" or units * inner > 65536 else backward > 0 or expected < 3
            g.close()
        finally:
            engine.set_option("graph_plan", "1")
    assert launches[0] * 2 < launches[2] and launches[0] == launches[1] and launches[2] == launches[3] >= 8 * steps
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows,cols,depth", [(100, 100, 20), (128, 128, 20), (90, 100, 30), (128, 128, 40), (255, 257, 12)])
def test_long_elementwise_chains_on_all_SMs_are_the_same_bits(engine, dtype, rows, cols, depth):
    """More pieces a level than the cluster has workers, over several levels: from the best one on, a launch on all SMs each, also where
    the last level alone would gain nothing by that."""
    results = []
    for plan in ("1", "0"):
        r = rng(rows + depth)
        up = lambda: engine.upload((r.standard_normal((rows, cols)) * 0.3).astype(dtype))  # noqa: E731
        engine.set_option("graph_plan", plan)
        try:
            g = Graph(engine, dtype)
            dx = engine.zeros((rows, cols), dtype)
            h, x = g.input(up()), g.weight(up(), dx)
            for k in range(depth):
                h = g.node(("SigmoidOperation", "TanhOperation", "GELUOperation", "LeakyReLUOperation")[k % 4], [h], scalar=0.01)
                h = g.node("HadamardProductOperation" if k % 2 else "MatrixAddOperation", [h, x])
            got, d = [], up()
            for _ in range(2):
                g.forward()
                n0 = engine.launch_count()
                g.backward(h, d)
                launches = engine.launch_count() - n0
                assert launches > depth if plan == "0" else launches < 6
                got += [g.data(h).numpy(), dx.numpy()]
            results.append(got)
            g.close()
        finally:
            engine.set_option("graph_plan", "1")
    for a, b in zip(*results):
        np.testing.assert_array_equal(a, b)

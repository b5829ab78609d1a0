"""Performance cases: what a program built on this framework has it do, through its public entry points.

Seven kinds of work, over the sizes they are used at:

  node       one MatrixMultiplyOperation -> activation node, Forward and Backward, the unit every managed operation
             class calls.  "buffers": "kept" passes the output buffers of the last pass again (a program with a static
             schedule), "new" lets the library allocate them (a program that follows the managed contract, where every
             Forward and Backward returns new matrices)
  mlp        one training step of a feed-forward network with softmax + cross-entropy or MSE: forward, loss, backward,
             clip, Adam.  "how": "recorded" replays a recorded launch sequence, "host" takes a batch from page-locked host
             memory and returns the loss to the host, "calls" makes the calls one by one on device-resident batches
  wide       the same step for wide GELU layers without biases, the data-parallel benchmark network and the share of it
             that one of several GPUs holds
  lstm       forward and full backpropagation through time of an LSTM layer, sequences handed over as host arrays
  swin       forward and full backward of a windowed self-attention block
  graph      a network built from a JSON architecture (an LSTM unrolled over time steps and layers): forward, loss
             gradients, the visitor's backward from all time steps, clip + Adam
  embedding  gather of table rows and the ordered scatter of their gradients, with word-like (skewed) indices

Every state has an engine of the process in common (one context per GPU, as the managed library has it).
"""
import math

import numpy as np
import torch

from parallelreverseautodiff_b200 import engine as E
from parallelreverseautodiff_b200.architecture import ArchitectureGraph
from parallelreverseautodiff_b200.networks import FeedForwardNetwork, LstmNetwork, SwinBlock

ACTS = {"leaky_relu": E.ACT_LEAKY_RELU, "sigmoid": E.ACT_SIGMOID, "tanh": E.ACT_TANH, "gelu": E.ACT_GELU}
SAVES_OUTPUT = ("sigmoid", "tanh")      # activations whose Backward reads their output
NP = {"f32": np.float32, "f64": np.float64}
TORCH = {"f32": torch.float32, "f64": torch.float64}
SIZE = {"f32": 4, "f64": 8}
ALPHA = 0.01

_eng = None


def _engine():
    global _eng
    if _eng is None:
        _eng = E.Engine(0)
    return _eng


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call there is: a hidden layer of a toy network; launches and host code are all of it
        {"name": "node-f32-small", "kind": "node", "dtype": "f32", "act": "leaky_relu", "m": 24, "k": 40, "n": 16,
         "buffers": "kept"},
        # benchmark configuration 1
        {"name": "node-f64-512", "kind": "node", "dtype": "f64", "act": "leaky_relu", "m": 512, "k": 784, "n": 256,
         "buffers": "new"},
        # a layer large enough for the tensor cores, called operation by operation
        {"name": "node-f32-8192", "kind": "node", "dtype": "f32", "act": "gelu", "m": 8192, "k": 2048, "n": 1536,
         "buffers": "new"},
        # a large double product with a ragged edge
        {"name": "node-f64-2048", "kind": "node", "dtype": "f64", "act": "tanh", "m": 2048, "k": 1536, "n": 1000,
         "buffers": "kept"},
        # benchmark configuration 2, a training loop with a fixed batch size
        {"name": "mlp-f32-256", "kind": "mlp", "dtype": "f32", "act": "leaky_relu", "loss": "cce", "batch": 256, "n_in": 784,
         "hidden": 512, "layers": 3, "n_out": 10, "how": "recorded"},
        # the double library fed from the host, an odd batch and odd widths
        {"name": "mlp-f64-host", "kind": "mlp", "dtype": "f64", "act": "sigmoid", "loss": "mse", "batch": 100, "n_in": 61,
         "hidden": 133, "layers": 4, "n_out": 7, "how": "host"},
        # benchmark configuration 5 on one GPU, the largest case
        {"name": "wide-f32-65536", "kind": "wide", "rows": 65536, "width": 4096, "layers": 8},
        # benchmark configuration 3
        {"name": "lstm-f64-64", "kind": "lstm", "dtype": "f64", "steps": 64, "batch": 32, "n_in": 128, "hidden": 256},
        # a short sequence in float, odd sizes
        {"name": "lstm-f32-12", "kind": "lstm", "dtype": "f32", "steps": 12, "batch": 7, "n_in": 24, "hidden": 56},
        # benchmark configuration 4
        {"name": "swin-f32-64", "kind": "swin", "images": 64, "windows": 64, "window": 49, "dim": 96, "heads": 3},
        # a two-layer LSTM from a JSON architecture over eight time steps
        {"name": "graph-f64-8x2", "kind": "graph", "dtype": "f64", "steps": 8, "layers": 2, "n_in": 32, "hidden": 64,
         "n_out": 8, "columns": 8},
        # a vocabulary's table in a language model
        {"name": "embedding-f32-50000", "kind": "embedding", "dtype": "f32", "n": 16384, "vocab": 50000, "dim": 512},
    ]


def _spread(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("node", "node", "mlp", "wide", "lstm", "swin", "graph", "embedding"))
    dtype = rng.choice(("f32", "f64"))
    act = rng.choice(sorted(ACTS))
    if kind == "node":
        top = 8192 if dtype == "f32" else 2048
        m, k, n = _spread(rng, 16, top), _spread(rng, 16, 2048), _spread(rng, 16, 2048)
        return {"kind": "node", "dtype": dtype, "act": act, "m": m, "k": k, "n": n, "buffers": rng.choice(("kept", "new"))}
    if kind == "mlp":
        return {"kind": "mlp", "dtype": dtype, "act": act, "loss": rng.choice(("cce", "mse")), "batch": _spread(rng, 16, 1024),
                "n_in": _spread(rng, 16, 1024), "hidden": _spread(rng, 16, 1024), "layers": rng.randint(2, 5),
                "n_out": _spread(rng, 2, 64), "how": rng.choice(("recorded", "host", "calls"))}
    if kind == "wide":
        return {"kind": "wide", "rows": _spread(rng, 1024, 32768), "width": _spread(rng, 512, 4096), "layers": rng.randint(2, 8)}
    if kind == "lstm":
        return {"kind": "lstm", "dtype": dtype, "steps": _spread(rng, 4, 64), "batch": _spread(rng, 1, 64),
                "n_in": _spread(rng, 8, 256), "hidden": _spread(rng, 16, 256)}
    if kind == "swin":
        dim, heads = rng.choice(((64, 2), (96, 3), (128, 4)))
        return {"kind": "swin", "images": _spread(rng, 1, 48), "windows": rng.choice((16, 64)), "window": rng.choice((16, 36, 49)),
                "dim": dim, "heads": heads}
    if kind == "graph":
        return {"kind": "graph", "dtype": dtype, "steps": _spread(rng, 1, 12), "layers": rng.randint(1, 3), "n_in": _spread(rng, 4, 64),
                "hidden": _spread(rng, 8, 128), "n_out": _spread(rng, 1, 16), "columns": _spread(rng, 1, 32)}
    return {"kind": "embedding", "dtype": dtype, "n": _spread(rng, 64, 32768), "vocab": _spread(rng, 128, 50000),
            "dim": _spread(rng, 16, 1024)}


# ---------------------------------------------------------------- between torch and the library
class _Shown:
    """A device matrix under the CUDA array interface; keeps it alive, and the owner of its memory where it is a view."""

    def __init__(self, m, owner):
        self.m, self.owner = m, owner
        self.__cuda_array_interface__ = {"shape": m.shape, "typestr": m.dtype.str, "data": (m.ptr, False), "version": 3}


def _tensor(m, owner=None):
    return torch.as_tensor(_Shown(m, owner), device="cuda")


class _Inputs:
    """Random device matrices from one seed."""

    def __init__(self, seed, dtype):
        self.eng, self.dtype = _engine(), dtype
        self.g = torch.Generator(device="cuda").manual_seed(seed)

    def _matrix(self, t):
        out = self.eng.empty(tuple(t.shape), NP[self.dtype])
        torch.cuda.synchronize()
        self.eng.copy(out, E.DeviceMatrix(self.eng, t.data_ptr(), t.shape, NP[self.dtype], owned=False))
        self.eng.sync()
        return out

    def normal_t(self, *shape, scale=1.0):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=TORCH[self.dtype]) * scale

    def uniform_t(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.g, device="cuda", dtype=TORCH[self.dtype]) * (hi - lo) + lo

    def normal(self, *shape, scale=1.0):
        return self._matrix(self.normal_t(*shape, scale=scale))

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return self._matrix(self.uniform_t(*shape, lo=lo, hi=hi))

    def onehot_t(self, rows, cols):
        c = torch.randint(0, cols, (rows,), generator=self.g, device="cuda")
        return torch.nn.functional.one_hot(c, cols).to(TORCH[self.dtype]).contiguous()

    def matrix(self, t):
        return self._matrix(t)


def prepare(case, seed):
    return {"node": _Node, "mlp": _Mlp, "wide": _Wide, "lstm": _Lstm, "swin": _Swin, "graph": _Graph,
            "embedding": _Embedding}[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---------------------------------------------------------------- node
class _Node:
    def __init__(self, case, seed):
        r = _Inputs(seed, case["dtype"])
        self.e, m, k, n = r.eng, case["m"], case["k"], case["n"]
        self.act, self.saves_output, self.kept = ACTS[case["act"]], case["act"] in SAVES_OUTPUT, case["buffers"] == "kept"
        self.A, self.B = r.uniform(m, k, lo=-1.0), r.normal(k, n, scale=math.sqrt(2.0 / k))
        self.dOut = r.normal(m, n)
        dt = NP[case["dtype"]]
        self.Z = self.e.empty((m, n), dt)
        if self.kept:
            self.Y, self.dPre = self.e.empty((m, n), dt), self.e.empty((m, n), dt)
            self.dA, self.dB = self.e.empty((m, k), dt), self.e.empty((k, n), dt)
            self.out = [_tensor(x) for x in (self.Y, self.dPre, self.dA, self.dB)]

    def run(self):
        e = self.e
        if self.kept:
            e.matmul_forward(self.A, self.B, Y=self.Y, Z_out=self.Z, act=self.act, act_alpha=ALPHA)
            e.act_backward(self.act, self.Y if self.saves_output else self.Z, self.dOut, ALPHA, out=self.dPre)
            e.matmul_backward(self.A, self.B, self.dPre, dA=self.dA, dB=self.dB)
            return self.out
        y = e.matmul_forward(self.A, self.B, Z_out=self.Z, act=self.act, act_alpha=ALPHA)
        dPre, dA, dB = e.matmul_act_backward(self.A, self.B, self.dOut, self.act, y if self.saves_output else self.Z, ALPHA)
        return [_tensor(x) for x in (y, dPre, dA, dB)]


# ---------------------------------------------------------------- feed-forward networks
class _Mlp:
    def __init__(self, case, seed):
        r = _Inputs(seed, case["dtype"])
        e = self.e = r.eng
        sizes = [case["n_in"]] + [case["hidden"]] * (case["layers"] - 1) + [case["n_out"]]
        cce = case["loss"] == "cce"
        net = self.net = FeedForwardNetwork(e, NP[case["dtype"]], sizes, hidden_act=ACTS[case["act"]], softmax_output=cce,
                                            loss=case["loss"])
        net.set_weights([r.normal_t(a, b, scale=math.sqrt(2.0 / a)).cpu().numpy() for a, b in zip(sizes[:-1], sizes[1:])],
                        [r.normal_t(1, b, scale=0.1).cpu().numpy() for b in sizes[1:]])
        rows = case["batch"]
        x = r.uniform_t(rows, sizes[0])
        t = r.onehot_t(rows, sizes[-1]) if cce else r.normal_t(rows, sizes[-1])
        self.how = case["how"]
        if self.how == "host":
            self.x, self.t = e.pinned_empty((rows, sizes[0]), net.dtype), e.pinned_empty((rows, sizes[-1]), net.dtype)
            self.x[...], self.t[...] = x.cpu().numpy(), t.cpu().numpy()
        else:
            self.x, self.t = r.matrix(x), r.matrix(t)
        if self.how == "recorded":
            self._step()                 # a recording needs the library's scratch at its final size
            e.sync()
            self.sequence = e.record(self._step)
            self.dX = _tensor(net.dX, net)
        self.state = [_tensor(m) for m in net.params + net.m + net.v]
        self.loss = _tensor(net.loss_dev)

    def __del__(self):
        if self.how == "recorded":
            self.sequence.close()

    def _step(self):
        self.net.forward(self.x)
        self.net.loss_value(self.t)
        self.net.backward(self.t)
        self.net.clip_and_optimize()

    def run(self):
        if self.how == "host":
            return [self.net.train_step_host(self.x, self.t), _tensor(self.net.dX, self.net)] + self.state
        if self.how == "recorded":
            self.sequence.launch()
            return [self.loss, self.dX] + self.state
        self._step()
        return [self.loss, _tensor(self.net.dX, self.net)] + self.state


class _Wide:
    def __init__(self, case, seed):
        r = _Inputs(seed, "f32")
        rows, w, layers = case["rows"], case["width"], case["layers"]
        net = self.net = FeedForwardNetwork(r.eng, np.float32, [w] * (layers + 1), hidden_act=E.ACT_GELU, output_act=E.ACT_GELU,
                                            use_bias=False)
        net.Parameters.LearningRate = 1e-5       # 1e-3 makes deep GELU networks diverge on random targets
        net.set_weights([r.normal_t(w, w, scale=math.sqrt(2.0 / w)).cpu().numpy() for _ in range(layers)])
        self.x, self.t = r.normal(rows, w), r.normal(rows, w)
        self.state = [_tensor(m) for m in net.params + net.m + net.v]
        self.loss = _tensor(net.loss_dev)

    def run(self):
        net = self.net
        net.forward(self.x)
        net.loss_value(self.t)
        net.backward(self.t)
        net.clip_and_optimize()
        return [self.loss, _tensor(net.dX, net)] + self.state


# ---------------------------------------------------------------- LSTM
class _Lstm:
    def __init__(self, case, seed):
        r = _Inputs(seed, case["dtype"])
        steps, batch, n_in, nh = case["steps"], case["batch"], case["n_in"], case["hidden"]
        net = self.net = LstmNetwork(r.eng, NP[case["dtype"]], n_in, nh, steps, batch)
        xavier = lambda a, b: r.uniform_t(a, b, lo=-1.0, hi=1.0).cpu().numpy() * math.sqrt(6.0 / (a + b))  # noqa: E731
        net.set_parameters({g: xavier(nh, n_in) for g in net.GATES}, {g: xavier(nh, nh) for g in net.GATES},
                           {g: r.normal_t(nh, scale=0.1).cpu().numpy() for g in net.GATES})
        self.x, self.y = (r.normal_t(steps, batch, n).cpu().numpy() for n in (n_in, nh))
        self.out = [_tensor(m, net) for m in [net.H, net.dX] + [d[g] for d in (net.dW, net.dU, net.db) for g in net.GATES]]

    def run(self):
        self.net.forward(self.x, self.y)
        self.net.backward()
        return self.out


# ---------------------------------------------------------------- windowed self-attention block
class _Swin:
    def __init__(self, case, seed):
        r = _Inputs(seed, "f32")
        d, tokens = case["dim"], case["images"] * case["windows"] * case["window"]
        blk = self.blk = SwinBlock(r.eng, np.float32, d, case["heads"], case["window"])
        he = lambda a, b: r.normal_t(a, b, scale=math.sqrt(2.0 / a)).cpu().numpy()  # noqa: E731
        bias = lambda n: r.normal_t(1, n, scale=0.1).cpu().numpy()  # noqa: E731
        blk.set_parameters({"Wqkv": he(d, 3 * d), "bqkv": bias(3 * d), "Wproj": he(d, d), "bproj": bias(d),
                            "W1": he(d, 4 * d), "b1": bias(4 * d), "W2": he(4 * d, d), "b2": bias(d)})
        self.x, self.d_out = r.normal(tokens, d), r.normal(tokens, d)
        self.grads = [_tensor(blk.g[k]) for k in sorted(blk.g)]

    def run(self):
        out = self.blk.forward(self.x)
        d_x = self.blk.backward(self.d_out)
        return [_tensor(out), _tensor(d_x)] + self.grads


# ---------------------------------------------------------------- JSON architecture
def _architecture():
    """An LSTM over column vectors (one column per sample): an input embedding per time step, the gates of every layer,
    an output projection per time step."""
    op = lambda id_, type_, inputs, grads=None: dict(  # noqa: E731
        {"id": id_, "type": type_, "inputs": inputs}, **({"gradientResultTo": grads} if grads else {}))
    mm, add = "MatrixMultiplyOperation", "MatrixAddOperation"
    start = [op("projectedInput", mm, ["We", "Input[t]"], ["DWe", None]),
             op("embeddedInput", add, ["projectedInput", "be"], [None, "Dbe"])]
    cell = []
    for g, act in (("f", "SigmoidOperation"), ("i", "SigmoidOperation"), ("c", "TanhOperation"), ("o", "SigmoidOperation")):
        cell += [op("w" + g, mm, [f"W{g}[layerIndex]", "currentInput"], [f"DW{g}[layerIndex]", None]),
                 op("u" + g, mm, [f"U{g}[layerIndex]", "previousHiddenState"], [f"DU{g}[layerIndex]", None]),
                 op(g + "Sum", "MatrixAddThreeOperation", ["w" + g, "u" + g, f"b{g}[layerIndex]"], [None, None, f"Db{g}[layerIndex]"]),
                 op(g + "Gate", act, [g + "Sum"])]
    cell += [op("kept", "HadamardProductOperation", ["fGate", "previousMemoryCellState"]),
             op("written", "HadamardProductOperation", ["iGate", "cGate"]),
             op("newC", add, ["kept", "written"]),
             op("cTanh", "TanhOperation", ["newC"]),
             op("newH", "HadamardProductOperation", ["oGate", "cTanh"])]
    end = [op("projectedOutput", mm, ["V", "lastHiddenState"], ["DV", None]),
           dict(op("output", add, ["projectedOutput", "bv"], [None, "Dbv"]), setResultTo="Output[t]")]
    return {"timeSteps": [{"startOperations": start, "layers": [{"operations": cell}], "endOperations": end}]}


class _Graph:
    def __init__(self, case, seed):
        r = _Inputs(seed, case["dtype"])
        e, dt = r.eng, NP[case["dtype"]]
        self.e, T, L, cols = e, case["steps"], case["layers"], case["columns"]
        n_in, nh, n_out = case["n_in"], case["hidden"], case["n_out"]
        shapes = {"We": (nh, n_in), "be": (nh, cols), "V": (n_out, nh), "bv": (n_out, cols)}
        layer_shapes = {w + g: (nh, cols) if w == "b" else (nh, nh) for g in "fico" for w in "WUb"}
        names = list(shapes) + [(l, k) for l in range(L) for k in layer_shapes]
        all_shapes = list(shapes.values()) + list(layer_shapes.values()) * L
        offsets, total = [], 0
        for a, b in all_shapes:              # one buffer for all parameters, every matrix at a 256-byte boundary
            offsets.append(total)
            total += -(-a * b // 64) * 64
        flat = [e.zeros((1, total), dt) for _ in range(4)]
        self.w, self.dw, self.m, self.v = ([f.view(s, o) for s, o in zip(all_shapes, offsets)] for f in flat)
        for (a, b), m, k in zip(all_shapes, self.w, names):
            scale = 0.1 if "b" in str(k) else 1 / math.sqrt(b)
            e.copy(m, r.normal(a, b, scale=scale))
        e.sync()
        p, d = dict(zip(names, self.w)), dict(zip(names, self.dw))
        x = [r.normal(n_in, cols) for _ in range(T)]
        self.target = [r.normal(n_out, cols) for _ in range(T)]
        h0, c0 = e.zeros((nh, cols), dt), e.zeros((nh, cols), dt)
        graph = self.graph = ArchitectureGraph(e, dt)
        for k in shapes:
            graph.AddWeight(k, lambda li, k=k: p[k]).AddGradient("D" + k, lambda li, k=k: d[k])
        for k in layer_shapes:
            graph.AddWeight(k, lambda li, k=k: p[li.Layer, k]).AddGradient("D" + k, lambda li, k=k: d[li.Layer, k])
        y = self.y = [e.empty((n_out, cols), dt) for _ in range(T)]
        graph.AddIntermediate("Input", lambda li: x[li.TimeStep]).AddIntermediate("Output", lambda li: y[li.TimeStep])
        graph.AddOperationFinder("currentInput", lambda li: graph[f"embeddedInput_{li.TimeStep}_0"] if li.Layer == 0
                                 else graph[f"newH_{li.TimeStep}_{li.Layer - 1}"])
        graph.AddOperationFinder("previousHiddenState", lambda li: h0 if li.TimeStep == 0 else graph[f"newH_{li.TimeStep - 1}_{li.Layer}"])
        graph.AddOperationFinder("previousMemoryCellState",
                                 lambda li: c0 if li.TimeStep == 0 else graph[f"newC_{li.TimeStep - 1}_{li.Layer}"])
        graph.AddOperationFinder("lastHiddenState", lambda li: graph[f"newH_{li.TimeStep}_{L - 1}"])
        graph.ConstructFromArchitecture(_architecture(), L, T)
        self.starts = [f"output_{t}_0" for t in range(T)]
        self.dy = [e.empty((n_out, cols), dt) for _ in range(T)]
        self.out = [_tensor(y) for y in self.y] + [_tensor(f) for f in flat]

    def __del__(self):
        self.graph.close()

    def run(self):
        e = self.e
        self.graph.forward()                 # and the copies of the outputs into self.y
        for y, t, dy in zip(self.y, self.target, self.dy):
            e.mse_backward(y, t, grad=dy)
        self.graph.backward(self.starts, self.dy)
        e.clip_adam(self.w, self.dw, self.m, self.v, E.CLIP_REFERENCE, 4.0, 1e-8, 1e-3, 0.9, 0.999, 1e-8, 1.0, zero_grad=True)
        return self.out


# ---------------------------------------------------------------- embedding
class _Embedding:
    def __init__(self, case, seed):
        r = _Inputs(seed, case["dtype"])
        self.e, n, self.vocab, dim = r.eng, case["n"], case["vocab"], case["dim"]
        # the k-th commonest word appears about 1 / k as often as the commonest; ids are spread over the table
        rank = torch.exp(r.uniform_t(n, 1).double() * math.log(self.vocab + 1)).long().clamp(1, self.vocab) - 1
        place = torch.randperm(self.vocab, generator=r.g, device="cuda")
        self.idx = r.matrix(place[rank].to(TORCH[case["dtype"]]).contiguous())
        self.W, self.dOut = r.normal(self.vocab, dim, scale=0.02), r.normal(n, dim)

    def run(self):
        y = self.e.embedding_forward(self.idx, self.W)
        dW = self.e.embedding_backward(self.idx, self.dOut, self.vocab)
        return [_tensor(y), _tensor(dW)]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Inputs read once, outputs and updated state written once; multiply-adds of the products, forward and backward."""
    kind = case["kind"]
    if kind == "node":
        m, k, n, s = case["m"], case["k"], case["n"], SIZE[case["dtype"]]
        return {"bytes": s * (2 * m * k + 2 * k * n + 4 * m * n), "flops": 6 * m * k * n}
    if kind in ("mlp", "wide"):
        if kind == "mlp":
            sizes = [case["n_in"]] + [case["hidden"]] * (case["layers"] - 1) + [case["n_out"]]
            rows, s, bias = case["batch"], SIZE[case["dtype"]], 1
        else:
            sizes, rows, s, bias = [case["width"]] * (case["layers"] + 1), case["rows"], 4, 0
        params = sum((a + bias) * b for a, b in zip(sizes[:-1], sizes[1:]))
        return {"bytes": s * (6 * params + rows * (2 * sizes[0] + sizes[-1])),
                "flops": sum(6 * rows * a * b for a, b in zip(sizes[:-1], sizes[1:]))}
    if kind == "lstm":
        tb, n_in, nh, s = case["steps"] * case["batch"], case["n_in"], case["hidden"], SIZE[case["dtype"]]
        params = 4 * nh * (n_in + nh + 1)
        return {"bytes": s * (2 * params + tb * (2 * n_in + 2 * nh)), "flops": 6 * tb * 4 * nh * (n_in + nh)}
    if kind == "swin":
        d, ws = case["dim"], case["window"]
        t = case["images"] * case["windows"] * ws
        params = d * 3 * d + d * d + 2 * d * 4 * d + 9 * d
        return {"bytes": 4 * (4 * t * d + 2 * params), "flops": 6 * t * (12 * d * d + 2 * ws * d)}
    if kind == "graph":
        T, L, nh, cols, s = case["steps"], case["layers"], case["hidden"], case["columns"], SIZE[case["dtype"]]
        params = nh * case["n_in"] + nh * cols + case["n_out"] * (nh + cols) + L * 4 * nh * (2 * nh + cols)
        macs = T * cols * (nh * case["n_in"] + L * 8 * nh * nh + case["n_out"] * nh)
        return {"bytes": s * (6 * params + T * cols * (case["n_in"] + 2 * case["n_out"])), "flops": 6 * macs}
    n, vocab, dim, s = case["n"], case["vocab"], case["dim"], SIZE[case["dtype"]]
    return {"bytes": s * (2 * n + 3 * n * dim + vocab * dim), "flops": n * dim}


def tolerance(case):
    """Sums of the data type taken in another order.  Adam divides a gradient by its own size, so a weight whose gradient is
    rounding alone may move by a learning rate either way: single values of a training step can differ by more."""
    kind = case["kind"]
    f64 = case.get("dtype") == "f64"
    if kind == "embedding":
        return "exact"                       # rows copied, and gradients added in the order of the input
    if kind in ("mlp", "wide", "graph"):
        return {"rel": 1e-11, "max": 0.1} if f64 else {"rel": 1e-4, "max": 0.1}
    if kind == "node":
        return {"rel": 1e-13, "max": 1e-11} if f64 else {"rel": 1e-5, "max": 1e-4}
    return {"rel": 1e-11} if f64 else {"rel": 5e-5}

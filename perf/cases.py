"""What a user of this library has it do, as cases that can be timed and compared.

A case is a dict of plain values. `listed()` gives the standing ones, `draw(rng)` another one of the same
ranges, `prepare(case, seed)` what a program has in hand before the call, `run(state)` one pass through the
public entry points, `work(case)` the bytes and operations that pass cannot do without and
`tolerance(case)` how far another correct implementation may be from it.

Kinds: products (`dot`, `batched_dot`), a fully-connected layer, one convolution, an Inception module, a
pooling layer, fused element-wise expressions, and whole training steps of the AlexNet and VGG model A
convolution stacks. Activations are (C, D, H, W, N), filters (C, T, R, S, K), as everywhere in the library.
"""
import math

import numpy as np
import torch

from nervanagpu_b200 import NervanaGPU
from nervanagpu_b200.convnet import NETWORKS, ConvStack
from nervanagpu_b200.layers import ConvLayer, DataLayer, FullLayer, Inception, Layer, PoolLayer
from nervanagpu_b200.nervanagpu import GPUTensor

_NP = {"f16": np.float16, "f32": np.float32}
_TORCH = {"f16": torch.float16, "f32": torch.float32}
_BYTES = {"f16": 2, "f32": 4}
# small enough that thousands of passes on one state leave the values as they are in use
_LEARNING_RATE = {"fc": -1e-6, "inception": -1e-7, "stack": -1e-8}


# ---- the cases -------------------------------------------------------------------------------------
def listed():
    return [
        # a product of a small model: one launch, all latency
        dict(name="dot_small", kind="dot", op="nn", m=128, n=128, k=128, relu=False, beta=0.0, sr=0),
        # a large square product, rounded stochastically, as in training with fp16 weights
        dict(name="dot_square_3072", kind="dot", op="tn", m=3072, n=3072, k=3072, relu=True, beta=0.0, sr=10),
        # odd sizes everywhere: 1001 classes, a last minibatch of 125, 4096 features and a bias
        dict(name="dot_ragged", kind="dot", op="nn", m=1001, n=125, k=4097, relu=False, beta=0.0, sr=0),
        # AlexNet's first fully-connected layer in training: forward, deltas, weight gradient, descent
        dict(name="fc_layer", kind="fc", nin=9216, nout=4096, n=128),
        # a recurrent layer over 32 time steps: shared weights forward, gradient summed over the steps
        dict(name="batched_dot", kind="batched", batch=32, m=512, n=128, k=512),
        # a video layer: 3x3x3, 64 -> 64 feature maps over 16 frames of 56x56, all three passes
        dict(name="conv_3d", kind="conv", N=32, C=64, K=64, D=16, H=56, W=56, T=3, R=3, S=3,
             pad_d=1, pad=1, str_d=1, stride=1),
        # GoogLeNet's first module, forward and backward: small 1x1, 3x3 and 5x5 layers, padded pooling
        dict(name="inception_module", kind="inception", N=128, C=192, H=28, n1=64, r3=96, n3=128, r5=16, n5=32, proj=32),
        # whole training steps: recorded once and replayed, as a training loop runs them
        dict(name="alexnet_step_128", kind="stack", net="alexnet", N=128, recorded=True),
        dict(name="vgg_a_step_64", kind="stack", net="vgg_a", N=64, recorded=True),
        # the shard of an AlexNet minibatch over 8 GPUs, each kernel launched from Python
        dict(name="alexnet_step_16_live", kind="stack", net="alexnet", N=16, recorded=False),
        # pooling over feature maps, frames and pixels at once, forward and backward
        dict(name="pool_4d", kind="pool", op="max", dtype="f16", N=32, C=64, D=16, H=56, W=56, J=2, T=2, R=2, S=2,
             pad=0, str_j=2, str_d=2, stride=2),
        # batch normalisation of a hidden layer as one expression: one short launch
        dict(name="batch_norm_4096x128", kind="ew", expr="batch_norm", dtype="f16", rows=4096, cols=128),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` from lo to hi, spread over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step)))
    return max(lo, min(hi, int(v) // step * step))


def _draw_conv(rng):
    while True:
        R = rng.choice([1, 1, 3, 3, 3, 5, 7])
        H = _log(rng, max(R, 7), 112)
        c = dict(kind="conv", N=_log(rng, 16, 128, 8), C=rng.choice([3, _log(rng, 16, 512), _log(rng, 16, 512, 16)]),
                 K=_log(rng, 16, 512, 8), D=1, H=H, W=H, T=1, R=R, S=R, pad_d=0, pad=R // 2, str_d=1,
                 stride=rng.choice([1, 1, 1, 2]))
        w = work(c)
        if 1e8 < w["flops"] < (4e11 if c["stride"] == 1 else 4e10) and w["bytes"] < 1.2e9:
            return c


def _draw_pool(rng):
    R, stride, pad = rng.choice([(3, 2, 0), (2, 2, 0), (3, 1, 1), (3, 3, 0)])
    H = _log(rng, 7, 112)
    return dict(kind="pool", op=rng.choice(["max", "max", "max", "avg"]), dtype=rng.choice(["f16", "f16", "f32"]),
                N=_log(rng, 16, 128, 8), C=_log(rng, 16, 128), D=1, H=H, W=H, J=1, T=1, R=R, S=R, pad=pad,
                str_j=1, str_d=1, stride=stride)


def _draw_ew(rng):
    expr, dtype = rng.choice(["batch_norm", "softmax", "momentum"]), rng.choice(["f16", "f16", "f32"])
    if expr == "batch_norm":        # one row per unit or per pixel of a feature map, one column per image
        return dict(kind="ew", expr=expr, dtype=dtype, rows=_log(rng, 64, 500000), cols=_log(rng, 16, 256))
    if expr == "softmax":           # classes down the columns
        return dict(kind="ew", expr=expr, dtype=dtype, rows=_log(rng, 10, 4096), cols=_log(rng, 8, 512))
    return dict(kind="ew", expr=expr, dtype=dtype, rows=_log(rng, 64, 8192), cols=_log(rng, 64, 8192))


def draw(rng):
    kind = rng.choice(["dot", "ragged", "fc", "batched", "conv", "conv", "inception", "stack", "pool", "ew", "ew"])
    if kind in ("dot", "ragged"):
        step = 8 if kind == "dot" else 1
        return dict(kind="dot", op=rng.choice(["nn", "nt", "tn"]), m=_log(rng, 16, 4096 if step == 8 else 2048, step),
                    n=_log(rng, 16, 4096 if step == 8 else 512, step), k=_log(rng, 16, 8192 if step == 8 else 4096, step),
                    relu=rng.random() < 0.5, beta=rng.choice([0.0, 0.0, 1.0]), sr=rng.choice([0, 0, 10]))
    if kind == "fc":
        return dict(kind="fc", nin=_log(rng, 256, 9216, 8), nout=_log(rng, 128, 4096, 8), n=_log(rng, 16, 256, 8))
    if kind == "batched":
        return dict(kind="batched", batch=_log(rng, 2, 64), m=_log(rng, 32, 1024, 8), n=_log(rng, 16, 256, 8),
                    k=_log(rng, 32, 1024, 8))
    if kind == "conv":
        return _draw_conv(rng)
    if kind == "inception":
        return dict(kind="inception", N=_log(rng, 16, 128, 16), C=_log(rng, 128, 512, 16), H=rng.choice([7, 14, 28]),
                    n1=_log(rng, 64, 256, 8), r3=_log(rng, 64, 160, 8), n3=_log(rng, 96, 320, 8), r5=_log(rng, 16, 48, 8),
                    n5=_log(rng, 32, 128, 8), proj=_log(rng, 32, 128, 8))
    if kind == "stack":
        net = rng.choice(["alexnet", "alexnet", "vgg_a"])
        return dict(kind="stack", net=net, N=_log(rng, 8, 120 if net == "alexnet" else 56, 8), recorded=rng.random() < 0.5)
    return _draw_pool(rng) if kind == "pool" else _draw_ew(rng)


# ---- what a pass needs -----------------------------------------------------------------------------
def _out(x, f, pad, stride):
    return -((f - x - 2 * pad - 1) // stride) if stride > 1 else x - f + 1 + 2 * pad


def _conv_sizes(c):
    """Elements of the input, the filters and the output, and operations of one pass."""
    pix = _out(c["D"], c["T"], c["pad_d"], c["str_d"]) * _out(c["H"], c["R"], c["pad"], c["stride"]) \
        * _out(c["W"], c["S"], c["pad"], c["stride"])
    taps = c["T"] * c["R"] * c["S"]
    return (c["C"] * c["D"] * c["H"] * c["W"] * c["N"], c["C"] * taps * c["K"], c["K"] * pix * c["N"],
            2.0 * c["N"] * c["K"] * pix * c["C"] * taps)


def _plain_conv(N, C, K, H, R, pad, stride):
    return dict(N=N, C=C, K=K, D=1, H=H, W=H, T=1, R=R, S=R, pad_d=0, pad=pad, str_d=1, stride=stride)


def work(case):
    c = case
    kind = c["kind"]
    if kind == "dot":
        size = c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"] * (2 if c["beta"] else 1)
        return {"bytes": 2.0 * size, "flops": 2.0 * c["m"] * c["n"] * c["k"]}
    if kind == "fc":
        # weights read, written back and their gradient written; input, output, deltas in and out
        w = c["nin"] * c["nout"]
        return {"bytes": 2.0 * (3 * w + 2 * c["n"] * (c["nin"] + c["nout"])), "flops": 6.0 * w * c["n"]}
    if kind == "batched":
        b, m, n, k = (c[x] for x in ("batch", "m", "n", "k"))
        return {"bytes": 2.0 * (2 * m * k + b * (k * n + 2 * m * n)), "flops": 4.0 * b * m * n * k}
    if kind == "conv":
        i, f, o, flops = _conv_sizes(c)
        return {"bytes": 2.0 * (2 * i + f + 2 * o) + 4.0 * f, "flops": 3 * flops}
    if kind == "inception":
        N, C, H = c["N"], c["C"], c["H"]
        convs = [(C, c["n1"], 1), (C, c["r3"], 1), (c["r3"], c["n3"], 3), (C, c["r5"], 1), (c["r5"], c["n5"], 5), (C, c["proj"], 1)]
        flops = weights = 0.0
        for cin, cout, r in convs:
            _, f, _, fl = _conv_sizes(_plain_conv(N, cin, cout, H, r, r // 2, 1))
            flops += 3 * fl
            weights += f
        K = c["n1"] + c["n3"] + c["n5"] + c["proj"]
        return {"bytes": 2.0 * N * H * H * (2 * C + 2 * K) + 8.0 * weights, "flops": flops}
    if kind == "stack":
        net = NETWORKS[c["net"]]
        C, H = net["C"], net["H"]
        flops, size = 0.0, 2.0 * C * H * H * c["N"]
        for i, (what, p) in enumerate(net["layers"]):
            if what == "conv":
                K, R, _, pad, stride = p
                _, f, o, fl = _conv_sizes(_plain_conv(c["N"], C, K, H, R, pad, stride))
                flops += fl * (3 if i else 2)
                size += 8.0 * f + 4.0 * o       # weights in and out, fp32 gradient; activations written and read again
                C, H = K, _out(H, R, pad, stride)
            else:
                H = _out(H, p[0], 0, p[2])
        return {"bytes": size, "flops": flops}
    if kind == "pool":
        i = c["C"] * c["D"] * c["H"] * c["W"] * c["N"]
        o = c["N"] * _out(c["C"], c["J"], 0, c["str_j"]) * _out(c["D"], c["T"], 0, c["str_d"]) \
            * _out(c["H"], c["R"], c["pad"], c["stride"]) * _out(c["W"], c["S"], c["pad"], c["stride"])
        return {"bytes": 2.0 * _BYTES[c["dtype"]] * (i + o), "flops": 1.0 * c["J"] * c["T"] * c["R"] * c["S"] * o}
    size = c["rows"] * c["cols"]
    esz = _BYTES[c["dtype"]]
    if c["expr"] == "momentum":                 # weights and velocity read and written, fp32 gradient read
        return {"bytes": size * (4.0 * esz + 4.0), "flops": 6.0 * size}
    return {"bytes": 2.0 * esz * size, "flops": 6.0 * size}


def tolerance(case):
    """Results are rounded to fp16 once (a relative error of 2^-11 at most, 2^-10 when stochastically) over fp32
    sums; chains round at every layer. Max-pooling picks values and adds a window's few errors in one order."""
    kind = case["kind"]
    if kind == "pool":
        return "exact" if case["op"] == "max" else {"rel": 1e-5 if case["dtype"] == "f32" else 1e-3}
    if kind == "ew":
        return {"rel": 1e-5 if case["dtype"] == "f32" else 1e-3}
    if kind == "stack":
        return {"rel": 3e-3}
    if kind in ("fc", "inception"):
        # an activation next to zero falls on either side of its ReLU: a few deltas come or go whole
        return {"rel": 1e-3 if kind == "fc" else 3e-3, "max": 0.5}
    return {"rel": 1e-3}


# ---- preparation -----------------------------------------------------------------------------------
class _Inputs(object):
    """Random device arrays of one seed, and library tensors over device arrays."""

    def __init__(self, ng, seed):
        self.ng = ng
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, shape, std=1.0, dtype="f16"):
        return (torch.randn(tuple(shape), generator=self.gen, device="cuda") * std).to(_TORCH[dtype])

    def uniform(self, shape, lo=0.0, hi=1.0, dtype="f16"):
        return (torch.rand(tuple(shape), generator=self.gen, device="cuda") * (hi - lo) + lo).to(_TORCH[dtype])

    def tensor(self, t):
        dtype = np.float16 if t.dtype == torch.float16 else np.float32
        return GPUTensor(self.ng, tuple(t.shape), dtype, gpudata=t.data_ptr(), rounding=self.ng.round_mode)


def _view(x):
    """A library tensor's memory as a torch tensor."""
    return torch.as_tensor(x, device="cuda")


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["pass"](state)


def _prepare_dot(c, seed):
    ng = NervanaGPU(stochastic_round=c["sr"], seed=seed)
    r = _Inputs(ng, seed)
    m, n, k = c["m"], c["n"], c["k"]
    a = r.normal((k, m) if c["op"][0] == "t" else (m, k))
    b = r.normal((n, k) if c["op"][1] == "t" else (k, n), std=0.1)
    out = r.normal((m, n))
    A, B, C = r.tensor(a), r.tensor(b), r.tensor(out)
    return {"pass": _run_dot, "ng": ng, "keep": (a, b), "A": A.T if c["op"][0] == "t" else A, "B": B.T if c["op"][1] == "t" else B,
            "C": C, "relu": c["relu"], "beta": c["beta"], "start": r.normal((m, n)) if c["beta"] else None, "out": out}


def _run_dot(s):
    if s["start"] is not None:
        s["out"].copy_(s["start"])      # the sum that the product is added to
    s["ng"].dot(s["A"], s["B"], s["C"], beta=s["beta"], relu=s["relu"])
    return s["out"]


def _prepare_batched(c, seed):
    ng = NervanaGPU()
    r = _Inputs(ng, seed)
    b, m, n, k = (c[x] for x in ("batch", "m", "n", "k"))
    t = {"W": r.normal((m, k), std=0.05), "X": r.uniform((b, k, n)), "E": r.normal((b, m, n), std=0.1),
         "Y": torch.empty((b, m, n), device="cuda", dtype=torch.float16),
         "G": torch.empty((m, k), device="cuda", dtype=torch.float16)}
    s = {key: r.tensor(v) for key, v in t.items()}
    s.update({"pass": _run_batched, "ng": ng, "keep": t, "Xt": s["X"].T})
    return s


def _run_batched(s):
    ng = s["ng"]
    ng.batched_dot(s["W"], s["X"], s["Y"], relu=True)
    ng.batched_dot(s["E"], s["Xt"], s["G"])
    return s["keep"]["Y"], s["keep"]["G"]


def _prepare_conv(c, seed):
    ng = NervanaGPU()
    r = _Inputs(ng, seed)
    layer = ng.conv_layer(np.float16, c["N"], c["C"], c["K"], c["D"], c["H"], c["W"], c["T"], c["R"], c["S"],
                          c["pad_d"], c["pad"], c["pad"], c["str_d"], c["stride"], c["stride"])
    t = {"I": r.uniform(layer.dimI), "F": r.normal(layer.dimF, std=(2.0 / (layer.sizeF // c["K"])) ** 0.5),
         "E": r.normal(layer.dimO, std=0.1)}
    for key, dim, dtype in (("O", layer.dimO, torch.float16), ("gI", layer.dimI, torch.float16), ("gF", layer.dimF, torch.float32)):
        t[key] = torch.empty(dim, device="cuda", dtype=dtype)
    s = {key: r.tensor(v) for key, v in t.items()}
    s.update({"pass": _run_conv, "ng": ng, "layer": layer, "keep": t})
    return s


def _run_conv(s):
    ng, layer = s["ng"], s["layer"]
    ng.fprop_conv(layer, s["I"], s["F"], s["O"], relu=True)
    ng.bprop_conv(layer, s["F"], s["E"], s["gI"])
    ng.update_conv(layer, s["I"], s["E"], s["gF"])
    return s["keep"]["O"], s["keep"]["gI"], s["keep"]["gF"]


def _weights(r, layer):
    """Values that keep the size of what passes through a layer with a ReLU."""
    fan_in = layer.sizeF // layer.dimF2[1 if isinstance(layer, ConvLayer) else 0]
    return r.normal(layer.dimF, std=(2.0 / fan_in) ** 0.5)


def _layer_state(ng, r, layer, trained, learning_rate):
    """A layer with its input, its weights and the deltas that the layer above it left."""
    x, e = r.uniform(layer.dimI), r.normal(layer.dimO, std=0.1)
    layer.init_activations()
    layer.init_deltas()
    for inner in trained:
        inner.init_weights(zeros=True)
        inner.weights.copy(r.tensor(_weights(r, inner)))
        inner.learning_rate = learning_rate
    outs = [_view(layer.fprop_out), _view(layer.bprop_out)]
    outs += [_view(v) for inner in trained for v in (inner.updat_out, inner.weights)]
    torch.cuda.synchronize()            # the weights' sources are freed here
    return {"pass": _run_layer, "ng": ng, "layer": layer, "X": r.tensor(x), "E": r.tensor(e), "keep": (x, e), "outs": outs}


def _run_layer(s):
    s["layer"].fprop(s["X"])
    s["layer"].bprop(s["E"])
    return s["outs"]


def _prepare_fc(c, seed):
    ng = NervanaGPU()
    layer = FullLayer(ng, np.float16, c["n"], c["nin"], c["nout"])
    return _layer_state(ng, _Inputs(ng, seed), layer, [layer], _LEARNING_RATE["fc"])


def _conv_conf(K, R):
    return {"layer": ConvLayer, "K": K, "R": R, "S": R, "pad_h": R // 2, "pad_w": R // 2}


def _prepare_inception(c, seed):
    ng = NervanaGPU()
    data = DataLayer(ng, np.float16, c["N"], c["C"], 1, c["H"], c["H"])
    pool = {"layer": PoolLayer, "op": "max", "R": 3, "S": 3, "str_h": 1, "str_w": 1, "pad_h": 1, "pad_w": 1}
    conf = {"layer": Inception, "partitions": [[_conv_conf(c["n1"], 1)], [_conv_conf(c["r3"], 1), _conv_conf(c["n3"], 3)],
                                               [_conv_conf(c["r5"], 1), _conv_conf(c["n5"], 5)], [pool, _conv_conf(c["proj"], 1)]]}
    module = Layer.create(ng, conf, data, np.float16)
    convs = [l for part in module.partitions for l in part if isinstance(l, ConvLayer)]
    return _layer_state(ng, _Inputs(ng, seed), module, convs, _LEARNING_RATE["inception"])


_streams = []


def _prepare_stack(c, seed):
    ng = NervanaGPU()
    if not _streams:
        _streams.append(ng.new_stream())
    ng.stream = _streams[0]
    stack = ConvStack(ng, NETWORKS[c["net"]], N=c["N"], seed=seed, learning_rate=_LEARNING_RATE["stack"])
    # weights that carry the activations through all layers; deltas whose sum over the images does not
    # cancel, as a loss's do: the gradients are then far above the rounding noise of the deltas
    r = _Inputs(ng, seed)
    new = [(l.weights, _weights(r, l)) for l in stack.convs] + [(stack.top_delta, r.uniform(stack.layers[-1].dimO, hi=0.01))]
    torch.cuda.synchronize()
    for old, values in new:
        old.copy(r.tensor(values))
    ng.synchronize()
    stack.step()
    sequence = ng.capture(stack.step) if c["recorded"] else None
    outs = [_view(stack.acts[-1]), _view(stack.grads_flat), _view(stack.weights_flat)]
    ng.synchronize()
    return {"pass": _run_stack, "stack": stack, "step": sequence.launch if sequence else stack.step, "outs": outs}


def _run_stack(s):
    s["step"]()
    return s["outs"]


def _prepare_pool(c, seed):
    ng = NervanaGPU()
    r = _Inputs(ng, seed)
    layer = ng.pool_layer(_NP[c["dtype"]], c["op"], c["N"], c["C"], c["D"], c["H"], c["W"], c["J"], c["T"], c["R"], c["S"],
                          0, 0, c["pad"], c["pad"], c["str_j"], c["str_d"], c["stride"], c["stride"])
    t = {"I": r.uniform(layer.dimI, dtype=c["dtype"]), "E": r.normal(layer.dimO, std=0.1, dtype=c["dtype"]),
         "O": torch.empty(layer.dimO, device="cuda", dtype=_TORCH[c["dtype"]]),
         "gI": torch.empty(layer.dimI, device="cuda", dtype=_TORCH[c["dtype"]])}
    s = {key: r.tensor(v) for key, v in t.items()}
    s.update({"pass": _run_pool, "ng": ng, "layer": layer, "keep": t})
    return s


def _run_pool(s):
    ng, layer = s["ng"], s["layer"]
    ng.fprop_pool(layer, s["I"], s["O"])
    ng.bprop_pool(layer, s["I"], s["E"], s["gI"])
    return s["keep"]["O"], s["keep"]["gI"]


def _prepare_ew(c, seed):
    ng = NervanaGPU()
    r = _Inputs(ng, seed)
    shape, dtype = (c["rows"], c["cols"]), c["dtype"]
    if c["expr"] == "momentum":
        t = {"W": r.normal(shape, std=0.02, dtype=dtype), "V": r.normal(shape, std=1e-3, dtype=dtype),
             "G": r.normal(shape, std=0.1, dtype="f32")}
    else:
        t = {"A": r.uniform(shape, dtype=dtype) if c["expr"] == "batch_norm" else r.normal(shape, std=2.0, dtype=dtype),
             "O": torch.empty(shape, device="cuda", dtype=_TORCH[dtype])}
    s = {key: r.tensor(v) for key, v in t.items()}
    s.update({"pass": globals()["_run_" + c["expr"]], "ng": ng, "keep": t})
    return s


def _run_batch_norm(s):
    ng, A = s["ng"], s["A"]
    s["O"][:] = (A - ng.mean(A, axis=1)) / ng.sqrt(ng.var(A, axis=1) + 1e-3)
    return s["keep"]["O"]


def _run_softmax(s):
    ng, A = s["ng"], s["A"]
    s["O"][:] = ng.exp(A - ng.max(A, axis=0)) / ng.sum(ng.exp(A - ng.max(A, axis=0)), axis=0)
    return s["keep"]["O"]


def _run_momentum(s):
    W, V, G = s["W"], s["V"], s["G"]
    V[:] = V * 0.9 - (G + W * 5e-4) * 1e-4
    W[:] = W + V
    return s["keep"]["W"], s["keep"]["V"]

"""The forward passes that users of this framework run, as measurable cases.

Each case goes through the public API (``nebula_b200.api``): whole networks through the network executor, single
layers through the per-layer plans with the reference's NCHW tensors, and the operator library.  Weights and inputs
are seeded synthetic tensors with the shapes, value ranges and distributions of ``nebula_b200.workloads``.
"""
import math

import numpy as np
import torch

from nebula_b200 import api, workloads

IMAGE_NETS = ("vgg16", "resnet50", "alexnet", "dbn")


def listed():
    return [
        # the benchmark network at its batch: offline classification of an image collection
        {"name": "vgg16_b256", "kind": "net", "net": "vgg16", "math": "tf32", "batch": 256, "image": 224},
        # a small batch in the mode that agrees with the fp32 CPU path to 1e-5
        {"name": "vgg16_b8_tf32x3", "kind": "net", "net": "vgg16", "math": "tf32x3", "batch": 8, "image": 224},
        # an ordinary server batch of the batch-normalised network with shortcuts
        {"name": "resnet50_b64", "kind": "net", "net": "resnet50", "math": "tf32", "batch": 64, "image": 224},
        # one image at a time: the latency of a deep network's launches
        {"name": "resnet50_b1", "kind": "net", "net": "resnet50", "math": "tf32", "batch": 1, "image": 224},
        # AlexNet at the batch of the reference's own configuration
        {"name": "alexnet_b16", "kind": "net", "net": "alexnet", "math": "tf32", "batch": 16, "image": 227},
        # the same network with exact fp32 products, the mode results are checked in
        {"name": "alexnet_b4_fp32", "kind": "net", "net": "alexnet", "math": "fp32", "batch": 4, "image": 227},
        # the recurrent benchmark: two layers of 1024 over 128 steps and a projection of every step
        {"name": "lstm2_t128_b64_h1024", "kind": "net", "net": "lstm2", "math": "tf32", "batch": 64, "steps": 128,
         "inputs": 1024, "hidden": 1024, "classes": 10000, "act": "linear"},
        # a language model of ordinary size: hidden width off the tile sizes, a batch off the powers of two
        {"name": "lstm2_t35_b20_h300", "kind": "net", "net": "lstm2", "math": "tf32", "batch": 20, "steps": 35,
         "inputs": 300, "hidden": 300, "classes": 10000, "act": "linear"},
        # the vanilla recurrent network of the workloads
        {"name": "rnn2_t16_b32_h256", "kind": "net", "net": "rnn2", "math": "tf32", "batch": 32, "steps": 16,
         "inputs": 256, "hidden": 256, "classes": 1000, "act": "tanh"},
        # the deep belief network: a few connected layers, bound by its weights
        {"name": "dbn_b32", "kind": "net", "net": "dbn", "math": "tf32", "batch": 32, "image": 128},
        # a Nebula build that calls the backend layer by layer with its own NCHW buffers: conv, conv, pool
        {"name": "layers_b32_c128_f256", "kind": "layers", "math": "tf32", "batch": 32, "channels": 128, "size": 56,
         "filters": 256, "residual": False},
        # a connected layer written with the operator library: _gemm_, _forward_bias_, activation
        {"name": "gemm_256x1024x1024", "kind": "gemm", "math": "fp32", "m": 256, "n": 1024, "k": 1024, "ta": False,
         "tb": True, "act": "relu"},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    which = rng.choice(["vgg16", "resnet50", "alexnet", "lstm2", "lstm2", "rnn2", "dbn", "layers", "gemm"])
    math_mode = "tf32" if rng.random() < 0.7 else "tf32x3"
    if which in ("vgg16", "resnet50"):
        image = 32 * rng.randint(2, 7)
        return {"kind": "net", "net": which, "math": math_mode, "batch": _log(rng, 1, 128 if math_mode == "tf32" else 40),
                "image": image}
    if which == "alexnet":
        m = rng.choice(["tf32", "tf32", "tf32x3", "fp32"])
        return {"kind": "net", "net": which, "math": m, "batch": _log(rng, 1, 16 if m == "fp32" else 128), "image": 227}
    if which in ("lstm2", "rnn2"):
        # widths: mostly multiples of 4, small ones of any value
        def width():
            w = _log(rng, 32, 1024)
            return w if w <= 200 else w // 4 * 4
        lstm = which == "lstm2"
        return {"kind": "net", "net": which, "math": math_mode, "batch": _log(rng, 1, 100), "steps": _log(rng, 2, 64),
                "inputs": width(), "hidden": width(), "classes": _log(rng, 10, 10000),
                "act": "linear" if lstm else rng.choice(["tanh", "relu", "logistic"])}
    if which == "dbn":
        return {"kind": "net", "net": which, "math": math_mode, "batch": _log(rng, 1, 256), "image": 16 * rng.randint(1, 8)}
    if which == "layers":
        return {"kind": "layers", "math": math_mode, "batch": _log(rng, 1, 48), "channels": 4 * _log(rng, 8, 64),
                "size": rng.randint(7, 64), "filters": 4 * _log(rng, 8, 64), "residual": rng.random() < 0.5}
    while True:
        m, n, k = _log(rng, 1, 2048), _log(rng, 16, 4096), _log(rng, 16, 4096)
        if m * n * k <= 1 << 32:
            return {"kind": "gemm", "math": "fp32", "m": m, "n": n, "k": k, "ta": rng.random() < 0.3, "tb": rng.random() < 0.6,
                    "act": rng.choice(["relu", "leaky", "logistic", "linear"])}


# ------------------------------------------------------------------- states
class _State:
    """What a user's program keeps: the handle, the network or the plans, and this call's tensors on the GPU."""

    def __init__(self):
        self.owned = []         # closed in reverse order

    def own(self, obj):
        self.owned.append(obj)
        return obj

    def __del__(self):
        for obj in reversed(self.owned):
            obj.close()


def _workload(case):
    net, b = case["net"], case["batch"]
    if net in ("lstm2", "rnn2"):
        kw = dict(batch=b, time_steps=case["steps"], input_size=case["inputs"], hidden=case["hidden"], classes=case["classes"])
        return workloads.lstm2(**kw) if net == "lstm2" else workloads.rnn2(act=case["act"], **kw)
    if net == "alexnet":
        return workloads.alexnet(b)
    return {"vgg16": workloads.vgg16, "resnet50": workloads.resnet50, "dbn": workloads.dbn}[net](
        batch=b, height=case["image"], width=case["image"])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _weights(w, seed):
    """The workload's weight stream (the distributions of Workload.make_weights), drawn on the GPU."""
    g = _generator(seed)
    out = torch.empty(w.weight_count(), device="cuda")
    pos = 0
    for p in w.params:
        a = out[pos:pos + int(np.prod(p.shape))]
        pos += a.numel()
        if p.init == "he":
            a.normal_(0.0, math.sqrt(2.0 / p.fan_in), generator=g)
        elif p.init == "zeros":
            a.zero_()
        elif p.init == "uniform":
            a.uniform_(-p.bound, p.bound, generator=g)
        elif p.init == "bn_scale":
            a.uniform_(0.8, 1.2, generator=g)
        elif p.init == "bn_var":
            a.uniform_(0.5, 1.5, generator=g)
        else:                   # bn_mean, bias_n01
            a.normal_(0.0, 0.1, generator=g)
    return out


def _net_input(w, seed):
    x = torch.empty(w.input_shape, device="cuda")
    g = _generator(seed + 1000003)
    return x.uniform_(0.0, 1.0, generator=g) if w.input_dist == "uniform01" else x.normal_(generator=g)


def _layer_list(case):
    """The convolutions of a `layers` case: (channels, filters, size, padding, batch-norm, activation)."""
    c, f = case["channels"], case["filters"]
    if case["residual"]:        # bottleneck on f channels, the shortcut adds the block's input
        return [(f, c, 1, 0, True, "leaky"), (c, c, 3, 1, True, "leaky"), (c, f, 1, 0, True, "linear")]
    return [(c, f, 3, 1, False, "relu"), (f, f, 3, 1, False, "relu")]


def _layer_data(case, seed):
    g = _generator(seed)
    def normal(*shape, std=1.0):
        return torch.empty(shape, device="cuda").normal_(0.0, std, generator=g)
    def uniform(n, lo, hi):
        return torch.empty(n, device="cuda").uniform_(lo, hi, generator=g)
    params = []
    for (c, f, k, p, bn, act) in _layer_list(case):
        params.append((normal(f, c, k, k, std=math.sqrt(2.0 / (c * k * k))), normal(f, std=0.1),
                       (uniform(f, 0.8, 1.2), normal(f, std=0.1), uniform(f, 0.5, 1.5)) if bn else None))
    x = normal(case["batch"], _layer_list(case)[0][0], case["size"], case["size"])
    return params, x


def _gemm_data(case, seed):
    g = _generator(seed)
    m, n, k = case["m"], case["n"], case["k"]
    a = torch.empty((k, m) if case["ta"] else (m, k), device="cuda").normal_(generator=g)
    b = torch.empty((n, k) if case["tb"] else (k, n), device="cuda").normal_(0.0, math.sqrt(2.0 / k), generator=g)
    return a, b, torch.empty(n, device="cuda").normal_(0.0, 0.1, generator=g)


def prepare(case, seed):
    s = _State()
    s.case = case
    s.handle = s.own(api.Handle(0, case["math"]))
    if case["kind"] == "net":
        w = _workload(case)
        s.net = s.own(api.Network(s.handle, w.cfg))
        s.net.load_weights(_weights(w, seed))
        s.x = _net_input(w, seed)
    elif case["kind"] == "layers":
        params, s.x = _layer_data(case, seed)
        s.convs = []
        for (c, f, k, p, bn, act), (wt, bias, bnp) in zip(_layer_list(case), params):
            plan = s.own(api.Conv2d(s.handle, case["batch"], c, case["size"], case["size"], f, k, 1, p, bn, act))
            plan.set_weights(wt, bias, bnp)
            s.convs.append(plan)
    else:
        s.a, s.b, s.bias = _gemm_data(case, seed)
    return s


def run(s):
    case = s.case
    if case["kind"] == "net":
        s.net.forward(s.x)
        logits = s.net.logits("cuda")
        if case["net"] in IMAGE_NETS:
            return {"logits": logits, "probabilities": s.net.output("cuda")}
        return {"logits": logits}
    if case["kind"] == "layers":
        outs, y = [], s.x
        for conv in s.convs:
            y = conv.forward(y)
            outs.append(y)
        outs.append(s.handle.shortcut(y, s.x, "leaky") if case["residual"] else s.handle.pool(y, 2, 2, 0, "max"))
        return outs
    m, n, k = case["m"], case["n"], case["k"]
    out = torch.empty((m, n), device="cuda")
    s.handle.gemm(case["ta"], case["tb"], m, n, k, 1.0, s.a, s.a.shape[1], s.b, s.b.shape[1], 0.0, out, n)
    s.handle.forward_bias(out, s.bias, n, 1, m)
    return s.handle.activation(out, case["act"])


# --------------------------------------------------------- work and accuracy
def work(case):
    if case["kind"] == "net":
        w = _workload(case)
        rows = case["batch"] * case.get("steps", 1)
        outputs = rows * w.classes * (2 if case["net"] in IMAGE_NETS else 1)
        return {"bytes": 4.0 * (w.weight_count() + int(np.prod(w.input_shape)) + outputs),
                "flops": w.flops_per_unit * case["batch"]}
    if case["kind"] == "layers":
        ls, px = _layer_list(case), case["batch"] * case["size"] ** 2
        weights = sum(c * f * k * k for c, f, k, p, bn, act in ls)
        last = px * ls[-1][1] if case["residual"] else case["batch"] * ls[-1][1] * (case["size"] // 2) ** 2
        return {"bytes": 4.0 * (weights + px * (ls[0][0] + sum(f for c, f, k, p, bn, act in ls)) + last),
                "flops": 2.0 * px * weights}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": 4.0 * (m * k + k * n + n + m * n), "flops": 2.0 * m * n * k}


def tolerance(case):
    # about four times the measured distance to exact(): TF32 rounds each operand to 11 bits, layer after layer; the
    # other modes are at the level of fp32 sums
    if case["math"] != "tf32":
        return {"rel": 2.5e-5, "max": 1e-3}
    return {"rel": 6e-3, "max": 0.1}


# ------------------------------------------------------------ 64-bit results
def _act(x, name):
    if name == "linear":
        return x
    if name == "relu":
        return x.clamp(min=0.0)
    if name == "leaky":
        return torch.where(x > 0, x, 0.1 * x)
    return torch.sigmoid(x) if name == "logistic" else torch.tanh(x)


def _conv(x, w, stride, padding):
    """Patches and one matrix product per group of images (the library's 64-bit convolutions are slow)."""
    n, (f, c, k, _) = x.shape[0], w.shape
    oh, ow = ((e + 2 * padding - k) // stride + 1 for e in x.shape[2:])
    y = torch.empty((n, f, oh, ow), device=x.device, dtype=x.dtype)
    group = max(1, int(2.0e8 / (c * k * k * oh * ow)))
    for i in range(0, n, group):
        cols = torch.nn.functional.unfold(x[i:i + group], k, padding=padding, stride=stride)
        y[i:i + group] = torch.matmul(w.reshape(f, -1), cols).reshape(-1, f, oh, ow)
    return y


def _pool(x, size, stride, padding, is_max):
    oh, ow = (x.shape[2] + 2 * padding) // stride, (x.shape[3] + 2 * padding) // stride
    more = [max(0, (o - 1) * stride + size - e - padding) for o, e in ((ow, x.shape[3]), (oh, x.shape[2]))]
    x = torch.nn.functional.pad(x, (padding, more[0], padding, more[1]), value=-1e8 if is_max else 0.0)
    y = torch.nn.functional.max_pool2d(x, size, stride) if is_max else torch.nn.functional.avg_pool2d(x, size, stride)
    return y[:, :, :oh, :ow]


def _shortcut(prev, conn, act):
    s = max(1, conn.shape[3] // prev.shape[3])
    part = conn[:, :prev.shape[1], ::s, ::s][:, :, :prev.shape[2], :prev.shape[3]]
    y = prev.clone()
    y[:, :part.shape[1], :part.shape[2], :part.shape[3]] += part
    return _act(y, act)


def _bn(y, bn):
    """(y - mean) / (sqrt(var) + 1e-5) * scale over channel 1."""
    if bn is None:
        return y
    scale, mean, var = (v.double().reshape((1, -1) + (1,) * (y.dim() - 2)) for v in bn)
    return (y - mean) / (var.sqrt() + 0.00001) * scale


def _sections(cfg):
    secs = []
    for line in cfg.splitlines():
        if line.startswith("["):
            secs.append((line.strip("[]"), {}))
        elif "=" in line:
            key, value = line.split("=")
            secs[-1][1][key] = value
    return secs[1:]


class _Stream:
    def __init__(self, w):
        self.w, self.pos = w, 0

    def take(self, *shape):
        n = int(np.prod(shape))
        self.pos += n
        return self.w[self.pos - n:self.pos].reshape(shape).double()

    def connected(self, outputs, inputs, bn):
        b, w = self.take(outputs), self.take(outputs, inputs)
        return b, w, (self.take(outputs), self.take(outputs), self.take(outputs)) if bn else None


def _apply(gate, x, act):
    b, w, bn = gate
    return _act(_bn(x @ w.T, bn) + b, act)


def _lstm(x, s, hidden, act, bn):
    gates = [s.connected(hidden, hidden if i < 4 else x.shape[2], bn) for i in range(8)]       # iW fW oW cW iU fU oU cU
    h = c = torch.zeros((x.shape[1], hidden), device=x.device, dtype=x.dtype)
    out = []
    for xt in x:
        zi, zf, zo, zg = (_apply(gates[i], h, act) + _apply(gates[i + 4], xt, act) for i in range(4))
        c = c * torch.sigmoid(zf) + torch.sigmoid(zi) * torch.tanh(zg)
        h = torch.tanh(c) * torch.sigmoid(zo)
        out.append(h)
    return torch.stack(out)


def _rnn(x, s, hidden, act, bn):
    gi, gh, go = (s.connected(hidden, n, bn) for n in (x.shape[2], hidden, hidden))
    out, state = [], None
    for t, xt in enumerate(x):
        a = _apply(gi, xt, act)
        h = _apply(gh, a if t == 0 else state, act)
        state = a + h
        out.append(_apply(go, h if t == 0 else state, act))
    return torch.stack(out)


def _exact_net(w, stream, x):
    s, outs, logits = _Stream(stream), [], None
    for name, o in _sections(w.cfg):
        act, bn = o.get("activation"), o.get("batch_normalize") == "1"
        if name == "convolutional":
            f, k = int(o["filters"]), int(o["size"])
            b, wt = s.take(f), s.take(f, x.shape[1], k, k)
            bnp = (s.take(f), s.take(f), s.take(f)) if bn else None
            x = _act(_bn(_conv(x, wt, int(o["stride"]), int(o["padding"])), bnp) + b.reshape(1, -1, 1, 1), act)
        elif name in ("maxpool", "avgpool"):
            size = int(o["size"])
            x = _pool(x, size, int(o["stride"]), int(o.get("padding", (size - 1) // 2)), name == "maxpool")
        elif name == "shortcut":
            x = _shortcut(x, outs[len(outs) - int(o["hops"])], act)
        elif name in ("connected", "rbm"):
            x = x.reshape(-1, x.shape[2]) if w.recurrent else x.reshape(x.shape[0], -1)
            x = _apply(s.connected(int(o["output"]), x.shape[1], bn), x, act)
            logits = x if name == "connected" else logits
        elif name in ("lstm", "rnn"):
            x = (_lstm if name == "lstm" else _rnn)(x, s, int(o["output"]), act, bn)
        elif name == "softmax":
            x = torch.softmax(x, 1)
        outs.append(x if any(n == "shortcut" for n, _ in _sections(w.cfg)) else None)
    return logits, x


def exact(case, seed):
    if case["kind"] == "net":
        w = _workload(case)
        stream, x = _weights(w, seed), _net_input(w, seed)
        if w.recurrent:
            return {"logits": _exact_net(w, stream, x.double())[0].reshape(-1)}
        parts = [_exact_net(w, stream, x[i:i + 32].double()) for i in range(0, case["batch"], 32)]
        return {"logits": torch.cat([p[0] for p in parts]).reshape(-1),
                "probabilities": torch.cat([p[1] for p in parts]).reshape(-1)}
    if case["kind"] == "layers":
        params, x = _layer_data(case, seed)
        outs, y = [], x.double()
        for (c, f, k, p, bn, act), (wt, bias, bnp) in zip(_layer_list(case), params):
            y = _act(_bn(_conv(y, wt.double(), 1, p), bnp) + bias.double().reshape(1, -1, 1, 1), act)
            outs.append(y)
        outs.append(_shortcut(y, x.double(), "leaky") if case["residual"] else _pool(y, 2, 2, 0, True))
        return outs
    a, b, bias = (t.double() for t in _gemm_data(case, seed))
    return _act((a.T if case["ta"] else a) @ (b.T if case["tb"] else b) + bias, case["act"])

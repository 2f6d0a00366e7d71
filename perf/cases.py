"""Performance cases of the framework: what a user's program has it do, through the public entry points.

Four families, each with the sizes of the benchmark configurations, small and ragged ones, Float32 and BFloat16
storage, inference and training:

  mlp   chains of Dense layers (optionally LayerNorm -> Dense blocks): inference, eager `trainstep`, one-graph
        `GraphedTrainStep`, each with logitcrossentropy and Adam resumed in mid-training
  norm  LayerNorm / BatchNorm: inference, or forward + gradient of sum(abs2, y)
  rnn   LSTM / GRU over a sequence: inference, or forward + gradient of sum(abs2, out)
  mha   MultiHeadAttention: inference (self- or cross-attention), or the pre-norm residual sublayer
        x + mha(layernorm(x)) forward + gradient
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "flux.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fluxb200 as F  # noqa: E402


def listed():
    mlp = {"kind": "mlp", "dtype": "f32", "in": 784, "width": 512, "depth": 2, "classes": 10, "norm": False}
    wide = {"kind": "mlp", "in": 4096, "width": 4096, "classes": 1000, "norm": True}
    return [
        # one sample through a small classifier: a request to a served model, all latency
        dict(mlp, name="mlp_infer_1", mode="infer", batch=1),
        # the last, shorter batch of an epoch, kernel by kernel as `train` runs it
        dict(mlp, name="mlp_train_100", mode="train", batch=100),
        # the MNIST-sized training step, captured once and replayed
        dict(mlp, name="mlp_graph_1024", mode="graph", batch=1024),
        # the data-parallel benchmark model on one GPU: 8 x [LayerNorm -> Dense(4096, gelu)] -> 1000 classes
        dict(wide, name="wide_graph_8192", mode="graph", dtype="f32", depth=8, batch=8192),
        # a bf16 model trained eagerly, with Float32 master weights in the optimiser
        dict(wide, name="wide_bf16_train_2048", mode="train", dtype="bf16", depth=3, batch=2048),
        # batch normalisation of image feature maps (W, H, C, N) in training
        {"name": "batchnorm_train", "kind": "norm", "layer": "batch", "mode": "grad", "space": 1024, "feat": 256, "batch": 128, "act": "relu"},
        # layer normalisation of odd-sized features
        {"name": "layernorm_odd_grad", "kind": "norm", "layer": "layer", "mode": "grad", "space": 1, "feat": 1001, "batch": 3000, "act": "identity"},
        # the recurrent benchmark: 256 dependent steps each way
        {"name": "lstm_512_grad", "kind": "rnn", "cell": "lstm", "mode": "grad", "in": 512, "hidden": 512, "steps": 256, "batch": 64},
        # a small sequence model with sizes nobody rounded
        {"name": "gru_odd_grad", "kind": "rnn", "cell": "gru", "mode": "grad", "in": 65, "hidden": 200, "steps": 50, "batch": 20},
        # the attention benchmark, as the sublayer of a decoder: causal, sequence 2048
        {"name": "mha_f32_grad", "kind": "mha", "dtype": "f32", "mode": "grad", "head": 64, "heads": 16, "lq": 2048, "lk": 2048, "batch": 8, "causal": True},
        # the same in BFloat16 storage
        {"name": "mha_bf16_grad", "kind": "mha", "dtype": "bf16", "mode": "grad", "head": 64, "heads": 16, "lq": 2048, "lk": 2048, "batch": 8, "causal": True},
        # cross-attention of a short query sequence over a longer memory, inference
        {"name": "mha_cross_infer", "kind": "mha", "dtype": "f32", "mode": "infer", "head": 64, "heads": 8, "lq": 77, "lk": 301, "batch": 3, "causal": False},
    ]


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """Log-uniform in [lo, hi]; two of three are multiples of 8 where that is possible, the rest as they come."""
    v = _logint(rng, lo, hi)
    if rng.random() < 0.67 and v >= 8:
        v = max(8, v - v % 8)
    return v


def _draw(rng):
    kind = rng.choice(("mlp", "norm", "rnn", "mha"))
    if kind == "mlp":
        mode = rng.choice(("infer", "train", "graph"))
        low = mode != "graph" and rng.random() < 0.4       # GraphedTrainStep takes Float32 models
        norm = rng.random() < 0.5
        c = {"kind": kind, "mode": mode, "dtype": "bf16" if low else "f32", "in": _size(rng, 16, 4096), "width": _size(rng, 32, 4096),
             "depth": rng.randint(1, 8 if norm else 4), "classes": _size(rng, 2, 1000), "norm": norm, "batch": _size(rng, 1, 8192)}
        if low:     # bf16 Dense layers take sizes that are multiples of 8
            for k in ("in", "width", "classes"):
                c[k] = max(8, c[k] - c[k] % 8)
        if norm:
            c["in"] = c["width"]
        return c
    if kind == "norm":
        layer = rng.choice(("layer", "batch"))
        c = {"kind": kind, "layer": layer, "mode": rng.choice(("infer", "grad")), "space": 1, "act": rng.choice(("identity", "relu"))}
        if layer == "layer":
            c.update(feat=_size(rng, 32, 8192), batch=_size(rng, 1, 16384))
        else:
            side = rng.choice((1, 7, 8, 14, 16, 28, 32))
            c.update(space=side * side, feat=_size(rng, 16, 512), batch=_size(rng, 2, 256))
        return c
    if kind == "rnn":
        return {"kind": kind, "cell": rng.choice(("lstm", "gru")), "mode": rng.choice(("infer", "grad")), "in": _size(rng, 8, 512),
                "hidden": _size(rng, 16, 768), "steps": _logint(rng, 1, 256), "batch": _size(rng, 1, 128)}
    mode = rng.choice(("infer", "grad"))
    cross = mode == "infer" and rng.random() < 0.5
    lk = _logint(rng, 4, 2048)
    return {"kind": kind, "dtype": rng.choice(("f32", "bf16")), "mode": mode, "head": rng.choice((32, 64, 64, 64, 128)),
            "heads": rng.randint(1, 16), "lq": _logint(rng, 1, 512) if cross else lk, "lk": lk, "batch": _logint(rng, 1, 16),
            "causal": not cross and rng.random() < 0.7}


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if w["flops"] <= 1.5e12 and w["bytes"] <= 1e9:
            return c


# ------------------------------------------------------------------------------------- inputs ---
def _normal(g, size, scale=1.0, shift=0.0):
    return F.B200Array(torch.randn(math.prod(size), generator=g, device="cuda") * scale + shift, size)


def _glorot(g, out, inp):
    bound = math.sqrt(6.0 / (out + inp))
    return F.B200Array((torch.rand(out * inp, generator=g, device="cuda") * 2 - 1) * bound, (out, inp))


def _dense(g, inp, out, act="identity"):
    return F.Dense(_glorot(g, out, inp), _normal(g, (out,), 0.01), act)


def _layernorm(g, d, act="identity"):
    ln = F.LayerNorm(d, sigma=act)
    ln.diag.scale = _normal(g, (d,), 0.1, 1.0)
    ln.diag.bias = _normal(g, (d,), 0.1)
    return ln


def _prepare_mlp(c, g):
    # relu in inference; gelu in training, whose gradients do not jump where a pre-activation rounds across zero
    act = "relu" if c["mode"] == "infer" and not c["norm"] else "gelu"
    layers, d = [], c["in"]
    for _ in range(c["depth"]):
        if c["norm"]:
            layers.append(_layernorm(g, d))
        layers.append(_dense(g, d, c["width"], act))
        d = c["width"]
    layers.append(_dense(g, d, c["classes"]))
    model = F.Chain(*layers)
    x = _normal(g, (c["in"], c["batch"]))
    if c["dtype"] == "bf16":
        model = F.bf16(model)
    s = {"model": model, "x": x}
    if c["mode"] == "infer":
        return s
    labels = torch.randint(1, c["classes"] + 1, (c["batch"],), generator=g, device="cuda", dtype=torch.int32)
    s["y"] = F.OneHotLabels(F.B200Array(labels, (c["batch"],)), c["classes"])
    # an optimiser in mid-training: both moments hold something, a thousand steps are behind it
    s["opt"] = opt = F.setup(F.Adam(1e-4), model)
    for p in opt.params:
        state = opt.leaves[id(p)].state
        state[0].t.copy_(torch.randn(p.numel(), generator=g, device="cuda") * 1e-4)
        state[1].t.copy_((torch.rand(p.numel(), generator=g, device="cuda") + 0.5) * 1e-8)
        state[2] = (0.9 ** 1000, 0.999 ** 1000)
    if c["mode"] == "graph":
        s["step"] = F.GraphedTrainStep(_mlp_loss, model, opt, (x, s["y"]))
    return s


def _prepare_norm(c, g):
    if c["layer"] == "layer":
        layer, size = _layernorm(g, c["feat"], c["act"]), (c["feat"], c["batch"])
    else:
        layer = F.BatchNorm(c["feat"], c["act"])
        layer.γ, layer.β = _normal(g, (c["feat"],), 0.1, 1.0), _normal(g, (c["feat"],), 0.1)
        layer.μ = _normal(g, (c["feat"],), 0.1, 0.5)
        layer.σ2 = F.B200Array(torch.rand(c["feat"], generator=g, device="cuda") + 3.5, (c["feat"],))
        side = math.isqrt(c["space"])
        size = (side, side, c["feat"], c["batch"])
    return {"model": layer, "x": _normal(g, size, 2.0, 0.5)}


def _prepare_rnn(c, g):
    rows = c["hidden"] * (4 if c["cell"] == "lstm" else 3)
    make = F.LSTM if c["cell"] == "lstm" else F.GRU
    rnn = make(_glorot(g, rows, c["in"]), _glorot(g, rows, c["hidden"]), _normal(g, (rows,), 0.01))
    return {"model": rnn, "x": _normal(g, (c["in"], c["steps"], c["batch"]))}


def _prepare_mha(c, g):
    e = c["head"] * c["heads"]
    mha = F.MultiHeadAttention(*[_glorot(g, e, e) for _ in range(4)], nheads=c["heads"])
    q = _normal(g, (e, c["lq"], c["batch"]))
    mask = F.make_causal_mask() if c["causal"] else None
    if c["mode"] == "grad":
        model = F.Chain(_layernorm(g, e), mha)
        return {"model": F.bf16(model) if c["dtype"] == "bf16" else model, "x": q, "mask": mask}
    kv = q if c["lq"] == c["lk"] else _normal(g, (e, c["lk"], c["batch"]))
    if c["dtype"] == "bf16":
        mha, low = F.bf16(mha), F.bf16(q)
        q, kv = low, (low if kv is q else F.bf16(kv))
    return {"model": mha, "x": q, "kv": kv, "mask": mask}


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = {"mlp": _prepare_mlp, "norm": _prepare_norm, "rnn": _prepare_rnn, "mha": _prepare_mha}[case["kind"]](case, g)
    s["case"] = case
    return s


# --------------------------------------------------------------------------------- one pass ---
def _mlp_loss(m, x, y):
    return F.logitcrossentropy(m(x), y)


def _sublayer(m, x, mask):
    y = F.add(x, m[1](m[0](x), mask=mask)[0])
    return F.sum_abs2(y), y


def _plain(v):
    """Framework arrays as the tensors behind them, through the containers a gradient comes in."""
    if isinstance(v, F.B200Array):
        return v.t
    if isinstance(v, dict):
        return {k: _plain(x) for k, x in v.items() if x is not None and not isinstance(x, (str, bool))}
    if isinstance(v, (tuple, list)):
        return [_plain(x) for x in v]
    return v


def _with_gradient(f, model):
    out, (grads,) = F.withgradient(f, model)
    return {"out": _plain(out), "grads": _plain(grads)}


def run(state):
    c, m, x = state["case"], state["model"], state["x"]
    if c["kind"] == "mlp":
        if c["mode"] == "infer":
            return _plain(m(x))
        loss = state["step"](x, state["y"]) if c["mode"] == "graph" else F.trainstep(_mlp_loss, m, (x, state["y"]), state["opt"])
        opt = state["opt"]
        out = [loss] + [p.t for p in opt.params]
        for p in opt.params:
            if p.ndim == 2:
                leaf = opt.leaves[id(p)]
                out += [leaf.state[0].t, leaf.state[1].t]
        return out
    if c["kind"] == "mha":
        mask = state["mask"]
        if c["mode"] == "infer":
            return _plain(m(x, state["kv"], mask=mask)[0])
        return _with_gradient(lambda model: _sublayer(model, x, mask), m)
    if c["mode"] == "infer":
        return _plain(m(x))

    def f(model):
        y = model(x)
        return F.sum_abs2(y), y

    out = _with_gradient(f, m)
    if c["kind"] == "norm" and c["layer"] == "batch":
        out["running"] = [m.μ.t, m.σ2.t]
    return out


# ------------------------------------------------------- what a pass cannot do without, and how close ---
def work(case):
    c = case
    grad = c["mode"] != "infer"
    if c["kind"] == "mlp":
        n, el = c["batch"], 2 if c["dtype"] == "bf16" else 4
        dims = [c["in"]] + [c["width"]] * c["depth"] + [c["classes"]]
        macs = sum(a * b for a, b in zip(dims, dims[1:]))
        params = macs + sum(dims[1:]) + (2 * c["width"] * c["depth"] if c["norm"] else 0)
        if not grad:
            return {"bytes": el * (params + n * c["classes"]) + 4 * n * c["in"], "flops": 2.0 * macs * n}
        # the first layer needs no gradient of its input unless a LayerNorm with parameters sits before it
        flops = 2.0 * n * (3 * macs - (0 if c["norm"] else dims[0] * dims[1]))
        # parameters (and the Float32 masters of bf16 ones) and both moments are read and written once
        return {"bytes": params * (24 + (2 if el == 2 else 0)) + 4 * n * (c["in"] + 1), "flops": flops}
    if c["kind"] == "norm":
        e = c["space"] * c["feat"] * c["batch"]
        # inference: x in, y out; training: x in, y out for the loss (a gradient of the layer's parameters only)
        return {"bytes": 4.0 * (2 * e + 4 * c["feat"]), "flops": (16.0 if grad else 6.0) * e}
    if c["kind"] == "rnn":
        i, h, tb = c["in"], c["hidden"], c["steps"] * c["batch"]
        gates = 4 if c["cell"] == "lstm" else 3
        params = gates * h * (i + h + 1)
        flops = 2.0 * gates * h * (i + h) * tb
        if grad:    # + dWi, dWh, Wh' dgates; the input gets no gradient
            flops += 2.0 * gates * h * (i + 2 * h) * tb
        return {"bytes": 4.0 * ((2 if grad else 1) * params + tb * (i + h)), "flops": flops}
    e, b, lq, lk = c["head"] * c["heads"], c["batch"], c["lq"], c["lk"]
    el = 2 if c["dtype"] == "bf16" else 4
    pairs = lq * (lq + 1) / 2 if c["causal"] else lq * lk
    proj = 2.0 * e * e * b * (2 * lq + 2 * lk)
    core = 4.0 * e * b * pairs
    if not grad:
        return {"bytes": float(el * (4 * e * e + e * b * (2 * lq + (0 if lq == lk else lk)))), "flops": proj + core}
    return {"bytes": 8.0 * e * e * el + 4.0 * 2 * e * b * lq, "flops": 3 * proj + 3.5 * core}


def tolerance(case):
    """Relative 2-norm errors of Float32 sums of the lengths at hand, or of BFloat16 storage (8 bits)."""
    c = case
    if c.get("dtype") == "bf16":
        return {"rel": 1e-2}
    if c["kind"] == "norm":
        return {"rel": 1e-5, "max": 1e-3}
    # products accumulate up to 2048 terms on the tensor cores between round-to-nearest adds; the attention sublayer
    # chains six of them
    return {"rel": 1e-4 if c["kind"] == "mha" and c["mode"] == "grad" else 5e-5, "max": 5e-3}

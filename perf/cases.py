"""The work that users of this library have it do, at sizes from the smallest call to whole training runs.

A program uses the library in two ways: through the layer calls (`ops`, one call per library call site that they stand
in for) and through `Network`, which owns the memory manager and the training step.  The cases below cover both:

  head   softmax, the loss, the seed of backward and the softmax gradient: the end of every step, a few short launches
  conv   one convolution layer trained: forward with bias, then data, filter and bias gradient
  fc     one fully connected layer trained: forward with bias, then data, filter and bias gradient
  stage  the bandwidth-bound layers between two convolutions: activation, normalisation across channels, max-pooling,
         forward and backward
  net    training through Network: a fresh batch from pinned host memory and a loss read back every step, and the
         parameters read out at the end, as a program that writes a checkpoint does

All arithmetic of the library is fp32 in, fp32 out; it has no other data type.  Both algorithm modes are used: PERF_OPT
where a program has memory to spare for workspace, MEMORY_OPT where it has not.
"""
import math
import weakref

import numpy as np
import torch

import vdnn_implementation_b200 as v

ALGO = {"MEMORY_OPT": "VDNN_MEMORY_OPT_ALGO", "PERF_OPT": "VDNN_PERF_OPT_ALGO"}
MODE = {"MEMORY_OPT": v.VDNN_MEMORY_OPT_ALGO, "PERF_OPT": v.VDNN_PERF_OPT_ALGO}
CONV_BWD_ALL = 3


def listed():
    return [
        # the end of a training step at batch 64 over 1000 classes: short launches, latency
        {"name": "head", "kind": "head", "rows": 64, "cols": 1000},
        # a small classifier (32 x 32 images) at batch 8, offloading everything: launches and host work per layer
        {"name": "net small", "kind": "net", "model": "small", "batch": 8, "image": 32, "width": 32, "classes": 10,
         "policy": "VDNN_ALL", "algo": "PERF_OPT", "steps": 4},
        # a convolution of odd extents and channel counts that are no multiple of a tile
        {"name": "conv ragged", "kind": "conv", "n": 5, "c": 48, "h": 27, "w": 31, "k": 80, "r": 3, "pad": 1, "stride": 1,
         "algo": "PERF_OPT"},
        # the second convolution of the AlexNet of the benchmark, where workspace is not to be had
        {"name": "conv 5x5 no workspace", "kind": "conv", "n": 64, "c": 96, "h": 27, "w": 27, "k": 256, "r": 5, "pad": 2, "stride": 1,
         "algo": "MEMORY_OPT"},
        # a first layer: three channels, large filter, stride 4
        {"name": "conv first layer", "kind": "conv", "n": 64, "c": 3, "h": 227, "w": 227, "k": 96, "r": 11, "pad": 0, "stride": 4,
         "algo": "PERF_OPT"},
        # VGG16: few channels on a large image ...
        {"name": "conv wide image", "kind": "conv", "n": 32, "c": 64, "h": 224, "w": 224, "k": 64, "r": 3, "pad": 1, "stride": 1,
         "algo": "PERF_OPT"},
        # ... and many channels on a small one
        {"name": "conv deep", "kind": "conv", "n": 64, "c": 256, "h": 28, "w": 28, "k": 512, "r": 3, "pad": 1, "stride": 1,
         "algo": "PERF_OPT"},
        # the first fully connected layer of VGG16
        {"name": "fc", "kind": "fc", "n": 64, "c": 25088, "k": 4096, "algo": "MEMORY_OPT"},
        # activation, normalisation and overlapping pooling behind AlexNet's first convolution
        {"name": "stage", "kind": "stage", "n": 64, "c": 96, "h": 55, "w": 55, "act": "RELU", "lrn": True, "win": 3, "stride": 2},
        # the three benchmark configurations: AlexNet with normalisation and no workspace, VGG16 resident, VGG16 offloaded
        {"name": "net alexnet baseline", "kind": "net", "model": "ALEXNET_LRN", "batch": 128, "policy": "BASELINE", "algo": "MEMORY_OPT",
         "steps": 8},
        {"name": "net vgg16 resident", "kind": "net", "model": "VGG16_64", "batch": 64, "policy": "VDNN_NONE", "algo": "PERF_OPT", "steps": 8},
        {"name": "net vgg16 offload", "kind": "net", "model": "VGG16_64", "batch": 32, "policy": "VDNN_ALL", "algo": "PERF_OPT", "steps": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case.  Sizes are logarithmic and mostly odd; convolutions and networks are bounded by their arithmetic."""
    kind = rng.choices(["head", "conv", "fc", "stage", "net"], [1, 5, 1, 2, 2])[0]
    if kind == "head":
        return {"kind": kind, "rows": _log(rng, 1, 256), "cols": _log(rng, 2, 4000)}
    if kind == "fc":
        return {"kind": kind, "n": _log(rng, 1, 256), "c": _log(rng, 64, 25088), "k": _log(rng, 10, 4096),
                "algo": rng.choice(["MEMORY_OPT", "PERF_OPT"])}
    if kind == "stage":
        side = _log(rng, 13, 224)
        c = _log(rng, 16, 512)
        n = max(1, min(128, int(_log(rng, 10 ** 5, 10 ** 8) / (side * side * c))))
        win, stride = rng.choice([(2, 2), (3, 2)])
        return {"kind": kind, "n": n, "c": c, "h": side, "w": max(13, side + rng.randint(-3, 3)),
                "act": rng.choices(["RELU", "TANH", "SIGMOID"], [4, 1, 1])[0], "lrn": rng.random() < 0.4, "win": win, "stride": stride}
    if kind == "conv":
        algo = rng.choices(["PERF_OPT", "MEMORY_OPT"], [3, 2])[0]
        if rng.random() < 0.2:      # a first layer
            r, stride, pad = rng.choice([(11, 4, 0), (3, 1, 1), (7, 2, 3), (5, 1, 2)])
            c, k, side = rng.choice([1, 3, 3, 3, 4]), 16 * rng.randint(2, 8), _log(rng, 32, 230)
        else:                       # an inner layer: block-sized channel counts more often than odd ones
            r, stride, pad = rng.choices([(3, 1, 1), (5, 1, 2), (3, 1, 0), (1, 1, 0), (3, 2, 1)], [6, 2, 1, 1, 1])[0]
            if rng.random() < 0.65:
                c, k = (rng.choice([32, 64, 96, 128, 192, 256, 384, 512]) for _ in range(2))
            else:
                c, k = _log(rng, 8, 512), _log(rng, 8, 512)
            side = _log(rng, 7, 224)
        w = max(r + stride, side + rng.randint(-4, 4))
        per_image = 2.0 * c * k * r * r * side * w / stride ** 2
        n = max(1, min(128, int(_log(rng, 10 ** 8, 4 * 10 ** 11) / per_image)))
        return {"kind": kind, "n": n, "c": c, "h": max(r + stride, side), "w": w, "k": k, "r": r, "pad": pad, "stride": stride, "algo": algo}
    algo, policy = rng.choice(["PERF_OPT", "MEMORY_OPT"]), rng.choice(["BASELINE", "VDNN_NONE", "VDNN_CONV", "VDNN_ALL"])
    if rng.random() < 0.7:
        return {"kind": kind, "model": "small", "batch": _log(rng, 1, 64), "image": rng.choice([24, 32, 48, 64]), "width": rng.choice([16, 32, 64, 96]),
                "classes": rng.choice([10, 37, 100]), "policy": policy, "algo": algo, "steps": rng.randint(1, 6)}
    model = rng.choice(["ALEXNET", "ALEXNET_LRN", "OVERFEAT", "VGG16_64"])
    return {"kind": kind, "model": model, "batch": _log(rng, 4, 16 if model == "VGG16_64" else 96), "policy": policy, "algo": algo,
            "steps": rng.randint(2, 4)}


# ---------------------------------------------------------------------------------------------------------------- layers

def _gradient(shape, gen):
    """What arrives from the layers above: small, differing in size from image to image, two thirds zero behind an activation."""
    g = torch.randn(shape, device="cuda", generator=gen) * 1e-3
    g *= torch.exp(torch.randn((shape[0],) + (1,) * (len(shape) - 1), device="cuda", generator=gen))
    return g * (torch.rand(shape, device="cuda", generator=gen) < 0.34)


def _activation(shape, gen):
    return torch.relu(torch.randn(shape, device="cuda", generator=gen))


def _conv_dims(c):
    return (c["h"] + 2 * c["pad"] - c["r"]) // c["stride"] + 1, (c["w"] + 2 * c["pad"] - c["r"]) // c["stride"] + 1


def _prepare_head(c, gen):
    rows, cols = c["rows"], c["cols"]
    x = torch.randn(rows, cols, device="cuda", generator=gen) * 2
    label = torch.zeros(rows, cols, device="cuda")
    label[torch.arange(rows, device="cuda"), torch.randint(cols, (rows,), device="cuda", generator=gen)] = 1
    return {"x": x, "label": label, "y": torch.empty_like(x), "seed": torch.empty_like(x), "dx": torch.empty_like(x),
            "loss": torch.empty(2, dtype=torch.float64, device="cuda")}


def _run_head(c, s):
    stream = torch.cuda.current_stream().cuda_stream
    rows, cols = c["rows"], c["cols"]
    v.ops.softmax_fwd(rows, cols, s["x"], s["y"], stream=stream)
    v.ops.loss(rows, cols, s["y"], s["label"], s["loss"], stream=stream)
    v.ops.sub(rows * cols, s["y"], s["label"], s["seed"], stream=stream)
    v.ops.softmax_bwd(rows, cols, s["y"], s["seed"], s["dx"], stream=stream)
    return {k: s[k] for k in ("y", "loss", "seed", "dx")}


def _prepare_conv(c, gen):
    p, q = _conv_dims(c)
    first = c["c"] <= 4
    d = v.ops.conv_desc(c["n"], c["c"], c["h"], c["w"], c["k"], c["r"], c["r"], (c["pad"],) * 2, (c["stride"],) * 2)
    mode = MODE[c["algo"]]
    space = max(v.ops.conv_workspace_bytes(op, mode, d) for op in (v.abi.CONV_FWD, CONV_BWD_ALL))
    shape = (c["n"], c["c"], c["h"], c["w"])
    s = {"d": d, "mode": mode, "space": space, "work": torch.empty(max(space, 16), dtype=torch.uint8, device="cuda"),
         "x": torch.randn(shape, device="cuda", generator=gen) if first else _activation(shape, gen),
         "w": torch.randn(c["k"], c["c"], c["r"], c["r"], device="cuda", generator=gen) * math.sqrt(2.0 / (c["c"] * c["r"] ** 2)),
         "b": torch.randn(c["k"], device="cuda", generator=gen) * 0.1,
         "dy": _gradient((c["n"], c["k"], p, q), gen)}
    for name, like in (("y", "dy"), ("dx", "x"), ("dw", "w"), ("db", "b")):
        s[name] = torch.empty_like(s[like])
    return s


def _run_conv(c, s):
    stream = torch.cuda.current_stream().cuda_stream
    v.ops.conv_fwd(s["d"], s["x"], s["w"], s["y"], bias=s["b"], algo_mode=s["mode"], workspace=s["work"], workspace_bytes=s["space"],
                   stream=stream)
    v.ops.conv_bwd_data_filter_bias(s["d"], s["w"], s["x"], s["dy"], s["dx"], s["dw"], s["db"], algo_mode=s["mode"], workspace=s["work"],
                                    workspace_bytes=s["space"], stream=stream)
    return {k: s[k] for k in ("y", "dx", "dw", "db")}


def _prepare_fc(c, gen):
    n, cin, k, mode = c["n"], c["c"], c["k"], MODE[c["algo"]]
    space = max(v.ops.sgemm_workspace_bytes(mode, *mnk) for mnk in ((k, n, cin), (cin, n, k), (cin, k, n)))
    s = {"mode": mode, "space": space, "work": torch.empty(max(space, 16), dtype=torch.uint8, device="cuda"),
         "x": _activation((n, cin), gen), "w": torch.randn(k, cin, device="cuda", generator=gen) * math.sqrt(2.0 / cin),
         "b": torch.randn(k, device="cuda", generator=gen) * 0.1, "dy": _gradient((n, k), gen)}
    for name, like in (("y", "dy"), ("dx", "x"), ("dw", "w"), ("db", "b")):
        s[name] = torch.empty_like(s[like])
    return s


def _run_fc(c, s):
    stream = torch.cuda.current_stream().cuda_stream
    n, cin, k = c["n"], c["c"], c["k"]
    how = {"algo_mode": s["mode"], "workspace": s["work"], "workspace_bytes": s["space"], "stream": stream}
    v.ops.sgemm(1, 0, k, n, cin, 1.0, s["w"], cin, s["x"], cin, 0.0, s["y"], k, **how)
    v.ops.add_bias(n, k, 1, s["b"], s["y"], stream=stream)
    v.ops.sgemm(0, 0, cin, n, k, 1.0, s["w"], cin, s["dy"], k, 0.0, s["dx"], cin, **how)
    v.ops.sgemm(0, 1, cin, k, n, 1.0, s["x"], cin, s["dy"], k, 0.0, s["dw"], cin, **how)
    v.ops.conv_bwd_bias(n, k, 1, s["dy"], s["db"], stream=stream)
    return {key: s[key] for key in ("y", "dx", "dw", "db")}


def _pool_dims(c):
    return (c["h"] - c["win"]) // c["stride"] + 1, (c["w"] - c["win"]) // c["stride"] + 1


def _prepare_stage(c, gen):
    shape = (c["n"], c["c"], c["h"], c["w"])
    x = torch.randn(shape, device="cuda", generator=gen)
    s = {"x": x, "dp": _gradient(shape[:2] + _pool_dims(c), gen), "act": getattr(v.ops, "ACT_" + c["act"])}
    for name in ("a", "da", "dx") + (("l", "dl") if c["lrn"] else ()):
        s[name] = torch.empty_like(x)
    s["p"] = torch.empty_like(s["dp"])
    return s


def _run_stage(c, s):
    stream = torch.cuda.current_stream().cuda_stream
    n, ch, h, w = c["n"], c["c"], c["h"], c["w"]
    window = ((c["win"],) * 2, (c["stride"],) * 2)
    count = n * ch * h * w
    v.ops.activation_fwd(s["act"], count, s["x"], s["a"], stream=stream)
    below, dbelow = ("l", "dl") if c["lrn"] else ("a", "da")
    if c["lrn"]:
        v.ops.lrn_fwd(n, ch, h * w, s["a"], s["l"], stream=stream)
    v.ops.maxpool_fwd(n, ch, h, w, *window, s[below], s["p"], stream=stream)
    v.ops.maxpool_bwd(n, ch, h, w, *window, s["p"], s["dp"], s[below], s[dbelow], stream=stream)
    if c["lrn"]:
        v.ops.lrn_bwd(n, ch, h * w, s["a"], s["l"], s["dl"], s["da"], stream=stream)
    v.ops.activation_bwd(s["act"], count, s["a"], s["da"], s["x"], s["dx"], stream=stream)
    return {k: s[k] for k in ("a", "l", "p", "dl", "da", "dx") if k in s}


# -------------------------------------------------------------------------------------------------------------- networks

def _small_net(c):
    """Two blocks of convolutions and a two-layer classifier, as (type, n, c, h, w, pad, pad, stride, stride, k, r, s)."""
    n, side, wide = c["batch"], c["image"], c["width"]
    half, quarter = side // 2, side // 4
    conv = lambda cin, k, at: (v.FC_CONV, n, cin, at, at, 1, 1, 1, 1, k, 3, 3)  # noqa: E731
    relu = lambda ch, at: (v.RELU, n, ch, at, at, 0, 0, 0, 0, 0, 0, 0)  # noqa: E731
    pool = lambda ch, at: (v.POOL, n, ch, at, at, 0, 0, 2, 2, 0, 2, 2)  # noqa: E731
    fc = lambda cin, k: (v.FC_GEMM, n, cin, 1, 1, 0, 0, 0, 0, k, 1, 1)  # noqa: E731
    return [conv(3, wide, side), relu(wide, side), conv(wide, wide, side), relu(wide, side), pool(wide, side),
            conv(wide, 2 * wide, half), relu(2 * wide, half), pool(2 * wide, half),
            fc(2 * wide * quarter ** 2, 128), relu(128, 1), fc(128, c["classes"]), (v.SOFTMAX, n, c["classes"], 1, 1, 0, 0, 0, 0, 0, 0, 0)]


def _network(c, device, seed=0):
    how = {"vdnn_type": c["policy"], "algo_mode": ALGO[c["algo"]], "device": device, "weight_seed_base": 3000 + 100 * (seed % 1000003)}
    if c["model"] == "small":
        return v.Network("CUSTOM_CNN", pool_bytes=4e9, learning_rate=1e-4, custom_layers=_small_net(c), **how)
    return v.Network(c["model"], batch_size=c["batch"], pool_bytes=24e9, learning_rate=1e-6, **how)


# A process has one Network at a time (it owns the device pool); a program that trains feeds it batch after batch.  So all
# states of a case share the network of the first of them, for as long as one of them lives, and differ in their batches.
_LIVE = weakref.WeakValueDictionary()


def _prepare_net(c, gen, seed):
    key = repr(sorted(c.items()))
    net, n = _LIVE.get(key), c["batch"]
    fresh = net is None
    if fresh:
        net = _LIVE[key] = _network(c, 0, seed)
    classes = net.output_size // n
    x = torch.randn(c["steps"], net.input_size, device="cuda", generator=gen)
    label = torch.zeros(c["steps"] * n, classes, device="cuda")
    label[torch.arange(len(label), device="cuda"), torch.randint(classes, (len(label),), device="cuda", generator=gen)] = 1
    trained = [(l, kind) for l in range(net.num_layers) for kind in (v.abi.TENSOR_WEIGHT, v.abi.TENSOR_BIAS) if net.tensor_size(l, kind)]
    for l, kind in trained:     # training resumes: biases are no longer the zeros of a new network
        if fresh and kind == v.abi.TENSOR_BIAS:
            net.write_tensor(l, kind, (torch.randn(net.tensor_size(l, kind), device="cuda", generator=gen) * 0.05).cpu().numpy())
    return {"net": net, "trained": trained, "x": x.cpu().pin_memory(), "label": label.view(c["steps"], -1).cpu().pin_memory()}


def _run_net(c, s):
    net, losses = s["net"], []
    for x, label in zip(s["x"], s["label"]):
        net.set_input(x, label)
        net.step()
        losses.append(net.loss())
    return {"loss": np.array(losses), "parameters": [net.read_tensor(l, kind) for l, kind in s["trained"]]}


# ----------------------------------------------------------------------------------------------------------- entry points

def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "net":
        s = _prepare_net(case, gen, seed)
    else:
        s = {"head": _prepare_head, "conv": _prepare_conv, "fc": _prepare_fc, "stage": _prepare_stage}[kind](case, gen)
    s["case"] = case
    return s


def run(state):
    case = state["case"]
    return {"head": _run_head, "conv": _run_conv, "fc": _run_fc, "stage": _run_stage, "net": _run_net}[case["kind"]](case, state)


def work(case):
    """Bytes: every input read once, every result written once.  Flops: 2 M N K for each of the three contractions of a layer.
    For a network the parameters are read and written and the batch is read in every step."""
    kind = case["kind"]
    if kind == "head":
        return {"bytes": 4.0 * case["rows"] * case["cols"] * 5 + 16, "flops": 0}
    if kind == "conv":
        p, q = _conv_dims(case)
        x, y = case["n"] * case["c"] * case["h"] * case["w"], case["n"] * case["k"] * p * q
        w = case["k"] * case["c"] * case["r"] ** 2
        return {"bytes": 4.0 * (2 * x + 2 * y + 2 * w + 2 * case["k"]), "flops": 6.0 * y * case["c"] * case["r"] ** 2}
    if kind == "fc":
        n, c, k = case["n"], case["c"], case["k"]
        return {"bytes": 4.0 * (2 * n * c + 2 * n * k + 2 * c * k + 2 * k), "flops": 6.0 * n * c * k}
    if kind == "stage":
        x = case["n"] * case["c"] * case["h"] * case["w"]
        p, q = _pool_dims(case)
        return {"bytes": 4.0 * (x * (6 if case["lrn"] else 4) + 2 * case["n"] * case["c"] * p * q), "flops": 0}
    net = _network(case, -1)
    flops, parameters = 0.0, 0
    for l, s in enumerate(net.layer_specs()):
        if s.type in (v.CONV, v.FC_CONV):
            p, q = v.ops.conv_out_dims(v.ops.conv_desc(s.n, s.c, s.h, s.w, s.k, s.r, s.s, (s.pad_h, s.pad_w), (s.stride_h, s.stride_w)))
            flops += 6.0 * s.n * s.k * p * q * s.c * s.r * s.s
        elif s.type == v.FC_GEMM:
            flops += 6.0 * s.n * s.k * s.c * s.h * s.w
        parameters += net.tensor_size(l, v.abi.TENSOR_WEIGHT) + net.tensor_size(l, v.abi.TENSOR_BIAS)
    return {"bytes": 4.0 * case["steps"] * (net.input_size + net.output_size + 2 * parameters), "flops": case["steps"] * flops}


def tolerance(case):
    """fp32 sums in another order; a gradient element of a long reduction may cancel to well below the tensor's typical size."""
    return {"rel": 1e-5, "max": 1e-3}

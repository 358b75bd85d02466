"""The work whose speed counts: what a training or inference program has this library do, as cases that can be timed.

A case is a dict of plain values.  "op" names the family:

  separable    depthwise 3x3 -> BN+ReLU -> 1x1 -> BN+ReLU, the block MobileNetV1 is made of, as the functional calls of a
               caller that drives the layers itself; forward with running statistics (inference) or forward and backward
  depthwise    one SpatialDepthWiseConvolution layer of a training step: output, input gradient, parameter gradients
  conv         one SpatialConvolutionMM / SpatialDilatedConvolution layer of a training step (a network's first layer has
               no input gradient)
  transposed   one SpatialFullConvolution layer of a training step
  batchnorm    one BatchNormalization layer: training forward and backward, or forward with running statistics
  maxpool      one SpatialMaxPooling layer of a training step, indices included
  mobilenet    one training step of a MobileNetV1 replica on its shard of the batch: forward, loss, backward, update

Everything is fp32 NCHW, the library's layout.  Programs keep a layer's output and gradient buffers from step to step, and
clear the gradient accumulators before each backward pass; both are so here.
"""
import math

import torch

from cunn_b200 import functional as F

DEV = "cuda"
EPS = 1e-5
RATE = 0.001     # learning rate of the training step


def listed():
    return [
        # The smallest work: one image through one block of a deployed network; latency and launches are what it costs.
        {"name": "separable_image", "op": "separable", "train": False, "N": 1, "C": 512, "H": 14, "W": 14, "K": 512, "stride": 1},
        # A block of a training step on maps that divide by nothing (crops, detection inputs) and a partial batch.
        {"name": "separable_train_odd", "op": "separable", "train": True, "N": 12, "C": 144, "H": 37, "W": 29, "K": 200, "stride": 1},
        # The largest depthwise maps of MobileNetV1 at 64 images a GPU.
        {"name": "depthwise_train", "op": "depthwise", "N": 64, "C": 32, "H": 112, "W": 112, "M": 1, "k": 3, "stride": 1, "pad": 1},
        # Depthwise layers that are not 3x3: wider windows, strided, ragged rows.
        {"name": "depthwise_5x5_odd", "op": "depthwise", "N": 32, "C": 96, "H": 57, "W": 43, "M": 1, "k": 5, "stride": 2, "pad": 2},
        # The ordinary convolutions of a classifier's body: 3x3 and 1x1 at 14x14, batch 128.
        {"name": "conv_3x3_train", "op": "conv", "N": 128, "C": 256, "H": 14, "W": 14, "K": 256, "k": 3, "stride": 1, "pad": 1,
         "dil": 1, "first": False},
        {"name": "conv_1x1_train", "op": "conv", "N": 128, "C": 1024, "H": 14, "W": 14, "K": 256, "k": 1, "stride": 1, "pad": 0,
         "dil": 1, "first": False},
        # A convolution that halves the map, as at the start of each stage of such a body.
        {"name": "conv_3x3_stride2_train", "op": "conv", "N": 64, "C": 128, "H": 56, "W": 56, "K": 256, "k": 3, "stride": 2, "pad": 1,
         "dil": 1, "first": False},
        # A 7x7 first layer on images: few channels, many taps, no input gradient.
        {"name": "conv_7x7_first", "op": "conv", "N": 32, "C": 3, "H": 224, "W": 224, "K": 64, "k": 7, "stride": 2, "pad": 3,
         "dil": 1, "first": True},
        # Upsampling by two, as generators and segmentation heads do it.
        {"name": "transposed_4x4_train", "op": "transposed", "N": 64, "C": 256, "H": 14, "W": 14, "K": 128, "k": 4, "stride": 2, "pad": 1},
        # Large normalisation and pooling layers of a training step.
        {"name": "batchnorm_train", "op": "batchnorm", "train": True, "N": 256, "C": 64, "H": 112, "W": 112},
        {"name": "maxpool_train", "op": "maxpool", "N": 256, "C": 64, "H": 112, "W": 112, "k": 3, "stride": 2, "pad": 1, "ceil": False},
        # A replica's whole step: the shard of 128 images that a GPU of eight takes of a batch of 1024.
        {"name": "mobilenet_step", "op": "mobilenet", "N": 128, "H": 224},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _channels(rng, lo, hi):
    """Most layers have channels in multiples of eight; some do not."""
    c = _log(rng, lo, hi)
    return c if rng.random() < 0.25 else max(8, c // 8 * 8)


def _map(rng, lo=7, hi=112):
    h = _log(rng, lo, hi)
    return h, h if rng.random() < 0.6 else max(lo, int(h * rng.uniform(0.6, 1.4)))


def _batch(rng, per_image, limit, hi=256):
    """A batch of 1 to `hi` images that keeps the work under `limit`."""
    return max(1, min(_log(rng, 1, hi), int(limit // max(per_image, 1))))


def draw(rng):
    op = rng.choice(["separable", "depthwise", "conv", "conv", "transposed", "batchnorm", "maxpool", "mobilenet"])
    h, w = _map(rng)
    if op == "separable":
        c, k, s = _channels(rng, 16, 1024), _channels(rng, 16, 1024), rng.choice([1, 1, 2])
        return {"op": op, "train": rng.random() < 0.6, "N": _batch(rng, max(c, k) * h * w, 1.5e7, 128), "C": c, "H": h, "W": w, "K": k,
                "stride": s}
    if op == "depthwise":
        c, k = _channels(rng, 16, 1024), rng.choice([3, 3, 3, 5, 7])
        m = rng.choice([1, 1, 1, 2])
        return {"op": op, "N": _batch(rng, c * m * h * w, 2.5e7), "C": c, "H": h, "W": w, "M": m, "k": k, "stride": rng.choice([1, 2]),
                "pad": k // 2}
    if op == "conv":
        first = rng.random() < 0.15
        k = rng.choice([3, 5, 7, 11]) if first else rng.choice([1, 1, 3, 3, 5])
        h, w = (h * 2, w * 2) if first else (h, w)
        s = rng.choice([2, 4]) if first else rng.choice([1, 1, 2])
        c, kk = (3, _channels(rng, 16, 128)) if first else (_channels(rng, 16, 1024), _channels(rng, 16, 1024))
        dil = 2 if not first and k == 3 and rng.random() < 0.2 else 1
        per = max(c * h * w * 40, kk * c * k * k * (h // s + 1) * (w // s + 1) / 20)
        return {"op": op, "N": _batch(rng, per, 1e9), "C": c, "H": h, "W": w, "K": kk, "k": k, "stride": s, "pad": dil * (k // 2),
                "dil": dil, "first": first}
    if op == "transposed":
        h, w = _map(rng, 4, 32)
        c, kk, k = _channels(rng, 16, 512), _channels(rng, 16, 512), rng.choice([2, 3, 4])
        return {"op": op, "N": _batch(rng, kk * c * k * k * h * w / 20, 1e9), "C": c, "H": h, "W": w, "K": kk, "k": k, "stride": 2,
                "pad": 0 if k == 2 else 1}
    if op == "batchnorm":
        c = _channels(rng, 8, 1024)
        return {"op": op, "train": rng.random() < 0.75, "N": _batch(rng, c * h * w, 2e8), "C": c, "H": h, "W": w}
    if op == "maxpool":
        c, k = _channels(rng, 8, 512), rng.choice([2, 3])
        return {"op": op, "N": _batch(rng, c * h * w, 2e8), "C": c, "H": h, "W": w, "k": k, "stride": 2, "pad": k // 2 if k == 3 else 0,
                "ceil": rng.random() < 0.3}
    return {"op": op, "N": _log(rng, 8, 128), "H": rng.choice([96, 128, 160, 192, 224])}


# ---- shapes ---------------------------------------------------------------------------------------------------------

def _out(size, k, stride, pad, dil=1):
    return (size + 2 * pad - (dil * (k - 1) + 1)) // stride + 1


def _conv_out(c):
    return tuple(_out(c[d], c["k"], c["stride"], c["pad"], c.get("dil", 1)) for d in "HW")


def _transposed_out(c):
    return tuple((c[d] - 1) * c["stride"] - 2 * c["pad"] + c["k"] for d in "HW")


def _pool_out(c):
    """Torch7's rule: with ceil_mode the last window must still start inside the input or its left padding."""
    out = []
    for d in "HW":
        span = c[d] + 2 * c["pad"] - c["k"]
        o = (-(-span // c["stride"]) if c["ceil"] else span // c["stride"]) + 1
        if c["pad"] and (o - 1) * c["stride"] >= c[d] + c["pad"]:
            o -= 1
        out.append(o)
    return tuple(out)


_NET_CHANNELS = (32, 64, 128, 128, 256, 256, 512, 512, 512, 512, 512, 512, 1024, 1024)
_NET_STRIDES = (1, 2, 1, 2, 1, 2, 1, 1, 1, 1, 1, 2, 1)
_NET_CLASSES = 1000


def _net_layers(H):
    """(C in, C out, kernel, stride, pad, groups, map in, map out) of every convolution, in parameter order."""
    rows, h = [], H

    def add(cin, cout, k, s, pad, groups):
        nonlocal h
        o = _out(h, k, s, pad)
        rows.append((cin, cout, k, s, pad, groups, h, o))
        h = o

    add(3, 32, 3, 2, 1, 1)
    for i, s in enumerate(_NET_STRIDES):
        add(_NET_CHANNELS[i], _NET_CHANNELS[i], 3, s, 1, _NET_CHANNELS[i])
        add(_NET_CHANNELS[i], _NET_CHANNELS[i + 1], 1, 1, 0, 1)
    return rows


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device=DEV)


def _uniform(g, bound, *shape):
    return (torch.rand(shape, generator=g, device=DEV) * 2 - 1) * bound


def _inputs(case, seed):
    """The tensors that a pass reads, by name."""
    g, c, op = _generator(seed), case, case["op"]
    if op == "separable":
        oh, ow = _out(c["H"], 3, c["stride"], 1), _out(c["W"], 3, c["stride"], 1)
        d = {"x": _normal(g, c["N"], c["C"], c["H"], c["W"]).relu_(),          # behind a ReLU, as inside a network
             "w1": _uniform(g, 1 / 3, 1, c["C"], 3, 3), "b1": _uniform(g, 1 / 3, 1, c["C"]),
             "w2": _uniform(g, c["C"] ** -0.5, c["K"], c["C"], 1, 1), "b2": _uniform(g, c["C"] ** -0.5, c["K"])}
        for i, n in ((1, c["C"]), (2, c["K"])):
            d["gamma%d" % i] = torch.rand(n, generator=g, device=DEV) + 0.5
            d["beta%d" % i] = _uniform(g, 0.5, n)
            d["rm%d" % i] = _uniform(g, 0.2, n)
            d["rv%d" % i] = torch.rand(n, generator=g, device=DEV) * 0.5 + 0.5
        if c["train"]:
            d["gy"] = _normal(g, c["N"], c["K"], oh, ow)
        return d
    if op == "depthwise":
        b = 1.0 / c["k"]
        return {"x": _normal(g, c["N"], c["C"], c["H"], c["W"]), "w": _uniform(g, b, c["M"], c["C"], c["k"], c["k"]),
                "b": _uniform(g, b, c["M"], c["C"]), "gy": _normal(g, c["N"], c["C"] * c["M"], *_conv_out(c))}
    if op == "conv":
        b = (c["C"] * c["k"] * c["k"]) ** -0.5
        return {"x": _normal(g, c["N"], c["C"], c["H"], c["W"]), "w": _uniform(g, b, c["K"], c["C"], c["k"], c["k"]),
                "b": _uniform(g, b, c["K"]), "gy": _normal(g, c["N"], c["K"], *_conv_out(c))}
    if op == "transposed":
        b = (c["C"] * c["k"] * c["k"]) ** -0.5
        return {"x": _normal(g, c["N"], c["C"], c["H"], c["W"]), "w": _uniform(g, b, c["C"], c["K"], c["k"], c["k"]),
                "b": _uniform(g, b, c["K"]), "gy": _normal(g, c["N"], c["K"], *_transposed_out(c))}
    if op == "batchnorm":
        n = c["C"]
        d = {"x": _normal(g, c["N"], n, c["H"], c["W"]).mul_(torch.rand(1, n, 1, 1, generator=g, device=DEV) + 0.5)
             .add_(_uniform(g, 1.0, 1, n, 1, 1)),
             "gamma": torch.rand(n, generator=g, device=DEV) + 0.5, "beta": _uniform(g, 0.5, n), "rm": _uniform(g, 0.5, n),
             "rv": torch.rand(n, generator=g, device=DEV) + 0.5}
        if c["train"]:
            d["gy"] = _normal(g, c["N"], n, c["H"], c["W"])
        return d
    if op == "maxpool":
        return {"x": _normal(g, c["N"], c["C"], c["H"], c["W"]), "gy": _normal(g, c["N"], c["C"], *_pool_out(c))}
    # mobilenet: images of unit scale, labels, the flat parameter buffer (weight, bias, gamma, beta per convolution, classifier)
    parts = []
    for cin, cout, k, _, _, groups, _, _ in _net_layers(c["H"]):
        fan = cin // groups * k * k
        parts += [_uniform(g, fan ** -0.5, cout * fan), _uniform(g, fan ** -0.5, cout),
                  torch.rand(cout, generator=g, device=DEV), torch.zeros(cout, device=DEV)]
    parts += [_uniform(g, 1024 ** -0.5, _NET_CLASSES * 1024), _uniform(g, 1024 ** -0.5, _NET_CLASSES)]
    return {"images": _normal(g, c["N"], 3, c["H"], c["H"]),
            "labels": torch.randint(1, _NET_CLASSES + 1, (c["N"],), generator=g, device=DEV),      # Lua counts from one
            "params": torch.cat(parts)}


def _grads(d, *names):
    """One flat accumulator, as a module's getParameters() lays it out, and a view of it for each parameter."""
    flat = torch.zeros(sum(d[n].numel() for n in names), device=DEV)
    views, at = {}, 0
    for n in names:
        views["g_" + n] = flat[at:at + d[n].numel()].view(d[n].shape)
        at += d[n].numel()
    return flat, views


def prepare(case, seed):
    c, op = case, case["op"]
    d = _inputs(c, seed)
    s = {"case": c, "in": d}
    if op == "mobilenet":
        from cunn_b200 import mobilenet as mb
        cfg = mb.Config(c["H"], 1, _NET_CLASSES)
        net = mb.MobileNetV1(cfg, torch.device(DEV, torch.cuda.current_device()), d.pop("params").cpu().numpy(), c["N"])
        s["net"], s["step"] = net, mb.DataParallelStep(net)
        return s
    if op == "separable" and c["train"]:
        s["flat"], s["g"] = _grads(d, "w1", "b1", "gamma1", "beta1", "w2", "b2", "gamma2", "beta2")
    elif op in ("depthwise", "conv", "transposed"):
        s["flat"], s["g"] = _grads(d, "w", "b")
        o = _transposed_out(c) if op == "transposed" else _conv_out(c)
        s["y"] = torch.empty_like(d["gy"])
        assert tuple(s["y"].shape[2:]) == o
        s["gx"] = torch.empty_like(d["x"])
    elif op == "batchnorm":
        s["y"] = torch.empty_like(d["x"])
        if c["train"]:
            s["flat"], s["g"] = _grads(d, "gamma", "beta")
            s["gx"] = torch.empty_like(d["x"])
            # statistics that training has settled: the running values are those of the batches
            var, mean = torch.var_mean(d["x"].double(), dim=(0, 2, 3), unbiased=d["x"].numel() > d["x"].shape[1])
            d["rm"], d["rv"] = mean.float(), var.float()
    elif op == "maxpool":
        s["y"] = torch.empty_like(d["gy"])
        s["ind"] = torch.empty(d["gy"].shape, dtype=torch.int64, device=DEV)
        s["gx"] = torch.empty_like(d["x"])
    if op == "separable":
        s["mid"] = [torch.empty((c["N"], n, _out(c["H"], 3, c["stride"], 1), _out(c["W"], 3, c["stride"], 1)), device=DEV)
                    for n in (c["C"], c["C"], c["K"], c["K"])]
        if c["train"]:
            s["gx"] = torch.empty_like(d["x"])
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------

def run(state):
    c, d = state["case"], state["in"]
    op = c["op"]
    if op == "separable":
        return _run_separable(state, c, d)
    if op == "depthwise":
        st, p, g = c["stride"], c["pad"], state["g"]
        state["flat"].zero_()
        y = F.dwconv_forward(d["x"], d["w"], d["b"], st, st, p, p, out=state["y"])
        gx = F.dwconv_grad_input(d["gy"], d["w"], c["H"], c["W"], st, st, p, p, out=state["gx"])
        F.dwconv_acc_grad(d["x"], d["gy"], g["g_w"], g["g_b"], st, st, p, p)
        return {"y": y, "gx": gx, **g}
    if op == "conv":
        st, p, dil, g = c["stride"], c["pad"], c["dil"], state["g"]
        state["flat"].zero_()
        geo = (st, st, p, p)
        if dil > 1:
            y = F.dilated_conv_forward(d["x"], d["w"], d["b"], *geo, dil, dil, out=state["y"])
            gx = F.dilated_conv_grad_input(d["gy"], d["w"], c["H"], c["W"], *geo, dil, dil, out=state["gx"])
            F.dilated_conv_acc_grad(d["x"], d["gy"], g["g_w"], g["g_b"], *geo, dil, dil)
            return {"y": y, "gx": gx, **g}
        y = F.convmm_forward(d["x"], d["w"], d["b"], *geo, out=state["y"])
        out = {"y": y}
        if not c["first"]:
            out["gx"] = F.convmm_grad_input(d["gy"], d["w"], c["H"], c["W"], *geo, out=state["gx"])
        F.convmm_acc_grad(d["x"], d["gy"], g["g_w"], g["g_b"], *geo)
        return {**out, **g}
    if op == "transposed":
        st, p, g = c["stride"], c["pad"], state["g"]
        state["flat"].zero_()
        y = F.full_conv_forward(d["x"], d["w"], d["b"], st, st, p, p, out=state["y"])
        gx = F.full_conv_grad_input(d["gy"], d["w"], c["H"], c["W"], st, st, p, p, out=state["gx"])
        F.full_conv_acc_grad(d["x"], d["gy"], g["g_w"], g["g_b"], st, st, p, p)
        return {"y": y, "gx": gx, **g}
    if op == "batchnorm":
        y, mean, std = F.batchnorm_forward(d["x"], d["gamma"], d["beta"], d["rm"], d["rv"], c["train"], 0.1, EPS, out=state["y"])
        if not c["train"]:
            return {"y": y}
        g = state["g"]
        state["flat"].zero_()
        gx = F.batchnorm_backward(d["x"], d["gy"], d["gamma"], d["rm"], d["rv"], mean, std, True, 1.0, EPS, g["g_gamma"], g["g_beta"],
                                  out=state["gx"])
        return {"y": y, "gx": gx, "mean": mean, "std": std, "running_mean": d["rm"], "running_var": d["rv"], **g}
    if op == "maxpool":
        k, st, p = c["k"], c["stride"], c["pad"]
        y, ind = F.maxpool_forward(d["x"], k, k, st, st, p, p, c["ceil"], out=state["y"], indices=state["ind"])
        gx = F.maxpool_backward(d["gy"], ind, c["H"], c["W"], k, k, st, st, p, p, c["ceil"], out=state["gx"])
        return {"y": y, "indices": ind, "gx": gx}
    loss = state["step"].train_step(d["images"], d["labels"], c["N"], RATE)
    return {"loss": loss, "params": state["net"].params, "bn_running": state["net"].bn_running}


def _run_separable(state, c, d):
    st = c["stride"]
    m1, a1, m2, a2 = state["mid"]
    train = c["train"]
    F.dwconv_forward(d["x"], d["w1"], d["b1"], st, st, 1, 1, out=m1)
    _, mean1, std1 = F.batchnorm_relu_forward(m1, d["gamma1"], d["beta1"], d["rm1"], d["rv1"], train, 0.1, EPS, out=a1)
    F.convmm_forward(a1, d["w2"], d["b2"], 1, 1, 0, 0, out=m2)
    _, mean2, std2 = F.batchnorm_relu_forward(m2, d["gamma2"], d["beta2"], d["rm2"], d["rv2"], train, 0.1, EPS, out=a2)
    if not train:
        return {"y": a2}
    g = state["g"]
    state["flat"].zero_()
    t = F.batchnorm_relu_backward(m2, d["gy"], d["gamma2"], d["beta2"], d["rm2"], d["rv2"], mean2, std2, True, 1.0, EPS, g["g_gamma2"],
                                  g["g_beta2"])
    F.convmm_acc_grad(a1, t, g["g_w2"], g["g_b2"], 1, 1, 0, 0)
    t = F.convmm_grad_input(t, d["w2"], m1.shape[2], m1.shape[3], 1, 1, 0, 0)
    t = F.batchnorm_relu_backward(m1, t, d["gamma1"], d["beta1"], d["rm1"], d["rv1"], mean1, std1, True, 1.0, EPS, g["g_gamma1"],
                                  g["g_beta1"])
    F.dwconv_acc_grad(d["x"], t, g["g_w1"], g["g_b1"], st, st, 1, 1)
    gx = F.dwconv_grad_input(t, d["w1"], c["H"], c["W"], st, st, 1, 1, out=state["gx"])
    # a bias in front of a normalisation has a gradient of zero but for rounding: it says nothing
    return {"y": a2, "gx": gx, "running": [d["rm1"], d["rv1"], d["rm2"], d["rv2"]],
            **{n: v for n, v in g.items() if n not in ("g_b1", "g_b2")}}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case):
    c, op = case, case["op"]
    if op == "separable":
        oh, ow = _out(c["H"], 3, c["stride"], 1), _out(c["W"], 3, c["stride"], 1)
        x, y = c["N"] * c["C"] * c["H"] * c["W"], c["N"] * c["K"] * oh * ow
        params = c["C"] * (9 + c["K"] + 5) + c["K"] * 5
        mults = c["N"] * oh * ow * c["C"] * (9 + c["K"])
        return {"bytes": 4 * ((x + y + params) * (2 if c["train"] else 1)), "flops": 2 * mults * (3 if c["train"] else 1)}
    if op == "depthwise":
        oh, ow = _conv_out(c)
        x, y, w = c["N"] * c["C"] * c["H"] * c["W"], c["N"] * c["C"] * c["M"] * oh * ow, c["C"] * c["M"] * (c["k"] ** 2 + 1)
        return {"bytes": 8 * (x + y + w), "flops": 6 * y * c["k"] ** 2}
    if op in ("conv", "transposed"):
        oh, ow = _conv_out(c) if op == "conv" else _transposed_out(c)
        x, y, w = c["N"] * c["C"] * c["H"] * c["W"], c["N"] * c["K"] * oh * ow, c["C"] * c["K"] * c["k"] ** 2 + c["K"]
        first = c.get("first", False)
        pixels = oh * ow if op == "conv" else c["H"] * c["W"]
        mults = c["N"] * pixels * c["C"] * c["K"] * c["k"] ** 2
        return {"bytes": 4 * (x * (1 if first else 2) + 2 * y + 2 * w), "flops": 2 * mults * (2 if first else 3)}
    if op == "batchnorm":
        n = c["N"] * c["C"] * c["H"] * c["W"]
        return {"bytes": 4 * n * (4 if c["train"] else 2), "flops": (14 if c["train"] else 2) * n}
    if op == "maxpool":
        oh, ow = _pool_out(c)
        x, y = c["N"] * c["C"] * c["H"] * c["W"], c["N"] * c["C"] * oh * ow
        return {"bytes": 8 * x + 16 * y, "flops": y * c["k"] ** 2 + y}
    mults, acts, params = 0, 0, _NET_CLASSES * 1025
    for cin, cout, k, _, _, groups, hin, hout in _net_layers(c["H"]):
        mults += cin // groups * k * k * cout * hout * hout
        acts += cout * hout * hout
        params += cin // groups * k * k * cout + 3 * cout
    # forward writes what the backward pass reads again: each convolution's result
    return {"bytes": 4 * (c["N"] * (3 * c["H"] ** 2 + 2 * acts) + 2 * params), "flops": 6 * c["N"] * mults}


def tolerance(case):
    op = case["op"]
    if op == "mobilenet":
        # A value next to a ReLU's zero falls on either side of it by the last bit, and its gradient with it: two correct
        # implementations are 1 to 2 per cent apart in the gradients, which the learning rate scales before they reach the weights.
        return {"rel": 3e-3, "max": 0.9}
    if op == "separable" and case["train"]:
        return {"rel": 5e-3, "max": 0.9}       # the same, with a value or two of a pass on the other side
    if op == "maxpool":
        return {"rel": 1e-6, "max": 1e-5, "differ": 0.0}
    if op in ("conv", "transposed"):
        return {"rel": 1e-4, "max": 2e-3}      # long sums: weight gradients over 400,000 pixels are up to 2.2e-5 off
    return {"rel": 1e-5, "max": 1e-4}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------

def _leaf(t):
    return t.double().requires_grad_(True)


def _bn_relu(x, gamma, beta, rm, rv, train):
    if train:
        var, mean = torch.var_mean(x, dim=(0, 2, 3), unbiased=False)
    else:
        mean, var = rm.double(), rv.double()
    y = (x - mean.view(1, -1, 1, 1)) * ((var + EPS).rsqrt() * gamma).view(1, -1, 1, 1) + beta.view(1, -1, 1, 1)
    return y.relu(), mean.detach(), var.detach()


def _settle(rm, rv, mean, var, count):
    return [0.9 * rm.double() + 0.1 * mean, 0.9 * rv.double() + 0.1 * var * count / max(count - 1, 1)]


def exact(case, seed):
    c, op = case, case["op"]
    conv = torch.nn.functional.conv2d
    d = _inputs(c, seed)
    if op == "separable":
        with torch.set_grad_enabled(c["train"]):
            names = ("w1", "b1", "gamma1", "beta1", "w2", "b2", "gamma2", "beta2")
            p = {n: _leaf(d[n]) for n in names}
            x = _leaf(d["x"])
            m1 = conv(x, p["w1"].view(c["C"], 1, 3, 3), p["b1"].view(-1), c["stride"], 1, 1, c["C"])
            a1, mean1, var1 = _bn_relu(m1, p["gamma1"], p["beta1"], d["rm1"], d["rv1"], c["train"])
            m2 = torch.einsum("kc,nchw->nkhw", p["w2"].view(c["K"], c["C"]), a1) + p["b2"].view(1, -1, 1, 1)
            a2, mean2, var2 = _bn_relu(m2, p["gamma2"], p["beta2"], d["rm2"], d["rv2"], c["train"])
        if not c["train"]:
            return {"y": a2}
        wanted = [n for n in names if n not in ("b1", "b2")]
        got = torch.autograd.grad(a2, [x] + [p[n] for n in wanted], d["gy"].double())
        count = m1.shape[0] * m1.shape[2] * m1.shape[3]
        return {"y": a2, "gx": got[0],
                "running": _settle(d["rm1"], d["rv1"], mean1, var1, count) + _settle(d["rm2"], d["rv2"], mean2, var2, count),
                **{"g_" + n: t for n, t in zip(wanted, got[1:])}}
    if op == "depthwise":
        x, w, b = _leaf(d["x"]), _leaf(d["w"]), _leaf(d["b"])
        # filter j of channel c gives output channel c * M + j
        y = conv(x, w.transpose(0, 1).reshape(c["C"] * c["M"], 1, c["k"], c["k"]), b.t().reshape(-1), c["stride"], c["pad"], 1, c["C"])
        gx, gw, gb = torch.autograd.grad(y, (x, w, b), d["gy"].double())
        return {"y": y, "gx": gx, "g_w": gw, "g_b": gb}
    if op in ("conv", "transposed"):
        x, w, b = _leaf(d["x"]), _leaf(d["w"]), _leaf(d["b"])
        if op == "conv":
            y = conv(x, w, b, c["stride"], c["pad"], c["dil"])
        else:
            y = torch.nn.functional.conv_transpose2d(x, w, b, c["stride"], c["pad"])
        gx, gw, gb = torch.autograd.grad(y, (x, w, b), d["gy"].double())
        return {"y": y, **({} if c.get("first") else {"gx": gx}), "g_w": gw, "g_b": gb}
    if op == "batchnorm":
        x = d["x"].double()
        if not c["train"]:
            scale = d["gamma"].double() * (d["rv"].double() + EPS).rsqrt()
            return {"y": (x - d["rm"].double().view(1, -1, 1, 1)) * scale.view(1, -1, 1, 1) + d["beta"].double().view(1, -1, 1, 1)}
        count = x.numel() // x.shape[1]
        var, mean = torch.var_mean(x, dim=(0, 2, 3), unbiased=False)
        std = (var + EPS).rsqrt()
        h = (x - mean.view(1, -1, 1, 1)) * std.view(1, -1, 1, 1)
        gy = d["gy"].double()
        gb, gg = gy.sum((0, 2, 3)), (gy * h).sum((0, 2, 3))
        gx = (gy - (gb / count).view(1, -1, 1, 1) - h * (gg / count).view(1, -1, 1, 1)) * (std * d["gamma"].double()).view(1, -1, 1, 1)
        y = h * d["gamma"].double().view(1, -1, 1, 1) + d["beta"].double().view(1, -1, 1, 1)
        # the running values were those of this batch before the pass, and stay so
        return {"y": y, "gx": gx, "mean": mean, "std": std, "running_mean": mean, "running_var": var * count / max(count - 1, 1),
                "g_gamma": gg, "g_beta": gb}
    if op == "maxpool":
        x = _leaf(d["x"])
        y, ind = torch.nn.functional.max_pool2d(x, c["k"], c["stride"], c["pad"], 1, c["ceil"], return_indices=True)
        gx, = torch.autograd.grad(y, x, d["gy"].double())
        return {"y": y, "indices": ind + 1, "gx": gx}
    # The forward pass on 64-bit values.  The weights after the step have no value that rounding approaches: one ReLU that
    # falls the other way moves every gradient in front of it.
    flat, at = d["params"].double(), 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return flat[at - n:at].view(shape)

    h, running = d["images"].double(), []
    for cin, cout, k, s, pad, groups, _, _ in _net_layers(c["H"]):
        w, b, gamma, beta = take(cout, cin // groups, k, k), take(cout), take(cout), take(cout)
        if k == 1:
            h = torch.einsum("kc,nchw->nkhw", w.view(cout, cin), h) + b.view(1, -1, 1, 1)
        else:
            h = conv(h, w, b, s, pad, 1, groups)
        count = h.numel() // cout
        h, mean, var = _bn_relu(h, gamma, beta, None, None, True)
        running += [0.1 * mean, 0.9 + 0.1 * var * count / max(count - 1, 1)]
    logits = h.mean((2, 3)) @ take(_NET_CLASSES, 1024).t() + take(_NET_CLASSES)
    loss = torch.nn.functional.cross_entropy(logits, d["labels"] - 1)
    return {"loss": loss.view(1), "params": None, "bn_running": torch.cat(running)}

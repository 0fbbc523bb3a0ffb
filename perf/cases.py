"""The work a user has this framework do, as a list of cases that a timing program can run.

A case is a dict of plain values; `prepare` builds what a program holds before the call (inputs,
compressed filters, chains), `run` is one pass through the public entry points.  The kinds:

  layer     one sparse (or depthwise) convolution on device tensors: sparse_conv2d[_fused]
  model     the conv layers of a network launched one after the other on their own inputs, the
            step that bench.py times
  chain     the conv stack of a network as a LayerChain, run eagerly or replayed as one CUDA graph
  host      host arrays in, host arrays out: cuda_sparse_conv2d (blocking, ordinary memory) or
            cuda_sparse_conv2d_async over four slots (page-locked memory)
  compress  a dense filter into its compressed forms, and those read back
  layout    NCHW -> NHWC -> NCHW on the device

Weights are N(0, 0.05) with a random zero mask, activations uniform[0, 1) with half of the entries
zero (what a ReLU leaves), as in the workload module; a chain's weights are scaled so that its
activations keep their magnitude from layer to layer.  Everything is made on the GPU from the seed.
"""
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_PKG = "tetris-artifact-evalution_b200"


def _package():
    if "tetris_b200" not in sys.modules:
        here = os.path.join(os.getcwd(), _PKG)
        spec = importlib.util.spec_from_file_location(
            "tetris_b200", os.path.join(here, "__init__.py"), submodule_search_locations=[here])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tetris_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tetris_b200"]


def _workloads():
    _package()
    return importlib.import_module("tetris_b200.workloads")


def _layer(n, h, w, ic, oc, ks, stride=1, sparsity=0.9, groups=1, pad=None, relu=False, tuned=False, deterministic=False):
    return {"kind": "layer", "n": n, "h": h, "w": w, "ic": ic, "oc": oc, "ks": ks, "stride": stride,
            "pad": ks // 2 if pad is None else pad, "groups": groups, "sparsity": sparsity, "relu": relu,
            "tuned": tuned, "deterministic": deterministic}


def listed():
    return [
        # the single-layer configuration at one image: the smallest call, where latency is all
        dict(_layer(1, 56, 56, 64, 64, 3), name="layer 3x3 64 b1"),
        # the last layer of YOLOv3's first detection head: 1x1, 255 channels (no multiple of
        # anything) on a 13x13 image
        dict(_layer(8, 13, 13, 1024, 255, 1, sparsity=0.875), name="layer 1x1 head 255 b8"),
        # a downsampling layer of YOLOv3 with its activation fused, chosen by the tuner
        dict(_layer(16, 104, 104, 128, 256, 3, stride=2, sparsity=0.875, relu=True, tuned=True), name="layer 3x3 s2 b16"),
        # the benchmark's step: every conv layer of VGG-19 on 16 images
        {"kind": "model", "net": "vgg19", "batch": 16, "size": 224, "tuned": True, "name": "model vgg19 b16"},
        # 53 layers, most of them 1x1: the network with the most launches per step
        {"kind": "model", "net": "resnet50", "batch": 16, "size": 224, "tuned": True, "name": "model resnet50 b16"},
        # serving one image: the forward pass of the conv stack as one CUDA graph
        {"kind": "chain", "net": "vgg19", "batch": 1, "size": 224, "graph": True, "name": "chain vgg19 b1 graph"},
        # depthwise and 1x1 layers in turn, bound by memory, a full batch
        {"kind": "chain", "net": "mobilenet", "batch": 16, "size": 224, "graph": True, "name": "chain mobilenet b16 graph"},
        # the same network on one image without a graph: launches and host work
        {"kind": "chain", "net": "mobilenet", "batch": 1, "size": 224, "graph": False, "name": "chain mobilenet b1 eager"},
        # the reference's own call: ordinary host arrays in and out, one layer
        {"kind": "host", "n": 8, "h": 28, "w": 28, "ic": 128, "oc": 128, "ks": 3, "stride": 1, "pad": 1,
         "sparsity": 0.8, "calls": 1, "pipelined": False, "name": "host blocking 28x28 b8"},
        # batches streamed from page-locked memory over the four pipeline slots
        {"kind": "host", "n": 8, "h": 56, "w": 56, "ic": 64, "oc": 64, "ks": 3, "stride": 1, "pad": 1,
         "sparsity": 0.8, "calls": 8, "pipelined": True, "name": "host pipelined 56x56 b8"},
        # loading a model: one of VGG-19's large filters
        {"kind": "compress", "ic": 512, "oc": 512, "ks": 3, "sparsity": 0.9, "name": "compress 512x512x3x3"},
        # a PyTorch tensor (NCHW) into the engine's layout and back
        {"kind": "layout", "n": 16, "c": 128, "h": 112, "w": 112, "name": "layout 128x112x112 b16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _channels(rng, lo, hi):
    """Channel counts: mostly multiples of 32 or 8 as in the networks, odd ones among them."""
    c = _log_int(rng, lo, hi)
    step = rng.choice([32, 32, 32, 8, 8, 1])
    return max(lo, min(hi, (c + step - 1) // step * step))


def _extent(size, ks, stride, pad):
    return (size + 2 * pad - ks) // stride + 1


def _draw_conv(rng):
    """A conv shape no costlier than the largest layers of VGG-19 at batch 16."""
    while True:
        n, h = _log_int(rng, 1, 16), _log_int(rng, 7, 224)
        w = h if rng.random() < 0.7 else _log_int(rng, 7, 224)
        ks = rng.choice([1, 1, 3, 3, 3, 5])
        stride = rng.choice([1, 1, 1, 2])
        ic, oc = _channels(rng, 16, 1024), _channels(rng, 16, 1024)
        if rng.random() < 0.1:  # a stem
            ic, ks, stride = 3, rng.choice([3, 7]), rng.choice([1, 2])
        pad = ks // 2
        oh, ow = _extent(h, ks, stride, pad), _extent(w, ks, stride, pad)
        if 2.0 * n * oh * ow * oc * ic * ks * ks <= 60e9 and 4.0 * n * (h * w * ic + oh * ow * oc) <= 410e6:
            sparsity = 0.5 if ic == 3 else round(rng.uniform(0.7, 0.97), 3)
            return n, h, w, ic, oc, ks, stride, pad, sparsity


def draw(rng):
    kind = rng.choice(["layer"] * 7 + ["depthwise", "model", "chain", "chain", "host", "host", "compress", "layout"])
    if kind == "layer":
        n, h, w, ic, oc, ks, stride, pad, sparsity = _draw_conv(rng)
        return _layer(n, h, w, ic, oc, ks, stride, sparsity, 1, pad, rng.random() < 0.3, rng.random() < 0.5, rng.random() < 0.1)
    if kind == "depthwise":
        while True:
            n, h, c, stride = _log_int(rng, 1, 16), _log_int(rng, 7, 224), _channels(rng, 16, 1024), rng.choice([1, 2])
            if 8.0 * n * h * h * c <= 410e6:
                return _layer(n, h, h, c, c, 3, stride, 0.0, c, 1, rng.random() < 0.5)
    if kind == "model":
        return {"kind": "model", "net": rng.choice(["vgg19", "resnet50", "mobilenet"]), "batch": _log_int(rng, 1, 16),
                "size": rng.randint(96, 224), "tuned": rng.random() < 0.5}
    if kind == "chain":
        return {"kind": "chain", "net": rng.choice(["vgg19", "mobilenet"]), "batch": _log_int(rng, 1, 16),
                "size": rng.randint(96, 224), "graph": rng.random() < 0.5}
    if kind == "host":
        while True:
            n, h, w, ic, oc, ks, stride, pad, sparsity = _draw_conv(rng)
            pipelined = rng.random() < 0.5
            if 4.0 * n * (h * w * ic + _extent(h, ks, stride, pad) * _extent(w, ks, stride, pad) * oc) <= 26e6:
                return {"kind": "host", "n": n, "h": h, "w": w, "ic": ic, "oc": oc, "ks": ks, "stride": stride, "pad": pad,
                        "sparsity": sparsity, "calls": rng.randint(4, 8) if pipelined else 1, "pipelined": pipelined}
    if kind == "compress":
        while True:
            ic, oc, ks = _channels(rng, 16, 1024), _channels(rng, 16, 1024), rng.choice([1, 3, 3, 5])
            if ic * oc * ks * ks <= 512 * 512 * 9:
                return {"kind": "compress", "ic": ic, "oc": oc, "ks": ks, "sparsity": round(rng.uniform(0.7, 0.97), 3)}
    while True:
        n, c, h, w = _log_int(rng, 1, 16), _channels(rng, 3, 1024), _log_int(rng, 7, 224), _log_int(rng, 7, 224)
        if 4.0 * n * c * h * w <= 103e6:
            return {"kind": "layout", "n": n, "c": c, "h": h, "w": w}


# ---- the networks, at any image size ------------------------------------------------------------
_POOL_AFTER = {"vgg19": {1, 3, 7, 11}, "mobilenet": set()}


def _net(case):
    """[(layer, relu, pool)] of the case's network, extents worked out for its image size."""
    wl, size = _workloads(), case["size"]
    layers = {"vgg19": wl.vgg19, "resnet50": wl.resnet50, "mobilenet": wl.mobilenet_v1}[case["net"]]()
    got, at = [], size
    for i, L in enumerate(layers):
        if case["net"] == "resnet50":  # branches: each layer's extent is its share of the image's
            at = -(-L.H * size // 224)
        sparsity = 0.875 if L.sparsity is None else L.sparsity
        got.append((L._replace(H=at, W=at, sparsity=sparsity), i in _POOL_AFTER.get(case["net"], ())))
        at = _extent(at, L.KS, L.stride, L.pad) // (2 if got[-1][1] else 1)
    return got


def _costs(L, batch):
    """(flops, input bytes, output bytes, weight bytes) of one layer launch."""
    oh, ow = _extent(L.H, L.KS, L.stride, L.pad), _extent(L.W, L.KS, L.stride, L.pad)
    size = L.OC * (L.IC if L.groups == 1 else 1) * L.KS * L.KS
    nnz = size * (1.0 - L.sparsity)
    return (2.0 * nnz * batch * oh * ow, 4.0 * batch * L.IC * L.H * L.W, 4.0 * batch * L.OC * oh * ow,
            8.0 * nnz + 4.0 * (L.OC + 1) if L.groups == 1 else 4.0 * size)


def _as_layer(case):
    return _workloads().Layer("layer", case["h"], case["w"], case["ic"], case["oc"], case["ks"], case["pad"], case["stride"],
                              case.get("groups", 1), case["sparsity"])


# ---- tensors ------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _weights(g, L, std=0.05, mask=None):
    """Dense OIHW float32 host array, `sparsity` of it zero; `mask`: generator of the zero mask."""
    shape = (L.OC, L.IC if L.groups == 1 else 1, L.KS, L.KS)
    w = torch.randn(shape, generator=g, device="cuda") * std
    w[w == 0] = std  # a drawn exact zero would blur the nonzero count
    if L.sparsity > 0:
        w *= torch.rand(shape, generator=mask or g, device="cuda") >= L.sparsity
    return w.cpu().numpy()


def _activations(g, *shape):
    x = torch.rand(shape, generator=g, device="cuda")
    return x * (torch.rand(shape, generator=g, device="cuda") >= 0.5)


def _prepare_layer(tb, g, L, n, stream, tuned, deterministic=False):
    f = tb.SparseFilter(_weights(g, L), L.IC, L.OC, L.KS, groups=L.groups, deterministic=deterministic)
    x = _activations(g, n, L.H, L.W, L.IC)
    y = torch.empty(n, _extent(L.H, L.KS, L.stride, L.pad), _extent(L.W, L.KS, L.stride, L.pad), L.OC, device="cuda")
    if tuned:
        tb.tune_sparse_conv2d(f, x, y, n, L.H, L.W, L.stride, L.pad, cuda_stream=stream)
    return (f, x, y, n, L.H, L.W, L.stride, L.pad)


class _DeviceArray:
    """The chain's output buffer as torch sees it (no copy); the tensor made from it keeps the
    chain, which owns that buffer, alive."""

    def __init__(self, chain, address, shape):
        self.chain = chain
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (address, False), "version": 3}


def prepare(case, seed):
    tb, g, kind = _package(), _generator(seed), case["kind"]
    stream = torch.cuda.current_stream()
    state = {"tb": tb, "case": case, "stream": stream}
    if kind == "layer":
        state["launch"] = _prepare_layer(tb, g, _as_layer(case), case["n"], stream, case["tuned"], case["deterministic"])
    elif kind == "model":
        state["launches"] = [_prepare_layer(tb, g, L, case["batch"], stream, case["tuned"]) for L, _ in _net(case)]
    elif kind == "chain":
        layers = []
        for L, pool in _net(case):
            fan_in = (L.IC if L.groups == 1 else 1) * L.KS * L.KS * (1.0 - L.sparsity)
            f = tb.SparseFilter(_weights(g, L, math.sqrt(2.0 / fan_in)), L.IC, L.OC, L.KS, groups=L.groups)
            layers.append((f, L.stride, L.pad, True, 2 if pool else 0))
        state["layers"] = layers
        state["input"] = _activations(g, case["batch"], case["size"], case["size"], 3)
        state["chain"] = tb.LayerChain(layers, case["batch"], case["size"], case["size"])
        address, h, w, c = state["chain"].output()
        state["output"] = torch.as_tensor(_DeviceArray(state["chain"], address, (case["batch"], h, w, c)), device="cuda")
        torch.cuda.synchronize()
        if case["graph"]:
            state["chain"].capture(state["input"])
    elif kind == "host":
        L = _as_layer(case)
        state["filter"] = tb.SparseFilter(_weights(g, L), L.IC, L.OC, L.KS)
        oh, ow = _extent(L.H, L.KS, L.stride, L.pad), _extent(L.W, L.KS, L.stride, L.pad)
        state["in"] = [_activations(g, case["n"], L.IC, L.H, L.W).cpu() for _ in range(case["calls"])]
        if case["pipelined"]:
            state["in"] = [x.pin_memory() for x in state["in"]]
            state["pinned_out"] = [torch.empty(case["n"], L.OC, oh, ow).pin_memory() for _ in state["in"]]
            state["out"] = [y.numpy() for y in state["pinned_out"]]
        state["pinned_in"], state["in"] = state["in"], [x.numpy() for x in state["in"]]
    elif kind == "compress":
        # the zero mask belongs to the case (the lengths of the compressed forms follow from it),
        # the values to the seed
        L = _workloads().Layer("filter", 1, 1, case["ic"], case["oc"], case["ks"], 0, 1, 1, case["sparsity"])
        state["weights"] = _weights(g, L, mask=_generator(0))
    else:
        n, c, h, w = case["n"], case["c"], case["h"], case["w"]
        state["nchw"] = _activations(g, n, c, h, w)
        state["nhwc"] = torch.empty(n, h, w, c, device="cuda")
        state["back"] = torch.empty(n, c, h, w, device="cuda")
    return state


def run(state):
    tb, case, kind = state["tb"], state["case"], state["case"]["kind"]
    if kind == "layer":
        if case["relu"]:
            tb.sparse_conv2d_fused(*state["launch"], cuda_stream=state["stream"])
        else:
            tb.sparse_conv2d(*state["launch"], cuda_stream=state["stream"])
        return state["launch"][2]
    if kind == "model":
        for launch in state["launches"]:
            tb.sparse_conv2d(*launch, cuda_stream=state["stream"])
        return [launch[2] for launch in state["launches"]]
    if kind == "chain":
        if case["graph"]:
            state["chain"].replay(cuda_stream=state["stream"])
        else:
            state["chain"].run(state["input"], cuda_stream=state["stream"])
        return state["output"]
    if kind == "host":
        shape = (case["n"], case["h"], case["w"], case["stride"], case["pad"])
        if not case["pipelined"]:
            return tb.cuda_sparse_conv2d(state["in"][0], state["filter"], *shape)
        for i, (x, y) in enumerate(zip(state["in"], state["out"])):
            tb.host_sync(0, i % 4)
            tb.cuda_sparse_conv2d_async(x, state["filter"], *shape, y, slot=i % 4)
        tb.host_sync(0, -1)
        return state["out"]
    if kind == "compress":
        f = tb.SparseFilter(state["weights"], case["ic"], case["oc"], case["ks"])
        forms = [a.view(np.int64) if a.dtype == np.uint64 else a for a in f.download() + f.download_lists()]
        f.close()
        return forms
    n, c, h, w = case["n"], case["c"], case["h"], case["w"]
    tb.nchw_to_nhwc(state["nchw"], state["nhwc"], n, c, h, w, cuda_stream=state["stream"])
    tb.nhwc_to_nchw(state["nhwc"], state["back"], n, c, h, w, cuda_stream=state["stream"])
    return state["nhwc"], state["back"]


def work(case):
    """What a pass cannot do without: inputs and weights read once, outputs written once, two
    operations per nonzero weight and output pixel.  A chain's activations between its layers are
    not among its inputs or outputs."""
    kind = case["kind"]
    if kind == "layer":
        flops, i, o, w = _costs(_as_layer(case), case["n"])
        return {"bytes": i + o + w, "flops": flops}
    if kind == "model":
        costs = [_costs(L, case["batch"]) for L, _ in _net(case)]
        return {"bytes": sum(i + o + w for _, i, o, w in costs), "flops": sum(c[0] for c in costs)}
    if kind == "chain":
        net = _net(case)
        costs = [_costs(L, case["batch"]) for L, _ in net]
        return {"bytes": costs[0][1] + costs[-1][2] + sum(c[3] for c in costs), "flops": sum(c[0] for c in costs)}
    if kind == "host":
        flops, i, o, w = _costs(_as_layer(case), case["n"])
        return {"bytes": case["calls"] * (i + o + w), "flops": case["calls"] * flops}
    if kind == "compress":  # the dense filter in, both compressed forms (8 bytes per nonzero each) out
        size = case["ic"] * case["oc"] * case["ks"] ** 2
        return {"bytes": 4.0 * size + 16.0 * size * (1.0 - case["sparsity"]), "flops": 0.0}
    return {"bytes": 4 * 4.0 * case["n"] * case["c"] * case["h"] * case["w"], "flops": 0.0}


def tolerance(case):
    if case["kind"] in ("compress", "layout"):
        return "exact"
    # 32-bit sums of a few thousand products; over a chain the layers' rounding adds up
    return {"rel": 3e-5 if case["kind"] == "chain" else 1e-5}

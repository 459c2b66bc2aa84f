"""The work that users of this framework have it do, as cases that can be timed.

Two kinds of cases, both through the public interface (``darknet_b200`` and the C ABI behind it):

* ``network``: a whole network, as the reference's programs use it.  ``call`` says how it is driven:
  ``predict`` is network_predict on a host image batch (the detector and classifier commands; the batch is ordinary
  ``calloc`` memory there, "pageable", or page-locked where the caller cares), ``stream`` is two batches in flight
  through submit / collect (a validation loop), ``forward`` is the device-resident pass whose outputs are handed to
  device buffers in Darknet's layout (what an attached Darknet process does with the whole network), with or without
  CUDA-graph replay.
* ``layer``: one layer entry point on device tensors, as an attached Darknet process (NCHW float tensors) or a program
  that builds its own pipeline (channels-last tensors) calls it.

Networks, image sizes and batches are those of the benchmark and the tests: YOLOv3 at 608 and its smaller input sizes
(multiples of 32 from 320 up), YOLOv3-tiny, ResNet-50 and Darknet-19 at 224 and 256; layers are shapes inside them.
Parameters are seeded He-normal weights with batchnorm statistics, images are uniform in [0, 1).
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import darknet_b200 as dn
from darknet_b200 import synth

MODES = {"tf32": dn.MODE_TF32, "bf16": dn.MODE_BF16, "fp32": dn.MODE_FP32}


# ---------------------------------------------------------------------------------------------------- the cases
def _network(name, net, size, batch, mode, call, host="", graph=False):
    return {"name": name, "kind": "network", "net": net, "size": size, "batch": batch, "mode": mode, "call": call, "host": host, "graph": graph}


def _conv(name, b, c, hw, n, size, stride, groups, mode, layout, act="leaky"):
    return {"name": name, "kind": "layer", "op": "conv", "batch": b, "c": c, "hw": hw, "n": n, "size": size, "stride": stride,
            "groups": groups, "mode": mode, "layout": layout, "act": act}


def _mem(name, op, b, c, hw, layout, dtype):
    return {"name": name, "kind": "layer", "op": op, "batch": b, "c": c, "hw": hw, "layout": layout, "dtype": dtype}


def listed():
    return [
        # a webcam or single-image detector on the small network: one image per call, latency is what its user sees
        _network("tiny416 b1 predict", "yolov3-tiny", 416, 1, "tf32", "predict", host="pageable"),
        # detection on frames that a decoder left on the GPU, one at a time, replayed as a CUDA graph
        _network("yolov3-608 b1 graph", "yolov3", 608, 1, "tf32", "forward", graph=True),
        # a detection service with small batches, reduced input size and precision, images in ordinary host memory
        _network("yolov3-416 b8 bf16 predict", "yolov3", 416, 8, "bf16", "predict", host="pageable"),
        # the validation loop of the detector: full-size batches of the headline benchmark, two in flight
        _network("yolov3-608 b64 stream", "yolov3", 608, 64, "tf32", "stream", host="pinned"),
        # classification of a large set, device-resident (the benchmark's batch)
        _network("resnet50-224 b256 forward", "resnet50", 224, 256, "tf32", "forward"),
        # the binarised classifier at the benchmark's batch
        _network("darknet19x-224 b128 forward", "darknet19-xnor", 224, 128, "tf32", "forward"),
        # classification of one image per call
        _network("resnet50-256 b1 predict", "resnet50", 256, 1, "tf32", "predict", host="pageable"),
        # a layer of an attached Darknet process: NCHW in, NCHW out (Darknet-53's middle stage)
        _conv("conv3x3 nchw", 16, 256, 52, 512, 3, 1, 1, "tf32", "nchw"),
        # a bottleneck layer in a channels-last pipeline, bf16
        _conv("conv1x1 nhwc bf16", 64, 512, 52, 256, 1, 1, 1, "bf16", "nhwc"),
        # the full-precision mode (and grouped layers, in the drawn cases): exact cross-checks, ResNeXt-style layers
        _conv("conv3x3 fp32", 8, 64, 104, 128, 3, 1, 1, "fp32", "nchw"),
        # the memory-bound layers; the largest map of the 2x2 pooling chain
        _mem("maxpool nhwc f32", "maxpool", 64, 128, 152, "nhwc", "f32"),
        # the classifier's tail, one image: the smallest call there is
        _mem("softmax b1", "softmax", 1, 1000, 1, "nhwc", "f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _strip(case):
    case.pop("name")
    return case


def draw(rng):
    what = rng.randrange(12)
    yolo_size = 32 * rng.randint(10, 19)
    mode = rng.choice(["tf32", "tf32", "bf16"])
    host = rng.choice(["pageable", "pinned"])
    if what == 0:
        return _strip(_network("", "yolov3-tiny", yolo_size, _log(rng, 1, 32), mode, "predict", host))
    if what == 1:
        return _strip(_network("", rng.choice(["yolov3", "yolov3", "yolov3-tiny"]), yolo_size, _log(rng, 1, 16), mode, "forward", graph=True))
    if what == 2:
        return _strip(_network("", "yolov3", yolo_size, _log(rng, 1, 24), mode, "predict", host))
    if what == 3:
        return _strip(_network("", "yolov3", yolo_size, _log(rng, 8, 64), mode, "stream", "pinned"))
    if what == 4:
        return _strip(_network("", "resnet50", rng.choice([224, 256]), _log(rng, 1, 192), mode, "forward", graph=rng.random() < 0.5))
    if what == 5:
        return _strip(_network("", "darknet19-xnor", rng.choice([192, 224, 256]), _log(rng, 1, 128), "tf32", "forward", graph=rng.random() < 0.5))
    if what == 6:
        return _strip(_network("", rng.choice(["resnet50", "darknet19"]), rng.choice([224, 256]), _log(rng, 1, 64), mode, "predict", host))
    if what in (7, 8, 9):
        hw = rng.choice([7, 13, 14, 19, 26, 28, 38, 52, 56, 76, 104, 112, 152, _log(rng, 7, 152)])
        size = rng.choice([1, 3, 3])
        stride = rng.choice([1, 1, 1, 2]) if size == 3 else 1
        if what == 9:
            groups = rng.choice([1, 1, 2, 32])
            c = 32 * _log(rng, 1, 16) if groups == 32 else 2 * _log(rng, 8, 256)
            n = 32 * _log(rng, 1, 16) if groups == 32 else 2 * _log(rng, 8, 256)
            cmode, most, layout = "fp32", 3e10, rng.choice(["nchw", "nhwc"])
        else:
            groups = 1
            c, n = (rng.choice([v, v, 8 * _log(rng, 2, 128)]) for v in (2 ** rng.randint(5, 10), 2 ** rng.randint(5, 10)))
            n = rng.choice([n, n, n, 255])
            cmode, most, layout = mode, 2e11, ("nchw" if what == 7 else "nhwc")
        one = 2.0 * n * (c // groups) * size * size * (hw // stride) ** 2
        # no more work than the listed layers, and no more than 2^28 elements in a tensor
        cap = max(1, min(64, int(most / one), int(2 ** 28 / (max(c, n) * hw * hw))))
        return _strip(_conv("", _log(rng, 1, cap), c, hw, n, size, stride, groups, cmode, layout, rng.choice(["leaky", "leaky", "linear"])))
    if what == 10:
        op = rng.choice(["maxpool", "upsample", "shortcut", "route", "yolo", "convert"])
        layout, dtype = rng.choice([("nhwc", "f32"), ("nhwc", "bf16"), ("nchw", "f32")])
        hw = rng.choice([7, 13, 19, 26, 38, 52, 76, 104, 152, _log(rng, 7, 152)])
        c = 255 if op == "yolo" else rng.choice([2 ** rng.randint(5, 10), 8 * _log(rng, 4, 128)])
        if op == "upsample":
            hw = min(hw, 76)
        cap = max(1, min(64, int(2 ** 27 / (c * hw * hw))))
        return _strip(_mem("", op, _log(rng, 1, cap), c, hw, layout, dtype))
    return _strip(_mem("", rng.choice(["softmax", "avgpool"]), _log(rng, 1, 256), rng.choice([10, 80, 1000, 1024, 2048, _log(rng, 10, 9000)]),
                       rng.choice([7, 8, 13]), rng.choice(["nhwc", "nchw"]), "f32"))


# ---------------------------------------------------------------------------------------------------- geometry
def _cfg(case):
    size, batch = case["size"], case["batch"]
    if case["net"] == "yolov3":
        return synth.yolov3_cfg(batch, size)
    if case["net"] == "yolov3-tiny":
        return synth.yolov3_tiny_cfg(batch, size)
    if case["net"] == "resnet50":
        return synth.resnet50_cfg(batch, size)
    return synth.darknet19_cfg(batch, size, xnor=case["net"] == "darknet19-xnor")


def _result_layers(cfg):
    """The layers whose outputs network_predict hands out: every [yolo] layer, or the last layer."""
    kinds = [k for k, _ in synth.parse_cfg(cfg)[1:]]
    return [i for i, k in enumerate(kinds) if k == "yolo"] or [len(kinds) - 1]


def _walk(cfg):
    """(flops, parameters, values of the result layers) of one image."""
    sections = synth.parse_cfg(cfg)
    net = sections[0][1]
    c, h, w = int(net["channels"]), int(net["height"]), int(net["width"])
    dims, flops, params = [], 0.0, 0
    for i, (kind, o) in enumerate(sections[1:]):
        if kind == "convolutional":
            n, size, stride = int(o["filters"]), int(o["size"]), int(o["stride"])
            pad = size // 2 if int(o["pad"]) else 0
            h, w = (h + 2 * pad - size) // stride + 1, (w + 2 * pad - size) // stride + 1
            flops += 2.0 * n * c * size * size * h * w
            params += n * c * size * size
            c = n
        elif kind == "maxpool":
            size, stride = int(o["size"]), int(o["stride"])
            h, w = (h - 1) // stride + 1, (w - 1) // stride + 1     # padding size-1
        elif kind == "upsample":
            h, w = 2 * h, 2 * w
        elif kind == "route":
            ids = [int(t) for t in o["layers"].split(",")]
            ids = [t if t >= 0 else i + t for t in ids]
            c, h, w = sum(dims[t][0] for t in ids), dims[ids[0]][1], dims[ids[0]][2]
        elif kind == "avgpool":
            h = w = 1
        dims.append((c, h, w))
    return flops, params, sum(a * b * d for a, b, d in (dims[i] for i in _result_layers(cfg)))


def _out_hw(case):
    """Output extent of a layer case's square map."""
    op, hw = case["op"], case["hw"]
    if op == "conv":
        return (hw + 2 * (case["size"] // 2) - case["size"]) // case["stride"] + 1
    return {"maxpool": (hw + 1 - 2) // 2 + 1, "upsample": 2 * hw, "avgpool": 1, "softmax": 1}.get(op, hw)


# ---------------------------------------------------------------------------------------------------- preparation
def _params(cfg, gen):
    """synth.seeded_params' distributions, drawn on the GPU."""
    out = []
    for s in synth.param_shapes(cfg):
        fan = s.size * s.size * (s.c // s.groups)
        w = torch.randn((s.n, s.c // s.groups, s.size, s.size), generator=gen, device="cuda") * math.sqrt(2.0 / fan)
        vec = torch.randn((2, s.n), generator=gen, device="cuda")
        uni = torch.rand((2, s.n), generator=gen, device="cuda")
        bn = (None, None, None)
        if s.batch_normalize:
            bn = ((0.9 + 0.2 * uni[0]).cpu().numpy(), (vec[1] * math.sqrt(0.1)).cpu().numpy(), (0.5 + uni[1]).cpu().numpy())
        out.append(synth.ConvParams(w.cpu().numpy(), (vec[0] * 0.1).cpu().numpy(), *bn, s.kind))
    return out


_streams = []


def _side_stream():
    """The one stream that a program which drives networks on device-resident images has (the legacy default stream takes no graphs)."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    return gen


def _prepare_network(case, seed):
    gen = _generator(seed)
    cfg = _cfg(case)
    params = _params(cfg, gen)
    net = dn.Network(cfg, None, MODES[case["mode"]], text=True)
    fd, path = tempfile.mkstemp(suffix=".weights")
    os.close(fd)
    try:
        synth.write_weights(path, params)
        net.load_weights(path)
    finally:
        os.unlink(path)
    layers = _result_layers(cfg)
    state = {"call": case["call"], "net": net, "layers": layers}
    shape = (case["batch"], 3, case["size"], case["size"])
    images = [torch.rand(shape, generator=gen, device="cuda") for _ in range(2 if case["call"] == "stream" else 1)]
    if case["call"] == "forward":
        net.enable_graph(bool(case["graph"]))
        stream = _side_stream()
        state.update(x=images[0], stream=stream, handle=stream.cuda_stream,
                     out=[torch.empty((case["batch"],) + net.layer_shape(i), device="cuda") for i in layers])
    else:
        host = [x.cpu() for x in images]
        state["x"] = [x.pin_memory() if case["host"] == "pinned" else np.array(x.numpy()) for x in host]
    return state


def _nhwc(t, dtype):
    """Channels-last copy of an NCHW tensor, channels padded with zeros to a multiple of 8."""
    n, c, h, w = t.shape
    out = torch.zeros((n, h, w, (c + 7) // 8 * 8), dtype=dtype, device="cuda")
    out[..., :c] = t.permute(0, 2, 3, 1)
    return out


def _tensor(t, layout, dtype):
    """(storage, dnb_tensor) of NCHW values in the layout and type a case asks for."""
    if layout == "nchw":
        t = t.contiguous()
        return t, dn.as_tensor(t, dn.NCHW)
    s = _nhwc(t, torch.bfloat16 if dtype == "bf16" else torch.float32)
    return s, dn.as_tensor(s, dn.NHWC, t.shape[1])


def _empty(b, c, hw, layout, dtype):
    if layout == "nchw":
        t = torch.zeros((b, c, hw, hw), device="cuda")
        return t, dn.as_tensor(t, dn.NCHW)
    t = torch.zeros((b, hw, hw, (c + 7) // 8 * 8), dtype=torch.bfloat16 if dtype == "bf16" else torch.float32, device="cuda")
    return t, dn.as_tensor(t, dn.NHWC, c)


def _prepare_layer(case, seed):
    gen = _generator(seed)
    op, b, c, hw, layout = case["op"], case["batch"], case["c"], case["hw"], case["layout"]
    dtype = case.get("dtype", case.get("mode"))
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda")  # noqa: E731
    if op == "conv":
        cfg = synth.single_conv_cfg(b, c, hw, hw, case["n"], case["size"], case["stride"], act=case["act"], groups=case["groups"])
        p = _params(cfg, gen)[0]
        plan = dn.ConvPlan(b, c, hw, hw, case["n"], case["size"], case["stride"], case["size"] // 2, case["groups"], True, case["act"],
                           False, MODES[case["mode"]])
        plan.set_params(p.weights, p.biases, p.scales, p.rolling_mean, p.rolling_variance)
        ins, out = [_tensor(rand(b, c, hw, hw), layout, dtype)], _empty(b, case["n"], _out_hw(case), layout, dtype)
        return {"op": op, "plan": plan, "ins": ins, "out": out}
    if op == "softmax":
        ins, out = [_tensor(3 * rand(b, c, 1, 1), layout, dtype)], _empty(b, c, 1, layout, dtype)
    elif op == "shortcut":
        ins, out = [_tensor(rand(b, c, hw, hw), layout, dtype) for _ in range(2)], _empty(b, c, hw, layout, dtype)
    elif op == "route":
        ins, out = [_tensor(rand(b, k, hw, hw), layout, dtype) for k in (c, 2 * c)], _empty(b, 3 * c, hw, layout, dtype)
    elif op == "yolo":
        ins, out = [_tensor(rand(b, c, hw, hw), layout, dtype)], _empty(b, c, hw, "nchw", "f32")
    elif op == "convert":      # the boundary of a channels-last pipeline: Darknet's layout to channels-last, or (an nchw case) back
        src = "nchw" if layout == "nhwc" else "nhwc"
        ins, out = [_tensor(rand(b, c, hw, hw), src, dtype)], _empty(b, c, hw, layout, dtype)
    else:                      # maxpool (size 2, stride 2), upsample (x2), avgpool
        ins, out = [_tensor(rand(b, c, hw, hw), layout, dtype)], _empty(b, c, _out_hw(case), layout, dtype)
    return {"op": op, "ins": ins, "out": out}


def prepare(case, seed):
    return (_prepare_network if case["kind"] == "network" else _prepare_layer)(case, seed)


# ---------------------------------------------------------------------------------------------------- one pass
class _Held(np.ndarray):
    """A result array in the network's own host memory that keeps the network alive with it."""


def _hold(array, net):
    array = array.view(_Held)
    array.net = net
    return array


def _results(net, layers, last):
    if len(layers) == 1:
        return [_hold(last, net)]
    return [_hold(net.yolo_output(i), net) for i in layers]


def _run_network(s):
    net = s["net"]
    if s["call"] == "forward":
        net.forward(s["x"], stream=s["handle"])
        for i, out in zip(s["layers"], s["out"]):
            dn.check(dn.lib().dnb_network_export_layer(net.handle, i, ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(s["handle"])))
        return s["out"]
    if s["call"] == "predict":
        return _results(net, s["layers"], net.predict(s["x"][0]))
    net.submit(s["x"][0])
    net.submit(s["x"][1])
    return [_results(net, s["layers"], net.collect()) for _ in range(2)]


def run(state):
    s = state
    if "net" in s:
        return _run_network(s)
    op, x, (out, y) = s["op"], s["ins"][0][1], s["out"]
    if op == "conv":
        s["plan"].forward(x, y)
    elif op == "maxpool":
        dn.maxpool(x, y, 2, 2)
    elif op == "upsample":
        dn.upsample(x, y, 2)
    elif op == "shortcut":
        dn.shortcut(x, s["ins"][1][1], y)
    elif op == "route":
        dn.route([x, s["ins"][1][1]], y)
    elif op == "yolo":
        dn.yolo(x, y, 3, 80)
    elif op == "convert":
        dn.convert(x, y)
    elif op == "avgpool":
        dn.avgpool(x, y)
    else:
        dn.softmax(x, y)
    return out


# ---------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    if case["kind"] == "network":
        flops, params, results = _walk(_cfg(case))
        per_weight = 2 if case["mode"] == "bf16" else 4
        batches = 2 if case["call"] == "stream" else 1
        images = case["batch"] * batches
        return {"bytes": images * 4.0 * (3 * case["size"] ** 2 + results) + batches * per_weight * params, "flops": images * flops}
    b, c, hw, op = case["batch"], case["c"], case["hw"], case["op"]
    ohw = _out_hw(case)
    if op == "conv":
        es = 2 if case["mode"] == "bf16" and case["layout"] == "nhwc" else 4
        weights = case["n"] * (c // case["groups"]) * case["size"] ** 2
        flops = 2.0 * b * weights * ohw * ohw
        return {"bytes": es * b * (c * hw * hw + case["n"] * ohw * ohw) + (2.0 if case["mode"] == "bf16" else 4.0) * weights, "flops": flops}
    es = 2 if case["dtype"] == "bf16" and case["layout"] == "nhwc" else 4
    inside, outside = (c, c) if op == "softmax" else (c * hw * hw, c * ohw * ohw)
    if op == "convert":     # one side is always f32 in Darknet's layout
        other = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": float(b * inside * (4 + other))}
    if op == "yolo":
        return {"bytes": float(b * inside * (es + 4))}
    many = {"shortcut": (2, 1), "route": (3, 3)}.get(op, (1, 1))
    return {"bytes": float(b * es * (many[0] * inside + many[1] * outside))}


def tolerance(case):
    if case["kind"] == "network":
        # outputs are stored as 32-bit floats, but every layer multiplies and stores TF32 (10 bits) or bf16 (7 bits) values
        return {"rel": 2e-2} if case["mode"] == "bf16" else {"rel": 1e-2 if case["net"] == "darknet19-xnor" else 5e-3}
    op = case["op"]
    if op == "conv":
        return {"rel": {"tf32": 1e-3, "bf16": 1e-2, "fp32": 1e-5}[case["mode"]]}
    if op in ("maxpool", "upsample", "route", "convert"):
        return "exact"
    return {"rel": 4e-3} if case["dtype"] == "bf16" and op != "yolo" else {"rel": 1e-5}

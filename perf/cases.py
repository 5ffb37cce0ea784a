"""Performance cases of the interpreter backend: what users of this framework have it do, through its public entry points.

A case names a workload (``kind``), its sizes and the way the data crosses the boundary (``io``):

* ``op``: one op owned by itself (``create_op``), its operands on the device, run by the synchronous ``invoke()``;
* ``resident``: the inputs are on the device already, ``launch()`` enqueues the module and the results stay in the device
  tensors (``tensor_device``): throughput runs, and hosts that chain the module with other GPU work;
* ``call``: ``module.run`` with host arrays, the one-line call of the Python binding (set every input, invoke, get every output);
* ``stream`` / ``stream_i8``: a serving loop over pinned buffers: ``set_tensor_async`` (or the already quantised
  ``set_tensor_async_i8``), ``launch``, ``get_tensor_into`` for every output.

Kinds: ``conv`` (one INT8 Conv2D op, the op sweep), the INT8 / BF16 networks of ``tpu_compiler_b200.graphs``, ``calibration``
(the two statistics passes and the threshold search over an fp32 ResNet-50) and ``tuner`` (the threshold auto-tuner over a
small fp32 residual network). Weights are those of the graph builders' own seeds, as a deployed network's are; the inputs
come from the seed that ``prepare`` is given.
"""
import functools
import math
import re

import numpy as np
import torch

from tpu_compiler_b200 import graphs, module
from tpu_compiler_b200.calibration import ActivationCalibrator
from tpu_compiler_b200.tuner import SimpleTuner

YOLO_RES = 128  # the detector's scales are chosen on a small image; every extent of it is the resolution over a power of two
DTYPE_BYTES = {"INT8": 1, "BF16": 2, "FP32": 4}


def listed():
    return [
        # the smallest call: one op of the sweep on one image, invoked by itself, a few microseconds of device time
        {"name": "conv3x3_n1_c64_hw56_op", "kind": "conv", "n": 1, "ic": 64, "oc": 64, "hw": 56, "k": 3, "stride": 1,
         "relu": True, "io": "op"},
        # one op of odd sizes: channels that are no multiple of 16, a stride, a ragged last tile, no activation
        {"name": "conv5x5_s2_n7_c72_o200", "kind": "conv", "n": 7, "ic": 72, "oc": 200, "hw": 45, "k": 5, "stride": 2,
         "relu": False, "io": "resident"},
        # interactive inference, image by image: configuration C1 through the call a script makes
        {"name": "resnet50_int8_b1_call", "kind": "resnet50_int8", "batch": 1, "res": 224, "io": "call"},
        # a batcher that sends what has come in: an odd, middling batch
        {"name": "resnet50_int8_b19", "kind": "resnet50_int8", "batch": 19, "res": 224, "io": "resident"},
        # the headline throughput configuration
        {"name": "resnet50_int8_b256", "kind": "resnet50_int8", "batch": 256, "res": 224, "io": "resident"},
        # serving from pinned buffers with inputs that the client has quantised
        {"name": "resnet50_int8_b64_stream_i8", "kind": "resnet50_int8", "batch": 64, "res": 224, "io": "stream_i8"},
        # depthwise-separable network, its configured batch
        {"name": "mobilenet_v2_b32", "kind": "mobilenet_v2_int8", "batch": 32, "res": 224, "width": 1.0, "io": "resident"},
        # a slimmer one on small images, a few at a time, from host arrays
        {"name": "mobilenet_v2_w075_r160_b7_call", "kind": "mobilenet_v2_int8", "batch": 7, "res": 160, "width": 0.75,
         "io": "call"},
        # detection: mixed INT8 / BF16 graph, fp32 frames in, three heads out
        {"name": "yolov4_b8_416_stream", "kind": "yolov4_style_int8", "batch": 8, "res": 416, "io": "stream"},
        # BF16 inference
        {"name": "resnet50_bf16_b128", "kind": "resnet50_bf16", "batch": 128, "res": 224, "io": "resident"},
        # calibration of a network on a small image set (configuration C5's batches of 64)
        {"name": "calibration_b64x2", "kind": "calibration", "batch": 64, "batches": 2, "bins": 2048},
        # threshold tuning of a small network on the images that fit beside it
        {"name": "tuner_16x64", "kind": "tuner", "batch": 16, "res": 64, "width": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    while True:
        case = _draw(rng)
        if case not in known:
            return case


def _draw(rng):
    kind = rng.choice(["conv", "conv", "resnet50_int8", "resnet50_int8", "mobilenet_v2_int8", "yolov4_style_int8",
                       "resnet50_bf16", "calibration", "tuner"])
    if kind == "conv":
        io = rng.choice(["op", "resident"])
        n, hw = (_log_int(rng, 1, 32), _log_int(rng, 7, 112)) if io == "op" else (_log_int(rng, 6, 32), _log_int(rng, 20, 112))
        return {"kind": kind, "n": n, "ic": _log_int(rng, 16, 512), "oc": _log_int(rng, 16, 512), "hw": hw,
                "k": rng.choice([1, 3, 3, 5]), "stride": rng.choice([1, 1, 2]), "relu": rng.random() < 0.5, "io": io}
    if kind == "resnet50_int8":
        io = rng.choice(["resident", "resident", "call", "stream", "stream_i8"])
        return {"kind": kind, "batch": _log_int(rng, 1, 48 if io == "call" else 256), "res": 224, "io": io}
    if kind == "mobilenet_v2_int8":
        io = rng.choice(["resident", "call", "stream_i8"])
        return {"kind": kind, "batch": _log_int(rng, 1, 48 if io == "call" else 128), "res": rng.choice([128, 160, 192, 224]),
                "width": rng.choice([0.5, 0.75, 1.0]), "io": io}
    if kind == "yolov4_style_int8":
        res = rng.choice([256, 320, 416])
        return {"kind": kind, "batch": _log_int(rng, 1, 12), "res": res, "io": rng.choice(["resident", "stream"])}
    if kind == "resnet50_bf16":
        return {"kind": kind, "batch": _log_int(rng, 1, 128), "res": 224, "io": rng.choice(["resident", "stream"])}
    if kind == "calibration":
        return {"kind": kind, "batch": _log_int(rng, 8, 64), "batches": rng.choice([1, 2]), "bins": rng.choice([1024, 2048])}
    return {"kind": kind, "batch": _log_int(rng, 4, 24), "res": rng.choice([32, 40, 48, 56, 64, 72]),
            "width": rng.choice([16, 24, 32])}


# ----------------------------------------------------------------------------------------------- graphs and weights
def _residual_fp32(width, res, seed=7001):
    """A small fp32 network of the auto-tuner's op set: stem, max pool, three residual blocks, average pool, classifier."""
    rng = np.random.default_rng(seed)
    b = graphs.GraphBuilder(seed, simulate=False)

    def conv(name, src, oc, k, relu=1):
        n, ic, h, w = b.shapes[src]
        f = b.weight(name + "_filter", rng.normal(0, math.sqrt(2.0 / (ic * k * k)), (oc, ic, k, k)))
        bi = b.weight(name + "_bias", rng.normal(0, 0.1, oc))
        p = k // 2
        return b.op("conv_2d", name, [src, f, bi], (n, oc, h, w), "FP32", kh=k, kw=k, sh=1, sw=1, pt=p, pb=p, pl=p, pr=p, dh=1,
                    dw=1, g=1, do_relu=relu, with_bias=1)

    b.op("input", "data", [], (1, 3, res, res), "FP32")
    conv("conv1", "data", width, 3)
    x = b.op("pool_max_2d", "pool1", ["conv1"], (1, width, res // 2, res // 2), "FP32", kh=2, kw=2, sh=2, sw=2, pt=0, pb=0,
             pl=0, pr=0)
    for i in range(3):
        y = conv("b%d_1" % i, x, width, 1)
        y = conv("b%d_2" % i, y, 2 * width, 3, relu=0)
        s = conv("b%d_s" % i, x, 2 * width, 1, relu=0)
        x = b.op("eltwise_add", "b%d" % i, [s, y], b.shapes[y], "FP32", do_relu=1)
    x = b.op("pool_avg_2d", "gap", [x], (1, 2 * width, 1, 1), "FP32", kh=res // 2, kw=res // 2, sh=res // 2, sw=res // 2,
             count_include_pad=1)
    f = b.weight("fc_filter", rng.normal(0, 0.2, (10, 2 * width)))
    bi = b.weight("fc_bias", rng.normal(0, 0.1, 10))
    b.op("fully_connected", "fc", [x, f, bi], (1, 10), "FP32", do_relu=0)
    return graphs.Model(b.text(), b.weights, ["data"], ["fc"])


@functools.lru_cache(maxsize=4)
def _model(kind, *sizes):
    """The network at batch 1: its text, weights and outputs do not depend on the inputs."""
    if kind == "conv":
        ic, oc, hw, k, stride, relu = sizes
        m = graphs.single_conv_i8(1, ic, oc, hw, k, stride, k // 2, relu=relu)
    elif kind == "calibration":
        m = graphs.resnet50_fp32(1)
    elif kind == "tuner":
        m = _residual_fp32(*sizes)
    elif kind == "mobilenet_v2_int8":
        m = graphs.mobilenet_v2_int8(1, res=sizes[0], width=sizes[1])
    elif kind == "yolov4_style_int8":
        m = graphs.yolov4_style_int8(1, res=YOLO_RES)
    else:
        m = getattr(graphs, kind)(1)
    return m.text, m.weights, m.outputs


def _sizes(case):
    keys = {"conv": ("ic", "oc", "hw", "k", "stride", "relu"), "mobilenet_v2_int8": ("res", "width"), "tuner": ("width", "res")}
    return tuple(case[k] for k in keys.get(case["kind"], ()))


def _network(case):
    """(module text at the case's batch, weights, output names)"""
    text, weights, outputs = _model(case["kind"], *_sizes(case))
    text = re.sub(r"shape=1\b", "shape=%d" % case.get("batch", case.get("n")), text)
    if case["kind"] == "yolov4_style_int8":
        text = re.sub(r"(shape=\d+,\d+),(\d+),(\d+)", lambda s: "%s,%d,%d" % (
            s[1], int(s[2]) * case["res"] // YOLO_RES, int(s[3]) * case["res"] // YOLO_RES), text)
    return text, weights, outputs


# ----------------------------------------------------------------------------------------------- inputs and state
def _inputs(case, seed):
    """This seed's inputs as host values: int8-valued for one op, images in the range the network was quantised for
    (uniform pixels, 0..1 for the detector), N(0, 1) clipped to [-3, 3] for the fp32 networks."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "conv":
        shape = (case["n"], case["ic"], case["hw"], case["hw"])
        return torch.randint(-128, 128, shape, generator=g, device="cuda").float().cpu()
    shape = (case["batch"], 3, case.get("res", 224), case.get("res", 224))
    if case["kind"] in ("calibration", "tuner"):
        return [torch.randn(shape, generator=g, device="cuda").clamp_(-3, 3).cpu() for _ in range(case.get("batches", 1))]
    x = torch.rand(shape, generator=g, device="cuda")
    if case["kind"] != "yolov4_style_int8":
        x = x.mul_(2).sub_(1)
    if case["io"] == "stream_i8":  # as the module's own quant op (threshold 1.0): round half away from zero, saturate
        x = x.mul_(128)
        x = (torch.sign(x) * torch.floor(x.abs() + 0.5)).clamp_(-128, 127).to(torch.int8)
    return x.cpu()


class _DeviceArray:
    def __init__(self, m, ptr, shape, typestr):
        self.module = m  # the storage is the module's: it lives as long as a view of it does
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


def _device_view(m, name):
    """The module's tensor where it lies on the device: [n, h, w, channels]."""
    t = m.tensor_device(name)
    n, c, h, w = (m.get_tensor_shape(name) + [1, 1, 1])[:4]
    typestr = {0: "|i1", 1: "<i2", 2: "<f4"}[t["dtype"]]
    return torch.as_tensor(_DeviceArray(m, t["ptr"], (n, h, w, t["pitch"]), typestr), device="cuda")[..., :c]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    x = _inputs(case, seed)
    text, weights, s.outputs = _network(case)
    if case["kind"] in ("calibration", "tuner"):
        m = s.model = module(0)
        m.load_text(text, weights)
        if case["kind"] == "calibration":
            batches = [b.pin_memory() for b in x]  # a loader with pin_memory=True
            s.calibrator = ActivationCalibrator(m, lambda: iter(batches), histogram_bin_num=case["bins"])
        else:
            s.images = x[0].numpy()
            s.text, s.weights = text, weights
            s.tables, s.stats = ActivationCalibrator(m, lambda: iter([s.images])).run_multi([2048, 1024, 512])
        return s
    m = s.model = module(0)
    if case["io"] == "op":
        m.set_weights(weights)
        s.op = [m.create_op(line) for line in text.splitlines()][-1]
    else:
        m.load_text(text, weights)
    s.input = m.get_input_details()[0]
    io = case["io"]
    if io == "call":
        s.x = x.numpy()
    elif io in ("op", "resident"):
        m.set_tensor(s.input, x.numpy())
        s.views = {n: _device_view(m, n) for n in s.outputs}
    else:
        s.x = x.pin_memory()
        s.y = {n: torch.empty(m.get_tensor_shape(n), pin_memory=True) for n in s.outputs}
    return s


def run(s):
    case, m = s.case, s.model
    if case["kind"] == "calibration":
        thresholds, stats = s.calibrator.run()
        return {"thresholds": np.array(list(thresholds.values()), np.float32),
                "statistics": np.array(list(stats.values()), np.float32)}
    if case["kind"] == "tuner":
        t = SimpleTuner(s.text, s.weights, s.tables, s.stats, s.images)
        best = t.run()
        distances = [d for per_op in t.distances.values() for d in per_op.values()]
        t.close()
        return {"thresholds": np.array(list(best.values()), np.float64), "distances": np.array(distances, np.float64)}
    if case["io"] == "call":
        return m.run(s.x)
    if case["io"] in ("op", "resident"):
        s.op.invoke() if case["io"] == "op" else m.launch()
        return s.views
    if case["io"] == "stream":
        m.set_tensor_async(s.input, s.x.data_ptr(), s.x.numel())
    else:
        m.set_tensor_async_i8(s.input + "_quant", s.x.data_ptr(), s.x.numel())
    m.launch()
    for n, y in s.y.items():
        m.get_tensor_into(n, y.data_ptr(), y.numel())
    return s.y


# ----------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    """Multiply-adds of the convolutions and inner products (two operations each); bytes of the inputs and the weights,
    read once, and of every result tensor, written once (all of them stay fetchable). The statistics passes also read the
    activations once more: a histogram needs the maximum first."""
    text, weights, _ = _network(case)
    shapes, flops, acts, wbytes = {}, 0.0, 0.0, 0.0
    for line in text.splitlines():
        kind, *rest = line.split()
        a = dict(t.split("=", 1) for t in rest)
        shape = shapes[a["name"]] = [int(d) for d in a["shape"].split(",")]
        size, es = float(np.prod(shape)), DTYPE_BYTES[a["dtype"]]
        if kind != "reshape":
            acts += size * es
        operands = a.get("in", "").split(",")
        if kind in ("conv_2d", "fully_connected"):
            w = weights[operands[1]]
            flops += 2.0 * size * w[0].size
            wbytes += w.size * es
    if case["kind"] == "calibration":
        return {"bytes": case["batches"] * (2 * acts + wbytes), "flops": case["batches"] * flops}
    if case["kind"] == "tuner":  # fp32 reference pass; per candidate an INT8 pass and the distance to the reference
        return {"bytes": acts * (1 + 3 * 1.25) + wbytes, "flops": 4 * flops}
    return {"bytes": acts + wbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "resnet50_bf16":
        return {"rel": 1e-2, "max": 8e-2}  # another order of the fp32 sums moves single BF16 roundings
    if case["kind"] in ("calibration", "tuner"):
        return {"rel": 1e-4}  # fp32 forward
    return "exact"  # INT8 values

"""Timed workloads of the framework, through its public entry points (mace_b200.hostapi, mace_b200.capi).

Whole networks as an engine runs them, and the operators that a program calls on device pointers: a case is
one configuration, listed() the ones to watch, draw() any other of the same ranges.

Networks (inputs and weights are seeded, uint8 NHWC / fp32 NCHW, square images):
  mobilenet   quantized MobileNet-v1 on a captured HostEngine
  resnet      fp32 ResNet-50 on a captured HostEngine with its operators merged and its memory planned
Operators:
  matmul_u8   quantized MatMul: any transposition, batched or not, per-column bias or none
  fc_u8       quantized FullyConnected: a weight matrix times a batch of vectors
  conv_u8     quantized Conv2D, NHWC, k x k
  conv_f32    fp32 Conv2D, NCHW; 3x3 stride 1 by Winograd with the kept transformed filter, as the engine does
  dwconv_f32  fp32 depthwise convolution, NCHW
  matmul_f32  fp32 MatMul, any transposition
"""
import functools
import math

import numpy as np
import torch

from mace_b200 import capi, hostapi
from mace_b200.harness import mobilenet_v1, resnet50

LARGEST_FLOPS = 4.0e11   # of a drawn operator case
LARGEST_BYTES = 1.5e9


def listed():
    return [
        # one photo classified for one request: host buffers in and out, nothing to hide latency behind
        {"name": "mobilenet_u8_request", "net": "mobilenet", "batch": 1, "image": 224, "host": True},
        # throughput serving, the batch already on the device
        {"name": "mobilenet_u8_b64", "net": "mobilenet", "batch": 64, "image": 224, "host": False},
        {"name": "resnet50_f32_request", "net": "resnet", "batch": 1, "image": 224, "host": True},
        {"name": "resnet50_f32_b256", "net": "resnet", "batch": 256, "image": 224, "host": False},
        # a square MatMul, A x B as stored, with bias
        {"name": "matmul_u8_1024", "op": "matmul_u8", "batch": 1, "m": 1024, "n": 1024, "k": 1024,
         "ta": False, "tb": False, "bias": True},
        # a few tokens against a large weight matrix
        {"name": "matmul_u8_few_rows", "op": "matmul_u8", "batch": 1, "m": 16, "n": 4096, "k": 4096,
         "ta": False, "tb": False, "bias": False},
        # sizes as they come: a batch of sequences of odd length
        {"name": "matmul_u8_odd", "op": "matmul_u8", "batch": 4, "m": 333, "n": 1001, "k": 777,
         "ta": False, "tb": True, "bias": True},
        # one vector through a large fully connected layer
        {"name": "fc_u8_4096", "op": "fc_u8", "batch": 1, "rows": 4096, "k": 4096},
        # a 3x3 layer of a quantized detector's backbone
        {"name": "conv_u8_3x3", "op": "conv_u8", "batch": 8, "hw": 56, "c": 64, "o": 128, "ksize": 3, "stride": 2},
        # a 3x3 layer of a residual network
        {"name": "conv_f32_winograd", "op": "conv_f32", "batch": 32, "hw": 56, "c": 64, "o": 64, "ksize": 3,
         "stride": 1},
        # a depthwise layer of a float MobileNet
        {"name": "dwconv_f32_3x3", "op": "dwconv_f32", "batch": 32, "hw": 112, "c": 64, "ksize": 3, "stride": 2},
        # attention scores: Q x K^T per head
        {"name": "matmul_f32_scores", "op": "matmul_f32", "batch": 12, "m": 384, "n": 384, "k": 64,
         "ta": False, "tb": True},
    ]


def _log(rng, low, high, step=1):
    """A whole number from low to high, spread over its logarithm, a multiple of step."""
    return max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))) / step)) * step)


def _draw_once(rng):
    kind = rng.choice(["mobilenet", "resnet", "matmul_u8", "matmul_u8", "fc_u8", "conv_u8", "conv_f32",
                       "dwconv_f32", "matmul_f32"])
    step = rng.choice([1, 16])   # sizes as they come, or the round ones that models like
    if kind in ("mobilenet", "resnet"):
        batch = _log(rng, 2, 96)
        return {"net": kind, "batch": batch, "image": rng.choice([128, 160, 192, 224]), "host": batch <= 4}
    if kind == "matmul_u8":
        if rng.random() < 0.35:
            return {"op": kind, "batch": _log(rng, 2, 64), "m": _log(rng, 32, 768, step), "n": _log(rng, 32, 768, step),
                    "k": _log(rng, 32, 768, step), "ta": rng.random() < 0.3, "tb": rng.random() < 0.5,
                    "bias": rng.random() < 0.5}
        return {"op": kind, "batch": 1, "m": _log(rng, 1, 4096), "n": _log(rng, 64, 4096, step),
                "k": _log(rng, 64, 4096, step), "ta": rng.random() < 0.2, "tb": rng.random() < 0.5,
                "bias": rng.random() < 0.5}
    if kind == "fc_u8":
        return {"op": kind, "batch": _log(rng, 1, 64), "rows": _log(rng, 100, 8192, step), "k": _log(rng, 64, 8192, step)}
    if kind == "matmul_f32":
        return {"op": kind, "batch": _log(rng, 1, 32), "m": _log(rng, 16, 1536, step), "n": _log(rng, 16, 1536, step),
                "k": _log(rng, 16, 1024, step), "ta": rng.random() < 0.3, "tb": rng.random() < 0.5}
    # feature maps: odd extents as well as the usual ones
    hw = rng.choice([7, 14, 28, 56, 112, rng.randint(7, 112)])
    case = {"op": kind, "batch": _log(rng, 1, 32), "hw": hw, "c": _log(rng, 16, 512, step)}
    if kind != "dwconv_f32":
        case["o"] = _log(rng, 16, 512, step)
    case["ksize"] = rng.choice([3, 3, 5] if kind == "dwconv_f32" else [1, 3, 3, 5])
    case["stride"] = rng.choice([1, 2])
    return case


def draw(rng):
    while True:
        case = _draw_once(rng)
        if "net" in case:
            return case
        w = work(case)
        if w["flops"] <= LARGEST_FLOPS and w["bytes"] <= LARGEST_BYTES:
            return case


# ---- what the cases share -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    """The program's one device context: its operators run in order on one stream."""
    return capi.Context(0)


class _Dev:
    """A torch tensor where the binding expects a device buffer."""

    def __init__(self, tensor):
        self.tensor = tensor
        self.ptr = tensor.data_ptr()


class _Engine:
    """Closes a HostEngine when nothing refers to it any more."""

    def __init__(self, engine):
        self.engine = engine

    def __del__(self):
        self.engine.close()


class _View:
    """A tensor of an engine, for torch.as_tensor; keeps the engine alive."""

    def __init__(self, owner, name, shape, typestr):
        self._owner = owner
        ptr, _ = owner.engine.device_ptr(name)
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False), "version": 2}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _bytes(g, *shape, low=0, high=256):
    return torch.randint(low, high, shape, generator=g, device="cuda", dtype=torch.uint8)


def _normal(g, *shape, std=1.0):
    return torch.randn(shape, generator=g, device="cuda") * std


def _bias_i32(g, n):
    return torch.round(_normal(g, n, std=1000.0)).to(torch.int32)


def _fixed_point(real):
    """real in (0, 1) as a Q31 multiplier in [2^30, 2^31) and a right shift."""
    q, e = math.frexp(real)
    mult = int(round(q * (1 << 31)))
    if mult == 1 << 31:
        mult, e = mult // 2, e + 1
    return mult, -e


def _output_scale(depth):
    """Uniform operands with central zero points: the accumulator's deviation is about
    sqrt(depth) * 74 * 74, and three of them fill half of the output's range."""
    return 127.0 / (3.0 * math.sqrt(depth) * 74.0 * 74.0)


def _same(size, ksize, stride):
    """Output extent and leading padding of SAME, the smaller half in front."""
    out = -(-size // stride)
    return out, max(0, (out - 1) * stride + ksize - size) // 2


# ---- networks -----------------------------------------------------------------------------

def _mobilenet_macs(image):
    fc = 1024 * mobilenet_v1.NUM_CLASSES
    return (mobilenet_v1.macs_per_image() - fc) * image ** 2 // 224 ** 2 + fc


@functools.lru_cache(maxsize=None)
def _resnet_graph():
    nodes, weights = resnet50.build(seed=0)
    return nodes, {k: v.shape for k, v in weights.items()}


def _mobilenet_layers(g, image):
    """He-normal weights quantized around a central zero point.  A ReLU's output keeps its input's mean
    square under such weights, so one output scale that covers four deviations serves every layer."""
    layers, s_in, rms = [], 1.0 / 255.0, math.sqrt(1.0 / 3.0)
    s_act = 4.0 * math.sqrt(2.0) * rms / 255.0

    def layer(kind, name, shape, channels, fan_in, stride=1, s_out=s_act, zp_out=0):
        std = math.sqrt(2.0 / fan_in)
        s_f, zp_f = 8.0 * std / 255.0, int(torch.randint(120, 137, (1,), generator=g, device="cuda"))
        w = torch.clamp(torch.round(_normal(g, *shape, std=std / s_f)) + zp_f, 1, 255).to(torch.uint8).cpu().numpy()
        bias = torch.round(_normal(g, channels, std=0.01 / (s_in * s_f))).to(torch.int32).cpu().numpy()
        layers.append(dict(kind=kind, name=name, w=w, s_f=s_f, zp_f=zp_f, bias=bias, bias_scale=s_in * s_f,
                           stride=stride, s_in=s_in, zp_in=0, s_out=s_out, zp_out=zp_out))
        return s_out

    s_in = layer("conv", "stem", (32, 3, 3, 3), 32, 27, 2)
    c = 32
    for i, (o, s) in enumerate(zip(mobilenet_v1.PW_OUT, mobilenet_v1.DW_STRIDE)):
        s_in = layer("dw", "dw%d" % (i + 1), (3, 3, c, 1), c, 9, s)
        s_in = layer("conv", "pw%d" % (i + 1), (o, 1, 1, c), o, c)
        c = o
    layers.append(dict(kind="pool", name="pool", kernel=image // 32, s_in=s_in, zp_in=0))
    layer("fc", "fc", (mobilenet_v1.NUM_CLASSES, 1, 1, c), mobilenet_v1.NUM_CLASSES, c, s_out=6.0 / 255.0, zp_out=128)
    return layers


def _resnet_weights(g, shapes):
    return {k: _normal(g, *s, std=math.sqrt(2.0 / math.prod(s[1:])) if len(s) == 4 else 0.01).cpu().numpy()
            for k, s in shapes.items()}


def _prepare_net(case, seed):
    g, batch, image = _generator(seed), case["batch"], case["image"]
    if case["net"] == "mobilenet":
        eng = mobilenet_v1.build_engine(hostapi, _mobilenet_layers(g, image), batch, image=image)
        x = _bytes(g, batch, image, image, 3).cpu()
        out_type, out_np, out_shape = "|u1", np.uint8, (batch, 1, 1, mobilenet_v1.NUM_CLASSES)
    else:
        nodes, shapes = _resnet_graph()
        eng = resnet50.build_engine(hostapi, nodes, _resnet_weights(g, shapes), batch, image=image)
        eng.share_subsampled_inputs()
        eng.fuse_activations()
        x = torch.rand((batch, 3, image, image), generator=g, device="cuda").cpu()
        out_type, out_np, out_shape = "<f4", np.float32, (batch, resnet50.NUM_CLASSES, 1, 1)
    owner = _Engine(eng)
    eng.write("input", x.numpy())
    eng.run()
    if case["net"] == "resnet":
        eng.fuse_residual_sums()
        eng.plan_memory()
        eng.write("input", x.numpy())
        eng.run()
    eng.capture()
    state = {"owner": owner}
    if case["host"]:
        state["keep"] = (x.pin_memory(), torch.empty(out_shape, dtype=getattr(torch, np.dtype(out_np).name)).pin_memory())
        state["x"], state["out"] = (t.numpy() for t in state["keep"])
    else:
        state["out"] = torch.as_tensor(_View(owner, "fc", out_shape, out_type), device="cuda")
    return state


def _run_net(s):
    if "x" in s:
        s["owner"].engine.run_host("input", s["x"], "fc", s["out"])
    else:
        s["owner"].engine.run()
    return s["out"]


# ---- operators ----------------------------------------------------------------------------

def _prepare_op(c, seed):
    g, op = _generator(seed), c["op"]
    s = {}
    if op == "matmul_u8":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        s["a"], s["b"] = _Dev(_bytes(g, b, m * k)), _Dev(_bytes(g, b, k * n))
        s["bias"] = _Dev(_bias_i32(g, n)) if c["bias"] else None
        s["out"] = _Dev(torch.empty((b, m, n), dtype=torch.uint8, device="cuda"))
        s["fixed"] = _fixed_point(_output_scale(k))
    elif op == "fc_u8":
        s["w"], s["x"] = _Dev(_bytes(g, c["rows"], c["k"])), _Dev(_bytes(g, c["batch"], c["k"]))
        s["bias"] = _Dev(_bias_i32(g, c["rows"]))
        s["out"] = _Dev(torch.empty((c["batch"], c["rows"]), dtype=torch.uint8, device="cuda"))
        s["scale"] = _output_scale(c["k"])
    elif op == "conv_u8":
        ho, _ = _same(c["hw"], c["ksize"], c["stride"])
        s["x"] = _Dev(_bytes(g, c["batch"], c["hw"], c["hw"], c["c"]))
        s["w"] = _Dev(_bytes(g, c["o"], c["ksize"], c["ksize"], c["c"], low=1))
        s["bias"] = _Dev(_bias_i32(g, c["o"]))
        s["out"] = _Dev(torch.empty((c["batch"], ho, ho, c["o"]), dtype=torch.uint8, device="cuda"))
        s["fixed"] = _fixed_point(_output_scale(c["ksize"] ** 2 * c["c"]))
    elif op == "matmul_f32":
        b, m, n, k = c["batch"], c["m"], c["n"], c["k"]
        s["a"], s["b"] = _Dev(_normal(g, b, m * k)), _Dev(_normal(g, b, k * n))
        s["out"] = _Dev(torch.empty((b, m, n), device="cuda"))
    else:
        depthwise = op == "dwconv_f32"
        ho, _ = _same(c["hw"], c["ksize"], c["stride"])
        o = c["c"] if depthwise else c["o"]
        fan_in = c["ksize"] ** 2 * (1 if depthwise else c["c"])
        s["x"] = _Dev(_normal(g, c["batch"], c["c"], c["hw"], c["hw"]))
        s["w"] = _Dev(_normal(g, *((1, o) if depthwise else (o, c["c"])), c["ksize"], c["ksize"],
                              std=math.sqrt(2.0 / fan_in)))
        s["bias"] = _Dev(_normal(g, o, std=0.1))
        s["out"] = _Dev(torch.empty((c["batch"], o, ho, ho), device="cuda"))
        if _winograd(c):
            t = (_winograd_tile(c) + 2) ** 2
            s["transformed"] = _Dev(torch.empty((t, o, c["c"]), device="cuda"))
            torch.cuda.synchronize()
            _context().winograd_transform_filter(s["w"], s["transformed"], c["c"], o, _winograd_tile(c))
    return s


def _winograd(c):
    return c["op"] == "conv_f32" and c["ksize"] == 3 and c["stride"] == 1


def _winograd_tile(c):
    return 6 if c["hw"] > 16 else 2


def _run_op(c, s):
    ctx, op = _context(), c["op"]
    if op == "matmul_u8":
        ctx.gemm_u8(s["a"], s["b"], s["bias"], s["out"], c["batch"], c["m"], c["n"], c["k"], 128, 120, *s["fixed"],
                    zp_c=127, a_col_major=c["ta"], b_col_major=c["tb"])
    elif op == "fc_u8":
        ctx.gemv_u8(s["w"], s["x"], s["bias"], s["out"], c["batch"], c["rows"], c["k"], 126, 121, s["scale"], 128)
    elif op == "matmul_f32":
        ctx.gemm_f32(s["a"], s["b"], s["out"], c["batch"], c["m"], c["n"], c["k"], a_col_major=c["ta"],
                     b_col_major=c["tb"])
    else:
        ho, pad = _same(c["hw"], c["ksize"], c["stride"])
        size = (c["batch"], c["hw"], c["hw"], c["c"]) if op == "conv_u8" else (c["batch"], c["c"], c["hw"], c["hw"])
        taps, strides = (c["ksize"], c["ksize"]), (c["stride"], c["stride"])
        if op == "conv_u8":
            ctx.conv2d_u8(s["x"], s["w"], s["bias"], s["out"], *size, c["o"], *taps, strides, (pad, pad), (ho, ho),
                          125, 131, *s["fixed"], 127)
        elif op == "dwconv_f32":
            ctx.dwconv_f32(s["x"], s["w"], s["bias"], s["out"], *size, 1, *taps, strides, (1, 1), (pad, pad),
                           (ho, ho), act=1)
        elif _winograd(c):
            ctx.winograd_f32(s["x"], s["w"], s["bias"], s["out"], *size, c["o"], (pad, pad), (ho, ho), act=1,
                             tile=_winograd_tile(c), transformed=s["transformed"])
        else:
            ctx.conv2d_f32(s["x"], s["w"], s["bias"], s["out"], *size, c["o"], *taps, strides, (1, 1), (pad, pad),
                           (ho, ho), act=1)
    return s["out"].tensor


# ---- the interface ------------------------------------------------------------------------

def prepare(case, seed):
    state = _prepare_net(case, seed) if "net" in case else _prepare_op(case, seed)
    state["case"] = case
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    return _run_net(state) if "net" in case else _run_op(case, state)


def work(case):
    """Inputs, weights and outputs moved once; two operations for a multiplication and its addition.
    (A Winograd convolution counts as the direct one.)"""
    c = case
    if c.get("net") == "mobilenet":
        weights = 4_250_000   # bytes, biases among them
        return {"bytes": c["batch"] * (c["image"] ** 2 * 3 + 1000) + weights, "flops": 2 * c["batch"] * _mobilenet_macs(c["image"])}
    if c.get("net") == "resnet":
        nodes, shapes = _resnet_graph()
        weights = sum(math.prod(s) for s in shapes.values())
        return {"bytes": 4 * (c["batch"] * (c["image"] ** 2 * 3 + 1000) + weights),
                "flops": 2 * c["batch"] * resnet50.macs_per_image(nodes, c["image"])}
    op = c["op"]
    if op in ("matmul_u8", "matmul_f32"):
        values = c["batch"] * (c["m"] * c["k"] + c["k"] * c["n"] + c["m"] * c["n"])
        return {"bytes": values * (4 if op == "matmul_f32" else 1), "flops": 2 * c["batch"] * c["m"] * c["n"] * c["k"]}
    if op == "fc_u8":
        return {"bytes": c["rows"] * c["k"] + c["batch"] * (c["k"] + c["rows"]) + 4 * c["rows"],
                "flops": 2 * c["batch"] * c["rows"] * c["k"]}
    ho, _ = _same(c["hw"], c["ksize"], c["stride"])
    o, depth = (c["c"], 1) if op == "dwconv_f32" else (c["o"], c["c"])
    values = c["batch"] * (c["hw"] ** 2 * c["c"] + ho * ho * o) + o * depth * c["ksize"] ** 2
    return {"bytes": values * (1 if op == "conv_u8" else 4) + 4 * o,
            "flops": 2 * c["batch"] * ho * ho * o * depth * c["ksize"] ** 2}


def tolerance(case):
    """Quantized results are whole numbers that every implementation has to hit."""
    if case.get("net") == "resnet":
        return {"rel": 3e-4}      # 53 fp32 layers, 16 of them F(6,3) or F(2,3) Winograd
    if case.get("net") == "mobilenet" or case["op"] in ("matmul_u8", "fc_u8", "conv_u8"):
        return "exact"
    if _winograd(case):
        return {"rel": 5e-5}
    # split tf32 products lose the lowest bits of every term, so the error grows with the depth
    depth = case["k"] if case["op"] == "matmul_f32" else case["ksize"] ** 2 * case["c"]
    return {"rel": 1e-5 if case["op"] == "dwconv_f32" else max(1e-5, 1.2e-8 * depth)}

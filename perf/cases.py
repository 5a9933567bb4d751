"""The work this package is used for, as a list of timed cases over its public entry points.

Every case is a dict of plain values; `kind` says which entry point it goes through:

  mlp         models.QuantizedMLP, called op by op: QuantizeLinear, three QLinearMatMul, DequantizeLinear
  quantize    ops.QuantizeLinear        (float to 8 bits)
  dequantize  ops.DequantizeLinear      (8 bits to float)
  lstm        ops.ElementWiseNvrtc on the pointwise group of an LSTM cell, from the fusion pass's own source text
  matmul      ops.MatMulInteger
  qmatmul     ops.QLinearMatMul
  conv        ops.QLinearConv through the operator's own signature (unpacked weights; NCHW or channels-last maps)
  dynconv     the chain a dynamically quantized convolution runs: MinMax, DynamicQuantParamsU8, QuantizeLinear with device
              scalars, ConvInteger with a device zero point and per-channel uint8 weights
  resnet50    models.ResNet50Int8, folded requantization: op by op, or captured by dataparallel.InferenceEngine
  mobilenetv2 models.MobileNetV2Int8, likewise

Inputs have the distributions the benchmark configurations name: images uniform in [0, 1), activations normal, quantized operands
uniform over their type, weights symmetric int8 per channel unless the case says otherwise.
"""
import importlib
import math

import numpy as np
import torch

_PACKAGE = "chainer-compiler_b200"  # not an identifier, hence importlib
_pkg = importlib.import_module(_PACKAGE)
ops = importlib.import_module(_PACKAGE + ".ops")
fusion = importlib.import_module(_PACKAGE + ".fusion")
models = importlib.import_module(_PACKAGE + ".models")
dataparallel = importlib.import_module(_PACKAGE + ".dataparallel")

_DEV = "cuda:0"
_FLOATS = {"float32": torch.float32, "float16": torch.float16}
_QTYPES = {"uint8": (torch.uint8, np.uint8, 0, 255), "int8": (torch.int8, np.int8, -128, 127)}


def listed():
    return [
        # a latency-bound request: five small operators, launched one after the other
        {"name": "mlp_b64", "kind": "mlp", "batch": 64, "packed": False},
        # the input batch of the image networks on its way to 8 bits
        {"name": "quantize_images_b256", "kind": "quantize", "n": 256 * 3 * 224 * 224, "zp": 0, "dtype": "uint8", "rne": False},
        # a feature map with a ragged number of values on its way back to float, signed with a zero point
        {"name": "dequantize_ragged", "kind": "dequantize", "n": 37 * 511 * 29 * 31 + 5, "zp": -3, "dtype": "int8"},
        # the fused elementwise group of the benchmark
        {"name": "lstm_4096", "kind": "lstm", "rows": 4096, "cols": 4096, "dtype": "float32"},
        # the smallest size of the integer matrix product sweep
        {"name": "matmul_1024", "kind": "matmul", "m": 1024, "n": 1024, "k": 1024, "b_dtype": "int8", "b_zp": "none"},
        # a product of odd extents with asymmetric weights quantized per column, as the quantizing pass makes of a Gemm
        {"name": "matmul_ragged", "kind": "matmul", "m": 509, "n": 3073, "k": 1283, "b_dtype": "uint8", "b_zp": "column"},
        # a large product of the same sweep, requantized
        {"name": "qmatmul_8192", "kind": "qmatmul", "m": 8192, "n": 8192, "k": 8192},
        # the operator as a graph of the reference calls it: NCHW in, NCHW out, weights as they are stored
        {"name": "conv_nchw_b256", "kind": "conv", "batch": 256, "c": 128, "h": 28, "w": 28, "m": 128, "k": 3, "stride": 1, "layout": "nchw",
         "depthwise": False, "x_zp": 0},
        # one convolution of a dynamically quantized graph
        {"name": "dynconv_b8", "kind": "dynconv", "batch": 8, "c": 64, "h": 56, "w": 56, "m": 64, "k": 3, "stride": 1},
        # the image networks at the batches they are benchmarked at, replayed from a CUDA graph
        {"name": "resnet50_b256", "kind": "resnet50", "batch": 256, "graph": True},
        {"name": "mobilenetv2_b512", "kind": "mobilenetv2", "batch": 512, "graph": True},
        # one image, operator by operator
        {"name": "resnet50_b1", "kind": "resnet50", "batch": 1, "graph": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extent(rng, lo, hi):
    """An extent between lo and hi, spread over the logarithm: as it falls, or rounded to a multiple of 16 as often."""
    v = _log_int(rng, lo, hi)
    return v if rng.random() < 0.5 else max(16, (v + 8) // 16 * 16)


def draw(rng):
    kind = rng.choice(["mlp", "quantize", "dequantize", "lstm", "matmul", "qmatmul", "conv", "dynconv", "resnet50", "mobilenetv2"])
    if kind == "mlp":
        return {"kind": kind, "batch": _log_int(rng, 1, 4096), "packed": rng.random() < 0.5}
    if kind in ("quantize", "dequantize"):
        dtype = rng.choice(["uint8", "uint8", "int8"])
        zp = rng.choice([0, rng.randint(1, 255)]) if dtype == "uint8" else rng.randint(-128, 127)
        case = {"kind": kind, "n": _log_int(rng, 1 << 10, 1 << 28), "zp": zp, "dtype": dtype}
        if kind == "quantize":
            case["rne"] = rng.random() < 0.3
        return case
    if kind == "lstm":
        return {"kind": kind, "rows": _log_int(rng, 1, 4096), "cols": _extent(rng, 32, 4096), "dtype": rng.choice(["float32", "float32", "float16"])}
    if kind in ("matmul", "qmatmul"):
        while True:
            m, n, k = _extent(rng, 1, 8192), _extent(rng, 16, 8192), _extent(rng, 16, 8192)
            # products whose extents fall as they may stay below the listed ragged one, the others below the listed large one
            if m * n * k <= (509 * 3073 * 1283 if k % 16 else 8192 ** 3):
                break
        case = {"kind": kind, "m": m, "n": n, "k": k}
        if kind == "matmul":
            case["b_dtype"] = rng.choice(["int8", "uint8"])
            case["b_zp"] = "none" if case["b_dtype"] == "int8" else rng.choice(["tensor", "column"])
        return case
    if kind == "conv":
        while True:
            hw = _log_int(rng, 7, 112)
            case = {"kind": kind, "batch": _log_int(rng, 1, 256), "c": _extent(rng, 16, 512), "h": hw, "w": max(7, hw + rng.choice([0, 0, -1, 3])),
                    "m": _extent(rng, 16, 512), "k": rng.choice([1, 3, 3, 5]), "stride": rng.choice([1, 1, 2]), "layout": rng.choice(["nchw", "nchw", "nhwc"]),
                    "depthwise": False, "x_zp": rng.choice([0, 0, rng.randint(1, 255)])}
            if case["layout"] == "nhwc" and rng.random() < 0.4:
                case.update(depthwise=True, m=case["c"], k=3)
            if _conv_macs(case) <= 256 * 28 * 28 * 128 * 128 * 9 and case["batch"] * case["c"] * case["h"] * case["w"] <= 1 << 27:
                return case
    if kind == "dynconv":
        while True:
            hw = _log_int(rng, 7, 112)
            case = {"kind": kind, "batch": _log_int(rng, 1, 64), "c": _extent(rng, 3, 256), "h": hw, "w": max(7, hw + rng.choice([0, 0, -1, 3])),
                    "m": _extent(rng, 16, 256), "k": rng.choice([1, 3, 3, 5]), "stride": rng.choice([1, 1, 2])}
            if _conv_macs(case) <= 8 * 56 * 56 * 64 * 64 * 9:
                return case
    return {"kind": kind, "batch": _log_int(rng, 1, 256 if kind == "resnet50" else 512), "graph": rng.random() < 0.5}


def _out_extent(case, key):
    return (case[key] + 2 * (case["k"] // 2) - case["k"]) // case["stride"] + 1


def _conv_macs(case):
    c = 1 if case.get("depthwise") else case["c"]
    return case["batch"] * case["m"] * _out_extent(case, "h") * _out_extent(case, "w") * c * case["k"] ** 2


# ---- inputs -------------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed))


def _uniform_q(shape, dtype, gen, lo=None):
    t, _, least, most = _QTYPES[dtype]
    return torch.randint(least if lo is None else lo, most + 1, shape, dtype=t, device=_DEV, generator=gen)


def _prepare_mlp(case, seed):
    net = models.QuantizedMLP(_DEV, seed=seed)
    return {"net": net, "x": torch.rand((case["batch"], 784), device=_DEV, generator=_gen(seed)), "packed": case["packed"]}


def _prepare_quantize(case, seed):
    zp = _QTYPES[case["dtype"]][1](case["zp"])
    if case["zp"] == 0 and case["dtype"] == "uint8":  # an image batch
        x, scale = torch.rand(case["n"], device=_DEV, generator=_gen(seed)), 1.0 / 255.0
    else:  # activations with both signs
        x, scale = torch.randn(case["n"], device=_DEV, generator=_gen(seed)), 8.0 / 255.0
    return {"x": x, "scale": scale, "zp": zp, "mode": ops.ROUND_RNE if case["rne"] else ops.ROUND_REF}


def _prepare_dequantize(case, seed):
    return {"x": _uniform_q((case["n"],), case["dtype"], _gen(seed)), "scale": 8.0 / 255.0, "zp": _QTYPES[case["dtype"]][1](case["zp"])}


def _prepare_lstm(case, seed):
    nodes = fusion.lstm_cell_group()
    group = fusion.fuse_elementwise(nodes, {}, ["c_next", "h"])[0]
    code = fusion.build_program(nodes, 1, group.inputs, group.outputs, dtype=case["dtype"])
    gen = _gen(seed)
    ins = [torch.randn((case["rows"], case["cols"]), device=_DEV, generator=gen).to(_FLOATS[case["dtype"]]) for _ in group.inputs]
    return {"inputs": ins, "outputs": len(group.outputs), "code": code}


def _prepare_matmul(case, seed):
    gen = _gen(seed)
    m, n, k = case["m"], case["n"], case["k"]
    state = {"a": _uniform_q((m, k), "uint8", gen), "a_zp": torch.tensor([128], dtype=torch.uint8, device=_DEV), "b_zp": None}
    state["b"] = _uniform_q((k, n), case["b_dtype"], gen, lo=-127 if case["b_dtype"] == "int8" else 0)
    if case["b_zp"] != "none":
        state["b_zp"] = torch.randint(100, 156, (n if case["b_zp"] == "column" else 1,), dtype=torch.uint8, device=_DEV, generator=gen)
    return state


def _prepare_qmatmul(case, seed):
    gen = _gen(seed)
    # the output scale leaves the products' spread inside the 8-bit range
    return {"a": _uniform_q((case["m"], case["k"]), "uint8", gen), "b": _uniform_q((case["k"], case["n"]), "int8", gen, lo=-127),
            "y_scale": 0.01 * 0.001 * 74.0 * 73.0 * math.sqrt(case["k"]) / 40.0}


def _prepare_conv(case, seed):
    gen = _gen(seed)
    c, m, k = case["c"], case["m"], case["k"]
    cg = 1 if case["depthwise"] else c
    x = _uniform_q((case["batch"], c, case["h"], case["w"]), "uint8", gen)
    if case["layout"] == "nhwc":
        x = x.contiguous(memory_format=torch.channels_last)
    return {"x": x, "w": _uniform_q((m, cg, k, k), "int8", gen, lo=-127), "w_scale": torch.rand(m, device=_DEV, generator=gen) * 1e-3 + 5e-4,
            "w_zp": torch.zeros(m, dtype=torch.int8, device=_DEV), "b": torch.randint(-2000, 2001, (m,), dtype=torch.int32, device=_DEV, generator=gen),
            "x_zp": np.uint8(case["x_zp"]), "y_scale": 0.02 * 1e-3 * 74.0 * 73.0 * math.sqrt(cg * k * k) / 40.0, "stride": (case["stride"],) * 2,
            "pad": (k // 2,) * 2, "group": c if case["depthwise"] else 1}


def _prepare_dynconv(case, seed):
    gen = _gen(seed)
    c, m, k = case["c"], case["m"], case["k"]
    return {"x": torch.randn((case["batch"], c, case["h"], case["w"]), device=_DEV, generator=gen), "w": _uniform_q((m, c, k, k), "uint8", gen),
            "w_zp": torch.randint(100, 156, (m,), dtype=torch.uint8, device=_DEV, generator=gen), "stride": (case["stride"],) * 2, "pad": (k // 2,) * 2}


def _prepare_network(case, seed):
    net = (models.ResNet50Int8 if case["kind"] == "resnet50" else models.MobileNetV2Int8)(case["batch"], _DEV, seed=seed)
    x = torch.rand((case["batch"], 3, 224, 224), device=_DEV, generator=_gen(seed))
    if case["graph"]:
        engine = dataparallel.InferenceEngine(net, fold=True)
        engine.prepare(x)
        return {"engine": engine}
    net.calibrate(x)
    return {"net": net, "x": x}


_PREPARE = {"mlp": _prepare_mlp, "quantize": _prepare_quantize, "dequantize": _prepare_dequantize, "lstm": _prepare_lstm, "matmul": _prepare_matmul,
            "qmatmul": _prepare_qmatmul, "conv": _prepare_conv, "dynconv": _prepare_dynconv, "resnet50": _prepare_network,
            "mobilenetv2": _prepare_network}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["kind"] = case["kind"]
    return state


# ---- one pass -----------------------------------------------------------------------------------------------------------


def _run_mlp(s):
    return s["net"].forward_packed(s["x"]) if s["packed"] else s["net"].forward(s["x"])


def _run_quantize(s):
    return ops.QuantizeLinear(s["x"], s["scale"], s["zp"], round_mode=s["mode"])


def _run_dequantize(s):
    return ops.DequantizeLinear(s["x"], s["scale"], s["zp"])


def _run_lstm(s):
    return ops.ElementWiseNvrtc(s["inputs"], s["outputs"], s["code"], 1)


def _run_matmul(s):
    return ops.MatMulInteger(s["a"], s["b"], s["a_zp"], s["b_zp"])


def _run_qmatmul(s):
    return ops.QLinearMatMul(s["a"], 0.01, np.uint8(128), s["b"], 0.001, np.int8(0), s["y_scale"], np.uint8(128))


def _run_conv(s):
    return ops.QLinearConv(s["x"], 0.02, s["x_zp"], s["w"], s["w_scale"], s["w_zp"], s["y_scale"], np.uint8(128), s["b"], s["stride"], s["pad"], s["group"])


def _run_dynconv(s):
    mm = ops.MinMax(s["x"])
    scale, zp = ops.DynamicQuantParamsU8(mm[0:1], mm[1:2])
    return ops.ConvInteger(ops.QuantizeLinear(s["x"], scale, zp), s["w"], zp, s["w_zp"], s["stride"], s["pad"]), scale, zp


def _run_network(s):
    if "engine" in s:
        return s["engine"].step_device()
    return s["net"].forward(s["x"], fold=True)


_RUN = {"mlp": _run_mlp, "quantize": _run_quantize, "dequantize": _run_dequantize, "lstm": _run_lstm, "matmul": _run_matmul, "qmatmul": _run_qmatmul,
        "conv": _run_conv, "dynconv": _run_dynconv, "resnet50": _run_network, "mobilenetv2": _run_network}


def run(state):
    return _RUN[state["kind"]](state)


# ---- what a pass cannot do without --------------------------------------------------------------------------------------


def _resnet50_counts():
    """(multiply-accumulates per image, weights) of models.ResNet50Int8 at 224 x 224."""
    macs, weights, hw, cin = 64 * 147 * 112 * 112, 64 * 147, 56, 64
    for blocks, mid, cout, stride in models.RESNET50_STAGES:
        for i in range(blocks):
            hw = hw // stride if i == 0 else hw
            layer = cin * mid + 9 * mid * mid + mid * cout + (cin * cout if i == 0 else 0)
            macs, weights, cin = macs + layer * hw * hw, weights + layer, cout
    return macs + cin * 1000, weights + 4 * cin * 1000


def _mobilenetv2_counts():
    macs, weights, hw, cin = 32 * 27 * 112 * 112, 32 * 27, 112, 32
    for t, c, n, s in models.MOBILENETV2_BLOCKS:
        for i in range(n):
            mid, out = cin * t, hw // s if i == 0 else hw
            expand = cin * mid if t != 1 else 0
            macs += expand * hw * hw + (9 * mid + mid * c) * out * out
            weights, hw, cin = weights + expand + 9 * mid + mid * c, out, c
    return macs + cin * 1280 * hw * hw + 1280 * 1000, weights + cin * 1280 + 4 * 1280 * 1000


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        weights = 784 * 1000 + 1000 * 1000 + 1000 * 10
        return {"bytes": case["batch"] * 4 * (784 + 10) + weights, "flops": 2 * case["batch"] * weights}
    if kind in ("quantize", "dequantize"):
        return {"bytes": 5 * case["n"], "flops": 2 * case["n"]}
    if kind == "lstm":
        n = case["rows"] * case["cols"]
        return {"bytes": 7 * n * (4 if case["dtype"] == "float32" else 2), "flops": 30 * n}  # five transcendental functions and four operations
    if kind in ("matmul", "qmatmul"):
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": m * k + k * n + m * n * (4 if kind == "matmul" else 1), "flops": 2 * m * n * k}
    if kind in ("conv", "dynconv"):
        x = case["batch"] * case["c"] * case["h"] * case["w"]
        y = case["batch"] * case["m"] * _out_extent(case, "h") * _out_extent(case, "w")
        w = case["m"] * (1 if case.get("depthwise") else case["c"]) * case["k"] ** 2
        return {"bytes": x + w + y if kind == "conv" else 4 * x + w + 4 * y, "flops": 2 * _conv_macs(case)}
    # networks: the image batch, the weights and the logits; the maps between the layers are the implementation's own affair
    macs, weights = _resnet50_counts() if kind == "resnet50" else _mobilenetv2_counts()
    return {"bytes": case["batch"] * 4 * (3 * 224 * 224 + 1000) + weights, "flops": 2 * case["batch"] * macs}


def tolerance(case):
    """Quantized values and integer accumulators are the same bytes whatever the order of the sums; floats agree to fp32 rounding (of
    the classifier's sums, or of the fused group's functions), half-precision results to their own spacing."""
    if case["kind"] == "lstm" and case["dtype"] == "float16":
        return {"rel": 1e-3}
    if case["kind"] in ("mlp", "dequantize", "lstm", "resnet50", "mobilenetv2"):
        return {"rel": 1e-5}
    if case["kind"] == "dynconv":
        return {"rel": 1e-6}
    return "exact"

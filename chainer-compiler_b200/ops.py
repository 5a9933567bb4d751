"""Host-side mirror of the reference's VM op bodies for the quantized hot path.

Each function has the name, argument order and argument meaning of the corresponding entry of
the reference's op table (``runtime/chxvm_defs.py:431-434,451-469``) and does what the reference's
``XxxOp::RunImpl`` does around the arithmetic: validate, allocate a fresh output, call the kernel.
The bodies themselves are native (``csrc/native.cc``, the extension ``_native``), because the host work of an interpreted
body costs several kernel launches; the functions here hold the signatures and their documentation.  The arithmetic
runs in ``libchxq.so`` through the C ABI; PyTorch supplies device memory and the current stream only.  There is no
fallback: without a CUDA device or without the built libraries every op raises.

Array arguments are ``torch`` CUDA tensors, logically NCHW / row-major as in the reference.
Activation maps that are ``channels_last`` in memory take the NHWC kernels (tensor cores,
depthwise kernel) as they are and yield ``channels_last`` outputs; plain contiguous NCHW maps yield NCHW outputs
(dense convolutions run on the tensor cores all the same, behind a pass that rewrites the map).  ``Scalar`` arguments are Python / numpy scalars; a zero point carries its dtype
as a numpy scalar (``np.uint8(3)``, ``np.int8(-1)``) the way ``StrictScalar`` does in the reference
(``runtime/strict_scalar.h:8-34``).
"""
import ctypes

import numpy as np
import torch

from . import _lib
from ._lib import (FLOAT16, FLOAT32, FLOAT64, INT8, NCHW, NHWC, PATH_AUTO, PATH_SIMT, PATH_TENSOR, ROUND_REF, ROUND_RNE, UINT8,  # noqa: F401
                   ChxqError, ConvGeom, QConvParams, check, lib)

_lib.lib()  # libchxq.so, or a clear error
try:
    from . import _native
except ImportError as e:
    raise _lib.ChxqLibraryError("_native.so is missing or does not load (%s); build it with `make -C %s` (this package has no fallback path)" % (e, _lib.CSRC))

_TORCH_Q = {torch.uint8: UINT8, torch.int8: INT8}


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "chxq ops run on CUDA tensors only (no CPU path exists)")


def _qcode(t, what):
    if t.dtype not in _TORCH_Q:
        raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "%s must be uint8 or int8, got %s" % (what, t.dtype))
    return _TORCH_Q[t.dtype]


def workspace(nbytes, device):
    """Scratch for one library call on the current stream, 256-byte aligned: a block of the caching allocator, the caller's until it lets
    go of the tensor.  (Calls on other streams and in other threads have their own.)"""
    return None if nbytes == 0 else torch.empty(int(nbytes), dtype=torch.uint8, device=device)


def _to_device_array(v, like, kind):
    """A parameter given as a number or host array, on the device of `like`; kind "f" makes it float32."""
    return torch.as_tensor(np.asarray(v, np.float32) if kind == "f" else np.asarray(v), device=like.device)


def _zp_scalar(zp, default_dtype=np.uint8):
    """(value, chxq dtype code) of an OptionalScalar zero point."""
    if zp is None:
        return 0, (UINT8 if default_dtype == np.uint8 else INT8)
    if isinstance(zp, torch.Tensor):
        if zp.numel() != 1:
            raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "a Scalar zero point must have one element")
        return int(zp.item()), _qcode(zp, "zero point")
    if isinstance(zp, (np.generic, np.ndarray)):
        dt = np.asarray(zp).dtype
        if dt == np.int8:
            return int(zp), INT8
        if dt == np.uint8:
            return int(zp), UINT8
        # runtime/ops/quantize.cc:19-25: the zero point's dtype is uint8 or int8, anything else CHECK-fails
        raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "a zero point must be uint8 or int8, got %s" % dt)
    # plain Python ints carry no dtype: the reference's default is uint8 (runtime/ops/quantize.cc:50-51)
    return int(zp), (UINT8 if default_dtype == np.uint8 else INT8)


def _is_channels_last(t):
    return t.dim() == 4 and t.is_contiguous(memory_format=torch.channels_last) and not (t.is_contiguous() and t.shape[1] != 1)


_native.setup(ChxqError, _zp_scalar, _to_device_array, np.uint8, np.int8)


def QuantizeLinear(x, y_scale, y_zero_point=None, round_mode=ROUND_REF):
    """runtime/chxvm_defs.py:451-453; body runtime/ops/quantize.cc:16-35,48-53.

    y_scale (and y_zero_point) may be one-element CUDA tensors: the scalars are then read by the kernel on the device, without
    the device-to-host read the reference's VM does per Scalar argument (runtime/chxvm_var.cc:70-76)."""
    return _native.quantize_linear(x, y_scale, y_zero_point, round_mode)


def DequantizeLinear(x, x_scale, x_zero_point=None):
    """runtime/chxvm_defs.py:454-456; body runtime/ops/quantize.cc:37-44,55-60."""
    return _native.dequantize_linear(x, x_scale, x_zero_point)


def _zp_array(zp, like, what):
    """OptionalArray zero point: device tensor of the operand's dtype with ndim <= 1."""
    if zp is None:
        return None, 0
    if not isinstance(zp, torch.Tensor):
        zp = torch.as_tensor(np.asarray(zp), device=like.device)
    _require_cuda(zp)
    if zp.dim() > 1:
        raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "%s must have at most one dimension" % what)  # runtime/ops/quantize.cc:105,109
    if zp.dtype != like.dtype:
        raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "%s must have the operand's dtype %s, got %s" % (what, like.dtype, zp.dtype))
    zp = zp.contiguous().reshape(-1)
    return zp, zp.numel()


def MatMulInteger(a, b, a_zero_point=None, b_zero_point=None, path=PATH_AUTO):
    """runtime/chxvm_defs.py:462-465; body runtime/ops/quantize.cc:96-114."""
    return _native.matmul_integer(a, b, a_zero_point, b_zero_point, path)


def QLinearMatMul(a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point, round_mode=ROUND_REF, path=PATH_AUTO):
    """ONNX QLinearMatMul.  The reference has no VM op for it: compiler/simplifier.cc:675-694 rewrites the
    node into DequantizeLinear, DequantizeLinear, MatMul, QuantizeLinear with scalar parameters; this is
    that chain as one kernel."""
    return _native.qlinear_matmul(a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point, round_mode, path)


def conv_geometry(x, w, strides, pads, group, auto_pad):
    """Geometry of a convolution the way the reference resolves it (runtime/chainerx_util.cc:180-200,276-311)."""
    return conv_geometry_from_shapes(tuple(x.shape), _qcode(x, "x"), tuple(w.shape), _qcode(w, "w"), strides, pads, group, auto_pad)


def conv_geometry_from_shapes(x_shape, x_code, w_shape, w_code, strides, pads, group, auto_pad):
    if len(x_shape) != 4 or len(w_shape) != 4:
        raise ChxqError(_lib.ERR_UNSUPPORTED, "convolutions over 2 spatial dimensions only")
    N, C, H, W = x_shape
    M, Cg, KH, KW = w_shape
    g = ConvGeom()
    s = (ctypes.c_int64 * 2)(*(list(strides) + [1, 1])[:2])
    p = (ctypes.c_int64 * 2)(*(list(pads) + [0, 0])[:2])
    check(lib().chxq_conv_resolve_geometry(N, C, H, W, M, Cg, KH, KW, s, len(strides), p, len(pads), group, (auto_pad or "").encode(),
                                           ctypes.byref(g)))
    g.x_dtype = x_code
    g.w_dtype = w_code
    return g


def ConvInteger(x, w, x_zero_point=None, w_zero_point=None, strides=(), pads=(), group=1, auto_pad="", path=PATH_AUTO):
    """runtime/chxvm_defs.py:466-469; body runtime/ops/quantize.cc:116-146.

    x_zero_point may be a one-element CUDA tensor of x's dtype (a zero point computed on the device): it is then read by the
    kernel, not by the host (on the tensor cores; tiny and grouped convolutions and PATH_SIMT on the general CUDA-core kernel)."""
    return _native.conv_integer(x, w, x_zero_point, w_zero_point, strides, pads, group, auto_pad, path)


def QLinearConv(x, x_scale, x_zero_point, w, w_scale, w_zero_point, y_scale, y_zero_point, b=None, strides=(), pads=(), group=1,
                auto_pad="", round_mode=ROUND_REF, path=PATH_AUTO, clamp_hi_q=None, residual=None, res_scale=1.0, res_zero_point=0,
                res_relu=True, out_scale=1.0, out_zero_point=0, fold_scales=False):
    """runtime/chxvm_defs.py:457-461; body runtime/ops/quantize.cc:62-94.

    The keyword arguments after ``auto_pad`` have no counterpart in the reference: ``clamp_hi_q`` folds a
    ReLU6 into the output range, ``residual`` (+ scales) fuses the DequantizeLinear, DequantizeLinear, Add,
    Relu, QuantizeLinear nodes that follow the convolution of a residual block into the epilogue,
    ``fold_scales`` requantizes with one multiplier per channel instead of a multiply and a divide.
    """
    return _native.qlinear_conv(x, w, strides, pads, group, auto_pad, path, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b,
                                round_mode, clamp_hi_q, residual, res_scale, res_zero_point, res_relu, out_scale, out_zero_point, fold_scales)


class PackedConv:
    """Constant weights of one QLinearConv / ConvInteger, packed once for the tensor-core path."""

    def __init__(self, w, w_zero_point, x_shape, strides=(), pads=(), group=1, auto_pad="", x_dtype=torch.uint8, x_layout=NHWC):
        _require_cuda(w)
        self.w = w.contiguous()
        self.g = conv_geometry_from_shapes(tuple(x_shape), _TORCH_Q[x_dtype], tuple(self.w.shape), _qcode(self.w, "w"), strides, pads, group,
                                           auto_pad)
        self.g.x_layout, self.g.y_layout = x_layout, NHWC
        self.zw, self.zw_len = _zp_array(w_zero_point, self.w, "w_zero_point")
        nbytes = lib().chxq_conv_prepack_bytes(ctypes.byref(self.g))
        self.flags = 0
        self.blob = None
        if nbytes:
            self.blob = torch.empty(int(nbytes), dtype=torch.uint8, device=w.device)
            flags = ctypes.c_int32(0)
            check(lib().chxq_conv_prepack(_ptr(self.w), ctypes.byref(self.g), _ptr(self.zw), self.zw_len, _ptr(self.blob), nbytes,
                                          ctypes.byref(flags), _stream()))
            self.flags = flags.value

    @property
    def eligible(self):
        return bool(self.flags & 1)


def QLinearConvPacked(x, packed, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b=None, round_mode=ROUND_REF,
                      clamp_hi_q=None, residual=None, res_scale=1.0, res_zero_point=0, res_relu=True, out_scale=1.0, out_zero_point=0,
                      out=None, fold_scales=False):
    """QLinearConv with weights packed by PackedConv; x must be a channels_last map of the packed geometry."""
    return _native.qlinear_conv_packed(x, packed, out, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b, round_mode, clamp_hi_q,
                                       residual, res_scale, res_zero_point, res_relu, out_scale, out_zero_point, fold_scales)


def QLinearConvChainPacked(x, packed1, conv1, packed2, conv2, out=None):
    """Two QLinearConvPacked calls as one kernel: `packed1` / `conv1` describe a convolution with 64, 128 or 256 output channels,
    `packed2` / `conv2` the 1x1, stride-1 convolution that is its only reader.  conv1 and conv2 are dicts of the keyword arguments
    QLinearConvPacked takes after `packed` (x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b, clamp_hi_q,
    fold_scales, and for conv2 the residual tail's residual, res_scale, res_zero_point, res_relu, out_scale, out_zero_point).  The
    map between the two convolutions is never written.  Bit-identical to the two calls in sequence; raises
    ChxqError(ERR_UNSUPPORTED) when the pair has no fused kernel (the caller then makes the two calls)."""
    return _native.qlinear_conv_chain_packed(x, packed1, packed2, out, *_chain_params(conv1), *_chain_params(conv2))


def _chain_params(c):
    return (c["x_scale"], c["x_zero_point"], c["w_scale"], c.get("w_zero_point"), c["y_scale"], c["y_zero_point"], c.get("b"),
            c.get("round_mode", ROUND_REF), c.get("clamp_hi_q"), c.get("residual"), c.get("res_scale", 1.0), c.get("res_zero_point", 0),
            c.get("res_relu", True), c.get("out_scale", 1.0), c.get("out_zero_point", 0), c.get("fold_scales", False))


def QLinearConvMaxPoolPacked(x, packed, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b=None, pool_kernel=3, pool_stride=2,
                             pool_pad=0, cover_all=False, round_mode=ROUND_REF, quant_round_mode=ROUND_REF, clamp_hi_q=None, out=None,
                             fold_scales=False):
    """QLinearConvPacked followed by MaxPoolU8(pool_kernel, pool_stride, pool_pad, cover_all) as one kernel; bit-identical to the
    two ops.  x: the uint8 map, or the fp32 tensor in front of a QuantizeLinear(x_scale, x_zero_point) (as
    QuantizeLinearConvPacked).  Only kernel 3 / stride 2 / pad 0 pooling behind a convolution whose packed K tile is 64 bytes
    (network stems); raises ChxqError(ERR_UNSUPPORTED) otherwise."""
    return _native.qlinear_conv_maxpool_packed(x, packed, pool_kernel, pool_stride, pool_pad, cover_all, quant_round_mode, out, x_scale, x_zero_point,
                                               w_scale, w_zero_point, y_scale, y_zero_point, b, round_mode, clamp_hi_q, None, 1.0, 0, True, 1.0, 0,
                                               fold_scales)


def ConvIntegerPacked(x, packed, x_zero_point=None):
    """ConvInteger with weights packed by PackedConv; x must be a channels_last map of the packed geometry."""
    return _native.conv_integer_packed(x, packed, x_zero_point)


def QuantizeLinearConvPacked(x, packed, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b=None, round_mode=ROUND_REF,
                             quant_round_mode=ROUND_REF, clamp_hi_q=None, out=None, fold_scales=False):
    """QuantizeLinear(x, x_scale, x_zero_point) fused into the packed QLinearConv that consumes it: x is the fp32 tensor (same
    layout as the packed geometry expects of the quantized map).  Only for stride-2 convolutions over at most 4 channels
    (network stems); bit-identical to the two ops run one after the other."""
    return _native.quantize_qlinear_conv_packed(x, packed, quant_round_mode, out, x_scale, x_zero_point, w_scale, w_zero_point, y_scale, y_zero_point, b,
                                                round_mode, clamp_hi_q, None, 1.0, 0, True, 1.0, 0, fold_scales)


def ElementWiseNvrtc(inputs, num_outputs, code, fusion_id):
    """runtime/chxvm_defs.py:431-434; body runtime/ops/nvrtc.cc:90-161: broadcast every input to the common
    shape, make it contiguous, allocate num_outputs arrays of that shape and dtype, run the generated kernel."""
    return _native.elementwise(inputs, num_outputs, code, fusion_id)


# ---- glue ops of a quantized CNN graph -------------------------------------------------------------

def MaxPoolU8(x, kernel, stride, pad=0, cover_all=False):
    """MaxPool (runtime/ops/pooling.cc:47-60) on a uint8 channels_last map."""
    return _native.maxpool_u8(x, kernel, stride, pad, cover_all)


def GlobalAveragePoolDequant(x, x_scale, x_zero_point=0):
    """DequantizeLinear followed by a global AveragePool (runtime/ops/pooling.cc:62-75) of a uint8 channels_last map -> [N, C] fp32."""
    return _native.global_avgpool_dq(x, x_scale, x_zero_point)


def Linear(x, w, b=None):
    """runtime/ops/connection.cc:12-15 (fp32): y = x w^T + b."""
    return _native.linear(x, w, b)


def QAddU8(a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point=0, relu=True, round_mode=ROUND_REF):
    """DequantizeLinear(a), DequantizeLinear(b), Add, Relu, QuantizeLinear in one pass (same memory layout in and out)."""
    return _native.qadd_u8(a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point, relu, round_mode)


def to_channels_last(x):
    """NCHW -> NHWC copy of a 1- or 4-byte map through the library's transpose kernel."""
    _require_cuda(x)
    if _is_channels_last(x):
        return x
    return _native.transpose_map(x.contiguous(), True)


def to_contiguous_nchw(x):
    _require_cuda(x)
    if x.is_contiguous():
        return x
    if not _is_channels_last(x):
        return x.contiguous()
    return _native.transpose_map(x, False)


def PrepareWeights(w, bn=None, conv_bias=None, epsilon=1e-5, to_int8=True, per_channel=True, return_folded=False):
    """Model preparation on the device: the Conv + BatchNormalization merge (compiler/merge.cc:142-215) followed by the weight
    quantizer (compiler/quantize.cc:70-129).  w: fp32 [M, ...]; bn: None or (scale, bias, mean, var), fp32 [M] each.
    Returns (q, scales, zero_points, folded_bias or None[, folded_w]); zero_points are int32."""
    _require_cuda(w)
    if w.dtype != torch.float32:
        raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "PrepareWeights: w must be float32")
    w = w.contiguous()
    M = w.shape[0]
    inner = w.numel() // M
    vec = lambda t: None if t is None else t.to(device=w.device, dtype=torch.float32).contiguous()  # noqa: E731
    gamma, beta, mean, var = (vec(t) for t in bn) if bn is not None else (None, None, None, None)
    conv_bias = vec(conv_bias)
    for t in (gamma, beta, mean, var, conv_bias):
        if t is not None and t.numel() != M:
            raise ChxqError(_lib.ERR_INVALID_ARGUMENT, "PrepareWeights: per-channel vectors need one entry per output channel")
    n = M if per_channel else 1
    q = torch.empty(w.shape, dtype=torch.int8 if to_int8 else torch.uint8, device=w.device)
    scales = torch.empty(n, dtype=torch.float32, device=w.device)
    zps = torch.empty(n, dtype=torch.int32, device=w.device)
    folded_bias = torch.empty(M, dtype=torch.float32, device=w.device) if bn is not None else None
    folded_w = torch.empty_like(w) if return_folded else None
    ws_bytes = lib().chxq_prepare_weights_workspace(M)
    ws = workspace(ws_bytes, w.device)
    p = lambda t: None if t is None else _ptr(t)  # noqa: E731
    check(lib().chxq_prepare_weights(_ptr(w), M, inner, p(gamma), p(beta), p(mean), p(var), float(epsilon), p(conv_bias), int(to_int8), int(per_channel),
                                     _ptr(q), _ptr(scales), _ptr(zps), p(folded_w), p(folded_bias), _ptr(ws), ws_bytes, _stream()))
    return (q, scales, zps, folded_bias, folded_w) if return_folded else (q, scales, zps, folded_bias)


def DynamicQuantParamsU8(rmin, rmax):
    """scale, zero point of the dynamic uint8 quantization of an activation from its ReduceMin / ReduceMax, as the Sub, Div,
    Floor, Cast nodes of compiler/quantize.cc:196-207 compute them, on the device: returns (float32[1], uint8[1]) CUDA tensors."""
    return _native.dynamic_params_u8(rmin, rmax)


def MinMax(x):
    """ReduceMin and ReduceMax of an fp32 tensor in one pass -> device tensor [min, max]."""
    return _native.minmax(x)


def device_status():
    """Raises if a bounded device-side wait expired since the last call (synchronises the stream)."""
    check(lib().chxq_device_status(_stream()))

// Host bodies of the VM ops over torch tensors: what ops.py's functions do around the C ABI -- check the arguments, allocate the
// output, find scratch, call the library on the current stream -- as a CPython extension (_native.so).
//
// Why native: the interpreted bodies (attribute look-ups, torch.empty, ctypes conversions) cost 12 us per QuantizeLinear and 22 us per
// packed QLinearConv, three to ten times the kernel launch itself, so that everything smaller than about a million elements and every
// network below a few dozen images ran at the speed of the interpreter.  A call through this file costs 3-5 us.  Functions take
// positional arguments only (METH_FASTCALL); ops.py holds the public signatures and their documentation.
//
// The interpreter lock is released around the library call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <stdarg.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/chxq.h"

namespace {

// ---- errors ---------------------------------------------------------------------------------------------------------------

struct OpError {
    int code;
    std::string msg;
};
struct PyErrSet {};  // a Python exception is already set

PyObject* g_error_class = nullptr;  // _lib.ChxqError
PyObject* g_helpers[3] = {};        // ops._zp_scalar, ops._to_device_array
PyTypeObject *g_np_uint8 = nullptr, *g_np_int8 = nullptr;

[[noreturn]] __attribute__((format(printf, 2, 3))) void fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    throw OpError{code, buf};
}

PyObject* raise(const OpError& e) {
    PyObject* exc = PyObject_CallFunction(g_error_class, "is", e.code, e.msg.c_str());
    if (exc) {
        PyErr_SetObject(g_error_class, exc);
        Py_DECREF(exc);
    }
    return nullptr;
}

// The interpreter lock, given up until the end of the scope -- also by an exception (a tensor without storage throws when it is asked for its
// address), which is turned into a Python one by code that needs the lock.
struct Unlocked {
    PyThreadState* save = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked&) = delete;
    ~Unlocked() { PyEval_RestoreThread(save); }
};

// Runs a library call without the interpreter lock and turns its status into an exception.
template <typename F>
void call(F&& f) {
    int rc;
    {
        const Unlocked unlocked;
        rc = f();
    }
    if (rc != CHXQ_OK) throw OpError{rc, chxq_last_error()};
}

#define OP_BEGIN     \
    HANDLE_TH_ERRORS \
    try {
#define OP_END                 \
    }                          \
    catch (const OpError& e) { \
        return raise(e);       \
    }                          \
    catch (const PyErrSet&) {  \
        return nullptr;        \
    }                          \
    END_HANDLE_TH_ERRORS

void need_args(const char* op, Py_ssize_t got, Py_ssize_t want) {
    if (got != want) {
        PyErr_Format(PyExc_TypeError, "%s: expected %zd arguments, got %zd", op, want, got);
        throw PyErrSet{};
    }
}

// ---- arguments ------------------------------------------------------------------------------------------------------------

inline bool is_tensor(PyObject* o) {
    return THPVariable_Check(o);
}

const at::Tensor& tensor(PyObject* o, const char* what) {
    if (!is_tensor(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor, got %s", what, Py_TYPE(o)->tp_name);
        throw PyErrSet{};
    }
    return THPVariable_Unpack(o);
}

void require_cuda(const at::Tensor& t) {
    if (!t.is_cuda()) fail(CHXQ_ERR_INVALID_ARGUMENT, "chxq ops run on CUDA tensors only (no CPU path exists)");
}

std::string dtype_name(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return "torch.float32";
        case at::kDouble: return "torch.float64";
        case at::kHalf: return "torch.float16";
        case at::kBFloat16: return "torch.bfloat16";
        case at::kByte: return "torch.uint8";
        case at::kChar: return "torch.int8";
        case at::kInt: return "torch.int32";
        case at::kLong: return "torch.int64";
        case at::kBool: return "torch.bool";
        default: return std::string("torch.") + c10::toString(t.scalar_type());
    }
}

int qcode(const at::Tensor& t, const char* what) {
    if (t.scalar_type() == at::kByte) return CHXQ_UINT8;
    if (t.scalar_type() == at::kChar) return CHXQ_INT8;
    fail(CHXQ_ERR_INVALID_ARGUMENT, "%s must be uint8 or int8, got %s", what, dtype_name(t).c_str());
}

inline at::ScalarType qtype(int code) {
    return code == CHXQ_UINT8 ? at::kByte : at::kChar;
}

double as_double(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyErrSet{};
    return v;
}

long as_long(PyObject* o) {
    if (PyLong_CheckExact(o)) {
        const long v = PyLong_AsLong(o);
        if (v == -1 && PyErr_Occurred()) throw PyErrSet{};
        return v;
    }
    PyObject* n = PyNumber_Long(o);  // int(o): numpy scalars, floats, one-element arrays
    if (!n) throw PyErrSet{};
    const long v = PyLong_AsLong(n);
    Py_DECREF(n);
    if (v == -1 && PyErr_Occurred()) throw PyErrSet{};
    return v;
}

bool as_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyErrSet{};
    return v != 0;
}

struct Zp {
    int value, code;
};

// An OptionalScalar zero point and the dtype it carries: absent and plain integers are uint8 (runtime/ops/quantize.cc:50-51); numpy
// scalars bring theirs; everything else (tensors, arrays, wrong types) goes through ops._zp_scalar.
Zp zp_scalar(PyObject* o) {
    if (o == Py_None) return {0, CHXQ_UINT8};
    if (Py_TYPE(o) == g_np_uint8) return {(int)as_long(o), CHXQ_UINT8};
    if (Py_TYPE(o) == g_np_int8) return {(int)as_long(o), CHXQ_INT8};
    if (PyLong_CheckExact(o)) return {(int)as_long(o), CHXQ_UINT8};
    PyObject* r = PyObject_CallOneArg(g_helpers[0], o);
    if (!r) throw PyErrSet{};
    Zp z{0, 0};
    if (!PyArg_ParseTuple(r, "ii", &z.value, &z.code)) {
        Py_DECREF(r);
        throw PyErrSet{};
    }
    Py_DECREF(r);
    return z;
}

bool is_channels_last(const at::Tensor& t) {
    return t.dim() == 4 && t.is_contiguous(at::MemoryFormat::ChannelsLast) && !(t.is_contiguous() && t.size(1) != 1);
}

bool is_device_scalar(PyObject* o) {
    if (!is_tensor(o)) return false;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.numel() == 1;
}

// A parameter that may come as a number or an array: a device tensor of it (kind "f": float32, "": its own type).
at::Tensor device_array(PyObject* o, const at::Tensor& like, const char* kind) {
    if (is_tensor(o)) return THPVariable_Unpack(o);
    PyObject* dev = THPVariable_Wrap(like);
    PyObject* r = PyObject_CallFunction(g_helpers[1], "OOs", o, dev, kind);
    Py_XDECREF(dev);
    if (!r) throw PyErrSet{};
    if (!is_tensor(r)) {
        Py_DECREF(r);
        PyErr_SetString(PyExc_TypeError, "expected a tensor");
        throw PyErrSet{};
    }
    at::Tensor t = THPVariable_Unpack(r);
    Py_DECREF(r);
    return t;
}

// Contiguous, or channels-last, or else a contiguous copy: the element order of the copy-free forms is the memory order.
at::Tensor dense(const at::Tensor& x) {
    return x.is_contiguous() || is_channels_last(x) ? x : x.contiguous();
}

at::Tensor empty_like_as(const at::Tensor& x, at::ScalarType dtype) {
    return at::detail::empty_strided_cuda(x.sizes(), x.strides(), dtype, x.device());
}

at::Tensor empty_map(at::IntArrayRef size, at::ScalarType dtype, const at::Tensor& like, bool channels_last) {
    return at::detail::empty_cuda(size, dtype, like.device(), channels_last ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous);
}

inline void* stream() {
    return c10::cuda::getCurrentCUDAStream().stream();
}

inline PyObject* wrap(at::Tensor&& t) {
    return THPVariable_Wrap(std::move(t));
}

// Zero point as an optional device array of the operand's dtype with at most one dimension.
struct ZpArray {
    at::Tensor t;
    const void* ptr = nullptr;
    int64_t len = 0;
};

ZpArray zp_array(PyObject* o, const at::Tensor& like, const char* what) {
    ZpArray z;
    if (o == Py_None) return z;
    z.t = device_array(o, like, "");
    require_cuda(z.t);
    if (z.t.dim() > 1) fail(CHXQ_ERR_INVALID_ARGUMENT, "%s must have at most one dimension", what);  // runtime/ops/quantize.cc:105,109
    if (z.t.scalar_type() != like.scalar_type())
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s must have the operand's dtype %s, got %s", what, dtype_name(like).c_str(), dtype_name(z.t).c_str());
    z.t = z.t.contiguous();
    z.ptr = z.t.data_ptr();
    z.len = z.t.numel();
    return z;
}

// ---- scratch --------------------------------------------------------------------------------------------------------------

// Scratch of one call, from the caching allocator on the device and stream the launch goes to: calls on several streams or threads stay
// independent of one another, a graph captured around a call owns its scratch with the rest of its pool, and the block is reused by whatever
// comes next on the stream.  (One grow-only buffer per device, as these bodies had, saves the allocator's half microsecond and lets two streams
// overwrite each other's operands.)
struct OwnScratch {
    at::Tensor t;
    void* get(size_t nbytes) {
        if (nbytes == 0) return nullptr;
        t = at::detail::empty_cuda({(int64_t)nbytes}, at::kByte, c10::Device(c10::kCUDA, c10::cuda::current_device()), std::nullopt);
        return t.data_ptr();
    }
    // For calls that have a form without scratch, which the library takes when it gets none.
    void* get_if_room(size_t nbytes) {
        try {
            return get(nbytes);
        } catch (const c10::OutOfMemoryError&) {
            return nullptr;
        }
    }
};

// ---- QLinearConv parameters -----------------------------------------------------------------------------------------------

// Whether a weight zero-point tensor holds only zeros, learned by ONE device-to-host read per tensor (and again after an in-place change,
// which bumps the tensor's version): weight zero points are graph constants, and symmetric int8 weights, the common case, have none.
// The C ABI treats a zero point that is present as non-zero, because it never reads device memory back; this op body is the place that
// may know better, as the reference's VM knows its constants at Init.  An entry holds a weak reference to the storage it describes, so
// that a tensor that reuses a freed tensor's address is read anew.
struct ZeroEntry {
    c10::weak_intrusive_ptr<c10::StorageImpl> storage;
    uint32_t version;
    bool zero;
};

bool weight_zero_points_are_zero(const at::Tensor& wz) {
    if (wz.is_inference()) return false;  // no version counter, so nothing learned about it can be kept: the general form
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing((cudaStream_t)stream(), &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
        return false;  // no synchronization during a capture: the general form
    static auto& cache = *new std::map<std::tuple<const void*, int64_t, int>, ZeroEntry>;
    const auto key = std::make_tuple((const void*)wz.data_ptr(), wz.numel(), (int)wz.scalar_type());
    const uint32_t version = wz._version();
    const auto it = cache.find(key);
    if (it != cache.end() && it->second.version == version && it->second.storage.lock().get() == wz.storage().unsafeGetStorageImpl()) return it->second.zero;
    bool zero;
    {
        const Unlocked unlocked;  // the read waits for the stream: other Python threads go on meanwhile
        zero = !wz.ne(0).any().item<bool>();
    }
    if (cache.size() > 4096) cache.clear();
    cache.insert_or_assign(key, ZeroEntry{c10::weak_intrusive_ptr<c10::StorageImpl>(wz.storage().getWeakStorageImpl()), version, zero});
    return zero;
}

struct ConvParams {
    chxq_qconv_params p;
    int y_code;
    at::Tensor w_scale, w_zp, bias;  // alive until the launch has been enqueued
};

// The sixteen trailing arguments of the QLinearConv family, in this order: x_scale, x_zero_point, w_scale, w_zero_point, y_scale,
// y_zero_point, b, round_mode, clamp_hi_q, residual, res_scale, res_zero_point, res_relu, out_scale, out_zero_point, fold_scales.
constexpr int kConvArgs = 16;

void conv_params(PyObject* const* a, const at::Tensor& like, const at::Tensor& w, bool packed, ConvParams* out) {
    chxq_qconv_params& p = out->p;
    memset(&p, 0, sizeof(p));
    p.fold_scales = as_bool(a[15]);
    const Zp zx = zp_scalar(a[1]), zy = zp_scalar(a[5]);
    out->w_scale = device_array(a[2], like, "f");
    out->w_zp = device_array(a[3], like, "");
    at::Tensor &ws = out->w_scale, &wz = out->w_zp;
    require_cuda(ws);
    require_cuda(wz);
    // runtime/ops/quantize.cc:76-77: scale and zero point agree in size and rank; rank is 0 or 1.
    if (ws.numel() != wz.numel() || ws.dim() != wz.dim() || ws.dim() > 1)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConv: w_scale and w_zero_point must both be 0-d or both be 1-d of equal length");
    if (ws.dim() == 1 && ws.size(0) != w.size(0))
        fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConv: per-channel w_scale needs one entry per output channel");  // :79
    if (ws.scalar_type() != at::kFloat || wz.scalar_type() != w.scalar_type())
        fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConv: w_scale must be float32 and w_zero_point must have w's dtype");
    ws = ws.contiguous();
    wz = wz.contiguous();
    p.x_scale = (float)as_double(a[0]);
    p.x_zero_point = zx.value;
    p.w_scale = static_cast<const float*>(ws.data_ptr());
    p.w_zero_point = wz.data_ptr();
    p.w_params_len = ws.numel();
    // symmetric weights: the kernels skip the weight zero-point term (and its input sums); packed weights carry that in their flags
    if (!packed && weight_zero_points_are_zero(wz)) p.w_zero_point = nullptr;
    p.y_scale = (float)as_double(a[4]);
    p.y_zero_point = zy.value;
    p.y_dtype = out->y_code = zy.code;
    if (a[6] != Py_None) {
        out->bias = tensor(a[6], "QLinearConv: bias");
        require_cuda(out->bias);
        if (out->bias.scalar_type() != at::kInt || out->bias.numel() != w.size(0))
            fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConv: bias must be int32 with one entry per output channel");
        out->bias = out->bias.contiguous();
        p.bias = static_cast<const int32_t*>(out->bias.data_ptr());
    }
    p.round_mode = (int32_t)as_long(a[7]);
    p.clamp_hi_q = a[8] == Py_None ? -1 : (int32_t)as_long(a[8]);
    if (a[9] != Py_None) {
        const at::Tensor& r = tensor(a[9], "QLinearConv: residual");
        require_cuda(r);
        p.residual = r.data_ptr();
        p.res_scale = (float)as_double(a[10]);
        p.res_zero_point = (int32_t)as_long(a[11]);
        p.res_relu = as_bool(a[12]);
        p.out_scale = (float)as_double(a[13]);
        p.out_zero_point = (int32_t)as_long(a[14]);
    }
}

// A fused residual is read with the output's indexing: a uint8 map of the output's shape and layout, and the tensor-core kernels read
// it 16 bytes at a time.
void check_residual(const char* op, PyObject* o, at::IntArrayRef y_size, bool channels_last) {
    if (o == Py_None) return;
    const at::Tensor& r = tensor(o, "residual");
    if (r.sizes() != y_size || r.scalar_type() != at::kByte || is_channels_last(r) != channels_last)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: residual must be a uint8 map with the output's shape and layout", op);
    if (channels_last && (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15u))
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: residual must start on a 16-byte boundary", op);
}

// Geometry of a convolution the way the reference resolves it (runtime/chainerx_util.cc:180-200,276-311).
void pair_of(PyObject* seq, int64_t* v, int* n, int64_t fill) {
    PyObject* f = PySequence_Fast(seq, "strides and pads must be sequences");
    if (!f) throw PyErrSet{};
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(f);
    v[0] = v[1] = fill;
    try {
        for (Py_ssize_t i = 0; i < len && i < 2; ++i) v[i] = as_long(PySequence_Fast_GET_ITEM(f, i));
    } catch (...) {
        Py_DECREF(f);
        throw;
    }
    Py_DECREF(f);
    *n = (int)len;
}

chxq_conv_geom geometry(const at::Tensor& x, const at::Tensor& w, PyObject* strides, PyObject* pads, PyObject* group, PyObject* auto_pad) {
    const int xc = qcode(x, "x"), wc = qcode(w, "w");
    if (x.dim() != 4 || w.dim() != 4) fail(CHXQ_ERR_UNSUPPORTED, "convolutions over 2 spatial dimensions only");
    int64_t s[2], p[2];
    int ns, np;
    pair_of(strides, s, &ns, 1);
    pair_of(pads, p, &np, 0);
    const char* ap = "";
    if (auto_pad != Py_None) {
        ap = PyUnicode_AsUTF8(auto_pad);
        if (!ap) throw PyErrSet{};
    }
    chxq_conv_geom g;
    const int rc = chxq_conv_resolve_geometry((int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), (int)w.size(0), (int)w.size(1), (int)w.size(2),
                                              (int)w.size(3), s, ns, p, np, (int)as_long(group), ap, &g);
    if (rc != CHXQ_OK) throw OpError{rc, chxq_last_error()};
    g.x_dtype = xc;
    g.w_dtype = wc;
    return g;
}

// Layouts: channels-last maps use the NHWC kernels.
void conv_io(at::Tensor* x, chxq_conv_geom* g, at::ScalarType dtype, at::Tensor* y) {
    const bool cl = is_channels_last(*x);
    if (!cl) *x = x->contiguous();
    g->x_layout = g->y_layout = cl ? CHXQ_NHWC : CHXQ_NCHW;
    *y = empty_map({g->N, g->M, g->Ho, g->Wo}, dtype, *x, cl);
}

// The fields of a PackedConv.
struct Packed {
    at::Tensor w, blob;
    chxq_conv_geom g;
    int flags;
};

PyObject *s_w, *s_blob, *s_g, *s_flags;

Packed packed_of(PyObject* o) {
    Packed k;
    auto get = [&](PyObject* name) {
        PyObject* v = PyObject_GetAttr(o, name);
        if (!v) throw PyErrSet{};
        return v;
    };
    PyObject* v = get(s_w);
    if (is_tensor(v)) k.w = THPVariable_Unpack(v);
    Py_DECREF(v);
    v = get(s_blob);
    if (is_tensor(v)) k.blob = THPVariable_Unpack(v);
    Py_DECREF(v);
    v = get(s_flags);
    k.flags = (int)PyLong_AsLong(v);
    Py_DECREF(v);
    v = get(s_g);
    Py_buffer view;
    if (PyObject_GetBuffer(v, &view, PyBUF_SIMPLE) != 0) {
        Py_DECREF(v);
        throw PyErrSet{};
    }
    const bool ok = view.len == (Py_ssize_t)sizeof(chxq_conv_geom);
    if (ok) memcpy(&k.g, view.buf, sizeof(k.g));
    PyBuffer_Release(&view);
    Py_DECREF(v);
    if (!ok || !k.w.defined()) {
        PyErr_SetString(PyExc_TypeError, "expected a PackedConv");
        throw PyErrSet{};
    }
    return k;
}

inline bool eligible(const Packed& k) {
    return (k.flags & 1) != 0;
}

bool matches_geometry(const at::Tensor& x, const chxq_conv_geom& g) {
    return x.dim() == 4 && x.size(0) == g.N && x.size(1) == g.C && x.size(2) == g.H && x.size(3) == g.W &&
           (g.x_layout == CHXQ_NHWC ? is_channels_last(x) : x.is_contiguous());
}

// `out` as given, or a fresh channels-last map.
at::Tensor output_map(const char* op, PyObject* out, at::IntArrayRef size, at::ScalarType dtype, const at::Tensor& like) {
    if (out == Py_None) return empty_map(size, dtype, like, true);
    const at::Tensor& y = tensor(out, "out");
    if (y.sizes() != size || !is_channels_last(y) || y.scalar_type() != dtype)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: out must be a channels_last map of the output's shape and dtype", op);
    return y;
}

// ---- ops ------------------------------------------------------------------------------------------------------------------

typedef PyObject* const* Args;

// x, y_scale, y_zero_point, round_mode
PyObject* quantize_linear(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("QuantizeLinear", n, 4);
    const at::Tensor& x0 = tensor(a[0], "QuantizeLinear: x");
    require_cuda(x0);
    if (x0.scalar_type() != at::kFloat) fail(CHXQ_ERR_INVALID_ARGUMENT, "QuantizeLinear: x must be float32, got %s", dtype_name(x0).c_str());
    const int mode = (int)as_long(a[3]);
    if (is_device_scalar(a[1])) {
        const at::Tensor& scale = THPVariable_Unpack(a[1]);
        if (scale.scalar_type() != at::kFloat) fail(CHXQ_ERR_INVALID_ARGUMENT, "QuantizeLinear: a device y_scale must be float32");
        at::Tensor zp;
        int code = CHXQ_UINT8;
        if (a[2] != Py_None && !is_device_scalar(a[2])) {
            const Zp z = zp_scalar(a[2]);
            code = z.code;
            zp = at::full({1}, z.value, at::TensorOptions().dtype(qtype(z.code)).device(x0.device()));
        } else if (a[2] != Py_None) {
            zp = THPVariable_Unpack(a[2]);
            code = qcode(zp, "QuantizeLinear: y_zero_point");
        }
        const at::Tensor x = dense(x0);
        at::Tensor y = empty_like_as(x, qtype(code));
        call([&] {
            return chxq_quantize_linear_dev(static_cast<const float*>(x.data_ptr()), x.numel(), static_cast<const float*>(scale.data_ptr()),
                                            zp.defined() ? zp.data_ptr() : nullptr, code, mode, y.data_ptr(), stream());
        });
        return wrap(std::move(y));
    }
    const Zp z = zp_scalar(a[2]);
    const float scale = (float)as_double(a[1]);
    const at::Tensor x = dense(x0);
    at::Tensor y = empty_like_as(x, qtype(z.code));
    call([&] { return chxq_quantize_linear(static_cast<const float*>(x.data_ptr()), x.numel(), scale, z.value, z.code, mode, y.data_ptr(), stream()); });
    return wrap(std::move(y));
    OP_END
}

// x, x_scale, x_zero_point
PyObject* dequantize_linear(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("DequantizeLinear", n, 3);
    const at::Tensor& x0 = tensor(a[0], "DequantizeLinear: x");
    require_cuda(x0);
    const int code = qcode(x0, "DequantizeLinear: x");
    const Zp z = zp_scalar(a[2]);
    const float scale = (float)as_double(a[1]);
    const at::Tensor x = dense(x0);
    at::Tensor y = empty_like_as(x, at::kFloat);
    call([&] { return chxq_dequantize_linear(x.data_ptr(), code, x.numel(), scale, z.value, static_cast<float*>(y.data_ptr()), stream()); });
    return wrap(std::move(y));
    OP_END
}

// a, b, a_zero_point, b_zero_point, path
PyObject* matmul_integer(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("MatMulInteger", n, 5);
    at::Tensor l = tensor(a[0], "MatMulInteger: a"), r = tensor(a[1], "MatMulInteger: b");
    require_cuda(l);
    require_cuda(r);
    const int cl = qcode(l, "MatMulInteger: a"), cr = qcode(r, "MatMulInteger: b");
    if (l.dim() < 2 || r.dim() < 2) fail(CHXQ_ERR_INVALID_ARGUMENT, "MatMulInteger: operands need at least two dimensions");
    const int64_t d = l.dim(), dr = r.dim();
    if (d > 2 && l.sizes().slice(0, d - 2) != r.sizes().slice(0, dr - 2))
        fail(CHXQ_ERR_UNSUPPORTED, "MatMulInteger: batched operands need equal leading dimensions");
    if (d != dr) fail(CHXQ_ERR_UNSUPPORTED, "MatMulInteger: operands need the same number of dimensions");
    const int64_t M = l.size(d - 2), K = l.size(d - 1), K2 = r.size(d - 2), N = r.size(d - 1);
    if (K != K2) fail(CHXQ_ERR_INVALID_ARGUMENT, "MatMulInteger: inner dimensions differ (%lld vs %lld)", (long long)K, (long long)K2);
    int64_t batch = 1;
    c10::SmallVector<int64_t, 5> size;
    for (int64_t i = 0; i < d - 2; ++i) {
        batch *= l.size(i);
        size.push_back(l.size(i));
    }
    size.push_back(M);
    size.push_back(N);
    l = l.contiguous();
    r = r.contiguous();
    const ZpArray za = zp_array(a[2], l, "a_zero_point"), zb = zp_array(a[3], r, "b_zero_point");
    const int path = (int)as_long(a[4]);
    at::Tensor y = empty_map(size, at::kInt, l, false);
    const size_t ws_bytes = path != CHXQ_PATH_SIMT ? chxq_matmul_integer_workspace(batch, M, N, K) : 0;
    OwnScratch own;
    void* ws = K % 16 != 0 ? own.get_if_room(ws_bytes) : own.get(ws_bytes);
    call([&] {
        return chxq_matmul_integer(l.data_ptr(), cl, r.data_ptr(), cr, batch, M, N, K, za.ptr, za.len, zb.ptr, zb.len, static_cast<int32_t*>(y.data_ptr()), ws,
                                   ws_bytes, path, stream());
    });
    return wrap(std::move(y));
    OP_END
}

// a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point, round_mode, path
PyObject* qlinear_matmul(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("QLinearMatMul", n, 10);
    at::Tensor l = tensor(a[0], "QLinearMatMul: a"), r = tensor(a[3], "QLinearMatMul: b");
    require_cuda(l);
    require_cuda(r);
    const int cl = qcode(l, "QLinearMatMul: a"), cr = qcode(r, "QLinearMatMul: b");
    if (l.dim() != 2 || r.dim() != 2 || l.size(1) != r.size(0)) fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearMatMul: expected [M,K] x [K,N]");
    const int64_t M = l.size(0), K = l.size(1), N = r.size(1);
    const Zp za = zp_scalar(a[2]), zb = zp_scalar(a[5]), zy = zp_scalar(a[7]);
    l = l.contiguous();
    r = r.contiguous();
    const float sa = (float)as_double(a[1]), sb = (float)as_double(a[4]), sy = (float)as_double(a[6]);
    const int mode = (int)as_long(a[8]), path = (int)as_long(a[9]);
    at::Tensor y = empty_map({M, N}, qtype(zy.code), l, false);
    const size_t ws_bytes = path != CHXQ_PATH_SIMT ? chxq_matmul_integer_workspace(1, M, N, K) : 0;
    OwnScratch own;
    void* ws = K % 16 != 0 ? own.get_if_room(ws_bytes) : own.get(ws_bytes);
    call([&] {
        return chxq_qlinear_matmul(l.data_ptr(), cl, sa, za.value, r.data_ptr(), cr, sb, zb.value, sy, zy.value, zy.code, M, N, K, mode, y.data_ptr(), ws,
                                   ws_bytes, path, stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, w, x_zero_point, w_zero_point, strides, pads, group, auto_pad, path
PyObject* conv_integer(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("ConvInteger", n, 9);
    at::Tensor x = tensor(a[0], "ConvInteger: x"), w = tensor(a[1], "ConvInteger: w");
    require_cuda(x);
    require_cuda(w);
    chxq_conv_geom g = geometry(x, w, a[4], a[5], a[6], a[7]);
    at::Tensor y;
    conv_io(&x, &g, at::kInt, &y);
    w = w.contiguous();
    int32_t* yp = static_cast<int32_t*>(y.data_ptr());
    if (is_device_scalar(a[2])) {
        const at::Tensor& zx = THPVariable_Unpack(a[2]);
        if (zx.scalar_type() != x.scalar_type()) fail(CHXQ_ERR_INVALID_ARGUMENT, "ConvInteger: a device x_zero_point must have x's dtype");
        const ZpArray zw = zp_array(a[3], w, "w_zero_point");
        OwnScratch own;
        const size_t ws_bytes = (int)as_long(a[8]) != CHXQ_PATH_SIMT ? chxq_conv_dev_workspace(&g) : 0;
        void* ws = own.get_if_room(ws_bytes);
        call([&] { return chxq_conv_integer_dev_ws(x.data_ptr(), w.data_ptr(), &g, zx.data_ptr(), zw.ptr, zw.len, yp, ws, ws_bytes, stream()); });
        return wrap(std::move(y));
    }
    const Zp zx = zp_scalar(a[2]);
    const ZpArray zw = zp_array(a[3], w, "w_zero_point");
    const int path = (int)as_long(a[8]);
    const size_t ws_bytes = path != CHXQ_PATH_SIMT ? chxq_conv_workspace(&g) : 0;
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] {
        return chxq_conv_integer(x.data_ptr(), w.data_ptr(), &g, a[2] != Py_None, zx.value, zw.ptr, zw.len, yp, ws, ws_bytes, path, stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, w, strides, pads, group, auto_pad, path, then the sixteen of conv_params
PyObject* qlinear_conv(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("QLinearConv", n, 7 + kConvArgs);
    at::Tensor x = tensor(a[0], "QLinearConv: x"), w = tensor(a[1], "QLinearConv: w");
    require_cuda(x);
    require_cuda(w);
    chxq_conv_geom g = geometry(x, w, a[2], a[3], a[4], a[5]);
    Args c = a + 7;
    ConvParams p;
    conv_params(c, x, w, false, &p);
    at::Tensor y;
    conv_io(&x, &g, qtype(p.y_code), &y);
    if (c[9] != Py_None) {
        const at::Tensor& r = THPVariable_Unpack(c[9]);
        if (r.sizes() != y.sizes() || r.scalar_type() != at::kByte || is_channels_last(r) != (g.y_layout == CHXQ_NHWC))
            fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConv: residual must be a uint8 map with the output's shape and layout");
    }
    w = w.contiguous();
    const int path = (int)as_long(a[6]);
    const size_t ws_bytes = path != CHXQ_PATH_SIMT ? chxq_conv_workspace(&g) : 0;
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] { return chxq_qlinear_conv(x.data_ptr(), w.data_ptr(), &g, &p.p, y.data_ptr(), ws, ws_bytes, path, stream()); });
    return wrap(std::move(y));
    OP_END
}

// x, packed, out, then the sixteen of conv_params
PyObject* qlinear_conv_packed(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("QLinearConvPacked", n, 3 + kConvArgs);
    const at::Tensor& x = tensor(a[0], "QLinearConvPacked: x");
    require_cuda(x);
    const Packed k = packed_of(a[1]);
    const chxq_conv_geom& g = k.g;
    if (!matches_geometry(x, g)) fail(CHXQ_ERR_INVALID_ARGUMENT, "QLinearConvPacked: x does not match the packed geometry / layout");
    Args c = a + 3;
    const int64_t size[4] = {g.N, g.M, g.Ho, g.Wo};
    check_residual("QLinearConvPacked", c[9], size, true);
    ConvParams p;
    conv_params(c, x, k.w, true, &p);
    at::Tensor y = output_map("QLinearConvPacked", a[2], size, qtype(p.y_code), x);
    if (!eligible(k)) fail(CHXQ_ERR_UNSUPPORTED, "QLinearConvPacked: this geometry is not eligible for the packed tensor-core path");
    const size_t ws_bytes = chxq_conv_packed_workspace(&g, p.p.x_zero_point, k.flags);
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] { return chxq_qlinear_conv_packed(x.data_ptr(), k.blob.data_ptr(), &g, &p.p, k.flags, y.data_ptr(), ws, ws_bytes, stream()); });
    return wrap(std::move(y));
    OP_END
}

// x, packed1, packed2, out, then the sixteen of conv_params for the first and for the second convolution
PyObject* qlinear_conv_chain_packed(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    const char* op = "QLinearConvChainPacked";
    need_args(op, n, 4 + 2 * kConvArgs);
    const at::Tensor& x = tensor(a[0], "QLinearConvChainPacked: x");
    require_cuda(x);
    const Packed k1 = packed_of(a[1]), k2 = packed_of(a[2]);
    const chxq_conv_geom &g1 = k1.g, &g2 = k2.g;
    if (!(x.dim() == 4 && x.size(0) == g1.N && x.size(1) == g1.C && x.size(2) == g1.H && x.size(3) == g1.W && is_channels_last(x)))
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: x does not match the packed geometry / layout", op);
    if (!eligible(k1) || !eligible(k2)) fail(CHXQ_ERR_UNSUPPORTED, "%s: a geometry is not eligible for the packed tensor-core path", op);
    Args c1 = a + 4, c2 = c1 + kConvArgs;
    if (c1[9] != Py_None) fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: only the second convolution may carry a residual tail", op);
    const int64_t size[4] = {g2.N, g2.M, g2.Ho, g2.Wo};
    check_residual(op, c2[9], size, true);
    ConvParams p1, p2;
    conv_params(c1, x, k1.w, true, &p1);
    conv_params(c2, x, k2.w, true, &p2);
    if (p1.y_code != CHXQ_UINT8 || p2.y_code != CHXQ_UINT8) fail(CHXQ_ERR_UNSUPPORTED, "%s: both outputs must be uint8", op);
    at::Tensor y = output_map(op, a[3], size, at::kByte, x);
    call([&] {
        return chxq_qlinear_conv_chain_packed(x.data_ptr(), k1.blob.data_ptr(), &g1, &p1.p, k1.flags, k2.blob.data_ptr(), &g2, &p2.p, k2.flags, y.data_ptr(),
                                              stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, packed, pool_kernel, pool_stride, pool_pad, cover_all, quant_round_mode, out, then the sixteen of conv_params
PyObject* qlinear_conv_maxpool_packed(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    const char* op = "QLinearConvMaxPoolPacked";
    need_args(op, n, 8 + kConvArgs);
    const at::Tensor& x = tensor(a[0], "QLinearConvMaxPoolPacked: x");
    require_cuda(x);
    const Packed k = packed_of(a[1]);
    const chxq_conv_geom& g = k.g;
    const bool f32 = x.scalar_type() == at::kFloat;
    if (!matches_geometry(x, g) || !(f32 || x.scalar_type() == at::kByte))
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: x does not match the packed geometry / layout", op);
    if (!eligible(k)) fail(CHXQ_ERR_UNSUPPORTED, "%s: this geometry is not eligible for the packed tensor-core path", op);
    ConvParams p;
    conv_params(a + 8, x, k.w, true, &p);
    if (p.y_code != CHXQ_UINT8) fail(CHXQ_ERR_UNSUPPORTED, "%s: the output must be uint8", op);
    const long kernel = as_long(a[2]), stride = as_long(a[3]), pad = as_long(a[4]);
    const bool cover_all = as_bool(a[5]);
    const int mode = (int)as_long(a[6]);
    auto pooled = [&](int extent) {  // floor division, as the quotient of a window larger than the map is negative
        const long v = extent + 2 * pad - kernel + (cover_all ? stride - 1 : 0);
        return (v >= 0 ? v / stride : -((-v + stride - 1) / stride)) + 1;
    };
    if (stride < 1) fail(CHXQ_ERR_UNSUPPORTED, "%s: bad pooling stride", op);
    at::Tensor y = a[7] != Py_None ? tensor(a[7], "out") : empty_map({g.N, g.M, pooled(g.Ho), pooled(g.Wo)}, at::kByte, x, true);
    const size_t ws_bytes = chxq_conv_packed_workspace(&g, p.p.x_zero_point, k.flags);
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] {
        return chxq_qlinear_conv_maxpool_packed(x.data_ptr(), f32, mode, k.blob.data_ptr(), &g, &p.p, k.flags, (int)kernel, (int)stride, (int)pad, cover_all,
                                                y.data_ptr(), ws, ws_bytes, stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, packed, quant_round_mode, out, then the sixteen of conv_params
PyObject* quantize_qlinear_conv_packed(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    const char* op = "QuantizeLinearConvPacked";
    need_args(op, n, 4 + kConvArgs);
    const at::Tensor& x = tensor(a[0], "QuantizeLinearConvPacked: x");
    require_cuda(x);
    const Packed k = packed_of(a[1]);
    const chxq_conv_geom& g = k.g;
    if (!matches_geometry(x, g) || x.scalar_type() != at::kFloat)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: x must be the fp32 tensor of the packed geometry / layout", op);
    ConvParams p;
    conv_params(a + 4, x, k.w, true, &p);
    const int mode = (int)as_long(a[2]);
    at::Tensor y = a[3] != Py_None ? tensor(a[3], "out") : empty_map({g.N, g.M, g.Ho, g.Wo}, qtype(p.y_code), x, true);
    if (!eligible(k)) fail(CHXQ_ERR_UNSUPPORTED, "%s: this geometry is not eligible for the packed tensor-core path", op);
    const size_t ws_bytes = chxq_conv_packed_workspace(&g, p.p.x_zero_point, k.flags);
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] {
        return chxq_quantize_qlinear_conv_packed(static_cast<const float*>(x.data_ptr()), mode, k.blob.data_ptr(), &g, &p.p, k.flags, y.data_ptr(), ws, ws_bytes,
                                                 stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, packed, x_zero_point
PyObject* conv_integer_packed(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("ConvIntegerPacked", n, 3);
    const at::Tensor& x = tensor(a[0], "ConvIntegerPacked: x");
    require_cuda(x);
    const Packed k = packed_of(a[1]);
    const chxq_conv_geom& g = k.g;
    if (!matches_geometry(x, g)) fail(CHXQ_ERR_INVALID_ARGUMENT, "ConvIntegerPacked: x does not match the packed geometry / layout");
    if (!eligible(k)) fail(CHXQ_ERR_UNSUPPORTED, "ConvIntegerPacked: this geometry is not eligible for the packed tensor-core path");
    const Zp zx = zp_scalar(a[2]);
    at::Tensor y = empty_map({g.N, g.M, g.Ho, g.Wo}, at::kInt, x, true);
    const size_t ws_bytes = chxq_conv_packed_workspace(&g, zx.value, k.flags);
    OwnScratch own;
    void* ws = own.get(ws_bytes);
    call([&] {
        return chxq_conv_integer_packed(x.data_ptr(), k.blob.data_ptr(), &g, a[2] != Py_None, zx.value, k.flags, static_cast<int32_t*>(y.data_ptr()), ws, ws_bytes,
                                        stream());
    });
    return wrap(std::move(y));
    OP_END
}

// inputs, num_outputs, code, fusion_id
PyObject* elementwise(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    const char* op = "ElementWiseNvrtc";
    need_args(op, n, 4);
    PyObject* seq = PySequence_Fast(a[0], "ElementWiseNvrtc: inputs must be a sequence of tensors");
    if (!seq) throw PyErrSet{};
    std::vector<at::Tensor> ins;
    try {
        for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(seq); ++i) ins.push_back(tensor(PySequence_Fast_GET_ITEM(seq, i), "ElementWiseNvrtc: input"));
    } catch (...) {
        Py_DECREF(seq);
        throw;
    }
    Py_DECREF(seq);
    if (ins.empty()) fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: no inputs", op);
    for (const at::Tensor& t : ins) require_cuda(t);
    const at::ScalarType dtype = ins[0].scalar_type();
    if (dtype != at::kHalf && dtype != at::kFloat && dtype != at::kDouble)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: dtype %s is not a float type", op, dtype_name(ins[0]).c_str());
    bool same = true;
    for (const at::Tensor& t : ins) {
        if (t.scalar_type() != dtype) fail(CHXQ_ERR_INVALID_ARGUMENT, "%s: all inputs must share one dtype", op);  // runtime/ops/nvrtc.cc:102
        same = same && t.sizes() == ins[0].sizes();
    }
    if (!same) {
        const std::vector<at::Tensor> full = at::broadcast_tensors(ins);
        ins.assign(full.begin(), full.end());
    }
    for (at::Tensor& t : ins) t = t.contiguous();
    const long n_out = as_long(a[1]);
    const char* code = PyUnicode_Check(a[2]) ? PyUnicode_AsUTF8(a[2]) : PyBytes_AsString(a[2]);
    if (!code) throw PyErrSet{};
    const int id = (int)as_long(a[3]);
    std::vector<const void*> in_ptrs;
    std::vector<void*> out_ptrs;
    std::vector<at::Tensor> outs;
    for (const at::Tensor& t : ins) in_ptrs.push_back(t.data_ptr());
    for (long i = 0; i < n_out; ++i) {
        outs.push_back(empty_map(ins[0].sizes(), dtype, ins[0], false));
        out_ptrs.push_back(outs.back().data_ptr());
    }
    const int dcode = dtype == at::kHalf ? CHXQ_FLOAT16 : (dtype == at::kFloat ? CHXQ_FLOAT32 : CHXQ_FLOAT64);
    call([&] {
        return chxq_eltwise_run(code, id, in_ptrs.data(), (int)in_ptrs.size(), out_ptrs.data(), (int)out_ptrs.size(), ins[0].numel(), dcode, stream());
    });
    PyObject* list = PyList_New((Py_ssize_t)outs.size());
    if (!list) throw PyErrSet{};
    for (size_t i = 0; i < outs.size(); ++i) {
        PyObject* o = wrap(std::move(outs[i]));
        if (!o) {
            Py_DECREF(list);
            throw PyErrSet{};
        }
        PyList_SET_ITEM(list, (Py_ssize_t)i, o);
    }
    return list;
    OP_END
}

// x, kernel, stride, pad, cover_all
PyObject* maxpool_u8(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("MaxPoolU8", n, 5);
    const at::Tensor& x = tensor(a[0], "MaxPoolU8: x");
    require_cuda(x);
    if (x.scalar_type() != at::kByte || !is_channels_last(x)) fail(CHXQ_ERR_INVALID_ARGUMENT, "MaxPoolU8: expected a uint8 channels_last map");
    const long kernel = as_long(a[1]), stride = as_long(a[2]), pad = as_long(a[3]);
    const bool cover_all = as_bool(a[4]);
    if (stride < 1) fail(CHXQ_ERR_INVALID_ARGUMENT, "MaxPool: bad geometry");
    auto pooled = [&](int64_t extent) {
        const int64_t v = extent + 2 * pad - kernel + (cover_all ? stride - 1 : 0);
        return (v >= 0 ? v / stride : -((-v + stride - 1) / stride)) + 1;
    };
    const int64_t Ho = pooled(x.size(2)), Wo = pooled(x.size(3));
    at::Tensor y = empty_map({x.size(0), x.size(1), Ho, Wo}, at::kByte, x, true);
    call([&] {
        return chxq_maxpool_u8_nhwc(static_cast<const uint8_t*>(x.data_ptr()), (int)x.size(0), (int)x.size(2), (int)x.size(3), (int)x.size(1), (int)kernel,
                                    (int)stride, (int)pad, (int)Ho, (int)Wo, static_cast<uint8_t*>(y.data_ptr()), stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, x_scale, x_zero_point
PyObject* global_avgpool_dq(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("GlobalAveragePoolDequant", n, 3);
    const at::Tensor& x = tensor(a[0], "GlobalAveragePoolDequant: x");
    require_cuda(x);
    if (x.scalar_type() != at::kByte || !is_channels_last(x))
        fail(CHXQ_ERR_INVALID_ARGUMENT, "GlobalAveragePoolDequant: expected a uint8 channels_last map");
    const float scale = (float)as_double(a[1]);
    const int zp = (int)as_long(a[2]);
    at::Tensor y = empty_map({x.size(0), x.size(1)}, at::kFloat, x, false);
    call([&] {
        return chxq_global_avgpool_dq_nhwc(static_cast<const uint8_t*>(x.data_ptr()), (int)x.size(0), (int)(x.size(2) * x.size(3)), (int)x.size(1), scale, zp,
                                           static_cast<float*>(y.data_ptr()), stream());
    });
    return wrap(std::move(y));
    OP_END
}

// x, w, b
PyObject* linear(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("Linear", n, 3);
    at::Tensor x = tensor(a[0], "Linear: x"), w = tensor(a[1], "Linear: w"), b;
    require_cuda(x);
    require_cuda(w);
    if (a[2] != Py_None) {
        b = tensor(a[2], "Linear: b");
        require_cuda(b);
        b = b.contiguous();
    }
    x = x.contiguous();
    w = w.contiguous();
    at::Tensor y = empty_map({x.size(0), w.size(0)}, at::kFloat, x, false);
    call([&] {
        return chxq_linear_f32(static_cast<const float*>(x.data_ptr()), static_cast<const float*>(w.data_ptr()),
                               b.defined() ? static_cast<const float*>(b.data_ptr()) : nullptr, (int)x.size(0), (int)x.size(1), (int)w.size(0),
                               static_cast<float*>(y.data_ptr()), stream());
    });
    return wrap(std::move(y));
    OP_END
}

// a, a_scale, a_zero_point, b, b_scale, b_zero_point, y_scale, y_zero_point, relu, round_mode
PyObject* qadd_u8(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("QAddU8", n, 10);
    const at::Tensor &l = tensor(a[0], "QAddU8: a"), &r = tensor(a[3], "QAddU8: b");
    require_cuda(l);
    require_cuda(r);
    if (l.sizes() != r.sizes() || l.scalar_type() != at::kByte || r.scalar_type() != at::kByte || l.strides() != r.strides())
        fail(CHXQ_ERR_INVALID_ARGUMENT, "QAddU8: operands must be uint8 maps of equal shape and layout");
    const float sa = (float)as_double(a[1]), sb = (float)as_double(a[4]), sy = (float)as_double(a[6]);
    const int za = (int)as_long(a[2]), zb = (int)as_long(a[5]), zy = (int)as_long(a[7]), mode = (int)as_long(a[9]);
    const bool relu = as_bool(a[8]);
    at::Tensor y = at::empty_like(l);
    call([&] {
        return chxq_qadd_u8(static_cast<const uint8_t*>(l.data_ptr()), sa, za, static_cast<const uint8_t*>(r.data_ptr()), sb, zb, l.numel(), sy, zy, relu, mode,
                            static_cast<uint8_t*>(y.data_ptr()), stream());
    });
    return wrap(std::move(y));
    OP_END
}

// rmin, rmax
PyObject* dynamic_params_u8(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("DynamicQuantParamsU8", n, 2);
    const at::Tensor &lo = tensor(a[0], "DynamicQuantParamsU8: rmin"), &hi = tensor(a[1], "DynamicQuantParamsU8: rmax");
    require_cuda(lo);
    require_cuda(hi);
    if (lo.scalar_type() != at::kFloat || hi.scalar_type() != at::kFloat || lo.numel() != 1 || hi.numel() != 1)
        fail(CHXQ_ERR_INVALID_ARGUMENT, "DynamicQuantParamsU8: rmin and rmax must be one-element float32 tensors");
    at::Tensor scale = empty_map({1}, at::kFloat, lo, false), zp = empty_map({1}, at::kByte, lo, false);
    call([&] {
        return chxq_dynamic_quant_params_u8(static_cast<const float*>(lo.data_ptr()), static_cast<const float*>(hi.data_ptr()),
                                            static_cast<float*>(scale.data_ptr()), static_cast<uint8_t*>(zp.data_ptr()), stream());
    });
    PyObject *s = wrap(std::move(scale)), *z = wrap(std::move(zp));
    if (!s || !z) {
        Py_XDECREF(s);
        Py_XDECREF(z);
        throw PyErrSet{};
    }
    PyObject* t = PyTuple_Pack(2, s, z);
    Py_DECREF(s);
    Py_DECREF(z);
    return t;
    OP_END
}

// x
PyObject* minmax(PyObject*, PyObject* o) {
    OP_BEGIN
    at::Tensor x = tensor(o, "MinMax: x");
    require_cuda(x);
    x = x.contiguous();
    at::Tensor y = empty_map({2}, at::kFloat, x, false);
    call([&] { return chxq_minmax_f32(static_cast<const float*>(x.data_ptr()), x.numel(), static_cast<float*>(y.data_ptr()), stream()); });
    return wrap(std::move(y));
    OP_END
}

// x, to_nhwc: the layout copies behind ops.to_channels_last and ops.to_contiguous_nchw
PyObject* transpose_map(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("layout transform", n, 2);
    const at::Tensor& x = tensor(a[0], "layout transform: x");
    require_cuda(x);
    const bool to_nhwc = as_bool(a[1]);
    at::Tensor y = empty_map(x.sizes(), x.scalar_type(), x, to_nhwc);
    call([&] {
        auto* f = to_nhwc ? chxq_nchw_to_nhwc : chxq_nhwc_to_nchw;
        return f(x.data_ptr(), (int)x.element_size(), (int)x.size(0), (int)x.size(1), (int)x.size(2), (int)x.size(3), 0, y.data_ptr(), stream());
    });
    return wrap(std::move(y));
    OP_END
}

// ChxqError, ops._zp_scalar, ops._to_device_array, numpy.uint8, numpy.int8
PyObject* setup(PyObject*, Args a, Py_ssize_t n) {
    OP_BEGIN
    need_args("setup", n, 5);
    for (int i = 0; i < 5; ++i) Py_INCREF(a[i]);
    g_error_class = a[0];
    g_helpers[0] = a[1];
    g_helpers[1] = a[2];
    g_np_uint8 = reinterpret_cast<PyTypeObject*>(a[3]);
    g_np_int8 = reinterpret_cast<PyTypeObject*>(a[4]);
    Py_RETURN_NONE;
    OP_END
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FAST(quantize_linear), FAST(dequantize_linear), FAST(matmul_integer), FAST(qlinear_matmul), FAST(conv_integer), FAST(qlinear_conv),
                           FAST(qlinear_conv_packed), FAST(qlinear_conv_chain_packed), FAST(qlinear_conv_maxpool_packed), FAST(quantize_qlinear_conv_packed),
                           FAST(conv_integer_packed), FAST(elementwise), FAST(maxpool_u8), FAST(global_avgpool_dq), FAST(linear), FAST(qadd_u8),
                           FAST(dynamic_params_u8), {"minmax", minmax, METH_O, nullptr}, FAST(transpose_map), FAST(setup),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", "Host bodies of the VM ops over the C ABI of libchxq.so.", -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
    s_w = PyUnicode_InternFromString("w");
    s_blob = PyUnicode_InternFromString("blob");
    s_g = PyUnicode_InternFromString("g");
    s_flags = PyUnicode_InternFromString("flags");
    return PyModule_Create(&g_module);
}

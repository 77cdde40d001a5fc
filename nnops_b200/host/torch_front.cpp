// The calls of nnops_b200/ops.py in their usual form, from torch tensors to the C ABI without the
// interpreter in between.  Each function here is handed what the Python function of the same name was, and
// either makes the call and returns its output, or returns None with nothing of the caller's touched, and the
// Python code carries on: for whatever is not a plain dense CUDA tensor of the expected type on the current device
// (tensor subclasses, tensors of a transform, other devices, sequences to convert), for options that
// only tests and measurements use, and for every mistake, which is thus reported where it always was.
//
// Why: marshalling an int8 call in Python took 16 us (argument checks, fifty fields, two allocations, a
// stream look-up), more than the device needs for most layers at decode sizes; this takes about 6.
//
// The functions of libnnb200 come as addresses from the library capi.py has loaded (bind()).
#include <Python.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ops/empty.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAFunctions.h>

#include <cmath>
#include <cstring>
#include <limits>

#include "../../include/nnb200.h"

namespace {

using Size = size_t (*)(const void*);
using Run = int (*)(const void*, void*);

struct Library {
    Size gemm_bytes = nullptr;
    Run gemm = nullptr;
    Size q4_bytes = nullptr;
    Run q4 = nullptr;
    Run quantize = nullptr;
    Run dequantize = nullptr;
    Size conv_bytes = nullptr;
    Run conv = nullptr;
} g_lib;

PyObject* g_error = nullptr;   // capi.check: raises for a status that is not ok

enum Key {
    kBias, kRelu, kActivation, kActAlpha, kActBeta, kMinClip, kMaxClip, kScaleA, kScaleW, kZpA, kZpW, kOutScale, kOutZp,
    kWorkspace, kEngine, kRw, kMinWorkspace, kAlpha, kOverlap, kStride, kDilation, kPadding, kGroups, kScaleX, kZpX, kKeys
};
const char* const kKeyNames[kKeys] = {"bias", "relu", "activation", "act_alpha", "act_beta", "min_clip", "max_clip", "scale_a",
                                      "scale_w", "zp_a", "zp_w", "out_scale", "out_zp", "workspace", "engine", "r_w",
                                      "min_workspace", "alpha", "overlap_previous", "stride", "dilation", "padding", "groups",
                                      "scale_x", "zp_x"};
PyObject* g_keys[kKeys];

const char* const kActivations[] = {"none", "relu", "gelu", "sigmoid", "tanh", "leaky_relu", "silu", "hard_swish", "elu", "relu6"};
const char* const kKinds[] = {"s32", "s8", "u8", "f32", "f16"};
const at::ScalarType kKindTypes[] = {at::kInt, at::kChar, at::kByte, at::kFloat, at::kHalf};

// Not a call for this file.
struct Elsewhere {};

[[noreturn]] void elsewhere() { throw Elsewhere{}; }

// The keyword arguments, sorted into their slots (borrowed references); null = not given.
struct Options {
    PyObject* at[kKeys] = {};

    Options(PyObject* dict, std::initializer_list<Key> known)
    {
        PyObject *name, *value;
        Py_ssize_t pos = 0;
        while (PyDict_Next(dict, &pos, &name, &value)) {
            int found = -1;
            for (Key k : known) {
                if (g_keys[k] == name) {
                    found = k;
                    break;
                }
            }
            if (found < 0) {
                elsewhere();   // unknown, or a name that is not the interned one
            }
            at[found] = value;
        }
    }
    PyObject* operator[](Key k) const { return at[k]; }
};

// A dense tensor with storage of its own on the current device, and exactly a torch.Tensor.
const at::Tensor& plain(PyObject* o, const c10::Device& dev)
{
    if (!THPVariable_CheckExact(o)) {
        elsewhere();
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.has_storage() || t.layout() != at::kStrided || t.device() != dev || t.is_neg() || t.is_conj()) {
        elsewhere();
    }
    return t;
}

c10::Device current_device(PyObject* first)
{
    if (!THPVariable_CheckExact(first)) {
        elsewhere();
    }
    const at::Tensor& t = THPVariable_Unpack(first);
    if (!t.is_cuda() || t.device().index() != c10::cuda::current_device()) {
        elsewhere();
    }
    return t.device();
}

double number(PyObject* o)
{
    if (PyFloat_CheckExact(o)) {
        return PyFloat_AS_DOUBLE(o);
    }
    if (!PyLong_CheckExact(o)) {
        elsewhere();
    }
    const double d = PyLong_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        elsewhere();
    }
    return d;
}

float real(PyObject* o, float otherwise) { return o == nullptr ? otherwise : static_cast<float>(number(o)); }

int64_t whole(PyObject* o)
{
    if (!PyLong_CheckExact(o)) {
        elsewhere();
    }
    int overflow = 0;
    const int64_t v = PyLong_AsLongLongAndOverflow(o, &overflow);
    if (overflow != 0) {
        elsewhere();
    }
    return v;
}

int32_t whole32(PyObject* o, int32_t otherwise)
{
    if (o == nullptr) {
        return otherwise;
    }
    const int64_t v = whole(o);
    if (v != static_cast<int32_t>(v)) {
        elsewhere();
    }
    return static_cast<int32_t>(v);
}

bool flag(PyObject* o, bool otherwise)
{
    if (o == nullptr) {
        return otherwise;
    }
    if (!PyBool_Check(o)) {
        elsewhere();
    }
    return o == Py_True;
}

template <size_t N>
int one_of(PyObject* o, const char* const (&names)[N], int otherwise)
{
    if (o == nullptr) {
        return otherwise;
    }
    if (!PyUnicode_CheckExact(o)) {
        elsewhere();
    }
    for (size_t i = 0; i < N; ++i) {
        if (PyUnicode_CompareWithASCIIString(o, names[i]) == 0) {
            return static_cast<int>(i);
        }
    }
    elsewhere();
}

// A quantization parameter: an array of `count` entries, or one number.
template <class T>
void parameter(PyObject* o, at::ScalarType type, const c10::Device& dev, int64_t count, const T*& array, T& single)
{
    array = nullptr;
    if (o == nullptr || o == Py_None) {
        return;
    }
    if (PyFloat_CheckExact(o) || PyLong_CheckExact(o)) {
        if constexpr (std::is_same_v<T, float>) {
            single = static_cast<float>(number(o));
        } else {
            single = whole32(o, 0);
        }
        return;
    }
    const at::Tensor& t = plain(o, dev);
    if (t.scalar_type() != type || !t.is_contiguous() || t.numel() != count) {
        elsewhere();
    }
    array = static_cast<const T*>(t.data_ptr());
}

const void* bias_of(PyObject* o, at::ScalarType type, const c10::Device& dev)
{
    if (o == nullptr || o == Py_None) {
        return nullptr;
    }
    const at::Tensor& t = plain(o, dev);
    if (t.scalar_type() != type || !t.is_contiguous()) {
        elsewhere();
    }
    return t.data_ptr();
}

at::Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const c10::Device& dev)
{
    return at::empty(sizes, at::TensorOptions().dtype(type).device(dev));
}

// Scratch for the call, if it has any use for some.  Memory that cannot be had is the Python code's business,
// which knows what the least is.
at::Tensor scratch(size_t bytes, const c10::Device& dev)
{
    try {
        return empty({static_cast<int64_t>(bytes)}, at::kByte, dev);
    } catch (const c10::OutOfMemoryError&) {
        elsewhere();
    }
}

void enqueue(Run run, const void* args, const c10::Device& dev, const char* what)
{
    void* stream = at::cuda::getCurrentCUDAStream(dev.index()).stream();
    int status;
    Py_BEGIN_ALLOW_THREADS
    status = run(args, stream);
    Py_END_ALLOW_THREADS
    if (status != NNB200_OK) {
        PyObject* r = PyObject_CallFunction(g_error, "is", status, what);
        Py_XDECREF(r);
        throw python_error();
    }
}

// What Python code sees of any function here.
template <class F>
PyObject* guarded(F&& f)
{
    try {
        return f();
    } catch (const Elsewhere&) {
        Py_RETURN_NONE;
    } catch (python_error& e) {
        e.restore();
        return nullptr;
    } catch (const c10::OutOfMemoryError&) {
        Py_RETURN_NONE;   // an output that does not fit: torch.empty says so
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

void expect(Py_ssize_t n, Py_ssize_t want)
{
    if (n != want) {
        elsewhere();
    }
}

at::Tensor run_gemm_i8(const at::Tensor& a, const at::Tensor& w, at::Tensor out, int kind, const nnb200_gemm_i8_args& options,
                       const c10::Device& dev)
{
    nnb200_gemm_i8_args g = options;
    const int64_t ad = a.dim(), wd = w.dim();
    const int64_t ab = ad == 3 ? a.size(0) : 1, wb = wd == 3 ? w.size(0) : 1;
    const int64_t m = a.size(-2), k = a.size(-1), n = w.size(-2);
    const bool made = !out.defined();
    if (made) {
        out = ad == 3 || wd == 3 ? empty({std::max(ab, wb), m, n}, kKindTypes[kind], dev) : empty({m, n}, kKindTypes[kind], dev);
    }
    const int64_t ob = out.dim() == 3 ? out.size(0) : 1;
    g.a = a.data_ptr();
    g.w = w.data_ptr();
    g.out = out.data_ptr();
    g.m = m;
    g.n = n;
    g.k = k;
    g.a_stride_m = a.stride(-2);
    g.a_stride_k = k > 1 ? a.stride(-1) : 1;
    g.w_stride_n = w.stride(-2);
    g.w_stride_k = k > 1 ? w.stride(-1) : 1;
    g.ldc = out.stride(-2);
    g.batch = std::max(ab, wb);
    g.a_batch_stride = ab > 1 ? a.stride(0) : 0;
    g.w_batch_stride = wb > 1 ? w.stride(0) : 0;
    g.out_batch_stride = ob > 1 ? out.stride(0) : 0;
    g.a_unsigned = a.scalar_type() == at::kByte ? 1 : 0;
    g.out_kind = kind;
    at::Tensor workspace;   // stream-ordered: may go when this returns
    if (const size_t need = g_lib.gemm_bytes(&g); need != 0) {
        workspace = scratch(need, dev);
        g.workspace = workspace.data_ptr();
        g.workspace_bytes = need;
    }
    enqueue(g_lib.gemm, &g, dev, "nnb200_gemm_i8");
    return out;
}

// Checks the operands' forms and fills in everything that does not depend on the output.
void gemm_operands(const at::Tensor& a, const at::Tensor& w)
{
    const int64_t ad = a.dim(), wd = w.dim();
    if (ad < 2 || ad > 3 || wd < 2 || wd > 3 || (a.scalar_type() != at::kChar && a.scalar_type() != at::kByte) ||
        w.scalar_type() != at::kChar || a.size(-1) != w.size(-1)) {
        elsewhere();
    }
    const int64_t ab = ad == 3 ? a.size(0) : 1, wb = wd == 3 ? w.size(0) : 1;
    if (ab != wb && ab != 1 && wb != 1) {
        elsewhere();
    }
}

void gemm_options(nnb200_gemm_i8_args& g, const Options& o, int kind, int64_t m, int64_t n, const c10::Device& dev)
{
    std::memset(&g, 0, sizeof(g));
    if ((o[kWorkspace] != nullptr && o[kWorkspace] != Py_None) || flag(o[kMinWorkspace], false)) {
        elsewhere();
    }
    static const char* const automatic[] = {"auto"};
    one_of(o[kEngine], automatic, 0);
    g.bias = bias_of(o[kBias], kind <= NNB200_OUT_U8 ? at::kInt : kKindTypes[kind], dev);
    g.relu = flag(o[kRelu], false) ? 1 : 0;
    g.activation = one_of(o[kActivation], kActivations, 0);
    g.act_alpha = real(o[kActAlpha], 0.0f);
    g.act_beta = real(o[kActBeta], 1.0f);
    g.min_clip = real(o[kMinClip], -std::numeric_limits<float>::infinity());
    g.max_clip = real(o[kMaxClip], std::numeric_limits<float>::infinity());
    g.scale_a_scalar = g.scale_w_scalar = 1.0f;
    parameter(o[kScaleA], at::kFloat, dev, m, g.scale_a, g.scale_a_scalar);
    parameter(o[kScaleW], at::kFloat, dev, n, g.scale_w, g.scale_w_scalar);
    parameter(o[kZpA], at::kInt, dev, m, g.zp_a, g.zp_a_scalar);
    parameter(o[kZpW], at::kInt, dev, n, g.zp_w, g.zp_w_scalar);
    g.zp_a_nonzero = g.zp_a != nullptr ? NNB200_ZP_NOT_KNOWN : 0;
    g.zp_w_nonzero = g.zp_w != nullptr ? NNB200_ZP_NOT_KNOWN : 0;
    g.out_scale = real(o[kOutScale], 1.0f);
    g.out_zp = whole32(o[kOutZp], 0);
    if (o[kRw] != nullptr && o[kRw] != Py_None) {
        g.r_w = static_cast<const int32_t*>(plain(o[kRw], dev).data_ptr());
    }
}

// gemm_i8(a, w, out_kind, out, kw)
PyObject* gemm_i8(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 5);
        const c10::Device dev = current_device(args[0]);
        const at::Tensor& a = plain(args[0], dev);
        const at::Tensor& w = plain(args[1], dev);
        const int kind = one_of(args[2], kKinds, 0);
        at::Tensor out;
        if (args[3] != Py_None) {
            out = plain(args[3], dev);
            if (out.dim() < 2 || out.dim() > 3) {
                elsewhere();
            }
        }
        gemm_operands(a, w);
        nnb200_gemm_i8_args g;
        gemm_options(g, Options(args[4], {kScaleA, kScaleW, kBias, kOutScale, kRelu, kOutZp, kActivation, kZpA, kZpW, kRw, kActAlpha,
                                          kActBeta, kMinClip, kMaxClip, kWorkspace, kEngine, kMinWorkspace}),
                     kind, a.size(-2), w.size(-2), dev);
        return THPVariable_Wrap(run_gemm_i8(a, w, std::move(out), kind, g, dev));
    });
}

at::ScalarType dtype_of(PyObject* o, at::ScalarType otherwise)
{
    if (o == Py_None) {
        return otherwise;
    }
    if (!THPDtype_Check(o)) {
        elsewhere();
    }
    return reinterpret_cast<THPDtype*>(o)->scalar_type;
}

// linear_q4_1(a, w_blocks | (qs, n, qs_pitch, dm, dm_pitch), k, out_dtype, out, kw)
PyObject* linear_q4_1(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 6);
        const c10::Device dev = current_device(args[0]);
        const at::Tensor& a = plain(args[0], dev);
        if (a.dim() != 2 || a.stride(1) != 1 || (a.scalar_type() != at::kHalf && a.scalar_type() != at::kFloat)) {
            elsewhere();
        }
        nnb200_q4_1_args q;
        std::memset(&q, 0, sizeof(q));
        if (PyTuple_CheckExact(args[1])) {
            q.w_blocks = reinterpret_cast<const void*>(whole(PyTuple_GET_ITEM(args[1], 0)));
            q.n = whole(PyTuple_GET_ITEM(args[1], 1));
            q.ldw_blocks = whole(PyTuple_GET_ITEM(args[1], 2));
            q.w_dm = reinterpret_cast<const void*>(whole(PyTuple_GET_ITEM(args[1], 3)));
            q.ld_dm = whole(PyTuple_GET_ITEM(args[1], 4));
        } else {
            const at::Tensor& w = plain(args[1], dev);
            if (w.scalar_type() != at::kByte || w.dim() != 2 || w.stride(1) != 1 || w.stride(0) % 20 != 0) {
                elsewhere();
            }
            q.w_blocks = w.data_ptr();
            q.n = w.size(0);
            q.ldw_blocks = w.stride(0) / 20;
        }
        q.k = whole(args[2]);
        const at::ScalarType type = dtype_of(args[3], a.scalar_type());
        const Options o(args[5], {kActivation, kBias, kAlpha, kActAlpha, kActBeta, kMinClip, kMaxClip, kEngine, kOverlap});
        static const char* const automatic[] = {"auto"};
        one_of(o[kEngine], automatic, 0);
        at::Tensor out;
        if (args[4] != Py_None) {
            out = plain(args[4], dev);
            if (out.dim() != 2 || out.stride(1) != 1) {
                elsewhere();
            }
        }
        const at::ScalarType out_type = out.defined() ? out.scalar_type() : type;
        if (out_type != at::kHalf && out_type != at::kFloat) {
            elsewhere();
        }
        q.bias = bias_of(o[kBias], out_type, dev);
        q.activation = one_of(o[kActivation], kActivations, 0);
        q.act_alpha = real(o[kActAlpha], 0.0f);
        q.act_beta = real(o[kActBeta], 1.0f);
        q.min_clip = real(o[kMinClip], -std::numeric_limits<float>::infinity());
        q.max_clip = real(o[kMaxClip], std::numeric_limits<float>::infinity());
        q.alpha = real(o[kAlpha], 1.0f);
        q.flags = flag(o[kOverlap], false) ? NNB200_Q4_FLAG_OVERLAP_PREVIOUS : 0;
        if (!out.defined()) {
            out = empty({a.size(0), q.n}, type, dev);
        }
        q.a = a.data_ptr();
        q.out = out.data_ptr();
        q.m = a.size(0);
        q.lda = a.stride(0);
        q.ldc = out.stride(0);
        q.a_f16 = a.scalar_type() == at::kHalf ? 1 : 0;
        q.out_f16 = out_type == at::kHalf ? 1 : 0;
        at::Tensor workspace;
        if (const size_t need = g_lib.q4_bytes(&q); need != 0) {
            workspace = scratch(need, dev);
            q.workspace = workspace.data_ptr();
            q.workspace_bytes = need;
        }
        enqueue(g_lib.q4, &q, dev, "nnb200_linear_q4_1");
        return THPVariable_Wrap(std::move(out));
    });
}

// quantize_linear / dequantize_linear (x, scale, zero_point, axis, out_dtype, out)
PyObject* quant(PyObject* const* args, Py_ssize_t nargs, bool quantize)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 6);
        const c10::Device dev = current_device(args[0]);
        const at::Tensor& x = plain(args[0], dev);
        const at::Tensor& scale = plain(args[1], dev);
        const at::Tensor& zp = plain(args[2], dev);
        const int64_t axis = whole(args[3]);
        const at::ScalarType type = dtype_of(args[4], at::kChar);
        const auto floating = [](at::ScalarType t) { return t == at::kFloat || t == at::kHalf; };
        const auto byte = [](at::ScalarType t) { return t == at::kChar || t == at::kByte; };
        at::Tensor y;
        if (args[5] != Py_None) {
            y = plain(args[5], dev);
        }
        const at::ScalarType to = y.defined() ? y.scalar_type() : type;
        if (!x.is_contiguous() || (quantize ? !floating(x.scalar_type()) || !byte(to) : !byte(x.scalar_type()) || !floating(to)) ||
            scale.scalar_type() != at::kFloat || !byte(zp.scalar_type()) || !scale.is_contiguous() || !zp.is_contiguous() ||
            scale.numel() != zp.numel() || axis >= x.dim() || (axis < 0 && x.dim() == 0)) {
            elsewhere();
        }
        // [outer][rows][inner]: one parameter for all, one per innermost row, or one per index of the axis.
        nnb200_quant_linear_args q;
        std::memset(&q, 0, sizeof(q));
        q.outer = q.rows = 1;
        q.inner = x.numel();
        if (scale.numel() > 1) {
            if (axis < 0) {
                q.inner = x.size(-1);
                q.rows = q.inner != 0 ? x.numel() / q.inner : 0;
            } else {
                q.inner = 1;
                for (int64_t d = 0; d < x.dim(); ++d) {
                    (d < axis ? q.outer : d == axis ? q.rows : q.inner) *= x.size(d);
                }
            }
        }
        if (q.rows != scale.numel()) {
            elsewhere();
        }
        if (!y.defined()) {
            y = empty(x.sizes(), type, dev);
        }
        q.x = x.data_ptr();
        q.y = y.data_ptr();
        q.scale = static_cast<const float*>(scale.data_ptr());
        q.zero_point = zp.data_ptr();
        q.zp_unsigned = zp.scalar_type() == at::kByte ? NNB200_ZP_U8 : NNB200_ZP_S8;
        q.float_f16 = (quantize ? x : y).scalar_type() == at::kHalf ? 1 : 0;
        q.int_unsigned = (quantize ? y : x).scalar_type() == at::kByte ? 1 : 0;
        enqueue(quantize ? g_lib.quantize : g_lib.dequantize, &q, dev, quantize ? "nnb200_quantize_linear" : "nnb200_dequantize_linear");
        return THPVariable_Wrap(std::move(y));
    });
}

PyObject* quantize_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return quant(args, nargs, true); }
PyObject* dequantize_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) { return quant(args, nargs, false); }

// linear_fp_act(a, w, scale_a, zp_a, act_dtype, kw)
PyObject* linear_fp_act(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 6);
        const c10::Device dev = current_device(args[0]);
        const at::Tensor& a = plain(args[0], dev);
        const at::Tensor& w = plain(args[1], dev);
        const at::ScalarType act = dtype_of(args[4], at::kChar);
        const bool f16 = a.scalar_type() == at::kHalf;
        if (a.dim() != 2 || (!f16 && a.scalar_type() != at::kFloat) || !a.is_contiguous() || (act != at::kChar && act != at::kByte) ||
            w.scalar_type() != at::kChar || w.dim() != 2 || w.size(1) != a.size(1)) {
            elsewhere();
        }
        const int64_t m = a.size(0), k = a.size(1);
        // One scale and zero point for all rows, or an array of scales and one or many zero points.
        const bool one = !THPVariable_Check(args[2]);
        const float* scale = nullptr;
        const int32_t* zp = nullptr;
        float scale_value = 1.0f;
        int32_t zp_value = 0;
        parameter(args[2], at::kFloat, dev, m, scale, scale_value);
        parameter(args[3], at::kInt, dev, m, zp, zp_value);
        if (args[2] == Py_None || args[3] == Py_None || (one && zp != nullptr)) {
            elsewhere();
        }
        const Options o(args[5], {kScaleW, kBias, kActivation, kZpW, kRelu, kActAlpha, kActBeta, kMinClip, kMaxClip, kOutScale, kOutZp,
                                  kRw, kWorkspace, kEngine, kMinWorkspace});
        const int kind = f16 ? NNB200_OUT_F16 : NNB200_OUT_F32;
        nnb200_gemm_i8_args g;
        gemm_options(g, o, kind, m, w.size(0), dev);
        g.scale_a = scale;
        g.scale_a_scalar = scale_value;
        g.zp_a = zp;
        g.zp_a_scalar = zp_value;
        g.zp_a_nonzero = zp != nullptr ? NNB200_ZP_NOT_KNOWN : 0;

        const at::Tensor aq = empty({m, k}, act, dev);
        nnb200_quant_linear_args q;
        std::memset(&q, 0, sizeof(q));
        q.x = a.data_ptr();
        q.y = aq.data_ptr();
        q.outer = 1;
        q.rows = one ? 1 : m;
        q.inner = one ? m * k : k;
        q.scale = one ? &scale_value : scale;
        q.zero_point = zp != nullptr ? static_cast<const void*>(zp) : &zp_value;
        q.zp_unsigned = one ? NNB200_PARAMS_HOST : (zp != nullptr ? NNB200_ZP_S32 : NNB200_ZP_HOST);
        q.float_f16 = f16 ? 1 : 0;
        q.int_unsigned = act == at::kByte ? 1 : 0;
        enqueue(g_lib.quantize, &q, dev, "nnb200_quantize_linear");
        return THPVariable_Wrap(run_gemm_i8(aq, w, at::Tensor(), kind, g, dev));
    });
}

void pair_of(PyObject* o, int64_t (&v)[2])
{
    if (o == nullptr) {
        return;
    }
    if (!PyTuple_CheckExact(o) || PyTuple_GET_SIZE(o) != 2) {
        elsewhere();
    }
    v[0] = whole(PyTuple_GET_ITEM(o, 0));
    v[1] = whole(PyTuple_GET_ITEM(o, 1));
}

// conv2d_i8(x, packed blob, (kh, kw, icg, oc), out_kind, out, kw), zero points of the filter as one number
PyObject* conv2d_i8(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 6);
        const c10::Device dev = current_device(args[0]);
        const at::Tensor& x = plain(args[0], dev);
        const at::Tensor& w = plain(args[1], dev);
        if (x.dim() != 4 || (x.scalar_type() != at::kByte && x.scalar_type() != at::kChar) || !PyTuple_CheckExact(args[2]) ||
            PyTuple_GET_SIZE(args[2]) != 4) {
            elsewhere();
        }
        const int kind = one_of(args[3], kKinds, 0);
        const Options o(args[5], {kStride, kDilation, kPadding, kGroups, kBias, kScaleX, kZpX, kScaleW, kZpW, kOutScale, kOutZp, kRelu,
                                  kActivation, kActAlpha, kActBeta, kMinClip, kMaxClip, kWorkspace});
        if (o[kWorkspace] != nullptr && o[kWorkspace] != Py_None) {
            elsewhere();
        }
        nnb200_conv2d_i8_args c;
        std::memset(&c, 0, sizeof(c));
        int64_t stride[2] = {1, 1}, dil[2] = {1, 1}, pad[2] = {0, 0};
        pair_of(o[kStride], stride);
        pair_of(o[kDilation], dil);
        pair_of(o[kPadding], pad);
        if (stride[0] < 1 || stride[1] < 1) {
            elsewhere();
        }
        c.batch = x.size(0);
        c.ih = x.size(1);
        c.iw = x.size(2);
        c.ic = x.size(3);
        c.kh = whole(PyTuple_GET_ITEM(args[2], 0));
        c.kw = whole(PyTuple_GET_ITEM(args[2], 1));
        c.oc = whole(PyTuple_GET_ITEM(args[2], 3));
        const int64_t reach_h = c.ih + 2 * pad[0] - ((c.kh - 1) * dil[0] + 1), reach_w = c.iw + 2 * pad[1] - ((c.kw - 1) * dil[1] + 1);
        if (reach_h < 0 || reach_w < 0) {
            elsewhere();   // no output row: the division there rounds down
        }
        c.oh = reach_h / stride[0] + 1;
        c.ow = reach_w / stride[1] + 1;
        c.stride_h = stride[0];
        c.stride_w = stride[1];
        c.dil_h = dil[0];
        c.dil_w = dil[1];
        c.pad_h = pad[0];
        c.pad_w = pad[1];
        c.groups = o[kGroups] != nullptr ? whole(o[kGroups]) : 1;
        c.in_stride_n = x.stride(0);
        c.in_stride_h = x.stride(1);
        c.in_stride_w = x.stride(2);
        c.in_stride_c = x.stride(3);
        c.weight_packed = 1;
        c.a_unsigned = x.scalar_type() == at::kByte ? 1 : 0;
        c.out_kind = kind;
        c.bias = static_cast<const void*>(bias_of(o[kBias], kind == NNB200_OUT_S8 || kind == NNB200_OUT_U8 ? at::kInt : kKindTypes[kind], dev));
        c.relu = flag(o[kRelu], false) ? 1 : 0;
        c.activation = one_of(o[kActivation], kActivations, 0);
        c.act_alpha = real(o[kActAlpha], 0.0f);
        c.act_beta = real(o[kActBeta], 1.0f);
        c.min_clip = real(o[kMinClip], -std::numeric_limits<float>::infinity());
        c.max_clip = real(o[kMaxClip], std::numeric_limits<float>::infinity());
        c.scale_w_scalar = 1.0f;
        parameter(o[kScaleW], at::kFloat, dev, c.oc, c.scale_w, c.scale_w_scalar);
        c.scale_x = real(o[kScaleX], 1.0f);
        c.zp_x = whole32(o[kZpX], 0);
        c.zp_w_scalar = whole32(o[kZpW], 0);   // an array: the Python code looks whether it holds anything
        c.out_scale = real(o[kOutScale], 1.0f);
        c.out_zp = whole32(o[kOutZp], 0);
        at::Tensor out;
        if (args[4] != Py_None) {
            out = plain(args[4], dev);
            if (out.dim() != 4) {
                elsewhere();
            }
        } else {
            out = empty({c.batch, c.oh, c.ow, c.oc}, kKindTypes[kind], dev);
        }
        c.out_stride_n = out.stride(0);
        c.out_stride_h = out.stride(1);
        c.out_stride_w = out.stride(2);
        c.input = x.data_ptr();
        c.weight = w.data_ptr();
        c.out = out.data_ptr();
        at::Tensor workspace;
        if (const size_t need = g_lib.conv_bytes(&c); need != 0) {
            workspace = scratch(need, dev);
            c.workspace = workspace.data_ptr();
            c.workspace_bytes = need;
        }
        enqueue(g_lib.conv, &c, dev, "nnb200_conv2d_i8");
        return THPVariable_Wrap(std::move(out));
    });
}

// bind(addresses in the order of Library, check)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs)
{
    return guarded([&]() -> PyObject* {
        expect(nargs, 9);
        const auto address = [&](int i) { return reinterpret_cast<void*>(whole(args[i])); };
        g_lib.gemm_bytes = reinterpret_cast<Size>(address(0));
        g_lib.gemm = reinterpret_cast<Run>(address(1));
        g_lib.q4_bytes = reinterpret_cast<Size>(address(2));
        g_lib.q4 = reinterpret_cast<Run>(address(3));
        g_lib.quantize = reinterpret_cast<Run>(address(4));
        g_lib.dequantize = reinterpret_cast<Run>(address(5));
        g_lib.conv_bytes = reinterpret_cast<Size>(address(6));
        g_lib.conv = reinterpret_cast<Run>(address(7));
        Py_INCREF(args[8]);
        Py_XDECREF(g_error);
        g_error = args[8];
        Py_RETURN_TRUE;
    });
}

PyMethodDef g_methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"gemm_i8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(gemm_i8)), METH_FASTCALL, nullptr},
    {"linear_q4_1", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_q4_1)), METH_FASTCALL, nullptr},
    {"quantize_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(quantize_linear)), METH_FASTCALL, nullptr},
    {"dequantize_linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(dequantize_linear)), METH_FASTCALL, nullptr},
    {"linear_fp_act", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_fp_act)), METH_FASTCALL, nullptr},
    {"conv2d_i8", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(conv2d_i8)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "torch_front", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_torch_front()
{
    for (int i = 0; i < kKeys; ++i) {
        g_keys[i] = PyUnicode_InternFromString(kKeyNames[i]);
    }
    return PyModule_Create(&g_module);
}

// CPython binding of the per-call entry points of the C ABI (include/b200q.h): takes torch tensors and
// RowScaledView objects, fills the ABI's structs and calls the function, without an intermediate Python
// object. A quantize + GEMM pair launches in about 4.6 us of driver time; marshalling the same call through
// ctypes structures cost another 5.6 us (M=1, K=N=2048: 10.2 us per Linear.forward, 5.4 us through this
// binding), so at small row counts the host, not the GPU, set the rate.
//
// Every function returns None when the call ran, raises the package's error type with the library's message
// when it failed, and returns NotImplemented for an argument it does not take itself (not a CUDA tensor, not
// 2-D, an unknown keyword, a view whose `c` was replaced; a tensor without storage or with symbolic sizes, as
// under vmap, functional transforms and tracing, whose accessors throw): the caller then goes the ctypes way,
// which either handles the argument or raises the error that belongs to it. The GIL is released around each call.
#include "b200q.h"
#include <torch/csrc/autograd/python_variable.h>
#include <cstring>

namespace {
PyObject *error_type = nullptr;  // breeze_tts_cpp_b200.B200QError
PyObject *view_method = nullptr; // RowScaledView.c as defined by the package
PyObject *name_values, *name_scales, *name_format, *name_group, *name_rotation, *name_c;

constexpr b200q_tensor kNone{nullptr, 0, 0, 0, 0, -1};

int type_code(c10::ScalarType type) {
    switch (type) {
    case c10::ScalarType::BFloat16: return B200Q_BF16;
    case c10::ScalarType::Half: return B200Q_F16;
    case c10::ScalarType::Float: return B200Q_F32;
    case c10::ScalarType::Int: return B200Q_I32;
    case c10::ScalarType::Char: return B200Q_I8;
    default: return -1;
    }
}
// A 1-D or 2-D CUDA tensor with a dense inner axis; false = not one (leave it to the caller's slow path).
bool tensor_of(PyObject *object, b200q_tensor &out, int code = -1) {
    if (object == Py_None) {
        out = kNone;
        return true;
    }
    if (!THPVariable_Check(object)) return false;
    const at::Tensor &t = THPVariable_Unpack(object);
    if (!t.is_cuda()) return false;
    const auto sizes = t.sizes();
    const auto strides = t.strides();
    const size_t dims = sizes.size();
    if ((dims != 1 && dims != 2) || strides[dims - 1] != 1) return false;
    const int64_t rows = dims == 2 ? sizes[0] : 1, cols = sizes[dims - 1];
    const int64_t stride = dims == 2 && rows > 1 && strides[0] != cols ? strides[0] : 0;
    if (code < 0) code = type_code(t.scalar_type());
    if (code < 0 || rows > INT32_MAX || cols > INT32_MAX || stride < 0 || stride > INT32_MAX) return false;
    out = {t.data_ptr(), int32_t(rows), int32_t(cols), int32_t(stride), code, t.get_device()};
    return true;
}
bool int_of(PyObject *object, int32_t &out) {
    if (!PyLong_Check(object)) return false;
    const long v = PyLong_AsLong(object);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    if (v < INT32_MIN || v > INT32_MAX) return false;
    out = int32_t(v);
    return true;
}
bool float_of(PyObject *object, float &out) {
    const double v = PyFloat_AsDouble(object);
    if (v == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    out = float(v);
    return true;
}
struct Ref { // owned reference
    PyObject *p;
    explicit Ref(PyObject *object) : p(object) {
        if (!p) PyErr_Clear();
    }
    ~Ref() { Py_XDECREF(p); }
    Ref(const Ref &) = delete;
};
bool view_of(PyObject *object, b200q_row_scaled &out) {
    const Ref c(PyObject_GetAttr(object, name_c));
    if (!c.p || !PyMethod_Check(c.p) || PyMethod_GET_FUNCTION(c.p) != view_method) return false;
    const Ref values(PyObject_GetAttr(object, name_values)), scales(PyObject_GetAttr(object, name_scales)),
        format(PyObject_GetAttr(object, name_format)), group(PyObject_GetAttr(object, name_group)),
        rotation(PyObject_GetAttr(object, name_rotation));
    int32_t code = 0;
    if (!values.p || !scales.p || !format.p || !group.p || !rotation.p) return false;
    return int_of(format.p, code) && code >= 0 && values.p != Py_None && scales.p != Py_None &&
           tensor_of(values.p, out.values, code) && tensor_of(scales.p, out.scales, B200Q_F32) &&
           int_of(group.p, out.group_size) && int_of(rotation.p, out.rotation_size);
}
// Device pointer of an int32 index tensor (the ABI takes the bare pointer).
bool rows_of(PyObject *object, const int32_t *&out) {
    if (object == Py_None) {
        out = nullptr;
        return true;
    }
    if (!THPVariable_Check(object)) return false;
    const at::Tensor &t = THPVariable_Unpack(object);
    if (!t.is_cuda() || t.scalar_type() != c10::ScalarType::Int) return false;
    out = static_cast<const int32_t *>(t.data_ptr());
    return true;
}
bool is(PyObject *key, const char *name) { return PyUnicode_CompareWithASCIIString(key, name) == 0; }

// Keyword dictionaries; absent (None or empty) is the ABI's default.
bool epilogue_of(PyObject *dict, b200q_epilogue &e) {
    e = {kNone, kNone, kNone, 1.f, 1.f, 1.f, .1f, 0, kNone, kNone, kNone, 1, 0, 1, nullptr};
    if (dict == Py_None) return true;
    if (!PyDict_Check(dict)) return false;
    PyObject *key, *value;
    Py_ssize_t at = 0;
    while (PyDict_Next(dict, &at, &key, &value)) {
        if (!PyUnicode_Check(key)) return false;
        const bool ok = is(key, "bias")                      ? tensor_of(value, e.bias)
                        : is(key, "residual")                ? tensor_of(value, e.residual)
                        : is(key, "activation")              ? int_of(value, e.activation)
                        : is(key, "gate")                    ? tensor_of(value, e.gate)
                        : is(key, "rows_per_sequence")       ? int_of(value, e.rows_per_sequence)
                        : is(key, "residual_f32")            ? tensor_of(value, e.residual_f32, B200Q_F32)
                        : is(key, "value_scale")             ? float_of(value, e.value_scale)
                        : is(key, "output_scale")            ? float_of(value, e.output_scale)
                        : is(key, "residual_scale")          ? float_of(value, e.residual_scale)
                        : is(key, "alpha")                   ? float_of(value, e.alpha)
                        : is(key, "condition")               ? tensor_of(value, e.condition)
                        : is(key, "raw")                     ? tensor_of(value, e.raw)
                        : is(key, "valid_rows_per_sequence") ? int_of(value, e.valid_rows_per_sequence)
                        : is(key, "input_repeat")            ? int_of(value, e.input_repeat)
                        : is(key, "residual_rows")           ? rows_of(value, e.residual_rows)
                                                             : false;
        if (!ok) return false;
    }
    return true;
}
bool fusion_of(PyObject *dict, b200q_norm_fusion &f) {
    f = {kNone, kNone, kNone, kNone, kNone, kNone, 1, nullptr};
    if (dict == Py_None) return true;
    if (!PyDict_Check(dict)) return false;
    PyObject *key, *value;
    Py_ssize_t at = 0;
    while (PyDict_Next(dict, &at, &key, &value)) {
        if (!PyUnicode_Check(key)) return false;
        const bool ok = is(key, "residual")            ? tensor_of(value, f.residual)
                        : is(key, "projection_bias")   ? tensor_of(value, f.projection_bias)
                        : is(key, "raw")               ? tensor_of(value, f.raw)
                        : is(key, "gate")              ? tensor_of(value, f.gate)
                        : is(key, "shift")             ? tensor_of(value, f.shift)
                        : is(key, "scale")             ? tensor_of(value, f.scale)
                        : is(key, "rows_per_sequence") ? int_of(value, f.rows_per_sequence)
                        : is(key, "source_rows")       ? rows_of(value, f.source_rows)
                                                       : false;
        if (!ok) return false;
    }
    return true;
}
bool empty(PyObject *dict) { return dict == Py_None || (PyDict_Check(dict) && !PyDict_GET_SIZE(dict)); }
template <class T> T *handle_of(PyObject *object) { // a Python int; 0 (a closed object) is rejected by the library
    void *p = PyLong_AsVoidPtr(object);
    if (!p) PyErr_Clear();
    return static_cast<T *>(p);
}

PyObject *declined() { Py_RETURN_NOTIMPLEMENTED; }
template <class Call> PyObject *finish(const char *name, Call &&call) {
    char message[512];
    message[0] = 0;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call(message, sizeof message);
    Py_END_ALLOW_THREADS
    if (!rc) Py_RETURN_NONE;
    PyErr_Format(error_type ? error_type : PyExc_RuntimeError, "%s: %s", name, message);
    return nullptr;
}
using Args = PyObject *const *;

PyObject *row_quantize(PyObject *, Args a, Py_ssize_t n) { // context, x, out
    b200q_tensor x;
    b200q_row_scaled out;
    if (n != 3 || !tensor_of(a[1], x) || !view_of(a[2], out)) return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_row_quantize", [&](char *m, size_t s) { return b200q_row_quantize(c, &x, &out, m, s); });
}
PyObject *quantized_norm(PyObject *, Args a, Py_ssize_t n) { // context, residual, update, weight, out, epsilon, gemma, scale
    b200q_tensor x, u, w, scale;
    b200q_row_scaled out;
    float epsilon;
    int32_t gemma;
    if (n != 8 || !tensor_of(a[1], x) || !tensor_of(a[2], u) || !tensor_of(a[3], w) || !view_of(a[4], out) ||
        !float_of(a[5], epsilon) || !int_of(a[6], gemma) || !tensor_of(a[7], scale))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_quantized_norm", [&](char *m, size_t s) {
        return b200q_quantized_norm(c, &x, &u, &w, &out, epsilon, gemma, &scale, m, s);
    });
}
PyObject *quantized_gated(PyObject *, Args a, Py_ssize_t n) { // context, x, out, kind
    b200q_tensor x;
    b200q_row_scaled out;
    int32_t kind;
    if (n != 4 || !tensor_of(a[1], x) || !view_of(a[2], out) || !int_of(a[3], kind)) return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_quantized_gated",
                  [&](char *m, size_t s) { return b200q_quantized_gated(c, &x, &out, kind, m, s); });
}
PyObject *linear(PyObject *, Args a, Py_ssize_t n) { // context, x, weight, out, epilogue
    b200q_row_scaled x, w;
    b200q_tensor out;
    b200q_epilogue e;
    if (n != 5 || !view_of(a[1], x) || !view_of(a[2], w) || !tensor_of(a[3], out) || !epilogue_of(a[4], e)) return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    const b200q_epilogue *ep = empty(a[4]) ? nullptr : &e;
    return finish("b200q_linear", [&](char *m, size_t s) { return b200q_linear(c, &x, &w, &out, ep, m, s); });
}
PyObject *linear_forward(PyObject *, Args a, Py_ssize_t n) { // context, x, weight, scratch, out, epilogue, quantized_output
    b200q_tensor x, out;
    b200q_row_scaled w, scratch, encoded;
    b200q_epilogue e;
    if (n != 7 || !tensor_of(a[1], x) || !view_of(a[2], w) || !view_of(a[3], scratch) || !tensor_of(a[4], out) ||
        !epilogue_of(a[5], e) || (a[6] != Py_None && !view_of(a[6], encoded)))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    const b200q_epilogue *ep = empty(a[5]) ? nullptr : &e;
    const b200q_row_scaled *q = a[6] == Py_None ? nullptr : &encoded;
    return finish("b200q_linear_forward",
                  [&](char *m, size_t s) { return b200q_linear_forward(c, &x, &w, &scratch, &out, ep, q, m, s); });
}
PyObject *layer_forward(PyObject *, Args a, Py_ssize_t n) { // context, layer, x, out, epilogue, quantized_output
    b200q_tensor x, out;
    b200q_row_scaled encoded;
    b200q_epilogue e;
    if (n != 6 || !tensor_of(a[2], x) || !tensor_of(a[3], out) || !epilogue_of(a[4], e) ||
        (a[5] != Py_None && !view_of(a[5], encoded)))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    auto *layer = handle_of<b200q_linear_layer>(a[1]);
    const b200q_epilogue *ep = empty(a[4]) ? nullptr : &e;
    const b200q_row_scaled *q = a[5] == Py_None ? nullptr : &encoded;
    return finish("b200q_linear_layer_forward",
                  [&](char *m, size_t s) { return b200q_linear_layer_forward(c, layer, &x, &out, ep, q, m, s); });
}
// context, layer, x, normalized, out, norm weight, norm bias, epsilon, fusion, epilogue, quantized_output
PyObject *layer_normalized_forward(PyObject *, Args a, Py_ssize_t n) {
    b200q_tensor x, normalized, out, weight, bias;
    b200q_row_scaled encoded;
    b200q_norm_fusion f;
    b200q_epilogue e;
    float epsilon;
    if (n != 11 || !tensor_of(a[2], x) || !tensor_of(a[3], normalized) || !tensor_of(a[4], out) || !tensor_of(a[5], weight) ||
        !tensor_of(a[6], bias) || !float_of(a[7], epsilon) || !fusion_of(a[8], f) || !epilogue_of(a[9], e) ||
        (a[10] != Py_None && !view_of(a[10], encoded)))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    auto *layer = handle_of<b200q_linear_layer>(a[1]);
    const b200q_epilogue *ep = empty(a[9]) ? nullptr : &e;
    const b200q_row_scaled *q = a[10] == Py_None ? nullptr : &encoded;
    return finish("b200q_linear_layer_normalized_forward", [&](char *m, size_t s) {
        return b200q_linear_layer_normalized_forward(c, layer, &x, &normalized, &out, &weight, &bias, epsilon, &f, ep, q, m, s);
    });
}
PyObject *pointwise(PyObject *, Args a, Py_ssize_t n) { // context, x, y, epilogue
    b200q_tensor x, y;
    b200q_epilogue e;
    if (n != 4 || !tensor_of(a[1], x) || !tensor_of(a[2], y) || !epilogue_of(a[3], e)) return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_pointwise", [&](char *m, size_t s) { return b200q_pointwise(c, &x, &y, &e, m, s); });
}
PyObject *pointwise_quantize(PyObject *, Args a, Py_ssize_t n) { // context, x, out, epilogue, retained
    b200q_tensor x, retained;
    b200q_row_scaled out;
    b200q_epilogue e;
    if (n != 5 || !tensor_of(a[1], x) || !view_of(a[2], out) || !epilogue_of(a[3], e) || !tensor_of(a[4], retained))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_pointwise_quantize",
                  [&](char *m, size_t s) { return b200q_pointwise_quantize(c, &x, &out, &e, &retained, m, s); });
}
PyObject *layer_norm_quantize(PyObject *, Args a, Py_ssize_t n) { // context, x, out, weight, bias, epsilon, fusion, retained
    b200q_tensor x, weight, bias, retained;
    b200q_row_scaled out;
    b200q_norm_fusion f;
    float epsilon;
    if (n != 8 || !tensor_of(a[1], x) || !view_of(a[2], out) || !tensor_of(a[3], weight) || !tensor_of(a[4], bias) ||
        !float_of(a[5], epsilon) || !fusion_of(a[6], f) || !tensor_of(a[7], retained))
        return declined();
    auto *c = handle_of<b200q_context>(a[0]);
    return finish("b200q_layer_norm_quantize", [&](char *m, size_t s) {
        return b200q_layer_norm_quantize(c, &x, &out, &weight, &bias, epsilon, &f, &retained, m, s);
    });
}
PyObject *bind(PyObject *, Args a, Py_ssize_t n) { // error type, RowScaledView.c
    if (n != 2) return declined();
    Py_XDECREF(error_type);
    Py_XDECREF(view_method);
    error_type = Py_NewRef(a[0]);
    view_method = Py_NewRef(a[1]);
    Py_RETURN_NONE;
}

// No C++ exception may reach the interpreter: what torch throws at an argument is left to the caller's slow path.
template <PyObject *(*Method)(PyObject *, Args, Py_ssize_t)> PyObject *guarded(PyObject *self, Args a, Py_ssize_t n) {
    try {
        return Method(self, a, n);
    } catch (...) {
        PyErr_Clear();
        return declined();
    }
}
#define B200Q_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B200Q_METHOD(row_quantize),   B200Q_METHOD(quantized_norm),      B200Q_METHOD(quantized_gated),
                         B200Q_METHOD(linear),         B200Q_METHOD(linear_forward),      B200Q_METHOD(layer_forward),
                         B200Q_METHOD(pointwise),      B200Q_METHOD(pointwise_quantize),  B200Q_METHOD(layer_norm_quantize),
                         B200Q_METHOD(layer_normalized_forward), B200Q_METHOD(bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module{PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};
} // namespace

PyMODINIT_FUNC PyInit__native() {
    name_values = PyUnicode_InternFromString("values");
    name_scales = PyUnicode_InternFromString("scales");
    name_format = PyUnicode_InternFromString("format");
    name_group = PyUnicode_InternFromString("group_size");
    name_rotation = PyUnicode_InternFromString("rotation_size");
    name_c = PyUnicode_InternFromString("c");
    return PyModule_Create(&module);
}

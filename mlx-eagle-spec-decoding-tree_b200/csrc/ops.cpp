// Operator calls from Python without the interpreter in between: argument checks, result allocation and the launch through
// the C ABI in one native call (a call spent ~14 us in Python around a launch of 2 us; here the whole call is ~4 us).
//
// Every function returns None when the arguments are anything but the plain case it knows (device, type, shape, layout) or something
// in it throws (a tensor without storage, no memory for the result); the Python operator then takes its own path, which handles or
// refuses them.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <climits>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "b200_eagle.h"

namespace {

// A CUDA tensor of `type` without gaps, or NULL.
const at::Tensor* plain(PyObject* o, at::ScalarType type) {
    if (!THPVariable_Check(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    return t.is_cuda() && t.scalar_type() == type && t.is_contiguous() ? &t : nullptr;
}

// The tensor's device index when it is the current one, else -1.
int on_current(const at::Tensor& t) {
    const int dev = t.get_device();
    return dev == c10::cuda::current_device() ? dev : -1;
}

bool same_device(int dev, const at::Tensor* t) { return t == nullptr || t->get_device() == dev; }

at::Tensor result(at::IntArrayRef sizes, const at::Tensor& like) {
    return at::detail::empty_cuda(sizes, at::kHalf, like.device(), c10::nullopt);
}

void* stream_of(int dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }

bool int_arg(PyObject* o, long* v) {
    *v = PyLong_AsLong(o);
    if (*v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

// qmm(x, w, s, b, group_size, bias, workspace) -> y
PyObject* qmm(PyObject* const* a, Py_ssize_t n) {
    long group;
    if (n != 7 || !int_arg(a[4], &group) || group != 64) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0], at::kHalf), *s = plain(a[2], at::kHalf), *b = plain(a[3], at::kHalf);
    const at::Tensor *bias = a[5] == Py_None ? nullptr : plain(a[5], at::kHalf), *ws = plain(a[6], at::kByte);
    if (!x || !s || !b || !ws || (a[5] != Py_None && !bias) || !THPVariable_Check(a[1])) Py_RETURN_NONE;
    const at::Tensor& w = THPVariable_Unpack(a[1]);
    if (!w.is_cuda() || (w.scalar_type() != at::kInt && w.scalar_type() != at::kUInt32) || !w.is_contiguous()) Py_RETURN_NONE;
    const int dev = on_current(*x);
    if (dev < 0 || !same_device(dev, s) || !same_device(dev, b) || !same_device(dev, &w) || !same_device(dev, bias) || !same_device(dev, ws) ||
        x->dim() < 1 || w.dim() != 2 || s->dim() != 2 || b->dim() != 2)
        Py_RETURN_NONE;
    const int64_t K = x->size(-1), N = w.size(0);
    if (K < 128 || K % 128 || w.size(1) * 8 != K || s->size(0) != N || s->size(1) * 64 != K || b->size(0) != N || b->size(1) * 64 != K) Py_RETURN_NONE;
    const int64_t M = x->numel() / K;
    if (M < 1 || M > INT_MAX || N > INT_MAX || (bias && bias->numel() != N)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 5> sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = N;
    at::Tensor y = result(sizes, *x);
    const int rc = b200_qmm(x->data_ptr(), static_cast<const uint32_t*>(w.data_ptr()), s->data_ptr(), b->data_ptr(), bias ? bias->data_ptr() : nullptr,
                            y.data_ptr(), (int)M, (int)N, (int)K, 64, 0, ws->data_ptr(), (size_t)ws->numel(), stream_of(dev));
    if (rc != B200_OK) Py_RETURN_NONE;                   // (nothing was launched: the Python operator reports it)
    return THPVariable_Wrap(std::move(y));
}

// qmm_tiled(x, wt, n, bias, workspace) -> y
PyObject* qmm_tiled(PyObject* const* a, Py_ssize_t n) {
    long N;
    if (n != 5 || !int_arg(a[2], &N)) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0], at::kHalf), *wt = plain(a[1], at::kByte), *ws = plain(a[4], at::kByte);
    const at::Tensor* bias = a[3] == Py_None ? nullptr : plain(a[3], at::kHalf);
    if (!x || !wt || !ws || (a[3] != Py_None && !bias) || x->dim() != 2) Py_RETURN_NONE;
    const int dev = on_current(*x);
    if (dev < 0 || !same_device(dev, wt) || !same_device(dev, bias) || !same_device(dev, ws)) Py_RETURN_NONE;
    const int64_t M = x->size(0), K = x->size(1);
    if (M < 1 || M > 32 || N < 8 || N > INT_MAX || K > INT_MAX || (bias && bias->numel() != N)) Py_RETURN_NONE;
    const size_t need = b200_qmm_tiled_bytes((int)N, (int)K);
    if (need == 0 || (size_t)wt->numel() < need) Py_RETURN_NONE;
    at::Tensor y = result({M, (int64_t)N}, *x);
    const int rc = b200_qmm_tiled(x->data_ptr(), wt->data_ptr(), nullptr, bias ? bias->data_ptr() : nullptr, nullptr, y.data_ptr(), (int)M, (int)N,
                                  (int)K, B200_EPI_NONE, ws->data_ptr(), (size_t)ws->numel(), stream_of(dev));
    if (rc != B200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
}

// rope_positions(inp, offsets, inv_freqs, scaling_factor) -> out
PyObject* rope_positions(PyObject* const* a, Py_ssize_t n) {
    if (n != 4) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0], at::kHalf), *pos = plain(a[1], at::kInt), *inv = plain(a[2], at::kFloat);
    const double scaling = PyFloat_AsDouble(a[3]);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        Py_RETURN_NONE;
    }
    if (!x || !pos || !inv || x->dim() != 4) Py_RETURN_NONE;
    const int dev = on_current(*x);
    const int64_t B = x->size(0), H = x->size(1), L = x->size(2), D = x->size(3);
    if (dev < 0 || !same_device(dev, pos) || !same_device(dev, inv) || pos->numel() != B * L || inv->numel() != D / 2) Py_RETURN_NONE;
    at::Tensor y = result(x->sizes(), *x);
    const int rc = b200_rope_positions(x->data_ptr(), static_cast<const int*>(pos->data_ptr()), static_cast<const float*>(inv->data_ptr()),
                                       (float)scaling, y.data_ptr(), (int)B, (int)H, (int)L, (int)D, stream_of(dev));
    if (rc != B200_OK) Py_RETURN_NONE;
    return THPVariable_Wrap(std::move(y));
}

// layer_pointers(layers, table[, fast]) -> 0: `table` (address of [layers][8] pointers in the order of b200_forward_desc.layer_table) holds
// the device pointers of the layers already, 1: it does now, -1: a layer is not as it should be (no re-laid-out weights, say).
// Runs ahead of every pass, so that a pass never sees the address of a tensor that has been replaced: ~0.35 us a layer.  `fast` (address of 32
// bits) becomes 1 if every re-laid-out matrix is known to allow the short expansion as it is now, as QLinear.scales_fast, 0 if not.  (Asked
// for every pass like the addresses: a matrix that has taken the place of one that was freed can have its address and its count of changes.)
PyObject* layer_pointers(PyObject*, PyObject* const* a, Py_ssize_t n) {
    static PyObject* const linears[] = {PyUnicode_InternFromString("qkv"), PyUnicode_InternFromString("o"), PyUnicode_InternFromString("gate"),
                                        PyUnicode_InternFromString("up"), PyUnicode_InternFromString("down")};
    static PyObject* const norms[] = {PyUnicode_InternFromString("input_norm"), PyUnicode_InternFromString("post_norm")};
    static PyObject* const tiled = PyUnicode_InternFromString("tiled");
    static PyObject* const bias = PyUnicode_InternFromString("bias");
    static PyObject* const fast_of = PyUnicode_InternFromString("_fast_of");
    void** table = (n == 2 || n == 3) && (PyList_Check(a[0]) || PyTuple_Check(a[0])) ? static_cast<void**>(PyLong_AsVoidPtr(a[1])) : nullptr;
    uint32_t* fast = table != nullptr && n == 3 ? static_cast<uint32_t*>(PyLong_AsVoidPtr(a[2])) : nullptr;
    if (PyErr_Occurred()) return nullptr;
    if (table == nullptr) return PyLong_FromLong(-1);
    if (fast != nullptr) *fast = 0;
    bool plain = true, same = true, all_fast = fast != nullptr;
    auto put = [&](PyObject* t, bool optional) {              // (borrowed, may be NULL)
        void* q = nullptr;
        if (t == nullptr || !THPVariable_Check(t)) plain = plain && optional && t == Py_None;
        else q = THPVariable_Unpack(t).data_ptr();
        same = same && *table == q;
        *table++ = q;
    };
    auto put_attr = [&](PyObject* o, PyObject* name, bool optional) {
        PyObject* t = o == nullptr ? nullptr : PyObject_GetAttr(o, name);
        if (t == nullptr) PyErr_Clear();
        put(t, optional);
        if (name == tiled && all_fast) {                         // (the tensor looked at, its count of changes then)
            PyObject* of = t == nullptr ? nullptr : PyObject_GetAttr(o, fast_of);
            if (of == nullptr) PyErr_Clear();
            all_fast = of != nullptr && PyTuple_Check(of) && PyTuple_GET_SIZE(of) == 2 && PyTuple_GET_ITEM(of, 0) == t && THPVariable_Check(t) &&
                       !THPVariable_Unpack(t).is_inference() && PyLong_AsLongLong(PyTuple_GET_ITEM(of, 1)) == (long long)THPVariable_Unpack(t)._version();
            if (PyErr_Occurred()) PyErr_Clear();                 // (no number there)
            Py_XDECREF(of);
        }
        Py_XDECREF(t);                                           // (the layer still holds it)
    };
    try {
        const Py_ssize_t layers = PySequence_Fast_GET_SIZE(a[0]);
        for (Py_ssize_t l = 0; l < layers; l++) {
            PyObject* layer = PySequence_Fast_GET_ITEM(a[0], l);
            if (!PyDict_Check(layer)) return PyLong_FromLong(-1);
            for (int i = 0; i < 5; i++) {
                PyObject* lin = PyDict_GetItem(layer, linears[i]);
                put_attr(lin, tiled, false);
                if (i == 0) put_attr(lin, bias, true);
            }
            for (PyObject* name : norms) put(PyDict_GetItem(layer, name), false);
        }
    } catch (const std::exception&) {                            // (a tensor without storage)
        plain = false;
    }
    if (fast != nullptr) *fast = plain && all_fast;
    return PyLong_FromLong(!plain ? -1 : (same ? 0 : 1));
}

// No C++ exception passes through the interpreter's frames: it would end the process.
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* caught(PyObject*, PyObject* const* a, Py_ssize_t n) {
    try {
        return F(a, n);
    } catch (const std::exception&) {
        Py_RETURN_NONE;
    }
}

#define FAST(name, f) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST("qmm", caught<qmm>), FAST("qmm_tiled", caught<qmm_tiled>), FAST("rope_positions", caught<rope_positions>),
                         FAST("layer_pointers", layer_pointers), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_b200ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200ops(void) { return PyModule_Create(&module); }

// The forward's host path in native code: what OrthoLinear.forward, _C_ops.forward and _C_ops.forward_multi do on every call that
// is the same as one before it -- checks, output, argument record, launch -- without going through Python and ctypes for each
// step.  Everything that is not plain (another dtype or device, a tensor subclass, a stream under capture with scratch, a record
// that has to be made) is left to the Python code: these functions then return None and have done nothing.
//
// The checks are the Python code's own: a record holds what it was made for (pointers and version counters of every buffer) and is
// compared with the module's present buffers on each call; nothing is remembered by the identity of an input.
#include <Python.h>

#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/torch.h>

#include <memory>

#include "../../include/ortho_b200.h"

namespace {

using multi_fn = int (*)(const ortho_b200_layer_desc *, int, const void *, int64_t, int64_t, void *, int64_t, void *);
using multi_ws_fn = int64_t (*)(const ortho_b200_layer_desc *, int, int64_t, int64_t);
using typed_fn = int (*)(const ortho_b200_layer_desc *, const void *, int, int, int64_t, int64_t, void *, void *, int64_t, void *);
multi_fn forward_multi = nullptr;
typed_fn forward_typed = nullptr;
multi_ws_fn multi_workspace = nullptr;

struct Ptr { const void *data; int64_t version; };
struct Record {
    ortho_b200_layer_desc desc;
    Ptr buf[5];                                  // base_weight, base_scales, ortho_values, ortho_col_indices, ortho_row_ptr
    const void *bias;
    int bias_type;
    bool has_bias, add_bias, active;             // add_bias: not one that the kernel adds; active: alpha > 0
    int64_t ws_bytes;
    void *ws_ptr;
    int64_t ws_gen;
    PyObject *ws;                                // the scratch's owner: `gen` and `tensor`
    PyObject *plan;                              // owner of desc.plan, or None: held, also while a launch runs without the lock
    int device;
    int type;                                    // ORTHO_B200_TYPE_* of activations and output
    bool converts;                               // activations of another type that the kernel needs as FP16
    bool takes;                                  // no: the kernel does not take that type, the FP16 record converts around
};
const char *kBuffers[5] = {"base_weight", "base_scales", "ortho_values", "ortho_col_indices", "ortho_row_ptr"};
PyObject *s_buffers[5], *s_bias, *s_gen, *s_tensor, *s_handle, *s_value, *s_fast;

void free_record(PyObject *cap)
{
    Record *r = static_cast<Record *>(PyCapsule_GetPointer(cap, "ortho_record"));
    if (!r) { PyErr_Clear(); return; }
    Py_XDECREF(r->ws);
    Py_XDECREF(r->plan);
    delete r;
}

// a plain CUDA tensor whose storage holds its values (no negation pending), or nullptr
const at::Tensor *plain(PyObject *o)
{
    if (!o || !THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor &t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || !t.has_storage() || t.layout() != at::kStrided || t.is_neg() || t.unsafeGetTensorImpl()->is_python_dispatch()) return nullptr;
    return &t;
}

bool same_buffers(const Record &r, PyObject *buffers, PyObject *params)
{
    for (int i = 0; i < 5; i++) {
        PyObject *o = PyDict_GetItemWithError(buffers, s_buffers[i]);
        if (!o || !THPVariable_Check(o)) return false;
        const at::Tensor &t = THPVariable_Unpack(o);
        if (!t.has_storage() || t.const_data_ptr() != r.buf[i].data) return false;
        if (i >= 2 && (int64_t)t._version() != r.buf[i].version) return false;      // the CSR buffers' contents
    }
    PyObject *b = PyDict_GetItemWithError(params, s_bias);
    if (!b) return false;
    if (b == Py_None) return !r.has_bias;
    if (!r.has_bias || !THPVariable_Check(b)) return false;
    const at::Tensor &t = THPVariable_Unpack(b);
    if (r.add_bias && (!plain(b) || t.dim() != 1)) return false;
    return t.has_storage() && (int)t.scalar_type() == r.bias_type && t.const_data_ptr() == r.bias;
}

// record(desc_address, plan or None, buffers, bias or None, active, ws, ws_gen, ws_ptr, ws_bytes, device, type, converts) -> capsule.
// converts: bytes of the FP16 copy, negative where the kernel does not take the type
PyObject *make_record(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 12) { PyErr_SetString(PyExc_TypeError, "record takes 12 arguments"); return nullptr; }
    HANDLE_TH_ERRORS
    auto r = std::make_unique<Record>();
    r->desc = *static_cast<const ortho_b200_layer_desc *>(PyLong_AsVoidPtr(a[0]));
    for (int i = 0; i < 5; i++) {
        PyObject *o = PyDict_GetItemWithError(a[2], s_buffers[i]);
        if (!o || !THPVariable_Check(o)) Py_RETURN_NONE;
        const at::Tensor &t = THPVariable_Unpack(o);
        // the base buffers' contents are read anew on each forward and may be tensors made in inference mode, which have no version
        r->buf[i] = Ptr{t.const_data_ptr(), i >= 2 ? (int64_t)t._version() : 0};
    }
    r->has_bias = a[3] != Py_None;
    if (r->has_bias) {
        if (!r->desc.bias_f32 && !plain(a[3])) Py_RETURN_NONE;
        const at::Tensor &b = THPVariable_Unpack(a[3]);
        r->bias = b.const_data_ptr();
        r->bias_type = (int)b.scalar_type();
        r->add_bias = !r->desc.bias_f32;
    }
    r->active = PyObject_IsTrue(a[4]) == 1;
    r->ws_gen = PyLong_AsLongLong(a[6]);
    r->ws_ptr = a[7] == Py_None ? nullptr : PyLong_AsVoidPtr(a[7]);
    r->ws_bytes = PyLong_AsLongLong(a[8]);
    r->device = (int)PyLong_AsLong(a[9]);
    r->type = (int)PyLong_AsLong(a[10]);
    const int64_t converts = PyLong_AsLongLong(a[11]);
    r->converts = converts > 0;
    r->takes = converts >= 0;
    if (PyErr_Occurred()) return nullptr;
    PyObject *cap = PyCapsule_New(r.get(), "ortho_record", free_record);
    if (!cap) return nullptr;
    r->plan = Py_NewRef(a[1]);
    r.release()->ws = Py_NewRef(a[5]);
    return cap;
    END_HANDLE_TH_ERRORS
}

// the record of a call, or None / nullptr (with an error set): a new reference
PyObject *find_record(PyObject *bound, int64_t M, void *stream, int type)
{
    PyObject *key = type == ORTHO_B200_TYPE_F16 ? Py_BuildValue("(LK)", (long long)M, (unsigned long long)(uintptr_t)stream)
                                                : Py_BuildValue("(LKi)", (long long)M, (unsigned long long)(uintptr_t)stream, type);
    if (!key) return nullptr;
    PyObject *b = PyDict_GetItemWithError(bound, key);
    Py_DECREF(key);
    if (b) return PyObject_GetAttr(b, s_fast);
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

// module(x, buffers, parameters, bound, alpha, in_features, out_features) -> output, an int status, or None
PyObject *module_forward(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "module takes 7 arguments"); return nullptr; }
    HANDLE_TH_ERRORS
    const at::Tensor *x = plain(a[0]);
    if (!x || x->dim() < 1) Py_RETURN_NONE;
    const auto dtype = x->scalar_type();
    int type = dtype == at::kHalf ? ORTHO_B200_TYPE_F16 : dtype == at::kBFloat16 ? ORTHO_B200_TYPE_BF16 : dtype == at::kFloat ? ORTHO_B200_TYPE_F32 : -1;
    if (type < 0) Py_RETURN_NONE;
    // the kernels read rows that follow one another, 16 bytes at a time; an FP16 copy of other activations is contiguous and aligned
    const bool in_order = x->is_contiguous();
    if (type != ORTHO_B200_TYPE_F16 && (!in_order || ((uintptr_t)x->const_data_ptr() & 15u) != 0)) type = ORTHO_B200_TYPE_F16;
    const int64_t K = PyLong_AsLongLong(a[5]), N = PyLong_AsLongLong(a[6]);
    const double alpha = PyFloat_AsDouble(a[4]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    if (x->size(-1) != K || x->numel() == 0 || K <= 0) Py_RETURN_NONE;
    const int64_t M = x->numel() / K;
    const int dev = x->get_device();
    if (c10::cuda::current_device() != dev) Py_RETURN_NONE;
    void *stream = (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    std::unique_ptr<PyObject, void (*)(PyObject *)> hold_rec(nullptr, [](PyObject *o) { Py_XDECREF(o); });
    Record *r = nullptr;
    at::Tensor as_half;                          // the FP16 copy of activations that are converted around the FP16 forward
    for (;;) {
        hold_rec.reset(find_record(a[3], M, stream, type));
        if (!hold_rec) return nullptr;
        if (hold_rec.get() == Py_None) Py_RETURN_NONE;
        r = static_cast<Record *>(PyCapsule_GetPointer(hold_rec.get(), "ortho_record"));
        if (!r) { PyErr_Clear(); Py_RETURN_NONE; }
        if (r->device != dev || r->type != type || (alpha > 0) != r->active || r->desc.N != N) Py_RETURN_NONE;
        if (r->takes) break;
        type = ORTHO_B200_TYPE_F16;              // (a record of that type takes it)
    }
    if (!same_buffers(*r, a[1], a[2])) Py_RETURN_NONE;
    at::Tensor bias;                             // in hand, whatever other threads replace during the launch
    if (r->add_bias) bias = THPVariable_Unpack(PyDict_GetItemWithError(a[2], s_bias));
    // the scratch of the record, held over the launch whatever other threads bind meanwhile
    PyObject *scratch = nullptr;
    if (r->ws_bytes) {
        scratch = PyObject_GetAttr(r->ws, s_tensor);
        PyObject *gen = scratch ? PyObject_GetAttr(r->ws, s_gen) : nullptr;
        const bool same = gen && PyLong_AsLongLong(gen) == r->ws_gen && scratch != Py_None;
        Py_XDECREF(gen);
        if (PyErr_Occurred()) { Py_XDECREF(scratch); return nullptr; }
        if (!same || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) { Py_DECREF(scratch); Py_RETURN_NONE; }
    }
    std::unique_ptr<PyObject, void (*)(PyObject *)> hold_scratch(scratch, [](PyObject *o) { Py_XDECREF(o); });
    const bool around = type == ORTHO_B200_TYPE_F16 && dtype != at::kHalf;
    if (around || !in_order) {
        as_half = x->to(at::kHalf).contiguous();
        if (!as_half.has_storage() || as_half.unsafeGetTensorImpl()->is_python_dispatch()) Py_RETURN_NONE;
        x = &as_half;
    }
    at::Tensor y;
    {
        c10::SmallVector<int64_t, 6> shape(x->sizes().begin(), x->sizes().end());
        shape.back() = N;
        y = at::empty(shape, at::TensorOptions().dtype(x->scalar_type()).device(x->device()));
    }
    if (!y.has_storage() || y.unsafeGetTensorImpl()->is_python_dispatch()) Py_RETURN_NONE;
    ortho_b200_layer_desc d = r->desc;
    d.y_f16 = y.mutable_data_ptr();
    d.alpha = (float)alpha;
    const void *xp = x->const_data_ptr();
    at::Tensor copy;                             // back with torch's allocator, in stream order, when the call returns
    if (r->converts) {
        copy = at::empty({M, K}, at::TensorOptions().dtype(at::kHalf).device(x->device()));
        if (!copy.has_storage() || copy.unsafeGetTensorImpl()->is_python_dispatch()) Py_RETURN_NONE;
    }
    void *ws = r->ws_ptr, *xs = r->converts ? copy.mutable_data_ptr() : nullptr;
    const int64_t ws_bytes = r->ws_bytes;
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = type == ORTHO_B200_TYPE_F16 ? forward_multi(&d, 1, xp, M, K, ws, ws_bytes, stream)
                                     : forward_typed(&d, xp, type, type, M, K, xs, ws, ws_bytes, stream);
    Py_END_ALLOW_THREADS
    // The typed call is routed anew each time: with other routing settings, or an alpha too small for FP32, it may be one that the kernels
    // do not take or that needs the FP16 copy this record has no room for.  It says so before it launches the forward.
    if (type != ORTHO_B200_TYPE_F16 && (st == ORTHO_B200_ERR_SHAPE || st == ORTHO_B200_ERR_ALIGN || st == ORTHO_B200_ERR_WORKSPACE)) Py_RETURN_NONE;
    if (st) return PyLong_FromLong(st);
    if (bias.defined()) y.add_(bias);
    if (around) y = y.to(dtype);
    return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}

// one layer's tensors -> record; false: leave it to Python (which raises where something is wrong)
bool layer(ortho_b200_layer_desc &d, PyObject *qw_, PyObject *qs_, PyObject *ov_, PyObject *oc_, PyObject *orp_, PyObject *y_, PyObject *plan,
           PyObject *bias, int64_t M, int64_t K, int dev)
{
    const at::Tensor *qw = plain(qw_), *qs = plain(qs_), *y = plain(y_), *ov = plain(ov_);
    if (!qw || !qs || !y || !ov) return false;
    if (qw->scalar_type() != at::kByte || qs->scalar_type() != at::kHalf || y->scalar_type() != at::kHalf) return false;
    if (y->dim() != 2 || !y->is_contiguous() || y->size(0) != M) return false;
    const int64_t N = y->size(1);
    if (qw->dim() != 2 || qw->size(0) != N || qw->size(1) != K / 2 || qs->numel() != N || !qw->is_contiguous() || !qs->is_contiguous()) return false;
    if (qw->get_device() != dev || qs->get_device() != dev || y->get_device() != dev || ov->get_device() != dev) return false;
    const int64_t nnz = ov->numel();
    d.plan = nullptr;
    if (plan && plan != Py_None) {
        PyObject *h = PyObject_GetAttr(plan, s_handle), *v = h && h != Py_None ? PyObject_GetAttr(h, s_value) : nullptr;
        void *p = v && v != Py_None ? PyLong_AsVoidPtr(v) : nullptr;
        Py_XDECREF(h); Py_XDECREF(v);
        if (PyErr_Occurred()) { PyErr_Clear(); return false; }
        if (!p) return false;
        d.plan = static_cast<const ortho_b200_plan *>(p);
    }
    d.ortho_values_f16 = nullptr; d.ortho_col_indices = nullptr; d.ortho_row_ptr = nullptr;
    if (nnz) {
        const at::Tensor *oc = plain(oc_), *orp = plain(orp_);
        if (!oc || !orp || ov->scalar_type() != at::kHalf || oc->scalar_type() != at::kInt || orp->scalar_type() != at::kInt) return false;
        if (orp->numel() != N + 1 || oc->numel() != nnz || oc->get_device() != dev || orp->get_device() != dev) return false;
        if (!ov->is_contiguous() || !oc->is_contiguous() || !orp->is_contiguous()) return false;
        d.ortho_values_f16 = ov->const_data_ptr();
        d.ortho_col_indices = static_cast<const int32_t *>(oc->const_data_ptr());
        d.ortho_row_ptr = static_cast<const int32_t *>(orp->const_data_ptr());
    }
    d.bias_f32 = nullptr;
    if (bias && bias != Py_None) {
        const at::Tensor *b = plain(bias);
        if (!b || b->scalar_type() != at::kFloat || b->numel() != N || !b->is_contiguous() || b->get_device() != dev) return false;
        d.bias_f32 = static_cast<const float *>(b->const_data_ptr());
    }
    d.q_weight = qw->const_data_ptr(); d.q_scales_f16 = qs->const_data_ptr();
    d.nnz = nnz; d.y_f16 = y->mutable_data_ptr(); d.N = N; d.ldy = 0; d.reserved = 0;
    return true;
}

// layers(list of 5-tuples, x, outputs, alphas, biases, plans, workspace): the launch -> int status, or None.
// alphas, biases and plans are lists / tuples or None; a workspace that is None or too small is replaced by a temporary.
PyObject *layers_forward(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "layers takes 7 arguments"); return nullptr; }
    HANDLE_TH_ERRORS
    const at::Tensor *x = plain(a[1]);
    if (!x || x->scalar_type() != at::kHalf || x->dim() != 2 || !x->is_contiguous()) Py_RETURN_NONE;
    const int64_t M = x->size(0), K = x->size(1);
    const int dev = x->get_device();
    if (c10::cuda::current_device() != dev) Py_RETURN_NONE;
    auto seq = [](PyObject *o) { return PyList_CheckExact(o) || PyTuple_CheckExact(o); };
    const Py_ssize_t nl = seq(a[0]) ? PySequence_Fast_GET_SIZE(a[0]) : 0;
    if (nl < 1 || nl > ORTHO_B200_MULTI_MAX_LAYERS) Py_RETURN_NONE;
    for (int i = 2; i < 6; i++)
        if (!(i > 2 && a[i] == Py_None) && (!seq(a[i]) || PySequence_Fast_GET_SIZE(a[i]) < nl)) Py_RETURN_NONE;
    ortho_b200_layer_desc d[ORTHO_B200_MULTI_MAX_LAYERS];
    memset(d, 0, sizeof(d));
    for (Py_ssize_t i = 0; i < nl; i++) {
        PyObject *t = PySequence_Fast_GET_ITEM(a[0], i);
        if (!seq(t) || PySequence_Fast_GET_SIZE(t) != 5) Py_RETURN_NONE;
        PyObject **f = PySequence_Fast_ITEMS(t);
        auto at = [&](int j) { return a[j] == Py_None ? nullptr : PySequence_Fast_GET_ITEM(a[j], i); };
        if (!layer(d[i], f[0], f[1], f[2], f[3], f[4], at(2), at(5), at(4), M, K, dev)) Py_RETURN_NONE;
        d[i].alpha = 1.f;
        if (a[3] != Py_None) {
            d[i].alpha = (float)PyFloat_AsDouble(at(3));
            if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
        }
    }
    const int64_t need = multi_workspace(d, (int)nl, M, K);
    if (need < 0) Py_RETURN_NONE;
    at::Tensor own;
    void *ws = nullptr;
    int64_t ws_bytes = 0;
    if (need) {
        const at::Tensor *given = a[6] == Py_None ? nullptr : plain(a[6]);
        if (a[6] != Py_None && (!given || given->get_device() != dev)) Py_RETURN_NONE;
        if (!given || (int64_t)given->nbytes() < need) {
            own = at::empty({need}, at::TensorOptions().dtype(at::kByte).device(x->device()));
            if (!own.has_storage() || own.unsafeGetTensorImpl()->is_python_dispatch()) Py_RETURN_NONE;
            given = &own;
        }
        ws = given->mutable_data_ptr();
        ws_bytes = (int64_t)given->nbytes();
    }
    const void *xp = x->const_data_ptr();
    void *stream = (void *)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = forward_multi(d, (int)nl, xp, M, K, ws, ws_bytes, stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(st);
    END_HANDLE_TH_ERRORS
}

// addresses of ortho_b200_forward_multi, ortho_b200_multi_workspace_bytes and ortho_b200_forward_typed in the loaded library
PyObject *set_library(PyObject *, PyObject *const *a, Py_ssize_t n)
{
    if (n != 3) { PyErr_SetString(PyExc_TypeError, "set_library takes 3 arguments"); return nullptr; }
    forward_multi = reinterpret_cast<multi_fn>(PyLong_AsVoidPtr(a[0]));
    multi_workspace = reinterpret_cast<multi_ws_fn>(PyLong_AsVoidPtr(a[1]));
    forward_typed = reinterpret_cast<typed_fn>(PyLong_AsVoidPtr(a[2]));
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"record", (PyCFunction)(void (*)(void))make_record, METH_FASTCALL, nullptr},
    {"module", (PyCFunction)(void (*)(void))module_forward, METH_FASTCALL, nullptr},
    {"layers", (PyCFunction)(void (*)(void))layers_forward, METH_FASTCALL, nullptr},
    {"set_library", (PyCFunction)(void (*)(void))set_library, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void)
{
    for (int i = 0; i < 5; i++) s_buffers[i] = PyUnicode_InternFromString(kBuffers[i]);
    s_bias = PyUnicode_InternFromString("bias");
    s_gen = PyUnicode_InternFromString("gen");
    s_tensor = PyUnicode_InternFromString("tensor");
    s_handle = PyUnicode_InternFromString("handle");
    s_value = PyUnicode_InternFromString("value");
    s_fast = PyUnicode_InternFromString("fast");
    PyObject *m = PyModule_Create(&module_def);
    // the torch it was compiled against: a module built for another one is not to be used
    if (m && PyModule_AddStringConstant(m, "torch_version", ORTHO_TORCH_VERSION) < 0) { Py_DECREF(m); return nullptr; }
    return m;
}

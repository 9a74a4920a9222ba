// The host side of a node's call, as a CPython extension: what DequantDot / DecodeAttention do between "the user has a
// tensor" and "the C ABI is called".
//
// A decode step is a chain of launches of a few microseconds each, so the time the host spends per launch is part of
// the step: through ctypes and torch's Python wrappers (descriptor fields, workspace lookup, current stream, nine
// converted arguments) a call took 13 to 19 us of host time for 4 to 8 us of GPU time.  Here a call is: look at the
// tensor, find the entry for its row count and type, allocate the output, take the current stream, call the C ABI.  A row
// count and type that has not been seen asks the node for its descriptor and workspace first (a prompt's length is new more
// often than not: 20 us where the Python path takes 28).
//
// The objects here never decide anything on their own.  Whatever is not the plain case (a tensor that is not a contiguous
// CUDA tensor of the right shape, an addend that is missing) makes the call return None, and the Python method runs its full
// path, which checks and raises.
//
// Entries are added and looked up under the interpreter lock.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>
#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <cstring>
#include <new>
#include <unordered_map>

#include "nnf_b200.h"

namespace
{
using LinearFn = int (*)(nnf_b200_ctx*, void*, const nnf_b200_linear_desc*, const void*, const nnf_b200_qweight*,
                         const nnf_b200_qweight*, const void*, const void*, void*, void*, size_t);
using AttnFn = int (*)(nnf_b200_ctx*, void*, const nnf_b200_attn_desc*, const void*, const void*, const void*, void*,
                       void*, void*, void*, size_t);
using AttnWsFn = size_t (*)(const nnf_b200_ctx*, const nnf_b200_attn_desc*);

// A tensor the C ABI can take as it is, or null.
const at::Tensor* plain_cuda(PyObject* o)
{
    if (!THPVariable_Check(o))
        return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda() || !t.is_contiguous())
        return nullptr;
    return &t;
}

int dtype_code(c10::ScalarType s)
{
    return s == at::kHalf ? NNF_B200_F16 : s == at::kFloat ? NNF_B200_F32 : -1;
}

PyObject* wrapped_empty(at::IntArrayRef sizes, c10::ScalarType dtype, c10::Device device)
{
    return THPVariable_Wrap(at::Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt)));
}

const void* address_of(PyObject* o)
{
    return o == Py_None ? nullptr : THPVariable_Unpack(o).const_data_ptr();
}

// A workspace: a tensor of bytes, or None.
bool is_workspace(PyObject* o)
{
    return o == Py_None || (THPVariable_Check(o) && THPVariable_Unpack(o).is_contiguous() && THPVariable_Unpack(o).itemsize() == 1);
}

size_t bytes_of(PyObject* ws)
{
    return ws == Py_None ? 0 : (size_t)THPVariable_Unpack(ws).numel();
}

// ---------------------------------------------------------------------------------------------------- linear

struct LinearEntry
{
    nnf_b200_linear_desc desc;
    PyObject* ws = nullptr; // the workspace, a tensor that this entry keeps alive, or None
    void* ws_data = nullptr;
    size_t ws_bytes = 0;
};

struct LinearCall
{
    PyObject_HEAD
    LinearFn fn;
    Py_buffer handle;
    nnf_b200_qweight w, w2;
    int has_w2, add;
    PyObject* gain;  // tensors or None: their addresses are read at every call
    PyObject* bias;
    PyObject* check; // Context.check: raises for a status that is not OK
    int64_t N, K;
    std::unordered_map<uint64_t, LinearEntry>* entries; // by row count and type
    const LinearEntry* last; // ... the one found last, and its key
    uint64_t last_key;
};
constexpr size_t kMaxEntries = 4096; // beyond that they are all let go and made again

void clear_entries(LinearCall* c)
{
    std::unordered_map<uint64_t, LinearEntry> old;
    old.swap(*c->entries);
    c->last = nullptr;
    for (auto& e : old)
        Py_DECREF(e.second.ws);
}

// Adds the entry that the node gives for a row count and type: (descriptor bytes, workspace or None).
bool add_entry(LinearCall* c, PyObject* node, int64_t M, int xd, LinearEntry* e, THPObjectPtr* ws)
{
    THPObjectPtr plan(PyObject_CallMethod(node, "_plan", "Li", (long long)M, xd));
    Py_buffer desc;
    PyObject* w;
    if (!plan || !PyArg_ParseTuple(plan.get(), "y*O", &desc, &w))
        return false;
    const bool ok = desc.len == (Py_ssize_t)sizeof e->desc && is_workspace(w);
    if (ok)
        memcpy(&e->desc, desc.buf, sizeof e->desc);
    PyBuffer_Release(&desc);
    if (!ok)
    {
        PyErr_SetString(PyExc_ValueError, "_plan: (descriptor bytes, workspace)");
        return false;
    }
    *ws = THPObjectPtr::dup(w);
    e->ws = w, e->ws_data = const_cast<void*>(address_of(w)), e->ws_bytes = bytes_of(w);
    if (c->entries->size() >= kMaxEntries)
        clear_entries(c);
    LinearEntry& slot = (*c->entries)[(uint64_t)M << 1 | (uint64_t)xd];
    THPObjectPtr before(slot.ws); // (another thread may have been here meanwhile)
    slot = *e;
    Py_INCREF(w);
    return true;
}

// The library's context, as the node's Context holds it now: null once that has been closed (the C ABI then refuses).
nnf_b200_ctx* context(const Py_buffer& handle)
{
    return *static_cast<nnf_b200_ctx* const*>(handle.buf);
}

// Takes a Context's handle (a ctypes.c_void_p; its storage is read at every call).
bool hold_handle(PyObject* o, Py_buffer* handle)
{
    if (PyObject_GetBuffer(o, handle, PyBUF_SIMPLE) < 0)
        return false;
    if (handle->len == (Py_ssize_t)sizeof(void*))
        return true;
    PyBuffer_Release(handle);
    PyErr_SetString(PyExc_ValueError, "handle size");
    return false;
}

// y = node(x) with x [..., K]; lead: the output takes x's leading dimensions instead of [M, N].
PyObject* linear_run(LinearCall* self, PyObject* node, PyObject* px, PyObject* pout, PyObject* paddend, bool lead)
{
    const at::Tensor* x = plain_cuda(px);
    if (!x)
        Py_RETURN_NONE;
    const int xd = dtype_code(x->scalar_type());
    const int64_t dims = x->dim();
    const int64_t K = self->K, N = self->N;
    if (xd < 0 || (lead ? dims < 1 : dims != 2) || x->size(dims - 1) != K || (self->add != 0) != (paddend != Py_None))
        Py_RETURN_NONE;
    const int64_t M = x->numel() / K;
    if (M < 1 || M > INT32_MAX)
        Py_RETURN_NONE;
    LinearEntry e; // a copy, and a reference to its workspace: the call below runs without the interpreter lock
    THPObjectPtr ws;
    const uint64_t key = (uint64_t)M << 1 | (uint64_t)xd;
    if (!self->last || self->last_key != key)
    {
        const auto known = self->entries->find(key);
        if (known != self->entries->end())
            self->last = &known->second, self->last_key = key; // (stays where it is until the table is cleared)
        else if (!add_entry(self, node, M, xd, &e, &ws))
            return nullptr;
    }
    if (!ws)
        e = *self->last, ws = THPObjectPtr::dup(e.ws);
    const c10::ScalarType yt = e.desc.y_dtype == NNF_B200_F16 ? at::kHalf : at::kFloat;
    const void* bias = nullptr;
    if (paddend != Py_None)
    {
        const at::Tensor* a = plain_cuda(paddend);
        if (!a || a->dim() != 2 || a->size(0) != M || a->size(1) != N || a->scalar_type() != yt)
            Py_RETURN_NONE;
        bias = a->const_data_ptr();
    }
    else
        bias = address_of(self->bias);
    THPObjectPtr out;
    if (pout == Py_None)
    {
        if (lead)
        {
            c10::SmallVector<int64_t, 6> sizes(x->sizes().begin(), x->sizes().end());
            sizes.back() = N;
            out = wrapped_empty(sizes, yt, x->device());
        }
        else
            out = wrapped_empty({M, N}, yt, x->device());
        if (!out)
            return nullptr;
    }
    else
    {
        const at::Tensor* o = plain_cuda(pout);
        if (!o || o->dim() != 2 || o->size(0) != M || o->size(1) != N || o->scalar_type() != yt)
            Py_RETURN_NONE;
        out = THPObjectPtr::dup(pout);
    }
    void* y = THPVariable_Unpack(out.get()).mutable_data_ptr();
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
    const void *px_data = x->const_data_ptr(), *gain = address_of(self->gain);
    nnf_b200_ctx* const ctx = context(self->handle);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = self->fn(ctx, stream, &e.desc, px_data, &self->w, self->has_w2 ? &self->w2 : nullptr, gain, bias, y,
                  e.ws_data, e.ws_bytes);
    Py_END_ALLOW_THREADS
    if (rc != NNF_B200_OK)
        return PyObject_CallFunction(self->check, "i", rc);
    return out.release();
}

// C++ exceptions leave as torch's own bindings would raise them (OutOfMemoryError for an allocation that failed, ...).
template <typename Body>
PyObject* guarded(Body&& body)
{
    try
    {
        return body();
    }
    catch (...)
    {
        torch::translate_exception_to_python(std::current_exception());
        return nullptr;
    }
}

// call(node, x, out, addend) -> tensor or None
PyObject* linear_call(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    if (n != 4)
        return PyErr_Format(PyExc_TypeError, "call(node, x, out, addend)");
    return guarded([&] { return linear_run(reinterpret_cast<LinearCall*>(self), args[0], args[1], args[2], args[3], false); });
}

// call_lead(node, x, wq) -> tensor or None: any leading dimensions; None too when wq is no longer the tensor the node was
// built for.
PyObject* linear_call_lead(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    if (n != 3)
        return PyErr_Format(PyExc_TypeError, "call_lead(node, x, wq)");
    return guarded([&]() -> PyObject* {
        LinearCall* c = reinterpret_cast<LinearCall*>(self);
        if (!THPVariable_Check(args[2]) || THPVariable_Unpack(args[2]).const_data_ptr() != c->w.wq)
            Py_RETURN_NONE;
        return linear_run(c, args[0], args[1], Py_None, Py_None, true);
    });
}

PyObject* linear_new(PyTypeObject* type, PyObject* args, PyObject*)
{
    unsigned long long fn;
    Py_buffer w, w2, handle;
    int add;
    long long N, K;
    PyObject *hobj, *gain, *bias, *check;
    w2.buf = nullptr;
    if (!PyArg_ParseTuple(args, "KOy*z*iOOOLL", &fn, &hobj, &w, &w2, &add, &gain, &bias, &check, &N, &K))
        return nullptr;
    const bool sizes = N > 0 && K > 0 && w.len == (Py_ssize_t)sizeof(nnf_b200_qweight) && (!w2.buf || w2.len == (Py_ssize_t)sizeof(nnf_b200_qweight));
    const bool held = sizes && hold_handle(hobj, &handle);
    auto* entries = held ? new (std::nothrow) std::unordered_map<uint64_t, LinearEntry>() : nullptr;
    LinearCall* c = entries ? reinterpret_cast<LinearCall*>(type->tp_alloc(type, 0)) : nullptr;
    if (!sizes)
        PyErr_SetString(PyExc_ValueError, "weight set or matrix size");
    else if (held && !entries)
        PyErr_NoMemory();
    if (!c)
    {
        delete entries;
        if (held)
            PyBuffer_Release(&handle);
    }
    if (c)
    {
        c->fn = reinterpret_cast<LinearFn>(fn);
        c->handle = handle;
        memcpy(&c->w, w.buf, sizeof c->w);
        c->has_w2 = w2.buf != nullptr;
        if (c->has_w2)
            memcpy(&c->w2, w2.buf, sizeof c->w2);
        c->add = add;
        c->gain = Py_NewRef(gain), c->bias = Py_NewRef(bias), c->check = Py_NewRef(check);
        c->N = N, c->K = K;
        c->entries = entries;
    }
    PyBuffer_Release(&w);
    if (w2.buf)
        PyBuffer_Release(&w2);
    return reinterpret_cast<PyObject*>(c);
}

void linear_dealloc(PyObject* self)
{
    LinearCall* c = reinterpret_cast<LinearCall*>(self);
    PyBuffer_Release(&c->handle);
    Py_XDECREF(c->gain);
    Py_XDECREF(c->bias);
    Py_XDECREF(c->check);
    clear_entries(c);
    delete c->entries;
    Py_TYPE(self)->tp_free(self);
}

PyMethodDef linear_methods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(linear_call)), METH_FASTCALL, nullptr},
    {"call_lead", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(linear_call_lead)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

// ---------------------------------------------------------------------------------------------------- attention

struct AttnCall
{
    PyObject_HEAD
    AttnFn fn;
    AttnWsFn ws_fn;
    Py_buffer handle;
    nnf_b200_attn_desc desc;
    PyObject* ws; // the workspace, kept alive, or None
    void* ws_data;
    size_t ws_bytes;
    PyObject* check;
};

const at::Tensor* half_of(PyObject* o, int64_t numel)
{
    const at::Tensor* t = plain_cuda(o);
    return t && t->scalar_type() == at::kHalf && t->numel() == numel ? t : nullptr;
}

// call(node, q, k_new, v_new, k_cache, v_cache, position, out) -> tensor or None
PyObject* attn_call(PyObject* self, PyObject* const* args, Py_ssize_t n)
{
    if (n != 8)
        return PyErr_Format(PyExc_TypeError, "call(node, q, k_new, v_new, k_cache, v_cache, position, out)");
    return guarded([&]() -> PyObject* {
        PyObject* const* a = args + 1;
        AttnCall* c = reinterpret_cast<AttnCall*>(self);
        const int64_t hd = (int64_t)c->desc.heads * c->desc.head_dim, kd = (int64_t)c->desc.kv_heads * c->desc.head_dim;
        const at::Tensor *q = half_of(a[0], hd), *k = half_of(a[1], kd), *v = half_of(a[2], kd);
        const at::Tensor *kc = half_of(a[3], kd * c->desc.capacity), *vc = half_of(a[4], kd * c->desc.capacity);
        if (!q || !k || !v || !kc || !vc || !PyLong_CheckExact(a[5]))
            Py_RETURN_NONE;
        const long position = PyLong_AsLong(a[5]);
        if (position < 0 || position >= c->desc.capacity)
        {
            PyErr_Clear();
            Py_RETURN_NONE;
        }
        nnf_b200_attn_desc d = c->desc;
        d.position = (int32_t)position;
        nnf_b200_ctx* const ctx = context(c->handle);
        const size_t need = c->ws_fn(ctx, &d);
        if (need > c->ws_bytes)
        {
            THPObjectPtr grown(PyObject_CallMethod(args[0], "_grown", "l", position));
            if (!grown)
                return nullptr;
            if (!is_workspace(grown.get()) || bytes_of(grown.get()) < need)
                Py_RETURN_NONE;
            PyObject* const before = c->ws;
            c->ws = grown.release();
            c->ws_data = const_cast<void*>(address_of(c->ws)), c->ws_bytes = bytes_of(c->ws);
            Py_DECREF(before);
        }
        // (referenced: the call below runs without the interpreter lock)
        THPObjectPtr ws = THPObjectPtr::dup(c->ws);
        const size_t ws_bytes = c->ws_bytes;
        void* const ws_data = c->ws_data;
        THPObjectPtr out;
        if (a[6] == Py_None)
        {
            out = wrapped_empty({1, hd}, at::kHalf, q->device());
            if (!out)
                return nullptr;
        }
        else
        {
            if (!half_of(a[6], hd))
                Py_RETURN_NONE;
            out = THPObjectPtr::dup(a[6]);
        }
        cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
        const void *qp = q->const_data_ptr(), *kp = k->const_data_ptr(), *vp = v->const_data_ptr();
        void *kcp = kc->mutable_data_ptr(), *vcp = vc->mutable_data_ptr();
        void* op = THPVariable_Unpack(out.get()).mutable_data_ptr();
        int rc;
        Py_BEGIN_ALLOW_THREADS
        rc = c->fn(ctx, stream, &d, qp, kp, vp, kcp, vcp, op, need ? ws_data : nullptr, need ? ws_bytes : 0);
        Py_END_ALLOW_THREADS
        if (rc != NNF_B200_OK)
            return PyObject_CallFunction(c->check, "i", rc);
        return out.release();
    });
}

PyObject* attn_new(PyTypeObject* type, PyObject* args, PyObject*)
{
    unsigned long long fn, ws_fn;
    Py_buffer desc, handle;
    PyObject *hobj, *ws, *check;
    if (!PyArg_ParseTuple(args, "KKOy*OO", &fn, &ws_fn, &hobj, &desc, &ws, &check))
        return nullptr;
    if (desc.len != (Py_ssize_t)sizeof(nnf_b200_attn_desc) || !is_workspace(ws))
    {
        PyBuffer_Release(&desc);
        return PyErr_Format(PyExc_ValueError, "descriptor size, or no workspace");
    }
    if (!hold_handle(hobj, &handle))
    {
        PyBuffer_Release(&desc);
        return nullptr;
    }
    AttnCall* c = reinterpret_cast<AttnCall*>(type->tp_alloc(type, 0));
    if (!c)
        PyBuffer_Release(&handle);
    else
    {
        c->fn = reinterpret_cast<AttnFn>(fn), c->ws_fn = reinterpret_cast<AttnWsFn>(ws_fn);
        c->handle = handle;
        memcpy(&c->desc, desc.buf, sizeof c->desc);
        c->ws = Py_NewRef(ws);
        c->ws_data = const_cast<void*>(address_of(ws)), c->ws_bytes = bytes_of(ws);
        c->check = Py_NewRef(check);
    }
    PyBuffer_Release(&desc);
    return reinterpret_cast<PyObject*>(c);
}

void attn_dealloc(PyObject* self)
{
    PyBuffer_Release(&reinterpret_cast<AttnCall*>(self)->handle);
    Py_XDECREF(reinterpret_cast<AttnCall*>(self)->ws);
    Py_XDECREF(reinterpret_cast<AttnCall*>(self)->check);
    Py_TYPE(self)->tp_free(self);
}

PyMethodDef attn_methods[] = {
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(attn_call)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject linear_type = {PyVarObject_HEAD_INIT(nullptr, 0)};
PyTypeObject attn_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host_calls", "Repeated calls of a node, without Python in between.", -1,
                          nullptr, nullptr, nullptr, nullptr, nullptr};
} // namespace

PyMODINIT_FUNC PyInit__host_calls(void)
{
    linear_type.tp_name = "nnfusion_b200._host_calls.LinearCall";
    linear_type.tp_basicsize = sizeof(LinearCall);
    linear_type.tp_flags = Py_TPFLAGS_DEFAULT;
    linear_type.tp_new = linear_new;
    linear_type.tp_dealloc = linear_dealloc;
    linear_type.tp_methods = linear_methods;
    attn_type.tp_name = "nnfusion_b200._host_calls.AttnCall";
    attn_type.tp_basicsize = sizeof(AttnCall);
    attn_type.tp_flags = Py_TPFLAGS_DEFAULT;
    attn_type.tp_new = attn_new;
    attn_type.tp_dealloc = attn_dealloc;
    attn_type.tp_methods = attn_methods;
    if (PyType_Ready(&linear_type) < 0 || PyType_Ready(&attn_type) < 0)
        return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m)
        return nullptr;
    if (PyModule_AddObjectRef(m, "LinearCall", reinterpret_cast<PyObject*>(&linear_type)) < 0 ||
        PyModule_AddObjectRef(m, "AttnCall", reinterpret_cast<PyObject*>(&attn_type)) < 0)
    {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}

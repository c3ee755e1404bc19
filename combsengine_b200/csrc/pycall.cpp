// Native side of the Python mirror's hot calls (kv.py, rope.py): one call per layer checks its tensors, finds the stream
// and enters the C ABI without ctypes' argument conversion.  A decode layer of a small batch takes the GPU five to ten
// microseconds, so this path is what such a step waits for.  Whatever a function here does not take (another type of
// object, a tensor that fails a check) it answers with `kSlow`, and the Python code goes its general way, which
// raises the error.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdint>
#include <vector>

namespace {

constexpr long kSlow = 1 << 20;  // no return code of the library

using AttentionFn = int32_t (*)(void*, int32_t, const void*, const void*, const void*, void*, double, int64_t, void*);
using RopeFn = int32_t (*)(void*, int32_t, const void*, const void*, const void*, const void*, const void*, void*, double, int64_t, void*);
using BeginFn = int32_t (*)(void*, void* const*, const int64_t*, const int64_t*, int32_t, void*);
using PopnFn = int32_t (*)(void*, int64_t, int64_t*);
AttentionFn attention_fn;
RopeFn rope_fn;
BeginFn begin_fn;
PopnFn popn_fn;
PyObject* handle_name;  // "_h"
PyObject* stream_name;  // "cuda_stream"

PyObject* slow() {
    PyErr_Clear();
    return PyLong_FromLong(kSlow);
}
bool as_int(PyObject* o, int64_t* v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLongLong(o);
    return !(*v == -1 && PyErr_Occurred());
}
bool as_ptr(PyObject* o, void** p) {
    if (!PyLong_Check(o)) return false;
    *p = PyLong_AsVoidPtr(o);
    return !PyErr_Occurred();
}
bool as_stream(PyObject* o, void** p) {
    if (o == Py_None) {
        *p = c10::cuda::getCurrentCUDAStream().stream();
        return true;
    }
    PyObject* s = PyObject_GetAttr(o, stream_name);
    const bool ok = s && as_ptr(s, p);
    Py_XDECREF(s);
    return ok;
}
const at::Tensor* tensor(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }
// an operand: contiguous on the GPU, of the arena's type, with as many elements as the step needs
const at::Tensor* operand(PyObject* o, int64_t bf16, int64_t numel) {
    const at::Tensor* t = tensor(o);
    return t && t->is_cuda() && t->is_contiguous() && t->scalar_type() == (bf16 ? at::kBFloat16 : at::kHalf) && t->numel() == numel ? t : nullptr;
}

// The calls of a layer share their tail: q, k, v, out, scale, window, stream, bf16, elements of q, elements of k.
struct Layer {
    const at::Tensor *q, *k, *v;
    at::Tensor made;
    PyObject* out_obj;
    void* out;
    void* stream;
    double scale;
    int64_t window = 0;
    bool parse(PyObject* const* a) {
        int64_t bf16, nq, nkv;
        if (!as_int(a[7], &bf16) || !as_int(a[8], &nq) || !as_int(a[9], &nkv)) return false;
        if (!(q = operand(a[0], bf16, nq)) || !(k = operand(a[1], bf16, nkv)) || !(v = operand(a[2], bf16, nkv))) return false;
        scale = PyFloat_AsDouble(a[4]);
        if (scale == -1.0 && PyErr_Occurred()) return false;
        if (a[5] != Py_None && !as_int(a[5], &window)) return false;
        if (!as_stream(a[6], &stream)) return false;
        out_obj = a[3];
        if (out_obj == Py_None) {
            made = at::empty_like(*q);
            out = made.data_ptr();
        } else {
            const at::Tensor* t = tensor(out_obj);
            if (!t) return false;
            out = t->data_ptr();
        }
        return true;
    }
    PyObject* result(int32_t rc) {
        if (rc != 0) return PyLong_FromLong(rc);
        return made.defined() ? THPVariable_Wrap(made) : Py_NewRef(out_obj);
    }
};

// attention(arena, layer, q, k, v, out, scale, window, stream, bf16, elements of q, of k) -> out, or a code
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void* arena;
    int64_t layer;
    Layer l;
    try {
        if (n != 12 || !as_ptr(a[0], &arena) || !as_int(a[1], &layer) || layer != (int32_t)layer || !l.parse(a + 2)) return slow();
        int32_t rc;
        Py_BEGIN_ALLOW_THREADS
        rc = attention_fn(arena, (int32_t)layer, l.q->data_ptr(), l.k->data_ptr(), l.v->data_ptr(), l.out, l.scale, l.window, l.stream);
        Py_END_ALLOW_THREADS
        return l.result(rc);
    } catch (...) {
        return slow();
    }
}
// attention_rope(arena, layer, rope, norm's address, then as above)
PyObject* attention_rope(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *arena, *rope, *norm;
    int64_t layer;
    Layer l;
    try {
        if (n != 14 || !as_ptr(a[0], &arena) || !as_int(a[1], &layer) || layer != (int32_t)layer || !as_ptr(a[2], &rope) || !as_ptr(a[3], &norm) ||
            !l.parse(a + 4))
            return slow();
        int32_t rc;
        Py_BEGIN_ALLOW_THREADS
        rc = rope_fn(arena, (int32_t)layer, rope, norm, l.q->data_ptr(), l.k->data_ptr(), l.v->data_ptr(), l.out, l.scale, l.window, l.stream);
        Py_END_ALLOW_THREADS
        return l.result(rc);
    } catch (...) {
        return slow();
    }
}
// begin_step(arena, sequences, new tokens, positions or None, stream) -> (code, tokens of the step), or kSlow
PyObject* begin_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void *arena, *stream;
    try {
        if (n != 5 || !as_ptr(a[0], &arena) || !PyList_Check(a[1]) || !PyList_Check(a[2]) || (a[3] != Py_None && !PyList_Check(a[3]))) return slow();
        const Py_ssize_t m = PyList_GET_SIZE(a[1]);
        auto same_length = [&] { return PyList_GET_SIZE(a[1]) == m && PyList_GET_SIZE(a[2]) == m && (a[3] == Py_None || PyList_GET_SIZE(a[3]) == m); };
        if (!same_length()) return slow();
        std::vector<void*> seqs((size_t)m + 1);
        std::vector<int64_t> news((size_t)m + 1), pos((size_t)m + 1);
        int64_t total = 0;
        for (Py_ssize_t i = 0; i < m; i++) {
            PyObject* s = Py_NewRef(PyList_GET_ITEM(a[1], i));
            PyObject* h = PyObject_GetAttr(s, handle_name);  // may run Python code, and that may change the lists
            const bool ok = h && as_ptr(h, &seqs[(size_t)i]);
            Py_XDECREF(h);
            Py_DECREF(s);
            if (!ok || !same_length() || !as_int(PyList_GET_ITEM(a[2], i), &news[(size_t)i])) return slow();
            if (a[3] != Py_None && !as_int(PyList_GET_ITEM(a[3], i), &pos[(size_t)i])) return slow();
            total += news[(size_t)i];
        }
        if (!as_stream(a[4], &stream)) return slow();
        int32_t rc;
        Py_BEGIN_ALLOW_THREADS
        rc = begin_fn(arena, seqs.data(), news.data(), a[3] == Py_None ? nullptr : pos.data(), (int32_t)m, stream);
        Py_END_ALLOW_THREADS
        return Py_BuildValue("(iL)", rc, (long long)total);
    } catch (...) {
        return slow();
    }
}
// popn(sequence, n) -> (code, tokens dropped), or kSlow
PyObject* popn(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void* seq;
    int64_t k, popped = 0;
    if (n != 2 || !as_ptr(a[0], &seq) || !as_int(a[1], &k)) return slow();
    int32_t rc;
    Py_BEGIN_ALLOW_THREADS
    rc = popn_fn(seq, k, &popped);
    Py_END_ALLOW_THREADS
    return Py_BuildValue("(iL)", rc, (long long)popped);
}
// bind(addresses of cbkv_attention, cbkv_attention_rope, cbkv_begin_step, cbkv_popn)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void* p[4];
    if (n != 4) { PyErr_SetString(PyExc_TypeError, "four addresses"); return nullptr; }
    for (int i = 0; i < 4; i++)
        if (!as_ptr(a[i], &p[i])) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "an address is an int"); return nullptr; }
    attention_fn = reinterpret_cast<AttentionFn>(p[0]);
    rope_fn = reinterpret_cast<RopeFn>(p[1]);
    begin_fn = reinterpret_cast<BeginFn>(p[2]);
    popn_fn = reinterpret_cast<PopnFn>(p[3]);
    Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(bind)), METH_FASTCALL, nullptr},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention)), METH_FASTCALL, nullptr},
    {"attention_rope", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(attention_rope)), METH_FASTCALL, nullptr},
    {"begin_step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(begin_step)), METH_FASTCALL, nullptr},
    {"popn", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(popn)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module{PyModuleDef_HEAD_INIT, "_pycall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__pycall(void) {
    handle_name = PyUnicode_InternFromString("_h");
    stream_name = PyUnicode_InternFromString("cuda_stream");
    PyObject* m = PyModule_Create(&module);
    if (m) PyModule_AddIntConstant(m, "SLOW", kSlow);
    return m;
}

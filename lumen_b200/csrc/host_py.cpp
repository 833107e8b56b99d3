// CPython side of the call path (module lumen_b200._host): reads tensors' pointers, shapes and strides and calls the C
// ABI without ctypes structures in between. A call of a compiled function or of an attention / GEMM entry is host work
// of a few microseconds in front of kernels that may take less: descriptors built attribute by attribute in Python took
// 2 us each, three times a kernel launch.
//
// Tensors are duck-typed as everywhere in the package: anything with data_ptr(), shape, stride() and dtype.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <algorithm>
#include <deque>
#include <new>
#include <unordered_map>
#include <vector>

#include "../../include/lumen_b200.h"

namespace {

struct Names {
    PyObject *dtype, *shape, *stride, *data_ptr, *is_cuda, *is_contiguous, *get_device;
} names;
PyObject* code_of = nullptr;     // dict: dtype object or name -> lb_dtype code, filled as dtypes are met
PyObject* code_miss = nullptr;   // callable(dtype) -> code, for the first meeting
PyObject* raise_error = nullptr; // callable(status): raises the library's error
PyObject* raw_stream = nullptr;     // callable(device index) -> torch's current stream handle, or None
PyObject* current_stream = nullptr; // callable() -> the caller's current stream handle

bool dtype_code(PyObject* t, int32_t* out) {
    PyObject* d = PyObject_GetAttr(t, names.dtype);
    if (!d) return false;
    PyObject* c = PyDict_GetItemWithError(code_of, d);  // borrowed
    if (c) {
        *out = (int32_t)PyLong_AsLong(c);
        Py_DECREF(d);
        return true;
    }
    if (PyErr_Occurred()) {
        Py_DECREF(d);
        return false;
    }
    PyObject* made = PyObject_CallOneArg(code_miss, d);
    bool ok = made && PyDict_SetItem(code_of, d, made) == 0;
    if (ok) *out = (int32_t)PyLong_AsLong(made);
    Py_XDECREF(made);
    Py_DECREF(d);
    return ok;
}

bool read_pointer(PyObject* t, void** out) {
    PyObject* p = PyObject_CallMethodNoArgs(t, names.data_ptr);
    if (!p) return false;
    *out = PyLong_AsVoidPtr(p);
    Py_DECREF(p);
    return !PyErr_Occurred();
}

// A sequence of at most LB_MAX_RANK integers (a tuple, as torch and this package give it, or what another framework does).
// Steals the reference.
bool read_longs(PyObject* tuple, int64_t* out, int32_t* count, const char* what) {
    bool ok = false;
    if (tuple && !PyTuple_Check(tuple)) Py_SETREF(tuple, PySequence_Tuple(tuple));
    if (tuple && PyTuple_GET_SIZE(tuple) <= LB_MAX_RANK) {
        *count = (int32_t)PyTuple_GET_SIZE(tuple);
        ok = true;
        for (int32_t k = 0; k < *count; k++) out[k] = PyLong_AsLongLong(PyTuple_GET_ITEM(tuple, k));
        if (PyErr_Occurred()) ok = false;
    } else if (tuple) {
        PyErr_Format(PyExc_TypeError, "a tensor's %s must be at most %d integers", what, LB_MAX_RANK);
    }
    Py_XDECREF(tuple);
    return ok;
}

bool truth(PyObject* b, bool* out) {  // steals b
    if (!b) return false;
    int v = PyObject_IsTrue(b);
    Py_DECREF(b);
    *out = v == 1;
    return v >= 0;
}

bool describe(PyObject* t, lb_tensor* out) {
    PyObject* cuda = PyObject_GetAttr(t, names.is_cuda);
    bool on_gpu = true;
    if (!cuda) PyErr_Clear();  // a tensor type without the attribute answers for itself
    else if (!truth(cuda, &on_gpu)) return false;
    if (!on_gpu) {
        PyErr_SetString(PyExc_ValueError, "expected a CUDA tensor");
        return false;
    }
    int32_t strides = 0;
    if (!dtype_code(t, &out->dtype) || !read_pointer(t, &out->ptr)) return false;
    if (!read_longs(PyObject_GetAttr(t, names.shape), out->shape, &out->rank, "shape")) return false;
    if (!read_longs(PyObject_CallMethodNoArgs(t, names.stride), out->stride, &strides, "stride")) return false;
    if (strides != out->rank) {
        PyErr_SetString(PyExc_TypeError, "a tensor needs as many strides as dimensions");
        return false;
    }
    return true;
}

PyObject* finish(int status) {
    if (status == LB_OK) Py_RETURN_NONE;
    PyObject* r = PyObject_CallFunction(raise_error, "i", status);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "the library reported an error");
    return nullptr;
}

bool wants(Py_ssize_t got, Py_ssize_t want) {
    if (got == want) return true;
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
    return false;
}

// setup(codes, miss, raise, current_stream, raw_stream)
PyObject* setup(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (!wants(n, 5)) return nullptr;
    Py_XSETREF(code_of, Py_NewRef(a[0]));
    Py_XSETREF(code_miss, Py_NewRef(a[1]));
    Py_XSETREF(raise_error, Py_NewRef(a[2]));
    Py_XSETREF(current_stream, Py_NewRef(a[3]));
    Py_XSETREF(raw_stream, Py_NewRef(a[4]));
    Py_RETURN_NONE;
}

bool attn_desc(PyObject* const* a, lb_attn_desc* d) {
    d->scale = (float)PyFloat_AsDouble(a[0]);
    d->causal = (int32_t)PyLong_AsLong(a[1]);
    d->causal_offset = PyLong_AsLongLong(a[2]);
    return !PyErr_Occurred();
}

// attention_fwd(scale, causal, offset, q, k, v, o, lse, stream)
PyObject* attention_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    lb_attn_desc d;
    lb_tensor t[5];
    if (!wants(n, 9) || !attn_desc(a, &d)) return nullptr;
    for (int k = 0; k < 5; k++)
        if (!describe(a[3 + k], &t[k])) return nullptr;
    void* stream = PyLong_AsVoidPtr(a[8]);
    if (PyErr_Occurred()) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = lb_attention_fwd(&d, &t[0], &t[1], &t[2], &t[3], &t[4], stream);
    Py_END_ALLOW_THREADS
    return finish(rc);
}

// attention_bwd_scratch_bytes(scale, causal, offset, q, k)
PyObject* attention_bwd_scratch_bytes(PyObject*, PyObject* const* a, Py_ssize_t n) {
    lb_attn_desc d;
    lb_tensor q, k;
    if (!wants(n, 5) || !attn_desc(a, &d) || !describe(a[3], &q) || !describe(a[4], &k)) return nullptr;
    return PyLong_FromSize_t(lb_attention_bwd_scratch_bytes(&d, &q, &k));
}

// attention_bwd(scale, causal, offset, q, k, v, o, dO, lse, delta, dq_accum or None, dq, dk, dv, scratch pointer, scratch bytes, stream)
PyObject* attention_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
    lb_attn_desc d;
    lb_tensor t[11];
    if (!wants(n, 17) || !attn_desc(a, &d)) return nullptr;
    const bool atomic = a[10] != Py_None;
    for (int k = 0; k < 11; k++)
        if ((k != 7 || atomic) && !describe(a[3 + k], &t[k])) return nullptr;
    void* scratch = PyLong_AsVoidPtr(a[14]);
    const size_t bytes = PyLong_AsSize_t(a[15]);
    void* stream = PyLong_AsVoidPtr(a[16]);
    if (PyErr_Occurred()) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = atomic ? lb_attention_bwd_atomic(&d, &t[0], &t[1], &t[2], &t[3], &t[4], &t[5], &t[6], &t[7], &t[8], &t[9], &t[10], stream)
                : lb_attention_bwd_scratch(&d, &t[0], &t[1], &t[2], &t[3], &t[4], &t[5], &t[6], &t[8], &t[9], &t[10], scratch, bytes, stream);
    Py_END_ALLOW_THREADS
    return finish(rc);
}

// gemm(a, b, out, aux or None, epilogue, kernel, scratch pointer, scratch bytes, stream)
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    lb_tensor ta, tb;
    lb_gemm_out out = {};
    lb_gemm_cfg cfg = {};
    if (!wants(n, 9) || !describe(a[0], &ta) || !describe(a[1], &tb) || !describe(a[2], &out.product)) return nullptr;
    if (a[3] != Py_None && !describe(a[3], &out.aux)) return nullptr;
    out.epilogue = (int32_t)PyLong_AsLong(a[4]);
    cfg.kernel = (int32_t)PyLong_AsLong(a[5]);
    cfg.scratch = PyLong_AsVoidPtr(a[6]);
    cfg.scratch_bytes = (size_t)PyLong_AsUnsignedLongLong(a[7]);
    void* stream = PyLong_AsVoidPtr(a[8]);
    if (PyErr_Occurred()) return nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = lb_gemm(&ta, &tb, &out, &cfg, stream);
    Py_END_ALLOW_THREADS
    return finish(rc);
}

// ---- the calls of one compiled function -----------------------------------------------------------------------------
// The signatures a `lumen_b200.compile`d function has met whose arguments are all tensors, by a hash of the arguments' types,
// dtypes and shapes and of the device: a call costs the same with one signature as with thousands (a cache that grows by a token a
// call). `call(args, stream, device)` finds the one that `args` match, runs its plan and returns its results; it returns None
// when the call needs the general path (an unknown signature, host or strided or foreign arguments).
struct Arg {
    PyObject* type;   // exact type
    PyObject* dtype;  // the dtype attribute
    int32_t rank;
    int64_t shape[LB_MAX_RANK];
};
struct Entry {
    std::vector<Arg> args;  // owns its references
    std::vector<char> torch;  // by argument: a torch tensor, which has to be on the GPU and contiguous
    long device;            // the GPU that the plan's workspace and results live on (-1: the process has one)
    const lb_plan* plan;
    void* workspace;
    std::vector<void*> outputs;
    PyObject *signature, *returned, *keep;  // keep: the last call's arguments, alive until the next call
};
struct CallTable {
    PyObject_HEAD
    std::deque<Entry>* entries;  // references stay valid while other threads add signatures
    std::unordered_multimap<uint64_t, Entry*>* index;
    std::vector<PyObject*>* types;  // the argument types of the entries (held by them): anything else is not looked up
    PyObject* latest;  // the signature object of the latest call
};

void drop(Entry& e) {
    for (Arg& a : e.args) Py_XDECREF(a.type), Py_XDECREF(a.dtype);
    Py_XDECREF(e.signature), Py_XDECREF(e.returned), Py_XDECREF(e.keep);
}
PyObject* table_new(PyTypeObject* type, PyObject*, PyObject*) {
    CallTable* t = (CallTable*)type->tp_alloc(type, 0);
    if (!t) return nullptr;
    t->entries = new (std::nothrow) std::deque<Entry>();
    t->index = new (std::nothrow) std::unordered_multimap<uint64_t, Entry*>();
    t->types = new (std::nothrow) std::vector<PyObject*>();
    t->latest = Py_NewRef(Py_None);
    if (!t->entries || !t->index || !t->types) {
        Py_DECREF(t);
        return PyErr_NoMemory();
    }
    return (PyObject*)t;
}
int table_traverse(CallTable* t, visitproc visit, void* arg) {
    if (t->entries)
        for (Entry& e : *t->entries) {
            Py_VISIT(e.signature);
            Py_VISIT(e.returned);
            Py_VISIT(e.keep);
        }
    Py_VISIT(t->latest);
    return 0;
}
int table_clear(CallTable* t) {
    std::deque<Entry> gone;
    if (t->index) t->index->clear();
    if (t->types) t->types->clear();
    if (t->entries) gone.swap(*t->entries);
    for (Entry& e : gone) drop(e);
    Py_CLEAR(t->latest);
    return 0;
}
void table_dealloc(CallTable* t) {
    PyObject_GC_UnTrack(t);
    table_clear(t);
    delete t->entries;
    delete t->index;
    delete t->types;
    Py_TYPE(t)->tp_free((PyObject*)t);
}

// What a call's argument is looked up by; the references are the caller's (`dtype` is new, `type` borrowed).
bool read_arg(PyObject* x, Arg* out) {
    out->type = (PyObject*)Py_TYPE(x);
    out->dtype = PyObject_GetAttr(x, names.dtype);
    return out->dtype && read_longs(PyObject_GetAttr(x, names.shape), out->shape, &out->rank, "shape");
}
bool hash_args(const Arg* args, size_t count, long device, uint64_t* out) {
    uint64_t h = (uint64_t)device + 0x9e3779b97f4a7c15ull;
    auto mix = [&](uint64_t v) { h = (h ^ v) * 0xff51afd7ed558ccdull, h ^= h >> 32; };
    for (size_t k = 0; k < count; k++) {
        const Py_hash_t d = PyObject_Hash(args[k].dtype);
        if (d == -1 && PyErr_Occurred()) return false;
        mix((uint64_t)(uintptr_t)args[k].type), mix((uint64_t)d), mix((uint64_t)args[k].rank);
        for (int32_t r = 0; r < args[k].rank; r++) mix((uint64_t)args[k].shape[r]);
    }
    *out = h;
    return true;
}

// add(args, torch_flags, device, plan handle, workspace pointer, output pointers, signature, returned)
PyObject* table_add(CallTable* t, PyObject* const* a, Py_ssize_t n) {
    if (!wants(n, 8)) return nullptr;
    if (!PyTuple_Check(a[0]) || !PyTuple_Check(a[1]) || !PyTuple_Check(a[5]) || PyTuple_GET_SIZE(a[0]) != PyTuple_GET_SIZE(a[1])) {
        PyErr_SetString(PyExc_TypeError, "add: tuples of arguments, flags and output pointers");
        return nullptr;
    }
    Entry e = {};
    try {
        e.device = PyLong_AsLong(a[2]);
        e.plan = (const lb_plan*)PyLong_AsVoidPtr(a[3]);
        e.workspace = PyLong_AsVoidPtr(a[4]);
        for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(a[5]); k++) e.outputs.push_back(PyLong_AsVoidPtr(PyTuple_GET_ITEM(a[5], k)));
        bool ok = !PyErr_Occurred();
        for (Py_ssize_t k = 0; ok && k < PyTuple_GET_SIZE(a[0]); k++) {
            e.args.push_back(Arg{});
            ok = read_arg(PyTuple_GET_ITEM(a[0], k), &e.args.back());
            Py_XINCREF(e.args.back().type);
            e.torch.push_back(PyTuple_GET_ITEM(a[1], k) == Py_True);
        }
        uint64_t h = 0;
        if (!ok || !hash_args(e.args.data(), e.args.size(), e.device, &h)) {
            drop(e);
            return nullptr;
        }
        for (const Arg& arg : e.args)
            if (std::find(t->types->begin(), t->types->end(), arg.type) == t->types->end()) t->types->push_back(arg.type);
        t->entries->push_back(e);
        e = {};  // the table's now
        Entry& kept = t->entries->back();
        kept.signature = Py_NewRef(a[6]), kept.returned = Py_NewRef(a[7]);
        t->index->emplace(h, &kept);
    } catch (const std::bad_alloc&) {
        drop(e);
        return PyErr_NoMemory();
    }
    Py_RETURN_NONE;
}

bool same_args(const Arg* got, const Entry& e) {
    for (size_t k = 0; k < e.args.size(); k++) {
        const Arg& want = e.args[k];
        if (got[k].type != want.type || got[k].rank != want.rank) return false;
        for (int32_t r = 0; r < want.rank; r++)
            if (got[k].shape[r] != want.shape[r]) return false;
        if (got[k].dtype != want.dtype) {
            const int same = PyObject_RichCompareBool(got[k].dtype, want.dtype, Py_EQ);
            if (same < 0) PyErr_Clear();
            if (same <= 0) return false;
        }
    }
    return true;
}
// 1: the torch tensor can be read where it is; 0: it cannot (on the host, strided, on another GPU); -1: a Python error
int in_place(PyObject* x, long device) {
    bool yes = false;
    if (!truth(PyObject_GetAttr(x, names.is_cuda), &yes)) return -1;
    if (!yes) return 0;
    if (!truth(PyObject_CallMethodNoArgs(x, names.is_contiguous), &yes)) return -1;
    if (!yes) return 0;
    if (device >= 0) {
        PyObject* g = PyObject_CallMethodNoArgs(x, names.get_device);
        if (!g) return -1;
        const long at = PyLong_AsLong(g);
        Py_DECREF(g);
        if (at != device) return PyErr_Occurred() ? -1 : 0;
    }
    return 1;
}

// The entry that the arguments match, or null (with a Python error set where reading one failed).
Entry* find(CallTable* t, PyObject* args, long device) {
    constexpr Py_ssize_t kMost = 64;
    const Py_ssize_t count = PyTuple_GET_SIZE(args);
    if (count > kMost) return nullptr;
    for (Py_ssize_t k = 0; k < count; k++)
        if (std::find(t->types->begin(), t->types->end(), (PyObject*)Py_TYPE(PyTuple_GET_ITEM(args, k))) == t->types->end()) return nullptr;
    Arg got[kMost];
    Py_ssize_t read = 0;
    bool ok = true;
    for (; ok && read < count; read++) ok = read_arg(PyTuple_GET_ITEM(args, read), &got[read]);
    Entry* found = nullptr;
    uint64_t h = 0;
    if (ok && hash_args(got, (size_t)count, device, &h)) {
        auto range = t->index->equal_range(h);
        for (auto it = range.first; it != range.second && !found; ++it)
            if ((Py_ssize_t)it->second->args.size() == count && it->second->device == device && same_args(got, *it->second)) found = it->second;
    }
    for (Py_ssize_t k = 0; k < read; k++) Py_XDECREF(got[k].dtype);
    return found;
}

// call(args, stream, device): stream 0 means the caller's current stream; `device`: the current device's index, on which the
// signature's memory and the arguments have to be (< 0: the process sees one GPU only)
PyObject* table_call(CallTable* t, PyObject* const* a, Py_ssize_t n) {
    if (!wants(n, 3)) return nullptr;
    PyObject* args = a[0];
    if (!PyTuple_Check(args)) {
        PyErr_SetString(PyExc_TypeError, "call: a tuple of arguments");
        return nullptr;
    }
    void* stream = PyLong_AsVoidPtr(a[1]);
    const long device = PyLong_AsLong(a[2]);
    if (PyErr_Occurred()) return nullptr;
    Entry* entry = find(t, args, device);
    if (!entry) {
        if (PyErr_Occurred()) return nullptr;
        Py_RETURN_NONE;
    }
    Entry& e = *entry;
    PyObject *returned = Py_NewRef(e.returned), *signature = Py_NewRef(e.signature);  // hold the plan and its memory
    const Py_ssize_t count = PyTuple_GET_SIZE(args);
    void* pointers[64];
    int usable = 1;
    bool torch = false;
    for (Py_ssize_t k = 0; usable == 1 && k < count; k++) {
        PyObject* x = PyTuple_GET_ITEM(args, k);
        if (e.torch[k]) torch = true, usable = in_place(x, device);
        if (usable == 1 && !read_pointer(x, &pointers[k])) usable = -1;
    }
    if (usable == 1 && !stream) {
        PyObject* s = torch && raw_stream != Py_None ? PyObject_CallFunction(raw_stream, "l", device < 0 ? 0L : device)
                                                     : PyObject_CallNoArgs(current_stream);
        if (s) stream = PyLong_AsVoidPtr(s);
        Py_XDECREF(s);
        if (PyErr_Occurred()) usable = -1;
    }
    if (usable != 1) {
        Py_DECREF(returned);
        Py_DECREF(signature);
        if (usable < 0) return nullptr;
        Py_RETURN_NONE;
    }
    PyObject* before = e.keep;
    e.keep = Py_NewRef(args);
    const lb_plan* plan = e.plan;
    void* workspace = e.workspace;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = lb_plan_run(plan, workspace, pointers, (int)count, e.outputs.data(), (int)e.outputs.size(), 0, -1, stream);
    Py_END_ALLOW_THREADS
    Py_XDECREF(before);
    Py_XSETREF(t->latest, signature);
    if (rc != LB_OK) {
        Py_DECREF(returned);
        return finish(rc);
    }
    return returned;
}

PyMethodDef table_methods[] = {
    {"add", (PyCFunction)(void (*)(void))table_add, METH_FASTCALL, "adds a signature"},
    {"call", (PyCFunction)(void (*)(void))table_call, METH_FASTCALL, "runs the matching signature's plan, or returns None"},
    {nullptr, nullptr, 0, nullptr},
};
PyMemberDef table_members[] = {
    {"latest", T_OBJECT, offsetof(CallTable, latest), 0, "the signature object of the latest call"},
    {nullptr, 0, 0, 0, nullptr},
};
PyTypeObject table_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyMethodDef methods[] = {
    {"setup", (PyCFunction)(void (*)(void))setup, METH_FASTCALL, "dtype codes and callbacks"},
    {"attention_fwd", (PyCFunction)(void (*)(void))attention_fwd, METH_FASTCALL, "lb_attention_fwd on tensors"},
    {"attention_bwd", (PyCFunction)(void (*)(void))attention_bwd, METH_FASTCALL, "lb_attention_bwd_scratch / lb_attention_bwd_atomic on tensors"},
    {"attention_bwd_scratch_bytes", (PyCFunction)(void (*)(void))attention_bwd_scratch_bytes, METH_FASTCALL, "lb_attention_bwd_scratch_bytes of tensors"},
    {"gemm", (PyCFunction)(void (*)(void))gemm, METH_FASTCALL, "lb_gemm on tensors"},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "the call path of lumen_b200 over the C ABI", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    names.dtype = PyUnicode_InternFromString("dtype");
    names.shape = PyUnicode_InternFromString("shape");
    names.stride = PyUnicode_InternFromString("stride");
    names.data_ptr = PyUnicode_InternFromString("data_ptr");
    names.is_cuda = PyUnicode_InternFromString("is_cuda");
    names.is_contiguous = PyUnicode_InternFromString("is_contiguous");
    names.get_device = PyUnicode_InternFromString("get_device");
    table_type.tp_name = "lumen_b200._host.CallTable";
    table_type.tp_basicsize = sizeof(CallTable);
    table_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
    table_type.tp_new = table_new;
    table_type.tp_dealloc = (destructor)table_dealloc;
    table_type.tp_traverse = (traverseproc)table_traverse;
    table_type.tp_clear = (inquiry)table_clear;
    table_type.tp_methods = table_methods;
    table_type.tp_members = table_members;
    if (PyType_Ready(&table_type) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&table_type);
    if (PyModule_AddObject(m, "CallTable", (PyObject*)&table_type) < 0) {
        Py_DECREF(&table_type);
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}

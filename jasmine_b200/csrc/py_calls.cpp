// The frequent calls of the Python plumbing (jasmine_b200/__init__.py) without ctypes: a tensor is described by reading its fields instead of by
// six calls into Python, the structs live on the stack.  What a call of the small operations costs is the host's part: 21 calls of a
// two-layer model of width 128 took 255 us for 91 us of kernels.
//
// Every function returns the call's status, or None for arguments that it leaves to the Python code: anything but plain dense CUDA tensors of the
// types that a jsm_mat knows (subclasses, wrappers of transforms, other types and ranks) and numbers outside the C types.  The
// library is the one that Python has loaded (bind).
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include "../../include/jasmine_b200.h"

namespace {

struct Library {
    decltype(&jsm_eval_elementwise) eval_elementwise;
    decltype(&jsm_eval_rows) eval_rows;
    decltype(&jsm_dot_f32) dot_f32;
    decltype(&jsm_embedding) embedding;
    decltype(&jsm_attn_prefill) attn_prefill;
    decltype(&jsm_attn_decode) attn_decode;
} L = {};

// a plain dense CUDA tensor: nothing between it and its memory
const at::Tensor* plain(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.layout() != c10::kStrided || !t.is_cuda()) return nullptr;
    constexpr c10::DispatchKeySet known = c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) |
                                          c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA);
    return (t.key_set().raw_repr() & ~known.raw_repr()) == 0 ? &t : nullptr;
}

int type_of(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return JSM_F32;
        case at::kBFloat16: return JSM_BF16;
        case at::kInt: return JSM_I32;
        default: return -1;
    }
}

bool as_mat(PyObject* o, jsm_mat& m) {
    const at::Tensor* t = plain(o);
    if (!t || (t->dim() != 1 && t->dim() != 2)) return false;
    const int type = type_of(*t);
    const int64_t rows = t->dim() == 1 ? 1 : t->size(0), cols = t->size(-1);
    if (type < 0 || rows > INT32_MAX || cols > INT32_MAX) return false;
    m.data = t->mutable_data_ptr();
    m.rows = (int32_t)rows; m.cols = (int32_t)cols;
    m.col_stride = t->stride(-1);
    m.row_stride = t->dim() == 1 ? cols * m.col_stride : t->stride(0);
    m.dtype = type;
    return true;
}
// address of a tensor, or null for None
bool as_pointer(PyObject* o, void*& p) {
    p = nullptr;
    if (o == Py_None) return true;
    const at::Tensor* t = plain(o);
    if (!t) return false;
    p = t->mutable_data_ptr();
    return true;
}
bool as_int(PyObject* o, int& v) {
    if (!PyLong_Check(o)) return false;
    int over = 0;
    const long x = PyLong_AsLongAndOverflow(o, &over);
    v = (int)x;
    return !over && x >= INT32_MIN && x <= INT32_MAX;
}
bool as_float(PyObject* o, float& v) {
    if (PyFloat_Check(o)) v = (float)PyFloat_AS_DOUBLE(o);
    else {
        int i;
        if (!as_int(o, i)) return false;
        v = (float)i;
    }
    return true;
}
// a list or tuple of (op,), (op, index) or (op, number)
bool as_program(PyObject* o, jsm_instr (&p)[JSM_MAX_INSTR], int& n) {
    if (!PyList_Check(o) && !PyTuple_Check(o)) return false;
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(o);
    if (len > JSM_MAX_INSTR) return false;
    n = (int)len;
    for (int k = 0; k < n; ++k) {
        PyObject* e = PySequence_Fast_GET_ITEM(o, k);
        if (!PyTuple_Check(e) || PyTuple_GET_SIZE(e) < 1 || !as_int(PyTuple_GET_ITEM(e, 0), p[k].op)) return false;
        p[k].arg = 0;
        p[k].imm = 0.0f;
        if (PyTuple_GET_SIZE(e) < 2) continue;
        PyObject* a = PyTuple_GET_ITEM(e, 1);
        if (p[k].op == JSM_OP_IMM || p[k].op == JSM_OP_POW ? !as_float(a, p[k].imm) : !as_int(a, p[k].arg)) return false;
    }
    return true;
}
bool as_leaves(PyObject* o, jsm_mat (&m)[JSM_MAX_LEAVES], int& n) {
    if (!PyList_Check(o) && !PyTuple_Check(o)) return false;
    const Py_ssize_t len = PySequence_Fast_GET_SIZE(o);
    if (len > JSM_MAX_LEAVES) return false;
    n = (int)len;
    for (int k = 0; k < n; ++k)
        if (!as_mat(PySequence_Fast_GET_ITEM(o, k), m[k])) return false;
    return true;
}

template <typename Call>
PyObject* status_of(Call call) {
    int s;
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    Py_BEGIN_ALLOW_THREADS
    s = (int)call(stream);
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(s);
}

#define JSM_FAST(name) PyObject* name(PyObject*, PyObject* const* a, Py_ssize_t n_args)
#define JSM_NEED(cond) do { if (!(cond)) Py_RETURN_NONE; } while (0)

JSM_FAST(bind) {  // address of the shared library's handle
    if (n_args != 1) return PyErr_Format(PyExc_TypeError, "bind(handle)");
    void* h = PyLong_AsVoidPtr(a[0]);
    if (PyErr_Occurred()) return nullptr;
    auto find = [&](auto& f, const char* name) { f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(h, name)); return f != nullptr; };
    if (!find(L.eval_elementwise, "jsm_eval_elementwise") || !find(L.eval_rows, "jsm_eval_rows") || !find(L.dot_f32, "jsm_dot_f32") ||
        !find(L.embedding, "jsm_embedding") || !find(L.attn_prefill, "jsm_attn_prefill") || !find(L.attn_decode, "jsm_attn_decode"))
        return PyErr_Format(PyExc_ImportError, "libjasmine_b200: a symbol is missing");
    Py_RETURN_NONE;
}

JSM_FAST(eval_elementwise) {  // instrs, leaves, out
    jsm_instr p[JSM_MAX_INSTR];
    jsm_mat l[JSM_MAX_LEAVES], out;
    int n, nl;
    JSM_NEED(n_args == 3 && as_program(a[0], p, n) && as_leaves(a[1], l, nl) && as_mat(a[2], out));
    return status_of([&](void* st) { return L.eval_elementwise(p, n, l, nl, out, st); });
}

JSM_FAST(eval_rows) {  // kind, axis, instrs, leaves, out, gain, bias, eps
    jsm_instr p[JSM_MAX_INSTR];
    jsm_mat l[JSM_MAX_LEAVES], out;
    int kind, axis, n, nl;
    void *gain, *bias;
    float eps;
    JSM_NEED(n_args == 8 && as_int(a[0], kind) && as_int(a[1], axis) && as_program(a[2], p, n) && as_leaves(a[3], l, nl) && as_mat(a[4], out) &&
             as_pointer(a[5], gain) && as_pointer(a[6], bias) && as_float(a[7], eps));
    return status_of([&](void* st) { return L.eval_rows(kind, axis, p, n, l, nl, (const float*)gain, (const float*)bias, eps, out, st); });
}

JSM_FAST(dot_f32) {  // A, B, out, bias, epilogue, residual
    jsm_mat A, B, out, bias, res;
    int epilogue;
    JSM_NEED(n_args == 6 && as_mat(a[0], A) && as_mat(a[1], B) && as_mat(a[2], out) && (a[3] == Py_None || as_mat(a[3], bias)) && as_int(a[4], epilogue) &&
             (a[5] == Py_None || as_mat(a[5], res)));
    const jsm_mat *pb = a[3] == Py_None ? nullptr : &bias, *pr = a[5] == Py_None ? nullptr : &res;
    return status_of([&](void* st) { return L.dot_f32(A, B, pb, epilogue, pr, out, st); });
}

JSM_FAST(embedding) {  // table, ids, pos_table, positions, out
    void *table, *ids, *pos, *at, *out;
    JSM_NEED(n_args == 5 && as_pointer(a[0], table) && as_pointer(a[1], ids) && as_pointer(a[2], pos) && as_pointer(a[3], at) && as_pointer(a[4], out));
    JSM_NEED(a[0] != Py_None && a[1] != Py_None && a[4] != Py_None);
    const at::Tensor &t = THPVariable_Unpack(a[0]), &i = THPVariable_Unpack(a[1]);
    const int type = type_of(t);
    JSM_NEED(type >= 0 && t.dim() >= 2 && i.dim() >= 1 && t.size(1) <= INT32_MAX && i.size(0) <= INT32_MAX);
    const int T = (int)i.size(0), d = (int)t.size(1);
    return status_of([&](void* st) { return L.embedding(table, pos, (const int32_t*)ids, (const int32_t*)at, out, (jsm_dtype)type, T, d, st); });
}

JSM_FAST(attn_prefill) {  // q, k, v, batch, Hq, Hkv, D, causal, scale, rope, impl, out
    void *q, *k, *v, *rope, *out;
    int batch, hq, hkv, d, causal, impl;
    float scale;
    JSM_NEED(n_args == 12 && as_pointer(a[0], q) && as_pointer(a[1], k) && as_pointer(a[2], v) && as_int(a[3], batch) && as_int(a[4], hq) && as_int(a[5], hkv) &&
             as_int(a[6], d) && as_int(a[7], causal) && as_float(a[8], scale) && as_pointer(a[9], rope) && as_int(a[10], impl) && as_pointer(a[11], out));
    JSM_NEED(a[0] != Py_None && a[1] != Py_None && a[2] != Py_None && a[11] != Py_None && batch > 0);
    const at::Tensor &tq = THPVariable_Unpack(a[0]), &tk = THPVariable_Unpack(a[1]);
    const int type = type_of(tq);
    JSM_NEED(type >= 0 && tq.dim() >= 1 && tk.dim() >= 1 && tq.size(0) <= INT32_MAX && tk.size(0) <= INT32_MAX);
    const int nq = (int)(tq.size(0) / batch), nk = (int)(tk.size(0) / batch);
    return status_of([&](void* st) { return L.attn_prefill(q, k, v, out, (jsm_dtype)type, batch, nq, nk, hq, hkv, d, causal, scale, (const float*)rope, impl, st); });
}

JSM_FAST(attn_decode) {  // q, pool, block_table, context_lens, Hq, Hkv, D, max_context, scale, rope, scratch, out
    void *q, *pool, *table, *lens, *rope, *scratch, *out;
    int hq, hkv, d, most;
    float scale;
    JSM_NEED(n_args == 12 && as_pointer(a[0], q) && as_pointer(a[1], pool) && as_pointer(a[2], table) && as_pointer(a[3], lens) && as_int(a[4], hq) &&
             as_int(a[5], hkv) && as_int(a[6], d) && as_int(a[7], most) && as_float(a[8], scale) && as_pointer(a[9], rope) && as_pointer(a[10], scratch) &&
             as_pointer(a[11], out));
    JSM_NEED(a[0] != Py_None && a[1] != Py_None && a[2] != Py_None && a[3] != Py_None && a[10] != Py_None && a[11] != Py_None);
    const at::Tensor &tq = THPVariable_Unpack(a[0]), &tt = THPVariable_Unpack(a[2]);
    JSM_NEED(tq.dim() >= 1 && tt.dim() >= 2 && tq.size(0) <= INT32_MAX && tt.size(1) <= INT32_MAX);
    const int n = (int)tq.size(0), pages = (int)tt.size(1);
    const int64_t pitch = tq.stride(0);
    return status_of([&](void* st) {
        return L.attn_decode(q, pitch, pool, (const int32_t*)table, pages, (const int32_t*)lens, n, hq, hkv, d, scale, (const float*)rope, most, scratch, out, st);
    });
}

// torch throws for tensors that keep their memory to themselves (sizes or addresses that are not to be read): the Python code meets the same and raises
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    try {
        return F(self, a, n);
    } catch (...) {
        Py_RETURN_NONE;
    }
}

#define JSM_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {JSM_METHOD(bind), JSM_METHOD(eval_elementwise), JSM_METHOD(eval_rows), JSM_METHOD(dot_f32), JSM_METHOD(embedding),
                         JSM_METHOD(attn_prefill), JSM_METHOD(attn_decode), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// torch: the torch whose headers this module has been built with, `<version> <revision>`.  The fields of a tensor are read at their places in that one.
PyMODINIT_FUNC PyInit__native() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch", JSM_TORCH) != 0) Py_CLEAR(m);
    return m;
}

// The host path of the Python front end for the calls that need no explanation: tensors exactly as the entry point
// wants them. Each function here checks that, makes the output, finds the stream and calls the C ABI in one step;
// where anything is not plain — another type, a view that has to be made contiguous, a shape that is an error —
// it returns None having done nothing, and the Python code beside it (luma_b200/high.py, low.py) runs as
// written there, with its conversions and its precise exceptions. Small calls are bound by this path: a decode
// step's two calls (append, attention) took 23 us of interpreter, ctypes and per-argument work for 8 us on the GPU;
// here they take 9, of which 5.5 are the two kernel launches.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <exception>
#include <type_traits>

#include "../../include/flash_attn.h"
#include "../../include/luma_nn_kernels.h"

namespace {

using Tensor = at::Tensor;

// The C ABI's functions by storage type (f32, f16, bf16), with every pointer as void*: the types are made from the
// headers' declarations, so that a changed argument list does not compile here. Addresses come from
// the ctypes handle of the library, so that both front ends drive the same copy of it.
template <class A> struct Erased { using type = A; };
template <class A> struct Erased<A*> { using type = void*; };
template <class A> struct Erased<const A*> { using type = const void*; };
template <class F> struct ErasedFn;
template <class... A> struct ErasedFn<int(A...)> { using type = int (*)(typename Erased<A>::type...); };
#define ERASED(fn) ErasedFn<decltype(fn)>::type
#define SAME(T, ...) static_assert(all_same<T, __VA_ARGS__>, #T)
template <class T, class... U> constexpr bool all_same = (std::is_same_v<T, U> && ...);
using BatchFn = ERASED(flash_attn_f32);
using BatchLseFn = ERASED(flash_attn_f32_lse);
using VarlenFn = ERASED(flash_attn_varlen_f32);
using VarlenTotalFn = ERASED(flash_attn_varlen_f16_total);
using KvFn = ERASED(flash_attn_with_kvcache_f32);
using AppendFn = ERASED(flash_attn_kvcache_append);
using SoftmaxFn = ERASED(luma_softmax_f32);
using ErrorFn = decltype(&flash_attn_last_error);
SAME(BatchFn, ERASED(flash_attn_f16), ERASED(flash_attn_bf16));
SAME(BatchLseFn, ERASED(flash_attn_f16_lse), ERASED(flash_attn_bf16_lse));
SAME(VarlenFn, ERASED(flash_attn_varlen_f16), ERASED(flash_attn_varlen_bf16));
SAME(VarlenTotalFn, ERASED(flash_attn_varlen_bf16_total));
SAME(KvFn, ERASED(flash_attn_with_kvcache_f16), ERASED(flash_attn_with_kvcache_bf16));
SAME(SoftmaxFn, ERASED(luma_softmax_f16), ERASED(luma_softmax_bf16));

struct Library {
    BatchFn batch[3];
    BatchLseFn batch_lse[3];
    VarlenFn varlen[3];
    VarlenTotalFn varlen_total[2];   // f16, bf16: with the row counts of the packed buffers
    KvFn kv[3];
    AppendFn append;
    SoftmaxFn softmax[3];
    ErrorFn last_error;
} lib;
PyObject* g_from_status = nullptr;   // luma_b200.error.from_status

int type_index(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return 0;
        case at::kHalf: return 1;
        case at::kBFloat16: return 2;
        default: return -1;
    }
}

// A plain CUDA tensor (no subclass), dense, on `device` (< 0: any so far).
bool plain(PyObject* o, const Tensor*& t, int& device) {
    if (!THPVariable_CheckExact(o)) return false;
    t = &THPVariable_Unpack(o);
    if (!t->defined() || !t->is_cuda() || t->layout() != at::kStrided || !t->is_contiguous()) return false;
    const int d = t->get_device();
    if (device < 0) device = d;
    return d == device;
}

bool as_int(PyObject* o, int& v) {
    if (!PyLong_CheckExact(o)) return false;
    int overflow = 0;
    const long long x = PyLong_AsLongLongAndOverflow(o, &overflow);
    if (overflow != 0 || x < INT32_MIN || x > INT32_MAX) return false;
    v = (int)x;
    return true;
}

// `None` -> 1 / sqrt(d)
bool as_scale(PyObject* o, int64_t d, float& scale) {
    if (o == Py_None) scale = (float)(1.0 / std::sqrt((double)d));
    else if (PyFloat_CheckExact(o)) scale = (float)PyFloat_AS_DOUBLE(o);
    else return false;
    return true;
}

void* stream_of(int device) { return (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }

bool fits(int64_t v) { return v >= 1 && v <= INT32_MAX; }

// Whether the buffer holds a * b * c * d elements; four ints multiply to 124 bits, which 64 do not hold.
bool holds(const Tensor& t, int64_t a, int64_t b, int64_t c, int64_t d) { return (__int128)a * b * c * d <= (__int128)t.numel(); }

bool head_size_ok(int64_t d) { return d == 32 || d == 64 || d == 128; }

// The library's status as the front end reports it: nullptr with the exception set, or `result`.
PyObject* finish(int code, PyObject* result) {
    if (code == 0) return result;
    Py_XDECREF(result);
    const char* msg = lib.last_error();
    PyObject* r = PyObject_CallFunction(g_from_status, "is", code, msg != nullptr ? msg : "");
    Py_XDECREF(r);
    if (r != nullptr) Py_RETURN_NONE;
    return nullptr;
}

#define PLAIN(cond) \
    if (!(cond)) Py_RETURN_NONE
#define WITHOUT_GIL(stmt)      \
    Py_BEGIN_ALLOW_THREADS     \
    stmt;                      \
    Py_END_ALLOW_THREADS

// attn(q, k, v, scale, start_pos, return_lse) -> o | (o, lse) | None
PyObject* attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 6);
    const Tensor *q, *k, *v;
    int dev = -1, start_pos;
    float scale;
    PLAIN(plain(a[0], q, dev) && plain(a[1], k, dev) && plain(a[2], v, dev) && as_int(a[4], start_pos) && start_pos >= 0);
    PLAIN(a[5] == Py_True || a[5] == Py_False);
    const int ti = type_index(*q);
    PLAIN(ti >= 0 && k->scalar_type() == q->scalar_type() && v->scalar_type() == q->scalar_type());
    PLAIN(q->dim() == 4 && k->dim() == 4 && k->sizes() == v->sizes());
    const int64_t b = q->size(0), sq = q->size(1), hq = q->size(2), d = q->size(3), skv = k->size(1), hkv = k->size(2);
    PLAIN(fits(b) && fits(sq) && fits(skv) && fits(hq) && fits(hkv) && k->size(0) == b && k->size(3) == d && head_size_ok(d) && hq % hkv == 0);
    PLAIN(as_scale(a[3], d, scale));
    Tensor o = at::empty_like(*q);
    void* st = stream_of(dev);
    int code;
    if (a[5] == Py_True) {
        Tensor lse = at::empty({b, hq, sq}, q->options().dtype(at::kFloat));
        WITHOUT_GIL(code = lib.batch_lse[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.data_ptr(), lse.data_ptr<float>(),
                                             (int)b, (int)sq, (int)skv, (int)hq, (int)hkv, (int)d, start_pos, scale, nullptr, st));
        if (code != 0) return finish(code, nullptr);
        PyObject* po = THPVariable_Wrap(std::move(o));
        PyObject* pl = THPVariable_Wrap(std::move(lse));
        PyObject* r = PyTuple_Pack(2, po, pl);
        Py_DECREF(po);
        Py_DECREF(pl);
        return r;
    }
    WITHOUT_GIL(code = lib.batch[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.data_ptr(), (int)b, (int)sq, (int)skv,
                                     (int)hq, (int)hkv, (int)d, start_pos, scale, nullptr, st));
    return finish(code, code == 0 ? THPVariable_Wrap(std::move(o)) : nullptr);
}

// low_attn(q, k, v, o, batch, q_seq_len, kv_seq_len, q_heads, kv_heads, head_size, start_pos, scale, mask, lse) -> True | None
// on the current stream of q's device
PyObject* low_attn(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 14);
    const Tensor *q, *k, *v, *o, *mask = nullptr, *lse = nullptr;
    int dev = -1, x[7];
    float scale;
    PLAIN(plain(a[0], q, dev) && plain(a[1], k, dev) && plain(a[2], v, dev) && plain(a[3], o, dev));
    for (int i = 0; i < 7; ++i) PLAIN(as_int(a[4 + i], x[i]) && x[i] >= (i == 6 ? 0 : 1));
    const int64_t b = x[0], sq = x[1], skv = x[2], hq = x[3], hkv = x[4], d = x[5];
    PLAIN(PyFloat_CheckExact(a[11]) && head_size_ok(d) && hq % hkv == 0);
    scale = (float)PyFloat_AS_DOUBLE(a[11]);
    const int ti = type_index(*q);
    PLAIN(ti >= 0 && k->scalar_type() == q->scalar_type() && v->scalar_type() == q->scalar_type() && o->scalar_type() == q->scalar_type());
    PLAIN(holds(*q, b, sq, hq, d) && holds(*o, b, sq, hq, d) && holds(*k, b, skv, hkv, d) && holds(*v, b, skv, hkv, d));
    if (a[12] != Py_None) PLAIN(plain(a[12], mask, dev) && mask->element_size() == 1 && holds(*mask, b, skv, 1, 1));
    if (a[13] != Py_None) PLAIN(plain(a[13], lse, dev) && lse->scalar_type() == at::kFloat && holds(*lse, b, hq, sq, 1));
    const uint8_t* mp = mask != nullptr ? (const uint8_t*)mask->const_data_ptr() : nullptr;
    void* st = stream_of(dev);
    int code;
    if (lse != nullptr) {
        WITHOUT_GIL(code = lib.batch_lse[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o->data_ptr(), lse->data_ptr<float>(),
                                             x[0], x[1], x[2], x[3], x[4], x[5], x[6], scale, mp, st));
    } else {
        WITHOUT_GIL(code = lib.batch[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o->data_ptr(), x[0], x[1], x[2], x[3], x[4],
                                         x[5], x[6], scale, mp, st));
    }
    if (code != 0) return finish(code, nullptr);
    Py_RETURN_TRUE;
}

// varlen(q, k, v, cu_q, cu_k, max_q, max_k, scale, block_table) -> o | None
PyObject* varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 9);
    const Tensor *q, *k, *v, *cu_q, *cu_k, *table = nullptr;
    int dev = -1, max_q, max_k;
    float scale;
    PLAIN(plain(a[0], q, dev) && plain(a[1], k, dev) && plain(a[2], v, dev) && plain(a[3], cu_q, dev) && plain(a[4], cu_k, dev));
    PLAIN(as_int(a[5], max_q) && as_int(a[6], max_k));
    const int ti = type_index(*q);
    PLAIN(ti >= 0 && k->scalar_type() == q->scalar_type() && v->scalar_type() == q->scalar_type());
    PLAIN(cu_q->scalar_type() == at::kInt && cu_k->scalar_type() == at::kInt && q->dim() == 3 && k->sizes() == v->sizes());
    const int64_t num_seqs = cu_q->numel() - 1, hq = q->size(1), d = q->size(2);
    int64_t block_size = 1, hkv, max_blocks = 0;
    if (a[8] != Py_None) {
        PLAIN(plain(a[8], table, dev) && table->scalar_type() == at::kInt && k->dim() == 4 && num_seqs > 0);
        block_size = k->size(1);
        hkv = k->size(2);
        max_blocks = table->numel() / num_seqs;
    } else {
        PLAIN(k->dim() == 3);
        hkv = k->size(1);
    }
    PLAIN(fits(num_seqs) && fits(hq) && fits(hkv) && fits(block_size) && max_blocks <= INT32_MAX && k->size(-1) == d && head_size_ok(d));
    PLAIN(as_scale(a[7], d, scale));
    Tensor o = at::empty_like(*q);
    void* st = stream_of(dev);
    int code;
    const int* tab = table != nullptr ? table->const_data_ptr<int>() : nullptr;
    const int paged = table != nullptr ? 1 : 0;
    if (ti > 0 && q->size(0) <= INT32_MAX && (paged || k->size(0) <= INT32_MAX)) {
        WITHOUT_GIL(code = lib.varlen_total[ti - 1](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.data_ptr(), cu_q->const_data_ptr<int>(),
                                                    cu_k->const_data_ptr<int>(), tab, (int)num_seqs, max_q, max_k, (int)hq, (int)hkv, (int)d, (int)block_size,
                                                    (int)max_blocks, paged, scale, (int)q->size(0), paged ? 0 : (int)k->size(0), st));
    } else {
        WITHOUT_GIL(code = lib.varlen[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.data_ptr(), cu_q->const_data_ptr<int>(),
                                          cu_k->const_data_ptr<int>(), tab, (int)num_seqs, max_q, max_k, (int)hq, (int)hkv, (int)d, (int)block_size,
                                          (int)max_blocks, paged, scale, st));
    }
    return finish(code, code == 0 ? THPVariable_Wrap(std::move(o)) : nullptr);
}

// kvcache(q, k_cache, v_cache, cache_seqlens, block_table, scale) -> o | None
PyObject* kvcache(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 6);
    const Tensor *q, *k, *v, *lens, *table;
    int dev = -1;
    float scale;
    PLAIN(plain(a[0], q, dev) && plain(a[1], k, dev) && plain(a[2], v, dev) && plain(a[3], lens, dev) && plain(a[4], table, dev));
    const int ti = type_index(*q);
    PLAIN(ti >= 0 && k->scalar_type() == q->scalar_type() && v->scalar_type() == q->scalar_type());
    PLAIN(q->dim() == 4 && k->dim() == 4 && k->sizes() == v->sizes() && table->dim() == 2);
    PLAIN(lens->scalar_type() == at::kInt && table->scalar_type() == at::kInt);
    const int64_t b = q->size(0), sq = q->size(1), hq = q->size(2), d = q->size(3), bs = k->size(1), hkv = k->size(2), mb = table->size(1);
    PLAIN(fits(b) && fits(sq) && fits(hq) && fits(hkv) && fits(bs) && fits(mb) && k->size(3) == d && head_size_ok(d));
    PLAIN(table->size(0) == b && lens->numel() == b && as_scale(a[5], d, scale));
    Tensor o = at::empty_like(*q);
    void* st = stream_of(dev);
    int code;
    WITHOUT_GIL(code = lib.kv[ti](q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), o.data_ptr(), table->const_data_ptr<int>(),
                                  lens->const_data_ptr<int>(), (int)b, (int)sq, (int)hq, (int)hkv, (int)d, (int)bs, (int)mb, scale, st));
    return finish(code, code == 0 ? THPVariable_Wrap(std::move(o)) : nullptr);
}

// append(k_new, v_new, k_cache, v_cache, block_tables, context_lens, num_seqs, n_new, kv_heads, head_size, block_size, max_blocks)
// -> True | None, on the current stream of k_new's device
PyObject* append(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 12);
    const Tensor *kn, *vn, *kc, *vc, *table, *lens;
    int dev = -1, x[6];
    PLAIN(plain(a[0], kn, dev) && plain(a[1], vn, dev) && plain(a[2], kc, dev) && plain(a[3], vc, dev) && plain(a[4], table, dev) && plain(a[5], lens, dev));
    for (int i = 0; i < 6; ++i) PLAIN(as_int(a[6 + i], x[i]) && x[i] >= 1);
    PLAIN(holds(*kn, x[0], x[1], x[2], x[3]) && holds(*vn, x[0], x[1], x[2], x[3]) && table->scalar_type() == at::kInt && lens->scalar_type() == at::kInt);
    void* st = stream_of(dev);
    int code;
    WITHOUT_GIL(code = lib.append(kn->const_data_ptr(), vn->const_data_ptr(), kc->data_ptr(), vc->data_ptr(), table->const_data_ptr<int>(),
                                  lens->const_data_ptr<int>(), x[0], x[1], x[2], x[3], (int)kn->element_size(), x[4], x[5], st));
    if (code != 0) return finish(code, nullptr);
    Py_RETURN_TRUE;
}

// softmax(x) -> y | None
PyObject* softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
    PLAIN(n == 1);
    const Tensor* x;
    int dev = -1;
    PLAIN(plain(a[0], x, dev));
    const int ti = type_index(*x);
    PLAIN(ti >= 0 && x->dim() >= 1 && fits(x->size(-1)) && x->numel() > 0);
    Tensor y = at::empty_like(*x);
    void* st = stream_of(dev);
    int code;
    WITHOUT_GIL(code = lib.softmax[ti](x->const_data_ptr(), y.data_ptr(), (long long)(x->numel() / x->size(-1)), (int)x->size(-1), st));
    return finish(code, code == 0 ? THPVariable_Wrap(std::move(y)) : nullptr);
}

// No C++ exception crosses into the interpreter: an allocation that fails in torch comes back as None, and the
// Python path raises what it always raised.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    try {
        return F(self, a, n);
    } catch (const std::exception&) {
        Py_RETURN_NONE;
    }
}

// bind(from_status, addresses): the C ABI's functions in the order of `Library`
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    const Py_ssize_t want = sizeof(Library) / sizeof(void*);
    if (n != 2 || !PyTuple_Check(a[1]) || PyTuple_GET_SIZE(a[1]) != want) {
        PyErr_SetString(PyExc_TypeError, "bind(from_status, addresses)");
        return nullptr;
    }
    void* at[sizeof(Library) / sizeof(void*)];
    for (Py_ssize_t i = 0; i < want; ++i) {
        at[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(a[1], i));
        if (at[i] == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
            return nullptr;
        }
    }
    static_assert(sizeof(void*) == sizeof(BatchFn), "function and data addresses have one size");
    std::memcpy(&lib, at, sizeof(lib));
    Py_INCREF(a[0]);
    Py_XSETREF(g_from_status, a[0]);
    Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast() {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(static_cast<PyObject* (*)(PyObject*, PyObject* const*, Py_ssize_t)>(F)));
}

PyMethodDef methods[] = {
    {"bind", fast<bind>(), METH_FASTCALL, nullptr},
    {"attn", fast<guarded<attn>>(), METH_FASTCALL, nullptr},
    {"low_attn", fast<guarded<low_attn>>(), METH_FASTCALL, nullptr},
    {"varlen", fast<guarded<varlen>>(), METH_FASTCALL, nullptr},
    {"kvcache", fast<guarded<kvcache>>(), METH_FASTCALL, nullptr},
    {"append", fast<guarded<append>>(), METH_FASTCALL, nullptr},
    {"softmax", fast<guarded<softmax>>(), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }

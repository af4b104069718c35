// Native step calls for the Python layer: unpacks the tensors of one decode step and calls the C ABI.
//
// A ctypes call with forty arguments costs about 20 us of host time (one conversion object per pointer, stride
// and size), more than the kernels of a short decode step take; here a step is one METH_FASTCALL function that
// reads pointers and strides from the tensors directly.  A `plan` (capsule) holds what does not change between
// steps: the cache descriptor, the parameters and the addresses of the engine's preallocated buffers.
//
// A call returns 0 (done), 1 (the tensors are not in a form the native path takes: the caller prepares them and
// calls again through the general path) or a negative FQ_ERR_* code.  What torch throws on the way (a tensor without storage
// has no address) becomes a Python exception.
#include <Python.h>

#include <atomic>
#include <cstring>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/flashquest_b200.h"

namespace {

struct Plan {
    int kind;                       // 4, 8: fq_int4_cache; 3: fq_turbo_cache
    fq_int4_cache c4;
    fq_turbo_cache c3;
    fq_decode_params prm;
    int device, cache_dtype, n_layers;
    float* scores; int64_t sc_sl;
    int32_t* compact; int64_t cp_sl;
    char* O; int64_t o_sl;          // bytes
    float* lse; int64_t lse_sl;
    char* ws; size_t ws_sl, ws_bytes;
    char* scratch; size_t scratch_sl, scratch_bytes;
    char *q_rot, *k_rot, *v_rot; int64_t qr_sl, kr_sl;     // (bytes between layers) rotated q / k and cast v of the patched forward, dense, cache dtype
    float* retention;               // (n_layers, H_q): written by the patched forward from the head pattern
    std::atomic<unsigned long long> launches{0};           // kernels that step() and forward() have launched
};

const char* kPlanName = "flashquest_b200.plan";

void free_plan(PyObject* cap) { delete static_cast<Plan*>(PyCapsule_GetPointer(cap, kPlanName)); }

Plan* plan_of(PyObject* o) { return static_cast<Plan*>(PyCapsule_GetPointer(o, kPlanName)); }

inline void* as_ptr(PyObject* o) { return reinterpret_cast<void*>(PyLong_AsUnsignedLongLong(o)); }

int dtype_of(const at::Tensor& t) {
    switch (t.scalar_type()) {
        case at::kHalf: return FQ_F16;
        case at::kBFloat16: return FQ_BF16;
        case at::kFloat: return FQ_F32;
        default: return -1;
    }
}

inline const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// on the GPU whose buffers the plan or cache holds: an address of another one would be read there
inline bool on_device(const at::Tensor& t, int device) { return t.is_cuda() && t.get_device() == device; }

// every row of a 16-bit tensor on a 16-byte boundary
bool rows_aligned(const at::Tensor& t) {
    if (reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
    for (int64_t i = 0; i + 1 < t.dim(); ++i)
        if (t.stride(i) % 8) return false;
    return true;
}

// equal strides wherever a stride is used: that of an axis of length 1 can be anything, also after contiguous()
bool same_layout(const at::Tensor& a, const at::Tensor& b) {
    if (a.sizes() != b.sizes()) return false;
    for (int64_t i = 0; i < a.dim(); ++i)
        if (a.size(i) != 1 && a.stride(i) != b.stride(i)) return false;
    return true;
}

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }

// The native calls run without the GIL, as ctypes calls do: a launch blocks while the stream's queue is full, and other
// Python threads go on meanwhile.  What comes from Python objects has been read before.
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

struct CountLaunches {
    Plan* plan;
    const unsigned long long before = fq_launches();
    explicit CountLaunches(Plan* p) : plan(p) {}
    ~CountLaunches() { plan->launches.fetch_add(fq_launches() - before, std::memory_order_relaxed); }
};

// plan(kind, cache_desc, params, device, n_layers, scores, sc_sl, compact, cp_sl, O, o_sl_bytes, lse, lse_sl,
//      ws, ws_sl, ws_bytes, scratch, scratch_sl, scratch_bytes, q_rot, qr_sl_bytes, k_rot, v_rot, kr_sl_bytes, retention):
// addresses and sizes as integers.  Every buffer has a part for each layer: layers of one cache may run on different streams.
PyObject* make_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 25) { PyErr_SetString(PyExc_TypeError, "plan() takes 25 arguments"); return nullptr; }
    Plan* p = new Plan();
    p->kind = static_cast<int>(PyLong_AsLong(a[0]));
    if (p->kind == 3) { p->c3 = *static_cast<const fq_turbo_cache*>(as_ptr(a[1])); p->cache_dtype = p->c3.kv_dtype; }
    else { p->c4 = *static_cast<const fq_int4_cache*>(as_ptr(a[1])); p->cache_dtype = p->c4.kv_dtype; }
    p->prm = *static_cast<const fq_decode_params*>(as_ptr(a[2]));
    p->device = static_cast<int>(PyLong_AsLong(a[3]));
    p->n_layers = static_cast<int>(PyLong_AsLong(a[4]));
    p->scores = static_cast<float*>(as_ptr(a[5])); p->sc_sl = PyLong_AsLongLong(a[6]);
    p->compact = static_cast<int32_t*>(as_ptr(a[7])); p->cp_sl = PyLong_AsLongLong(a[8]);
    p->O = static_cast<char*>(as_ptr(a[9])); p->o_sl = PyLong_AsLongLong(a[10]);
    p->lse = static_cast<float*>(as_ptr(a[11])); p->lse_sl = PyLong_AsLongLong(a[12]);
    p->ws = static_cast<char*>(as_ptr(a[13])); p->ws_sl = PyLong_AsSize_t(a[14]); p->ws_bytes = PyLong_AsSize_t(a[15]);
    p->scratch = static_cast<char*>(as_ptr(a[16])); p->scratch_sl = PyLong_AsSize_t(a[17]); p->scratch_bytes = PyLong_AsSize_t(a[18]);
    p->q_rot = static_cast<char*>(as_ptr(a[19])); p->qr_sl = PyLong_AsLongLong(a[20]);
    p->k_rot = static_cast<char*>(as_ptr(a[21])); p->v_rot = static_cast<char*>(as_ptr(a[22])); p->kr_sl = PyLong_AsLongLong(a[23]);
    p->retention = static_cast<float*>(as_ptr(a[24]));
    if (PyErr_Occurred()) { delete p; return nullptr; }
    return PyCapsule_New(p, kPlanName, free_plan);
    END_HANDLE_TH_ERRORS
}

int run_layer(const Plan* p, int layer, int seen, const void* k, const void* v, int64_t sb, int64_t sh, int64_t ss, int n_new,
              const void* q, int q_dtype, int64_t q_sb, int64_t q_sh, const fq_decode_params* prm, void* stream) {
    float* sc = p->scores + layer * p->sc_sl;
    int32_t* cp = p->compact + layer * p->cp_sl;
    char* O = p->O + layer * p->o_sl;
    float* lse = p->lse + layer * p->lse_sl;
    char* ws = p->ws + static_cast<size_t>(layer) * p->ws_sl;
    if (p->kind == 3)
        return fq_decode_layer_turbo(&p->c3, layer, seen, k, v, sb, sh, ss, n_new, q, q_dtype, q_sb, q_sh, prm, sc, cp,
                                     p->scratch + static_cast<size_t>(layer) * p->scratch_sl, p->scratch_bytes, O, lse, ws, p->ws_bytes, stream);
    if (p->kind == 8)
        return fq_decode_layer_int8(&p->c4, layer, seen, k, v, sb, sh, ss, n_new, q, q_dtype, q_sb, q_sh, prm, sc, cp,
                                    O, lse, ws, p->ws_bytes, stream);
    return fq_decode_layer_int4(&p->c4, layer, seen, k, v, sb, sh, ss, n_new, q, q_dtype, q_sb, q_sh, prm, sc, cp,
                                O, lse, ws, p->ws_bytes, stream);
}

// step(plan, layer, seen, k, v, q, params | 0): k, v (B,H_kv,n,D) of the cache's dtype, q (B,H_q,1,D) or (B,H_q,D)
PyObject* step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "step() takes 7 arguments"); return nullptr; }
    Plan* p = plan_of(a[0]);
    if (!p) return nullptr;
    const int layer = static_cast<int>(PyLong_AsLong(a[1])), seen = static_cast<int>(PyLong_AsLong(a[2]));
    const at::Tensor *k = tensor_of(a[3]), *v = tensor_of(a[4]), *q = tensor_of(a[5]);
    const fq_decode_params* prm = static_cast<const fq_decode_params*>(as_ptr(a[6]));
    if (PyErr_Occurred()) return nullptr;
    if (!k || !v || !q) return PyLong_FromLong(1);
    const int B = p->kind == 3 ? p->c3.B : p->c4.B, Hkv = p->kind == 3 ? p->c3.Hkv : p->c4.Hkv, D = p->kind == 3 ? p->c3.D : p->c4.D;
    const int Hq = p->prm.Hq;
    const int qd = static_cast<int>(q->dim());
    const bool ok = k->dim() == 4 && v->dim() == 4 && (qd == 3 || (qd == 4 && q->size(2) == 1)) && on_device(*k, p->device) && on_device(*v, p->device) && on_device(*q, p->device) &&
                    dtype_of(*k) == p->cache_dtype && dtype_of(*v) == p->cache_dtype && dtype_of(*q) >= 0 &&
                    same_layout(*k, *v) && k->size(0) == B && k->size(1) == Hkv && k->size(3) == D &&
                    k->stride(3) == 1 && q->size(0) == B && q->size(1) == Hq && q->size(qd - 1) == D && q->stride(qd - 1) == 1 &&
                    (p->kind != 3 || ((Hq == 1 || q->stride(1) == D) && (B == 1 || q->stride(0) == static_cast<int64_t>(Hq) * D)));
    // the INT8 append takes 16-byte aligned rows only (the other two refuse the rest themselves)
    if (!ok || (p->kind == 8 && k->size(2) > 0 && !(rows_aligned(*k) && rows_aligned(*v)))) return PyLong_FromLong(1);
    const int64_t q_sb = p->kind == 3 ? static_cast<int64_t>(Hq) * D : q->stride(0), q_sh = p->kind == 3 ? D : q->stride(1);
    const fq_decode_params par = prm ? *prm : p->prm;
    int rc;
    {
        const NoGil released;
        const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(p->device));
        const CountLaunches counted(p);
        rc = run_layer(p, layer, seen, k->data_ptr(), v->data_ptr(), k->stride(0), k->stride(1), k->stride(2), static_cast<int>(k->size(2)),
                       q->data_ptr(), dtype_of(*q), q_sb, q_sh, &par, stream_of(p->device));
    }
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// forward(plan, layer, seen, q, k, v, cos, sin, params | 0, pattern | None): one new token of the patched attention forward.
// q (B,1,H_q*D), k, v (B,1,H_kv*D): the projections as the linears return them; cos, sin (B or 1,1,D) of the same dtype;
// pattern (H_kv,) bool, read by the launch: retrieval heads keep the parameters' retention, streaming heads 0.
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10) { PyErr_SetString(PyExc_TypeError, "forward() takes 10 arguments"); return nullptr; }
    Plan* p = plan_of(a[0]);
    if (!p) return nullptr;
    const int layer = static_cast<int>(PyLong_AsLong(a[1])), seen = static_cast<int>(PyLong_AsLong(a[2]));
    const at::Tensor* t[5];
    for (int i = 0; i < 5; ++i) t[i] = tensor_of(a[3 + i]);
    const fq_decode_params* prm = static_cast<const fq_decode_params*>(as_ptr(a[8]));
    if (PyErr_Occurred()) return nullptr;
    const int B = p->kind == 3 ? p->c3.B : p->c4.B, Hkv = p->kind == 3 ? p->c3.Hkv : p->c4.Hkv, D = p->kind == 3 ? p->c3.D : p->c4.D;
    const int Hq = p->prm.Hq;
    const int dt = t[0] ? dtype_of(*t[0]) : -1;
    // outside the rotary launch's dtypes and sizes the caller's general path says what is not supported
    if ((dt != FQ_F16 && dt != FQ_BF16) || (p->cache_dtype != FQ_F16 && p->cache_dtype != FQ_BF16) || D > 128 || D % 2) return PyLong_FromLong(1);
    for (int i = 0; i < 5; ++i) {
        if (!t[i] || !on_device(*t[i], p->device) || dtype_of(*t[i]) != dt || t[i]->dim() != 3 || t[i]->size(1) != 1 || t[i]->stride(2) != 1) return PyLong_FromLong(1);
        const int64_t width = i == 0 ? static_cast<int64_t>(Hq) * D : i < 3 ? static_cast<int64_t>(Hkv) * D : D;
        if (t[i]->size(2) != width || !(t[i]->size(0) == B || (i >= 3 && t[i]->size(0) == 1))) return PyLong_FromLong(1);
    }
    const at::Tensor* pat = a[9] == Py_None ? nullptr : tensor_of(a[9]);
    if (a[9] != Py_None && (!pat || !on_device(*pat, p->device) || pat->scalar_type() != at::kBool || pat->dim() != 1 || pat->size(0) != Hkv))
        return PyLong_FromLong(1);
    const int64_t cs = t[3]->size(0) == 1 ? 0 : t[3]->stride(0), ss = t[4]->size(0) == 1 ? 0 : t[4]->stride(0);
    fq_decode_params par = prm ? *prm : p->prm;
    float* ret = p->retention + static_cast<int64_t>(layer) * Hq;
    if (pat) par.retention_per_head = ret;
    int rc;
    {
        const NoGil released;
        const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(p->device));
        const CountLaunches counted(p);
        void* st = stream_of(p->device);
        char *q_rot = p->q_rot + layer * p->qr_sl, *k_rot = p->k_rot + layer * p->kr_sl, *v_rot = p->v_rot + layer * p->kr_sl;
        rc = fq_rope_qkv_pattern(t[0]->data_ptr(), t[0]->stride(0), t[1]->data_ptr(), t[1]->stride(0), t[2]->data_ptr(), t[2]->stride(0), dt,
                         t[3]->data_ptr(), cs, t[4]->data_ptr(), ss, B, Hq, Hkv, D, q_rot, k_rot, v_rot, p->cache_dtype,
                                 pat ? static_cast<const uint8_t*>(pat->data_ptr()) : nullptr, pat ? pat->stride(0) : 0, par.retention, ret, st);
        if (rc == 0)
            rc = run_layer(p, layer, seen, k_rot, v_rot, static_cast<int64_t>(Hkv) * D, D, D, 1, q_rot, p->cache_dtype,
                           static_cast<int64_t>(Hq) * D, D, &par, st);
    }
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// append(kv_bits, cache descriptor, device, layer, seen, k, v): k, v (B,H_kv,n,D) of the cache's dtype
PyObject* append(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) { PyErr_SetString(PyExc_TypeError, "append() takes 7 arguments"); return nullptr; }
    const int kind = static_cast<int>(PyLong_AsLong(a[0])), device = static_cast<int>(PyLong_AsLong(a[2]));
    const void* desc = as_ptr(a[1]);
    const int layer = static_cast<int>(PyLong_AsLong(a[3])), seen = static_cast<int>(PyLong_AsLong(a[4]));
    const at::Tensor *k = tensor_of(a[5]), *v = tensor_of(a[6]);
    if (PyErr_Occurred()) return nullptr;
    const auto* c3 = static_cast<const fq_turbo_cache*>(desc);
    const auto* c4 = static_cast<const fq_int4_cache*>(desc);
    const int B = kind == 3 ? c3->B : c4->B, Hkv = kind == 3 ? c3->Hkv : c4->Hkv, D = kind == 3 ? c3->D : c4->D;
    const int dt = kind == 3 ? c3->kv_dtype : c4->kv_dtype;
    if (!k || !v || (dt != FQ_F16 && dt != FQ_BF16) || k->dim() != 4 || !on_device(*k, device) || !on_device(*v, device) ||
        dtype_of(*k) != dt || dtype_of(*v) != dt || !same_layout(*k, *v) ||
        k->size(0) != B || k->size(1) != Hkv || k->size(3) != D || k->stride(3) != 1 || k->size(2) < 1)
        return PyLong_FromLong(1);
    const int nn = static_cast<int>(k->size(2));
    int rc;
    {
        const NoGil released;
        const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));
        void* st = stream_of(device);
        rc = kind == 3 ? fq_append_kv_turbo(c3, layer, seen, k->data_ptr(), v->data_ptr(), k->stride(0), k->stride(1), k->stride(2), nn, st)
                       : fq_append_kv_int4(c4, layer, seen, k->data_ptr(), v->data_ptr(), k->stride(0), k->stride(1), k->stride(2), nn, st);
    }
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// addresses(tensors, known): the tensors' addresses packed into bytes; `known` itself where it holds the same ones
PyObject* addresses(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    constexpr Py_ssize_t MAX = 16;
    if (n != 2 || !PyTuple_Check(a[0]) || PyTuple_GET_SIZE(a[0]) > MAX) { PyErr_SetString(PyExc_TypeError, "addresses() takes a tuple of up to 16 tensors and bytes"); return nullptr; }
    const void* at[MAX];
    const Py_ssize_t count = PyTuple_GET_SIZE(a[0]), size = count * static_cast<Py_ssize_t>(sizeof(void*));
    for (Py_ssize_t i = 0; i < count; ++i) {
        const at::Tensor* t = tensor_of(PyTuple_GET_ITEM(a[0], i));
        if (!t) { PyErr_SetString(PyExc_TypeError, "addresses() takes tensors"); return nullptr; }
        at[i] = t->data_ptr();
    }
    if (PyBytes_Check(a[1]) && PyBytes_GET_SIZE(a[1]) == size && std::memcmp(PyBytes_AS_STRING(a[1]), at, size) == 0) return Py_NewRef(a[1]);
    return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(at), size);
    END_HANDLE_TH_ERRORS
}

// launches() of the calling thread, launches(plan) of the plan's calls
PyObject* launches(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n == 0) return PyLong_FromUnsignedLongLong(fq_launches());
    const Plan* p = plan_of(a[0]);
    return p ? PyLong_FromUnsignedLongLong(p->launches.load(std::memory_order_relaxed)) : nullptr;
}

PyMethodDef kMethods[] = {
    {"launches", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(launches)), METH_FASTCALL, nullptr},
    {"addresses", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(addresses)), METH_FASTCALL, nullptr},
    {"append", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(append)), METH_FASTCALL, nullptr},
    {"plan", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(make_plan)), METH_FASTCALL, nullptr},
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(step)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(forward)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fq_bind", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fq_bind(void) { return PyModule_Create(&kModule); }

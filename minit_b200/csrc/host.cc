// Host side of the hot module calls (CPython extension minit_b200._host): argument checks, output allocation, workspace
// look-up and the call into the C ABI, without the Python frames around them.
//
// A decode linear takes 6 us on the GPU and its Python wrapper took 18 us per call (device context, stream object, five
// tensors' properties, a 17-argument ctypes call), so a program of single small calls waited for the host.
//
// Every function takes the plain case only -- dense CUDA tensors of exactly torch.Tensor, no active mode or transform, shapes
// and types that the Python wrapper would accept, a workspace that is already large enough, status MT_OK -- and returns None
// for anything else: the wrapper then runs its own checks and call, which raise or allocate as they always did.  Nothing is
// kept between calls but the tables of workspaces, which belong to the wrappers.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <cmath>
#include "../../include/minit_b200.h"

namespace {

PyObject* g_workspaces = nullptr;       // (device index, stream) -> uint8 tensor: linears
PyObject* g_att_workspaces = nullptr;   // the same for attention_decode

const c10::DispatchKeySet& refused_keys() {
    static const c10::DispatchKeySet keys({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::FuncTorchBatched,
                                           c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                           c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::Functionalize,
                                           c10::DispatchKey::Batched, c10::DispatchKey::Conjugate, c10::DispatchKey::Negative,
                                           c10::DispatchKey::ZeroTensor});
    return keys;
}

bool modes_active() {
    return at::impl::PythonTorchFunctionTLS::stack_len() > 0 || c10::impl::tls_local_dispatch_key_set().included_.has_any(refused_keys());
}

// One call's tensors: all dense, contiguous, on one device.
struct Call {
    c10::DeviceIndex dev = -1;
    bool ok = !modes_active();

    const at::Tensor* tensor(PyObject* o) {
        if (!ok || !THPVariable_CheckExact(o)) { ok = false; return nullptr; }
        const at::Tensor& t = THPVariable_Unpack(o);
        if (!t.defined() || !t.is_cuda() || t.layout() != c10::kStrided || !t.has_storage() || t.key_set().has_any(refused_keys()) || !t.is_contiguous()) {
            ok = false;
            return nullptr;
        }
        if (dev < 0) dev = t.get_device();
        else if (dev != t.get_device()) ok = false;
        return &t;
    }
    const at::Tensor* optional(PyObject* o) { return o == Py_None ? nullptr : tensor(o); }
    void need(bool c) { ok = ok && c; }
};

void* ptr(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
bool is(const at::Tensor& t, c10::ScalarType s) { return t.scalar_type() == s; }
int dtype_code(const at::Tensor& t) { return is(t, at::kHalf) ? MT_F16 : is(t, at::kBFloat16) ? MT_BF16 : -1; }

// x [*ms, K] times a GPTQ weight: the contract of the Python wrappers' checks.
struct Linear {
    const at::Tensor *x, *qw, *qz, *sc, *bias;
    int64_t m = 0, n = 0, k = 0, g = 0;
    int bits, dtype = -1;
    Linear(Call& c, PyObject* x_, PyObject* qw_, PyObject* qz_, PyObject* sc_, PyObject* bias_, int bits_)
        : x(c.tensor(x_)), qw(c.tensor(qw_)), qz(c.optional(qz_)), sc(c.tensor(sc_)), bias(c.optional(bias_)), bits(bits_) {
        c.need(bits == 4 || bits == 8);
        if (!c.ok) return;
        const int pack = 32 / bits;
        c.need(x->dim() >= 1 && qw->dim() == 2 && sc->dim() == 2 && is(*qw, at::kInt));
        if (!c.ok) return;
        k = x->size(-1); n = qw->size(1); g = sc->size(0);
        dtype = dtype_code(*x);
        c.need(dtype >= 0 && k > 0 && n > 0 && g > 0 && x->numel() > 0 && k == qw->size(0) * pack && sc->size(1) == n && sc->scalar_type() == x->scalar_type());
        if (qz) c.need(qz->dim() == 2 && qz->size(0) == g && qz->size(1) == n / pack && is(*qz, at::kInt));
        if (bias) c.need(bias->dim() == 1 && bias->size(0) == n && bias->scalar_type() == x->scalar_type());
        c.need(n < INT32_MAX && k < INT32_MAX && x->numel() / (k > 0 ? k : 1) < INT32_MAX);
        if (c.ok) m = x->numel() / k;
    }
    at::Tensor result(int64_t cols) const {
        auto sizes = x->sizes().vec();
        sizes.back() = cols;
        return at::empty(sizes, x->options());
    }
};

// The wrapper's workspace of this device and stream, if it is large enough.
at::Tensor workspace(PyObject* table, c10::DeviceIndex dev, cudaStream_t st, size_t need) {
    PyObject* key = Py_BuildValue("(iK)", int(dev), (unsigned long long)(uintptr_t)st);
    if (!key) { PyErr_Clear(); return {}; }
    PyObject* v = PyDict_GetItemWithError(table, key);
    Py_DECREF(key);
    if (!v) { PyErr_Clear(); return {}; }
    if (!THPVariable_CheckExact(v)) return {};
    at::Tensor t = THPVariable_Unpack(v);
    return size_t(t.numel()) >= need ? t : at::Tensor();
}

// fn(stream, workspace) -> status, with the device current and the GIL released
template <typename F>
bool launch(const Call& c, PyObject* table, size_t need, F&& fn) {
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(c.dev).stream();
    at::Tensor ws;
    if (table) {
        ws = workspace(table, c.dev, st, need);
        if (!ws.defined()) return false;
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fn(st, ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? size_t(ws.numel()) : 0);
    Py_END_ALLOW_THREADS
    return rc == MT_OK;
}

long as_long(PyObject* o, Call& c) {
    if (!PyLong_CheckExact(o)) { c.ok = false; return 0; }
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); c.ok = false; }
    c.need(v >= INT32_MIN && v <= INT32_MAX);
    return v;
}

template <typename F>
PyObject* guarded(Py_ssize_t nargs, Py_ssize_t want, F&& body) {
    if (nargs != want) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }
    try {
        Call c;
        at::Tensor out;
        if (c.ok) out = body(c);
        if (out.defined()) return THPVariable_Wrap(std::move(out));
    } catch (...) {      // out of memory and the like: the wrapper meets it again and raises it
        PyErr_Clear();
    }
    Py_RETURN_NONE;
}

struct Guard {           // the call's device is current while it is sized and launched
    c10::cuda::OptionalCUDAGuard g;
    explicit Guard(const Call& c) { g.set_index(c.dev); }
};

// (x, qweight, zeros, scales, groups, bias, bits, flags)
PyObject* qgemm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 8, [&](Call& c) -> at::Tensor {
        const int bits = int(as_long(a[6], c)), flags = int(as_long(a[7], c));
        const Linear l(c, a[0], a[1], a[2], a[3], a[5], bits);
        const at::Tensor* groups = c.optional(a[4]);
        if (c.ok && groups) c.need(groups->dim() == 1 && groups->size(0) == l.k && is(*groups, at::kInt));
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = l.result(l.n);
        const bool done = launch(c, g_workspaces, mt_workspace_bytes(l.m, l.n, l.k, bits), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_qgemm(st, ptr(l.x), (const uint32_t*)ptr(l.qw), (const int32_t*)ptr(groups), (const uint32_t*)ptr(l.qz), ptr(l.sc), ptr(l.bias),
                            out.data_ptr(), l.m, l.n, l.k, l.g, bits, l.dtype, ws, wb, flags);
        });
        return done ? out : at::Tensor();
    });
}

// (x, qweight_sorted, zeros, scales, perm, bias, bits, flags)
PyObject* qgemm_ordered(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 8, [&](Call& c) -> at::Tensor {
        const int bits = int(as_long(a[6], c)), flags = int(as_long(a[7], c));
        const Linear l(c, a[0], a[1], a[2], a[3], a[5], bits);
        const at::Tensor* perm = c.tensor(a[4]);
        if (c.ok) c.need(perm->dim() == 1 && perm->size(0) == l.k && is(*perm, at::kInt));
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = l.result(l.n), scratch;
        if (l.m > 2) scratch = at::empty({l.m, l.k}, l.x->options());
        const bool done = launch(c, g_workspaces, mt_workspace_bytes(l.m, l.n, l.k, bits), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_qgemm_ordered(st, ptr(l.x), (const int32_t*)ptr(perm), scratch.defined() ? scratch.data_ptr() : nullptr, (const uint32_t*)ptr(l.qw),
                                    (const uint32_t*)ptr(l.qz), ptr(l.sc), ptr(l.bias), out.data_ptr(), l.m, l.n, l.k, l.g, bits, l.dtype, ws, wb, flags);
        });
        return done ? out : at::Tensor();
    });
}

// (x, qweight, zeros, scales, groups, residual, bias, bits, flags)
PyObject* qgemm_residual(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 9, [&](Call& c) -> at::Tensor {
        const int bits = int(as_long(a[7], c)), flags = int(as_long(a[8], c));
        const Linear l(c, a[0], a[1], a[2], a[3], a[6], bits);
        const at::Tensor* groups = c.optional(a[4]);
        const at::Tensor* res = c.tensor(a[5]);
        if (c.ok && groups) c.need(groups->dim() == 1 && groups->size(0) == l.k && is(*groups, at::kInt));
        if (c.ok) c.need(res->scalar_type() == l.x->scalar_type() && res->numel() == l.m * l.n);
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = l.result(l.n);
        const bool done = launch(c, g_workspaces, mt_workspace_bytes(l.m, l.n, l.k, bits), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_qgemm_residual(st, ptr(l.x), (const uint32_t*)ptr(l.qw), (const int32_t*)ptr(groups), (const uint32_t*)ptr(l.qz), ptr(l.sc), ptr(l.bias),
                                     ptr(res), out.data_ptr(), l.m, l.n, l.k, l.g, bits, l.dtype, ws, wb, flags, nullptr, 0, 1, 0);
        });
        return done ? out : at::Tensor();
    });
}

// (x, qweight, zeros, scales, bias, bits, flags): gate / up interleaved columns
PyObject* qgemm_swiglu(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 7, [&](Call& c) -> at::Tensor {
        const int bits = int(as_long(a[5], c)), flags = int(as_long(a[6], c));
        const Linear l(c, a[0], a[1], a[2], a[3], a[4], bits);
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = l.result(l.n / 2), scratch;
        if (l.m > 2 || l.n % 128 || (l.k / l.g) % 32) scratch = at::empty({l.m, l.n}, l.x->options());
        const bool done = launch(c, g_workspaces, mt_workspace_bytes(l.m, l.n, l.k, bits), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_qgemm_swiglu(st, ptr(l.x), (const uint32_t*)ptr(l.qw), (const uint32_t*)ptr(l.qz), ptr(l.sc), ptr(l.bias), out.data_ptr(),
                                   scratch.defined() ? scratch.data_ptr() : nullptr, l.m, l.n, l.k, l.g, bits, l.dtype, ws, wb, flags);
        });
        return done ? out : at::Tensor();
    });
}

// (x, qweight, zeros, scales, bias, cos, sin, k_cache, v_cache, query heads, offset, bits, flags)
PyObject* qkv_rope(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 13, [&](Call& c) -> at::Tensor {
        const int64_t hq = as_long(a[9], c), offset = as_long(a[10], c);
        const int bits = int(as_long(a[11], c)), flags = int(as_long(a[12], c));
        const Linear l(c, a[0], a[1], a[2], a[3], a[4], bits);
        const at::Tensor *cs = c.tensor(a[5]), *sn = c.tensor(a[6]), *kc = c.tensor(a[7]), *vc = c.tensor(a[8]);
        if (!c.ok) return {};
        c.need(l.x->dim() == 2 && kc->dim() == 3 && kc->sizes() == vc->sizes() && kc->scalar_type() == l.x->scalar_type() &&
               vc->scalar_type() == l.x->scalar_type() && cs->dim() == 2 && cs->sizes() == sn->sizes() && is(*cs, at::kFloat) && is(*sn, at::kFloat));
        if (!c.ok) return {};
        const int64_t cap = kc->size(0), hkv = kc->size(1), d = kc->size(2);
        c.need(hq > 0 && l.n == (hq + 2 * hkv) * d && cs->size(1) * 2 == d && cap < INT32_MAX && cs->size(0) < INT32_MAX);
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor q = at::empty({l.m, hq, d}, l.x->options()), scratch;
        if (l.m > 2 || d != 128 || (l.k / l.g) % 32) scratch = at::empty({l.m, l.n}, l.x->options());
        const bool done = launch(c, g_workspaces, mt_workspace_bytes(l.m, l.n, l.k, bits), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_qgemm_rope_append(st, ptr(l.x), (const uint32_t*)ptr(l.qw), (const uint32_t*)ptr(l.qz), ptr(l.sc), ptr(l.bias), (const float*)ptr(cs),
                                        (const float*)ptr(sn), q.data_ptr(), ptr(kc), ptr(vc), scratch.defined() ? scratch.data_ptr() : nullptr, l.m, hq, hkv,
                                        d, l.k, l.g, bits, l.dtype, offset, nullptr, cap, cs->size(0), ws, wb, flags);
        });
        return done ? q : at::Tensor();
    });
}

// (q, k_cache, v_cache, offset)
PyObject* attention_decode(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 4, [&](Call& c) -> at::Tensor {
        const int64_t offset = as_long(a[3], c);
        const at::Tensor *q = c.tensor(a[0]), *kc = c.tensor(a[1]), *vc = c.tensor(a[2]);
        if (!c.ok) return {};
        c.need(q->dim() == 3 && kc->dim() == 3 && kc->sizes() == vc->sizes() && kc->scalar_type() == q->scalar_type() &&
               vc->scalar_type() == q->scalar_type() && dtype_code(*q) >= 0 && q->numel() > 0);
        if (!c.ok) return {};
        const int64_t m = q->size(0), hq = q->size(1), d = q->size(2), hkv = kc->size(1);
        c.need(kc->size(2) == d && hkv > 0 && offset >= 0 && offset + m <= kc->size(0) && offset + m < INT32_MAX);
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = at::empty({m, hq * d}, q->options());
        const int len = int(offset + m);
        const bool done = launch(c, g_att_workspaces, mt_attention_workspace_bytes(m, hkv, len), [&](cudaStream_t st, void* ws, size_t wb) {
            return mt_attention_decode(st, ptr(q), ptr(kc), ptr(vc), out.data_ptr(), m, hq, hkv, d, offset, nullptr, len, float(1.0 / std::sqrt(double(d))),
                                       ws, wb, dtype_code(*q));
        });
        return done ? out : at::Tensor();
    });
}

// (q, k_cache, v_cache, offset, offsets): the scratch is the call's own
PyObject* attention(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 5, [&](Call& c) -> at::Tensor {
        const int64_t offset = as_long(a[3], c);
        const at::Tensor *q = c.tensor(a[0]), *kc = c.tensor(a[1]), *vc = c.tensor(a[2]), *offs = c.optional(a[4]);
        if (!c.ok) return {};
        c.need(q->dim() == 4 && kc->dim() == 4 && kc->sizes() == vc->sizes() && kc->scalar_type() == q->scalar_type() &&
               vc->scalar_type() == q->scalar_type() && dtype_code(*q) >= 0 && q->numel() > 0 && kc->numel() > 0);
        if (!c.ok) return {};
        const int64_t b = q->size(0), m = q->size(1), hq = q->size(2), d = q->size(3), cap = kc->size(1), hkv = kc->size(2);
        c.need(kc->size(0) == b && kc->size(3) == d && hq % hkv == 0 && b < INT32_MAX && m < INT32_MAX && hq < INT32_MAX && cap < INT32_MAX && d <= 256);
        if (offs) c.need(offs->dim() == 1 && offs->size(0) == b && is(*offs, at::kInt));
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = at::empty({b, m, hq * d}, q->options()), ws;
        const size_t need = mt_attention_batch_workspace_bytes(m, hq, hkv, d);
        if (need) ws = at::empty({int64_t(need)}, q->options().dtype(at::kByte));
        const bool done = launch(c, nullptr, 0, [&](cudaStream_t st, void*, size_t) {
            return mt_attention_batch(st, ptr(q), ptr(kc), ptr(vc), out.data_ptr(), (const int32_t*)ptr(offs), b, m, hq, hkv, d, offset, cap,
                                      float(1.0 / std::sqrt(double(d))), need ? ws.data_ptr() : nullptr, need, dtype_code(*q));
        });
        return done ? out : at::Tensor();
    });
}

// (x, weight, eps)
PyObject* rms_norm(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    return guarded(nargs, 3, [&](Call& c) -> at::Tensor {
        const at::Tensor *x = c.tensor(a[0]), *w = c.tensor(a[1]);
        c.need(PyFloat_CheckExact(a[2]));
        if (!c.ok) return {};
        c.need(x->dim() >= 1 && w->dim() == 1 && w->size(0) == x->size(-1) && w->scalar_type() == x->scalar_type() && dtype_code(*x) >= 0 && x->numel() > 0);
        if (!c.ok) return {};
        const int64_t h = x->size(-1), rows = x->numel() / h;
        c.need(rows < INT32_MAX && h < INT32_MAX);
        if (!c.ok) return {};
        const Guard guard(c);
        at::Tensor out = at::empty(x->sizes(), x->options());
        const float eps = float(PyFloat_AS_DOUBLE(a[2]));
        const bool done = launch(c, nullptr, 0, [&](cudaStream_t st, void*, size_t) {
            return mt_rms_norm(st, ptr(x), ptr(w), out.data_ptr(), rows, h, eps, dtype_code(*x));
        });
        return done ? out : at::Tensor();
    });
}

// (linear workspaces, attention workspaces)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
    if (nargs != 2 || !PyDict_CheckExact(a[0]) || !PyDict_CheckExact(a[1])) { PyErr_SetString(PyExc_TypeError, "two dicts expected"); return nullptr; }
    Py_INCREF(a[0]); Py_INCREF(a[1]);
    Py_XSETREF(g_workspaces, a[0]);
    Py_XSETREF(g_att_workspaces, a[1]);
    Py_RETURN_NONE;
}

#define MT_FN(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MT_FN(bind), MT_FN(qgemm), MT_FN(qgemm_ordered), MT_FN(qgemm_residual), MT_FN(qgemm_swiglu), MT_FN(qkv_rope),
                         MT_FN(attention_decode), MT_FN(attention), MT_FN(rms_norm), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    PyObject* m = PyModule_Create(&module);
    if (m && PyModule_AddStringConstant(m, "torch_version", MT_TORCH_VERSION) < 0) { Py_DECREF(m); return nullptr; }
    return m;
}

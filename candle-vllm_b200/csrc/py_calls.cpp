// py_calls.cpp -- the operators that a decode step calls most, as native Python functions over the C ABI.
//
// A call of a few microseconds on the GPU was entered through 10 to 26 us of Python: shape and type checks, views that change nothing, an allocation, a foreign-function call with a
// dozen arguments, the error check.  Here a call whose arguments are plain -- torch tensors of the exact class, on the current device, contiguous, of the types the kernel takes -- is
// checked, allocated for and launched natively.  Anything else returns None and the caller goes the way through Python: nothing is accepted here that is refused there.  So do the calls
// that find no workspace or too small a one, an operator's first and those that grow it.
// [Host time, us a call, Python -> here: Linear.forward 12.8 -> 4.2, QMatMul.forward 16.6 -> 7.4, silu_mul 10.2 -> 4.2, PagedAttention.forward (decode, with its cache write) 25.2 -> 9.7,
// latent decode with its cache write 26 -> less than the GPU's 13.8 (one sequence of 1000 keys); a
// call that is left to Python 0.3 more than without the look.]
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <dlfcn.h>

#include "b200_backend.h"

namespace {

// the library's functions, from the copy of the library that the package has loaded
struct Library {
    decltype(&linear_16bit) linear = nullptr;
    decltype(&qmatmul_f32) qmatmul = nullptr;
    decltype(&qmatmul_workspace_bytes) qmatmul_bytes = nullptr;
    decltype(&silu_mul) silu = nullptr;
    decltype(&reshape_and_cache) cache = nullptr;
    decltype(&paged_attention_decode) decode = nullptr;
    decltype(&paged_attention_decode_workspace_bytes) decode_bytes = nullptr;
    decltype(&paged_attention_prefill) prefill = nullptr;
    decltype(&concat_and_cache_mla) latent_cache = nullptr;
    decltype(&mla_paged_attention) latent = nullptr;
    decltype(&mla_paged_decode_workspace_bytes) latent_bytes = nullptr;
    decltype(&b200_last_error) last_error = nullptr;
    decltype(&b200_device_cc) cc = nullptr;
    bool ready = false;
} L;

// A tensor of torch's own class with memory on a device, contiguous or of rows [heads, width] a stride apart, or null.  (Subclasses, fake and batched tensors: not here.)
const at::Tensor* rows(PyObject* o) {
    if (!THPVariable_CheckExact(o)) return nullptr;
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || t.layout() != at::kStrided || !t.is_cuda() || !t.has_storage() || t.is_neg() || t.is_conj()) return nullptr;
    if (t.unsafeGetTensorImpl()->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Python,
                                                                       c10::DispatchKey::Functionalize, c10::DispatchKey::Batched}))) return nullptr;
    return t.is_contiguous() || (t.dim() == 3 && t.stride(2) == 1 && t.stride(1) == t.size(2)) ? &t : nullptr;
}
const at::Tensor* plain(PyObject* o) {
    const at::Tensor* t = rows(o);
    return t && t->is_contiguous() ? t : nullptr;
}
int64_t row_stride(const at::Tensor& t) { return t.is_contiguous() ? t.size(1) * t.size(2) : t.stride(0); }
bool here(const at::Tensor& t, int device) { return t.get_device() == device; }
int type16(const at::Tensor& t) { return t.scalar_type() == at::kBFloat16 ? B200_BF16 : (t.scalar_type() == at::kHalf ? B200_F16 : -1); }
bool fits(int64_t v) { return v > 0 && v <= INT32_MAX; }

struct Unlocked {                  // the interpreter lock is not held while the library runs: a launch may wait for room in the queue
    PyThreadState* s = PyEval_SaveThread();
    ~Unlocked() { PyEval_RestoreThread(s); }
};

// the result, or the code of the error that the call recorded: the caller raises it (its message is the library's last, of this thread)
PyObject* result(at::Tensor&& out) {
    if (const int e = L.last_error()) return PyLong_FromLong(e);
    return THPVariable_Wrap(std::move(out));
}

at::Tensor fresh(at::IntArrayRef sizes, const at::Tensor& like, at::ScalarType type) { return at::empty(sizes, at::TensorOptions().dtype(type).device(like.device())); }

// The caller's numbers.  False for what converts to none (None, a float where an integer belongs): Python's way decides what becomes of it.
bool known(bool ok) {
    if (!ok) PyErr_Clear();
    return ok;
}
bool number(PyObject* o, int64_t& v) { v = PyLong_AsLongLong(o); return known(v != -1 || !PyErr_Occurred()); }
bool number(PyObject* o, double& v) { v = PyFloat_AsDouble(o); return known(v != -1.0 || !PyErr_Occurred()); }
bool number(PyObject* o, bool& v) { const int t = PyObject_IsTrue(o); v = t > 0; return known(t >= 0); }

// linear(x, weight, bias or None)
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 3) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]), *b = a[2] == Py_None ? nullptr : plain(a[2]);
    if (!x || !w || (a[2] != Py_None && !b) || w->dim() != 2 || x->dim() < 1) Py_RETURN_NONE;
    const int64_t n = w->size(0), k = w->size(1), m = k > 0 ? x->numel() / k : 0;
    const int type = type16(*x), dev = x->get_device();
    if (type < 0 || w->scalar_type() != x->scalar_type() || x->size(-1) != k || !fits(m) || !fits(n) || !fits(k) || k % 8 || n % 8) Py_RETURN_NONE;
    if (b && (b->scalar_type() != x->scalar_type() || b->numel() != n || !here(*b, dev))) Py_RETURN_NONE;
    if (dev != c10::cuda::current_device() || !here(*w, dev) || L.cc() < 100) Py_RETURN_NONE;
    at::DimVector sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    at::Tensor out = fresh(sizes, *x, x->scalar_type());
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked u;
        L.linear(x->data_ptr(), w->data_ptr(), b ? b->data_ptr() : nullptr, out.data_ptr(), (int32_t)m, (int32_t)n, (int32_t)k, type, st);
    }
    return result(std::move(out));
    END_HANDLE_TH_ERRORS
}

// qmatmul(x f32, blocks, n, k, ggml type, workspace or None)
PyObject* py_qmatmul(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 6 || a[5] == Py_None) Py_RETURN_NONE;
    const at::Tensor *x = plain(a[0]), *w = plain(a[1]), *ws = plain(a[5]);
    if (!x || !w || !ws || x->dim() < 1 || x->scalar_type() != at::kFloat || w->scalar_type() != at::kByte || ws->scalar_type() != at::kByte) Py_RETURN_NONE;
    int64_t n, k, type;
    if (!number(a[2], n) || !number(a[3], k) || !number(a[4], type)) Py_RETURN_NONE;
    const int64_t m = k > 0 ? x->numel() / k : 0;
    const int dev = x->get_device();
    if (x->size(-1) != k || !fits(m) || !fits(n) || !fits(k) || dev != c10::cuda::current_device() || !here(*w, dev) || !here(*ws, dev) || L.cc() < 100) Py_RETURN_NONE;
    if ((uint64_t)ws->numel() < L.qmatmul_bytes((int32_t)m, (int32_t)n, (int32_t)k)) Py_RETURN_NONE;
    at::DimVector sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = n;
    at::Tensor out = fresh(sizes, *x, at::kFloat);
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked u;
        L.qmatmul(static_cast<const float*>(x->data_ptr()), w->data_ptr(), static_cast<float*>(out.data_ptr()), (int32_t)m, (int32_t)n, (int32_t)k, (int32_t)type, 0, ws->data_ptr(),
                  (size_t)ws->numel(), st);
    }
    return result(std::move(out));
    END_HANDLE_TH_ERRORS
}

// silu_mul(gate f32, up f32) -> f32
PyObject* py_silu_mul(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 2) Py_RETURN_NONE;
    const at::Tensor *g = plain(a[0]), *u = plain(a[1]);
    if (!g || !u || g->scalar_type() != at::kFloat || u->scalar_type() != at::kFloat || g->sizes() != u->sizes() || g->numel() < 1) Py_RETURN_NONE;
    const int dev = g->get_device();
    if (dev != c10::cuda::current_device() || !here(*u, dev) || L.cc() < 100) Py_RETURN_NONE;
    at::Tensor out = fresh(g->sizes(), *g, at::kFloat);
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked un;
        L.silu(static_cast<const float*>(g->data_ptr()), static_cast<const float*>(u->data_ptr()), out.data_ptr(), g->numel(), B200_F32, st);
    }
    return result(std::move(out));
    END_HANDLE_TH_ERRORS
}

// paged_attention(prompt, q [T, H, hd], k, v [T, G, hd] (rows any stride apart: parts of a fused projection), k_cache, v_cache [blocks, bs, G, hd], slots i64, tables i32 [B, W], lens i32 [B] or None, cu_q, cu_k i32 [B + 1] or None,
//                 workspace or None, heads, kv heads, head dim, longest query, window, scale, cap, e4m3 cache)
// decode: lens and a workspace; prompt: cu_q and cu_k.  An error of the cache write comes back as its negative code.
PyObject* py_paged_attention(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 20) Py_RETURN_NONE;
    bool prompt, e4m3;
    if (!number(*a++, prompt)) Py_RETURN_NONE;
    const at::Tensor *q = plain(a[0]), *k = rows(a[1]), *v = rows(a[2]), *kc = plain(a[3]), *vc = plain(a[4]), *slots = plain(a[5]), *bt = plain(a[6]);
    if (!q || !k || !v || !kc || !vc || !slots || !bt) Py_RETURN_NONE;
    const at::Tensor *lens = prompt || a[7] == Py_None ? nullptr : plain(a[7]), *cu_q = prompt ? plain(a[8]) : nullptr, *cu_k = prompt ? plain(a[9]) : nullptr, *ws = prompt || a[10] == Py_None ? nullptr : plain(a[10]);
    if (prompt ? (!cu_q || !cu_k) : (!lens || !ws)) Py_RETURN_NONE;
    int64_t H, G, hd, window, longest = 0;
    double scale, cap;
    if (!number(a[11], H) || !number(a[12], G) || !number(a[13], hd) || (prompt && !number(a[14], longest)) || !number(a[15], window) || !number(a[16], scale) || !number(a[17], cap) ||
        !number(a[18], e4m3)) Py_RETURN_NONE;
    const int type = type16(*q), dev = q->get_device();
    auto words = [&](const at::Tensor& t) { return t.scalar_type() == at::kInt || t.scalar_type() == at::kUInt32; };
    if (type < 0 || q->dim() != 3 || q->size(1) != H || q->size(2) != hd || k->dim() != 3 || v->dim() != 3 || k->sizes() != v->sizes() || k->size(1) != G || k->size(2) != hd) Py_RETURN_NONE;
    if (k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || kc->dim() != 4 || kc->sizes() != vc->sizes() || kc->scalar_type() != vc->scalar_type()) Py_RETURN_NONE;
    if (kc->size(2) != G || kc->size(3) != hd || slots->scalar_type() != at::kLong || slots->numel() != k->size(0) || !words(*bt) || bt->dim() != 2) Py_RETURN_NONE;
    const int cache_type = e4m3 || kc->scalar_type() == at::kByte ? B200_FP8_E4M3 : type;
    if (cache_type == B200_FP8_E4M3 ? kc->scalar_type() != at::kByte : kc->scalar_type() != q->scalar_type()) Py_RETURN_NONE;
    const int64_t T = q->size(0), bs = kc->size(1), nb = kc->size(0), W = bt->size(1), seqs = prompt ? cu_q->numel() - 1 : T;
    if (!fits(T) || !fits(k->size(0)) || !fits(seqs) || !fits(W) || !fits(bs) || !fits(nb) || !fits(H) || !fits(G) || !fits(hd) || bt->size(0) < seqs || window < 0 || window > INT32_MAX) Py_RETURN_NONE;
    if (prompt ? (!words(*cu_q) || !words(*cu_k) || cu_k->numel() != cu_q->numel() || !fits(longest) || !here(*cu_q, dev) || !here(*cu_k, dev))
               : (!words(*lens) || lens->numel() < T || ws->scalar_type() != at::kByte || !here(*lens, dev) || !here(*ws, dev))) Py_RETURN_NONE;
    for (const at::Tensor* t : {k, v, kc, vc, slots, bt}) if (!here(*t, dev)) Py_RETURN_NONE;
    if (dev != c10::cuda::current_device() || L.cc() < 100) Py_RETURN_NONE;
    if (!prompt && (uint64_t)ws->numel() < L.decode_bytes((int32_t)T, (int32_t)H, (int32_t)hd, (int32_t)W, (int32_t)bs)) Py_RETURN_NONE;
    at::Tensor out = fresh(q->sizes(), *q, q->scalar_type());
    int write_error = 0;
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked u;
        L.cache(k->data_ptr(), v->data_ptr(), kc->data_ptr(), vc->data_ptr(), static_cast<const int64_t*>(slots->data_ptr()), (int32_t)k->size(0), (int32_t)G, (int32_t)hd, (int32_t)bs,
                row_stride(*k), row_stride(*v), type, cache_type, B200_KV_FLASH, st);
        write_error = L.last_error();
        const auto* tables = static_cast<const uint32_t*>(bt->data_ptr());
        if (write_error) {
        } else if (prompt)
            L.prefill(out.data_ptr(), q->data_ptr(), kc->data_ptr(), vc->data_ptr(), tables, static_cast<const uint32_t*>(cu_q->data_ptr()), static_cast<const uint32_t*>(cu_k->data_ptr()),
                      (int32_t)seqs, (int32_t)T, (int32_t)longest, (int32_t)H, (int32_t)G, (int32_t)hd, (int32_t)bs, (int32_t)W, (float)scale, (float)cap, (int32_t)window, type, cache_type, B200_KV_FLASH, st);
        else
            L.decode(out.data_ptr(), q->data_ptr(), kc->data_ptr(), vc->data_ptr(), tables, static_cast<const uint32_t*>(lens->data_ptr()), (int32_t)T, (int32_t)H, (int32_t)G, (int32_t)hd,
                     (int32_t)bs, (int32_t)W, nb, (float)scale, (float)cap, (int32_t)window, type, cache_type, B200_KV_FLASH, type, ws->data_ptr(), (size_t)ws->numel(), st);
    }
    if (write_error) return PyLong_FromLong(-write_error);
    return result(std::move(out));
    END_HANDLE_TH_ERRORS
}

// latent_cache(ckv [T, R], k_pe [T, P], their caches [blocks, bs, 1, R] and [.., P], slots i64 [T]) -> 0 or the error's code
PyObject* py_latent_cache(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 5) Py_RETURN_NONE;
    const at::Tensor *c = plain(a[0]), *r = plain(a[1]), *cc = plain(a[2]), *rc = plain(a[3]), *slots = plain(a[4]);
    if (!c || !r || !cc || !rc || !slots || c->dim() != 2 || r->dim() != 2 || cc->dim() != 4 || rc->dim() != 4) Py_RETURN_NONE;
    const int type = type16(*c), dev = c->get_device();
    if (type < 0 || cc->scalar_type() != c->scalar_type() || r->scalar_type() != c->scalar_type() || rc->scalar_type() != c->scalar_type() || slots->scalar_type() != at::kLong) Py_RETURN_NONE;
    const int64_t T = c->size(0), R = c->size(1), P = r->size(1);
    if (!fits(T) || !fits(R) || !fits(P) || r->size(0) != T || slots->numel() != T || cc->size(3) != R || rc->size(3) != P || cc->size(2) != 1 || rc->size(2) != 1) Py_RETURN_NONE;
    for (const at::Tensor* t : {r, cc, rc, slots}) if (!here(*t, dev)) Py_RETURN_NONE;
    if (dev != c10::cuda::current_device() || L.cc() < 100) Py_RETURN_NONE;
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked u;
        L.latent_cache(c->data_ptr(), r->data_ptr(), cc->data_ptr(), rc->data_ptr(), static_cast<const int64_t*>(slots->data_ptr()), (int32_t)T, (int32_t)R, (int32_t)P, type, st);
    }
    return PyLong_FromLong(L.last_error());
    END_HANDLE_TH_ERRORS
}

// latent_decode(q [B, H, R], q_pe [B, H, P], caches, tables i32 [B, W], lens i32 [B], scale): one row per sequence
PyObject* py_latent_decode(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
    HANDLE_TH_ERRORS
    if (!L.ready || n_args != 7) Py_RETURN_NONE;
    const at::Tensor *q = plain(a[0]), *qp = plain(a[1]), *cc = plain(a[2]), *rc = plain(a[3]), *bt = plain(a[4]), *lens = plain(a[5]);
    double scale;
    if (!q || !qp || !cc || !rc || !bt || !lens || q->dim() != 3 || qp->dim() != 3 || cc->dim() != 4 || rc->dim() != 4 || bt->dim() != 2 || !number(a[6], scale)) Py_RETURN_NONE;
    const int type = type16(*q), dev = q->get_device();
    if (type < 0 || qp->scalar_type() != q->scalar_type() || cc->scalar_type() != q->scalar_type() || rc->scalar_type() != q->scalar_type()) Py_RETURN_NONE;
    const int64_t B = q->size(0), H = q->size(1), R = q->size(2), P = qp->size(2), W = bt->size(1), nb = cc->size(0), bs = cc->size(1);
    if (!fits(B) || !fits(H) || !fits(R) || !fits(P) || !fits(W) || !fits(nb) || !fits(bs) || qp->size(0) != B || qp->size(1) != H || bt->size(0) != B || lens->numel() != B) Py_RETURN_NONE;
    if (cc->size(2) != 1 || rc->size(2) != 1 || cc->size(3) != R || rc->size(3) != P || rc->size(0) != nb || rc->size(1) != bs) Py_RETURN_NONE;
    if (bt->scalar_type() != at::kInt || lens->scalar_type() != at::kInt) Py_RETURN_NONE;
    for (const at::Tensor* t : {qp, cc, rc, bt, lens}) if (!here(*t, dev)) Py_RETURN_NONE;
    if (dev != c10::cuda::current_device() || L.cc() < 100) Py_RETURN_NONE;
    const size_t need = L.latent_bytes((int32_t)B, (int32_t)H, (int32_t)W, (int32_t)bs);
    if (need > (size_t)INT64_MAX) Py_RETURN_NONE;
    at::Tensor out = fresh(q->sizes(), *q, q->scalar_type()), ws = fresh({(int64_t)need}, *q, at::kByte);
    const int64_t st = reinterpret_cast<int64_t>(c10::cuda::getCurrentCUDAStream(dev).stream());
    {
        Unlocked u;
        L.latent(out.data_ptr(), q->data_ptr(), qp->data_ptr(), cc->data_ptr(), rc->data_ptr(), static_cast<const uint32_t*>(bt->data_ptr()), static_cast<const uint32_t*>(lens->data_ptr()),
                 nullptr, (int32_t)B, (int32_t)B, (int32_t)H, (int32_t)R, (int32_t)P, (int32_t)bs, (int32_t)W, nb, (float)scale, type, ws.data_ptr(), need, st);
    }
    return result(std::move(out));
    END_HANDLE_TH_ERRORS
}

// bind(path of the library that is loaded)
PyObject* py_bind(PyObject*, PyObject* path) {
    const char* p = PyUnicode_AsUTF8(path);
    if (!p) return nullptr;
    void* h = dlopen(p, RTLD_NOW | RTLD_NOLOAD);
    if (!h) { PyErr_Format(PyExc_ImportError, "%s is not loaded", p); return nullptr; }
    bool ok = true;
    auto find = [&](auto& f, const char* name) { f = reinterpret_cast<std::remove_reference_t<decltype(f)>>(dlsym(h, name)); ok = ok && f; };
    find(L.linear, "linear_16bit"); find(L.qmatmul, "qmatmul_f32"); find(L.qmatmul_bytes, "qmatmul_workspace_bytes"); find(L.silu, "silu_mul"); find(L.cache, "reshape_and_cache");
    find(L.decode, "paged_attention_decode"); find(L.decode_bytes, "paged_attention_decode_workspace_bytes"); find(L.prefill, "paged_attention_prefill");
    find(L.latent_cache, "concat_and_cache_mla"); find(L.latent, "mla_paged_attention"); find(L.latent_bytes, "mla_paged_decode_workspace_bytes");
    find(L.last_error, "b200_last_error"); find(L.cc, "b200_device_cc");
    if (!ok) { PyErr_Format(PyExc_ImportError, "%s lacks a function", p); return nullptr; }
    L.ready = true;
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {{"bind", py_bind, METH_O, nullptr},
                          {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_linear)), METH_FASTCALL, nullptr},
                          {"qmatmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_qmatmul)), METH_FASTCALL, nullptr},
                          {"silu_mul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_silu_mul)), METH_FASTCALL, nullptr},
                          {"paged_attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_paged_attention)), METH_FASTCALL, nullptr},
                          {"latent_cache", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_latent_cache)), METH_FASTCALL, nullptr},
                          {"latent_decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_latent_decode)), METH_FASTCALL, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&kModule); }

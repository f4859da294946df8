// Native half of the torch front end (api.py): fills the C-ABI parameter blocks straight from the tensors, allocates
// results and scratch, and calls libltc_attn.so.
//
// Why it is native: the small calls of this library run for 5 to 10 us on the GPU, while filling an
// ltca_attn_params block field by field through ctypes, asking for the workspace size and allocating two results took
// the host about 18 us per forward and 25 us per decode step - the calls were bound by the interpreter.  Here a call
// is one argument vector, two allocations without the dispatcher, and the launch itself.
//
// Every function takes its arguments by position (the Python methods of Context give them names and defaults) and enqueues
// on the context's stream like the C ABI does.  The C call itself runs without the interpreter lock, as calls through
// ctypes do: threads that drive contexts of their own enqueue side by side, and a launch queue that is full holds up only
// the thread that met it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>

#include "../../include/ltc_attn.h"

namespace {

PyObject* g_error_class = nullptr;      // api.LtcaError, set once at import
PyObject* g_memory_class = nullptr;     // torch.OutOfMemoryError

// Thrown when a Python exception has been set; the entry wrapper turns it into a null return.
struct PyErrorSet {};

[[noreturn]] void raise(PyObject* type, const char* msg) {
    PyErr_SetString(type, msg);
    throw PyErrorSet();
}
inline void require(bool ok, const char* msg) {
    if (!ok) raise(PyExc_AssertionError, msg);
}

struct Host {
    PyObject_HEAD
    ltca_ctx* ctx;
    int device;
    at::Tensor* ws;      // scratch, grown on demand and kept
};

void check(const Host* h, int rc) {
    if (rc == 0) return;
    PyObject* e = PyObject_CallFunction(g_error_class ? g_error_class : PyExc_RuntimeError, "is", rc,
                                        ltca_last_error(h->ctx));
    if (e) {
        PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(e)), e);
        Py_DECREF(e);
    }
    throw PyErrorSet();
}

// f() without the interpreter lock; it touches no Python object, and whatever it reads is held by the caller.
template <typename F>
int unlocked(F f) {
    struct Release {
        PyThreadState* state = PyEval_SaveThread();
        ~Release() { PyEval_RestoreThread(state); }
    } release;
    return f();
}

// ---- argument access ---------------------------------------------------------------------------
inline bool given(PyObject* o) { return o && o != Py_None; }
inline const at::Tensor& tensor(PyObject* o) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a tensor");
    return THPVariable_Unpack(o);
}
inline double number(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet();
    return v;
}
inline int64_t integer(PyObject* o) {
    if (PyLong_Check(o)) {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
        return v;
    }
    PyObject* i = PyNumber_Long(o);
    if (!i) throw PyErrorSet();
    const long long v = PyLong_AsLongLong(i);
    Py_DECREF(i);
    if (v == -1 && PyErr_Occurred()) throw PyErrorSet();
    return v;
}
// Any whole number, modulo 2^64 (what a ctypes field of that type takes).
inline uint64_t word64(PyObject* o) {
    PyObject* i = PyNumber_Long(o);
    if (!i) throw PyErrorSet();
    const unsigned long long v = PyLong_AsUnsignedLongLongMask(i);
    Py_DECREF(i);
    if (v == (unsigned long long)-1 && PyErr_Occurred()) throw PyErrorSet();
    return v;
}
inline int truth(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PyErrorSet();
    return v;
}

inline at::Tensor empty(const Host* h, at::IntArrayRef sizes, at::ScalarType t) {
    return at::Tensor(at::detail::empty_cuda(sizes, t, at::Device(at::kCUDA, (c10::DeviceIndex)h->device), std::nullopt));
}
inline PyObject* wrap(at::Tensor t) {
    PyObject* o = THPVariable_Wrap(std::move(t));
    if (!o) throw PyErrorSet();
    return o;
}
// The caller's tensor or a new one, as a new reference.
inline PyObject* result(PyObject* given_obj, const at::Tensor& t) {
    if (given(given_obj)) {
        Py_INCREF(given_obj);
        return given_obj;
    }
    return wrap(t);
}

// Undefined for zero bytes.  The result is a reference of its own: while the lock is released another thread may have
// the scratch of this context grow.
at::Tensor workspace(Host* h, size_t bytes) {
    if (bytes == 0) return at::Tensor();
    if (!h->ws->defined() || (size_t)h->ws->numel() < bytes) {
        *h->ws = at::Tensor();           // give the old block back before the larger one is taken
        *h->ws = empty(h, {(int64_t)bytes}, at::kByte);
    }
    return *h->ws;
}

// ---- the attention core ------------------------------------------------------------------------
inline ltca_strides strides(const at::Tensor& t) {
    require(t.dim() == 4 && (t.stride(3) == 1 || t.size(3) == 1), "head_dim must be contiguous");
    return ltca_strides{t.stride(0), t.stride(1), t.stride(2)};
}
inline void same_shape(const at::Tensor& t, int64_t B, int64_t H, int64_t S, int64_t D, const char* msg) {
    require(t.dim() == 4 && t.size(0) == B && t.size(1) == H && t.size(2) == S && t.size(3) == D, msg);
}

struct Core {
    ltca_attn_params p;
    int64_t B, H, Sq, Sk, D;
    at::ScalarType dtype;
};

// Shape, storage type and options that forward, backward and decode share.
void fill(Core& c, const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, PyObject* scale, int causal, PyObject* keep_mask,
          PyObject* kv_len, PyObject* score_clamp, int mode) {
    std::memset(&c.p, 0, sizeof(c.p));
    require(q.is_cuda() && k.is_cuda() && v.is_cuda(), "q, k and v must be CUDA tensors");
    require(q.dim() == 4 && k.dim() == 4, "tensors are [batch, heads, seq, head_dim]");
    c.B = q.size(0); c.H = q.size(1); c.Sq = q.size(2); c.D = q.size(3); c.Sk = k.size(2);
    same_shape(k, c.B, c.H, c.Sk, c.D, "k must be [batch, heads, keys, head_dim]");
    same_shape(v, c.B, c.H, c.Sk, c.D, "v must have the shape of k");
    c.dtype = q.scalar_type();
    require(k.scalar_type() == c.dtype && v.scalar_type() == c.dtype, "q, k and v must have one dtype");
    ltca_attn_params& p = c.p;
    if (c.dtype == at::kFloat) p.dtype = LTCA_F32;
    else if (c.dtype == at::kBFloat16) p.dtype = LTCA_BF16;
    else raise(PyExc_TypeError, "unsupported dtype: the tensors must be float32 or bfloat16");
    p.B = (int32_t)c.B; p.H = (int32_t)c.H; p.Sq = (int32_t)c.Sq; p.Sk = (int32_t)c.Sk; p.D = (int32_t)c.D;
    p.mode = mode;
    p.causal = causal;
    p.scale = given(scale) ? (float)number(scale) : (float)(1.0 / std::sqrt((double)c.D));
    p.score_clamp = given(score_clamp) ? (float)number(score_clamp) : 0.f;
    p.q = q.data_ptr(); p.q_strides = strides(q);
    p.k = k.data_ptr(); p.k_strides = strides(k);
    p.v = v.data_ptr(); p.v_strides = strides(v);
    if (given(keep_mask)) {
        const at::Tensor& m = tensor(keep_mask);
        require(m.scalar_type() == at::kFloat && m.is_contiguous() && m.dim() == 3 && m.size(0) == c.B && m.size(1) == c.Sq &&
                    m.size(2) == c.Sk, "keep_mask must be contiguous float32 [batch, queries, keys]");
        p.keep_mask = static_cast<const float*>(m.data_ptr());
    }
    if (given(kv_len)) {
        const at::Tensor& n = tensor(kv_len);
        require(n.scalar_type() == at::kInt && n.is_contiguous() && n.dim() == 1 && n.size(0) == c.B,
                "kv_len must be contiguous int32 [batch]");
        p.kv_len = static_cast<const int32_t*>(n.data_ptr());
    }
}

// The scratch of a call, which keeps it until it returns.
template <typename Params>
at::Tensor attach(Host* h, Params& p, size_t bytes) {
    at::Tensor ws = workspace(h, bytes);
    if (ws.defined()) {
        p.workspace = ws.data_ptr();
        p.workspace_bytes = (size_t)ws.numel();
    }
    return ws;
}

// out / lse: the caller's tensors, or new ones of the shape that the call writes.
void outputs(Host* h, Core& c, PyObject* out_obj, PyObject* lse_obj, at::Tensor& o, at::Tensor& lse) {
    o = given(out_obj) ? tensor(out_obj) : empty(h, {c.B, c.H, c.Sq, c.D}, c.dtype);
    lse = given(lse_obj) ? tensor(lse_obj) : empty(h, {c.B, c.H, c.Sq}, at::kFloat);
    same_shape(o, c.B, c.H, c.Sq, c.D, "out must have the shape of q");
    require(o.scalar_type() == c.dtype, "out must have the dtype of q");
    c.p.o = o.data_ptr();
    c.p.o_strides = strides(o);
    c.p.lse = static_cast<float*>(lse.data_ptr());
}

// (q, k, v, scale, causal, keep_mask, kv_len, score_clamp, mode, out, lse)
PyObject* attn_fwd(Host* h, PyObject* const* a) {
    Core c;
    fill(c, tensor(a[0]), tensor(a[1]), tensor(a[2]), a[3], truth(a[4]), a[5], a[6], a[7], (int)integer(a[8]));
    at::Tensor o, lse;
    outputs(h, c, a[9], a[10], o, lse);
    size_t need = 0;
    ltca_attn_workspace_bytes(&c.p, 0, &need);
    const at::Tensor ws = attach(h, c.p, need);
    check(h, unlocked([&] { return ltca_attn_fwd(h->ctx, &c.p); }));
    return Py_BuildValue("NN", result(a[9], o), result(a[10], lse));
}

// (q, k, v, kv_len, scale, keep_mask, score_clamp, out, lse)
PyObject* attn_decode(Host* h, PyObject* const* a) {
    Core c;
    fill(c, tensor(a[0]), tensor(a[1]), tensor(a[2]), a[4], 0, a[5], a[3], a[6], LTCA_MODE_FP32);
    at::Tensor o, lse;
    outputs(h, c, a[7], a[8], o, lse);
    size_t need = 0;
    ltca_attn_decode_workspace_bytes(&c.p, &need);
    const at::Tensor ws = attach(h, c.p, need);
    check(h, unlocked([&] { return ltca_attn_decode(h->ctx, &c.p); }));
    return Py_BuildValue("NN", result(a[7], o), result(a[8], lse));
}

// (q, k, v, o, lse, dout, scale, causal, keep_mask, kv_len, score_clamp, mode, dq, dk, dv, deterministic)
PyObject* attn_bwd(Host* h, PyObject* const* a) {
    Core c;
    fill(c, tensor(a[0]), tensor(a[1]), tensor(a[2]), a[6], truth(a[7]), a[8], a[9], a[10], (int)integer(a[11]));
    const at::Tensor& o = tensor(a[3]);
    const at::Tensor& dout = tensor(a[5]);
    same_shape(o, c.B, c.H, c.Sq, c.D, "o must have the shape of q");
    same_shape(dout, c.B, c.H, c.Sq, c.D, "dout must have the shape of q");
    require(o.scalar_type() == c.dtype && dout.scalar_type() == c.dtype, "o and dout must have the dtype of q");
    ltca_attn_params& p = c.p;
    p.o = o.data_ptr(); p.o_strides = strides(o);
    p.lse = given(a[4]) ? static_cast<float*>(tensor(a[4]).data_ptr()) : nullptr;
    p.dout = dout.data_ptr(); p.do_strides = strides(dout);
    const int64_t shape_q[4] = {c.B, c.H, c.Sq, c.D}, shape_k[4] = {c.B, c.H, c.Sk, c.D};
    at::Tensor g[3];
    for (int i = 0; i < 3; ++i) {
        const int64_t* s = i == 0 ? shape_q : shape_k;
        g[i] = given(a[12 + i]) ? tensor(a[12 + i]) : empty(h, at::IntArrayRef(s, 4), c.dtype);
    }
    p.dq = g[0].data_ptr(); p.dq_strides = strides(g[0]);
    p.dk = g[1].data_ptr(); p.dk_strides = strides(g[1]);
    p.dv = g[2].data_ptr(); p.dv_strides = strides(g[2]);
    p.bwd_deterministic = truth(a[15]);
    size_t need = 0;
    ltca_attn_workspace_bytes(&p, 1, &need);
    const at::Tensor ws = attach(h, p, need);
    check(h, unlocked([&] { return ltca_attn_bwd(h->ctx, &p); }));
    return Py_BuildValue("NNN", result(a[12], g[0]), result(a[13], g[1]), result(a[14], g[2]));
}

// ---- the modules -------------------------------------------------------------------------------
// x, wq, wk, wv, wo, B, S, H, head_width, scale, causal, time_major, use_residual, use_layer_norm, gamma, beta,
// keep_mask, mode, bq, bk, bv, bo   (the first kModuleArgs arguments of every module call)
constexpr int kModuleArgs = 22;

inline const float* f32_or_null(PyObject* o) { return given(o) ? static_cast<const float*>(tensor(o).data_ptr()) : nullptr; }
inline const float* bias(PyObject* o) {
    if (!given(o)) return nullptr;
    const at::Tensor& b = tensor(o);
    require(b.scalar_type() == at::kFloat && b.is_contiguous(), "biases must be contiguous float32");
    return static_cast<const float*>(b.data_ptr());
}

void fill_module(ltca_tsa_params& p, PyObject* const* a) {
    std::memset(&p, 0, sizeof(p));
    const at::Tensor& x = tensor(a[0]);
    p.B = (int32_t)integer(a[5]); p.S = (int32_t)integer(a[6]);
    p.H = (int32_t)integer(a[7]); p.head_width = (int32_t)integer(a[8]);
    require(x.is_cuda() && x.dim() == 2 && x.size(0) == (int64_t)p.B * p.S && x.scalar_type() == at::kFloat && x.is_contiguous(),
            "x must be a contiguous float32 CUDA tensor [batch * seq, input_dim]");
    p.E = (int32_t)x.size(1);
    const int64_t E = p.E, HW = (int64_t)p.H * p.head_width;
    const float* w[4];
    for (int i = 0; i < 4; ++i) {
        const at::Tensor& t = tensor(a[1 + i]);
        require(t.dim() == 2 && t.size(0) == (i < 3 ? E : HW) && t.size(1) == (i < 3 ? HW : E),
                "wq, wk, wv are [input_dim, heads * head_width], wo is [heads * head_width, input_dim]");
        w[i] = static_cast<const float*>(t.data_ptr());
    }
    p.x = static_cast<const float*>(x.data_ptr());
    p.wq = w[0]; p.wk = w[1]; p.wv = w[2]; p.wo = w[3];
    p.scale = (float)number(a[9]);
    p.causal = truth(a[10]); p.time_major = truth(a[11]);
    p.use_residual = truth(a[12]); p.use_layer_norm = truth(a[13]);
    if (given(a[14])) { p.ln_gamma = f32_or_null(a[14]); p.ln_beta = f32_or_null(a[15]); }
    p.keep_mask = f32_or_null(a[16]);
    p.mode = (int32_t)integer(a[17]);
    p.bq = bias(a[18]); p.bk = bias(a[19]); p.bv = bias(a[20]); p.bo = bias(a[21]);
}

void attach_saved(ltca_tsa_params& p, PyObject* saved, int reuse) {
    if (!given(saved)) return;
    const at::Tensor& s = tensor(saved);
    p.saved = s.data_ptr();
    p.saved_bytes = (size_t)s.numel();
    p.reuse_forward = reuse;
}
// weight_cache: None or (buffer, valid).  The result keeps the buffer for the call.
at::Tensor attach_weight_cache(ltca_tsa_params& p, PyObject* cache) {
    if (!given(cache)) return at::Tensor();
    PyObject* buf = PySequence_GetItem(cache, 0);
    PyObject* valid = buf ? PySequence_GetItem(cache, 1) : nullptr;
    if (!valid) { Py_XDECREF(buf); throw PyErrorSet(); }
    at::Tensor t;
    if (THPVariable_Check(buf)) t = THPVariable_Unpack(buf);
    const int v = PyObject_IsTrue(valid);
    if (t.defined()) { p.weight_cache = t.data_ptr(); p.weight_cache_bytes = (size_t)t.numel(); p.weight_cache_valid = v; }
    Py_DECREF(buf);
    Py_DECREF(valid);
    if (!t.defined()) raise(PyExc_TypeError, "weight_cache is (buffer, valid)");
    if (v < 0) throw PyErrorSet();
    return t;
}

at::Tensor attach_module(Host* h, ltca_tsa_params& p, int which) {
    size_t need = 0;
    check(h, ltca_tsa_workspace_bytes(&p, which, &need));
    return attach(h, p, need);
}

PyObject* module_forward(Host* h, ltca_tsa_params& p, const at::Tensor& x) {
    at::Tensor out = empty(h, x.sizes(), at::kFloat);
    p.out = static_cast<float*>(out.data_ptr());
    const at::Tensor ws = attach_module(h, p, 0);
    check(h, unlocked([&] { return ltca_tsa_fwd(h->ctx, &p); }));
    return wrap(std::move(out));
}

// (module arguments, saved, weight_cache)
PyObject* tsa_fwd(Host* h, PyObject* const* a) {
    ltca_tsa_params p;
    fill_module(p, a);
    const at::Tensor cache = attach_weight_cache(p, a[kModuleArgs + 1]);
    attach_saved(p, a[kModuleArgs], 0);
    return module_forward(h, p, tensor(a[0]));
}

// (module arguments, dy, saved, reuse_forward, weight_cache)
PyObject* tsa_bwd(Host* h, PyObject* const* a) {
    ltca_tsa_params p;
    fill_module(p, a);
    const at::Tensor& dy = tensor(a[kModuleArgs]);
    const at::Tensor cache = attach_weight_cache(p, a[kModuleArgs + 3]);
    attach_saved(p, a[kModuleArgs + 1], truth(a[kModuleArgs + 2]));
    const at::Tensor& x = tensor(a[0]);
    at::Tensor dx = empty(h, x.sizes(), at::kFloat);
    // the four weight gradients are views of one allocation, so a multi-GPU caller sums them over the ranks with a
    // single collective on that allocation (shard.sum_weight_grads) without packing them
    const int64_t E = p.E, HW = (int64_t)p.H * p.head_width;
    at::Tensor flat = empty(h, {4 * E * HW}, at::kFloat);
    float* base = static_cast<float*>(flat.data_ptr());
    p.dy = static_cast<const float*>(dy.data_ptr());
    p.dx = static_cast<float*>(dx.data_ptr());
    p.dwq = base; p.dwk = base + E * HW; p.dwv = base + 2 * E * HW; p.dwo = base + 3 * E * HW;
    const at::Tensor ws = attach_module(h, p, 3);
    check(h, unlocked([&] { return ltca_tsa_bwd(h->ctx, &p); }));
    PyObject* out[5] = {wrap(std::move(dx)), nullptr, nullptr, nullptr, nullptr};
    for (int i = 0; i < 4; ++i) {
        const int64_t size[2] = {i < 3 ? E : HW, i < 3 ? HW : E}, stride[2] = {size[1], 1};
        auto view = c10::make_intrusive<c10::TensorImpl>(c10::Storage(flat.storage()), flat.key_set(), flat.dtype());
        view->set_sizes_and_strides(size, stride);
        view->set_storage_offset(i * E * HW);
        out[1 + i] = wrap(at::Tensor(std::move(view)));
    }
    return Py_BuildValue("NNNNN", out[0], out[1], out[2], out[3], out[4]);
}

// The FlashAttention form: LayerNorm first, dropout last.
void fill_fa(ltca_tsa_params& p, PyObject* const* a) {
    fill_module(p, a);
    p.pre_norm = 1;
    p.dropout_prob = (float)number(a[kModuleArgs]);
    p.dropout_seed = word64(a[kModuleArgs + 1]);
    p.score_clamp = (float)number(a[kModuleArgs + 2]);
}

// (module arguments, dropout_prob, dropout_seed, score_clamp)
PyObject* fa_fwd(Host* h, PyObject* const* a) {
    ltca_tsa_params p;
    fill_fa(p, a);
    return module_forward(h, p, tensor(a[0]));
}

// (module arguments, dropout_prob, dropout_seed, score_clamp, dy) -> dict of gradients
PyObject* fa_bwd(Host* h, PyObject* const* a) {
    ltca_tsa_params p;
    fill_fa(p, a);
    const at::Tensor& x = tensor(a[0]);
    p.dy = static_cast<const float*>(tensor(a[kModuleArgs + 3]).data_ptr());
    const int64_t E = p.E, HW = (int64_t)p.H * p.head_width;
    struct Grad { const char* name; at::Tensor t; float** slot; };
    auto f32 = [&](at::IntArrayRef s) { return empty(h, s, at::kFloat); };
    Grad g[11] = {
        {"dx", f32(x.sizes()), &p.dx}, {"dwq", f32({E, HW}), &p.dwq}, {"dwk", f32({E, HW}), &p.dwk},
        {"dwv", f32({E, HW}), &p.dwv}, {"dwo", f32({HW, E}), &p.dwo}, {"dbq", f32({HW}), &p.dbq},
        {"dbk", f32({HW}), &p.dbk}, {"dbv", f32({HW}), &p.dbv}, {"dbo", f32({E}), &p.dbo},
        {"dgamma", at::Tensor(), &p.dgamma}, {"dbeta", at::Tensor(), &p.dbeta}};
    const int n = p.use_layer_norm ? 11 : 9;
    if (n == 11) { g[9].t = f32({E}); g[10].t = f32({E}); }
    for (int i = 0; i < n; ++i) *g[i].slot = static_cast<float*>(g[i].t.data_ptr());
    const at::Tensor ws = attach_module(h, p, 3);
    check(h, unlocked([&] { return ltca_tsa_bwd(h->ctx, &p); }));
    PyObject* d = PyDict_New();
    if (!d) throw PyErrorSet();
    for (int i = 0; i < n; ++i) {
        PyObject* t = wrap(std::move(g[i].t));
        PyDict_SetItemString(d, g[i].name, t);
        Py_DECREF(t);
    }
    return d;
}

// (nbytes): the context's scratch, at least that large; None for zero bytes.
PyObject* host_workspace(Host* h, PyObject* const* a) {
    at::Tensor ws = workspace(h, (size_t)integer(a[0]));
    if (!ws.defined()) Py_RETURN_NONE;
    return wrap(std::move(ws));
}

// (): the context is gone; later calls fail with LTCA_ERR_INVALID.
PyObject* host_close(Host* h, PyObject* const*) {
    h->ctx = nullptr;
    *h->ws = at::Tensor();
    Py_RETURN_NONE;
}

// ---- Python type -------------------------------------------------------------------------------
template <PyObject* (*F)(Host*, PyObject* const*), int kArgs>
PyObject* entry(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    if (n != kArgs) {
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", kArgs, n);
        return nullptr;
    }
    try {
        return F(reinterpret_cast<Host*>(self), args);
    } catch (const PyErrorSet&) {
        return nullptr;
    } catch (const c10::OutOfMemoryError& e) {
        PyErr_SetString(g_memory_class ? g_memory_class : PyExc_MemoryError, e.what_without_backtrace());
        return nullptr;
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return nullptr;
    }
}

#define LTCA_METHOD(name, args) \
    {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<name, args>)), METH_FASTCALL, nullptr}
PyMethodDef host_methods[] = {
    LTCA_METHOD(attn_fwd, 11),
    LTCA_METHOD(attn_bwd, 16),
    LTCA_METHOD(attn_decode, 9),
    LTCA_METHOD(tsa_fwd, kModuleArgs + 2),
    LTCA_METHOD(tsa_bwd, kModuleArgs + 4),
    LTCA_METHOD(fa_fwd, kModuleArgs + 3),
    LTCA_METHOD(fa_bwd, kModuleArgs + 4),
    {"workspace", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<host_workspace, 1>)), METH_FASTCALL, nullptr},
    {"close", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<host_close, 0>)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

int host_init(PyObject* self, PyObject* args, PyObject*) {
    unsigned long long ctx = 0;
    int device = 0;
    if (!PyArg_ParseTuple(args, "Ki", &ctx, &device)) return -1;
    Host* h = reinterpret_cast<Host*>(self);
    h->ctx = reinterpret_cast<ltca_ctx*>(static_cast<uintptr_t>(ctx));
    h->device = device;
    if (!h->ws) h->ws = new at::Tensor();
    return 0;
}
void host_dealloc(PyObject* self) {
    delete reinterpret_cast<Host*>(self)->ws;
    Py_TYPE(self)->tp_free(self);
}

PyTypeObject HostType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* set_error_classes(PyObject*, PyObject* args) {
    PyObject *failed, *memory;
    if (!PyArg_ParseTuple(args, "OO", &failed, &memory)) return nullptr;
    Py_INCREF(failed);
    Py_XSETREF(g_error_class, failed);
    Py_INCREF(memory);
    Py_XSETREF(g_memory_class, memory);
    Py_RETURN_NONE;
}
PyMethodDef module_methods[] = {{"set_error_classes", set_error_classes, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Native half of the torch front end.", -1, module_methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    HostType.tp_name = "cuda_ltc_b200._host.Host";
    HostType.tp_basicsize = sizeof(Host);
    HostType.tp_flags = Py_TPFLAGS_DEFAULT;
    HostType.tp_doc = "Calls of one ltca_ctx: Host(context address, device).";
    HostType.tp_new = PyType_GenericNew;
    HostType.tp_init = host_init;
    HostType.tp_dealloc = host_dealloc;
    HostType.tp_methods = host_methods;
    if (PyType_Ready(&HostType) < 0) return nullptr;
    PyObject* m = PyModule_Create(&module_def);
    if (!m) return nullptr;
    Py_INCREF(&HostType);
    if (PyModule_AddObject(m, "Host", reinterpret_cast<PyObject*>(&HostType)) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}

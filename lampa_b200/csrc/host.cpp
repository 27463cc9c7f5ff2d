// Native host path of the eager entry points: argument checks, output and workspace allocation and the C ABI call
// behind one Python call each, bound with METH_FASTCALL (no argument-parsing layer in between).
//
// Why: a decode step or a short sequence takes the GPU 5 - 100 us, and the same steps written in Python (a dozen
// ctypes conversions, attribute reads and small tensor calls) took the host 40 - 60 us per call, so the GPU waited.
//
// Every function takes its arguments in canonical form: CUDA tensors on one device, contiguous, of the types the
// kernels read.  For anything else (and for every call that has to raise) it returns None without side effects; the
// Python layer then raises, or converts the arguments and calls again.  Nothing is kept from one call to the next
// except the address of a device's status word.
#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>

#include "../../include/lampa_b200.h"

namespace {

using at::Tensor;

constexpr int MAX_DEVICES = 64;
int32_t* g_status[MAX_DEVICES] = {nullptr};     // device int32[4], owned by lampa_b200._lib
PyObject* g_lib_module = nullptr;                // lampa_b200._lib

struct PyError {};                               // a Python exception is set

struct Call {
    int dev;
    void* stream;
    int32_t* status;
};

PyObject* lib_module() {
    if (!g_lib_module) g_lib_module = PyImport_ImportModule("lampa_b200._lib");
    if (!g_lib_module) throw PyError();
    return g_lib_module;
}

Call begin(const Tensor& t) {
    Call c;
    c.dev = t.get_device();
    c.stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c.dev).stream();
    if (c.dev >= MAX_DEVICES) throw PyError();
    if (!g_status[c.dev]) {
        PyObject* w = PyObject_CallMethod(lib_module(), "status_word_of", "i", c.dev);
        if (!w) throw PyError();
        g_status[c.dev] = (int32_t*)THPVariable_Unpack(w).data_ptr();
        Py_DECREF(w);
    }
    c.status = g_status[c.dev];
    return c;
}

void check(int rc, const char* what) {
    if (rc == LAMPA_OK) return;
    PyObject* r = PyObject_CallMethod(lib_module(), "check", "is", rc, what);   // raises
    Py_XDECREF(r);
    throw PyError();
}

// LAMPA_B200_CHECK=1: synchronise and raise on a device-side error after the call
void debug_check(const Call& c) {
    const char* e = std::getenv("LAMPA_B200_CHECK");
    if (!e || !*e || (e[0] == '0' && !e[1])) return;
    PyObject* r = PyObject_CallMethod(lib_module(), "check_status_of", "i", c.dev);
    if (!r) throw PyError();
    Py_DECREF(r);
}

int dtype_code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kBFloat16: return LAMPA_BF16;
        case at::kHalf: return LAMPA_F16;
        case at::kFloat: return LAMPA_F32;
        default: return -1;
    }
}

// The tensor behind an argument, or null for None.  `ok` turns false for anything else.
const Tensor* tensor_or_none(PyObject* o, bool& ok) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) { ok = false; return nullptr; }
    return &THPVariable_Unpack(o);
}
// A tensor the kernels can read as it is, on device `dev` (dev < 0: any, and sets it)
const Tensor* dense(PyObject* o, int& dev, bool& ok) {
    if (!THPVariable_Check(o)) { ok = false; return nullptr; }
    const Tensor* t = &THPVariable_Unpack(o);
    if (!t->is_cuda() || !t->is_contiguous() || (dev >= 0 && t->get_device() != dev)) { ok = false; return nullptr; }
    dev = t->get_device();
    return t;
}
const Tensor* dense_or_none(PyObject* o, int& dev, bool& ok) { return o == Py_None ? nullptr : dense(o, dev, ok); }

bool wants_grad(std::initializer_list<const Tensor*> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t && t->requires_grad()) return true;
    return false;
}

Tensor empty(at::IntArrayRef size, at::ScalarType st, int dev) {
    return at::detail::empty_cuda(size, st, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt);
}
void* ptr(const Tensor* t) { return t ? t->data_ptr() : nullptr; }
PyObject* none() { Py_RETURN_NONE; }

PyObject* pack(std::initializer_list<PyObject*> items) {
    PyObject* t = PyTuple_New((Py_ssize_t)items.size());
    Py_ssize_t i = 0;
    for (PyObject* o : items) PyTuple_SET_ITEM(t, i++, o);
    return t;
}
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* wrap_or_none(const Tensor& t) { if (t.defined()) return THPVariable_Wrap(t); Py_RETURN_NONE; }

// 1024-byte aligned scratch inside a fresh tensor (which the caller keeps until the launches are enqueued)
void* workspace(size_t bytes, int dev, Tensor& hold) {
    hold = empty({(int64_t)bytes + 1024}, at::kByte, dev);
    return (void*)(((uintptr_t)hold.data_ptr() + 1023) & ~(uintptr_t)1023);
}

int levels_required(int64_t T) {
    const int64_t nt = (T + 63) / 64;
    int e = 0;
    while (((int64_t)1 << e) < nt) ++e;
    return 7 + e;
}

// The reference's hint about head-first input (shared by the gated-delta entry points)
void warn_layout(int64_t T, int64_t H) {
    if (T >= H) return;
    if (PyErr_WarnFormat(PyExc_UserWarning, 1,
            "Input tensor shape suggests potential format mismatch: seq_len (%lld) < num_heads (%lld). "
            "This may indicate the inputs were passed in head-first format [B, H, T, ...] "
            "when head_first=False was specified. "
            "Please verify your input tensor format matches the expected shape [B, T, H, ...].",
            (long long)T, (long long)H) < 0) throw PyError();
}

// ---- gated-delta rules ----------------------------------------------------------------------------
struct MixerArgs {
    const Tensor *q, *k, *v, *g, *beta, *lam;
    lampa_gdn_desc d;
    int dev = -1;
};

// q, k [B,T,H,K], v [B,T,H,V], g, beta [B,T,H], lam [B,T,H,L] or None
// `entry`: called straight from a public function that refuses fp32 q/k/v and hints at head-first input
bool mixer_args(PyObject* const* a, MixerArgs& m, bool entry) {
    bool ok = true;
    m.q = dense(a[0], m.dev, ok); m.k = dense(a[1], m.dev, ok); m.v = dense(a[2], m.dev, ok);
    m.g = dense(a[3], m.dev, ok); m.beta = dense(a[4], m.dev, ok); m.lam = dense_or_none(a[5], m.dev, ok);
    if (!ok || m.q->dim() != 4 || m.v->dim() != 4 || m.g->dim() != 3 || m.k->sizes() != m.q->sizes() || m.beta->sizes() != m.g->sizes()) return false;
    const auto qs = m.q->sizes(), vs = m.v->sizes(), gs = m.g->sizes();
    if (vs.slice(0, 3) != qs.slice(0, 3) || gs != qs.slice(0, 3)) return false;
    if (m.lam && (m.lam->dim() != 4 || m.lam->sizes().slice(0, 3) != gs)) return false;
    const int dt = dtype_code(*m.q), gdt = dtype_code(*m.g), ldt = m.lam ? dtype_code(*m.lam) : LAMPA_F32;
    if (dt < 0 || (entry && dt == LAMPA_F32) || gdt < 0 || ldt < 0) return false;
    if (m.k->scalar_type() != m.q->scalar_type() || m.v->scalar_type() != m.q->scalar_type() || m.beta->scalar_type() != m.g->scalar_type()) return false;
    for (int64_t s : qs) if (s <= 0 || s > INT32_MAX) return false;
    m.d.B = (int32_t)qs[0]; m.d.T = (int32_t)qs[1]; m.d.H = (int32_t)qs[2]; m.d.K = (int32_t)qs[3]; m.d.V = (int32_t)vs[3];
    m.d.L = m.lam ? (int32_t)m.lam->size(3) : 0;
    m.d.nseq = 0;
    m.d.qkv_dtype = dt; m.d.gb_dtype = gdt; m.d.lam_dtype = ldt;
    m.d.use_l2norm = 1; m.d.scale = 1.f;
    return m.d.K <= 256;
}

// (o, states, counts, arrivals): the counts and, in the word behind them, the arrival counter of the decode steps
PyObject* with_words(const Tensor& o, const Tensor& states, const Tensor& words, at::IntArrayRef counts) {
    const int64_t n = words.numel() - 1;
    return pack({wrap(o), wrap(states), wrap(words.narrow(0, 0, n).view(counts)), wrap(words.narrow(0, n, 1))});
}

// gdn(q, k, v, g, beta, lam|None, h0|None, cu|None, out_perm|None, scale|None, l2norm, want_state, entry)
//   plain rule: (o, final state | None); hierarchical: (o, None), or (o, states, counts, arrivals) with want_state
PyObject* gdn(PyObject* const* a) {
    MixerArgs m;
    const bool entry = a[12] == Py_True;
    if (!mixer_args(a, m, entry)) return none();
    bool ok = true;
    const Tensor* h0 = dense_or_none(a[6], m.dev, ok);
    const Tensor* cu = dense_or_none(a[7], m.dev, ok);
    const Tensor* perm = dense_or_none(a[8], m.dev, ok);
    if (!ok || (entry && wants_grad({m.q, m.k, m.v, m.g, m.beta, m.lam, h0}))) return none();
    if (cu && (cu->scalar_type() != at::kLong || cu->dim() != 1 || cu->numel() < 2 || m.d.B != 1)) return none();
    if (perm && (perm->scalar_type() != at::kLong || perm->dim() != 1 || perm->numel() > (int64_t)m.d.B * m.d.T)) return none();
    m.d.nseq = cu ? (int32_t)cu->numel() - 1 : 0;
    const int64_t N = cu ? m.d.nseq : m.d.B;
    if (h0 && (h0->scalar_type() != at::kFloat || h0->sizes() != at::IntArrayRef({N, (int64_t)m.d.H, (int64_t)m.d.K, (int64_t)m.d.V}))) return none();
    if (m.lam && !cu && m.d.L < levels_required(m.d.T)) return none();
    m.d.use_l2norm = a[10] == Py_True;
    if (!m.lam) m.d.scale = a[9] == Py_None ? (float)std::pow((double)m.d.K, -0.5) : (float)PyFloat_AsDouble(a[9]);
    if (PyErr_Occurred()) throw PyError();
    const bool want_state = a[11] == Py_True;
    if (entry) warn_layout(m.d.T, m.d.H);

    const Call c = begin(*m.q);
    size_t bytes = 0;
    check(lampa_gdn_workspace_bytes(&m.d, &bytes), "lampa_gdn_workspace_bytes");
    Tensor hold, o = empty({m.d.B, m.d.T, m.d.H, m.d.V}, m.q->scalar_type(), m.dev);
    void* ws = workspace(bytes, m.dev, hold);
    if (!m.lam) {
        Tensor ht;
        if (want_state) ht = empty({N, m.d.H, m.d.K, m.d.V}, at::kFloat, m.dev);
        check(lampa_gdn_fwd(&m.d, ptr(m.q), ptr(m.k), ptr(m.v), ptr(m.g), ptr(m.beta), (const float*)ptr(h0), (const int64_t*)ptr(cu),
                            o.data_ptr(), want_state ? (float*)ht.data_ptr() : nullptr, ws, bytes, c.status, c.stream), "lampa_gdn_fwd");
        debug_check(c);
        return pack({wrap(o), wrap_or_none(ht)});
    }
    if (perm)
        check(lampa_hgdn_fwd_scatter(&m.d, ptr(m.q), ptr(m.k), ptr(m.v), ptr(m.g), ptr(m.beta), ptr(m.lam), (const int64_t*)ptr(cu),
                                     (const int64_t*)ptr(perm), perm->numel(), o.data_ptr(), ws, bytes, c.status, c.stream), "lampa_hgdn_fwd");
    else
        check(lampa_hgdn_fwd(&m.d, ptr(m.q), ptr(m.k), ptr(m.v), ptr(m.g), ptr(m.beta), ptr(m.lam), (const int64_t*)ptr(cu),
                             o.data_ptr(), ws, bytes, c.status, c.stream), "lampa_hgdn_fwd");
    if (!want_state) {
        debug_check(c);
        return pack({wrap(o), none()});
    }
    Tensor states = empty({N, m.d.H, m.d.K, m.d.V, m.d.L}, at::kFloat, m.dev), words = empty({N * m.d.L + 1}, at::kInt, m.dev);
    int32_t* counts = (int32_t*)words.data_ptr();
    check(lampa_hgdn_final_state_counted(&m.d, ptr(m.k), ptr(m.v), ptr(m.g), ptr(m.beta), (const int64_t*)ptr(cu), ws, bytes,
                                         (float*)states.data_ptr(), counts, counts + N * m.d.L, c.status, c.stream), "lampa_hgdn_final_state");
    debug_check(c);
    return with_words(o, states, words, {N, m.d.L});
}

// prefill(q, k, v, g, beta, lam, entry) -> (o, states, counts [L], arrivals)
PyObject* prefill(PyObject* const* a) {
    MixerArgs m;
    const bool entry = a[6] == Py_True;
    if (!mixer_args(a, m, entry) || !m.lam || (entry && wants_grad({m.q, m.k, m.v, m.g, m.beta, m.lam}))) return none();
    const int T0 = m.d.T - m.d.T % 64;
    if (T0 > 0 && m.d.L < levels_required(T0)) return none();
    if (entry) warn_layout(m.d.T, m.d.H);
    const Call c = begin(*m.q);
    lampa_gdn_desc whole = m.d;
    whole.T = T0;
    size_t bytes = 0;
    check(lampa_gdn_workspace_bytes(&whole, &bytes), "lampa_gdn_workspace_bytes");
    Tensor hold, o = empty({m.d.B, m.d.T, m.d.H, m.d.V}, m.q->scalar_type(), m.dev);
    void* ws = workspace(bytes, m.dev, hold);
    Tensor states = empty({m.d.B, m.d.H, m.d.K, m.d.V, m.d.L}, at::kFloat, m.dev), words = empty({m.d.L + 1}, at::kInt, m.dev);
    int32_t* counts = (int32_t*)words.data_ptr();
    check(lampa_hgdn_prefill_counted(&m.d, ptr(m.q), ptr(m.k), ptr(m.v), ptr(m.g), ptr(m.beta), ptr(m.lam), o.data_ptr(), ws, bytes,
                                     (float*)states.data_ptr(), counts, counts + m.d.L, c.status, c.stream), "lampa_hgdn_prefill");
    debug_check(c);
    return with_words(o, states, words, {m.d.L});
}

// step(q, k, v, g, beta, lam, states, counts, arrivals, entry): one token per row, q [B,1,H,K] (or [B,H,K]) -> o of v's shape
PyObject* step(PyObject* const* a) {
    bool ok = true;
    int dev = -1;
    const bool entry = a[9] == Py_True;
    const Tensor *q = dense(a[0], dev, ok), *k = dense(a[1], dev, ok), *v = dense(a[2], dev, ok), *g = dense(a[3], dev, ok),
                 *beta = dense(a[4], dev, ok), *lam = dense(a[5], dev, ok), *states = dense(a[6], dev, ok),
                 *counts = dense(a[7], dev, ok), *arrivals = dense(a[8], dev, ok);
    if (!ok || (entry && wants_grad({q, k, v, g, beta, lam}))) return none();
    const int64_t nd = q->dim();
    if ((nd != 3 && nd != 4) || (nd == 4 && q->size(1) != 1) || v->dim() != nd || lam->dim() != nd || g->dim() != nd - 1) return none();
    if (k->sizes() != q->sizes() || beta->sizes() != g->sizes() || v->sizes().slice(0, nd - 1) != q->sizes().slice(0, nd - 1) ||
        lam->sizes().slice(0, nd - 1) != g->sizes() || g->sizes() != q->sizes().slice(0, nd - 1)) return none();
    const int64_t B = q->size(0), H = q->size(nd - 2), K = q->size(nd - 1), V = v->size(nd - 1), L = lam->size(nd - 1);
    const int dt = dtype_code(*q), gdt = dtype_code(*g), ldt = dtype_code(*lam);
    if (B <= 0 || H <= 0 || dt < 0 || (entry && dt == LAMPA_F32) || gdt < 0 || ldt < 0) return none();
    if (k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || beta->scalar_type() != g->scalar_type()) return none();
    if (states->scalar_type() != at::kFloat || states->sizes() != at::IntArrayRef({B, H, K, V, L}) || counts->scalar_type() != at::kInt ||
        counts->numel() < L || arrivals->scalar_type() != at::kInt || arrivals->numel() < 1) return none();
    if (entry) warn_layout(1, H);
    const Call c = begin(*q);
    lampa_gdn_desc d;
    d.B = (int32_t)B; d.T = 1; d.H = (int32_t)H; d.K = (int32_t)K; d.V = (int32_t)V; d.L = (int32_t)L; d.nseq = 0;
    d.qkv_dtype = dt; d.gb_dtype = gdt; d.lam_dtype = ldt; d.use_l2norm = 1; d.scale = 1.f;
    Tensor o = empty(v->sizes(), q->scalar_type(), dev);
    check(lampa_hgdn_step_counted(&d, ptr(q), ptr(k), ptr(v), ptr(g), ptr(beta), ptr(lam), (float*)states->data_ptr(),
                                  (int32_t*)counts->data_ptr(), (int32_t*)arrivals->data_ptr(), o.data_ptr(), c.status, c.stream),
          "lampa_hgdn_step_counted");
    debug_check(c);
    return wrap(o);
}

#include "host_lsh.inc"
#include "host_model.inc"
#include "host_hept.inc"

template <PyObject* (*F)(PyObject* const*), int N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != N) { PyErr_Format(PyExc_TypeError, "expected %d arguments, got %d", N, (int)n); return nullptr; }
    try {
        return F(args);
    } catch (const PyError&) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "lampa_b200 host call failed");
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}
#define ENTRY(name, n) {#name, (PyCFunction)(void*)&entry<name, n>, METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    ENTRY(gdn, 13), ENTRY(prefill, 7), ENTRY(step, 10),
    ENTRY(lsh_hash, 8), ENTRY(segsort, 4), ENTRY(permute_rows, 5), ENTRY(invert_perm, 1), ENTRY(bucket_sort, 4), ENTRY(ordering, 3),
    ENTRY(model_forward, 6), ENTRY(region_inputs, 3), ENTRY(hept_core, 11),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Native host path of lampa_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module_def); }

// The calls a decode loop makes, as a CPython extension over the C ABI: arguments go from Python objects straight to
// the entry points of krk_cuda.h. A small matrix takes 5 us on the device; through ctypes a call cost 9-14 us of
// interpreter time (argument objects, a Python-level current_stream(), the foreign-function layer), so a token of
// eager calls ran at the host's pace. Nothing is computed or kept here: kraken_b200/capi.py is the interface, and an error code
// of the library becomes the exception capi registers.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>

#include "krk_cuda.h"

namespace {

PyObject *g_raise = nullptr;     // capi's (rc, where) -> raises
PyObject *g_address = nullptr;   // capi's ctypes pointer -> int

PyObject *fail(int rc, const char *where) {
    PyObject *r = PyObject_CallFunction(g_raise, "is", rc, where);
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed with %d", where, rc);
    return nullptr;
}

// One argument list; a conversion that fails leaves a Python error set and `ok` false.
struct Args {
    PyObject *const *a;
    bool ok = true;
    int64_t i(int k) {
        const long long v = PyLong_AsLongLong(a[k]);
        if (v == -1 && PyErr_Occurred()) ok = false;
        return v;
    }
    // An address: an integer, None, or whatever ctypes takes for a void pointer.
    uintptr_t addr(int k) {
        if (a[k] == Py_None) return 0;
        PyObject *o = PyLong_Check(a[k]) ? nullptr : PyObject_CallOneArg(g_address, a[k]);
        if (!o && !PyLong_Check(a[k])) {
            ok = false;
            return 0;
        }
        const uintptr_t v = (uintptr_t)PyLong_AsUnsignedLongLongMask(o ? o : a[k]);
        Py_XDECREF(o);
        if (PyErr_Occurred()) ok = false;
        return v;
    }
    void *backend(int k) {
        if (!PyLong_Check(a[k])) {
            if (ok) PyErr_SetString(PyExc_TypeError, "the backend is closed");
            ok = false;
            return nullptr;
        }
        return (void *)addr(k);
    }
    float f(int k) {
        const double v = PyFloat_AsDouble(a[k]);
        if (v == -1.0 && PyErr_Occurred()) ok = false;
        return (float)v;
    }
    bool b(int k) {
        const int v = PyObject_IsTrue(a[k]);
        if (v < 0) ok = false;
        return v > 0;
    }
    const at::Tensor *tensor(PyObject *o) {
        if (!THPVariable_Check(o)) {
            if (ok) PyErr_Format(PyExc_TypeError, "expected a torch tensor, got %s", Py_TYPE(o)->tp_name);
            ok = false;
            return nullptr;
        }
        return &THPVariable_Unpack(o);
    }
    const at::Tensor *t(int k) { return tensor(a[k]); }
    static void *ptr(const at::Tensor *x) { return x ? const_cast<void *>(x->const_data_ptr()) : nullptr; }
    void *p(int k) { return ptr(t(k)); }
    const at::Tensor *t_or_none(int k) { return a[k] == Py_None ? nullptr : t(k); }
    void *stream(int k) {
        if (a[k] == Py_None) return c10::cuda::getCurrentCUDAStream().stream();
        PyObject *s = PyObject_GetAttrString(a[k], "cuda_stream");
        if (!s) {
            ok = false;
            return nullptr;
        }
        void *v = PyLong_AsVoidPtr(s);
        Py_DECREF(s);
        if (!v && PyErr_Occurred()) ok = false;
        return v;
    }
};

at::Tensor empty_like_device(const at::Tensor &like, at::IntArrayRef sizes, at::ScalarType type) {
    return at::empty(sizes, like.options().dtype(type).requires_grad(false));
}

#define KRK_NARGS(count, name)                                                                                    \
    if (n != (count)) {                                                                                           \
        PyErr_Format(PyExc_TypeError, name " takes %d arguments, got %zd", (count), n);                           \
        return nullptr;                                                                                           \
    }
#define KRK_TRY try {
#define KRK_CATCH                                                                                                 \
    }                                                                                                             \
    catch (const std::exception &e) {                                                                             \
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());                                     \
        return nullptr;                                                                                           \
    }

PyObject *set_raise(PyObject *, PyObject *f) {
    Py_INCREF(f);
    Py_XSETREF(g_raise, f);
    Py_RETURN_NONE;
}
PyObject *set_address(PyObject *, PyObject *f) {
    Py_INCREF(f);
    Py_XSETREF(g_address, f);
    Py_RETURN_NONE;
}

PyObject *gemv(PyObject *, PyObject *const *a, Py_ssize_t n) {   // x, w, wt, n_out, n_in, out, accumulate, stream
    KRK_NARGS(8, "gemv")
    KRK_TRY
    Args g{a};
    const at::Tensor *x = g.t(0);
    const void *w = g.p(1);
    const int wt = (int)g.i(2);
    const int64_t n_out = g.i(3), n_in = g.i(4);
    const bool acc = g.b(6);
    const at::Tensor *out = g.t_or_none(5);
    void *st = g.stream(7);
    if (!g.ok) return nullptr;
    const int64_t rows = x->dim() == 1 ? 1 : x->size(0);
    at::Tensor made;
    if (!out) {
        if (acc) {
            PyErr_SetString(PyExc_ValueError, "accumulate needs an existing output");
            return nullptr;
        }
        made = empty_like_device(*x, {rows, n_out}, at::kFloat);
        out = &made;
    }
    void *y = Args::ptr(out), *xp = Args::ptr(x);
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_gemv(y, xp, w, wt, n_out, n_in, rows, acc, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "gemv");
    if (made.defined()) return THPVariable_Wrap(made);
    Py_INCREF(a[5]);
    return a[5];
    KRK_CATCH
}

// A list or tuple argument of up to KRK_CUDA_MAX_GROUP items, as a borrowed fast sequence.
struct Seq {
    PyObject *s;
    Py_ssize_t n = 0;
    explicit Seq(PyObject *o) : s(PySequence_Fast(o, "expected a sequence")) {
        if (s) n = PySequence_Fast_GET_SIZE(s);
    }
    ~Seq() { Py_XDECREF(s); }
    PyObject *operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(s, i); }
};

PyObject *gemv_group(PyObject *, PyObject *const *a, Py_ssize_t n) {   // xs, ws, wts, n_outs, n_in, outs, fuse, stream
    KRK_NARGS(8, "gemv_group")
    KRK_TRY
    Args g{a};
    Seq xs(a[0]), ws(a[1]), wts(a[2]), nos(a[3]);
    if (!xs.s || !ws.s || !wts.s || !nos.s) return nullptr;
    const Py_ssize_t m = ws.n;
    if (m > KRK_CUDA_MAX_GROUP) return fail(KRK_CUDA_EARG, "gemv_group");
    if (xs.n != m || wts.n != m || nos.n != m) {
        PyErr_SetString(PyExc_ValueError, "gemv_group: argument lists of unequal length");
        return nullptr;
    }
    void *y[KRK_CUDA_MAX_GROUP];
    const void *x[KRK_CUDA_MAX_GROUP], *w[KRK_CUDA_MAX_GROUP];
    int wt[KRK_CUDA_MAX_GROUP];
    int64_t n_out[KRK_CUDA_MAX_GROUP];
    PyObject *outs = a[5];
    if (outs == Py_None) {
        outs = PyList_New(m);
        if (!outs) return nullptr;
    } else {
        Py_INCREF(outs);
    }
    for (Py_ssize_t i = 0; i < m && g.ok; i++) {
        const at::Tensor *wi = g.tensor(ws[i]);
        x[i] = Args::ptr(g.tensor(xs[i]));
        w[i] = Args::ptr(wi);
        Args item{PySequence_Fast_ITEMS(wts.s)}, size{PySequence_Fast_ITEMS(nos.s)};
        wt[i] = (int)item.i((int)i);
        n_out[i] = size.i((int)i);
        g.ok = g.ok && item.ok && size.ok;
        if (g.ok && a[5] == Py_None) PyList_SET_ITEM(outs, i, THPVariable_Wrap(empty_like_device(*wi, {n_out[i]}, at::kFloat)));
    }
    const int64_t n_in = g.i(4);
    const bool fuse = g.b(6);
    void *st = g.stream(7);
    if (g.ok) {
        Seq ys(outs);
        if (!ys.s || ys.n != m) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "gemv_group: as many outputs as matrices are needed");
            g.ok = false;
        }
        for (Py_ssize_t i = 0; i < m && g.ok; i++) y[i] = Args::ptr(g.tensor(ys[i]));
    }
    if (!g.ok) {
        Py_DECREF(outs);
        return nullptr;
    }
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_gemv_group(y, x, w, wt, n_out, n_in, (int)m, fuse, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) {
        Py_DECREF(outs);
        return fail(rc, "gemv_group");
    }
    return outs;
    KRK_CATCH
}

PyObject *gemm(PyObject *, PyObject *const *a, Py_ssize_t n) {   // x, w, wt, n_out, n_in, out, workspace, stream
    KRK_NARGS(8, "gemm")
    KRK_TRY
    Args g{a};
    const at::Tensor *x = g.t(0);
    const void *w = g.p(1);
    const int wt = (int)g.i(2);
    const int64_t n_out = g.i(3), n_in = g.i(4);
    const at::Tensor *out = g.t_or_none(5), *ws = g.t_or_none(6);
    void *st = g.stream(7);
    if (!g.ok) return nullptr;
    const int64_t rows = x->size(0);
    const int xt = x->scalar_type() == at::kHalf ? KRK_CUDA_X_F16 : KRK_CUDA_X_F32;
    at::Tensor made_ws, made;
    if (!ws) {
        const size_t need = krk_cuda_gemm_workspace_bytes(xt, n_out, n_in, rows);
        if (need) {
            made_ws = empty_like_device(*x, {(int64_t)need}, at::kByte);
            ws = &made_ws;
        }
    }
    if (!out) {
        made = empty_like_device(*x, {rows, n_out}, at::kFloat);
        out = &made;
    }
    void *y = Args::ptr(out), *xp = Args::ptr(x), *wp = Args::ptr(ws);
    const size_t ws_bytes = ws ? (size_t)ws->numel() : 0;
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_gemm(y, xp, xt, w, wt, n_out, n_in, rows, wp, ws_bytes, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "gemm");
    if (made.defined()) return THPVariable_Wrap(made);
    Py_INCREF(a[5]);
    return a[5];
    KRK_CATCH
}

PyObject *silu_mul(PyObject *, PyObject *const *a, Py_ssize_t n) {   // gate, up, out, stream
    KRK_NARGS(4, "silu_mul")
    KRK_TRY
    Args g{a};
    const at::Tensor *gate = g.t(0), *out = g.t_or_none(2);
    const void *up = g.p(1);
    void *st = g.stream(3);
    if (!g.ok) return nullptr;
    at::Tensor made;
    if (!out) {
        made = at::empty_like(*gate, gate->options().requires_grad(false));   // with its strides: the kernel goes through the memory as it lies
        out = &made;
    }
    void *y = Args::ptr(out), *gp = Args::ptr(gate);
    const int64_t count = gate->numel();
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_silu_mul(y, gp, up, count, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "silu_mul");
    if (made.defined()) return THPVariable_Wrap(made);
    Py_INCREF(a[2]);
    return a[2];
    KRK_CATCH
}

PyObject *embed(PyObject *, PyObject *const *a, Py_ssize_t n) {   // table, wt, n_vocab, n_embd, tokens, out, stream
    KRK_NARGS(7, "embed")
    KRK_TRY
    Args g{a};
    const at::Tensor *table = g.t(0), *tokens = g.t(4), *out = g.t_or_none(5);
    const int wt = (int)g.i(1);
    const int64_t n_vocab = g.i(2), n_embd = g.i(3);
    void *st = g.stream(6);
    if (!g.ok) return nullptr;
    at::Tensor made;
    if (!out) {
        made = empty_like_device(*table, {tokens->numel(), n_embd}, at::kFloat);
        out = &made;
    }
    void *y = Args::ptr(out), *tp = Args::ptr(table), *ip = Args::ptr(tokens);
    const int64_t n_tok = tokens->numel();
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_embed(y, tp, wt, n_vocab, n_embd, ip, n_tok, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "embed");
    if (made.defined()) return THPVariable_Wrap(made);
    Py_INCREF(a[5]);
    return a[5];
    KRK_CATCH
}

// logits, k, pen_mask, rep_pen, softcap, temp, want_mass, workspace, stream -> (ids, vals, mass or None)
PyObject *logits_topk(PyObject *, PyObject *const *a, Py_ssize_t n) {
    KRK_NARGS(9, "logits_topk")
    KRK_TRY
    Args g{a};
    const at::Tensor *logits = g.t(0), *pen = g.t_or_none(2), *ws = g.t_or_none(7);
    const int64_t k = g.i(1);
    const float rep_pen = g.f(3), softcap = g.f(4), temp = g.f(5);
    const bool want_mass = g.b(6);
    void *st = g.stream(8);
    if (!g.ok) return nullptr;
    at::Tensor made_ws, mass;
    if (!ws) {
        const size_t need = krk_cuda_logits_topk_workspace_bytes(logits->numel(), (int)k);
        made_ws = empty_like_device(*logits, {(int64_t)(need > 16 ? need : 16)}, at::kByte);
        ws = &made_ws;
    }
    at::Tensor ids = empty_like_device(*logits, {k}, at::kInt), vals = empty_like_device(*logits, {k}, at::kFloat);
    if (want_mass) mass = empty_like_device(*logits, {1}, at::kFloat);
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_logits_topk(Args::ptr(logits), logits->numel(), (int)k, Args::ptr(pen), rep_pen, softcap, temp, Args::ptr(&ids),
                                                     Args::ptr(&vals), want_mass ? Args::ptr(&mass) : nullptr, Args::ptr(ws), (size_t)ws->numel(), st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "logits_topk");
    PyObject *r = PyTuple_New(3);
    if (!r) return nullptr;
    PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(ids));
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(vals));
    if (want_mass) {
        PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(mass));
    } else {
        Py_INCREF(Py_None);
        PyTuple_SET_ITEM(r, 2, Py_None);
    }
    return r;
    KRK_CATCH
}

// The krk_cuda_expert_bank behind capi's ctypes structure (which offers its memory as a buffer).
struct Bank {
    Py_buffer view{};
    bool ok;
    explicit Bank(PyObject *o) : ok(PyObject_GetBuffer(o, &view, PyBUF_SIMPLE) == 0) {
        if (ok && view.len < (Py_ssize_t)sizeof(krk_cuda_expert_bank)) {
            PyErr_SetString(PyExc_TypeError, "expected an ExpertBank");
            PyBuffer_Release(&view);
            ok = false;
        }
    }
    ~Bank() {
        if (ok) PyBuffer_Release(&view);
    }
    const krk_cuda_expert_bank *get() const { return static_cast<const krk_cuda_expert_bank *>(view.buf); }
};

PyObject *moe_ffn(PyObject *, PyObject *const *a, Py_ssize_t n) {   // x, ids, wts, bank, out, workspace, stream
    KRK_NARGS(7, "moe_ffn")
    KRK_TRY
    Args g{a};
    Bank bank(a[3]);
    if (!bank.ok) return nullptr;
    const at::Tensor *x = g.t(0), *ids = g.t(1), *wts = g.t(2), *out = g.t_or_none(4), *ws = g.t_or_none(5);
    void *st = g.stream(6);
    if (!g.ok) return nullptr;
    const int64_t n_tok = ids->size(0);
    const int k = (int)ids->size(1);
    at::Tensor made, made_ws;
    if (!ws) {
        const size_t need = krk_cuda_moe_workspace_bytes(bank.get(), k, n_tok);
        made_ws = empty_like_device(*x, {(int64_t)(need > 16 ? need : 16)}, at::kByte);
        ws = &made_ws;
    }
    if (!out) {
        made = empty_like_device(*x, {n_tok, bank.get()->n_embd}, at::kFloat);
        out = &made;
    }
    void *y = Args::ptr(out), *wp = Args::ptr(ws);
    const size_t ws_bytes = (size_t)ws->numel();
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_moe_ffn(y, Args::ptr(x), Args::ptr(ids), Args::ptr(wts), bank.get(), k, n_tok, wp, ws_bytes, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "moe_ffn");
    if (made.defined()) return THPVariable_Wrap(made);
    Py_INCREF(a[4]);
    return a[4];
    KRK_CATCH
}

PyObject *moe_ffn_routed(PyObject *, PyObject *const *a, Py_ssize_t n) {   // x, logits, k, bank, out, workspace, stream -> (y, ids, wts)
    KRK_NARGS(7, "moe_ffn_routed")
    KRK_TRY
    Args g{a};
    Bank bank(a[3]);
    if (!bank.ok) return nullptr;
    const at::Tensor *x = g.t(0), *logits = g.t(1), *out = g.t_or_none(4), *ws = g.t_or_none(5);
    const int64_t k = g.i(2);
    void *st = g.stream(6);
    if (!g.ok) return nullptr;
    const int64_t n_tok = logits->size(0), n_expert = logits->size(1);
    at::Tensor ids = empty_like_device(*x, {n_tok, k}, at::kInt), wts = empty_like_device(*x, {n_tok, k}, at::kFloat), made, made_ws;
    if (!ws) {
        const size_t need = krk_cuda_moe_workspace_bytes(bank.get(), (int)k, n_tok);
        made_ws = empty_like_device(*x, {(int64_t)(need > 16 ? need : 16)}, at::kByte);
        ws = &made_ws;
    }
    if (!out) {
        made = empty_like_device(*x, {n_tok, bank.get()->n_embd}, at::kFloat);
        out = &made;
    }
    void *y = Args::ptr(out), *wp = Args::ptr(ws);
    const size_t ws_bytes = (size_t)ws->numel();
    int rc;
    Py_BEGIN_ALLOW_THREADS rc = krk_cuda_moe_ffn_routed(y, Args::ptr(x), Args::ptr(logits), (int)n_expert, Args::ptr(&ids), Args::ptr(&wts),
                                                        bank.get(), (int)k, n_tok, wp, ws_bytes, st);
    Py_END_ALLOW_THREADS
    if (rc != 0) return fail(rc, "moe_ffn_routed");
    PyObject *r = PyTuple_New(3);
    if (!r) return nullptr;
    if (made.defined()) {
        PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(made));
    } else {
        Py_INCREF(a[4]);
        PyTuple_SET_ITEM(r, 0, a[4]);
    }
    PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(ids));
    PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(wts));
    return r;
    KRK_CATCH
}

// ---- the CudaBackend object: device and host addresses are plain integers -------------------------------------

PyObject *backend_upload(PyObject *, PyObject *const *a, Py_ssize_t n) {   // be, dst, host_src, bytes, off
    KRK_NARGS(5, "backend_upload")
    Args g{a};
    void *be = g.backend(0), *dst = (void *)g.addr(1);
    const void *src = (const void *)g.addr(2);
    const size_t bytes = (size_t)g.i(3), off = (size_t)g.i(4);
    if (!g.ok) return nullptr;
    Py_BEGIN_ALLOW_THREADS krk_cuda_backend_upload(be, dst, src, bytes, off);
    Py_END_ALLOW_THREADS Py_RETURN_NONE;
}
PyObject *backend_download(PyObject *, PyObject *const *a, Py_ssize_t n) {   // be, host_dst, src, bytes, off
    KRK_NARGS(5, "backend_download")
    Args g{a};
    void *be = g.backend(0), *dst = (void *)g.addr(1);
    const void *src = (const void *)g.addr(2);
    const size_t bytes = (size_t)g.i(3), off = (size_t)g.i(4);
    if (!g.ok) return nullptr;
    Py_BEGIN_ALLOW_THREADS krk_cuda_backend_download(be, dst, src, bytes, off);
    Py_END_ALLOW_THREADS Py_RETURN_NONE;
}
PyObject *backend_gemm(PyObject *, PyObject *const *a, Py_ssize_t n) {   // be, out, x, w, wt, n_out, n_in, rows
    KRK_NARGS(8, "backend_gemm")
    Args g{a};
    void *be = g.backend(0), *out = (void *)g.addr(1);
    const void *x = (const void *)g.addr(2), *w = (const void *)g.addr(3);
    const int wt = (int)g.i(4);
    const int64_t n_out = g.i(5), n_in = g.i(6), rows = g.i(7);
    if (!g.ok) return nullptr;
    Py_BEGIN_ALLOW_THREADS krk_cuda_backend_gemm(be, out, x, w, wt, n_out, n_in, rows);
    Py_END_ALLOW_THREADS Py_RETURN_NONE;
}
PyObject *backend_gemm_accumulate(PyObject *, PyObject *const *a, Py_ssize_t n) {   // be, dst, x, w, wt, n_out, n_in, rows
    KRK_NARGS(8, "backend_gemm_accumulate")
    Args g{a};
    void *be = g.backend(0), *dst = (void *)g.addr(1);
    const void *x = (const void *)g.addr(2), *w = (const void *)g.addr(3);
    const int wt = (int)g.i(4);
    const int64_t n_out = g.i(5), n_in = g.i(6), rows = g.i(7);
    if (!g.ok) return nullptr;
    int r;
    Py_BEGIN_ALLOW_THREADS r = krk_cuda_backend_gemm_accumulate(be, dst, x, w, wt, n_out, n_in, rows);
    Py_END_ALLOW_THREADS
    return PyBool_FromLong(r);
}
// be, outs, x, ws, wt, n_outs, n_in, rows, silu, wts or None, xs or None -> (ran in one launch, silu folded)
PyObject *backend_gemm_group(PyObject *, PyObject *const *a, Py_ssize_t n) {
    KRK_NARGS(11, "backend_gemm_group")
    KRK_TRY
    Args g{a};
    Seq outs(a[1]), ws(a[3]), nos(a[5]);
    if (!outs.s || !ws.s || !nos.s) return nullptr;
    const size_t m = (size_t)ws.n;
    PyObject *empty = PyTuple_New(0);
    Seq wts(a[9] == Py_None ? empty : a[9]), xs(a[10] == Py_None ? empty : a[10]);
    Py_DECREF(empty);
    if (!wts.s || !xs.s) return nullptr;
    if ((size_t)outs.n != m || (size_t)nos.n != m || (a[9] != Py_None && (size_t)wts.n != m) || (a[10] != Py_None && (size_t)xs.n != m)) {
        PyErr_SetString(PyExc_ValueError, "gemm_group: argument lists of unequal length");
        return nullptr;
    }
    std::vector<void *> y(m);
    std::vector<const void *> w(m), x(m);
    std::vector<int64_t> n_out(m);
    std::vector<int> wt(m);
    Args fo{PySequence_Fast_ITEMS(outs.s)}, fw{PySequence_Fast_ITEMS(ws.s)}, fn{PySequence_Fast_ITEMS(nos.s)}, ft{PySequence_Fast_ITEMS(wts.s)},
        fx{PySequence_Fast_ITEMS(xs.s)};
    for (size_t i = 0; i < m; i++) {
        y[i] = (void *)fo.addr((int)i);
        w[i] = (const void *)fw.addr((int)i);
        n_out[i] = fn.i((int)i);
        if (a[9] != Py_None) wt[i] = (int)ft.i((int)i);
        if (a[10] != Py_None) x[i] = (const void *)fx.addr((int)i);
    }
    void *be = g.backend(0);
    const void *x0 = (const void *)g.addr(2);
    const int wt0 = (int)g.i(4);
    const int64_t n_in = g.i(6), rows = g.i(7);
    const bool silu = g.b(8);
    if (!g.ok || !fo.ok || !fw.ok || !fn.ok || !ft.ok || !fx.ok) return nullptr;
    int fused = 0, ran;
    Py_BEGIN_ALLOW_THREADS ran = krk_cuda_backend_gemm_group_ex(be, y.data(), x0, w.data(), wt0, n_out.data(), n_in, (int)m, rows, silu, &fused,
                                                                a[9] != Py_None ? wt.data() : nullptr, a[10] != Py_None ? x.data() : nullptr);
    Py_END_ALLOW_THREADS
    return PyTuple_Pack(2, ran ? Py_True : Py_False, fused ? Py_True : Py_False);
    KRK_CATCH
}

#define KRK_FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"set_raise", set_raise, METH_O, nullptr},
                         {"set_address", set_address, METH_O, nullptr},
                         KRK_FAST(gemv),
                         KRK_FAST(gemv_group),
                         KRK_FAST(gemm),
                         KRK_FAST(silu_mul),
                         KRK_FAST(embed),
                         KRK_FAST(logits_topk),
                         KRK_FAST(moe_ffn),
                         KRK_FAST(moe_ffn_routed),
                         KRK_FAST(backend_upload),
                         KRK_FAST(backend_download),
                         KRK_FAST(backend_gemm),
                         KRK_FAST(backend_gemm_accumulate),
                         KRK_FAST(backend_gemm_group),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}   // namespace

PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&module); }

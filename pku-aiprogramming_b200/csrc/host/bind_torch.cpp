// The functions of functional.py over torch CUDA tensors, as one CPython extension (`_ttorch`): argument checks,
// output allocation and the C-ABI call without a Python object per pointer.
//
// A call on small tensors is all host work: through ctypes it took 30-40 us (checks in Python, one ctypes object
// per pointer, a device context manager, torch.empty through the dispatcher) against 3-10 us of kernels.
//
// Every function takes its arguments positionally, in the order functional.py passes them, and returns
//   its result;
//   None  -- an argument does not fit; functional.py then finds out which and words the error;
//   int   -- the status of a C-ABI call that failed; functional.py raises it through capi.check.
// The GIL is released around the C-ABI call, as ctypes does.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "tt_attn.h"

namespace {

using at::Tensor;

// A contiguous CUDA tensor argument; null where the argument is not one.
const Tensor* cuda_arg(PyObject* o) {
    if (!THPVariable_Check(o)) return nullptr;
    const Tensor& t = THPVariable_Unpack(o);
    return (t.is_cuda() && t.is_contiguous()) ? &t : nullptr;
}
// An optional buffer argument: None gives null; `ok` turns false for anything that is not a tensor.
const Tensor* opt_arg(PyObject* o, bool* ok) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_Check(o)) {
        *ok = false;
        return nullptr;
    }
    return &THPVariable_Unpack(o);
}
void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const Tensor* t) { return t ? t->data_ptr() : nullptr; }

bool float_type(const Tensor& t) { return t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat; }
int tt_type(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? TT_BF16 : TT_F32; }
bool same_shape(const Tensor& a, const Tensor& b) { return a.sizes() == b.sizes(); }

Tensor make(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
Tensor make_like(const Tensor& t) { return make(t.sizes(), t.scalar_type(), t); }
Tensor make_bytes(size_t n, const Tensor& like) { return make({(int64_t)n}, at::kByte, like); }

// The caller's device for the time of the call: allocation, current stream and launches follow it.
struct OnDevice {
    int before = -1;
    void* stream;
    explicit OnDevice(const Tensor& t) {
        const int want = t.get_device(), now = c10::cuda::current_device();
        if (now != want) {
            before = now;
            c10::cuda::set_device((c10::DeviceIndex)want);
        }
        stream = (void*)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)want).stream();
    }
    ~OnDevice() {   // an error here was the call's own already; a destructor that throws ends the process
        try {
            if (before >= 0) c10::cuda::set_device((c10::DeviceIndex)before);
        } catch (const std::exception&) {
        }
    }
};

// float argument or None: whatever float() takes
bool scale_arg(PyObject* o, float* out) {
    *out = 0.f;
    if (o == Py_None) return true;
    PyObject* x = PyNumber_Float(o);
    if (!x) return false;
    *out = (float)PyFloat_AS_DOUBLE(x);
    Py_DECREF(x);
    return true;
}
// integer argument: whatever int() takes
bool int_arg(PyObject* o, int64_t* out) {
    PyObject* x = PyNumber_Long(o);
    if (!x) return false;
    *out = PyLong_AsLongLong(x);
    Py_DECREF(x);
    return !(*out == -1 && PyErr_Occurred());
}
bool fits32(int64_t x) { return x == (int32_t)x; }

PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap_or(PyObject* given, const Tensor& made) {   // the caller's own object where it gave one
    if (given != Py_None) {
        Py_INCREF(given);
        return given;
    }
    if (!made.defined()) Py_RETURN_NONE;
    return wrap(made);
}
template <typename... P>
PyObject* pack(P*... items) {
    PyObject* r = PyTuple_New(sizeof...(items));
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(r, i++, items), ...);
    return r;
}
PyObject* failed(int rc) { return PyLong_FromLong(rc); }

// c10 errors (out of memory among them) become the Python exceptions that torch itself raises
template <typename F>
PyObject* guarded(F&& f) {
    try {
        return f();
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* torch = PyImport_ImportModule("torch");
        PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
        PyErr_SetString(type ? type : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(type);
        Py_XDECREF(torch);
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// the GIL is taken again on every way out
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
#define TT_CALL(rc, expr) \
    const int rc = [&] {  \
        NoGil released;   \
        return (expr);    \
    }()

// q [B,H,S,D], k and v [B,Hkv,L,D] of one type
bool attn_args(PyObject* oq, PyObject* ok, PyObject* ov, const Tensor** q, const Tensor** k, const Tensor** v,
               tt_attn_desc* d) {
    if (!(*q = cuda_arg(oq)) || !(*k = cuda_arg(ok)) || !(*v = cuda_arg(ov))) return false;
    const Tensor &tq = **q, &tk = **k, &tv = **v;
    if (tq.dim() != 4 || tk.dim() != 4 || tv.dim() != 4 || !float_type(tq)) return false;
    if (tk.scalar_type() != tq.scalar_type() || tv.scalar_type() != tq.scalar_type() || !same_shape(tk, tv)) return false;
    const int64_t B = tq.size(0), H = tq.size(1), hkv = tk.size(1);
    if (tk.size(0) != B || hkv < 1 || H % hkv != 0 || tk.size(3) != tq.size(3)) return false;
    *d = tt_attn_desc{(int32_t)B, (int32_t)H, (int32_t)tq.size(2), (int32_t)tk.size(2), (int32_t)tq.size(3), tt_type(tq), 0,
                      0.f, (int32_t)hkv};
    return true;
}
bool lens_arg(PyObject* o, int64_t B, const int32_t** p) {
    *p = nullptr;
    if (o == Py_None) return true;
    const Tensor* t = cuda_arg(o);
    if (!t || t->scalar_type() != at::kInt || t->dim() != 1 || t->size(0) != B) return false;
    *p = (const int32_t*)t->data_ptr();
    return true;
}
// The caller's workspace when it is large enough, else a new one of at least `least` bytes.
const Tensor* workspace_arg(const Tensor* given, size_t need, size_t least, const Tensor& like, Tensor* made, size_t* bytes) {
    if (given && given->nbytes() >= need) {
        *bytes = given->nbytes();
        return given;
    }
    *bytes = need > least ? need : least;
    if (*bytes == 0) return given;
    *made = make_bytes(*bytes, like);
    return made;
}

// (q, k, v, causal, scale, out, lse, need_lse, kv_lens) -> (out, lse)
PyObject* attention_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *q, *k, *v;
        tt_attn_desc d;
        const int32_t* lens;
        bool fits = true;
        if (n != 9 || !attn_args(a[0], a[1], a[2], &q, &k, &v, &d) || !lens_arg(a[8], d.B, &lens)) Py_RETURN_NONE;
        const Tensor *out = opt_arg(a[5], &fits), *lse = opt_arg(a[6], &fits);
        const int causal = PyObject_IsTrue(a[3]), need_lse = PyObject_IsTrue(a[7]);
        if (!fits) Py_RETURN_NONE;
        if (causal < 0 || need_lse < 0 || !scale_arg(a[4], &d.scale)) return nullptr;
        d.causal = causal;
        OnDevice dev(*q);
        Tensor new_out, new_lse;
        if (!out) new_out = make_like(*q);
        if (!lse && need_lse) new_lse = make({d.B, d.H, d.S}, at::kFloat, *q);
        void* po = out ? ptr(out) : ptr(new_out);
        float* pl = (float*)(lse ? ptr(lse) : new_lse.defined() ? ptr(new_lse) : nullptr);
        TT_CALL(rc, lens ? tt_attn_fwd_padded(&d, ptr(q), ptr(k), ptr(v), lens, po, pl, dev.stream)
                         : tt_attn_fwd(&d, ptr(q), ptr(k), ptr(v), po, pl, dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap_or(a[5], new_out), wrap_or(a[6], new_lse));
    });
}

// (q, k, v, out, lse, dout, causal, scale, workspace, kv_lens) -> (dq, dk, dv)
PyObject* attention_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *q, *k, *v;
        tt_attn_desc d;
        const int32_t* lens;
        bool fits = true;
        if (n != 10 || !attn_args(a[0], a[1], a[2], &q, &k, &v, &d) || !lens_arg(a[9], d.B, &lens)) Py_RETURN_NONE;
        const Tensor *out = cuda_arg(a[3]), *lse = cuda_arg(a[4]), *dout = cuda_arg(a[5]), *ws = opt_arg(a[8], &fits);
        if (!out || !lse || !dout || !fits || !same_shape(*out, *q) || !same_shape(*dout, *q) ||
            out->scalar_type() != q->scalar_type() || dout->scalar_type() != q->scalar_type() ||
            lse->scalar_type() != at::kFloat || lse->dim() != 3 || lse->size(0) != d.B || lse->size(1) != d.H || lse->size(2) != d.S)
            Py_RETURN_NONE;
        const int causal = PyObject_IsTrue(a[6]);
        if (causal < 0 || !scale_arg(a[7], &d.scale)) return nullptr;
        d.causal = causal;
        OnDevice dev(*q);
        Tensor made;
        size_t bytes;
        ws = workspace_arg(ws, tt_attn_bwd_workspace_bytes(&d), 256, *q, &made, &bytes);
        Tensor dq = make_like(*q), dk = make_like(*k), dv = make_like(*v);
        TT_CALL(rc, lens ? tt_attn_bwd_padded(&d, ptr(q), ptr(k), ptr(v), lens, ptr(out), (const float*)ptr(lse), ptr(dout), ptr(dq),
                                              ptr(dk), ptr(dv), ptr(ws), bytes, dev.stream)
                         : tt_attn_bwd(&d, ptr(q), ptr(k), ptr(v), ptr(out), (const float*)ptr(lse), ptr(dout), ptr(dq), ptr(dk),
                                       ptr(dv), ptr(ws), bytes, dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap(dq), wrap(dk), wrap(dv));
    });
}

// packed batches: q [total_q,H,D], k [total_k,Hkv,D], cu_q and cu_k int32 [n_seq + 1]
bool varlen_args(PyObject* const* a, const Tensor** q, const Tensor** k, const Tensor** v, const Tensor** cq, const Tensor** ck,
                 tt_varlen_desc* d, bool* raised) {
    *raised = false;
    if (!(*q = cuda_arg(a[0])) || !(*k = cuda_arg(a[1])) || !(*v = cuda_arg(a[2])) || !(*cq = cuda_arg(a[3])) || !(*ck = cuda_arg(a[4])))
        return false;
    const Tensor &tq = **q, &tk = **k;
    if (tq.dim() != 3 || tk.dim() != 3 || tq.scalar_type() != at::kBFloat16 || tk.scalar_type() != at::kBFloat16) return false;
    for (const Tensor* c : {*cq, *ck})
        if (c->scalar_type() != at::kInt || c->dim() != 1 || c->numel() != (*cq)->numel()) return false;
    if (tk.size(2) != tq.size(2) || tk.size(1) < 1 || tq.size(1) % tk.size(1) != 0) return false;
    int64_t mq, mk;
    if (!int_arg(a[5], &mq) || !int_arg(a[6], &mk)) {
        *raised = true;
        return false;
    }
    if (!fits32(mq) || !fits32(mk)) return false;
    *d = tt_varlen_desc{(int32_t)(*cq)->numel() - 1, (int32_t)tq.size(1), (int32_t)tk.size(1), (int32_t)tq.size(2), TT_BF16, 0, 0.f, (int32_t)mq,
                        (int32_t)mk, tq.size(0), tk.size(0)};
    return true;
}

// (q, k, v, cu_q, cu_k, max_q, max_k, causal, scale, out, lse) -> (out, lse)
PyObject* attention_forward_varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *q, *k, *v, *cq, *ck;
        tt_varlen_desc d;
        bool raised, fits = true;
        if (n != 11) Py_RETURN_NONE;
        if (!varlen_args(a, &q, &k, &v, &cq, &ck, &d, &raised)) {
            if (raised) return nullptr;
            Py_RETURN_NONE;
        }
        const Tensor *out = opt_arg(a[9], &fits), *lse = opt_arg(a[10], &fits);
        const int causal = PyObject_IsTrue(a[7]);
        if (!fits) Py_RETURN_NONE;
        if (causal < 0 || !scale_arg(a[8], &d.scale)) return nullptr;
        d.causal = causal;
        OnDevice dev(*q);
        Tensor new_out, new_lse;
        if (!out) new_out = make_like(*q);
        if (!lse) new_lse = make({q->size(1), q->size(0)}, at::kFloat, *q);
        TT_CALL(rc, tt_attn_fwd_varlen(&d, ptr(q), ptr(k), ptr(v), (const int32_t*)ptr(cq), (const int32_t*)ptr(ck),
                                       out ? ptr(out) : ptr(new_out), (float*)(lse ? ptr(lse) : ptr(new_lse)), dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap_or(a[9], new_out), wrap_or(a[10], new_lse));
    });
}

// (q, k, v, cu_q, cu_k, max_q, max_k, out, lse, dout, causal, scale, workspace) -> (dq, dk, dv)
PyObject* attention_backward_varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *q, *k, *v, *cq, *ck;
        tt_varlen_desc d;
        bool raised, fits = true;
        if (n != 13) Py_RETURN_NONE;
        if (!varlen_args(a, &q, &k, &v, &cq, &ck, &d, &raised)) {
            if (raised) return nullptr;
            Py_RETURN_NONE;
        }
        const Tensor *out = opt_arg(a[7], &fits), *lse = opt_arg(a[8], &fits), *dout = opt_arg(a[9], &fits), *ws = opt_arg(a[12], &fits);
        if (!fits || !out || !lse || !dout) Py_RETURN_NONE;
        const int causal = PyObject_IsTrue(a[10]);
        if (causal < 0 || !scale_arg(a[11], &d.scale)) return nullptr;
        d.causal = causal;
        OnDevice dev(*q);
        Tensor made;
        size_t bytes;
        ws = workspace_arg(ws, tt_attn_bwd_varlen_workspace_bytes(&d), 256, *q, &made, &bytes);
        Tensor dq = make_like(*q), dk = make_like(*k), dv = make_like(*v);
        TT_CALL(rc, tt_attn_bwd_varlen(&d, ptr(q), ptr(k), ptr(v), (const int32_t*)ptr(cq), (const int32_t*)ptr(ck), ptr(out),
                                       (const float*)ptr(lse), ptr(dout), ptr(dq), ptr(dk), ptr(dv), ptr(ws), bytes, dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap(dq), wrap(dk), wrap(dv));
    });
}

// (q, k, v, scale, out, lse, workspace, need_lse) -> (out, lse)
PyObject* attention_decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *q, *k, *v;
        tt_attn_desc d;
        bool fits = true;
        if (n != 8 || !attn_args(a[0], a[1], a[2], &q, &k, &v, &d) || d.S != 1) Py_RETURN_NONE;
        const Tensor *out = opt_arg(a[4], &fits), *lse = opt_arg(a[5], &fits), *ws = opt_arg(a[6], &fits);
        const int need_lse = PyObject_IsTrue(a[7]);
        if (!fits) Py_RETURN_NONE;
        if (need_lse < 0 || !scale_arg(a[3], &d.scale)) return nullptr;
        OnDevice dev(*q);
        Tensor new_out, new_lse, made;
        if (!out) new_out = make_like(*q);
        if (!lse && need_lse) new_lse = make({d.B, d.H, 1}, at::kFloat, *q);
        size_t bytes;
        ws = workspace_arg(ws, tt_attn_decode_workspace_bytes(&d), 0, *q, &made, &bytes);
        TT_CALL(rc, tt_attn_decode(&d, ptr(q), ptr(k), ptr(v), out ? ptr(out) : ptr(new_out),
                                   (float*)(lse ? ptr(lse) : new_lse.defined() ? ptr(new_lse) : nullptr), ptr(ws), bytes, dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap_or(a[4], new_out), wrap_or(a[5], new_lse));
    });
}

// (q, k_pool, v_pool, block_table, seq_lens, max_len, scale, out, lse, workspace, need_lse) -> (out, lse)
PyObject* attention_decode_paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        if (n != 11) Py_RETURN_NONE;
        const Tensor *q = cuda_arg(a[0]), *k = cuda_arg(a[1]), *v = cuda_arg(a[2]);
        if (!q || !k || !v || q->dim() != 4 || k->dim() != 4 || q->size(2) != 1 || q->scalar_type() != at::kBFloat16 ||
            k->scalar_type() != at::kBFloat16 || v->scalar_type() != at::kBFloat16 || k->size(3) != q->size(3) || !same_shape(*k, *v))
            Py_RETURN_NONE;
        const int64_t B = q->size(0), H = q->size(1), hkv = k->size(1);
        const int32_t* lens;
        if (hkv < 1 || H % hkv != 0 || !lens_arg(a[4], B, &lens)) Py_RETURN_NONE;
        int32_t page = 0, max_pages = 0;
        int64_t L = k->size(2);
        const int32_t* table = nullptr;
        if (a[3] != Py_None) {
            const Tensor* t = cuda_arg(a[3]);
            if (!t || t->scalar_type() != at::kInt || t->dim() != 2 || t->size(0) != B) Py_RETURN_NONE;
            table = (const int32_t*)t->data_ptr();
            page = (int32_t)k->size(2);
            max_pages = (int32_t)t->size(1);
            L = (int64_t)page * max_pages;
        } else if (k->size(0) != B) {
            Py_RETURN_NONE;
        }
        if (a[5] != Py_None && !int_arg(a[5], &L)) return nullptr;
        if ((!table && L > k->size(2)) || !fits32(L)) Py_RETURN_NONE;
        bool fits = true;
        const Tensor *out = opt_arg(a[7], &fits), *lse = opt_arg(a[8], &fits), *ws = opt_arg(a[9], &fits);
        const int need_lse = PyObject_IsTrue(a[10]);
        if (!fits) Py_RETURN_NONE;
        tt_attn_desc d{(int32_t)B, (int32_t)H, 1, (int32_t)L, (int32_t)q->size(3), TT_BF16, 0, 0.f, (int32_t)hkv};
        if (need_lse < 0 || !scale_arg(a[6], &d.scale)) return nullptr;
        OnDevice dev(*q);
        Tensor new_out, new_lse, made;
        if (!out) new_out = make_like(*q);
        if (!lse && need_lse) new_lse = make({B, H, 1}, at::kFloat, *q);
        size_t bytes;
        ws = workspace_arg(ws, tt_attn_decode_workspace_bytes(&d), 0, *q, &made, &bytes);
        TT_CALL(rc, tt_attn_decode_paged(&d, ptr(q), ptr(k), ptr(v), table, lens, page, max_pages, out ? ptr(out) : ptr(new_out),
                                         (float*)(lse ? ptr(lse) : new_lse.defined() ? ptr(new_lse) : nullptr), ptr(ws), bytes,
                                         dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap_or(a[7], new_out), wrap_or(a[8], new_lse));
    });
}

void rows_of(const Tensor& t, int64_t* rows, int32_t* cols) {
    *cols = t.dim() ? (int32_t)t.size(-1) : 0;
    *rows = *cols ? t.numel() / *cols : 0;
}

// (x, out) -> out
PyObject* softmax_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor* x = n == 2 ? cuda_arg(a[0]) : nullptr;
        bool fits = true;
        if (!x || !float_type(*x) || x->dim() < 1) Py_RETURN_NONE;
        const Tensor* out = opt_arg(a[1], &fits);
        if (!fits) Py_RETURN_NONE;
        int64_t rows;
        int32_t cols;
        rows_of(*x, &rows, &cols);
        OnDevice dev(*x);
        Tensor made;
        if (!out) made = make_like(*x);
        TT_CALL(rc, tt_softmax_fwd(ptr(x), out ? ptr(out) : ptr(made), rows, cols, tt_type(*x), dev.stream));
        return rc != TT_OK ? failed(rc) : wrap_or(a[1], made);
    });
}

// (y, dy, dx) -> dx
PyObject* softmax_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *y = n == 3 ? cuda_arg(a[0]) : nullptr, *dy = n == 3 ? cuda_arg(a[1]) : nullptr;
        bool fits = true;
        if (!y || !dy || !float_type(*y) || y->scalar_type() != dy->scalar_type() || !same_shape(*y, *dy) || y->dim() < 1) Py_RETURN_NONE;
        const Tensor* dx = opt_arg(a[2], &fits);
        if (!fits) Py_RETURN_NONE;
        int64_t rows;
        int32_t cols;
        rows_of(*y, &rows, &cols);
        OnDevice dev(*y);
        Tensor made;
        if (!dx) made = make_like(*y);
        TT_CALL(rc, tt_softmax_bwd(ptr(y), ptr(dy), dx ? ptr(dx) : ptr(made), rows, cols, tt_type(*y), dev.stream));
        return rc != TT_OK ? failed(rc) : wrap_or(a[2], made);
    });
}

// x [..., in], w [in, out] of one type
bool fc_args(PyObject* ox, PyObject* ow, const Tensor** x, const Tensor** w, int64_t* rows, int32_t* fin, int32_t* fout) {
    if (!(*x = cuda_arg(ox)) || !(*w = cuda_arg(ow))) return false;
    const Tensor &tx = **x, &tw = **w;
    if (!float_type(tx) || tx.scalar_type() != tw.scalar_type() || tw.dim() != 2 || tx.dim() < 1 || tx.size(-1) != tw.size(0)) return false;
    *fin = (int32_t)tw.size(0);
    *fout = (int32_t)tw.size(1);
    *rows = *fin ? tx.numel() / *fin : 0;
    return true;
}
bool layer_output(const Tensor& y, const Tensor& x, int32_t fout) {
    return y.dim() == x.dim() && y.size(-1) == fout && y.sizes().slice(0, y.dim() - 1) == x.sizes().slice(0, x.dim() - 1);
}

// (x, w, bias, out) -> y
PyObject* fc_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *x, *w;
        int64_t rows;
        int32_t fin, fout;
        bool fits = true;
        if (n != 4 || !fc_args(a[0], a[1], &x, &w, &rows, &fin, &fout)) Py_RETURN_NONE;
        const Tensor *bias = opt_arg(a[2], &fits), *out = opt_arg(a[3], &fits);
        if (!fits || (bias && (!bias->is_cuda() || bias->scalar_type() != x->scalar_type() || bias->dim() != 1 || bias->size(0) != fout)))
            Py_RETURN_NONE;
        OnDevice dev(*x);
        Tensor made;
        if (!out) {
            c10::SmallVector<int64_t, 5> shape(x->sizes().begin(), x->sizes().end());
            shape.back() = fout;
            made = make(shape, x->scalar_type(), *x);
        }
        TT_CALL(rc, tt_fc_fwd(ptr(x), ptr(w), ptr(bias), out ? ptr(out) : ptr(made), rows, fin, fout, tt_type(*x), dev.stream));
        return rc != TT_OK ? failed(rc) : wrap_or(a[3], made);
    });
}

// (x, w, dy, need_dx, need_dw, need_db, scalar_bias, workspace) -> (dx, dw, db)
PyObject* fc_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        const Tensor *x, *w;
        int64_t rows;
        int32_t fin, fout;
        bool fits = true;
        if (n != 8 || !fc_args(a[0], a[1], &x, &w, &rows, &fin, &fout)) Py_RETURN_NONE;
        const Tensor *dy = cuda_arg(a[2]), *ws = opt_arg(a[7], &fits);
        if (!fits || !dy || dy->scalar_type() != x->scalar_type() || !layer_output(*dy, *x, fout)) Py_RETURN_NONE;
        int flag[4];
        for (int i = 0; i < 4; ++i)
            if ((flag[i] = PyObject_IsTrue(a[3 + i])) < 0) return nullptr;
        OnDevice dev(*x);
        Tensor dx, dw, db, made;
        if (flag[0]) dx = make_like(*x);
        if (flag[1]) dw = make_like(*w);
        if (flag[2]) db = make({flag[3] ? 1 : (int64_t)fout}, x->scalar_type(), *x);
        size_t bytes = 0;
        ws = workspace_arg(ws, flag[2] ? tt_fc_bwd_workspace_bytes(rows, fin, fout, tt_type(*x)) : 0, 0, *x, &made, &bytes);
        auto at = [](const Tensor& t) { return t.defined() ? ptr(t) : nullptr; };
        TT_CALL(rc, tt_fc_bwd(ptr(x), ptr(w), ptr(dy), at(dx), at(dw), at(db), flag[3], rows, fin, fout, tt_type(*x), ptr(ws), bytes,
                              dev.stream));
        if (rc != TT_OK) return failed(rc);
        return pack(wrap_or(Py_None, dx), wrap_or(Py_None, dw), wrap_or(Py_None, db));
    });
}

#define TT_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    TT_METHOD(attention_forward), TT_METHOD(attention_backward), TT_METHOD(attention_forward_varlen),
    TT_METHOD(attention_backward_varlen), TT_METHOD(attention_decode), TT_METHOD(attention_decode_paged),
    TT_METHOD(softmax_forward), TT_METHOD(softmax_backward), TT_METHOD(fc_forward), TT_METHOD(fc_backward),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_ttorch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ttorch(void) { return PyModule_Create(&module); }

// The calls that an eager step makes most, from Python to the kernel library without ctypes in between: checks,
// allocation of the result, the current stream and the launch in one C function per operation.
//
// A prompt step of a small model is bound by its host: some ten operations a layer, each 12 to 20 us of Python (argument
// checks one attribute at a time, ctypes conversions of up to 25 arguments), against kernels of 5 to 50 us.  Here an
// operation takes 4 to 6 us, most of it the launch itself.
//
// The functions accept what the kernels' ordinary Python wrappers (`csrc/ops.py`) accept in everyday use and return None,
// having done nothing, for everything else: the wrapper then goes on as before, and says what is wrong if something is.
// Results: a tensor, or the C entry point's code as an int (0: done).  Nothing is kept between calls but the entry
// points' addresses.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

namespace {

typedef const void* P;
struct Entries {
    int (*add_rmsnorm)(P, P, P, void*, P, void*, int, int, float, int, void*);
    int (*qk_norm_rope_kv)(void*, int, P, P, float, P, int, P, P, void*, void*, int, int, int, int, int, int, int, int, int, float, void*);
    int (*gated_act)(P, void*, int, int, int, int, int, int, void*);
    int (*gemm_skinny)(P, P, P, void*, int, int, int, int, int, int, int, int, int, int, void*);
    int (*gemm_tcgen05_columns)(P, P, P, void*, int, int, int, int, int, int, int, int, int, void*, void*);
    int (*gemm_tcgen05_pair)(P, P, P, void*, int, int, int, int, int, int, int, int, void*, void*);
    int (*gemm_turned)(P, P, void*, int, int, int, int, int, int, int, int, int, int, void*, void*);
    int (*prefill)(P, int, int, P, P, int, P, int, P, P, P, void*, int, float, int, int, int, int, int, int, int, void*, int, void*, void*);
    int (*decode)(P, int, P, P, P, int, P, P, P, void*, int, void*, int, float, int, int, int, int, int, int, int, int, int, void*);
} entry;

const int DTYPE_F32 = 0, DTYPE_BF16 = 1;   // the library's codes

// ---- arguments ----------------------------------------------------------------------------------------
// A plain CUDA tensor, or null (of a subclass too: what intercepts torch's calls has to see them).
struct Arg {
    const at::Tensor* t = nullptr;
    explicit Arg(PyObject* o) {
        if (!THPVariable_CheckExact(o)) return;
        const at::Tensor& x = THPVariable_Unpack(o);
        if (x.is_cuda() && x.layout() == at::kStrided) t = &x;
    }
    explicit operator bool() const { return t != nullptr; }
    const at::Tensor& operator*() const { return *t; }
    const at::Tensor* operator->() const { return t; }
};
// The same, where None is allowed: `ok` is false if it is neither.
struct Optional {
    Arg a;
    bool ok;
    explicit Optional(PyObject* o) : a(o), ok(o == Py_None || bool(a)) {}
    explicit operator bool() const { return bool(a); }
    void* ptr() const { return a ? a->data_ptr() : nullptr; }
    bool is(at::ScalarType s) const { return ok && (!a || a->scalar_type() == s); }
};
inline bool is(const Arg& a, at::ScalarType s) { return a && a->scalar_type() == s; }
inline bool is16(const Arg& a) { return is(a, at::kBFloat16); }
inline int code_of(at::ScalarType s) { return s == at::kFloat ? DTYPE_F32 : s == at::kBFloat16 ? DTYPE_BF16 : -1; }
inline bool aligned16(const at::Tensor& t) { return ((uintptr_t)t.data_ptr() & 15) == 0; }
inline bool small(int64_t x) { return x >= 0 && x <= 0x7fffffff; }

// Whole numbers, truth values and floats; an argument of another kind (or out of range) sets `bad`.
struct Scalars {
    bool bad = false;
    int i(PyObject* o) {
        int overflow = 0;
        const long v = PyLong_Check(o) ? PyLong_AsLongAndOverflow(o, &overflow) : (bad = true, 0);
        if (overflow || v != (int)v) bad = true;
        return (int)v;
    }
    void* p(PyObject* o) {   // (an address; none is 0)
        void* v = PyLong_Check(o) ? PyLong_AsVoidPtr(o) : nullptr;
        if (!v) {
            PyErr_Clear();
            bad = true;
        }
        return v;
    }
    float f(PyObject* o) {
        if (PyFloat_Check(o)) return (float)PyFloat_AS_DOUBLE(o);
        return (float)i(o);
    }
};
inline at::Tensor fresh(int64_t rows, int64_t cols, at::ScalarType s, const at::Tensor& like) {
    return at::empty({rows, cols}, like.options().dtype(s));
}
inline void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
inline PyObject* result(int code, at::Tensor out) { return code ? PyLong_FromLong(code) : THPVariable_Wrap(std::move(out)); }
#define NOT_HERE Py_RETURN_NONE
#define LAUNCH(code, call)       \
    int code;                    \
    {                            \
        void* s = stream();      \
        Py_BEGIN_ALLOW_THREADS   \
        code = call;             \
        Py_END_ALLOW_THREADS     \
    }

inline bool tcgen05_takes(const at::Tensor& a, const at::Tensor& w) {
    return a.dim() == 2 && w.dim() == 2 && a.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && a.size(1) == w.size(1) &&
           a.size(1) % 8 == 0 && w.size(0) % 16 == 0 && a.stride(1) == 1 && w.stride(1) == 1 && a.stride(0) % 8 == 0 &&
           w.stride(0) % 8 == 0 && aligned16(a) && aligned16(w) && small(a.stride(0)) && small(w.stride(0)) && small(a.size(0)) &&
           small(w.size(0));
}
inline bool skinny_takes(const at::Tensor& a, const at::Tensor& w) {
    return a.dim() == 2 && w.dim() == 2 && a.size(0) > 0 && a.size(0) <= 8 && a.size(1) == w.size(1) && a.size(1) % 32 == 0 &&
           a.stride(1) == 1 && w.stride(1) == 1 && a.stride(0) % 8 == 0 && w.stride(0) % 8 == 0 && aligned16(a) && aligned16(w) &&
           small(a.stride(0)) && small(w.stride(0)) && small(w.size(0));
}

// ---- operations ---------------------------------------------------------------------------------------
// (residual, delta, weight, eps, out_dtype, rows, residual_out, update_residual)
PyObject* add_rmsnorm(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) NOT_HERE;
    Arg residual(o[0]), weight(o[2]);
    Optional delta(o[1]), rows(o[5]), residual_out(o[6]);
    Scalars sc;
    const float eps = sc.f(o[3]);
    if (sc.bad || !THPDtype_Check(o[4]) || !is(residual, at::kFloat) || !is(weight, at::kFloat) || !delta.ok || !rows.is(at::kInt) ||
        !residual_out.ok)
        NOT_HERE;
    const at::ScalarType kind = ((THPDtype*)o[4])->scalar_type;
    const int code = code_of(kind);
    if (code < 0 || residual->dim() != 2 || !residual->is_contiguous() || weight->numel() != residual->size(1)) NOT_HERE;
    if (delta && (delta.a->scalar_type() != kind || !delta.a->is_contiguous() || delta.a->sizes() != residual->sizes())) NOT_HERE;
    const int64_t width = residual->size(1), count = rows ? rows.a->numel() : residual->size(0);
    if (!small(width) || !small(count)) NOT_HERE;
    const int update = !rows && delta ? PyObject_IsTrue(o[7]) : 0;
    if (update < 0) return nullptr;   // (its truth value raised)
    void* sums = rows ? residual_out.ptr() : (update ? residual->data_ptr() : nullptr);
    at::Tensor out = fresh(count, width, kind, *residual);
    LAUNCH(rc, entry.add_rmsnorm(residual->data_ptr(), delta.ptr(), rows.ptr(), sums, weight->data_ptr(), out.data_ptr(), (int)count,
                                 (int)width, eps, code, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

// (qkv, q_weight, k_weight, eps, inv_freq, rot_dim, positions, slot_mapping, k_pool, v_pool, heads, kv heads, head size,
//  value size, interleaved, value heads, magnitude)
PyObject* qk_norm_rope_kv(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 17) NOT_HERE;
    Arg qkv(o[0]), positions(o[6]);
    Optional qw(o[1]), kw(o[2]), inv_freq(o[4]), slots(o[7]), k_pool(o[8]), v_pool(o[9]);
    Scalars sc;
    const float eps = sc.f(o[3]), magnitude = sc.f(o[16]);
    const int rot = sc.i(o[5]), H = sc.i(o[10]), Hk = sc.i(o[11]), D = sc.i(o[12]), Dv = sc.i(o[13]), turned = sc.i(o[14]), Hv = sc.i(o[15]);
    if (sc.bad || !qkv || !is(positions, at::kInt) || !qw.is(at::kFloat) || !kw.is(at::kFloat) || !inv_freq.is(at::kFloat) || !slots.ok ||
        !k_pool.ok || !v_pool.ok)
        NOT_HERE;
    const int code = code_of(qkv->scalar_type());
    if (code < 0 || qkv->dim() != 2 || !qkv->is_contiguous() || !small(qkv->size(0)) || !small(qkv->size(1))) NOT_HERE;
    if ((qw && qw.a->numel() != D) || (kw && kw.a->numel() != D) || (inv_freq && inv_freq.a->numel() * 2 != rot)) NOT_HERE;
    int page = 1;
    if (slots) {
        if (!k_pool || !v_pool) NOT_HERE;
        const at::Tensor &k = *k_pool.a, &v = *v_pool.a;
        if (k.scalar_type() != qkv->scalar_type() || k.dim() != 4 || v.dim() != 4 || !k.is_contiguous() || !v.is_contiguous() ||
            k.size(1) != Hk || k.size(3) != D || v.size(1) != Hv || v.size(2) != k.size(2) || v.size(3) != Dv || !small(k.size(2)))
            NOT_HERE;
        page = (int)k.size(2);
    }
    LAUNCH(rc, entry.qk_norm_rope_kv(qkv->data_ptr(), (int)qkv->size(1), qw.ptr(), kw.ptr(), eps, inv_freq.ptr(), rot, positions->data_ptr(),
                                     slots.ptr(), k_pool.ptr(), v_pool.ptr(), (int)qkv->size(0), H, Hk, D, page, code, Dv, turned, Hv,
                                     magnitude, s));
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// (gate_up, activation's code, block, out dtype)
PyObject* gated_act(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) NOT_HERE;
    Arg x(o[0]);
    Scalars sc;
    const int act = sc.i(o[1]), block = sc.i(o[2]);
    if (sc.bad || !x || !THPDtype_Check(o[3])) NOT_HERE;
    const at::ScalarType kind = ((THPDtype*)o[3])->scalar_type;
    const int in = code_of(x->scalar_type()), to = code_of(kind);
    if (in < 0 || to < 0 || x->dim() != 2 || !x->is_contiguous() || x->size(1) % 2 || !small(x->size(0)) || !small(x->size(1))) NOT_HERE;
    at::Tensor out = fresh(x->size(0), x->size(1) / 2, kind, *x);
    LAUNCH(rc, entry.gated_act(x->data_ptr(), out.data_ptr(), (int)x->size(0), (int)(x->size(1) / 2), act, block, in, to, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

// (a, w, out dtype): the library product, or a kernel of ours for a few rows; without a bias
PyObject* gemm_bf16(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 3) NOT_HERE;
    Arg a(o[0]), w(o[1]);
    if (!is16(a) || !is16(w) || !THPDtype_Check(o[2]) || a->dim() != 2 || w->dim() != 2 || a->size(1) != w->size(1)) NOT_HERE;
    const at::ScalarType kind = ((THPDtype*)o[2])->scalar_type;
    const int code = code_of(kind);
    if (code < 0) NOT_HERE;
    if (skinny_takes(*a, *w)) {
        at::Tensor out = fresh(a->size(0), w->size(0), kind, *a);
        LAUNCH(rc, entry.gemm_skinny(a->data_ptr(), w->data_ptr(), nullptr, out.data_ptr(), (int)a->size(0), (int)w->size(0), (int)a->size(1),
                                     (int)a->stride(0), (int)w->stride(0), (int)w->size(0), 0, -1, code, 0, s));
        return result(rc, std::move(out));
    }
    at::Tensor out;
    {
        pybind11::gil_scoped_release unlocked;
        out = kind == at::kFloat ? at::mm(*a, w->t(), at::kFloat) : at::mm(*a, w->t());
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// (a, w, bias, epilogue code, activation, columns of a tile or 0, pair, the error word's address)
PyObject* gemm_tcgen05(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) NOT_HERE;
    Arg a(o[0]), w(o[1]);
    Optional bias(o[2]);
    Scalars sc;
    const int code = sc.i(o[3]), act = sc.i(o[4]), columns = sc.i(o[5]), pair = sc.i(o[6]);
    void* const error = sc.p(o[7]);
    if (sc.bad || !a || !w || !bias.is(at::kFloat) || !tcgen05_takes(*a, *w)) NOT_HERE;
    const int64_t M = a->size(0), N = w->size(0), cols = code == 1 ? N / 2 : N;
    if ((bias && bias.a->numel() != N) || cols % 8) NOT_HERE;
    at::Tensor out = fresh(M, cols, at::kBFloat16, *a);
    LAUNCH(rc, pair ? entry.gemm_tcgen05_pair(a->data_ptr(), w->data_ptr(), bias.ptr(), out.data_ptr(), (int)M, (int)N, (int)a->size(1),
                                              (int)a->stride(0), (int)w->stride(0), (int)cols, code, act, error, s)
                    : entry.gemm_tcgen05_columns(a->data_ptr(), w->data_ptr(), bias.ptr(), out.data_ptr(), (int)M, (int)N, (int)a->size(1),
                                                 (int)a->stride(0), (int)w->stride(0), (int)cols, code, act, columns, error, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

// (a, w, gated, activation, out dtype, w is ready, the error word's address)
PyObject* gemm_turned(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) NOT_HERE;
    Arg a(o[0]), w(o[1]);
    Scalars sc;
    const int gated = sc.i(o[2]), act = sc.i(o[3]), ready = sc.i(o[5]);
    void* const error = sc.p(o[6]);
    if (sc.bad || !a || !w || !THPDtype_Check(o[4]) || !tcgen05_takes(*a, *w)) NOT_HERE;
    const at::ScalarType kind = ((THPDtype*)o[4])->scalar_type;
    const int64_t M = a->size(0), N = w->size(0), cols = gated ? N / 2 : N;
    if (code_of(kind) < 0 || cols % 8) NOT_HERE;
    at::Tensor out = fresh(M, cols, kind, *a);
    LAUNCH(rc, entry.gemm_turned(a->data_ptr(), w->data_ptr(), out.data_ptr(), (int)M, (int)N, (int)a->size(1), (int)a->stride(0),
                                 (int)w->stride(0), (int)cols, gated, act, code_of(kind), ready, error, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

PyObject* tcgen05_supported(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 2) NOT_HERE;
    Arg a(o[0]), w(o[1]);
    if (!a || !w || a->dim() != 2 || w->dim() != 2 || a->size(1) != w->size(1)) NOT_HERE;
    return PyBool_FromLong(tcgen05_takes(*a, *w));
    END_HANDLE_TH_ERRORS
}

// Queries, pools, block table and the result that the two attention calls have in common.
struct Attention {
    Arg q, k, v, table;
    Optional out;
    Attention(PyObject* q_, PyObject* k_, PyObject* v_, PyObject* table_, PyObject* out_) : q(q_), k(k_), v(v_), table(table_), out(out_) {}
    bool fine(int D) const {
        return is16(q) && is16(k) && is16(v) && is(table, at::kInt) && out.is(at::kBFloat16) && table->dim() == 2 && table->is_contiguous() &&
               k->dim() == 4 && v->dim() == 4 && k->is_contiguous() && v->is_contiguous() && k->size(3) == D && v->size(3) == D &&
               small(k->size(0)) && small(k->size(2)) && small(table->size(1));
    }
};

// (q, row stride, k_pool, v_pool, block table, cu_seqlens, kv_offsets, scale, window, heads, kv heads, head size, requests,
//  max_new, tokens, seq_list, out, scratch, max_splits, the error word's address)
PyObject* prefill_attention(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 20) NOT_HERE;
    Attention x(o[0], o[2], o[3], o[4], o[16]);
    Arg cu(o[5]), offsets(o[6]);
    Optional list(o[15]), scratch(o[17]);
    Scalars sc;
    const int ld = sc.i(o[1]), window = sc.i(o[8]), H = sc.i(o[9]), Hk = sc.i(o[10]), D = sc.i(o[11]), requests = sc.i(o[12]),
              max_new = sc.i(o[13]), tokens = sc.i(o[14]), splits = sc.i(o[18]);
    const float scale = sc.f(o[7]);
    void* const error = sc.p(o[19]);
    if (sc.bad || !x.fine(D) || !cu || !offsets || !list.ok || !scratch.is(at::kFloat)) NOT_HERE;
    at::Tensor out = x.out ? *x.out.a : fresh(tokens, (int64_t)H * D, at::kBFloat16, *x.q);
    LAUNCH(rc, entry.prefill(x.q->data_ptr(), ld, tokens, x.k->data_ptr(), x.v->data_ptr(), (int)x.k->size(0), x.table->data_ptr(),
                             (int)x.table->size(1), cu->data_ptr(), offsets->data_ptr(), list.ptr(), out.data_ptr(), H * D, scale, window,
                             requests, max_new, H, Hk, D, (int)x.k->size(2), scratch.ptr(), splits, error, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

// (q, row stride, k_pool, v_pool, block table, seq_of_token, positions, scale, window, heads, kv heads, head size, requests,
//  token_rows, out, out rows, scratch, max_splits, piece tiles, single tokens, shape)
PyObject* decode_attention(PyObject*, PyObject* const* o, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 21) NOT_HERE;
    Attention x(o[0], o[2], o[3], o[4], o[14]);
    Arg seq(o[5]), positions(o[6]);
    Optional rows(o[13]), scratch(o[16]);
    Scalars sc;
    const int ld = sc.i(o[1]), window = sc.i(o[8]), H = sc.i(o[9]), Hk = sc.i(o[10]), D = sc.i(o[11]), requests = sc.i(o[12]),
              out_rows = sc.i(o[15]), splits = sc.i(o[17]), tiles = sc.i(o[18]), early = sc.i(o[19]), shape = sc.i(o[20]);
    const float scale = sc.f(o[7]);
    if (sc.bad || !x.fine(D) || !seq || !positions || !rows.ok || !scratch.is(at::kFloat)) NOT_HERE;
    at::Tensor out = x.out ? *x.out.a : fresh(out_rows, (int64_t)H * D, at::kBFloat16, *x.q);
    LAUNCH(rc, entry.decode(x.q->data_ptr(), ld, x.k->data_ptr(), x.v->data_ptr(), x.table->data_ptr(), (int)x.table->size(1), rows.ptr(),
                            seq->data_ptr(), positions->data_ptr(), scratch.ptr(), splits, out.data_ptr(), H * D, scale, window, requests, H,
                            Hk, D, (int)x.k->size(2), tiles, early, shape, s));
    return result(rc, std::move(out));
    END_HANDLE_TH_ERRORS
}

// (path of the kernel library): looks the entry points up; once, before any other call
PyObject* bind(PyObject*, PyObject* arg) {
    const char* path = PyUnicode_AsUTF8(arg);
    if (!path) return nullptr;
    void* lib = dlopen(path, RTLD_NOW);
    if (!lib) return PyErr_Format(PyExc_OSError, "%s", dlerror());
    const struct { const char* name; void** at; } wanted[] = {
        {"vx_add_rmsnorm", (void**)&entry.add_rmsnorm},
        {"vx_qk_norm_rope_kv_shared", (void**)&entry.qk_norm_rope_kv},
        {"vx_gated_act", (void**)&entry.gated_act},
        {"vx_gemm_skinny_act", (void**)&entry.gemm_skinny},
        {"vx_gemm_tcgen05_columns", (void**)&entry.gemm_tcgen05_columns},
        {"vx_gemm_tcgen05_pair", (void**)&entry.gemm_tcgen05_pair},
        {"vx_gemm_turned", (void**)&entry.gemm_turned},
        {"vx_paged_prefill_attention_tc", (void**)&entry.prefill},
        {"vx_paged_decode_attention_shape", (void**)&entry.decode},
    };
    for (const auto& w : wanted) {
        *w.at = dlsym(lib, w.name);
        if (!*w.at) return PyErr_Format(PyExc_OSError, "%s has no %s", path, w.name);
    }
    Py_RETURN_NONE;
}

#define FAST(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"bind", bind, METH_O, nullptr}, FAST(add_rmsnorm), FAST(qk_norm_rope_kv), FAST(gated_act), FAST(gemm_bf16),
                         FAST(gemm_tcgen05), FAST(gemm_turned), FAST(tcgen05_supported), FAST(prefill_attention), FAST(decode_attention),
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "velox_b200_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_velox_b200_calls() { return PyModule_Create(&module); }

// Python binding of the typed ops (metaltile_b200/ops.py) over the C ABI of include/mtcuda.h.
//
// A small call is bound by its host side: through ctypes the argument checks, the output allocation, the stream look-up
// and the conversion of a dozen arguments took 12-18 us of Python per call on a kernel of 3-5 us.  Here the tensors are
// looked at in C++ (no attribute of a tensor crosses into Python), the output comes straight from the caching allocator
// and the C ABI is called directly.  The module adds nothing to what the ops do: same arguments, checks and errors.
//
// Compiled by build.py with the host compiler against the headers of the installed PyTorch, linked to libmtcuda.so.
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/mtcuda.h"

namespace {

// ---- helpers -------------------------------------------------------------------------------------
struct PyErr {};                                // a Python exception is set

[[noreturn]] void raise(PyObject *type, const std::string &msg) {
    PyErr_SetString(type, msg.c_str());
    throw PyErr{};
}

const at::Tensor &tensor(PyObject *o, const char *what) {
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, std::string(what) + " must be a torch.Tensor");
    return THPVariable_Unpack(o);
}

long long integer(PyObject *o) {
    if (PyLong_Check(o)) {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) throw PyErr{};
        return v;
    }
    PyObject *n = PyNumber_Index(o);
    if (!n) throw PyErr{};
    const long long v = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (v == -1 && PyErr_Occurred()) throw PyErr{};
    return v;
}

int act_dtype(const at::Tensor &t) {            // -1: not an activation type
    switch (t.scalar_type()) {
        case at::kFloat: return MTC_F32;
        case at::kHalf: return MTC_F16;
        case at::kBFloat16: return MTC_BF16;
        default: return -1;
    }
}
int need_dtype(const at::Tensor &t) {
    const int dt = act_dtype(t);
    if (dt < 0) raise(PyExc_KeyError, std::string("dtype must be float32, float16 or bfloat16, got ") + c10::toString(t.scalar_type()));
    return dt;
}

void need_contiguous(std::initializer_list<const at::Tensor *> ts) {
    for (const at::Tensor *t : ts)
        if (!t->is_contiguous()) raise(PyExc_ValueError, "operands must be contiguous");
}

at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Tensor &like) {
    if (like.is_cuda()) return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
    return at::empty(size, like.options().dtype(type));
}

void check_out(const at::Tensor &out, int64_t M, int64_t N, const at::Tensor &like) {
    if (out.device() != like.device() || out.scalar_type() != like.scalar_type())
        raise(PyExc_TypeError, "out must live on the same device and have the dtype of x");
    if (out.numel() != M * N || !out.is_contiguous())
        raise(PyExc_ValueError, "out must be a contiguous block of M*N = " + std::to_string(M * N) +
                                    " elements (a column slice of a wider tensor with M > 1 is not)");
}

void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// Without the interpreter lock: an allocation and an entry of the library may wait (a full launch queue, a block that grows, the
// first load of a kernel) while other Python threads have work, on another GPU for instance.  Nothing of Python's inside; a C++
// exception takes the lock again on its way out.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    Unlocked() = default;
    Unlocked(const Unlocked &) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};
template <typename F>
int unlocked(F &&f) {
    const Unlocked u;
    return f();
}

// ---- the Context of a call ---------------------------------------------------------------------------
// ops.context(device) makes a device's Context on first use; it is looked up here once per device.
PyObject *g_context_fn = nullptr;               // ops.context
PyObject *g_by_device[64] = {};                 // what it returned
PyObject *s_handle = nullptr, *s_check = nullptr;

struct Call {
    PyObject *obj;                              // the Context (borrowed)
    mtc_ctx *h;

    Call(PyObject *given, const at::Tensor &on) {
        obj = given;
        if (given == Py_None || PyObject_IsTrue(given) == 0) {
            const int dev = on.is_cuda() ? on.device().index() : -1;
            if (dev >= 0 && dev < 64 && g_by_device[dev]) {
                obj = g_by_device[dev];
            } else {
                if (!g_context_fn) raise(PyExc_RuntimeError, "the binding is not set up (metaltile_b200.ops does it on import)");
                PyObject *d = THPVariable_Wrap(on);
                PyObject *device = d ? PyObject_GetAttrString(d, "device") : nullptr;
                Py_XDECREF(d);
                if (!device) throw PyErr{};
                obj = PyObject_CallOneArg(g_context_fn, device);
                Py_DECREF(device);
                if (!obj) throw PyErr{};
                if (dev >= 0 && dev < 64) g_by_device[dev] = obj;         // kept for the life of the process, like ops' own cache
                else Py_DECREF(obj);                                      // the cache of ops.context holds it
            }
        }
        load();
    }
    void load() {
        PyObject *v = PyObject_GetAttr(obj, s_handle);
        if (!v) throw PyErr{};
        h = v == Py_None ? nullptr : static_cast<mtc_ctx *>(PyLong_AsVoidPtr(v));
        Py_DECREF(v);
        if (PyErr_Occurred()) throw PyErr{};
    }
    void check(int rc) const {                  // Context._check raises MetalTileError with the context's message
        if (rc == MTC_OK) return;
        PyObject *code = PyLong_FromLong(rc);
        PyObject *r = code ? PyObject_CallMethodOneArg(obj, s_check, code) : nullptr;
        Py_XDECREF(code);
        Py_XDECREF(r);
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "mtcuda call failed");
        throw PyErr{};
    }
};

PyObject *wrap(at::Tensor t) {
    PyObject *o = THPVariable_Wrap(std::move(t));
    if (!o) throw PyErr{};
    return o;
}
PyObject *same(PyObject *o) {
    Py_INCREF(o);
    return o;
}

void nargs(Py_ssize_t n, Py_ssize_t want) {
    if (n != want) raise(PyExc_TypeError, "wrong number of arguments");
}

using Args = PyObject *const *;

// x as rows of its last dimension: (contiguous tensor of the rows, rows, K)
struct Rows {
    at::Tensor held;                            // only when a reshape made a new tensor
    const at::Tensor *t;
    int64_t M, K;
    explicit Rows(const at::Tensor &x) : t(&x) {
        if (x.dim() == 0) raise(PyExc_IndexError, "x must have at least one dimension");
        K = x.size(-1);
        if (!x.is_contiguous()) {
            held = x.reshape({-1, K});
            t = &held;
        }
        M = K > 0 ? x.numel() / K : 0;
    }
};

// The checks of a dense product: x [.., K], w [N, K*bits/32], scales / biases [N, K/group].
struct Dense {
    const at::Tensor &w, &scales, &biases, &x;
    Rows rows;
    int64_t bits, group, N;
    int dt;
    Dense(PyObject *w_, PyObject *s_, PyObject *b_, PyObject *x_, long long bits_, long long group_)
        : w(tensor(w_, "w")), scales(tensor(s_, "scales")), biases(tensor(b_, "biases")), x(tensor(x_, "x")), rows(x), bits(bits_),
          group(group_) {
        if (!(w.is_cuda() && scales.is_cuda() && biases.is_cuda() && x.is_cuda())) raise(PyExc_ValueError, "all operands must be CUDA tensors");
        if (w.scalar_type() != at::kInt && w.scalar_type() != at::kUInt32)
            raise(PyExc_TypeError, "w must hold packed 32-bit words (torch.int32 / torch.uint32)");
        dt = act_dtype(x);
        if (dt < 0 || scales.scalar_type() != x.scalar_type() || biases.scalar_type() != x.scalar_type())
            raise(PyExc_TypeError, "x, scales and biases must share one dtype in {f32, f16, bf16}");
        if (group <= 0) raise(group == 0 ? PyExc_ZeroDivisionError : PyExc_ValueError, "group_size must be positive");
        if (w.dim() != 2) raise(PyExc_ValueError, "w must be [N, K*bits/32]");
        N = w.size(0);
        if (w.size(1) * 32 != rows.K * bits)
            raise(PyExc_ValueError, "w has " + std::to_string(w.size(1)) + " words per row, expected K*bits/32 = " +
                                        std::to_string(static_cast<double>(rows.K * bits) / 32));
        if (scales.dim() != 2 || scales.size(0) != N || scales.size(1) != rows.K / group || biases.sizes() != scales.sizes())
            raise(PyExc_ValueError, "scales/biases must be [N, K/group_size]");
        need_contiguous({&w, &scales, &biases, rows.t});
    }
};

// ---- ops -----------------------------------------------------------------------------------------
// dense(which, w, scales, biases, x, bits, group_size, out, ctx): which 0 = qmv, 1 = qmm
PyObject *dense(Args a, Py_ssize_t n) {
    nargs(n, 9);
    const long long which = integer(a[0]);
    Dense d(a[1], a[2], a[3], a[4], integer(a[5]), integer(a[6]));
    const bool given = a[7] != Py_None;
    at::Tensor out = given ? tensor(a[7], "out") : at::Tensor();
    if (given) check_out(out, d.rows.M, d.N, d.x);
    const Call c(a[8], d.x);
    c.check(unlocked([&] {
        if (!given) out = empty({d.rows.M, d.N}, d.x.scalar_type(), d.x);
        return (which ? mtc_qmm : mtc_qmv)(c.h, stream(), d.w.data_ptr(), d.scales.data_ptr(), d.biases.data_ptr(), d.rows.t->data_ptr(),
                                           out.data_ptr(), static_cast<int>(d.rows.M), static_cast<int>(d.N), static_cast<int>(d.rows.K),
                                           static_cast<int>(d.bits), static_cast<int>(d.group), d.dt);
    }));
    return given ? same(a[7]) : wrap(std::move(out));
}

// qmv_batched(mats, x, bits, group_size, out, ctx)
PyObject *qmv_batched(Args a, Py_ssize_t n) {
    nargs(n, 6);
    PyObject *mats = PySequence_Fast(a[0], "mats must be a sequence of (w, scales, biases)");
    if (!mats) throw PyErr{};
    struct Hold { PyObject *o; ~Hold() { Py_DECREF(o); } } hold{mats};
    const Py_ssize_t count = PySequence_Fast_GET_SIZE(mats);
    const at::Tensor &x = tensor(a[1], "x");
    const Rows rows(x);
    const long long bits = integer(a[2]), group = integer(a[3]);
    const bool one = rows.M == 1;
    mtc_qmv_desc descs[4] = {};
    at::Tensor outs[4], whole;
    int64_t total = 0, ns[4] = {};
    if (count < 1 || count > 4) {
        const Call c(a[5], x);
        c.check(mtc_qmv_batched(c.h, stream(), descs, static_cast<int>(count)));         // (refused at once)
    }
    // held: another thread may change a list of the caller's while the lock is let go below
    struct Parts {
        PyObject *p[4][3] = {};
        PyObject **operator[](Py_ssize_t i) { return p[i]; }
        ~Parts() {
            for (auto &m : p)
                for (PyObject *o : m) Py_XDECREF(o);
        }
    } parts;
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject *m = PySequence_Fast_GET_ITEM(mats, i);
        if (PyTuple_Check(m) && PyTuple_GET_SIZE(m) == 3) {
            for (int j = 0; j < 3; ++j) parts[i][j] = same(PyTuple_GET_ITEM(m, j));
        } else if (PyList_Check(m) && PyList_GET_SIZE(m) == 3) {
            for (int j = 0; j < 3; ++j) parts[i][j] = same(PyList_GET_ITEM(m, j));
        } else {
            raise(PyExc_ValueError, "mats must hold (w, scales, biases) triples");
        }
        ns[i] = tensor(parts[i][0], "w").size(0);
        total += ns[i];
    }
    PyObject *xrows = rows.held.defined() ? THPVariable_Wrap(rows.held) : same(a[1]);
    if (!xrows) throw PyErr{};
    Hold hold_x{xrows};
    if (one) {
        if (a[4] == Py_None) {
            const Unlocked u;
            whole = empty({1, total}, x.scalar_type(), x);
        } else {
            whole = tensor(a[4], "out");
        }
    }
    int64_t col = 0;
    for (Py_ssize_t i = 0; i < count; ++i) {
        Dense d(parts[i][0], parts[i][1], parts[i][2], xrows, bits, group);
        void *dst = nullptr;
        if (!one) {
            {
                const Unlocked u;
                outs[i] = empty({rows.M, ns[i]}, x.scalar_type(), x);
            }
            dst = outs[i].data_ptr();
        } else if (a[4] == Py_None) {
            dst = static_cast<char *>(whole.data_ptr()) + col * static_cast<int64_t>(x.element_size());     // tiles of one row, side by side
        } else {
            const at::Tensor tile = whole.slice(1, col, col + ns[i]);
            check_out(tile, 1, ns[i], x);
            dst = tile.data_ptr();
        }
        mtc_qmv_desc &q = descs[i];
        q.w = d.w.data_ptr();
        q.scales = d.scales.data_ptr();
        q.biases = d.biases.data_ptr();
        q.x = d.rows.t->data_ptr();
        q.outs[0] = dst;
        q.n_outs = 1;
        q.M = static_cast<int>(rows.M);
        q.N = static_cast<int>(ns[i]);
        q.K = static_cast<int>(rows.K);
        q.bits = static_cast<int>(bits);
        q.group_size = static_cast<int>(group);
        q.dtype = d.dt;
        col += ns[i];
    }
    const Call c(a[5], x);
    c.check(unlocked([&] { return mtc_qmv_batched(c.h, stream(), descs, static_cast<int>(count)); }));
    if (one) return a[4] == Py_None ? wrap(std::move(whole)) : same(a[4]);
    PyObject *list = PyList_New(count);
    if (!list) throw PyErr{};
    for (Py_ssize_t i = 0; i < count; ++i) {
        PyObject *o = THPVariable_Wrap(outs[i]);
        if (!o) {
            Py_DECREF(list);
            throw PyErr{};
        }
        PyList_SET_ITEM(list, i, o);
    }
    return list;
}

// qvm(w, scales, biases, x, bits, group_size, out, ctx)
PyObject *qvm(Args a, Py_ssize_t n) {
    nargs(n, 8);
    const at::Tensor &w = tensor(a[0], "w"), &s = tensor(a[1], "scales"), &b = tensor(a[2], "biases"), &x = tensor(a[3], "x");
    const long long bits = integer(a[4]), group = integer(a[5]);
    need_contiguous({&w, &s, &b, &x});
    const Rows rows(x);
    if (bits <= 0 || group <= 0) raise(PyExc_ZeroDivisionError, "bits and group_size must be positive");
    const int64_t N = w.size(1) * 32 / bits;
    if (w.size(0) != rows.K || s.dim() != 2 || s.size(0) != rows.K / group || s.size(1) != N || b.sizes() != s.sizes())
        raise(PyExc_ValueError, "w must be [K, N*bits/32] and scales / biases [K/group_size, N]");
    const bool given = a[6] != Py_None;
    at::Tensor out = given ? tensor(a[6], "out") : at::Tensor();
    if (given) check_out(out, rows.M, N, x);
    const Call c(a[7], x);
    const int dt = need_dtype(x);
    c.check(unlocked([&] {
        if (!given) out = empty({rows.M, N}, x.scalar_type(), x);
        return mtc_qvm(c.h, stream(), w.data_ptr(), s.data_ptr(), b.data_ptr(), x.data_ptr(), out.data_ptr(), static_cast<int>(rows.M),
                       static_cast<int>(N), static_cast<int>(rows.K), static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    return given ? same(a[6]) : wrap(std::move(out));
}

// rms_norm_qmv(w, scales, biases, x, norm_weight, eps, bits, group_size, out, ctx)
PyObject *rms_norm_qmv(Args a, Py_ssize_t n) {
    nargs(n, 10);
    const at::Tensor &w = tensor(a[0], "w"), &s = tensor(a[1], "scales"), &b = tensor(a[2], "biases"), &x = tensor(a[3], "x"),
                     &nw = tensor(a[4], "norm_weight");
    const double eps = PyFloat_AsDouble(a[5]);
    if (eps == -1.0 && PyErr_Occurred()) throw PyErr{};
    const long long bits = integer(a[6]), group = integer(a[7]);
    const int64_t K = x.numel(), N = w.size(0);
    if (nw.numel() != K || w.size(1) * 32 != K * bits)
        raise(PyExc_ValueError, "x and norm_weight must have K elements and w must be [N, K*bits/32]");
    const bool given = a[8] != Py_None;
    at::Tensor out = given ? tensor(a[8], "out") : at::Tensor();
    if (given) check_out(out, 1, N, x);
    const Call c(a[9], x);
    const int dt = need_dtype(x);
    c.check(unlocked([&] {
        if (!given) out = empty({1, N}, x.scalar_type(), x);
        return mtc_rms_norm_qmv(c.h, stream(), x.data_ptr(), nw.data_ptr(), static_cast<float>(eps), w.data_ptr(), s.data_ptr(), b.data_ptr(),
                                out.data_ptr(), static_cast<int>(N), static_cast<int>(K), static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    return given ? same(a[8]) : wrap(std::move(out));
}

// swiglu(gate, up, out, ctx)
PyObject *swiglu(Args a, Py_ssize_t n) {
    nargs(n, 4);
    const at::Tensor &g = tensor(a[0], "gate"), &u = tensor(a[1], "up");
    const bool given = a[2] != Py_None;
    at::Tensor out = given ? tensor(a[2], "out") : at::Tensor();
    const Call c(a[3], g);
    const int dt = need_dtype(g);
    c.check(unlocked([&] {
        if (!given) out = g.is_contiguous() ? empty(g.sizes(), g.scalar_type(), g) : at::empty_like(g);
        return mtc_swiglu(c.h, stream(), g.data_ptr(), u.data_ptr(), out.data_ptr(), static_cast<size_t>(g.numel()), dt);
    }));
    return given ? same(a[2]) : wrap(std::move(out));
}

// moe_router_topk(logits, k, norm_topk_prob, ctx) -> (indices, weights)
PyObject *moe_router_topk(Args a, Py_ssize_t n) {
    nargs(n, 4);
    const at::Tensor &l = tensor(a[0], "logits");
    if (l.dim() != 2) raise(PyExc_ValueError, "logits must be [rows, n_experts]");
    const int64_t k = integer(a[1]), norm = integer(a[2]);
    at::Tensor idx, wts;
    const Call c(a[3], l);
    const int dt = need_dtype(l);
    c.check(unlocked([&] {
        idx = empty({l.size(0), k}, at::kInt, l);
        wts = empty({l.size(0), k}, l.scalar_type(), l);
        return mtc_moe_router_topk(c.h, stream(), l.data_ptr(), idx.data_ptr(), wts.data_ptr(), static_cast<int>(l.size(0)),
                                   static_cast<int>(l.size(1)), static_cast<int>(k), static_cast<int>(norm), dt);
    }));
    PyObject *i = wrap(std::move(idx)), *w = THPVariable_Wrap(std::move(wts));
    PyObject *t = w ? PyTuple_Pack(2, i, w) : nullptr;
    Py_DECREF(i);
    Py_XDECREF(w);
    if (!t) throw PyErr{};
    return t;
}

// moe_sort(topk_idx, n_experts, ctx) -> (sort_token_idx, inv_perm, expert_offsets, row_expert)
PyObject *moe_sort(Args a, Py_ssize_t n) {
    nargs(n, 3);
    const at::Tensor &idx = tensor(a[0], "topk_idx");
    if (idx.dim() != 2) raise(PyExc_ValueError, "topk_idx must be [n_tokens, k]");
    const int64_t T = idx.size(0), k = idx.size(1), E = integer(a[1]);
    at::Tensor r[4];
    const Call c(a[2], idx);
    c.check(unlocked([&] {
        r[0] = empty({T * k}, at::kInt, idx);
        r[1] = empty({T, k}, at::kInt, idx);
        r[2] = empty({E + 1}, at::kInt, idx);
        r[3] = empty({T * k}, at::kInt, idx);
        return mtc_moe_sort(c.h, stream(), idx.data_ptr(), static_cast<int>(T), static_cast<int>(k), static_cast<int>(E), r[0].data_ptr(),
                            r[1].data_ptr(), r[2].data_ptr(), r[3].data_ptr());
    }));
    PyObject *t = PyTuple_New(4);
    if (!t) throw PyErr{};
    for (int i = 0; i < 4; ++i) {
        PyObject *o = THPVariable_Wrap(std::move(r[i]));
        if (!o) {
            Py_DECREF(t);
            throw PyErr{};
        }
        PyTuple_SET_ITEM(t, i, o);
    }
    return t;
}

// moe_permute(tokens, sort_token_idx, out, ctx)
PyObject *moe_permute(Args a, Py_ssize_t n) {
    nargs(n, 4);
    const at::Tensor &tok = tensor(a[0], "tokens"), &idx = tensor(a[1], "sort_token_idx");
    const int64_t rows = idx.numel(), hidden = tok.size(1);
    const bool given = a[2] != Py_None;
    at::Tensor out = given ? tensor(a[2], "out") : at::Tensor();
    const Call c(a[3], tok);
    const int dt = need_dtype(tok);
    c.check(unlocked([&] {
        if (!given) out = empty({rows, hidden}, tok.scalar_type(), tok);
        return mtc_moe_permute(c.h, stream(), tok.data_ptr(), idx.data_ptr(), out.data_ptr(), static_cast<int>(rows), static_cast<int>(hidden), dt);
    }));
    return given ? same(a[2]) : wrap(std::move(out));
}

// moe_unpermute(expert_outputs, inv_perm, weights, out, ctx)
PyObject *moe_unpermute(Args a, Py_ssize_t n) {
    nargs(n, 5);
    const at::Tensor &eo = tensor(a[0], "expert_outputs"), &inv = tensor(a[1], "inv_perm"), &wts = tensor(a[2], "weights");
    if (inv.dim() != 2) raise(PyExc_ValueError, "inv_perm must be [n_tokens, k]");
    const int64_t T = inv.size(0), k = inv.size(1), hidden = eo.size(1);
    const bool given = a[3] != Py_None;
    at::Tensor out = given ? tensor(a[3], "out") : at::Tensor();
    const Call c(a[4], eo);
    const int dt = need_dtype(eo);
    c.check(unlocked([&] {
        if (!given) out = empty({T, hidden}, eo.scalar_type(), eo);
        return mtc_moe_unpermute(c.h, stream(), eo.data_ptr(), inv.data_ptr(), wts.data_ptr(), out.data_ptr(), static_cast<int>(T),
                                 static_cast<int>(hidden), static_cast<int>(k), dt);
    }));
    return given ? same(a[3]) : wrap(std::move(out));
}

// gather_qmm(x, w, scales, biases, bits, group_size, expert_offsets, indices, out, ctx)
PyObject *gather_qmm(Args a, Py_ssize_t n) {
    nargs(n, 10);
    if ((a[6] == Py_None) == (a[7] == Py_None)) raise(PyExc_ValueError, "give exactly one of expert_offsets and indices");
    const at::Tensor &x = tensor(a[0], "x"), &w = tensor(a[1], "w"), &s = tensor(a[2], "scales"), &b = tensor(a[3], "biases");
    const long long bits = integer(a[4]), group = integer(a[5]);
    if (x.dim() != 2) raise(PyExc_ValueError, "x must be [rows, k_in]");
    const int64_t M = x.size(0), K = x.size(1);
    if (w.dim() != 3 || w.size(2) * 32 != K * bits) raise(PyExc_ValueError, "w must be [E, n_out, k_in*bits/32]");
    const int64_t E = w.size(0), N = w.size(1);
    if (group <= 0) raise(PyExc_ZeroDivisionError, "group_size must be positive");
    if (s.dim() != 3 || s.size(0) != E || s.size(1) != N || s.size(2) != K / group || b.sizes() != s.sizes())
        raise(PyExc_ValueError, "scales/biases must be [E, n_out, k_in/group_size]");
    need_contiguous({&x, &w, &s, &b});
    const bool given = a[8] != Py_None;
    at::Tensor out = given ? tensor(a[8], "out") : at::Tensor();
    if (given) check_out(out, M, N, x);
    const void *off = a[6] == Py_None ? nullptr : tensor(a[6], "expert_offsets").data_ptr();
    const void *ids = a[7] == Py_None ? nullptr : tensor(a[7], "indices").data_ptr();
    const Call c(a[9], x);
    const int dt = need_dtype(x);
    c.check(unlocked([&] {
        if (!given) out = empty({M, N}, x.scalar_type(), x);
        return mtc_gather_qmm(c.h, stream(), x.data_ptr(), w.data_ptr(), s.data_ptr(), b.data_ptr(), off, ids, out.data_ptr(),
                              static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(E), static_cast<int>(bits),
                              static_cast<int>(group), dt);
    }));
    return given ? same(a[8]) : wrap(std::move(out));
}

// (w, scales, biases) of one stacked expert matrix
struct Stacked {
    const at::Tensor *t[3];
    mtc_qmat m;
    Stacked(PyObject *o, const char *what) {
        if (!PyTuple_Check(o) && !PyList_Check(o)) raise(PyExc_TypeError, std::string(what) + " must be (w, scales, biases)");
        if (PySequence_Fast_GET_SIZE(o) < 3) raise(PyExc_IndexError, std::string(what) + " must be (w, scales, biases)");
        for (int j = 0; j < 3; ++j) t[j] = &tensor(PySequence_Fast_GET_ITEM(o, j), what);
        m.w = t[0]->data_ptr();
        m.scales = t[1]->data_ptr();
        m.biases = t[2]->data_ptr();
    }
};

// moe_experts(x, gate, up, down, bits, group_size, expert_offsets, sort_token_idx, out, ctx)
PyObject *moe_experts(Args a, Py_ssize_t n) {
    nargs(n, 10);
    const at::Tensor &x = tensor(a[0], "x");
    const Stacked g(a[1], "gate"), u(a[2], "up"), d(a[3], "down");
    const long long bits = integer(a[4]), group = integer(a[5]);
    if (x.dim() != 2 || g.t[0]->dim() != 3 || d.t[0]->dim() != 3)
        raise(PyExc_ValueError, "gate / up must be [E, inter, hidden*bits/32] and down [E, hidden, inter*bits/32] for x [rows, hidden]");
    const int64_t E = g.t[0]->size(0), inter = g.t[0]->size(1), hidden = d.t[0]->size(1);
    const at::Tensor &off = tensor(a[6], "expert_offsets");
    const at::Tensor *order = a[7] == Py_None ? nullptr : &tensor(a[7], "sort_token_idx");
    const int64_t M = order ? order->numel() : x.size(0);
    if (x.size(1) != hidden || g.t[0]->size(2) * 32 != hidden * bits || d.t[0]->size(2) * 32 != inter * bits)
        raise(PyExc_ValueError, "gate / up must be [E, inter, hidden*bits/32] and down [E, hidden, inter*bits/32] for x [rows, hidden]");
    need_contiguous({&x, g.t[0], g.t[1], g.t[2], u.t[0], u.t[1], u.t[2], d.t[0], d.t[1], d.t[2]});
    const bool given = a[8] != Py_None;
    at::Tensor out = given ? tensor(a[8], "out") : at::Tensor();
    if (given) check_out(out, M, hidden, x);
    const Call c(a[9], x);
    const int dt = need_dtype(x);
    c.check(unlocked([&] {
        if (!given) out = empty({M, hidden}, x.scalar_type(), x);
        return mtc_moe_experts(c.h, stream(), x.data_ptr(), order ? order->data_ptr() : nullptr, static_cast<int>(x.size(0)), &g.m, &u.m, &d.m,
                               off.data_ptr(), out.data_ptr(), static_cast<int>(M), static_cast<int>(hidden), static_cast<int>(inter),
                               static_cast<int>(E), static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    return given ? same(a[8]) : wrap(std::move(out));
}

// affine_quantize(w, bits, group_size, ctx) -> (packed, scales, biases)
PyObject *affine_quantize(Args a, Py_ssize_t n) {
    nargs(n, 4);
    const at::Tensor &w = tensor(a[0], "w");
    const long long bits = integer(a[1]), group = integer(a[2]);
    if (!w.is_contiguous()) raise(PyExc_ValueError, "w must be contiguous");
    if (w.dim() == 0) raise(PyExc_IndexError, "w must have at least one dimension");
    if (group <= 0) raise(PyExc_ZeroDivisionError, "group_size must be positive");
    const int64_t K = w.size(-1);
    if (K % group || (group * bits) % 32)
        raise(PyExc_ValueError, "the last dimension must hold whole groups and group_size * bits must be a multiple of 32");
    at::Tensor r[3];
    const Call c(a[3], w);
    const int dt = need_dtype(w);
    c.check(unlocked([&] {
        std::vector<int64_t> shape(w.sizes().begin(), w.sizes().end());
        shape.back() = K * bits / 32;
        r[0] = empty(shape, at::kInt, w);
        shape.back() = K / group;
        r[1] = empty(shape, w.scalar_type(), w);
        r[2] = empty(shape, w.scalar_type(), w);
        return mtc_affine_quantize(c.h, stream(), w.data_ptr(), r[0].data_ptr(), r[1].data_ptr(), r[2].data_ptr(), static_cast<size_t>(w.numel()),
                                   static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    PyObject *t = PyTuple_New(3);
    if (!t) throw PyErr{};
    for (int i = 0; i < 3; ++i) {
        PyObject *o = THPVariable_Wrap(std::move(r[i]));
        if (!o) {
            Py_DECREF(t);
            throw PyErr{};
        }
        PyTuple_SET_ITEM(t, i, o);
    }
    return t;
}

// affine_dequantize(w, scales, biases, bits, group_size, ctx)
PyObject *affine_dequantize(Args a, Py_ssize_t n) {
    nargs(n, 6);
    const at::Tensor &w = tensor(a[0], "w"), &s = tensor(a[1], "scales"), &b = tensor(a[2], "biases");
    const long long bits = integer(a[3]), group = integer(a[4]);
    need_contiguous({&w, &s, &b});
    if (bits == 0) raise(PyExc_ZeroDivisionError, "bits must be positive");
    if (w.dim() == 0) raise(PyExc_IndexError, "w must have at least one dimension");
    std::vector<int64_t> shape(w.sizes().begin(), w.sizes().end());
    shape.back() = w.size(-1) * 32 / bits;
    at::Tensor out;
    const Call c(a[5], w);
    const int dt = need_dtype(s);
    c.check(unlocked([&] {
        out = empty(shape, s.scalar_type(), w);
        return mtc_affine_dequantize(c.h, stream(), w.data_ptr(), s.data_ptr(), b.data_ptr(), out.data_ptr(), static_cast<size_t>(out.numel()),
                                     static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    return wrap(std::move(out));
}

// dequant_gather(weight, scales, biases, indices, bits, group_size, ctx)
PyObject *dequant_gather(Args a, Py_ssize_t n) {
    nargs(n, 7);
    const at::Tensor &w = tensor(a[0], "weight"), &s = tensor(a[1], "scales"), &b = tensor(a[2], "biases"), &idx = tensor(a[3], "indices");
    const long long bits = integer(a[4]), group = integer(a[5]);
    need_contiguous({&w, &s, &b, &idx});
    if (bits == 0) raise(PyExc_ZeroDivisionError, "bits must be positive");
    const int64_t vocab = w.size(0), hidden = w.size(1) * 32 / bits, T = idx.numel();
    at::Tensor out;
    const Call c(a[6], w);
    const int dt = need_dtype(s);
    c.check(unlocked([&] {
        out = empty({T, hidden}, s.scalar_type(), w);
        return mtc_dequant_gather(c.h, stream(), w.data_ptr(), s.data_ptr(), b.data_ptr(), idx.data_ptr(), out.data_ptr(), static_cast<size_t>(T),
                                  static_cast<int>(hidden), static_cast<int>(vocab), static_cast<int>(bits), static_cast<int>(group), dt);
    }));
    return wrap(std::move(out));
}

// unpack_codes(w, K, bits, ctx)
PyObject *unpack_codes(Args a, Py_ssize_t n) {
    nargs(n, 4);
    const at::Tensor &w = tensor(a[0], "w");
    const int64_t K = integer(a[1]), bits = integer(a[2]), N = w.size(0);
    at::Tensor codes;
    const Call c(a[3], w);
    c.check(unlocked([&] {
        codes = empty({N, K}, at::kByte, w);
        return mtc_unpack_codes(c.h, stream(), w.data_ptr(), codes.data_ptr(), static_cast<int>(N), static_cast<int>(K), static_cast<int>(bits));
    }));
    return wrap(std::move(codes));
}

// ---- module ----------------------------------------------------------------------------------------
PyObject *set_context(PyObject *, PyObject *fn) {
    Py_INCREF(fn);
    Py_XSETREF(g_context_fn, fn);
    Py_RETURN_NONE;
}

// C++ exceptions (ours and torch's) become Python ones at this boundary
template <PyObject *(*F)(Args, Py_ssize_t)>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        return F(args, n);
    } catch (const PyErr &) {
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

#define OP(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    OP(dense), OP(qmv_batched), OP(qvm), OP(rms_norm_qmv), OP(swiglu), OP(moe_router_topk), OP(moe_sort), OP(moe_permute), OP(moe_unpermute),
    OP(gather_qmm), OP(moe_experts), OP(affine_quantize), OP(affine_dequantize), OP(dequant_gather), OP(unpack_codes),
    {"set_context", set_context, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "typed ops on torch tensors over the C ABI of libmtcuda.so", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
    s_handle = PyUnicode_InternFromString("_handle");
    s_check = PyUnicode_InternFromString("_check");
    PyObject *m = s_handle && s_check ? PyModule_Create(&module) : nullptr;
    if (m && PyModule_AddStringConstant(m, "torch_version", MTC_TORCH_VERSION) != 0) Py_CLEAR(m);       // ops.py compares it with the PyTorch in the process
    return m;
}

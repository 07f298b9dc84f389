// Host side of the Python mirror: what lisa_b200/ops.py does between a caller's tensors and the C ABI -- checks, output
// allocation, argument tables, the current stream -- as compiled functions.  A decode step is dozens of calls of a few
// microseconds of GPU time each; the same steps in Python (tensor methods, ctypes conversion of fifteen arguments) took 25 to
// 40 us a call and were the bound of every small case.
//
// torch is the allocator and the source of streams here, nothing else: every product is a call of the C ABI
// (include/lisa_cuda.h).  Each function raises the LisaError that the Python form raised.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <vector>

#include "lisa_cuda.h"

namespace {

PyObject *g_error_class = nullptr;

struct LisaFailure {
    int code;
    std::string message;
};
struct PythonFailure {};  // a Python exception is already set

[[noreturn]] void refuse(int code, const char *message) { throw LisaFailure{code, message}; }

void check(int rc) {
    if (rc != LISA_OK) throw LisaFailure{rc, lisa_cuda_last_error_string()};
}
// A call of the library without the interpreter's lock: where a stream's queue is full a launch waits, and other threads (among them
// those that such a stream may be waiting for) go on.
template <typename F>
void enqueue(F &&call) {
    struct Unlocked {
        PyThreadState *state = PyEval_SaveThread();
        ~Unlocked() { PyEval_RestoreThread(state); }
    };
    int rc;
    {
        Unlocked here;
        rc = call();
    }
    check(rc);
}

// A tensor argument; `optional` lets None through as an undefined tensor.
const at::Tensor &tensor(PyObject *o, bool optional = false) {
    static const at::Tensor none;
    if (o == Py_None && optional) return none;
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "expected a torch.Tensor, got %s", Py_TYPE(o)->tp_name);
        throw PythonFailure{};
    }
    return THPVariable_Unpack(o);
}
void need_cuda(const at::Tensor &t) {
    if (t.defined() && !t.is_cuda()) refuse(LISA_ERR_BAD_ARG, "tensor is not on a CUDA device (no CPU fallback)");
}
int64_t integer(PyObject *o) {
    if (PyLong_CheckExact(o)) {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) throw PythonFailure{};
        return v;
    }
    PyObject *n = PyNumber_Index(o);
    if (!n) throw PythonFailure{};
    const long long v = PyLong_AsLongLong(n);
    Py_DECREF(n);
    if (v == -1 && PyErr_Occurred()) throw PythonFailure{};
    return v;
}
double real(PyObject *o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw PythonFailure{};
    return v;
}
bool truth(PyObject *o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw PythonFailure{};
    return v != 0;
}
at::Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const at::Tensor &like) {
    return at::detail::empty_cuda(size, dtype, like.device(), std::nullopt);
}
at::Tensor empty(at::IntArrayRef size, const at::Tensor &like) { return empty(size, like.scalar_type(), like); }
// The stream of a call: None: the current one; else an object with a `cuda_stream`, or the handle itself.  While this lives, tensors are
// allocated and copied on that stream, so that what ends with the call (contiguous copies, workspaces) goes back to the pool of
// the stream that still reads it.  Outputs belong to the caller's current stream (`output`).
class CallStream {
  public:
    explicit CallStream(PyObject *o) : caller_(c10::cuda::getCurrentCUDAStream()), handle_(caller_.stream()) {
        if (o == Py_None) return;
        if (PyObject *h = PyObject_GetAttrString(o, "cuda_stream")) {
            handle_ = handle(h);
            Py_DECREF(h);
        } else {
            PyErr_Clear();
            handle_ = handle(o);
        }
        if (handle_ != caller_.stream()) guard_.reset_stream(c10::cuda::getStreamFromExternal(handle_, caller_.device_index()));
    }
    operator lisa_stream_t() const { return handle_; }
    at::Tensor output(at::IntArrayRef size, at::ScalarType dtype, const at::Tensor &like) const {
        c10::cuda::OptionalCUDAStreamGuard back;
        if (handle_ != caller_.stream()) back.reset_stream(caller_);
        return empty(size, dtype, like);
    }
    at::Tensor output(at::IntArrayRef size, const at::Tensor &like) const { return output(size, like.scalar_type(), like); }

  private:
    static cudaStream_t handle(PyObject *o) { return reinterpret_cast<cudaStream_t>(integer(o)); }
    c10::cuda::CUDAStream caller_;
    cudaStream_t handle_;
    c10::cuda::OptionalCUDAStreamGuard guard_;
};
int dtype_code(const at::Tensor &t) {
    switch (t.scalar_type()) {
        case at::kBFloat16: return LISA_BF16;
        case at::kHalf: return LISA_F16;
        case at::kFloat: return LISA_F32;
        default: throw LisaFailure{LISA_ERR_UNSUPPORTED, "unsupported compute dtype torch." + std::string(c10::toString(t.scalar_type()))};
    }
}
at::Tensor whole(const at::Tensor &t) { return !t.defined() || t.is_contiguous() ? t : t.contiguous(); }
at::Tensor words(const at::Tensor &w) {
    if (w.scalar_type() != at::kInt && w.scalar_type() != at::kUInt32)
        throw LisaFailure{LISA_ERR_BAD_ARG, "packed weights must be uint32 words, got torch." + std::string(c10::toString(w.scalar_type()))};
    return whole(w);
}
const void *ptr(const at::Tensor &t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void *out_ptr(const at::Tensor &t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
template <typename T>
const T *ptr_of(const at::Tensor &t) { return reinterpret_cast<const T *>(ptr(t)); }
template <typename T>
T *out_of(const at::Tensor &t) { return reinterpret_cast<T *>(out_ptr(t)); }

// x's leading sizes followed by n
c10::SmallVector<int64_t, 5> with_last(const at::Tensor &x, int64_t n) {
    c10::SmallVector<int64_t, 5> s(x.sizes().begin(), x.sizes().end());
    s.back() = n;
    return s;
}
int64_t rows_of(const at::Tensor &x, int64_t k) { return k > 0 ? x.numel() / k : 0; }
PyObject *wrap(const at::Tensor &t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}
PyObject *list_of(const at::Tensor *t, int count) {
    PyObject *l = PyList_New(count);
    if (!l) throw PythonFailure{};
    for (int i = 0; i < count; ++i) PyList_SET_ITEM(l, i, THPVariable_Wrap(t[i]));
    return l;
}
PyObject *tuple_of(std::initializer_list<PyObject *> items) {  // steals the references
    PyObject *t = PyTuple_New(static_cast<Py_ssize_t>(items.size()));
    Py_ssize_t i = 0;
    for (PyObject *o : items) PyTuple_SET_ITEM(t, i++, o);
    return t;
}

// One to three (weight, scales, biases) and their outputs, as the tables of the C ABI.
constexpr int kMaxLinears = 16;  // (more than the library takes: it is the one that refuses them)
struct Linears {
    int count = 0;
    at::Tensor keep[kMaxLinears][3], y[kMaxLinears];
    const uint32_t *w[kMaxLinears];
    const void *s[kMaxLinears], *b[kMaxLinears];
    void *out[kMaxLinears];
    int64_t n[kMaxLinears];
    void add(PyObject *w_o, PyObject *s_o, PyObject *b_o) {
        const at::Tensor &wt = tensor(w_o), &st = tensor(s_o), &bt = tensor(b_o);
        need_cuda(wt);
        need_cuda(st);
        need_cuda(bt);
        keep[count][0] = words(wt);
        keep[count][1] = whole(st);
        keep[count][2] = whole(bt);
        w[count] = ptr_of<uint32_t>(keep[count][0]);
        s[count] = ptr(keep[count][1]);
        b[count] = ptr(keep[count][2]);
        n[count] = keep[count][0].size(0);
        ++count;
    }
    void read(PyObject *seq) {
        PyObject *fast = PySequence_Fast(seq, "linears: a sequence of (weight, scales, biases)");
        if (!fast) throw PythonFailure{};
        const Py_ssize_t c = PySequence_Fast_GET_SIZE(fast);
        try {
            if (c > kMaxLinears) refuse(LISA_ERR_BAD_ARG, "one to three linears");
            for (Py_ssize_t i = 0; i < c; ++i) {
                PyObject *one = PySequence_Fast(PySequence_Fast_GET_ITEM(fast, i), "a linear is (weight, scales, biases)");
                if (!one) throw PythonFailure{};
                try {
                    if (PySequence_Fast_GET_SIZE(one) != 3) {
                        PyErr_SetString(PyExc_ValueError, "a linear is (weight, scales, biases)");
                        throw PythonFailure{};
                    }
                    add(PySequence_Fast_GET_ITEM(one, 0), PySequence_Fast_GET_ITEM(one, 1), PySequence_Fast_GET_ITEM(one, 2));
                } catch (...) {
                    Py_DECREF(one);
                    throw;
                }
                Py_DECREF(one);
            }
        } catch (...) {
            Py_DECREF(fast);
            throw;
        }
        Py_DECREF(fast);
    }
    void fit(int i, int64_t k, int64_t group_size, int64_t bits, const char *message) const {
        if (bits <= 0 || keep[i][0].size(-1) * 32 / bits != k || keep[i][1].size(-1) * group_size != k) refuse(LISA_ERR_BAD_ARG, message);
    }
};

using Args = PyObject *const *;

template <typename F>
PyObject *guarded(Py_ssize_t got, Py_ssize_t want, F &&body) {
    if (got != want) {
        PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, got);
        return nullptr;
    }
    try {
        return body();
    } catch (const PythonFailure &) {
    } catch (const LisaFailure &f) {
        if (PyObject *e = PyObject_CallFunction(g_error_class, "is", f.code, f.message.c_str())) {
            PyErr_SetObject(g_error_class, e);
            Py_DECREF(e);
        }
    } catch (const std::exception &e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

// x, w, scales, biases, transpose, group_size, bits, stream, out, flags
PyObject *quantized_matmul(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 10, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]), &w0 = tensor(a[1]), &s0 = tensor(a[2]), &b0 = tensor(a[3], true), &out = tensor(a[8], true);
        need_cuda(x);
        need_cuda(w0);
        need_cuda(s0);
        need_cuda(b0);
        const CallStream stream(a[7]);
        const int64_t k = x.size(-1), m = rows_of(x, k), gs = integer(a[5]), bits = integer(a[6]);
        const at::Tensor xc = whole(x), w = words(w0), s = whole(s0), b = whole(b0);
        const int64_t n = w.size(0);
        if (bits <= 0 || w.size(-1) * 32 / bits != k || s.size(-1) * gs != k) refuse(LISA_ERR_BAD_ARG, "quantized_matmul: shapes of x, w and scales disagree");
        const at::Tensor y = out.defined() ? out : stream.output(with_last(x, n), x);
        const int transpose = truth(a[4]);
        const unsigned flags = static_cast<unsigned>(integer(a[9]));
        enqueue([&] {
            return lisa_cuda_quantized_matmul_ex(stream, ptr(xc), m, k, ptr_of<uint32_t>(w), ptr(s), ptr(b), n, transpose, static_cast<int>(gs),
                                            static_cast<int>(bits), dtype_code(xc), out_ptr(y), flags);
        });
        return wrap(out.defined() ? y.reshape(with_last(x, n)) : y);
    });
}

// x, linears, transpose, group_size, bits, stream, flags
PyObject *quantized_matmul_siblings(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 7, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]);
        need_cuda(x);
        const CallStream stream(a[5]);
        const int64_t k = x.size(-1), m = rows_of(x, k), gs = integer(a[3]), bits = integer(a[4]);
        const at::Tensor xc = whole(x);
        Linears l;
        l.read(a[1]);
        for (int i = 0; i < l.count; ++i) {
            l.fit(i, k, gs, bits, "quantized_matmul_siblings: shapes of x, w and scales disagree");
            l.y[i] = stream.output(with_last(x, l.n[i]), x);
            l.out[i] = out_ptr(l.y[i]);
        }
        const int transpose = truth(a[2]);
        const unsigned flags = static_cast<unsigned>(integer(a[6]));
        enqueue([&] {
            return lisa_cuda_quantized_matmul_siblings(stream, ptr(xc), m, k, l.count, l.w, l.s, l.b, l.n, transpose, static_cast<int>(gs),
                                                  static_cast<int>(bits), dtype_code(xc), l.out, flags);
        });
        return list_of(l.y, l.count);
    });
}

// x, residual, norm_weight, eps, linears, group_size, bits, write_norm, stream, flags
PyObject *quantized_matmul_addnorm(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 10, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]), &r = tensor(a[1]), &nw = tensor(a[2]);
        need_cuda(x);
        need_cuda(r);
        need_cuda(nw);
        const CallStream stream(a[8]);
        const int64_t k = x.size(-1), m = rows_of(x, k), gs = integer(a[5]), bits = integer(a[6]);
        const at::Tensor xc = whole(x), rc = whole(r), nc = whole(nw);
        if (rc.numel() != xc.numel()) throw std::runtime_error("shape '" + std::to_string(m) + " x " + std::to_string(k) + "' is invalid for the residual");
        Linears l;
        l.read(a[4]);
        for (int i = 0; i < l.count; ++i) {
            l.fit(i, k, gs, bits, "quantized_matmul_addnorm: shapes of x, w and scales disagree");
            l.y[i] = stream.output(with_last(x, l.n[i]), x);
            l.out[i] = out_ptr(l.y[i]);
        }
        const at::Tensor total = stream.output(x.sizes(), x), normed = truth(a[7]) ? stream.output(x.sizes(), x) : at::Tensor();
        const unsigned flags = static_cast<unsigned>(integer(a[9]));
        const float eps = static_cast<float>(real(a[3]));
        enqueue([&] {
            return lisa_cuda_quantized_matmul_addnorm(stream, ptr(xc), ptr(rc), ptr(nc), eps, m, k, l.count, l.w, l.s, l.b,
                                                 l.n, 1, static_cast<int>(gs), static_cast<int>(bits), dtype_code(xc), l.out, out_ptr(total),
                                                 out_ptr(normed), flags);
        });
        return tuple_of({list_of(l.y, l.count), wrap(total), wrap(normed)});
    });
}

// gate, up, w, scales, biases, group_size, bits, write_act, stream, flags
PyObject *quantized_matmul_swiglu(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 10, [&]() -> PyObject * {
        const at::Tensor &g = tensor(a[0]), &u = tensor(a[1]);
        need_cuda(g);
        need_cuda(u);
        const CallStream stream(a[8]);
        const int64_t k = g.size(-1), m = rows_of(g, k), gs = integer(a[5]), bits = integer(a[6]);
        const at::Tensor gc = whole(g), uc = whole(u);
        if (uc.numel() != gc.numel()) throw std::runtime_error("swiglu: gate and up differ in size");
        Linears l;
        l.add(a[2], a[3], a[4]);
        const at::Tensor y = stream.output(with_last(g, l.n[0]), g), act = truth(a[7]) ? stream.output(g.sizes(), g) : at::Tensor();
        // decode rows: a place for the activation, so that the library may form it once (rows too long for the one-launch kernels then run as
        // two steps)
        const at::Tensor scratch = !act.defined() && m > 2 && m <= 8 && gs == 64 && bits != 8 ? empty(g.sizes(), g) : act;
        const unsigned flags = static_cast<unsigned>(integer(a[9]));
        enqueue([&] {
            return lisa_cuda_quantized_matmul_swiglu(stream, ptr(gc), ptr(uc), m, k, l.w[0], l.s[0], l.b[0], l.n[0], 1, static_cast<int>(gs),
                                                static_cast<int>(bits), dtype_code(gc), out_ptr(y), out_ptr(scratch), flags);
        });
        return tuple_of({wrap(y), wrap(act)});
    });
}

// w, scales, biases, ids, group_size, bits, stream
PyObject *dequantize_rows(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 7, [&]() -> PyObject * {
        const at::Tensor &ids = tensor(a[3]);
        need_cuda(ids);
        const CallStream stream(a[6]);
        Linears l;
        l.add(a[0], a[1], a[2]);
        const int64_t gs = integer(a[4]), bits = integer(a[5]);
        if (bits <= 0) refuse(LISA_ERR_UNSUPPORTED, "dequantize_rows: bits must be 2, 4 or 8");
        const at::Tensor &s = l.keep[0][1];
        const int64_t k = l.keep[0][0].size(-1) * 32 / bits;
        const at::Tensor flat = whole(ids.scalar_type() == at::kInt ? ids : ids.to(at::kInt));
        c10::SmallVector<int64_t, 5> size(ids.sizes().begin(), ids.sizes().end());
        size.push_back(k);
        const at::Tensor out = stream.output(size, s);
        enqueue([&] {
            return lisa_cuda_dequantize_rows(stream, l.w[0], l.s[0], l.b[0], ptr_of<int32_t>(flat), flat.numel(), l.n[0], k, static_cast<int>(gs),
                                        static_cast<int>(bits), dtype_code(s), out_ptr(out));
        });
        return wrap(out);
    });
}

// fmt, weights, input, stream
PyObject *packed_matvec(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 4, [&]() -> PyObject * {
        const at::Tensor &w = tensor(a[1]), &x = tensor(a[2]);
        need_cuda(w);
        need_cuda(x);
        const CallStream stream(a[3]);
        const int code = static_cast<int>(integer(a[0]));
        if (w.dim() != 2 || w.scalar_type() != at::kByte || !w.is_contiguous()) refuse(LISA_ERR_BAD_ARG, "unsupported GGUF quantized matvec layout");
        if (x.dim() != 2 || x.scalar_type() != at::kFloat) refuse(LISA_ERR_BAD_ARG, "invalid GGUF matvec input rows");
        const int64_t rows = w.size(0), row_bytes = w.size(1), tokens = x.size(0);
        const int64_t block = code == LISA_GGUF_Q2_K ? 84 : code == LISA_GGUF_Q4_K ? 144 : code == LISA_GGUF_Q5_K ? 176 : 0;
        if (block && row_bytes % block == 0 && x.size(1) != row_bytes / block * 256)
            refuse(LISA_ERR_BAD_ARG, "GGUF matvec input width does not match the packed rows");
        const at::Tensor xc = whole(x), y = stream.output({tokens, rows}, x);
        enqueue([&] {
            return lisa_cuda_gguf_packed_matvec(stream, code, ptr_of<uint8_t>(w), rows, row_bytes, ptr_of<float>(xc), tokens, out_of<float>(y));
        });
        return wrap(y);
    });
}

// fmt, weights, input, workspace, stream
PyObject *packed_matmul(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 5, [&]() -> PyObject * {
        const at::Tensor &w = tensor(a[1]), &x = tensor(a[2]);
        at::Tensor ws = tensor(a[3], true);
        need_cuda(w);
        need_cuda(x);
        const CallStream stream(a[4]);
        const int code = static_cast<int>(integer(a[0]));
        if (w.dim() != 2 || w.scalar_type() != at::kByte || !w.is_contiguous()) refuse(LISA_ERR_BAD_ARG, "unsupported GGUF quantized matvec layout");
        if (x.dim() != 2 || x.scalar_type() != at::kFloat) refuse(LISA_ERR_BAD_ARG, "invalid GGUF matvec input rows");
        const int64_t rows = w.size(0), row_bytes = w.size(1), tokens = x.size(0);
        const size_t need = lisa_cuda_gguf_packed_matmul_workspace_bytes(tokens, row_bytes, code);
        if (!ws.defined() && need) ws = empty({static_cast<int64_t>(need)}, at::kByte, x);
        const at::Tensor xc = whole(x), y = stream.output({tokens, rows}, x);
        enqueue([&] {
            return lisa_cuda_gguf_packed_matmul(stream, code, ptr_of<uint8_t>(w), rows, row_bytes, ptr_of<float>(xc), tokens, out_of<float>(y),
                                           out_ptr(ws), ws.defined() ? static_cast<size_t>(ws.numel()) : 0);
        });
        return wrap(y);
    });
}

// fmt, weights, input, ids, stream
PyObject *expert_matvec(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 5, [&]() -> PyObject * {
        const at::Tensor &w = tensor(a[1]), &x = tensor(a[2]), &ids = tensor(a[3]);
        need_cuda(w);
        need_cuda(x);
        need_cuda(ids);
        const CallStream stream(a[4]);
        const int code = static_cast<int>(integer(a[0]));
        if (w.dim() != 3 || w.scalar_type() != at::kByte || !w.is_contiguous()) refuse(LISA_ERR_BAD_ARG, "unsupported GGUF quantized matvec layout");
        if (ids.dim() != 2 || ids.scalar_type() != at::kInt || x.dim() != 3 || x.scalar_type() != at::kFloat || x.size(0) != ids.size(0))
            refuse(LISA_ERR_BAD_ARG, "invalid GGUF expert matvec geometry");
        const int64_t tokens = ids.size(0), top_k = ids.size(1), rows = w.size(1);
        const at::Tensor xc = whole(x), ic = whole(ids), y = stream.output({tokens, top_k, rows}, x);
        enqueue([&] {
            return lisa_cuda_gguf_expert_matvec(stream, code, ptr_of<uint8_t>(w), w.size(0), rows, w.size(2), ptr_of<float>(xc), tokens, x.size(1),
                                           ptr_of<int32_t>(ic), top_k, out_of<float>(y));
        });
        return wrap(y);
    });
}

// x, w, scales, biases, lhs_indices, rhs_indices, transpose, group_size, bits, sorted_indices, stream, workspace
PyObject *gather_qmm(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 12, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]), &w0 = tensor(a[1]), &s0 = tensor(a[2]), &b0 = tensor(a[3], true), &lhs = tensor(a[4], true), &rhs = tensor(a[5], true);
        at::Tensor ws = tensor(a[11], true);
        for (const at::Tensor *t : {&x, &w0, &s0, &b0, &rhs}) need_cuda(*t);
        const CallStream stream(a[10]);
        const int64_t k = x.size(-1), rows = rows_of(x, k), experts = w0.size(0), n = w0.size(-2);
        const at::Tensor xc = whole(x), w = words(w0), s = whole(s0), b = whole(b0);
        const at::Tensor y = stream.output(with_last(x, n), x);
        const size_t need = lisa_cuda_gather_qmm_workspace_bytes(rows, experts);
        if (!ws.defined() && need) ws = empty({static_cast<int64_t>(need)}, at::kByte, x);
        const at::Tensor ids = !rhs.defined() ? rhs : whole(rhs.scalar_type() == at::kInt ? rhs : rhs.to(at::kInt));
        const int transpose = truth(a[6]);
        const int sorted = truth(a[9]);
        const int gs = static_cast<int>(integer(a[7]));
        const int bits = static_cast<int>(integer(a[8]));
        enqueue([&] {
            return lisa_cuda_gather_qmm(stream, ptr(xc), rows, k, ptr_of<uint32_t>(w), ptr(s), ptr(b), ptr_of<int32_t>(lhs), ptr_of<int32_t>(ids),
                                   experts, n, transpose, gs, bits, sorted, dtype_code(xc), out_ptr(y), out_ptr(ws), ws.defined() ? static_cast<size_t>(ws.numel()) : 0);
        });
        return wrap(y);
    });
}

// x, linears, rhs_indices, group_size, bits, stream, workspace
PyObject *gather_qmm_siblings(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 7, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]), &rhs = tensor(a[2]);
        at::Tensor ws = tensor(a[6], true);
        need_cuda(x);
        need_cuda(rhs);
        const CallStream stream(a[5]);
        const int64_t k = x.size(-1), rows = rows_of(x, k);
        const at::Tensor xc = whole(x), ids = whole(rhs.scalar_type() == at::kInt ? rhs : rhs.to(at::kInt));
        Linears l;
        l.read(a[1]);
        if (l.count < 1) refuse(LISA_ERR_BAD_ARG, "gather_qmm_siblings: one to three linears");
        const int64_t experts = l.keep[0][0].size(0), n = l.keep[0][0].size(-2);
        for (int i = 0; i < l.count; ++i) {
            if (l.keep[i][0].size(0) != experts || l.keep[i][0].size(-2) != n) refuse(LISA_ERR_BAD_ARG, "gather_qmm_siblings: the linears must have one shape");
            l.y[i] = stream.output(with_last(x, n), x);
            l.out[i] = out_ptr(l.y[i]);
        }
        const size_t need = lisa_cuda_gather_qmm_workspace_bytes(rows, experts);
        if (!ws.defined() && need) ws = empty({static_cast<int64_t>(need)}, at::kByte, x);
        const int gs = static_cast<int>(integer(a[3]));
        const int bits = static_cast<int>(integer(a[4]));
        enqueue([&] {
            return lisa_cuda_gather_qmm_siblings(stream, ptr(xc), rows, k, l.count, l.w, l.s, l.b, ptr_of<int32_t>(ids), experts, n, 1,
                                            gs, bits, 1, dtype_code(xc), l.out, out_ptr(ws),
                                            ws.defined() ? static_cast<size_t>(ws.numel()) : 0);
        });
        return list_of(l.y, l.count);
    });
}

// x, logits, gate (w, s, b), up, down (nine tensors), group_size, bits, top_k, decode_slots
PyObject *moe_block(PyObject *, Args a, Py_ssize_t na) {
    return guarded(na, 15, [&]() -> PyObject * {
        const at::Tensor &x = tensor(a[0]), &lg = tensor(a[1]);
        need_cuda(x);
        need_cuda(lg);
        Linears l;
        for (int i = 0; i < 3; ++i) l.add(a[2 + 3 * i], a[3 + 3 * i], a[4 + 3 * i]);
        const at::Tensor xc = whole(x), logits = whole(lg.scalar_type() == at::kFloat ? lg : lg.to(at::kFloat));
        const int64_t gs = integer(a[11]), bits = integer(a[12]);
        for (int i = 0; i < 3; ++i)
            for (const at::Tensor &t : l.keep[i])
                if (t.dim() != 3) refuse(LISA_ERR_BAD_ARG, "moe_block: weights, scales and biases have three dimensions: experts, rows, columns");
        if (logits.dim() != 2 || x.dim() < 1) refuse(LISA_ERR_BAD_ARG, "moe_block: shapes of x, the logits and the experts disagree");
        const int64_t tokens = logits.size(0), hidden = x.size(-1), experts = l.keep[0][0].size(0), inter = l.keep[0][0].size(1);
        if (logits.size(1) != experts || xc.numel() != tokens * hidden) refuse(LISA_ERR_BAD_ARG, "moe_block: shapes of x, the logits and the experts disagree");
        if (bits < 1 || bits > 32 || gs < 1) refuse(LISA_ERR_UNSUPPORTED, "moe_block: bits must be 2 or 4");
        // the kernels take every size from here: each tensor has to have it
        for (int i = 0; i < 3; ++i) {
            const int64_t n = i < 2 ? inter : hidden, k = i < 2 ? hidden : inter;
            const at::Tensor &w = l.keep[i][0], &sc = l.keep[i][1], &bi = l.keep[i][2];
            if (w.size(0) != experts || w.size(1) != n || w.size(2) * 32 != k * bits || sc.size(0) != experts || sc.size(1) != n || sc.size(2) * gs != k ||
                bi.sizes() != sc.sizes())
                refuse(LISA_ERR_BAD_ARG, i == 0 ? "moe_block: shapes of the gate projection, its scales and biases disagree with x and the logits"
                                       : i == 1 ? "moe_block: shapes of the up projection, its scales and biases disagree with the gate's"
                                                : "moe_block: shapes of the down projection, its scales and biases disagree with the gate's");
            if (sc.element_size() != 2 || bi.element_size() != 2) refuse(LISA_ERR_BAD_ARG, "moe_block: scales and biases must be 16-bit");
        }
        const int top_k = static_cast<int>(integer(a[13]));
        const size_t need = lisa_cuda_moe_block_workspace_bytes(tokens, experts, top_k, hidden, inter);
        const at::Tensor ws = empty({static_cast<int64_t>(need)}, at::kByte, x), out = empty({tokens, hidden}, x);
        const int64_t decode_slots = integer(a[14]);
        const lisa_stream_t stream = c10::cuda::getCurrentCUDAStream().stream();
        enqueue([&] {
            return lisa_cuda_moe_block(stream, ptr(xc), ptr_of<float>(logits), tokens, experts, top_k, hidden, inter, l.w[0], l.s[0], l.b[0],
                                  l.w[1], l.s[1], l.b[1], l.w[2], l.s[2], l.b[2], static_cast<int>(gs), static_cast<int>(bits),
                                  dtype_code(xc), decode_slots, out_ptr(out), out_ptr(ws), need);
        });
        return wrap(out);
    });
}

PyObject *set_error_class(PyObject *, PyObject *cls) {
    Py_INCREF(cls);
    Py_XSETREF(g_error_class, cls);
    Py_RETURN_NONE;
}

#define LISA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(&name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {LISA_METHOD(quantized_matmul), LISA_METHOD(quantized_matmul_siblings), LISA_METHOD(quantized_matmul_addnorm),
                           LISA_METHOD(quantized_matmul_swiglu), LISA_METHOD(dequantize_rows), LISA_METHOD(packed_matvec),
                           LISA_METHOD(packed_matmul), LISA_METHOD(expert_matvec), LISA_METHOD(gather_qmm),
                           LISA_METHOD(gather_qmm_siblings), LISA_METHOD(moe_block), {"set_error_class", &set_error_class, METH_O, nullptr},
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_lisa_torch", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__lisa_torch() { return PyModule_Create(&g_module); }

// The host side of the package's operators: argument checks, output allocation and the call of the C ABI, in C++ for the
// Python functions of the same names.  An operator call through ctypes cost 17-20 us of host time (a dozen boxed
// integers, a stream object, an allocation through the Python bindings), more than most small kernels run; from here it
// costs a few.  The functions of libsfbert_b200.so come in as addresses (bind), so that the package decides which build
// of the library it runs on.
#include <Python.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <cmath>
#include <string>
#include "../../include/sfbert_b200.h"

namespace {

// ---- the library -----------------------------------------------------------------------------------------------------
#define SFB_FUNCTIONS(X)                                                                                                 \
    X(sfb_last_error) X(sfb_bst_sgemm_nt) X(sfb_masked_softmax) X(sfb_bst_sgemm_xn) X(sfb_masked_softmax_grad) X(sfb_linear) \
    X(sfb_linear_nt) X(sfb_linear_residual) X(sfb_embedding) X(sfb_csr_attention) X(sfb_csr_attention_planned) X(sfb_csr_workspace) X(sfb_rowdot) X(sfb_fused_sddmm_softmax_grad)                  \
    X(sfb_fused_sddmm_softmax) X(sfb_fused_attention) X(sfb_fused_attention_slice) X(sfb_bias_residual_layernorm)         \
    X(sfb_bias_gelu) X(sfb_attention_backward)
struct Lib {
#define DECL(f) decltype(&::f) f = nullptr;
    SFB_FUNCTIONS(DECL)
#undef DECL
} L;

PyObject *error_type = nullptr;      // SfbError: one class, however often the package is loaded

struct Raised {};                    // a Python exception is set

[[noreturn]] void raise(PyObject *type, const char *text)
{
    PyErr_SetString(type, text);
    throw Raised();
}
inline void require(bool ok, const char *text)
{
    if (!ok) raise(PyExc_AssertionError, text);
}
inline void check(int rc)
{
    if (rc != 0) raise(error_type, L.sfb_last_error());
}
// While this exists other Python threads run: a launch waits when the stream's queue is full, for as long as the GPU is behind.
struct Unlocked {
    PyThreadState *state = PyEval_SaveThread();
    Unlocked() {}
    Unlocked(const Unlocked &) = delete;
    ~Unlocked() { PyEval_RestoreThread(state); }
};
// One call of the library.  Its arguments are evaluated before other threads are let in.
template <typename... P, typename... A>
inline void call(int (*f)(P...), A... a)
{
    int rc;
    {
        Unlocked others;
        rc = f(a...);
    }
    check(rc);                           // the library's message is the thread's own
}

// ---- Python objects ----------------------------------------------------------------------------------------------------
struct Ref {                         // an owned reference
    PyObject *o;
    explicit Ref(PyObject *p) : o(p) { if (!p) throw Raised(); }
    Ref(const Ref &) = delete;
    ~Ref() { Py_DECREF(o); }
};
enum Name { n_heads, n_nb, n_block_size, n_blocks, n_nn_max, n_nt_lut, n_nn_lut, n_tn_lut, n_tn_max, n_mask_np, n_mask_t,
            n_wo, n_w1, n_w2, n_bo, n_b1, n_b2, n_g1, n_g2, n_be1, n_be2, n_fused_qkv, n_names };
const char *const name_text[n_names] = {"heads", "nb", "block_size", "blocks", "nn_max", "nt_lut", "nn_lut", "tn_lut", "tn_max",
                                        "mask_np", "mask_t", "wo", "w1", "w2", "bo", "b1", "b2", "g1", "g2", "be1", "be2", "fused_qkv"};
PyObject *names[n_names];

inline uint32_t attr_u32(PyObject *o, Name n)
{
    Ref v(PyObject_GetAttr(o, names[n]));
    const long x = PyLong_AsLong(v.o);
    if (x == -1 && PyErr_Occurred()) throw Raised();
    return (uint32_t)x;
}
inline const at::Tensor &tensor(PyObject *o)
{
    if (!THPVariable_Check(o)) raise(PyExc_TypeError, "expected a torch.Tensor");
    return THPVariable_Unpack(o);
}
inline void *ptr(const at::Tensor &t) { return t.const_data_ptr() == nullptr ? nullptr : const_cast<void *>(t.const_data_ptr()); }
inline void *ptr_or_null(PyObject *o) { return o == Py_None ? nullptr : ptr(tensor(o)); }
// the attribute keeps its tensor alive for the call (the object outlives it)
inline void *attr_ptr(PyObject *o, Name n)
{
    Ref v(PyObject_GetAttr(o, names[n]));
    return ptr_or_null(v.o);
}
inline double number(PyObject *o)
{
    const double x = PyFloat_AsDouble(o);
    if (x == -1.0 && PyErr_Occurred()) throw Raised();
    return x;
}
inline bool truth(PyObject *o)
{
    const int x = PyObject_IsTrue(o);
    if (x < 0) throw Raised();
    return x != 0;
}
inline long integer(PyObject *o)
{
    const long x = PyLong_AsLong(o);
    if (x == -1 && PyErr_Occurred()) throw Raised();
    return x;
}
// a size that something is divided by: 0 is Python's ZeroDivisionError, and never reaches the division (which would kill the process)
inline int64_t divisor(int64_t n)
{
    if (n == 0) raise(PyExc_ZeroDivisionError, "division by a size that is 0");
    return n;
}
inline at::ScalarType scalar_type(int tag)
{
    return tag == SFB_F32 ? at::kFloat : tag == SFB_BF16 ? at::kBFloat16 : at::kHalf;
}
inline int tag(const at::Tensor &t)
{
    const at::ScalarType s = t.scalar_type();
    if (s == at::kFloat) return SFB_F32;
    if (s == at::kBFloat16) return SFB_BF16;
    if (s == at::kHalf) return SFB_F16;
    PyErr_SetString(PyExc_KeyError, c10::toString(s));
    throw Raised();
}
inline sfb_stream_t stream() { return (sfb_stream_t)c10::cuda::getCurrentCUDAStream().stream(); }
inline at::Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Tensor &like)
{
    return at::detail::empty_cuda(size, type, like.device(), std::nullopt);
}
inline at::Tensor alike(const at::Tensor &t) { return t.is_contiguous() ? empty(t.sizes(), t.scalar_type(), t) : at::empty_like(t); }
inline at::Tensor out_or(PyObject *out, const at::Tensor &like) { return out == Py_None ? alike(like) : tensor(out); }
inline PyObject *wrap(const at::Tensor &t) { return THPVariable_Wrap(t); }

// ---- layouts -------------------------------------------------------------------------------------------------------------
struct Lay {
    PyObject *o;
    uint32_t heads, nb, bs, blocks, nn_max;
    explicit Lay(PyObject *lay)
        : o(lay), heads(attr_u32(lay, n_heads)), nb(attr_u32(lay, n_nb)), bs(attr_u32(lay, n_block_size)), blocks(attr_u32(lay, n_blocks)),
          nn_max(attr_u32(lay, n_nn_max)) {}
    void *get(Name n) const { return attr_ptr(o, n); }
};
struct Dims {
    uint32_t B, L, H, d;
    Dims(const at::Tensor &q, const Lay &lay)
    {
        require(q.dim() == 4, "expected a [B, L, H, d] tensor");
        B = (uint32_t)q.size(0); L = (uint32_t)q.size(1); H = (uint32_t)q.size(2); d = (uint32_t)q.size(3);
        require(L == lay.nb * lay.bs, "sequence length does not match the layout");
        require(lay.heads == 1 || lay.heads == H, "the layout's heads are neither 1 nor the tensor's");
    }
};

// ---- operators (each also used by the compositions below) -------------------------------------------------------------------
at::Tensor bst_sgemm_nt(const at::Tensor &q, const at::Tensor &k, const Lay &lay, int out_tag)
{
    const Dims n(q, lay);
    at::Tensor s = empty({n.B, n.H, lay.blocks, lay.bs, lay.bs}, scalar_type(out_tag), q);
    call(L.sfb_bst_sgemm_nt, stream(), lay.get(n_nt_lut), ptr(q), ptr(k), ptr(s), tag(q), out_tag, lay.bs, lay.blocks, n.B, lay.nb, lay.nb, n.H,
                             n.d, lay.heads, lay.blocks);
    return s;
}

at::Tensor bst_sgemm(const at::Tensor &p, const at::Tensor &v, const Lay &lay, bool trans)
{
    const Dims n(v, lay);
    at::Tensor o = alike(v);
    call(L.sfb_bst_sgemm_xn, stream(), lay.get(trans ? n_tn_lut : n_nn_lut), ptr(p), ptr(v), ptr(o), tag(p), tag(v), lay.bs, lay.blocks, n.B,
                             lay.nb, lay.nb, n.H, n.d, lay.heads, lay.blocks + lay.nb, trans ? SFB_TN_OP : SFB_NN_OP, 0, 0,
                             trans ? attr_u32(lay.o, n_tn_max) : lay.nn_max);
    return o;
}

at::Tensor masked_softmax(const at::Tensor &s, const Lay &lay, float scale, int out_tag, bool use_mask)
{
    require(s.dim() >= 2, "expected a [B, H, blocks, bs, bs] tensor");
    at::Tensor y = empty(s.sizes(), scalar_type(out_tag), s);
    call(L.sfb_masked_softmax, stream(), lay.get(n_nn_lut), use_mask ? lay.get(n_mask_t) : nullptr, ptr(s), ptr(y), tag(s), out_tag, lay.bs,
                               lay.blocks, (uint32_t)s.size(0), (uint32_t)s.size(1), lay.nb, lay.heads, lay.blocks + lay.nb, lay.nn_max, lay.heads,
                               scale);
    return y;
}

at::Tensor masked_softmax_grad(const at::Tensor &dy, const at::Tensor &y, const Lay &lay, float scale)
{
    require(dy.scalar_type() == y.scalar_type() && dy.sizes() == y.sizes(), "dy and y differ in type or shape");
    at::Tensor dx = alike(y);
    call(L.sfb_masked_softmax_grad, stream(), lay.get(n_nn_lut), ptr(dy), ptr(y), ptr(dx), tag(y), lay.bs, lay.blocks, (uint32_t)y.size(0),
                                    (uint32_t)y.size(1), lay.nb, lay.heads, lay.blocks + lay.nb, lay.nn_max, scale);
    return dx;
}

at::Tensor rowdot(const at::Tensor &a, const at::Tensor &b)
{
    require(a.sizes() == b.sizes() && a.scalar_type() == b.scalar_type() && a.is_contiguous() && b.is_contiguous(),
            "a and b must be contiguous and alike");
    const int64_t d = divisor(a.size(-1));
    at::Tensor out = empty(a.sizes().slice(0, a.dim() - 1), at::kFloat, a);
    call(L.sfb_rowdot, stream(), (float *)ptr(out), ptr(a), ptr(b), (uint64_t)(a.numel() / d), (uint32_t)d, tag(a));
    return out;
}

at::Tensor fused_sddmm_softmax_grad(const at::Tensor &dout, const at::Tensor &v, const at::Tensor &p, const at::Tensor &delta, const Lay &lay,
                                    float scale)
{
    const Dims n(dout, lay);
    require(p.scalar_type() == dout.scalar_type() && dout.scalar_type() == v.scalar_type(), "P, dO and V differ in type");
    require(delta.scalar_type() == at::kFloat && delta.dim() == 3 && delta.size(0) == n.B && delta.size(1) == n.L && delta.size(2) == n.H,
            "delta is not a float [B, L, H] tensor");
    at::Tensor ds = alike(p);
    call(L.sfb_fused_sddmm_softmax_grad, stream(), lay.get(n_nt_lut), ptr(dout), ptr(v), ptr(p), (const float *)ptr(delta), ptr(ds), tag(p), lay.bs,
                                         lay.blocks, n.B, lay.nb, n.H, n.d, lay.heads, lay.blocks, scale);
    return ds;
}

at::Tensor fused_sddmm_softmax(const at::Tensor &q, const at::Tensor &k, const Lay &lay, float scale, int out_tag, bool use_mask)
{
    const Dims n(q, lay);
    at::Tensor y = empty({n.B, n.H, lay.blocks, lay.bs, lay.bs}, scalar_type(out_tag), q);
    call(L.sfb_fused_sddmm_softmax, stream(), lay.get(n_nn_lut), ptr(q), ptr(k), use_mask ? lay.get(n_mask_np) : nullptr, ptr(y), tag(q), out_tag,
                                    lay.bs, lay.blocks, n.B, lay.nb, lay.nb, n.H, n.d, lay.heads, lay.blocks, lay.heads, scale);
    return y;
}

// the two dimensions of a weight: k and n
inline void weight_dims(const at::Tensor &w, bool nt, int64_t &k, int64_t &n)
{
    require(w.dim() == 2, "the weight must have two dimensions");
    k = divisor(w.size(nt ? 1 : 0));
    n = w.size(nt ? 0 : 1);
}
void linear_into(const at::Tensor &x, const at::Tensor &w, const void *bias, int act, bool nt, const at::Tensor &out)
{
    int64_t k, n;
    weight_dims(w, nt, k, n);
    require(x.size(-1) == k && x.scalar_type() == w.scalar_type() && x.is_contiguous() && w.is_contiguous(),
            "x and w must be contiguous, of one type and of matching sizes");
    auto f = nt ? L.sfb_linear_nt : L.sfb_linear;
    call(f, stream(), ptr(out), ptr(x), ptr(w), (const float *)bias, (uint32_t)(x.numel() / k), (uint32_t)n, (uint32_t)k, tag(x), act);
}

at::Tensor linear(const at::Tensor &x, const at::Tensor &w, const void *bias, int act, bool nt)
{
    int64_t k, n;
    weight_dims(w, nt, k, n);
    at::Tensor out;
    if (x.dim() == 2) {
        out = empty({x.size(0), n}, x.scalar_type(), x);
    } else {
        std::vector<int64_t> size(x.sizes().begin(), x.sizes().end());
        size.back() = n;
        out = empty(size, x.scalar_type(), x);
    }
    linear_into(x, w, bias, act, nt, out);
    return out;
}

// ---- the Python functions ------------------------------------------------------------------------------------------------------
#define FUNCTION(name, count)                                                      \
    PyObject *name##_body(PyObject *const *a);                                     \
    PyObject *name##_call(PyObject *, PyObject *const *args, Py_ssize_t given)     \
    {                                                                              \
        HANDLE_TH_ERRORS                                                           \
        try {                                                                      \
            if (given != count) raise(PyExc_TypeError, #name ": expected " #count " arguments"); \
            return name##_body(args);                                              \
        } catch (const Raised &) {                                                 \
            return nullptr;                                                        \
        }                                                                          \
        END_HANDLE_TH_ERRORS                                                       \
    }                                                                              \
    PyObject *name##_body(PyObject *const *a)

// (q, k, lay, out_tag)
FUNCTION(py_bst_sgemm_nt, 4) { return wrap(bst_sgemm_nt(tensor(a[0]), tensor(a[1]), Lay(a[2]), (int)integer(a[3]))); }
// (s, lay, scale, out_tag, use_mask)
FUNCTION(py_masked_softmax, 5)
{
    return wrap(masked_softmax(tensor(a[0]), Lay(a[1]), (float)number(a[2]), (int)integer(a[3]), truth(a[4])));
}
// (p, v, lay, trans)
FUNCTION(py_bst_sgemm, 4) { return wrap(bst_sgemm(tensor(a[0]), tensor(a[1]), Lay(a[2]), truth(a[3]))); }
// (dy, y, lay, scale)
FUNCTION(py_masked_softmax_grad, 4) { return wrap(masked_softmax_grad(tensor(a[0]), tensor(a[1]), Lay(a[2]), (float)number(a[3]))); }
FUNCTION(py_rowdot, 2) { return wrap(rowdot(tensor(a[0]), tensor(a[1]))); }
// (do, v, p, delta, lay, scale)
FUNCTION(py_fused_sddmm_softmax_grad, 6)
{
    return wrap(fused_sddmm_softmax_grad(tensor(a[0]), tensor(a[1]), tensor(a[2]), tensor(a[3]), Lay(a[4]), (float)number(a[5])));
}
// (q, k, lay, scale, out_tag, use_mask)
FUNCTION(py_fused_sddmm_softmax, 6)
{
    return wrap(fused_sddmm_softmax(tensor(a[0]), tensor(a[1]), Lay(a[2]), (float)number(a[3]), (int)integer(a[4]), truth(a[5])));
}
// (x, w, bias, act, out, nt)
FUNCTION(py_linear, 6)
{
    const at::Tensor &x = tensor(a[0]), &w = tensor(a[1]);
    const void *bias = ptr_or_null(a[2]);
    const int act = (int)integer(a[3]);
    const bool nt = truth(a[5]);
    if (a[4] == Py_None) return wrap(linear(x, w, bias, act, nt));
    linear_into(x, w, bias, act, nt, tensor(a[4]));
    Py_INCREF(a[4]);
    return a[4];
}
// (table, ids, pos)
FUNCTION(py_embedding, 3)
{
    const at::Tensor &table = tensor(a[0]), &ids = tensor(a[1]);
    require(ids.dim() == 2 && table.dim() == 2, "ids must be [B, L] and the table [vocab, hidden]");
    require(ids.scalar_type() == at::kInt && ids.is_contiguous() && table.is_contiguous(), "ids must be int32 and contiguous, like the table");
    const int64_t B = ids.size(0), len = ids.size(1), vocab = table.size(0), hidden = table.size(1);
    at::Tensor out = empty({B, len, hidden}, table.scalar_type(), table), bad = empty({1}, at::kInt, table);
    call(L.sfb_embedding, stream(), ptr(out), ptr(table), (const int32_t *)ptr(ids), ptr_or_null(a[2]), (uint32_t)B, (uint32_t)len,
                          (uint32_t)hidden, (uint32_t)vocab, tag(table), (uint32_t *)ptr(bad));
    Ref o(wrap(out)), n(wrap(bad));
    return PyTuple_Pack(2, o.o, n.o);
}
// (q, k, v, rowptr, colidx, scale)
FUNCTION(py_csr_attention, 6)
{
    const at::Tensor &q = tensor(a[0]), &rowptr = tensor(a[3]), &colidx = tensor(a[4]);
    require(q.dim() == 4, "expected a [B, L, H, d] tensor");
    require(rowptr.scalar_type() == at::kInt && colidx.scalar_type() == at::kInt && rowptr.numel() == q.size(1) + 1,
            "rowptr and colidx must be int32, rowptr of L + 1 elements");
    at::Tensor o = alike(q), bad = empty({1}, at::kInt, q);
    const int64_t nnz = colidx.numel();
    const uint64_t bytes = nnz < (1ll << 31) ? L.sfb_csr_workspace((uint32_t)nnz, (uint32_t)q.size(1)) : 0;
    if (bytes) {
        at::Tensor ws = empty({(int64_t)bytes}, at::kByte, q);
        call(L.sfb_csr_attention_planned, stream(), (const int32_t *)ptr(rowptr), (const int32_t *)ptr(colidx), (uint32_t)nnz, ptr(q),
                                          ptr(tensor(a[1])), ptr(tensor(a[2])), ptr(o), tag(q), (uint32_t)q.size(0), (uint32_t)q.size(1),
                                          (uint32_t)q.size(2), (uint32_t)q.size(3), (float)number(a[5]), (uint32_t *)ptr(bad), ptr(ws));
        Ref r(wrap(o)), n(wrap(bad));
        return PyTuple_Pack(2, r.o, n.o);
    }
    call(L.sfb_csr_attention, stream(), (const int32_t *)ptr(rowptr), (const int32_t *)ptr(colidx), ptr(q), ptr(tensor(a[1])), ptr(tensor(a[2])),
                              ptr(o), tag(q), (uint32_t)q.size(0), (uint32_t)q.size(1), (uint32_t)q.size(2), (uint32_t)q.size(3),
                              (float)number(a[5]), (uint32_t *)ptr(bad));
    Ref r(wrap(o)), n(wrap(bad));
    return PyTuple_Pack(2, r.o, n.o);
}
inline float scale_or(PyObject *o, uint32_t d) { return o == Py_None ? (float)(1.0 / std::sqrt((double)divisor(d))) : (float)number(o); }
// (q, k, v, lay, scale, use_mask, out)
FUNCTION(py_fused_attention, 7)
{
    const at::Tensor &q = tensor(a[0]);
    const Lay lay(a[3]);
    const Dims n(q, lay);
    at::Tensor o = out_or(a[6], q);
    call(L.sfb_fused_attention, stream(), lay.get(n_nn_lut), ptr(q), ptr(tensor(a[1])), ptr(tensor(a[2])), ptr(o),
                                truth(a[5]) ? lay.get(n_mask_np) : nullptr, tag(q), lay.bs, lay.blocks, n.B, lay.nb, n.H, n.d, lay.heads, lay.blocks,
                                lay.heads, scale_or(a[4], n.d), lay.nn_max);
    return wrap(o);
}
// Row pitch (elements) of a [B, L, H, d] view whose heads are a slice of a wider tensor: rows of one batch element and
// batch elements themselves must follow each other at that pitch.
uint64_t row_pitch(const at::Tensor &t)
{
    require(t.dim() == 4, "expected a [B, L, H, d] tensor");
    const int64_t B = t.size(0), len = t.size(1), H = t.size(2), d = t.size(3), sl = t.stride(1);
    require(t.stride(3) == 1 && t.stride(2) == d && sl >= H * d && (B == 1 || t.stride(0) == len * sl),
            "not a head slice of a [B, L, H_total, d] tensor");
    return (uint64_t)sl;
}
FUNCTION(py_fused_attention_slice, 7)
{
    const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]);
    const Lay lay(a[3]);
    const Dims n(q, lay);
    at::Tensor o = a[6] == Py_None ? empty(q.sizes(), q.scalar_type(), q) : tensor(a[6]);
    const uint64_t pitch = row_pitch(q);
    require(row_pitch(k) == pitch && row_pitch(v) == pitch, "q, k and v have different row pitches");
    call(L.sfb_fused_attention_slice, stream(), lay.get(n_nn_lut), ptr(q), ptr(k), ptr(v), ptr(o), truth(a[5]) ? lay.get(n_mask_np) : nullptr,
                                      tag(q), lay.bs, lay.blocks, n.B, lay.nb, n.H, n.d, lay.heads, lay.blocks, lay.heads, scale_or(a[4], n.d),
                                      lay.nn_max, pitch, row_pitch(o));
    return wrap(o);
}
// (x, bias, resid, gain, beta, want_sum, out)
FUNCTION(py_bias_residual_layernorm, 7)
{
    const at::Tensor &x = tensor(a[0]);
    require(x.dim() == 2, "expected an [m, hidden] tensor");
    const int64_t m = x.size(0), hidden = x.size(1);
    at::Tensor out = out_or(a[6], x), sum, mean = empty({m}, at::kFloat, x), rstd = empty({m}, at::kFloat, x);
    if (truth(a[5])) sum = alike(x);
    call(L.sfb_bias_residual_layernorm, stream(), ptr(out), sum.defined() ? ptr(sum) : nullptr, (float *)ptr(mean), (float *)ptr(rstd), ptr(x),
                                        (const float *)ptr_or_null(a[1]), ptr_or_null(a[2]), (const float *)ptr(tensor(a[3])),
                                        (const float *)ptr(tensor(a[4])), (uint32_t)m, (uint32_t)hidden, tag(x));
    Ref o(wrap(out)), mu(wrap(mean)), rs(wrap(rstd));
    if (!sum.defined()) return PyTuple_Pack(4, o.o, Py_None, mu.o, rs.o);
    Ref s(wrap(sum));
    return PyTuple_Pack(4, o.o, s.o, mu.o, rs.o);
}
// (x, bias, out)
FUNCTION(py_bias_gelu, 3)
{
    const at::Tensor &x = tensor(a[0]);
    require(x.dim() == 2, "expected an [m, n] tensor");
    at::Tensor out = out_or(a[2], x);
    call(L.sfb_bias_gelu, stream(), ptr(out), ptr(x), (const float *)ptr_or_null(a[1]), (uint32_t)x.size(0), (uint32_t)x.size(1), tag(x));
    return wrap(out);
}

// One encoder layer on x [m, hidden], every projection on the library's kernels (the package's encoder.py states the order
// of operations): (x, w, lay, heads, pre, scale).  The activations between the first and the last operation live in one
// workspace in which what is no longer needed is written over -- the FFN's activations take the place of Q, K, V and the
// attention's output, both branch outputs share a slot -- so that a layer touches less memory than L2 holds more often.
FUNCTION(py_encoder_layer, 6)
{
    const at::Tensor &x = tensor(a[0]);
    PyObject *w = a[1];
    const Lay lay(a[2]);
    require(x.dim() == 2, "expected an [m, hidden] tensor");
    const int64_t heads = divisor(integer(a[3])), m = x.size(0), hidden = x.size(1), d = hidden / heads, len = divisor((int64_t)lay.nb * lay.bs);
    const bool pre = truth(a[4]);
    const float scale = (float)number(a[5]);
    require(x.is_contiguous() && heads > 0 && hidden % heads == 0 && m % len == 0, "x must be contiguous, whole sequences of whole heads");
    const int64_t B = m / len;
    require(lay.heads == 1 || lay.heads == heads, "the layout's heads are neither 1 nor the tensor's");
    Ref qkv(PyObject_CallMethodNoArgs(w, names[n_fused_qkv]));
    if (!PyTuple_Check(qkv.o) || PyTuple_GET_SIZE(qkv.o) != 2) raise(PyExc_TypeError, "fused_qkv() returns a pair");
    Ref o_wo(PyObject_GetAttr(w, names[n_wo])), o_w1(PyObject_GetAttr(w, names[n_w1])), o_w2(PyObject_GetAttr(w, names[n_w2]));
    const at::Tensor &wqkv = tensor(PyTuple_GET_ITEM(qkv.o, 0)), &wo = tensor(o_wo.o), &w1 = tensor(o_w1.o), &w2 = tensor(o_w2.o);
    const void *bqkv = ptr(tensor(PyTuple_GET_ITEM(qkv.o, 1)));
    const float *bo = (const float *)attr_ptr(w, n_bo), *b1 = (const float *)attr_ptr(w, n_b1), *b2 = (const float *)attr_ptr(w, n_b2),
                *g1 = (const float *)attr_ptr(w, n_g1), *be1 = (const float *)attr_ptr(w, n_be1), *g2 = (const float *)attr_ptr(w, n_g2),
                *be2 = (const float *)attr_ptr(w, n_be2);
    require(wqkv.dim() == 2 && wo.dim() == 2 && w1.dim() == 2 && w2.dim() == 2, "a weight of the layer does not have two dimensions");
    const int64_t ffn = w1.size(1);
    require(wqkv.size(0) == hidden && wqkv.size(1) == 3 * hidden && wo.size(0) == hidden && wo.size(1) == hidden && w1.size(0) == hidden &&
                w2.size(0) == ffn && w2.size(1) == hidden && wqkv.is_contiguous() && wo.is_contiguous() && w1.is_contiguous() && w2.is_contiguous(),
            "a weight does not fit the layer");
    const int t = tag(x);
    require(tag(wqkv) == t && tag(wo) == t && tag(w1) == t && tag(w2) == t, "x and the weights differ in type");
    const int64_t wide = std::max(4 * hidden, ffn);
    at::Tensor ws = empty({m * (wide + 2 * hidden)}, x.scalar_type(), x), out = empty({m, hidden}, x.scalar_type(), x);
    char *base = (char *)ptr(ws);
    const int64_t row = m * x.element_size();
    char *p_qkv = base, *p_attn = base + row * 3 * hidden, *p_ffn = base, *p_a = base + row * wide, *p_b = p_a + row * hidden;
    const sfb_stream_t s = stream();
    const uint32_t um = (uint32_t)m, uh = (uint32_t)hidden, uf = (uint32_t)ffn;
    const void *lut = lay.get(n_nn_lut), *px = ptr(x), *pwqkv = ptr(wqkv), *pwo = ptr(wo), *pw1 = ptr(w1), *pw2 = ptr(w2);
    void *pout = ptr(out);
    int rc = 0;
    auto done = [&](int r) { return (rc = r) == 0; };
    auto attention = [&](const void *h) {
        // Q, K and V are column slices of the [m, 3 * hidden] result
        const int64_t col = hidden * x.element_size();
        return done(L.sfb_linear(s, p_qkv, h, pwqkv, (const float *)bqkv, um, 3 * uh, uh, t, SFB_ACT_NONE)) &&
               done(L.sfb_fused_attention_slice(s, lut, p_qkv, p_qkv + col, p_qkv + 2 * col, p_attn, nullptr, t, lay.bs, lay.blocks, (uint32_t)B,
                                                lay.nb, (uint32_t)heads, (uint32_t)d, lay.heads, lay.blocks, lay.heads, scale, lay.nn_max, 3 * hidden,
                                                hidden));
    };
    {
        Unlocked others;                     // once for all launches of the layer
        if (pre) {
            // h = LN(x); a = Attn(h) Wo; h2, x1 = LN(x + a + bo) and the sum; out = x1 + GELU(h2 W1 + b1) W2 + b2
            (void)(done(L.sfb_bias_residual_layernorm(s, p_b, nullptr, nullptr, nullptr, px, nullptr, nullptr, g1, be1, um, uh, t)) &&
                   attention(p_b) &&
                   done(L.sfb_linear(s, p_a, p_attn, pwo, nullptr, um, uh, uh, t, SFB_ACT_NONE)) &&
                   done(L.sfb_bias_residual_layernorm(s, p_b, p_a, nullptr, nullptr, p_a, bo, px, g2, be2, um, uh, t)) &&
                   done(L.sfb_linear(s, p_ffn, p_b, pw1, b1, um, uf, uh, t, SFB_ACT_GELU)) &&
                   done(L.sfb_linear_residual(s, pout, p_ffn, pw2, b2, p_a, um, uh, uf, t)));
        } else {
            // x1 = LN(x + Attn(x) Wo + bo); out = LN(x1 + GELU(x1 W1 + b1) W2 + b2)
            (void)(attention(px) &&
                   done(L.sfb_linear(s, p_a, p_attn, pwo, nullptr, um, uh, uh, t, SFB_ACT_NONE)) &&
                   done(L.sfb_bias_residual_layernorm(s, p_b, nullptr, nullptr, nullptr, p_a, bo, px, g1, be1, um, uh, t)) &&
                   done(L.sfb_linear(s, p_ffn, p_b, pw1, b1, um, uf, uh, t, SFB_ACT_GELU)) &&
                   done(L.sfb_linear(s, p_a, p_ffn, pw2, nullptr, um, uh, uf, t, SFB_ACT_NONE)) &&
                   done(L.sfb_bias_residual_layernorm(s, pout, nullptr, nullptr, nullptr, p_a, b2, p_b, g2, be2, um, uh, t)));
        }
    }
    check(rc);
    return wrap(out);
}

// (do, q, k, v, p, o, lay, scale) -> (dq, dk, dv), the softmax gradient fused with dP
FUNCTION(py_attention_backward_fused, 8)
{
    const at::Tensor &dout = tensor(a[0]), &q = tensor(a[1]), &k = tensor(a[2]), &v = tensor(a[3]), &p = tensor(a[4]), &o = tensor(a[5]);
    const Lay lay(a[6]);
    const float scale = (float)number(a[7]);
    const Dims n(q, lay);
    const int t = tag(q);
    void *tn = lay.get(n_tn_lut);
    const uint32_t tn_max = attr_u32(lay.o, n_tn_max);
    // dS on chip where the library has the kernels for it, otherwise operator by operator
    auto tidy = [](const at::Tensor &x) { return x.is_contiguous() && ((uintptr_t)ptr(x) & 31) == 0; };
    if (t != SFB_F32 && lay.bs == 64 && n.d == 64 && lay.blocks && lay.nn_max && tn_max && (lay.nb <= 256 || (lay.nn_max <= 128 && tn_max <= 128)) && tag(k) == t &&
        tag(v) == t && tag(p) == t && tag(o) == t && tag(dout) == t && tidy(q) && tidy(k) && tidy(v) && tidy(p) && tidy(o) && tidy(dout) &&
        (int64_t)n.B * n.H * lay.blocks * 64 < (1ll << 31) - 64 && (int64_t)n.B * n.L < (1ll << 31)) {
        require(o.sizes() == dout.sizes() && dout.sizes() == q.sizes(), "q, o and dO differ in shape");
        at::Tensor delta = empty({n.B, n.H, n.L}, at::kFloat, q), dq = alike(q), dk = alike(k), dv = alike(v);
        call(L.sfb_attention_backward, stream(), lay.get(n_nn_lut), tn, ptr(q), ptr(k), ptr(v), ptr(p), ptr(o), ptr(dout), (float *)ptr(delta), ptr(dq),
                                       ptr(dk), ptr(dv), t, lay.bs, lay.blocks, n.B, lay.nb, n.H, n.d, lay.heads, lay.blocks + lay.nb, lay.nn_max,
                                       tn_max, scale);
        Ref x(wrap(dq)), y(wrap(dk)), z(wrap(dv));
        return PyTuple_Pack(3, x.o, y.o, z.o);
    }
    at::Tensor dv = bst_sgemm(p, dout, lay, true);
    at::Tensor ds = fused_sddmm_softmax_grad(dout, v, p, rowdot(dout, o), lay, scale);
    at::Tensor dk = bst_sgemm(ds, q, lay, true), dq = bst_sgemm(ds, k, lay, false);
    Ref x(wrap(dq)), y(wrap(dk)), z(wrap(dv));
    return PyTuple_Pack(3, x.o, y.o, z.o);
}
// (do, q, k, v, p, lay, scale, s_tag) -> (dq, dk, dv), the five operators one after another
FUNCTION(py_attention_backward, 8)
{
    const at::Tensor &dout = tensor(a[0]), &q = tensor(a[1]), &k = tensor(a[2]), &v = tensor(a[3]), &p = tensor(a[4]);
    const Lay lay(a[5]);
    const float scale = (float)number(a[6]);
    const int st = (int)integer(a[7]);
    at::Tensor dv = bst_sgemm(p, dout, lay, true);
    at::Tensor dp = bst_sgemm_nt(dout, v, lay, st);
    at::Tensor ds = masked_softmax_grad(dp, tag(p) == st ? p : p.to(scalar_type(st)), lay, scale);
    at::Tensor dk = bst_sgemm(ds, q, lay, true), dq = bst_sgemm(ds, k, lay, false);
    Ref x(wrap(dq)), y(wrap(dk)), z(wrap(dv));
    return PyTuple_Pack(3, x.o, y.o, z.o);
}

// bind(addresses by name): which build of the library the functions call
PyObject *py_bind(PyObject *, PyObject *args)
{
    PyObject *table;
    if (!PyArg_ParseTuple(args, "O!", &PyDict_Type, &table)) return nullptr;
#define GET(f)                                                                             \
    {                                                                                      \
        PyObject *v = PyDict_GetItemString(table, #f);                                     \
        if (!v) { PyErr_SetString(PyExc_KeyError, #f); return nullptr; }                   \
        L.f = (decltype(L.f))PyLong_AsVoidPtr(v);                                          \
        if (!L.f && PyErr_Occurred()) return nullptr;                                      \
    }
    SFB_FUNCTIONS(GET)
#undef GET
    Py_RETURN_NONE;
}
// the functions bind() takes
PyObject *py_wanted(PyObject *, PyObject *)
{
#define TEXT(f) #f " "
    return PyUnicode_FromString(SFB_FUNCTIONS(TEXT));
#undef TEXT
}

#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))py_##name##_call, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_VARARGS, nullptr}, {"wanted", py_wanted, METH_NOARGS, nullptr},
    ENTRY(bst_sgemm_nt), ENTRY(masked_softmax), ENTRY(bst_sgemm), ENTRY(masked_softmax_grad), ENTRY(rowdot), ENTRY(fused_sddmm_softmax_grad),
    ENTRY(fused_sddmm_softmax), ENTRY(linear), ENTRY(embedding), ENTRY(csr_attention), ENTRY(fused_attention), ENTRY(fused_attention_slice),
    ENTRY(bias_residual_layernorm), ENTRY(bias_gelu), ENTRY(encoder_layer), ENTRY(attention_backward_fused), ENTRY(attention_backward),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void)
{
    for (int i = 0; i < n_names; i++)
        if (!names[i] && !(names[i] = PyUnicode_InternFromString(name_text[i]))) return nullptr;
    if (!error_type && !(error_type = PyErr_NewException("sfbert_b200.SfbError", PyExc_RuntimeError, nullptr))) return nullptr;
    PyObject *m = PyModule_Create(&module);
    if (m && PyModule_AddObjectRef(m, "SfbError", error_type) < 0) Py_CLEAR(m);
    return m;
}

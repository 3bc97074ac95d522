// Native call path of the Python operators: reads the tensors' pointers, sizes and strides, allocates the outputs and
// enqueues the library's entry points (include/mamba_b200.h) without going through ctypes.
//
// A decode step is three calls whose kernels take 3-13 us each; building the argument structs field by field in Python
// cost 25-45 us per call, so small calls were bound by the host.  Here a call costs 3-6 us.
//
// Every function takes exactly the arguments of its operator and returns None when the call is not one it can pass on as
// it is -- a wrong shape or dtype, a tensor that needs converting or copying first, a CPU tensor, an input that requires
// a gradient, an error code of the library.  The Python operator then runs its own checks, which convert or raise.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/mamba_b200.h"

namespace {

using at::Tensor;

// An argument that is a tensor or None.  `bad` collects everything that sends the call to Python.
struct Arg {
    const Tensor *t = nullptr;
    bool has() const { return t != nullptr; }
    const Tensor &operator*() const { return *t; }
    const Tensor *operator->() const { return t; }
    void *ptr() const { return t ? t->data_ptr() : nullptr; }
};

Arg take(PyObject *o, bool &bad, bool optional = false)
{
    Arg a;
    if (o == Py_None) {
        if (!optional) bad = true;
        return a;
    }
    if (!THPVariable_Check(o)) {
        bad = true;
        return a;
    }
    a.t = &THPVariable_Unpack(o);
    if (!a.t->is_cuda()) bad = true;
    return a;
}

int code(at::ScalarType t)
{
    switch (t) {
    case at::kFloat: return MB200_F32;
    case at::kHalf: return MB200_F16;
    case at::kBFloat16: return MB200_BF16;
    default: return -1;
    }
}

bool shape(const Tensor &t, std::initializer_list<int64_t> s) { return t.sizes() == at::IntArrayRef(s); }
void strides(int64_t *dst, const Tensor &t, int n)
{
    for (int i = 0; i < n; ++i) dst[i] = t.stride(i);
}
// fp32, one-dimensional of n elements, contiguous
bool is_vec(const Arg &a, int64_t n) { return !a.has() || (a->scalar_type() == at::kFloat && a->dim() == 1 && a->size(0) == n && a->is_contiguous()); }
bool small(const Tensor &t)
{
    for (int64_t s : t.sizes())
        if (s > INT32_MAX) return false;
    return true;
}
bool wants_grad(std::initializer_list<Arg> args)
{
    if (!c10::GradMode::is_enabled()) return false;
    for (const Arg &a : args)
        if (a.has() && a->requires_grad()) return true;
    return false;
}
bool one_device(const Tensor &ref, std::initializer_list<Arg> args)
{
    for (const Arg &a : args)
        if (a.has() && a->device() != ref.device()) return false;
    return true;
}

Tensor empty(at::IntArrayRef size, at::ScalarType dtype, c10::Device dev)
{
    return at::detail::empty_cuda(size, dtype, dev, std::nullopt);
}
// empty_like without the dispatcher: keeps the strides of a dense tensor in any dimension order
Tensor empty_as(const Tensor &t)
{
    if (t.is_contiguous()) return empty(t.sizes(), t.scalar_type(), t.device());
    if (t.is_non_overlapping_and_dense()) return at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device());
    return at::empty_like(t);
}
Tensor bytes(size_t n, c10::Device dev) { return empty({(int64_t)n}, at::kByte, dev); }

void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

PyObject *wrap(const Tensor &t) { return THPVariable_Wrap(t); }

#define DECLINE() Py_RETURN_NONE
#define GUARD_BEGIN try {
#define GUARD_END                                                     \
    }                                                                 \
    catch (const std::exception &e)                                   \
    {                                                                 \
        PyErr_SetString(PyExc_RuntimeError, e.what());                \
        return nullptr;                                               \
    }

// ---------------------------------------------------------------------------------------------------- Mamba-1
// Fills what forward and backward have in common; false sends the call to Python.
template <class ARGS>
bool scan_common(ARGS &a, const Arg &u, const Arg &delta, const Arg &A, const Arg &B, const Arg &C, const Arg &D, const Arg &z, const Arg &bias,
                 bool softplus)
{
    if (u->dim() != 3 || delta->sizes() != u->sizes() || delta->scalar_type() != u->scalar_type() || !small(*u)) return false;
    const int64_t batch = u->size(0), dim = u->size(1), L = u->size(2);
    if (code(u->scalar_type()) < 0 || u->stride(2) != 1 || delta->stride(2) != 1) return false;
    if (A->scalar_type() != at::kFloat || A->dim() != 2 || A->size(0) != dim) return false;
    const int64_t N = A->size(1);
    if (!is_vec(D, dim) || !is_vec(bias, dim)) return false;
    if (z.has() && (z->sizes() != u->sizes() || z->scalar_type() != u->scalar_type() || z->stride(2) != 1)) return false;
    if (!one_device(*u, {delta, A, B, C, D, z, bias})) return false;
    const bool bv = B->dim() >= 3, cv = C->dim() >= 3;
    const int64_t G = bv ? (B->dim() == 4 ? B->size(1) : 1) : (cv ? (C->dim() == 4 ? C->size(1) : 1) : 1);
    auto bc = [&](const Arg &t, bool var, int64_t *st) {
        if (!var) {
            if (t->dim() != 2 || t->scalar_type() != at::kFloat || !shape(*t, {dim, N}) || t->stride(1) != 1) return false;
            strides(st, *t, 2);
            return true;
        }
        if (t->scalar_type() != u->scalar_type() || t->stride(-1) != 1) return false;
        if (t->dim() == 3) {
            if (G != 1 || !shape(*t, {batch, N, L})) return false;
            st[0] = t->stride(0); st[1] = t->stride(0); st[2] = t->stride(1);
            // the group stride of a single group is never used; it has to look like an ordinary row stride
            st[1] = t->stride(1) * N;
            return true;
        }
        if (t->dim() != 4 || !shape(*t, {batch, G, N, L})) return false;
        strides(st, *t, 3);
        return true;
    };
    if (!bc(B, bv, a.B_stride) || !bc(C, cv, a.C_stride)) return false;
    a.u = u.ptr(); a.delta = delta.ptr(); a.A = static_cast<const float *>(A.ptr());
    a.B = B.ptr(); a.C = C.ptr(); a.D = static_cast<const float *>(D.ptr()); a.z = z.ptr(); a.delta_bias = static_cast<const float *>(bias.ptr());
    a.batch = (int)batch; a.dim = (int)dim; a.seqlen = (int)L; a.dstate = (int)N; a.ngroups = (int)G;
    a.io_dtype = code(u->scalar_type());
    a.B_variable = bv; a.C_variable = cv; a.delta_softplus = softplus;
    a.device = u->device().index();
    strides(a.u_stride, *u, 2);
    strides(a.delta_stride, *delta, 2);
    if (z.has()) strides(a.z_stride, *z, 2);
    strides(a.A_stride, *A, 2);
    return true;
}

// (u, delta, A, B, C, D, z, delta_bias, delta_softplus, return_last_state) -> out | (out, last_state) | None
PyObject *scan_fwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 10;
    if (bad) DECLINE();
    const Arg u = take(v[0], bad), delta = take(v[1], bad), A = take(v[2], bad), B = take(v[3], bad), C = take(v[4], bad), D = take(v[5], bad, true),
              z = take(v[6], bad, true), bias = take(v[7], bad, true);
    if (bad || wants_grad({u, delta, A, B, C, D, z, bias})) DECLINE();
    mb200_scan_args a = {};
    if (!scan_common(a, u, delta, A, B, C, D, z, bias, PyObject_IsTrue(v[8]) == 1)) DECLINE();
    const bool want_last = PyObject_IsTrue(v[9]) == 1;
    const Tensor out = empty_as(*delta);
    if (out.stride(2) != 1) DECLINE();
    Tensor last, scratch;
    if (want_last) last = empty({a.batch, a.dim, a.dstate}, at::kFloat, u->device());
    a.out = out.data_ptr();
    a.last_state = want_last ? static_cast<float *>(last.data_ptr()) : nullptr;
    strides(a.out_stride, out, 2);
    size_t need = 0;
    if (mb200_scan_scratch_bytes(&a, &need) != MB200_OK) DECLINE();
    if (need) {
        scratch = bytes(need, u->device());
        a.scratch = scratch.data_ptr();
        a.scratch_bytes = need;
    }
    if (mb200_selective_scan_fwd(&a, stream_of(*u)) != MB200_OK) DECLINE();
    if (!want_last) return wrap(out);
    return Py_BuildValue("(NN)", wrap(out), wrap(last));
    GUARD_END
}

// (u, delta, A, B, C, D, z, delta_bias, dout, delta_softplus) -> (du, ddelta, dA, dB, dC, dD, dz, ddelta_bias) | None
PyObject *scan_bwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 10;
    if (bad) DECLINE();
    const Arg u = take(v[0], bad), delta = take(v[1], bad), A = take(v[2], bad), B = take(v[3], bad), C = take(v[4], bad), D = take(v[5], bad, true),
              z = take(v[6], bad, true), bias = take(v[7], bad, true), dout = take(v[8], bad);
    if (bad) DECLINE();
    mb200_scan_bwd_args a = {};
    if (!scan_common(a, u, delta, A, B, C, D, z, bias, PyObject_IsTrue(v[9]) == 1)) DECLINE();
    if (dout->sizes() != u->sizes() || dout->scalar_type() != u->scalar_type() || dout->stride(2) != 1 || dout->device() != u->device()) DECLINE();
    const c10::Device dev = u->device();
    const Tensor du = empty_as(*u), dd = empty_as(*delta);
    Tensor dz;
    if (z.has()) dz = empty_as(*z);
    if (du.stride(2) != 1 || dd.stride(2) != 1 || (z.has() && dz.stride(2) != 1)) DECLINE();
    // the fp32 accumulators each in a storage of its own: autograd keeps what it is given as .grad
    const Tensor dA = empty(A->sizes(), at::kFloat, dev);
    const Tensor dB = empty(B->sizes(), at::kFloat, dev), dC = empty(C->sizes(), at::kFloat, dev);
    Tensor dD, db;
    if (D.has()) dD = empty(D->sizes(), at::kFloat, dev);
    if (bias.has()) db = empty(bias->sizes(), at::kFloat, dev);
    auto floats = [](const Tensor &t) { return static_cast<float *>(t.data_ptr()); };
    a.dout = dout.ptr(); a.du = du.data_ptr(); a.ddelta = dd.data_ptr(); a.dz = z.has() ? dz.data_ptr() : nullptr;
    a.dA = floats(dA); a.dB = floats(dB); a.dC = floats(dC);
    a.dD = D.has() ? floats(dD) : nullptr;
    a.ddelta_bias = bias.has() ? floats(db) : nullptr;
    strides(a.dout_stride, *dout, 2);
    strides(a.du_stride, du, 2);
    strides(a.ddelta_stride, dd, 2);
    if (z.has()) strides(a.dz_stride, dz, 2);
    size_t need = 0;
    if (mb200_scan_bwd_scratch_bytes(&a, &need) != MB200_OK) DECLINE();
    const Tensor scratch = bytes(std::max<size_t>(need, 16), dev);
    a.scratch = scratch.data_ptr();
    a.scratch_bytes = need;
    if (mb200_selective_scan_bwd(&a, stream_of(*u)) != MB200_OK) DECLINE();
    auto opt = [](bool on, const Tensor &t) -> PyObject * {
        if (on) return wrap(t);
        Py_RETURN_NONE;
    };
    return Py_BuildValue("(NNNNNNNN)", wrap(du), wrap(dd), wrap(dA), wrap(dB.to(B->scalar_type())), wrap(dC.to(C->scalar_type())), opt(D.has(), dD),
                         opt(z.has(), dz), opt(bias.has(), db));
    GUARD_END
}

// ---------------------------------------------------------------------------------------------------- decode
// (state, x, dt, A, B, C, D, z, dt_bias, dt_softplus, state_batch_indices) -> out | None
PyObject *state_update(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 11;
    if (bad) DECLINE();
    const Arg state = take(v[0], bad), x = take(v[1], bad), dt = take(v[2], bad), A = take(v[3], bad), B = take(v[4], bad), C = take(v[5], bad),
              D = take(v[6], bad, true), z = take(v[7], bad, true), bias = take(v[8], bad, true), idx = take(v[10], bad, true);
    if (bad || !one_device(*x, {state, dt, A, B, C, D, z, bias, idx})) DECLINE();
    const bool heads = state->dim() == 4;
    if (!heads && state->dim() != 3) DECLINE();
    const int64_t H = heads ? state->size(1) : 1, P = state->size(-2), N = state->size(-1), batch = x->size(0);
    if (!small(*state) || batch > INT32_MAX) DECLINE();
    mb200_ssu_args a = {};
    // (batch, heads, dim)-shaped tensors, the heads dimension absent in the flat form
    auto bhp = [&](const Arg &t, int64_t *st) {
        if (heads) {
            if (!shape(*t, {batch, H, P})) return false;
            strides(st, *t, 3);
        } else {
            if (!shape(*t, {batch, P})) return false;
            st[0] = t->stride(0); st[1] = 0; st[2] = t->stride(1);
        }
        return true;
    };
    auto hp = [&](const Arg &t, int64_t *st) {
        if (!t.has()) return true;
        if (t->scalar_type() != at::kFloat) return false;
        if (t->dim() == 2) {
            if (!shape(*t, {H, P})) return false;
            strides(st, *t, 2);
        } else {
            if (H != 1 || !shape(*t, {P})) return false;
            st[0] = 0; st[1] = t->stride(0);
        }
        return true;
    };
    if (!bhp(x, a.x_stride) || !bhp(dt, a.dt_stride)) DECLINE();
    if (z.has() && (z->scalar_type() != x->scalar_type() || !bhp(z, a.z_stride))) DECLINE();
    if (!hp(D, a.D_stride) || !hp(bias, a.dt_bias_stride)) DECLINE();
    if (A->scalar_type() != at::kFloat) DECLINE();
    if (A->dim() == 3) {
        if (!shape(*A, {H, P, N})) DECLINE();
        strides(a.A_stride, *A, 3);
    } else {
        if (H != 1 || !shape(*A, {P, N})) DECLINE();
        a.A_stride[0] = 0; a.A_stride[1] = A->stride(0); a.A_stride[2] = A->stride(1);
    }
    const int64_t G = B->dim() == 3 ? B->size(1) : 1;
    auto bgn = [&](const Arg &t, int64_t *st) {
        if (t->dim() == 3) {
            if (!shape(*t, {batch, G, N})) return false;
            strides(st, *t, 3);
        } else {
            if (G != 1 || !shape(*t, {batch, N})) return false;
            st[0] = t->stride(0); st[1] = 0; st[2] = t->stride(1);
        }
        return true;
    };
    if (G <= 0 || H % G || !bgn(B, a.B_stride) || !bgn(C, a.C_stride) || B->scalar_type() != C->scalar_type()) DECLINE();
    if (idx.has()) {
        if (idx->scalar_type() != at::kInt || !shape(*idx, {batch}) || !idx->is_contiguous()) DECLINE();
    } else if (state->size(0) != batch) {
        DECLINE();
    }
    a.state_dtype = code(state->scalar_type()); a.x_dtype = code(x->scalar_type()); a.dt_dtype = code(dt->scalar_type());
    a.bc_dtype = code(B->scalar_type());
    if (a.state_dtype < 0 || a.x_dtype < 0 || a.dt_dtype < 0 || a.bc_dtype < 0) DECLINE();
    const Tensor out = empty_as(*x);
    a.state = state.ptr(); a.x = x.ptr(); a.dt = dt.ptr(); a.A = static_cast<const float *>(A.ptr()); a.B = B.ptr(); a.C = C.ptr();
    a.D = static_cast<const float *>(D.ptr()); a.z = z.ptr(); a.dt_bias = static_cast<const float *>(bias.ptr()); a.out = out.data_ptr();
    a.state_batch_indices = static_cast<const int32_t *>(idx.ptr());
    a.batch = (int)batch; a.nheads = (int)H; a.dim = (int)P; a.dstate = (int)N; a.ngroups = (int)G;
    a.dt_softplus = PyObject_IsTrue(v[9]) == 1;
    a.device = x->device().index();
    if (heads) {
        strides(a.state_stride, *state, 4);
        strides(a.out_stride, out, 3);
    } else {
        a.state_stride[0] = state->stride(0); a.state_stride[1] = 0; a.state_stride[2] = state->stride(1); a.state_stride[3] = state->stride(2);
        a.out_stride[0] = out.stride(0); a.out_stride[1] = 0; a.out_stride[2] = out.stride(1);
    }
    if (mb200_selective_state_update(&a, stream_of(*x)) != MB200_OK) DECLINE();
    return wrap(out);
    GUARD_END
}

// ---------------------------------------------------------------------------------------------------- conv1d
bool conv_weights(const Arg &w, const Arg &bias, int64_t dim)
{
    if (w->dim() != 2 || w->size(0) != dim || !w->is_contiguous() || code(w->scalar_type()) < 0) return false;
    return !bias.has() || (bias->dim() == 1 && bias->size(0) == dim && bias->is_contiguous() && bias->scalar_type() == w->scalar_type());
}
// None or "silu" / "swish"; -1 for anything else
int activation_code(PyObject *o)
{
    if (o == Py_None) return 0;
    if (!PyUnicode_Check(o)) return -1;
    return PyUnicode_CompareWithASCIIString(o, "silu") == 0 || PyUnicode_CompareWithASCIIString(o, "swish") == 0 ? 1 : -1;
}

// (x, weight, bias, seq_idx, activation) -> out | None
PyObject *conv1d_fwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 5;
    if (bad) DECLINE();
    const Arg x = take(v[0], bad), w = take(v[1], bad), bias = take(v[2], bad, true), sid = take(v[3], bad, true);
    const int act = activation_code(v[4]);
    if (bad || act < 0 || x->dim() != 3 || !small(*x) || code(x->scalar_type()) < 0) DECLINE();
    const int64_t batch = x->size(0), dim = x->size(1), L = x->size(2);
    if (!conv_weights(w, bias, dim) || !one_device(*x, {w, bias, sid}) || (x->stride(2) != 1 && x->stride(1) != 1)) DECLINE();
    if (sid.has() && (sid->scalar_type() != at::kInt || !shape(*sid, {batch, L}) || !sid->is_contiguous())) DECLINE();
    mb200_conv1d_args a = {};
    const Tensor out = empty_as(*x);
    a.x = x.ptr(); a.weight = w.ptr(); a.bias = bias.ptr(); a.seq_idx = static_cast<const int32_t *>(sid.ptr()); a.out = out.data_ptr();
    a.batch = (int)batch; a.dim = (int)dim; a.seqlen = (int)L; a.width = (int)w->size(1);
    a.io_dtype = code(x->scalar_type()); a.w_dtype = code(w->scalar_type()); a.activation = act; a.device = x->device().index();
    strides(a.x_stride, *x, 3);
    strides(a.out_stride, out, 3);
    if (mb200_causal_conv1d_fwd(&a, stream_of(*x)) != MB200_OK) DECLINE();
    return wrap(out);
    GUARD_END
}

// (x, conv_state, weight, bias, activation) -> out | None
PyObject *conv1d_update(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 5;
    if (bad) DECLINE();
    const Arg x = take(v[0], bad), st = take(v[1], bad), w = take(v[2], bad), bias = take(v[3], bad, true);
    const int act = activation_code(v[4]);
    if (bad || act < 0 || x->dim() != 2 || !small(*x) || code(x->scalar_type()) < 0) DECLINE();
    const int64_t batch = x->size(0), dim = x->size(1);
    if (!conv_weights(w, bias, dim) || !one_device(*x, {w, bias, st})) DECLINE();
    if (st->dim() != 3 || st->size(0) != batch || st->size(1) != dim || st->scalar_type() != x->scalar_type()) DECLINE();
    mb200_conv1d_update_args a = {};
    const Tensor out = empty_as(*x);
    a.x = x.ptr(); a.weight = w.ptr(); a.bias = bias.ptr(); a.conv_state = st.ptr(); a.out = out.data_ptr();
    a.batch = (int)batch; a.dim = (int)dim; a.width = (int)w->size(1); a.state_len = (int)st->size(2);
    a.io_dtype = code(x->scalar_type()); a.w_dtype = code(w->scalar_type()); a.activation = act; a.device = x->device().index();
    strides(a.x_stride, *x, 2);
    strides(a.out_stride, out, 2);
    strides(a.state_stride, *st, 3);
    if (mb200_causal_conv1d_update(&a, stream_of(*x)) != MB200_OK) DECLINE();
    return wrap(out);
    GUARD_END
}

// ---------------------------------------------------------------------------------------------------- gated RMSNorm
bool norm_weights(const Arg &w, const Arg &bias, int64_t ncols)
{
    if (w->dim() != 1 || w->size(0) != ncols || !w->is_contiguous() || code(w->scalar_type()) < 0) return false;
    return !bias.has() || (bias->dim() == 1 && bias->size(0) == ncols && bias->is_contiguous() && bias->scalar_type() == w->scalar_type());
}
// Rows of a (..., ncols) tensor at one stride: 2-d tensors as they are, others only when contiguous.
bool row_stride(const Tensor &t, int64_t &st)
{
    if (t.dim() < 1 || t.stride(-1) != 1) return false;
    if (t.dim() == 2) { st = t.stride(0); return true; }
    if (!t.is_contiguous()) return false;
    st = t.size(-1);
    return true;
}

// (x, weight, bias, z, eps, group_size, norm_before_gate) -> out | None
PyObject *rmsnorm(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 7;
    if (bad) DECLINE();
    const Arg x = take(v[0], bad), w = take(v[1], bad), bias = take(v[2], bad, true), z = take(v[3], bad, true);
    if (bad || x->dim() < 1 || code(x->scalar_type()) < 0 || x->numel() == 0) DECLINE();
    const int64_t ncols = x->size(-1);
    const int64_t group = v[5] == Py_None ? ncols : PyLong_AsLongLong(v[5]);
    const double eps = PyFloat_AsDouble(v[4]);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        DECLINE();
    }
    if (ncols > INT32_MAX || group <= 0 || ncols % group || !norm_weights(w, bias, ncols) || !one_device(*x, {w, bias, z})) DECLINE();
    mb200_rmsnorm_args a = {};
    if (!row_stride(*x, a.x_stride)) DECLINE();
    if (z.has() && (z->sizes() != x->sizes() || z->scalar_type() != x->scalar_type() || !row_stride(*z, a.z_stride))) DECLINE();
    const Tensor out = empty(x->sizes(), x->scalar_type(), x->device());
    a.x = x.ptr(); a.z = z.ptr(); a.weight = w.ptr(); a.bias = bias.ptr(); a.out = out.data_ptr();
    a.nrows = x->numel() / ncols; a.ncols = (int)ncols; a.group_size = (int)group;
    a.io_dtype = code(x->scalar_type()); a.w_dtype = code(w->scalar_type()); a.norm_before_gate = PyObject_IsTrue(v[6]) == 1;
    a.eps = (float)eps; a.device = x->device().index();
    a.out_stride = ncols;
    if (mb200_rmsnorm_gated_fwd(&a, stream_of(*x)) != MB200_OK) DECLINE();
    return wrap(out);
    GUARD_END
}

// ---------------------------------------------------------------------------------------------------- SSD
struct Limits { float lo, hi; };
// (lo, hi) of dt_limit; the library wants a finite upper end
bool dt_limits(PyObject *o, Limits &l)
{
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 2) return false;
    const double lo = PyFloat_AsDouble(PyTuple_GET_ITEM(o, 0)), hi = PyFloat_AsDouble(PyTuple_GET_ITEM(o, 1));
    if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    l.lo = (float)lo;
    l.hi = (float)(hi < 3.0e38 ? hi : 3.0e38);
    return true;
}

// (x, dt, A, B, C, chunk_size, D, z, dt_bias, initial_states, seq_idx, cu_seqlens, dt_softplus, dt_limit, return_final_states,
//  return_varlen_states) -> (out, final_states, varlen_states, status) | None
PyObject *ssd_fwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 16;
    if (bad) DECLINE();
    const Arg x = take(v[0], bad), dt = take(v[1], bad), A = take(v[2], bad), B = take(v[3], bad), C = take(v[4], bad), D = take(v[6], bad, true),
              z = take(v[7], bad, true), bias = take(v[8], bad, true), init = take(v[9], bad, true), sid = take(v[10], bad, true);
    const bool want_final = PyObject_IsTrue(v[14]) == 1, want_varlen = PyObject_IsTrue(v[15]) == 1;
    Arg cu;
    if (want_varlen) cu = take(v[11], bad);
    const long chunk = PyLong_Check(v[5]) ? PyLong_AsLong(v[5]) : -1;
    Limits lim;
    if (bad || chunk <= 0 || chunk > 1024 || !dt_limits(v[13], lim)) DECLINE();
    if (x->dim() != 4 || B->dim() != 4 || !small(*x) || !small(*B)) DECLINE();
    const int64_t batch = x->size(0), L = x->size(1), H = x->size(2), P = x->size(3), G = B->size(2), N = B->size(3);
    if (L == 0 || batch == 0 || G == 0 || H % G) DECLINE();
    const at::ScalarType io = x->scalar_type();
    if (code(io) < 0 || code(dt->scalar_type()) < 0 || B->scalar_type() != io || C->scalar_type() != io) DECLINE();
    if (!shape(*B, {batch, L, G, N}) || C->sizes() != B->sizes() || !shape(*dt, {batch, L, H}) || !is_vec(A, H) || !is_vec(bias, H)) DECLINE();
    if (x->stride(3) != 1 || B->stride(3) != 1 || C->stride(3) != 1) DECLINE();
    if (z.has() && (z->sizes() != x->sizes() || z->scalar_type() != io || z->stride(3) != 1)) DECLINE();
    if (D.has() && (D->scalar_type() != at::kFloat || !D->is_contiguous() || !(shape(*D, {H, P}) || shape(*D, {H})))) DECLINE();
    if (init.has() && (init->scalar_type() != at::kFloat || !init->is_contiguous() || !shape(*init, {batch, H, P, N}))) DECLINE();
    if (sid.has() && (sid->scalar_type() != at::kInt || !sid->is_contiguous() || !shape(*sid, {batch, L}))) DECLINE();
    if (cu.has() && (cu->scalar_type() != at::kInt || !cu->is_contiguous() || cu->dim() != 1 || cu->size(0) < 1 || batch != 1)) DECLINE();
    if (!one_device(*x, {dt, A, B, C, D, z, bias, init, sid, cu})) DECLINE();
    const c10::Device dev = x->device();
    mb200_ssd_args a = {};
    a.batch = (int)batch; a.seqlen = (int)L; a.nheads = (int)H; a.headdim = (int)P; a.ngroups = (int)G; a.dstate = (int)N; a.chunk_size = (int)chunk;
    a.io_dtype = code(io); a.dt_dtype = code(dt->scalar_type()); a.dt_softplus = PyObject_IsTrue(v[12]) == 1;
    a.D_has_hdim = D.has() && D->dim() == 2;
    a.dt_min = lim.lo; a.dt_max = lim.hi;
    a.phases = MB200_SSD_PHASE_ALL;
    a.device = dev.index();
    size_t need = 0;
    if (mb200_ssd_scratch_bytes(&a, &need) != MB200_OK) DECLINE();
    const Tensor out = empty_as(*x), scratch = bytes(std::max<size_t>(need, 256), dev), status = bytes(256, dev);
    if (out.stride(3) != 1) DECLINE();
    Tensor fin, var;
    if (want_final) fin = empty({batch, H, P, N}, at::kFloat, dev);
    if (cu.has()) var = empty({cu->size(0) - 1, H, P, N}, at::kFloat, dev);
    a.x = x.ptr(); a.dt = dt.ptr(); a.A = static_cast<const float *>(A.ptr()); a.B = B.ptr(); a.C = C.ptr(); a.D = static_cast<const float *>(D.ptr());
    a.z = z.ptr(); a.dt_bias = static_cast<const float *>(bias.ptr()); a.seq_idx = static_cast<const int32_t *>(sid.ptr());
    a.initial_states = static_cast<const float *>(init.ptr()); a.out = out.data_ptr();
    a.final_states = want_final ? static_cast<float *>(fin.data_ptr()) : nullptr;
    a.scratch = scratch.data_ptr(); a.scratch_bytes = need;
    a.status = static_cast<int32_t *>(status.data_ptr());
    if (cu.has()) {
        a.cu_seqlens = static_cast<const int32_t *>(cu.ptr());
        a.varlen_states = static_cast<float *>(var.data_ptr());
        a.num_seqs = (int)cu->size(0) - 1;
    }
    strides(a.x_stride, *x, 3);
    strides(a.dt_stride, *dt, 3);
    strides(a.B_stride, *B, 3);
    strides(a.C_stride, *C, 3);
    strides(a.out_stride, out, 3);
    if (z.has()) strides(a.z_stride, *z, 3);
    if (mb200_ssd_chunk_scan_fwd(&a, stream_of(*x)) != MB200_OK) DECLINE();
    auto opt = [](bool on, const Tensor &t) -> PyObject * {
        if (on) return wrap(t);
        Py_RETURN_NONE;
    };
    return Py_BuildValue("(NNNN)", wrap(out), opt(want_final, fin), opt(cu.has(), var), wrap(status));
    GUARD_END
}

// The Mamba-2 block after its input projection.  (zxbcdt, conv1d_weight, conv1d_bias, dt_bias, A, D, chunk_size, initial_states,
// seq_idx, dt_limit, return_final_states, activation, rmsnorm_weight, rmsnorm_eps, outproj_weight, outproj_bias, headdim,
// ngroups, norm_before_gate) -> (out, final_states | None, status) | None.  Handles blocks without a non-SSM part, whose
// conv, scan and norm read their column ranges of zxbcdt and of the conv's output in place.
PyObject *block_fwd(PyObject *, PyObject *const *v, Py_ssize_t n)
{
    GUARD_BEGIN
    bool bad = n != 19;
    if (bad) DECLINE();
    const Arg zx = take(v[0], bad), cw = take(v[1], bad), cb = take(v[2], bad, true), bias = take(v[3], bad), A = take(v[4], bad), D = take(v[5], bad),
              init = take(v[7], bad, true), sid = take(v[8], bad, true), nw = take(v[12], bad, true), ow = take(v[14], bad, true),
              ob = take(v[15], bad, true);
    const int act = activation_code(v[11]);
    const long chunk = PyLong_Check(v[6]) ? PyLong_AsLong(v[6]) : -1, G = PyLong_Check(v[17]) ? PyLong_AsLong(v[17]) : -1;
    long P = v[16] == Py_None ? 0 : (PyLong_Check(v[16]) ? PyLong_AsLong(v[16]) : -1);
    Limits lim;
    if (bad || act < 0 || chunk <= 0 || chunk > 1024 || G <= 0 || P < 0 || !dt_limits(v[9], lim)) DECLINE();
    if (wants_grad({zx, cw, cb, bias, A, D, init, nw, ow, ob})) DECLINE();
    const double eps = PyFloat_AsDouble(v[13]);
    if (PyErr_Occurred()) {
        PyErr_Clear();
        DECLINE();
    }
    if (zx->dim() != 3 || zx->stride(2) != 1 || !small(*zx) || code(zx->scalar_type()) < 0) DECLINE();
    const at::ScalarType io = zx->scalar_type();
    if (D->dim() == 2) P = D->size(1);
    if (D->dim() < 1 || D->dim() > 2 || P <= 0 || D->scalar_type() != at::kFloat || !D->is_contiguous()) DECLINE();
    const int64_t batch = zx->size(0), L = zx->size(1), H = D->size(0), dim = H * P, ch = cw->dim() == 2 ? cw->size(0) : 0;
    if (H % G || ch <= dim || (ch - dim) % (2 * G)) DECLINE();
    const int64_t N = (ch - dim) / (2 * G);
    if (zx->size(2) != dim + ch + H || batch == 0 || L == 0) DECLINE();
    if (!conv_weights(cw, cb, ch) || !is_vec(A, H) || !is_vec(bias, H)) DECLINE();
    if (init.has() && (init->scalar_type() != at::kFloat || !init->is_contiguous() || !shape(*init, {batch, H, P, N}))) DECLINE();
    if (sid.has() && (sid->scalar_type() != at::kInt || !sid->is_contiguous() || !shape(*sid, {batch, L}))) DECLINE();
    if (nw.has() && !norm_weights(nw, Arg(), dim)) DECLINE();
    if (!ow.has() && ob.has()) DECLINE();
    if (nw.has() && batch > 1 && zx->stride(0) != L * zx->stride(1)) DECLINE();      // the norm wants its rows at one stride
    if (!one_device(*zx, {cw, cb, bias, A, D, init, sid, nw, ow, ob})) DECLINE();
    const c10::Device dev = zx->device();
    void *stream = stream_of(*zx);
    const size_t e = at::elementSize(io);
    const int iocode = code(io);
    const int64_t sb = zx->stride(0), sl = zx->stride(1);
    char *zp = static_cast<char *>(zx.ptr()), *xbc = zp + dim * e, *dtp = xbc + ch * e;      // z | x B C | dt

    const Tensor conv = empty({batch, L, ch}, io, dev);
    {
        mb200_conv1d_args a = {};
        a.x = xbc; a.weight = cw.ptr(); a.bias = cb.ptr(); a.seq_idx = static_cast<const int32_t *>(sid.ptr()); a.out = conv.data_ptr();
        a.batch = (int)batch; a.dim = (int)ch; a.seqlen = (int)L; a.width = (int)cw->size(1);
        a.io_dtype = iocode; a.w_dtype = code(cw->scalar_type()); a.activation = act; a.device = dev.index();
        a.x_stride[0] = sb; a.x_stride[1] = 1; a.x_stride[2] = sl;
        a.out_stride[0] = L * ch; a.out_stride[1] = 1; a.out_stride[2] = ch;
        if (mb200_causal_conv1d_fwd(&a, stream) != MB200_OK) DECLINE();
    }
    const bool want_final = PyObject_IsTrue(v[10]) == 1;
    Tensor y = empty({batch, L, dim}, io, dev), fin;
    const Tensor status = bytes(256, dev);
    if (want_final) fin = empty({batch, H, P, N}, at::kFloat, dev);
    {
        mb200_ssd_args a = {};
        a.batch = (int)batch; a.seqlen = (int)L; a.nheads = (int)H; a.headdim = (int)P; a.ngroups = (int)G; a.dstate = (int)N; a.chunk_size = (int)chunk;
        a.io_dtype = iocode; a.dt_dtype = iocode; a.dt_softplus = 1; a.D_has_hdim = D->dim() == 2;
        a.dt_min = lim.lo; a.dt_max = lim.hi; a.phases = MB200_SSD_PHASE_ALL; a.device = dev.index();
        size_t need = 0;
        if (mb200_ssd_scratch_bytes(&a, &need) != MB200_OK) DECLINE();
        const Tensor scratch = bytes(std::max<size_t>(need, 256), dev);
        char *cp = static_cast<char *>(conv.data_ptr());
        a.x = cp; a.B = cp + dim * e; a.C = cp + (dim + G * N) * e; a.dt = dtp;
        a.A = static_cast<const float *>(A.ptr()); a.D = static_cast<const float *>(D.ptr()); a.dt_bias = static_cast<const float *>(bias.ptr());
        a.z = nw.has() ? nullptr : zp;
        a.seq_idx = static_cast<const int32_t *>(sid.ptr()); a.initial_states = static_cast<const float *>(init.ptr());
        a.out = y.data_ptr(); a.final_states = want_final ? static_cast<float *>(fin.data_ptr()) : nullptr;
        a.scratch = scratch.data_ptr(); a.scratch_bytes = need; a.status = static_cast<int32_t *>(status.data_ptr());
        auto set = [](int64_t *d, int64_t s0, int64_t s1, int64_t s2) { d[0] = s0; d[1] = s1; d[2] = s2; };
        set(a.x_stride, L * ch, ch, P);
        set(a.B_stride, L * ch, ch, N);
        set(a.C_stride, L * ch, ch, N);
        set(a.dt_stride, sb, sl, 1);
        set(a.z_stride, sb, sl, P);
        set(a.out_stride, L * dim, dim, P);
        if (mb200_ssd_chunk_scan_fwd(&a, stream) != MB200_OK) DECLINE();
    }
    if (nw.has()) {
        mb200_rmsnorm_args a = {};
        a.x = y.data_ptr(); a.z = zp; a.weight = nw.ptr(); a.out = y.data_ptr();      // in place: a row is read before it is written
        a.nrows = batch * L; a.ncols = (int)dim; a.group_size = (int)(dim / G);
        a.io_dtype = iocode; a.w_dtype = code(nw->scalar_type()); a.norm_before_gate = PyObject_IsTrue(v[18]) == 1;
        a.eps = (float)eps; a.device = dev.index();
        a.x_stride = dim; a.z_stride = sl; a.out_stride = dim;
        if (mb200_rmsnorm_gated_fwd(&a, stream) != MB200_OK) DECLINE();
    }
    if (ow.has()) y = ob.has() ? at::linear(y, *ow, *ob) : at::linear(y, *ow);
    return Py_BuildValue("(NNN)", wrap(y), want_final ? wrap(fin) : (Py_INCREF(Py_None), Py_None), wrap(status));
    GUARD_END
}

#define ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {ENTRY(scan_fwd), ENTRY(scan_bwd), ENTRY(state_update), ENTRY(conv1d_fwd), ENTRY(conv1d_update),
                         ENTRY(rmsnorm), ENTRY(ssd_fwd), ENTRY(block_fwd), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native call path of the mamba_b200 operators.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }

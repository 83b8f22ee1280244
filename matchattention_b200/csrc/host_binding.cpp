// Host side of the eager entry points in matchattention_b200/ops.py as a CPython extension: argument checks, output
// allocation and the call through the C ABI (include/matchattn.h) in one step.
//
// Why: a small operator call runs about 10 us on the device, while checking six tensors attribute by attribute in
// Python, a torch custom-op dispatch and a ctypes call with 19 arguments took about 60 us on the host.  Here it is
// about 6 us, most of it the launch itself and two tensor allocations.
//
// Every function returns None when it does not cover its arguments (a tensor subclass or wrapper, a tracing,
// function or dispatch mode, a wrong type, shape, device or layout); the caller then takes the Python path, which handles the rest
// and words the errors.  Nothing is kept between calls.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/PyInterpreter.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <cstdio>
#include <cstring>
#include <optional>

#include "../../include/matchattn.h"

namespace {

using at::Tensor;

// ---- arguments ------------------------------------------------------------------------------------------

// No functional transform (vmap, grad, functionalisation) is active.
bool untransformed()
{
    using c10::DispatchKey;
    static const c10::DispatchKeySet modes({DispatchKey::FuncTorchDynamicLayerFrontMode, DispatchKey::FuncTorchDynamicLayerBackMode,
                                            DispatchKey::Functionalize});
    return !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes);
}

// A torch function mode that has to see the calls.  (The one behind torch.set_default_device only places new tensors.)
bool function_mode()
{
    if (!at::impl::torch_function_mode_enabled()) return false;
    for (int64_t i = 0; i < at::impl::PythonTorchFunctionTLS::stack_len(); ++i) {
        PyObject *mode = at::impl::PythonTorchFunctionTLS::get_stack_at(i)->ptr(getPyInterpreter());
        if (std::strcmp(Py_TYPE(mode)->tp_name, "DeviceContext") != 0) return true;
    }
    return false;
}

// ... nor any mode that has to see the operators of this call (function and dispatch modes, tracing).
bool eager()
{
    using c10::DispatchKey;
    static const c10::DispatchKeySet modes({DispatchKey::Python, DispatchKey::PythonDispatcher, DispatchKey::PreDispatch});
    return untransformed() && !c10::impl::TorchDispatchModeTLS::any_modes_set() && !function_mode() &&
           !c10::impl::tls_local_dispatch_key_set().included_.has_any(modes) && !torch::jit::tracer::isTracing();
}

// A plain CUDA tensor (not wrapped by a transform; with `exact`, not an instance of a subclass either).
bool cuda_tensor(PyObject *o, Tensor &t, bool exact = true)
{
    using c10::DispatchKey;
    if (exact ? !THPVariable_CheckExact(o) : !THPVariable_Check(o)) return false;
    t = THPVariable_Unpack(o);
    static const c10::DispatchKeySet wrapped({DispatchKey::Python, DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper,
                                              DispatchKey::Functionalize, DispatchKey::Conjugate, DispatchKey::Negative,
                                              DispatchKey::ZeroTensor});
    return t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(wrapped);
}

int dtype_code(const Tensor &t)
{
    switch (t.scalar_type()) {
    case at::kFloat: return MATCHATTN_F32;
    case at::kHalf: return MATCHATTN_F16;
    case at::kBFloat16: return MATCHATTN_BF16;
    default: return -1;
    }
}

bool to_int(PyObject *o, int64_t &v)
{
    v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return v >= -(1LL << 31) && v < (1LL << 31);
}

bool to_float(PyObject *o, double &v)
{
    v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) {
        PyErr_Clear();
        return false;
    }
    return true;
}

// win_r: an int, or a list or tuple of two
bool to_window(PyObject *o, int64_t &rx, int64_t &ry)
{
    if (PyLong_Check(o)) {
        if (!to_int(o, rx)) return false;
        ry = rx;
        return true;
    }
    if (!PyList_Check(o) && !PyTuple_Check(o)) return false;
    return PySequence_Fast_GET_SIZE(o) == 2 && to_int(PySequence_Fast_GET_ITEM(o, 0), rx) && to_int(PySequence_Fast_GET_ITEM(o, 1), ry);
}

bool to_attn_type(PyObject *o, int &code)
{
    if (!PyUnicode_Check(o)) return false;
    if (PyUnicode_CompareWithASCIIString(o, "l1_norm") == 0) code = MATCHATTN_L1_NORM;
    else if (PyUnicode_CompareWithASCIIString(o, "dot_product") == 0) code = MATCHATTN_DOT_PRODUCT;
    else return false;
    return true;
}

bool shaped(const Tensor &t, const Tensor &like, std::initializer_list<int64_t> shape)
{
    return t.scalar_type() == like.scalar_type() && t.device() == like.device() && t.sizes() == at::IntArrayRef(shape.begin(), shape.size()) &&
           t.is_contiguous();
}

// ---- the call -------------------------------------------------------------------------------------------

void *data(const Tensor &t) { return t.data_ptr(); }
void *data_or_null(const std::optional<Tensor> &t) { return t.has_value() ? t->data_ptr() : nullptr; }

// Runs `call(stream)` with the tensor's device current and without the GIL; false and a Python error on failure.
template <typename Call>
bool enqueue(const Tensor &t, Call call)
{
    int status;
    {
        const c10::cuda::CUDAGuard guard(t.device());
        void *stream = c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
        Py_BEGIN_ALLOW_THREADS
        status = call(stream);
        Py_END_ALLOW_THREADS
    }
    if (status == MATCHATTN_OK) return true;
    PyErr_Format(PyExc_RuntimeError, "matchattn_b200: %s (status %d)", matchattn_strerror(status), status);
    return false;
}

// PyTorch exceptions (out of memory in an allocation, ...) as Python exceptions.
template <PyObject *(*F)(PyObject *const *, Py_ssize_t)>
PyObject *entry(PyObject *, PyObject *const *args, Py_ssize_t n)
{
    HANDLE_TH_ERRORS
    return F(args, n);
    END_HANDLE_TH_ERRORS
}

PyObject *not_covered() { Py_RETURN_NONE; }

// ---- training: the operator as an autograd function ------------------------------------------------------
// Only the inputs are saved: the backward recomputes scores and softmaxes.

// the name under which torch.profiler shows the operator: that of the custom op
constexpr const char *kOpName = "matchattn_b200::fused_forward_ops";

void check_status(int status)
{
    TORCH_CHECK(status == MATCHATTN_OK, "matchattn_b200: ", matchattn_strerror(status), " (status ", status, ")");
}

struct MatchAttentionFn : torch::autograd::Function<MatchAttentionFn> {
    static torch::autograd::variable_list forward(torch::autograd::AutogradContext *ctx, const Tensor &mo, const Tensor &q, const Tensor &k,
                                                  const Tensor &v, int64_t H, int64_t W, int64_t r, double scale)
    {
        const int64_t B = q.size(0), Nq = q.size(1), C = q.size(2), h = mo.size(2), M = (2 * r + 2) * (2 * r + 2);
        Tensor out = at::empty({B, Nq, C}, q.options()), attn = at::empty({B, Nq, h, M}, q.options());
        const c10::cuda::CUDAGuard device(q.device());
        RECORD_FUNCTION(kOpName, std::vector<c10::IValue>({mo, q, k, v}));
        check_status(matchattn_fused_forward(data(mo), data(q), data(k), data(v), data(out), data(attn), B, H, W, h, C / h, r, r,
                                             dtype_code(q), MATCHATTN_L1_NORM, static_cast<float>(scale), 0, H,
                                             c10::cuda::getCurrentCUDAStream(q.device().index()).stream()));
        ctx->save_for_backward({mo, q, k, v});
        ctx->saved_data["H"] = H;
        ctx->saved_data["W"] = W;
        ctx->saved_data["r"] = r;
        ctx->saved_data["scale"] = scale;
        ctx->set_materialize_grads(false);
        return {out, attn};
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads)
    {
        const auto saved = ctx->get_saved_variables();
        const Tensor &mo = saved[0], &q = saved[1], &k = saved[2], &v = saved[3];
        const int64_t H = ctx->saved_data["H"].toInt(), W = ctx->saved_data["W"].toInt(), r = ctx->saved_data["r"].toInt();
        const int64_t B = q.size(0), C = q.size(2), h = mo.size(2);
        Tensor d_out = grads[0].defined() ? grads[0].contiguous().resolve_neg() : at::zeros_like(q);
        Tensor d_attn = grads[1].defined() ? grads[1].contiguous().resolve_neg() : Tensor();
        Tensor d_q = at::empty_like(q), d_mo = ctx->needs_input_grad(0) ? at::empty_like(mo) : Tensor();
        const float scale = static_cast<float>(ctx->saved_data["scale"].toDouble());
        const c10::cuda::CUDAGuard guard(q.device());
        void *stream = c10::cuda::getCurrentCUDAStream(q.device().index()).stream();
        void *dattn = d_attn.defined() ? data(d_attn) : nullptr, *dmo = d_mo.defined() ? data(d_mo) : nullptr;
        const size_t bytes = matchattn_backward_workspace_bytes(B, H, W, h, C / h, r, dtype_code(q), 0, H);
        // without room for the workspace (8 bytes per query, head and tap) the accumulating call below serves
        Tensor ws;
        if (bytes != 0) {
            try {
                ws = at::empty({static_cast<int64_t>(bytes)}, q.options().dtype(at::kByte));
            } catch (const c10::OutOfMemoryError &) {
            }
        }
        if (ws.defined()) {
            Tensor d_k = at::empty_like(k), d_v = at::empty_like(v);
            const int status = matchattn_fused_backward_ws(data(mo), data(q), data(k), data(v), data(d_out), dattn, data(d_q), data(d_k), data(d_v),
                                                           dmo, B, H, W, h, C / h, r, r, dtype_code(q), MATCHATTN_L1_NORM, scale, 0, H, data(ws),
                                                           bytes, stream);
            if (status != MATCHATTN_ERR_VARIANT) {       // that one: a tensor is not 32-byte aligned
                check_status(status);
                return {d_mo, d_q, d_k, d_v, Tensor(), Tensor(), Tensor(), Tensor()};
            }
        }
        Tensor d_k = at::zeros(k.sizes(), k.options().dtype(at::kFloat)), d_v = at::zeros(v.sizes(), v.options().dtype(at::kFloat));
        check_status(matchattn_fused_backward(data(mo), data(q), data(k), data(v), data(d_out), dattn, data(d_q), static_cast<float *>(data(d_k)),
                                              static_cast<float *>(data(d_v)), dmo, B, H, W, h, C / h, r, r, dtype_code(q), MATCHATTN_L1_NORM,
                                              scale, 0, H, stream));
        return {d_mo, d_q, d_k.to(k.scalar_type()), d_v.to(v.scalar_type()), Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// ---- entry points ---------------------------------------------------------------------------------------

// The tensors of an operator call, checked; `rows` = query rows of the band.
struct Operands {
    Tensor mo, q, k, v;
    int64_t B, Nq, C, h;
    int dtype;
    bool read(PyObject *const *a, int64_t H, int64_t W, int64_t rows, bool exact = true)
    {
        if (!cuda_tensor(a[0], mo, exact) || !cuda_tensor(a[1], q, exact) || !cuda_tensor(a[2], k, exact) || !cuda_tensor(a[3], v, exact)) return false;
        dtype = dtype_code(q);
        if (dtype < 0 || q.dim() != 3 || mo.dim() != 4) return false;
        B = q.size(0);
        Nq = q.size(1);
        C = q.size(2);
        h = mo.size(2);
        return h > 0 && C % h == 0 && Nq == rows * W && shaped(q, q, {B, Nq, C}) && shaped(mo, q, {B, Nq, h, 2}) &&
               shaped(k, q, {B, H * W, C}) && shaped(v, q, {B, H * W, C});
    }
};

// module_forward(max_offset, q, k, v, H, W, win_r, attn_num, attn_type, scale) -> (out, attn)
PyObject *module_forward(PyObject *const *a, Py_ssize_t n)
{
    Operands o;
    int64_t H, W, rx, ry, M;
    int type;
    double scale;
    if (n != 10 || !to_int(a[4], H) || !to_int(a[5], W) || !to_window(a[6], rx, ry) || !to_int(a[7], M) || !to_attn_type(a[8], type) ||
        !to_float(a[9], scale) || rx < 0 || ry < 0 || M != (2 * rx + 2) * (2 * ry + 2) || !eager() || !o.read(a, H, W, H))
        return not_covered();
    if (at::GradMode::is_enabled() && (o.mo.requires_grad() || o.q.requires_grad() || o.k.requires_grad() || o.v.requires_grad())) {
        if (type != MATCHATTN_L1_NORM || rx != ry) return not_covered();
        torch::autograd::variable_list out;
        {
            pybind11::gil_scoped_release release;
            out = MatchAttentionFn::apply(o.mo, o.q, o.k, o.v, H, W, rx, scale);
        }
        return Py_BuildValue("(NN)", THPVariable_Wrap(out[0]), THPVariable_Wrap(out[1]));
    }
    if (PyLong_Check(a[6])) return not_covered();      // the custom op wants a list
    Tensor out = at::empty({o.B, o.Nq, o.C}, o.q.options()), attn = at::empty({o.B, o.Nq, o.h, M}, o.q.options());
    RECORD_FUNCTION(kOpName, std::vector<c10::IValue>({o.mo, o.q, o.k, o.v}));
    if (!enqueue(o.q, [&](void *stream) {
            return matchattn_fused_forward(data(o.mo), data(o.q), data(o.k), data(o.v), data(out), data(attn), o.B, H, W, o.h, o.C / o.h, rx, ry,
                                           o.dtype, type, static_cast<float>(scale), 0, H, stream);
        }))
        return nullptr;
    return Py_BuildValue("(NN)", THPVariable_Wrap(out), THPVariable_Wrap(attn));
}

// autograd(max_offset, q, k, v, H, W, r, scale) -> (out, attn) with a grad_fn
PyObject *autograd(PyObject *const *a, Py_ssize_t n)
{
    Operands o;
    int64_t H, W, r;
    double scale;
    if (n != 8 || !to_int(a[4], H) || !to_int(a[5], W) || !to_int(a[6], r) || !to_float(a[7], scale) || r < 0 || !untransformed() || !o.read(a, H, W, H, false))
        return not_covered();
    torch::autograd::variable_list out;
    {
        pybind11::gil_scoped_release release;
        out = MatchAttentionFn::apply(o.mo, o.q, o.k, o.v, H, W, r, scale);
    }
    return Py_BuildValue("(NN)", THPVariable_Wrap(out[0]), THPVariable_Wrap(out[1]));
}

// launch(max_offset, q, k, v, out, attn or None, H, W, win_r, attn_type, scale, q_row_begin, q_row_end) -> True
PyObject *launch(PyObject *const *a, Py_ssize_t n)
{
    Operands o;
    Tensor out;
    std::optional<Tensor> attn;
    int64_t H, W, rx, ry, r0, r1;
    int type;
    double scale;
    if (n != 13 || !to_int(a[6], H) || !to_int(a[7], W) || !to_window(a[8], rx, ry) || !to_attn_type(a[9], type) || !to_float(a[10], scale) ||
        !to_int(a[11], r0) || !to_int(a[12], r1) || rx < 0 || ry < 0 || !eager() || !o.read(a, H, W, r1 - r0) || !cuda_tensor(a[4], out) ||
        !shaped(out, o.q, {o.B, o.Nq, o.C}))
        return not_covered();
    if (a[5] != Py_None) {
        Tensor t;
        if (!cuda_tensor(a[5], t) || !shaped(t, o.q, {o.B, o.Nq, o.h, (2 * rx + 2) * (2 * ry + 2)})) return not_covered();
        attn = t;
    }
    if (!enqueue(o.q, [&](void *stream) {
            return matchattn_fused_forward(data(o.mo), data(o.q), data(o.k), data(o.v), data(out), data_or_null(attn), o.B, H, W, o.h, o.C / o.h,
                                           rx, ry, o.dtype, type, static_cast<float>(scale), r0, r1, stream);
        }))
        return nullptr;
    Py_RETURN_TRUE;
}

// cross_core(max_offset, q, k, v, gate or None, H, W, r, scale, clamp, kv_shift) -> [B, N, C + h*(2r+2)^2]
PyObject *cross_core(PyObject *const *a, Py_ssize_t n)
{
    Operands o;
    std::optional<Tensor> gate;
    int64_t H, W, r, shift;
    double scale;
    if (n != 11 || !to_int(a[5], H) || !to_int(a[6], W) || !to_int(a[7], r) || !to_float(a[8], scale) || !to_int(a[10], shift) || r < 0 ||
        !eager() || !o.read(a, H, W, H))
        return not_covered();
    const int clamp = PyObject_IsTrue(a[9]);
    if (clamp < 0) {
        PyErr_Clear();
        return not_covered();
    }
    if (a[4] != Py_None) {
        Tensor t;
        if (!cuda_tensor(a[4], t) || !shaped(t, o.q, {o.B, o.Nq, o.C})) return not_covered();
        gate = t;
    }
    const int64_t width = o.C + o.h * (2 * r + 2) * (2 * r + 2);
    Tensor buf = at::empty({o.B, o.Nq, width}, o.q.options());
    if (!enqueue(o.q, [&](void *stream) {
            return matchattn_fused_forward_glue(data(o.mo), data(o.q), data(o.k), data(o.v), data_or_null(gate), data(buf),
                                                static_cast<char *>(data(buf)) + o.C * buf.element_size(), o.B, H, W, o.h, o.C / o.h, r, r, o.dtype,
                                                MATCHATTN_L1_NORM, static_cast<float>(scale), 0, H, clamp, width, width, shift, stream);
        }))
        return nullptr;
    return THPVariable_Wrap(buf);
}

// self_core(max_offset, q, k, v, H, W, r, scale, clamp) -> out
PyObject *self_core(PyObject *const *a, Py_ssize_t n)
{
    Operands o;
    int64_t H, W, r;
    double scale;
    if (n != 9 || !to_int(a[4], H) || !to_int(a[5], W) || !to_int(a[6], r) || !to_float(a[7], scale) || r < 0 || !eager() || !o.read(a, H, W, H))
        return not_covered();
    const int clamp = PyObject_IsTrue(a[8]);
    if (clamp < 0) {
        PyErr_Clear();
        return not_covered();
    }
    Tensor out = at::empty({o.B, o.Nq, o.C}, o.q.options());
    if (!enqueue(o.q, [&](void *stream) {
            return matchattn_fused_forward_glue(data(o.mo), data(o.q), data(o.k), data(o.v), nullptr, data(out), nullptr, o.B, H, W, o.h, o.C / o.h,
                                                r, r, o.dtype, MATCHATTN_L1_NORM, static_cast<float>(scale), 0, H, clamp, 0, 0, 0, stream);
        }))
        return nullptr;
    return THPVariable_Wrap(out);
}

// upsample_field(field, mask, factor) -> [B, f*H, f*W, D]
PyObject *upsample_field(PyObject *const *a, Py_ssize_t n)
{
    Tensor field, mask;
    int64_t f;
    if (n != 3 || !to_int(a[2], f) || f <= 0 || !eager() || !cuda_tensor(a[0], field) || !cuda_tensor(a[1], mask) || dtype_code(field) < 0 ||
        field.dim() != 4)
        return not_covered();
    const int64_t B = field.size(0), H = field.size(1), W = field.size(2), D = field.size(3);
    if (mask.scalar_type() != field.scalar_type() || mask.device() != field.device() || mask.sizes() != at::IntArrayRef({B, 9 * f * f, H, W}))
        return not_covered();
    field = field.contiguous();
    mask = mask.contiguous();
    Tensor out = at::empty({B, H * f, W * f, D}, field.options());
    if (!enqueue(field, [&](void *stream) {
            return matchattn_upsample_field(data(field), data(mask), data(out), B, H, W, D, f, dtype_code(field), stream);
        }))
        return nullptr;
    return THPVariable_Wrap(out);
}

// stereo_volume(correlation) -> [2B, W, H, W]
PyObject *stereo_volume(PyObject *const *a, Py_ssize_t n)
{
    Tensor corr;
    if (n != 1 || !eager() || !cuda_tensor(a[0], corr) || dtype_code(corr) < 0 || corr.dim() != 4 || corr.size(2) != corr.size(3))
        return not_covered();
    corr = corr.contiguous();
    const int64_t B = corr.size(0), H = corr.size(1), W = corr.size(2);
    Tensor vol = at::empty({2 * B, W, H, W}, corr.options());
    if (!enqueue(corr, [&](void *stream) { return matchattn_stereo_volume(data(corr), data(vol), B, H, W, dtype_code(corr), stream); }))
        return nullptr;
    return THPVariable_Wrap(vol);
}

// consistency_mask(field, threshold) -> [B, H, W, 1]
PyObject *consistency_mask(PyObject *const *a, Py_ssize_t n)
{
    Tensor field;
    double threshold;
    if (n != 2 || !to_float(a[1], threshold) || !eager() || !cuda_tensor(a[0], field) || dtype_code(field) < 0 || field.dim() != 4 ||
        field.size(3) != 2 || field.size(0) % 2 != 0)
        return not_covered();
    field = field.contiguous();
    const int64_t B = field.size(0), H = field.size(1), W = field.size(2);
    Tensor mask = at::empty({B, H, W, 1}, field.options());
    if (!enqueue(field, [&](void *stream) {
            return matchattn_consistency_mask(data(field), data(mask), nullptr, B, H, W, static_cast<float>(threshold), dtype_code(field), stream);
        }))
        return nullptr;
    return THPVariable_Wrap(mask);
}

// local_disparity(volume) -> [B, H, W, 2]
PyObject *local_disparity(PyObject *const *a, Py_ssize_t n)
{
    Tensor vol;
    if (n != 1 || !eager() || !cuda_tensor(a[0], vol) || dtype_code(vol) < 0 || vol.dim() != 4 || vol.size(0) % 2 != 0 || vol.size(1) < 5)
        return not_covered();
    vol = vol.contiguous();
    const int64_t B = vol.size(0), D = vol.size(1), H = vol.size(2), W = vol.size(3);
    Tensor flow = at::empty({B, H, W, 2}, vol.options());
    if (!enqueue(vol, [&](void *stream) {
            return matchattn_local_disparity(data(vol), data(flow), nullptr, nullptr, B, D, H, W, dtype_code(vol), stream);
        }))
        return nullptr;
    return THPVariable_Wrap(flow);
}

// flow_init(correlation, H, W) -> (flow [2B, H, W, 2], prob [2B, H, W, N])
PyObject *flow_init(PyObject *const *a, Py_ssize_t n)
{
    Tensor corr;
    int64_t H, W;
    if (n != 3 || !to_int(a[1], H) || !to_int(a[2], W) || H <= 0 || W <= 0 || !eager() || !cuda_tensor(a[0], corr) || dtype_code(corr) < 0 ||
        corr.dim() != 3 || corr.size(1) != H * W || corr.size(2) != H * W)
        return not_covered();
    corr = corr.contiguous();
    const int64_t B = corr.size(0), N = H * W;
    Tensor prob = at::empty({2 * B, H, W, N}, corr.options()), flow = at::empty({2 * B, H, W, 2}, corr.options());
    const int64_t bytes = static_cast<int64_t>(matchattn_flow_init_scratch_bytes(B, H, W));
    Tensor scratch = at::empty({bytes}, corr.options().dtype(at::kByte));
    if (!enqueue(corr, [&](void *stream) {
            return matchattn_flow_init(data(corr), data(prob), data(flow), nullptr, nullptr, data(scratch), bytes, B, H, W, dtype_code(corr), stream);
        }))
        return nullptr;
    return Py_BuildValue("(NN)", THPVariable_Wrap(flow), THPVariable_Wrap(prob));
}

#define MA_ENTRY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MA_ENTRY(module_forward),   MA_ENTRY(autograd),        MA_ENTRY(launch),    MA_ENTRY(cross_core), MA_ENTRY(self_core),
                         MA_ENTRY(upsample_field),   MA_ENTRY(stereo_volume),   MA_ENTRY(consistency_mask), MA_ENTRY(local_disparity),
                         MA_ENTRY(flow_init),        {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }

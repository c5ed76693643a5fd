// The eager call path in native code: checks, allocation, autograd and the call of the C ABI in
// one step, for plain CUDA tensors outside any tracing or transform.
//
// What bounds a small call is not the GPU but the host's way to the launch.  Measured on B200's
// host with a decoder layer's shapes (300 queries): through the Python operators (checks,
// dispatcher, autograd.Function in Python, ctypes) a forward call took 69 us and forward +
// backward 256-270 us, of which the kernels run 6 and 45.
//
// deformops_b200/registry/msda.py tries this path first.  It answers None, and has done nothing,
// whenever a call is anything but the ordinary one - fake or subclassed tensors, dispatch or
// function modes, functorch, forward-mode AD, float64, operands that need a conversion or that
// are wrong - and the Python operators (deformops_b200/ops.py) take the call as before: they
// are what tracing, transforms and error messages go through.
//
// The C ABI is bound by address (bind()), so that this module and the Python side share the one
// copy of the library that deformops_b200/_loader.py loaded.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>

#include <atomic>
#include <cstdlib>

#include "../../include/msda_b200.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;

struct Abi {
    decltype(&msda_b200_forward) forward = nullptr;
    decltype(&msda_b200_backward) backward = nullptr;
    decltype(&msda_b200_forward_offsets) forward_offsets = nullptr;
    decltype(&msda_b200_backward_offsets) backward_offsets = nullptr;
    decltype(&msda_b200_backward_workspace_bytes) workspace_bytes = nullptr;
    decltype(&msda_b200_last_error) last_error = nullptr;
    decltype(&msda_b200_column_sums) column_sums = nullptr;
    decltype(&msda_b200_column_sums_scratch_bytes) column_sums_scratch_bytes = nullptr;
    decltype(&msda_b200_backward_offsets_workspace_bytes) offsets_workspace_bytes = nullptr;
} abi;

// One call: the operands as the kernels take them.  `ref` is undefined when `points` holds
// locations, else `points` holds predicted offsets.
struct Call {
    const Tensor &value, &shapes, &starts, &ref, &points, &attn;
    bool softmax;
    int64_t B, S, G, D, Q, L, K;

    Call(const Tensor &value_, const Tensor &shapes_, const Tensor &starts_, const Tensor &ref_,
         const Tensor &points_, const Tensor &attn_, bool softmax_)
        : value(value_), shapes(shapes_), starts(starts_), ref(ref_), points(points_), attn(attn_),
          softmax(softmax_), B(value.size(0)), S(value.size(1)), G(value.size(2)), D(value.size(3)),
          Q(points.size(1)), L(points.size(3)), K(points.size(4)) {}
};

int dtype_code(at::ScalarType t) {
    return t == at::kFloat      ? MSDA_B200_F32
           : t == at::kHalf     ? MSDA_B200_F16
           : t == at::kBFloat16 ? MSDA_B200_BF16
                                : -1;
}

void check_status(int status, const char *what) {
    if (status == MSDA_B200_OK) return;
    TORCH_CHECK_VALUE(status != MSDA_B200_INVALID_ARGUMENT && status != MSDA_B200_UNSUPPORTED, what,
                      " failed with status ", status, ": ", abi.last_error());
    TORCH_CHECK(false, what, " failed with status ", status, ": ", abi.last_error());
}

// torch allocations are 512-byte aligned; only an offset view can break 16-byte alignment
Tensor aligned(const Tensor &t) {
    return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0
               ? t
               : t.clone(at::MemoryFormat::Contiguous);
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device &device) {
    return Tensor(at::detail::empty_cuda(size, type, device, std::nullopt));
}

Tensor run_forward(const Call &c) {
    RECORD_FUNCTION(c.ref.defined() ? "deformops_b200::msda_offsets_forward"
                                    : (c.softmax ? "deformops_b200::msda_softmax_forward"
                                                 : "deformops_b200::msda_forward"),
                    std::vector<c10::IValue>());
    const at::Device device = c.value.device();
    const c10::cuda::CUDAGuard on_device(device);
    const int dtype = dtype_code(c.value.scalar_type());
    const Tensor value = aligned(c.value), points = aligned(c.points), attn = aligned(c.attn);
    Tensor out = empty({c.B, c.Q, c.G * c.D}, c.value.scalar_type(), device);
    void *stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    const auto *shapes = static_cast<const int64_t *>(c.shapes.const_data_ptr());
    const auto *starts = static_cast<const int64_t *>(c.starts.const_data_ptr());
    int st;
    if (c.ref.defined()) {
        const Tensor ref = aligned(c.ref);
        st = abi.forward_offsets(value.const_data_ptr(), shapes, starts,
                                 static_cast<const float *>(ref.const_data_ptr()), (int)ref.size(3),
                                 points.const_data_ptr(), dtype_code(points.scalar_type()),
                                 attn.const_data_ptr(), out.mutable_data_ptr(), c.B, c.S, c.G, c.D, c.Q,
                                 c.L, c.K, dtype, c.softmax, device.index(), stream);
    } else {
        st = abi.forward(value.const_data_ptr(), shapes, starts,
                         static_cast<const float *>(points.const_data_ptr()), attn.const_data_ptr(),
                         out.mutable_data_ptr(), c.B, c.S, c.G, c.D, c.Q, c.L, c.K, dtype, c.softmax,
                         device.index(), stream);
    }
    check_status(st, c.ref.defined() ? "msda_b200_forward_offsets" : "msda_b200_forward");
    return out;
}

// (grad_value, grad of the points, grad_attn)
variable_list run_backward(const Call &c, const Tensor &grad_in) {
    RECORD_FUNCTION(c.ref.defined() ? "deformops_b200::msda_offsets_backward"
                                    : (c.softmax ? "deformops_b200::msda_softmax_backward"
                                                 : "deformops_b200::msda_backward"),
                    std::vector<c10::IValue>());
    const at::Device device = c.value.device();
    const c10::cuda::CUDAGuard on_device(device);
    const int dtype = dtype_code(c.value.scalar_type());
    const Tensor value = aligned(c.value), points = aligned(c.points), attn = aligned(c.attn);
    const Tensor grad_out = aligned(grad_in.to(c.value.scalar_type()).contiguous());
    Tensor grad_value = empty(c.value.sizes(), c.value.scalar_type(), device);
    Tensor grad_points = empty(c.points.sizes(), c.points.scalar_type(), device);
    Tensor grad_attn = empty(c.attn.sizes(), c.attn.scalar_type(), device);
    const int64_t nbytes = (c.ref.defined() ? abi.offsets_workspace_bytes : abi.workspace_bytes)(
        c.B, c.S, c.G, c.D, c.Q, c.L, c.K, dtype, c.softmax);
    Tensor scratch;
    if (nbytes > 0) scratch = empty({nbytes}, at::kByte, device);
    void *scratch_ptr = nbytes > 0 ? scratch.mutable_data_ptr() : nullptr;
    void *stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    const auto *shapes = static_cast<const int64_t *>(c.shapes.const_data_ptr());
    const auto *starts = static_cast<const int64_t *>(c.starts.const_data_ptr());
    int st;
    if (c.ref.defined()) {
        const Tensor ref = aligned(c.ref);
        st = abi.backward_offsets(value.const_data_ptr(), shapes, starts,
                                  static_cast<const float *>(ref.const_data_ptr()), (int)ref.size(3),
                                  points.const_data_ptr(), dtype_code(points.scalar_type()),
                                  attn.const_data_ptr(), grad_out.const_data_ptr(),
                                  grad_value.mutable_data_ptr(), grad_points.mutable_data_ptr(),
                                  grad_attn.mutable_data_ptr(), scratch_ptr, nbytes, 0, c.B, c.S, c.G,
                                  c.D, c.Q, c.L, c.K, dtype, c.softmax, 1, device.index(), stream);
    } else {
        st = abi.backward(value.const_data_ptr(), shapes, starts,
                          static_cast<const float *>(points.const_data_ptr()), attn.const_data_ptr(),
                          grad_out.const_data_ptr(), grad_value.mutable_data_ptr(),
                          static_cast<float *>(grad_points.mutable_data_ptr()),
                          grad_attn.mutable_data_ptr(), scratch_ptr, nbytes, 0, c.B, c.S, c.G, c.D, c.Q,
                          c.L, c.K, dtype, c.softmax, 1, device.index(), stream);
    }
    check_status(st, c.ref.defined() ? "msda_b200_backward_offsets" : "msda_b200_backward");
    return {grad_value, grad_points, grad_attn};
}

// The autograd formula; differentiable once, like the Python one.
template <bool SOFTMAX>
struct MsdaFunction : torch::autograd::Function<MsdaFunction<SOFTMAX>> {
    static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &value, const Tensor &shapes,
                          const Tensor &starts, const std::optional<Tensor> &maybe_ref,
                          const Tensor &points, const Tensor &attn) {
        const Tensor ref = maybe_ref.value_or(Tensor());
        ctx->save_for_backward({value, shapes, starts, ref, points, attn});
        ctx->set_materialize_grads(false);
        at::AutoDispatchBelowADInplaceOrView below;
        return run_forward(Call(value, shapes, starts, ref, points, attn, SOFTMAX));
    }
    static variable_list backward(torch::autograd::AutogradContext *ctx, const variable_list &grads) {
        if (!grads[0].defined()) return variable_list(6);
        const variable_list saved = ctx->get_saved_variables();
        variable_list out;
        {
            at::AutoDispatchBelowADInplaceOrView below;
            out = run_backward(
                Call(saved[0], saved[1], saved[2], saved[3], saved[4], saved[5], SOFTMAX), grads[0]);
        }
        if (at::GradMode::is_enabled() && grads[0].requires_grad()) {
            for (Tensor &t : out) t.requires_grad_(true);
            torch::autograd::DelayedError once(
                "trying to differentiate twice a function that was marked with @once_differentiable",
                (int64_t)out.size());
            out = once.apply(std::move(out));
        }
        return {out[0], Tensor(), Tensor(), Tensor(), out[1], out[2]};
    }
};

// ---- projections with a bias gradient of our own ------------------------------------------------
Tensor column_sums(const Tensor &x) {
    const at::Device device = x.device();
    const c10::cuda::CUDAGuard on_device(device);
    Tensor out = empty({x.size(1)}, x.scalar_type(), device);
    Tensor scratch = empty({abi.column_sums_scratch_bytes(x.size(0), x.size(1))}, at::kByte, device);
    check_status(abi.column_sums(x.const_data_ptr(), out.mutable_data_ptr(), scratch.mutable_data_ptr(),
                                 x.size(0), x.size(1), dtype_code(x.scalar_type()),
                                 c10::cuda::getCurrentCUDAStream(device.index()).stream()),
                 "msda_b200_column_sums");
    return out;
}

Tensor bias_gradient(const Tensor &g) {
    // a graph of the gradients needs an operator that has a derivative itself
    return at::GradMode::is_enabled() && g.requires_grad() ? g.sum(0) : column_sums(g.contiguous());
}

// y = x W^T + b for each of one or two (W, b); the gradients of x meet in one tensor
struct LinearFunction : torch::autograd::Function<LinearFunction> {
    static variable_list forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &w0,
                                 const Tensor &b0, const std::optional<Tensor> &w1,
                                 const std::optional<Tensor> &b1) {
        ctx->save_for_backward({x, w0, w1.value_or(Tensor())});
        ctx->set_materialize_grads(false);
        at::AutoDispatchBelowADInplaceOrView below;
        variable_list out = {at::linear(x, w0, b0)};
        if (w1) out.push_back(at::linear(x, *w1, *b1));
        return out;
    }
    static variable_list backward(torch::autograd::AutogradContext *ctx, const variable_list &grads) {
        const variable_list saved = ctx->get_saved_variables();
        const Tensor &x = saved[0];
        const Tensor rows = x.reshape({-1, x.size(-1)});
        variable_list out(5);
        for (size_t i = 0; i < grads.size(); ++i) {
            if (!grads[i].defined()) continue;
            const Tensor &w = saved[1 + i];
            const Tensor g = grads[i].reshape({-1, grads[i].size(-1)});
            if (ctx->needs_input_grad(0)) {
                if (!out[0].defined())
                    out[0] = at::mm(g, w);
                else
                    out[0] = at::GradMode::is_enabled() ? at::addmm(out[0], g, w) : out[0].addmm_(g, w);
            }
            if (ctx->needs_input_grad(1 + 2 * i)) out[1 + 2 * i] = at::mm(g.t(), rows);
            if (ctx->needs_input_grad(2 + 2 * i)) out[2 + 2 * i] = bias_gradient(g);
        }
        if (out[0].defined()) out[0] = out[0].view(x.sizes());
        return out;
    }
};

// ---- acceptance ------------------------------------------------------------------------------
bool plain_thread_state() {
    if (at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
        torch::jit::tracer::isTracing())
        return false;
    // anything beyond what an eager thread includes (Python, functorch, functionalization, ...)
    const c10::DispatchKeySet usual({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView});
    return (c10::impl::tls_local_dispatch_key_set().included_ - usual).empty();
}

bool plain_tensor(const Tensor &t, const at::Device &device) {
    static const c10::DispatchKeySet unusual(
        {c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::FuncTorchBatched,
         c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Batched, c10::DispatchKey::Functionalize,
         c10::DispatchKey::Conjugate, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
    return t.defined() && t.is_cuda() && t.device() == device && t.layout() == at::kStrided &&
           !t.key_set().has_any(unusual) && !torch::autograd::isFwGradDefined(t);
}

bool supported_device(const at::Device &device) {
    // compute capability 10.x only; asked once per device
    static std::atomic<int> known[64];
    const int i = device.index();
    if (i < 0 || i >= 64) return false;
    int state = known[i].load(std::memory_order_relaxed);
    if (state == 0) {
        state = at::cuda::getDeviceProperties(i)->major == 10 ? 1 : 2;
        known[i].store(state, std::memory_order_relaxed);
    }
    return state == 1;
}

// DEFORMOPS_VALIDATE asks for checks that read the level table: those live on the Python side
bool validation_asked() {
    const char *v = std::getenv("DEFORMOPS_VALIDATE");
    return v != nullptr && v[0] != '\0' && !(v[0] == '0' && v[1] == '\0');
}

// The same conditions as check_msda_call and unsupported_reason of the Python side, for the
// forms that need no conversion.
bool acceptable(const Tensor &value, const Tensor &shapes, const Tensor &starts, const Tensor &points,
                const Tensor &attn) {
    if (value.dim() != 4 || points.dim() != 6 || (attn.dim() != 4 && attn.dim() != 5)) return false;
    const int dtype = dtype_code(value.scalar_type());
    if (dtype < 0 || attn.scalar_type() != value.scalar_type()) return false;
    const int64_t B = value.size(0), G = value.size(2), D = value.size(3), Q = points.size(1),
                  L = points.size(3), K = points.size(4);
    if (value.numel() == 0 || points.numel() == 0 || L > 16) return false;
    if (D % (dtype == MSDA_B200_F32 ? 4 : 8) != 0) return false;
    if (points.size(0) != B || points.size(2) != G || points.size(5) != 2) return false;
    if (attn.size(0) != B || attn.size(1) != Q || attn.size(2) != G) return false;
    if (attn.dim() == 4 ? attn.size(3) != L * K : (attn.size(3) != L || attn.size(4) != K)) return false;
    return shapes.scalar_type() == at::kLong && starts.scalar_type() == at::kLong && shapes.dim() == 2 &&
           starts.dim() == 1 && shapes.size(0) == L && shapes.size(1) == 2 && starts.size(0) == L &&
           shapes.is_contiguous() && starts.is_contiguous();
}

Tensor differentiable_call(const Tensor &value_in, const Tensor &shapes, const Tensor &starts,
                           const Tensor &ref_in, const Tensor &points_in, const Tensor &attn_in,
                           bool softmax) {
    const Tensor value = value_in.contiguous(), points = points_in.contiguous(), attn = attn_in.contiguous();
    const Tensor ref = ref_in.defined() ? ref_in.contiguous() : ref_in;
    if (at::GradMode::is_enabled() &&
        !c10::impl::tls_is_dispatch_key_excluded(c10::DispatchKey::AutogradCUDA) &&
        (value.requires_grad() || points.requires_grad() || attn.requires_grad())) {
        const std::optional<Tensor> maybe_ref = ref.defined() ? std::optional<Tensor>(ref) : std::nullopt;
        return softmax ? MsdaFunction<true>::apply(value, shapes, starts, maybe_ref, points, attn)
                       : MsdaFunction<false>::apply(value, shapes, starts, maybe_ref, points, attn);
    }
    at::AutoDispatchBelowADInplaceOrView below;
    return run_forward(Call(value, shapes, starts, ref, points, attn, softmax));
}

bool all_plain(PyObject *const *args, Py_ssize_t n) {
    for (Py_ssize_t i = 0; i < n; ++i)
        if (!THPVariable_CheckExact(args[i])) return false;
    return true;
}

// msda(value, spatial_shapes, level_start_index, locations, weights, softmax) -> Tensor | None
PyObject *py_msda(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 6, "msda takes six arguments");
    if (abi.forward == nullptr || !all_plain(args, 5) || !plain_thread_state() || validation_asked())
        Py_RETURN_NONE;
    const Tensor &value = THPVariable_Unpack(args[0]), &shapes = THPVariable_Unpack(args[1]),
                 &starts = THPVariable_Unpack(args[2]), &points = THPVariable_Unpack(args[3]),
                 &attn = THPVariable_Unpack(args[4]);
    const at::Device device = value.device();
    for (const Tensor *t : {&value, &shapes, &starts, &points, &attn})
        if (!plain_tensor(*t, device)) Py_RETURN_NONE;
    if (points.scalar_type() != at::kFloat || !supported_device(device) ||
        !acceptable(value, shapes, starts, points, attn))
        Py_RETURN_NONE;
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = differentiable_call(value, shapes, starts, Tensor(), points, attn, args[5] == Py_True);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// msda_offsets(value, spatial_shapes, level_start_index, reference_points, offsets, weights,
//              softmax) -> Tensor | None
PyObject *py_msda_offsets(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 7, "msda_offsets takes seven arguments");
    if (abi.forward == nullptr || !all_plain(args, 6) || !plain_thread_state() || validation_asked())
        Py_RETURN_NONE;
    const Tensor &value = THPVariable_Unpack(args[0]), &shapes = THPVariable_Unpack(args[1]),
                 &starts = THPVariable_Unpack(args[2]), &ref = THPVariable_Unpack(args[3]),
                 &points = THPVariable_Unpack(args[4]), &attn = THPVariable_Unpack(args[5]);
    const at::Device device = value.device();
    for (const Tensor *t : {&value, &shapes, &starts, &ref, &points, &attn})
        if (!plain_tensor(*t, device)) Py_RETURN_NONE;
    if (!supported_device(device) || !acceptable(value, shapes, starts, points, attn)) Py_RETURN_NONE;
    if (points.scalar_type() != at::kFloat && points.scalar_type() != value.scalar_type()) Py_RETURN_NONE;
    // a gradient of the reference points, or their conversion, is formed on the Python side
    if (ref.dim() != 4 || ref.scalar_type() != at::kFloat || ref.requires_grad() ||
        ref.size(0) != points.size(0) || ref.size(1) != points.size(1) || ref.size(2) != points.size(3) ||
        (ref.size(3) != 2 && ref.size(3) != 4))
        Py_RETURN_NONE;
    Tensor out;
    {
        pybind11::gil_scoped_release no_gil;
        out = differentiable_call(value, shapes, starts, ref, points, attn, args[6] == Py_True);
    }
    return THPVariable_Wrap(std::move(out));
    END_HANDLE_TH_ERRORS
}

// Below this many rows torch's own reduction is as quick and its call shorter.
constexpr int64_t kLinearRows = 2048;

bool linear_acceptable(const Tensor &x, const Tensor &w, const Tensor &b) {
    return w.dim() == 2 && b.dim() == 1 && w.size(1) == x.size(-1) && b.size(0) == w.size(0) &&
           w.scalar_type() == x.scalar_type() && b.scalar_type() == x.scalar_type();
}

// linear(x, weight, bias) -> Tensor | None;
// linear_pair(x, weight, bias, weight, bias) -> (Tensor, Tensor) | None
template <int N>
PyObject *py_linear(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 1 + 2 * N, "wrong number of arguments");
    if (abi.forward == nullptr || !all_plain(args, nargs) || !plain_thread_state() ||
        !at::GradMode::is_enabled() || at::autocast::is_autocast_enabled(at::kCUDA) ||
        c10::impl::tls_is_dispatch_key_excluded(c10::DispatchKey::AutogradCUDA))
        Py_RETURN_NONE;
    const Tensor &x = THPVariable_Unpack(args[0]);
    const at::Device device = x.device();
    bool grad = false;
    for (Py_ssize_t i = 0; i < nargs; ++i) {
        const Tensor &t = THPVariable_Unpack(args[i]);
        if (!plain_tensor(t, device)) Py_RETURN_NONE;
        grad = grad || t.requires_grad();
    }
    if (!grad || dtype_code(x.scalar_type()) < 0 || x.dim() < 2 || !x.is_contiguous() || x.size(-1) == 0 ||
        x.numel() / x.size(-1) < kLinearRows || !supported_device(device))
        Py_RETURN_NONE;
    for (int i = 0; i < N; ++i)
        if (!linear_acceptable(x, THPVariable_Unpack(args[1 + 2 * i]), THPVariable_Unpack(args[2 + 2 * i])))
            Py_RETURN_NONE;
    variable_list out;
    {
        pybind11::gil_scoped_release no_gil;
        std::optional<Tensor> w1, b1;
        if constexpr (N == 2) w1 = THPVariable_Unpack(args[3]), b1 = THPVariable_Unpack(args[4]);
        out = LinearFunction::apply(x, THPVariable_Unpack(args[1]), THPVariable_Unpack(args[2]), w1, b1);
    }
    if constexpr (N == 1) return THPVariable_Wrap(std::move(out[0]));
    THPObjectPtr a(THPVariable_Wrap(std::move(out[0]))), b(THPVariable_Wrap(std::move(out[N - 1])));
    if (!a || !b) return nullptr;
    return PyTuple_Pack(2, a.get(), b.get());
    END_HANDLE_TH_ERRORS
}

// bind(addresses of the ABI functions in the order of struct Abi)
PyObject *py_bind(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    HANDLE_TH_ERRORS
    TORCH_CHECK(nargs == 9, "bind takes nine addresses");
    void *p[9];
    for (int i = 0; i < 9; ++i) {
        p[i] = PyLong_AsVoidPtr(args[i]);
        if (p[i] == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null address");
            return nullptr;
        }
    }
    abi.backward = reinterpret_cast<decltype(abi.backward)>(p[1]);
    abi.forward_offsets = reinterpret_cast<decltype(abi.forward_offsets)>(p[2]);
    abi.backward_offsets = reinterpret_cast<decltype(abi.backward_offsets)>(p[3]);
    abi.workspace_bytes = reinterpret_cast<decltype(abi.workspace_bytes)>(p[4]);
    abi.last_error = reinterpret_cast<decltype(abi.last_error)>(p[5]);
    abi.column_sums = reinterpret_cast<decltype(abi.column_sums)>(p[6]);
    abi.column_sums_scratch_bytes = reinterpret_cast<decltype(abi.column_sums_scratch_bytes)>(p[7]);
    abi.offsets_workspace_bytes = reinterpret_cast<decltype(abi.offsets_workspace_bytes)>(p[8]);
    abi.forward = reinterpret_cast<decltype(abi.forward)>(p[0]);
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

template <typename F>
PyCFunction as_method(F f) {
    return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f));
}

PyMethodDef methods[] = {
    {"msda", as_method(py_msda), METH_FASTCALL, nullptr},
    {"msda_offsets", as_method(py_msda_offsets), METH_FASTCALL, nullptr},
    {"linear", as_method(py_linear<1>), METH_FASTCALL, nullptr},
    {"linear_pair", as_method(py_linear<2>), METH_FASTCALL, nullptr},
    {"bind", as_method(py_bind), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "msda_b200_host", nullptr, -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_msda_b200_host() { return PyModule_Create(&module); }

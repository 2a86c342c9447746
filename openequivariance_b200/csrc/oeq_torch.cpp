// The operators as torch library ops with native kernels: checks, output allocation, launch and autograd without
// the interpreter.  A call through Python kernels cost 30 us forward and 100 us more for a backward pass, several
// times what the GPU needs for a small molecule.
//
// Every operator object registers its own ops (as the reference does, openequivariance/implementations/
// TensorProductBase.py:236-298): a forward op, a gradient op that returns the list of input gradients, both
// differentiable.  All arguments are tensors: `inputs` operands, for the gradient op the output gradient, then the
// index arrays of a convolution, so that one boxed kernel serves every operator.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <atomic>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/oeq_b200.h"

namespace {

using at::Tensor;
using c10::OperatorHandle;
using c10::Stack;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Op {
    oeq_tp* tp = nullptr;
    oeq_conv* conv = nullptr;
    bool deterministic = false, shared = false;
    int inputs = 3;                 // x, y, w; a convolution whose weights are all 1 has no w
    int index = 0;                  // rows, cols[, sender order]
    int64_t x_dim = 0, y_dim = 0, z_dim = 0, w_numel = 0;
    at::ScalarType dtype = at::kFloat;
    std::optional<OperatorHandle> forward, gradient, second;
    std::atomic<bool> call_second{false};   // the caller replaced the fused second derivatives by the op `second`
    std::mutex mutex;
    std::vector<Tensor> scratch;    // large backward scratch, per device
};

void check(int rc) { TORCH_CHECK(rc == OEQ_OK, "oeq_b200: ", oeq_last_error()); }

// Argument i of the n on top of the stack.
const Tensor& arg(const Stack& stack, int n, int i) { return stack[stack.size() - n + i].toTensor(); }

void check_inputs(const Op& op, const Stack& stack, int n) {
    for (int i = 0; i < n; ++i)
        TORCH_CHECK(arg(stack, n, i).is_cuda(), "openequivariance_b200 runs on CUDA tensors only (there is no CPU fallback)");
    const Tensor &x = arg(stack, n, 0), &y = arg(stack, n, 1);
    TORCH_CHECK_VALUE(x.dim() == 2 && x.size(1) == op.x_dim, op.conv ? "node features must be [nodes, " : "first input must be [batch, ",
                      op.x_dim, "], got ", x.sizes());
    int64_t rows_n = x.size(0);
    if (op.conv) {
        const Tensor &rows = arg(stack, n, n - op.index), &cols = arg(stack, n, n - op.index + 1);
        TORCH_CHECK_VALUE(rows.dim() == 1 && cols.sizes() == rows.sizes(), "rows and cols must be 1-D and of equal length");
        TORCH_CHECK_VALUE(rows.scalar_type() == at::kLong && cols.scalar_type() == at::kLong, "rows and cols must be int64");
        rows_n = rows.size(0);
        if (op.deterministic) {
            const Tensor& perm = arg(stack, n, n - 1);
            TORCH_CHECK_VALUE(perm.sizes() == rows.sizes() && perm.scalar_type() == at::kLong, "sender_perm must be int64 and as long as rows");
        }
    }
    TORCH_CHECK_VALUE(y.dim() == 2 && y.size(0) == rows_n && y.size(1) == op.y_dim, op.conv ? "edge features must be [" : "second input must be [",
                      rows_n, ", ", op.y_dim, "], got ", y.sizes());
    TORCH_CHECK_VALUE(x.scalar_type() == op.dtype && y.scalar_type() == op.dtype, "tensors must be ", op.dtype);
    if (op.inputs == 3) {
        const Tensor& w = arg(stack, n, 2);
        TORCH_CHECK_VALUE(op.shared ? (w.dim() == 1 && w.size(0) == op.w_numel) : (w.dim() == 2 && w.size(0) == rows_n && w.size(1) == op.w_numel),
                          "weights must be [", op.shared ? "" : std::to_string(rows_n) + ", ", op.w_numel, "], got ", w.sizes());
        TORCH_CHECK_VALUE(w.scalar_type() == op.dtype, "tensors must be ", op.dtype);
    }
}

const int64_t* index_ptr(const Tensor& t) { return static_cast<const int64_t*>(t.const_data_ptr()); }

// ---------------------------------------------------------------- CUDA kernels

struct ForwardKernel final : c10::OperatorKernel {
    Op* op;
    explicit ForwardKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle&, c10::DispatchKeySet, Stack* stack) {
        const int n = op->inputs + op->index;
        check_inputs(*op, *stack, n);
        const Tensor x = arg(*stack, n, 0).contiguous(), y = arg(*stack, n, 1).contiguous();
        const Tensor w = op->inputs == 3 ? arg(*stack, n, 2).contiguous() : Tensor();
        const void* wp = op->inputs == 3 ? w.const_data_ptr() : nullptr;
        c10::cuda::CUDAGuard guard(x.device());
        Tensor z = at::empty({x.size(0), op->z_dim}, x.options());
        void* st = c10::cuda::getCurrentCUDAStream().stream();
        if (op->tp) {
            check(oeq_tp_forward(op->tp, x.size(0), x.const_data_ptr(), y.const_data_ptr(), wp, z.mutable_data_ptr(), st));
        } else {
            const Tensor rows = arg(*stack, n, op->inputs).contiguous(), cols = arg(*stack, n, op->inputs + 1).contiguous();
            check(oeq_conv_forward(op->conv, x.size(0), rows.size(0), x.const_data_ptr(), y.const_data_ptr(), wp, index_ptr(rows),
                                   index_ptr(cols), z.mutable_data_ptr(), nullptr, 0, st));
        }
        torch::jit::drop(*stack, n);
        stack->emplace_back(std::move(z));
    }
};

// Scratch of the deterministic backward pass.  Up to 256 MB come from the caching allocator call by call, safe with
// any number of streams; more is kept on the operator (allocating it again and again would flush a full device's
// cache): a quarter of it when the device cannot spare the whole, none when not even that.
Tensor backward_scratch(Op& op, int64_t nodes, int64_t edges, const at::TensorOptions& options) {
    const size_t want = oeq_conv_workspace_bytes(op.conv, nodes, edges);
    if (want == 0) return Tensor();
    const auto bytes = options.dtype(at::kByte);
    if (want <= (256u << 20)) return at::empty({(int64_t)want}, bytes);
    const size_t device = (size_t)options.device().index();
    std::lock_guard<std::mutex> lock(op.mutex);
    if (op.scratch.size() <= device) op.scratch.resize(device + 1);
    Tensor& kept = op.scratch[device];
    if (kept.defined() && (size_t)kept.numel() >= want) return kept;
    kept = Tensor();
    for (size_t size : {want, want / 4}) {
        try {
            kept = at::empty({(int64_t)size}, bytes);
            break;
        } catch (const c10::OutOfMemoryError&) {
        }
    }
    return kept;
}

struct GradientKernel final : c10::OperatorKernel {
    Op* op;
    explicit GradientKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle&, c10::DispatchKeySet, Stack* stack) {
        const int n = op->inputs + 1 + op->index;
        check_inputs(*op, *stack, n);
        const Tensor x = arg(*stack, n, 0).contiguous(), y = arg(*stack, n, 1).contiguous();
        const Tensor w = op->inputs == 3 ? arg(*stack, n, 2).contiguous() : Tensor();
        const Tensor dz = arg(*stack, n, op->inputs).contiguous();
        TORCH_CHECK_VALUE(dz.dim() == 2 && dz.size(0) == x.size(0) && dz.size(1) == op->z_dim && dz.scalar_type() == op->dtype,
                          "output gradient must be [", x.size(0), ", ", op->z_dim, "] of ", op->dtype, ", got ", dz.sizes());
        c10::cuda::CUDAGuard guard(x.device());
        Tensor dx = at::empty_like(x), dy = at::empty_like(y), dw = op->inputs == 3 ? at::empty_like(w) : Tensor();
        const void* wp = op->inputs == 3 ? w.const_data_ptr() : nullptr;
        void* dwp = op->inputs == 3 ? dw.mutable_data_ptr() : nullptr;
        void* st = c10::cuda::getCurrentCUDAStream().stream();
        Tensor ws;
        if (op->tp) {
            const size_t bytes = oeq_tp_workspace_bytes(op->tp, x.size(0));
            if (bytes) ws = at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
            check(oeq_tp_backward(op->tp, x.size(0), x.const_data_ptr(), y.const_data_ptr(), wp, dz.const_data_ptr(), dx.mutable_data_ptr(),
                                  dy.mutable_data_ptr(), dwp, bytes ? ws.mutable_data_ptr() : nullptr, bytes, st));
        } else {
            const Tensor rows = arg(*stack, n, op->inputs + 1).contiguous(), cols = arg(*stack, n, op->inputs + 2).contiguous();
            const Tensor perm = op->deterministic ? arg(*stack, n, op->inputs + 3).contiguous() : Tensor();
            ws = op->deterministic ? backward_scratch(*op, x.size(0), rows.size(0), x.options()) : Tensor();
            check(oeq_conv_backward(op->conv, x.size(0), rows.size(0), x.const_data_ptr(), y.const_data_ptr(), wp, dz.const_data_ptr(),
                                    index_ptr(rows), index_ptr(cols), perm.defined() ? index_ptr(perm) : nullptr, dx.mutable_data_ptr(),
                                    dy.mutable_data_ptr(), dwp, ws.defined() ? ws.mutable_data_ptr() : nullptr,
                                    ws.defined() ? (size_t)ws.numel() : 0, st));
        }
        torch::jit::drop(*stack, n);
        c10::List<Tensor> out;
        out.push_back(std::move(dx));
        out.push_back(std::move(dy));
        if (op->inputs == 3) out.push_back(std::move(dw));
        stack->emplace_back(std::move(out));
    }
};

// Second derivatives of the batch product in one launch (oeq_tp_has_double_backward).
variable_list tp_second(const Op& op, at::ArrayRef<Tensor> in) {
    variable_list c, out;
    for (const Tensor& t : in) c.push_back(t.contiguous());
    c10::cuda::CUDAGuard guard(c[0].device());
    for (int i = 0; i < 4; ++i) out.push_back(at::empty_like(c[i]));
    check(oeq_tp_double_backward(op.tp, c[0].size(0), c[0].const_data_ptr(), c[1].const_data_ptr(), c[2].const_data_ptr(),
                                 c[3].const_data_ptr(), c[4].const_data_ptr(), c[5].const_data_ptr(), c[6].const_data_ptr(),
                                 out[0].mutable_data_ptr(), out[1].mutable_data_ptr(), out[2].mutable_data_ptr(),
                                 out[3].mutable_data_ptr(), c10::cuda::getCurrentCUDAStream().stream()));
    return out;
}

// Second derivatives of the convolution in its fused launches; empty where the library has none here (the caller composes
// them).
variable_list conv_second(Op& op, at::ArrayRef<Tensor> in, at::ArrayRef<Tensor> index) {
    if (!oeq_conv_has_double_backward(op.conv)) return {};
    variable_list c, out, idx;
    for (const Tensor& t : in) c.push_back(t.contiguous());
    for (const Tensor& t : index) idx.push_back(t.contiguous());
    c10::cuda::CUDAGuard guard(c[0].device());
    for (int i = 0; i < 4; ++i) out.push_back(at::empty_like(c[i]));
    const int64_t nodes = c[0].size(0), edges = idx[0].size(0);
    Tensor ws = op.deterministic ? backward_scratch(op, nodes, edges, c[0].options()) : Tensor();
    const int rc = oeq_conv_double_backward(
        op.conv, nodes, edges, c[0].const_data_ptr(), c[1].const_data_ptr(), c[2].const_data_ptr(), c[3].const_data_ptr(),
        c[4].const_data_ptr(), c[5].const_data_ptr(), c[6].const_data_ptr(), index_ptr(idx[0]), index_ptr(idx[1]),
        op.deterministic ? index_ptr(idx[2]) : nullptr, out[0].mutable_data_ptr(), out[1].mutable_data_ptr(), out[2].mutable_data_ptr(),
        out[3].mutable_data_ptr(), ws.defined() ? ws.mutable_data_ptr() : nullptr, ws.defined() ? (size_t)ws.numel() : 0,
        c10::cuda::getCurrentCUDAStream().stream());
    if (rc == OEQ_ERR_UNSUPPORTED) return {};
    check(rc);
    return out;
}

// ---------------------------------------------------------------- autograd

Tensor call_forward(const Op& op, at::ArrayRef<Tensor> in) {
    Stack stack(in.begin(), in.end());
    op.forward->callBoxed(stack);
    return stack.back().toTensor();
}
variable_list call_list(const OperatorHandle& handle, at::ArrayRef<Tensor> in) {
    Stack stack(in.begin(), in.end());
    handle.callBoxed(stack);
    return stack.back().toTensorVector();
}
variable_list joined(std::initializer_list<Tensor> a, at::ArrayRef<Tensor> index) {
    variable_list v(a);
    v.insert(v.end(), index.begin(), index.end());
    return v;
}
// One gradient per forward argument: none for the operator, the given ones, none for the index arrays.
variable_list per_argument(variable_list grads, const Op& op) {
    grads.insert(grads.begin(), Tensor());
    grads.resize(grads.size() + op.index);
    return grads;
}

struct ForwardFn : torch::autograd::Function<ForwardFn> {
    static Tensor forward(AutogradContext* ctx, Op* op, at::TensorList in) {
        ctx->saved_data["op"] = reinterpret_cast<int64_t>(op);
        ctx->save_for_backward(in.vec());
        at::AutoDispatchBelowADInplaceOrView guard;
        return call_forward(*op, in);
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        Op& op = *reinterpret_cast<Op*>(ctx->saved_data["op"].toInt());
        variable_list in = ctx->get_saved_variables();
        in.insert(in.begin() + op.inputs, grads[0]);
        return per_argument(call_list(*op.gradient, in), op);
    }
};

struct GradientFn : torch::autograd::Function<GradientFn> {
    static variable_list forward(AutogradContext* ctx, Op* op, at::TensorList in) {
        ctx->saved_data["op"] = reinterpret_cast<int64_t>(op);
        ctx->save_for_backward(in.vec());
        at::AutoDispatchBelowADInplaceOrView guard;
        return call_list(*op->gradient, in);
    }
    // The product is trilinear in (x, y, w).  With cotangents (ex, ey, ew) of (dX, dY, dW):
    //   d/d(dz) = f(ex, y, w) + f(x, ey, w) + f(x, y, ew);  d/dx = dX(ey, w, dz) + dX(y, ew, dz), likewise y and w.
    static variable_list backward(AutogradContext* ctx, variable_list e) {
        Op& op = *reinterpret_cast<Op*>(ctx->saved_data["op"].toInt());
        const variable_list s = ctx->get_saved_variables();
        const at::ArrayRef<Tensor> idx(s.data() + op.inputs + 1, (size_t)op.index);
        const Tensor &x = s[0], &y = s[1], &dz = s[op.inputs];
        if (op.inputs == 2) {
            variable_list a = call_list(*op.gradient, joined({e[0], e[1], dz}, idx));
            return per_argument({a[0], a[1], call_forward(op, joined({e[0], y}, idx)) + call_forward(op, joined({x, e[1]}, idx))}, op);
        }
        const Tensor& w = s[2];
        if (!at::GradMode::is_enabled()) {
            // nothing differentiates through this result: launches that read a row's arrays once
            if (op.tp && oeq_tp_has_double_backward(op.tp)) return per_argument(tp_second(op, {x, y, w, dz, e[0], e[1], e[2]}), op);
        }
        if (op.conv && !at::GradMode::is_enabled()) {
            variable_list all = op.second && op.call_second ? call_list(*op.second, joined({x, y, w, dz, e[0], e[1], e[2]}, idx))
                                                            : conv_second(op, {x, y, w, dz, e[0], e[1], e[2]}, idx);
            if (all.size() == 4) return per_argument(std::move(all), op);
        }
        variable_list a = call_list(*op.gradient, joined({e[0], e[1], w, dz}, idx));    // dX(ey, w), dY(ex, w)
        variable_list b = call_list(*op.gradient, joined({x, y, e[2], dz}, idx));       // dX(y, ew), dY(x, ew)
        variable_list c = call_list(*op.gradient, joined({e[0], y, w, dz}, idx));       // dW(ex, y)
        variable_list d = call_list(*op.gradient, joined({x, e[1], w, dz}, idx));       // dW(x, ey)
        Tensor gz = call_forward(op, joined({e[0], y, w}, idx)) + call_forward(op, joined({x, e[1], w}, idx)) +
                    call_forward(op, joined({x, y, e[2]}, idx));
        return per_argument({a[0] + b[0], a[1] + b[1], c[2] + d[2], gz}, op);
    }
};

template <bool GRADIENT>
struct AutogradKernel final : c10::OperatorKernel {
    Op* op;
    explicit AutogradKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle& handle, c10::DispatchKeySet keys, Stack* stack) {
        const int diff = op->inputs + (GRADIENT ? 1 : 0), n = diff + op->index;
        bool needed = false;
        if (at::GradMode::is_enabled())
            for (int i = 0; i < diff; ++i) needed |= arg(*stack, n, i).requires_grad();
        if (!needed) {
            at::AutoDispatchBelowADInplaceOrView guard;
            handle.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
            return;
        }
        variable_list in;
        in.reserve(n);
        for (int i = 0; i < n; ++i) in.push_back(arg(*stack, n, i));
        torch::jit::drop(*stack, n);
        if constexpr (GRADIENT) stack->emplace_back(c10::List<Tensor>(GradientFn::apply(op, at::TensorList(in))));
        else stack->emplace_back(ForwardFn::apply(op, at::TensorList(in)));
    }
};

std::deque<torch::Library>& libraries() {
    static auto* l = new std::deque<torch::Library>();      // ops stay registered until the process ends
    return *l;
}
std::map<std::string, Op*>& operators() {       // by the name of their forward op
    static auto* m = new std::map<std::string, Op*>();
    return *m;
}
std::mutex register_mutex;
thread_local std::string register_error;

}  // namespace

extern "C" {

const char* oeq_torch_error() { return register_error.c_str(); }

// Registers the forward op and the gradient op of one operator (`tp` or `conv`) in the namespace
// openequivariance_b200.  `second`: name of an op (registered by the caller) that may replace the fused second
// derivatives (oeq_torch_call_second), or null.
int oeq_torch_register(const char* forward, const char* gradient, const char* second, oeq_tp* tp, oeq_conv* conv, int deterministic,
                       int shared, int has_weights, int f64, int64_t x_dim, int64_t y_dim, int64_t z_dim, int64_t w_numel) {
    try {
        std::lock_guard<std::mutex> lock(register_mutex);
        Op* op = new Op();          // lives as long as the ops
        op->tp = tp;
        op->conv = conv;
        op->deterministic = deterministic != 0;
        op->shared = shared != 0;
        op->inputs = has_weights ? 3 : 2;
        op->index = conv ? (deterministic ? 3 : 2) : 0;
        op->x_dim = x_dim;
        op->y_dim = y_dim;
        op->z_dim = z_dim;
        op->w_numel = w_numel;
        op->dtype = f64 ? at::kDouble : at::kFloat;
        const std::string in = has_weights ? "Tensor L1_in, Tensor L2_in, Tensor weights" : "Tensor L1_in, Tensor L2_in";
        const std::string idx = !conv ? "" : (deterministic ? ", Tensor rows, Tensor cols, Tensor transpose_perm" : ", Tensor rows, Tensor cols");
        const std::string ns = "openequivariance_b200";
        libraries().emplace_back(torch::Library::FRAGMENT, ns, std::nullopt, __FILE__, __LINE__);
        torch::Library& lib = libraries().back();
        lib.def((std::string(forward) + "(" + in + idx + ") -> Tensor").c_str());
        lib.def((std::string(gradient) + "(" + in + ", Tensor L3_grad" + idx + ") -> Tensor[]").c_str());
        auto boxed = [](auto functor) { return torch::CppFunction::makeFromBoxedFunctor(std::move(functor)); };
        lib.impl(forward, torch::dispatch(c10::DispatchKey::CUDA, boxed(std::make_unique<ForwardKernel>(op))));
        lib.impl(gradient, torch::dispatch(c10::DispatchKey::CUDA, boxed(std::make_unique<GradientKernel>(op))));
        lib.impl(forward, torch::dispatch(c10::DispatchKey::Autograd, boxed(std::make_unique<AutogradKernel<false>>(op))));
        lib.impl(gradient, torch::dispatch(c10::DispatchKey::Autograd, boxed(std::make_unique<AutogradKernel<true>>(op))));
        auto& dispatcher = c10::Dispatcher::singleton();
        op->forward = dispatcher.findSchemaOrThrow((ns + "::" + forward).c_str(), "");
        op->gradient = dispatcher.findSchemaOrThrow((ns + "::" + gradient).c_str(), "");
        if (second) op->second = dispatcher.findSchemaOrThrow((ns + "::" + second).c_str(), "");
        operators()[forward] = op;
        return 0;
    } catch (const std::exception& e) {
        register_error = e.what();
        return 1;
    }
}

// Whether the second backward pass of the operator with this forward op calls its op `second` (see oeq_torch_register)
// instead of the library's fused launches.
int oeq_torch_call_second(const char* forward, int call) {
    std::lock_guard<std::mutex> lock(register_mutex);
    auto it = operators().find(forward);
    if (it == operators().end()) return 1;
    it->second->call_second = call != 0;
    return 0;
}

}  // extern "C"

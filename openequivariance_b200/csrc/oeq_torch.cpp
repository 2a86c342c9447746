// The operators as torch library ops with native kernels: checks, output allocation, launch and autograd without
// the interpreter.  A call through Python kernels cost 30 us forward and 100 us more for a backward pass, several
// times what the GPU needs for a small molecule.
//
// Every operator object registers its own ops (as the reference does, openequivariance/implementations/
// TensorProductBase.py:236-298): a forward op, a gradient op that returns the list of input gradients, both
// differentiable.  All arguments are tensors: `inputs` operands, for the gradient op the output gradient, then the
// index arrays of a convolution, so that one boxed kernel serves every operator.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
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
    struct Kept {
        Tensor memory;
        std::optional<c10::cuda::CUDAStream> stream;    // whose work uses it
        size_t wanted = 0;          // size that was asked for (the device may have had less)
    };
    std::mutex mutex;
    std::map<c10::DeviceIndex, Kept> kept;  // large backward scratch
};

void check(int rc) { TORCH_CHECK(rc == OEQ_OK, "oeq_b200: ", oeq_last_error()); }

typedef at::ArrayRef<Tensor> Args;

void check_inputs(const Op& op, Args in) {
    const int n = (int)in.size();
    for (const Tensor& t : in)
        TORCH_CHECK(t.is_cuda(), "openequivariance_b200 runs on CUDA tensors only (there is no CPU fallback)");
    const Tensor &x = in[0], &y = in[1];
    TORCH_CHECK_VALUE(x.dim() == 2 && x.size(1) == op.x_dim, op.conv ? "node features must be [nodes, " : "first input must be [batch, ",
                      op.x_dim, "], got ", x.sizes());
    int64_t rows_n = x.size(0);
    if (op.conv) {
        const Tensor &rows = in[n - op.index], &cols = in[n - op.index + 1];
        TORCH_CHECK_VALUE(rows.dim() == 1 && cols.sizes() == rows.sizes(), "rows and cols must be 1-D and of equal length");
        TORCH_CHECK_VALUE(rows.scalar_type() == at::kLong && cols.scalar_type() == at::kLong, "rows and cols must be int64");
        rows_n = rows.size(0);
        if (op.deterministic) {
            const Tensor& perm = in[n - 1];
            TORCH_CHECK_VALUE(perm.sizes() == rows.sizes() && perm.scalar_type() == at::kLong, "sender_perm must be int64 and as long as rows");
        }
    }
    TORCH_CHECK_VALUE(y.dim() == 2 && y.size(0) == rows_n && y.size(1) == op.y_dim, op.conv ? "edge features must be [" : "second input must be [",
                      rows_n, ", ", op.y_dim, "], got ", y.sizes());
    TORCH_CHECK_VALUE(x.scalar_type() == op.dtype && y.scalar_type() == op.dtype, "tensors must be ", op.dtype);
    if (op.inputs == 3) {
        const Tensor& w = in[2];
        TORCH_CHECK_VALUE(op.shared ? (w.dim() == 1 && w.size(0) == op.w_numel) : (w.dim() == 2 && w.size(0) == rows_n && w.size(1) == op.w_numel),
                          "weights must be [", op.shared ? "" : std::to_string(rows_n) + ", ", op.w_numel, "], got ", w.sizes());
        TORCH_CHECK_VALUE(w.scalar_type() == op.dtype, "tensors must be ", op.dtype);
    }
}

const int64_t* index_ptr(const Tensor& t) { return static_cast<const int64_t*>(t.const_data_ptr()); }

// ---------------------------------------------------------------- CUDA kernels

// Operands x, y[, w], then the index arrays.
Tensor forward_cuda(const Op& op, Args in) {
    check_inputs(op, in);
    const auto x = in[0].expect_contiguous(), y = in[1].expect_contiguous();
    const auto w = in[op.inputs == 3 ? 2 : 0].expect_contiguous();
    const void* wp = op.inputs == 3 ? w->const_data_ptr() : nullptr;
    c10::cuda::CUDAGuard guard(x->device());
    Tensor z = at::empty({x->size(0), op.z_dim}, x->options());
    void* st = c10::cuda::getCurrentCUDAStream().stream();
    if (op.tp) {
        Tensor ws;      // of this call: safe with any number of streams
        const size_t bytes = oeq_tp_forward_workspace_bytes(op.tp);
        if (bytes) ws = at::empty({(int64_t)bytes}, x->options().dtype(at::kByte));
        check(oeq_tp_forward_ws(op.tp, x->size(0), x->const_data_ptr(), y->const_data_ptr(), wp, z.mutable_data_ptr(),
                                bytes ? ws.mutable_data_ptr() : nullptr, bytes, st));
    } else {
        const auto rows = in[op.inputs].expect_contiguous(), cols = in[op.inputs + 1].expect_contiguous();
        check(oeq_conv_forward(op.conv, x->size(0), rows->size(0), x->const_data_ptr(), y->const_data_ptr(), wp, index_ptr(*rows),
                               index_ptr(*cols), z.mutable_data_ptr(), nullptr, 0, st));
    }
    return z;
}

// Memory for the library to use as scratch: a quarter of what it wants when the device cannot spare the whole, none when
// not even that.
Tensor scratch_memory(size_t want, const at::TensorOptions& bytes) {
    for (size_t size : {want, want / 4}) {
        try {
            return at::empty({(int64_t)size}, bytes);
        } catch (const c10::OutOfMemoryError&) {
        }
    }
    return Tensor();
}

// Scratch of the deterministic backward pass, which runs without it too.  Up to 256 MB come from the caching allocator
// call by call; more is kept on the operator (allocating it again and again would flush a full device's cache).  Kept
// memory serves one stream, the last to ask: another stream's call gives it back to the pool of the former one, whose
// allocations come after its pending work, and takes memory of its own.  The lock is held until the launches that use kept
// memory are on the stream, so that the launches of two threads on one stream do not mix.  A captured call, whose graph may
// run at any time on any stream, takes memory from the graph's pool.
struct Scratch {
    std::unique_lock<std::mutex> lock;
    Tensor memory;
    void* data() const { return memory.defined() ? memory.mutable_data_ptr() : nullptr; }
    size_t bytes() const { return memory.defined() ? (size_t)memory.numel() : 0; }
};
Scratch backward_scratch(Op& op, int64_t nodes, int64_t edges, const at::TensorOptions& options) {
    const size_t want = oeq_conv_workspace_bytes(op.conv, nodes, edges);
    if (want == 0) return {};
    const auto bytes = options.dtype(at::kByte);
    if (want <= (256u << 20) || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
        return {{}, scratch_memory(want, bytes)};
    const auto stream = c10::cuda::getCurrentCUDAStream();
    std::unique_lock<std::mutex> lock(op.mutex);
    Op::Kept& kept = op.kept[stream.device_index()];
    const bool enough = kept.memory.defined() && ((size_t)kept.memory.numel() >= want || kept.wanted == want);
    if (!enough || kept.stream != stream) {
        kept.memory = Tensor();
        kept.memory = scratch_memory(want, bytes);
        kept.stream = stream;
        kept.wanted = want;
    }
    return {std::move(lock), kept.memory};
}

// Operands x, y[, w], the output gradient, then the index arrays.
variable_list gradient_cuda(Op& op, Args in) {
    check_inputs(op, in);
    const auto x = in[0].expect_contiguous(), y = in[1].expect_contiguous();
    const auto w = in[op.inputs == 3 ? 2 : 0].expect_contiguous();
    const auto dz = in[op.inputs].expect_contiguous();
    TORCH_CHECK_VALUE(dz->dim() == 2 && dz->size(0) == x->size(0) && dz->size(1) == op.z_dim && dz->scalar_type() == op.dtype,
                      "output gradient must be [", x->size(0), ", ", op.z_dim, "] of ", op.dtype, ", got ", dz->sizes());
    c10::cuda::CUDAGuard guard(x->device());
    variable_list out{at::empty_like(*x), at::empty_like(*y)};
    if (op.inputs == 3) out.push_back(at::empty_like(*w));
    const void* wp = op.inputs == 3 ? w->const_data_ptr() : nullptr;
    void *dxp = out[0].mutable_data_ptr(), *dyp = out[1].mutable_data_ptr(), *dwp = op.inputs == 3 ? out[2].mutable_data_ptr() : nullptr;
    void* st = c10::cuda::getCurrentCUDAStream().stream();
    if (op.tp) {
        // Half of the workspace, a quarter ... when the device cannot spare the whole: the library then goes through the
        // batch in blocks or with other kernels, as long as the partial weight gradients fit.
        const size_t want = oeq_tp_workspace_bytes(op.tp, x->size(0));
        for (size_t bytes = want;; bytes /= 2) {
            Tensor ws;
            try {
                if (bytes) ws = at::empty({(int64_t)bytes}, x->options().dtype(at::kByte));
            } catch (const c10::OutOfMemoryError&) {
                if (bytes / 2 < want / 64) throw;
                continue;
            }
            const int rc = oeq_tp_backward(op.tp, x->size(0), x->const_data_ptr(), y->const_data_ptr(), wp, dz->const_data_ptr(), dxp, dyp,
                                           dwp, bytes ? ws.mutable_data_ptr() : nullptr, bytes, st);
            TORCH_CHECK_WITH(OutOfMemoryError, rc != OEQ_ERR_INVALID || bytes == want, "out of memory: ", want, " bytes of workspace");
            check(rc);
            break;
        }
    } else {
        const auto rows = in[op.inputs + 1].expect_contiguous(), cols = in[op.inputs + 2].expect_contiguous();
        const auto perm = in[op.inputs + (op.deterministic ? 3 : 1)].expect_contiguous();
        const Scratch ws = op.deterministic ? backward_scratch(op, x->size(0), rows->size(0), x->options()) : Scratch();
        check(oeq_conv_backward(op.conv, x->size(0), rows->size(0), x->const_data_ptr(), y->const_data_ptr(), wp, dz->const_data_ptr(),
                                index_ptr(*rows), index_ptr(*cols), op.deterministic ? index_ptr(*perm) : nullptr, dxp, dyp, dwp,
                                ws.data(), ws.bytes(), st));
    }
    return out;
}

// The arguments on top of the stack.
variable_list pop(Stack* stack, int n) {
    variable_list in;
    in.reserve(n);
    for (auto it = stack->end() - n; it != stack->end(); ++it) in.push_back(std::move(*it).toTensor());
    torch::jit::drop(*stack, n);
    return in;
}
struct ForwardKernel final : c10::OperatorKernel {
    Op* op;
    explicit ForwardKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle&, c10::DispatchKeySet, Stack* stack) {
        stack->emplace_back(forward_cuda(*op, pop(stack, op->inputs + op->index)));
    }
};
struct GradientKernel final : c10::OperatorKernel {
    Op* op;
    explicit GradientKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle&, c10::DispatchKeySet, Stack* stack) {
        stack->emplace_back(c10::List<Tensor>(gradient_cuda(*op, pop(stack, op->inputs + 1 + op->index))));
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
    const Scratch ws = op.deterministic ? backward_scratch(op, nodes, edges, c[0].options()) : Scratch();
    const int rc = oeq_conv_double_backward(
        op.conv, nodes, edges, c[0].const_data_ptr(), c[1].const_data_ptr(), c[2].const_data_ptr(), c[3].const_data_ptr(),
        c[4].const_data_ptr(), c[5].const_data_ptr(), c[6].const_data_ptr(), index_ptr(idx[0]), index_ptr(idx[1]),
        op.deterministic ? index_ptr(idx[2]) : nullptr, out[0].mutable_data_ptr(), out[1].mutable_data_ptr(), out[2].mutable_data_ptr(),
        out[3].mutable_data_ptr(), ws.data(), ws.bytes(),
        c10::cuda::getCurrentCUDAStream().stream());
    if (rc == OEQ_ERR_UNSUPPORTED) return {};
    check(rc);
    return out;
}

// ---------------------------------------------------------------- autograd

// The gradients that an autograd node computes.  Plain CUDA tensors that nothing differentiates go straight to the
// kernels; anything else (tracing modes, tensor subclasses, batched tensors, negated or zero tensors whose memory does not
// hold their values, derivatives of the derivative) through the dispatcher.
bool direct(Args in) {
    using c10::DispatchKey;
    const auto tls = c10::impl::tls_local_dispatch_key_set().included_;
    if (at::GradMode::is_enabled() || tls.has(DispatchKey::Python) || tls.has(DispatchKey::PythonTLSSnapshot) ||
        tls.has(DispatchKey::FuncTorchDynamicLayerFrontMode) || tls.has(DispatchKey::Functionalize))
        return false;
    // keys of a dense CUDA tensor; a tensor with any other one is not plain
    static const uint64_t plain = c10::DispatchKeySet({DispatchKey::CUDA, DispatchKey::ADInplaceOrView, DispatchKey::AutogradCUDA, DispatchKey::AutocastCUDA}).raw_repr();
    for (const Tensor& t : in)
        if (!t.defined() || !t.is_cuda() || (t.key_set().raw_repr() & ~plain) != 0) return false;
    return true;
}
Tensor call_forward(const Op& op, Args in) {
    if (direct(in)) return forward_cuda(op, in);
    Stack stack(in.begin(), in.end());
    op.forward->callBoxed(stack);
    return stack.back().toTensor();
}
variable_list call_boxed(const OperatorHandle& handle, Args in) {
    Stack stack(in.begin(), in.end());
    handle.callBoxed(stack);
    return stack.back().toTensorVector();
}
variable_list call_gradient(Op& op, Args in) { return direct(in) ? gradient_cuda(op, in) : call_boxed(*op.gradient, in); }
variable_list joined(std::initializer_list<Tensor> a, Args index) {
    variable_list v;
    v.reserve(a.size() + index.size());
    v.insert(v.end(), a.begin(), a.end());
    v.insert(v.end(), index.begin(), index.end());
    return v;
}

// Saved operands (the index arrays among them), and next edges for the differentiable ones alone: a good deal less per
// call than torch::autograd::Function, which wraps every argument.
struct OpNode : torch::autograd::Node {
    Op* op;
    std::vector<torch::autograd::SavedVariable> saved;
    OpNode(Op* o, const variable_list& in, int diff) : op(o) {
        saved.reserve(in.size());
        for (const Tensor& t : in) saved.emplace_back(t, false);
        set_next_edges(torch::autograd::collect_next_edges(Args(in.data(), (size_t)diff)));
    }
    variable_list operands() {
        std::lock_guard<std::mutex> lock(mutex_);
        variable_list v;
        v.reserve(saved.size() + 1);
        for (const auto& s : saved) v.push_back(s.unpack());
        return v;
    }
    // (release_variables is not overridden: the operands live as long as the graph, so that a second backward pass through
    // a result needs no retain_graph, as with the reference's nodes, which keep their operands as attributes.)
};

struct ForwardNode final : OpNode {
    using OpNode::OpNode;
    std::string name() const override { return "OeqForwardBackward"; }
    variable_list apply(variable_list&& grads) override {
        variable_list in = operands();
        // (nothing flows in from a later node that gave no gradient: zeros, and zero gradients out)
        if (!grads[0].defined()) grads[0] = in[0].new_zeros_symint({in[0].sym_size(0), op->z_dim});
        in.insert(in.begin() + op->inputs, std::move(grads[0]));
        return call_gradient(*op, in);
    }
};

struct GradientNode final : OpNode {
    using OpNode::OpNode;
    std::string name() const override { return "OeqGradientBackward"; }
    // The product is trilinear in (x, y, w).  With cotangents (ex, ey, ew) of (dX, dY, dW):
    //   d/d(dz) = f(ex, y, w) + f(x, ey, w) + f(x, y, ew);  d/dx = dX(ey, w, dz) + dX(y, ew, dz), likewise y and w.
    variable_list apply(variable_list&& e) override {
        Op& o = *op;
        const variable_list s = operands();
        for (int i = 0; i < o.inputs; ++i)
            if (!e[i].defined()) e[i] = at::zeros_like(s[i]);
        const Args idx(s.data() + o.inputs + 1, (size_t)o.index);
        const Tensor &x = s[0], &y = s[1], &dz = s[o.inputs];
        if (o.inputs == 2) {
            variable_list a = call_gradient(o, joined({e[0], e[1], dz}, idx));
            return {a[0], a[1], call_forward(o, joined({e[0], y}, idx)) + call_forward(o, joined({x, e[1]}, idx))};
        }
        const Tensor& w = s[2];
        if (!at::GradMode::is_enabled()) {
            // nothing differentiates through this result: launches that read a row's arrays once
            const variable_list all_in{x, y, w, dz, e[0], e[1], e[2]};
            if (o.tp && oeq_tp_has_double_backward(o.tp) && direct(all_in)) return tp_second(o, all_in);
            if (o.conv) {
                variable_list all;
                if (o.second && o.call_second) all = call_boxed(*o.second, joined({x, y, w, dz, e[0], e[1], e[2]}, idx));
                else if (direct(all_in)) all = conv_second(o, all_in, idx);
                if (all.size() == 4) return all;
            }
        }
        variable_list a = call_gradient(o, joined({e[0], e[1], w, dz}, idx));    // dX(ey, w), dY(ex, w)
        variable_list b = call_gradient(o, joined({x, y, e[2], dz}, idx));       // dX(y, ew), dY(x, ew)
        variable_list c = call_gradient(o, joined({e[0], y, w, dz}, idx));       // dW(ex, y)
        variable_list d = call_gradient(o, joined({x, e[1], w, dz}, idx));       // dW(x, ey)
        Tensor gz = call_forward(o, joined({e[0], y, w}, idx)) + call_forward(o, joined({x, e[1], w}, idx)) +
                    call_forward(o, joined({x, y, e[2]}, idx));
        return {a[0] + b[0], a[1] + b[1], c[2] + d[2], gz};
    }
};

template <bool GRADIENT>
struct AutogradKernel final : c10::OperatorKernel {
    Op* op;
    explicit AutogradKernel(Op* o) : op(o) {}
    void operator()(const OperatorHandle& handle, c10::DispatchKeySet keys, Stack* stack) {
        const int diff = op->inputs + (GRADIENT ? 1 : 0), n = diff + op->index;
        // no tangents: below this kernel they would be dropped, and the derivative would come out as zero
        for (int i = 0; i < diff; ++i)
            TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined((*stack)[stack->size() - n + i].toTensor()),
                                        "openequivariance_b200: the operators have no forward-mode derivative");
        bool needed = false;
        if (at::GradMode::is_enabled())
            for (int i = 0; i < diff; ++i) needed |= (*stack)[stack->size() - n + i].toTensor().requires_grad();
        if (!needed) {
            at::AutoDispatchBelowADInplaceOrView guard;
            handle.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
            return;
        }
        variable_list in;
        in.reserve(n);
        for (auto it = stack->end() - n; it != stack->end(); ++it) in.push_back(it->toTensor());
        typedef std::conditional_t<GRADIENT, GradientNode, ForwardNode> NodeT;
        auto node = std::shared_ptr<NodeT>(new NodeT(op, in, diff), torch::autograd::deleteNode);
        {
            at::AutoDispatchBelowADInplaceOrView guard;
            handle.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
        }
        if constexpr (GRADIENT) {
            variable_list out = stack->back().toTensorVector();
            for (Tensor& t : out) torch::autograd::set_history(t, node);
            stack->back() = c10::List<Tensor>(std::move(out));
        } else {
            Tensor z = stack->back().toTensor();
            torch::autograd::set_history(z, node);
            stack->back() = std::move(z);
        }
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
        // (fake kernels and autograd are registered: a graph may hold these ops even where only such ops are allowed)
        const std::vector<at::Tag> tags{at::Tag::pt2_compliant_tag};
        lib.def((std::string(forward) + "(" + in + idx + ") -> Tensor").c_str(), tags);
        lib.def((std::string(gradient) + "(" + in + ", Tensor L3_grad" + idx + ") -> Tensor[]").c_str(), tags);
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

// The gradient passes of a convolution's object on raw pointers (any number of receivers), with the scratch that its ops
// keep: `forward` names its forward op; the current device and stream are those of the calling thread.  Returns the
// library's code; `scratch`: the memory used.  EX null: first derivatives into dX, dY, dW (and no dZ gradient).
int oeq_torch_conv_gradients(const char* forward, int64_t nodes, int64_t edges, const void* X, const void* Y, const void* W, const void* dZ,
                             const void* EX, const void* EY, const void* EW, const int64_t* rows, const int64_t* cols, const int64_t* perm,
                             void* dX, void* dY, void* dW, void* GdZ, int64_t* scratch_bytes, void** scratch) {
    try {
        Op* op = nullptr;
        {
            std::lock_guard<std::mutex> lock(register_mutex);
            auto it = operators().find(forward);
            TORCH_CHECK(it != operators().end(), "no such operator");
            op = it->second;
        }
        const auto stream = c10::cuda::getCurrentCUDAStream();
        const Scratch ws = op->deterministic ? backward_scratch(*op, nodes, edges, at::TensorOptions().device(stream.device())) : Scratch();
        *scratch_bytes = (int64_t)ws.bytes();
        *scratch = ws.data();
        if (EX) return oeq_conv_double_backward(op->conv, nodes, edges, X, Y, W, dZ, EX, EY, EW, rows, cols, perm, dX, dY, dW, GdZ,
                                                ws.data(), ws.bytes(), stream.stream());
        return oeq_conv_backward(op->conv, nodes, edges, X, Y, W, dZ, rows, cols, perm, dX, dY, dW, ws.data(), ws.bytes(), stream.stream());
    } catch (const std::exception& e) {
        register_error = e.what();
        return -1;
    }
}

}  // extern "C"

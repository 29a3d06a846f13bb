// Host path of the Python package, in native code: argument checks, output allocation, workspaces, autograd nodes and the
// calls into the C ABI (include/inferno_b200_attn.h), on torch tensors.
//
// The kernels know nothing of torch; this module is the one place where the two meet.  It finds the ABI's entry points in
// the shared object it is given (bind), so that another build of the library (the range-checked one) can stand in.
//
// Why native: a forward + backward of a small problem keeps the GPU busy for 25-50 us, and the same path written in Python
// (autograd.Function, ctypes marshalling of 30 arguments, views for the slices of a packed projection) took the host 200 us
// (4 x 4 heads, T = 128, fp32) -- small calls were bound by it.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/version.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <dlfcn.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <deque>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <utility>
#include <vector>

#include "../../include/inferno_b200_attn.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::Variable;
using torch::autograd::variable_list;

// ---- the C ABI, resolved once ----------------------------------------------------
struct Abi {
    decltype(&ib200_attn_workspace_bytes) workspace_bytes = nullptr;
    decltype(&ib200_attn_fwd_strided) attn_fwd = nullptr;
    decltype(&ib200_attn_fwd_chunk) attn_fwd_chunk = nullptr;
    decltype(&ib200_attn_bwd_strided) attn_bwd = nullptr;
    decltype(&ib200_linear_workspace_bytes) linear_workspace_bytes = nullptr;
    decltype(&ib200_linear_fwd_ws) linear_fwd = nullptr;
    decltype(&ib200_linear_bwd_ws) linear_bwd = nullptr;
    decltype(&ib200_attn_set_timing_events) set_timing_events = nullptr;
    decltype(&ib200_status_string) status_string = nullptr;
    PyObject* error_class = nullptr;      // the package's exception type, constructed from (status, where)
};
Abi g_abi;

// A status other than IB200_OK from the library.  It reaches Python as the package's own exception type, from the caller's thread
// (guarded) and from autograd's worker threads (in_node) alike.
struct StatusError : std::runtime_error {
    int status;
    const char* where;
    StatusError(int s, const char* w)
        : std::runtime_error(std::string(w) + ": " + g_abi.status_string(s) + " (status " + std::to_string(s) + ")"), status(s), where(w) {}
};
inline void check_status(int rc, const char* where) {
    if (rc != IB200_OK) throw StatusError(rc, where);
}

// ---- workspaces: caller-owned scratch of the C ABI, one per (device, stream), grown on demand ----------------------
// The number of entries is bounded by the number of streams a process uses (torch hands out a fixed pool of them).  A call
// holds its entry's lock while it issues its launches, so two host threads that share a stream cannot interleave the
// launches of two passes over one scratch buffer.  The table is never destroyed: at process exit the CUDA context may
// already be gone.  Attention and projections have a buffer each: a graph captured with the one must not lose it because an
// eager call of the other needs more.
struct Workspace {
    std::mutex launching;
    Tensor buf;            // attention; begins with the status header
    Tensor linear;
};
std::mutex g_ws_mutex;
std::map<std::pair<int, int64_t>, std::unique_ptr<Workspace>>& workspace_table() {
    static auto* t = new std::map<std::pair<int, int64_t>, std::unique_ptr<Workspace>>();
    return *t;
}
Workspace& workspace_of(int device, cudaStream_t stream) {
    const std::pair<int, int64_t> key{device, reinterpret_cast<int64_t>(stream)};
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    auto& slot = workspace_table()[key];
    if (!slot) slot = std::make_unique<Workspace>();
    return *slot;
}
// under ws.launching
Tensor empty_bytes(size_t bytes, c10::Device device) { return at::empty({static_cast<int64_t>(bytes)}, at::TensorOptions().dtype(at::kByte).device(device)); }
void reserve(Tensor& buf, size_t bytes, c10::Device device) {
    if (!buf.defined() || static_cast<size_t>(buf.numel()) < bytes) buf = empty_bytes(bytes, device);
}
// A projection's scratch.  While the stream is being captured it comes from the graph's own memory, and goes back there after the
// call: the graph then depends on nothing that a later call could replace.
Tensor linear_scratch(Workspace& ws, size_t bytes, c10::Device device) {
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return empty_bytes(bytes, device);
    reserve(ws.linear, bytes, device);
    return ws.linear;
}

// ---- timing events queued by a harness: one {start, stop} pair per attention call, forward and backward ----------------
struct TimingQueue {
    std::mutex m;
    std::deque<std::pair<cudaEvent_t, cudaEvent_t>> fwd, bwd;
    std::atomic<bool> any{false};
};
TimingQueue g_timing;
struct TimingScope {
    bool on = false;
    explicit TimingScope(bool backward) {
        if (!g_timing.any) return;
        std::lock_guard<std::mutex> lock(g_timing.m);
        auto& q = backward ? g_timing.bwd : g_timing.fwd;
        if (q.empty()) return;
        const auto ev = q.front();
        q.pop_front();
        g_timing.any = !g_timing.fwd.empty() || !g_timing.bwd.empty();
        auto e = [](cudaEvent_t x) { return reinterpret_cast<ib200_event_t>(x); };
        on = backward ? g_abi.set_timing_events(nullptr, nullptr, e(ev.first), e(ev.second)) == IB200_OK
                      : g_abi.set_timing_events(e(ev.first), e(ev.second), nullptr, nullptr) == IB200_OK;
    }
    ~TimingScope() {
        if (on) g_abi.set_timing_events(nullptr, nullptr, nullptr, nullptr);
    }
};

// ---- attention: checks and layouts -----------------------------------------------
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? IB200_DTYPE_F32 : IB200_DTYPE_BF16; }

void check_inputs(std::initializer_list<const Tensor*> ts) {
    const Tensor& q = **ts.begin();
    TORCH_CHECK_VALUE(q.dim() == 4, "causal_attention expects [B, H, T, D] tensors");
    for (const Tensor* t : ts) {
        TORCH_CHECK(t->is_cuda(), "causal_attention: tensor is not on a CUDA device (there is no CPU path)");
        TORCH_CHECK(t->device() == q.device(), "causal_attention: tensors are on different devices");
        TORCH_CHECK_TYPE(t->scalar_type() == q.scalar_type() && (t->scalar_type() == at::kFloat || t->scalar_type() == at::kBFloat16),
                         "causal_attention: dtype must be float32 or bfloat16, the same for all tensors");
        TORCH_CHECK_VALUE(t->sizes() == q.sizes(), "causal_attention: q, k, v (and dO) must have the same shape");
    }
}
// Caller-supplied outputs: any strides the kernels can address.
void check_like(const Tensor& t, const Tensor& q, const char* name) {
    TORCH_CHECK_VALUE(t.sizes() == q.sizes() && t.scalar_type() == q.scalar_type() && t.device() == q.device(), "causal_attention: `", name,
                      "` must match q in shape, dtype and device");
}
// The log-sum-exp vector is addressed densely by the kernels.
void check_lse_of(const Tensor& lse, c10::Device device, int64_t B, int64_t H, int64_t T) {
    TORCH_CHECK_VALUE(lse.scalar_type() == at::kFloat && lse.device() == device && lse.dim() == 3 && lse.size(0) == B && lse.size(1) == H &&
                          lse.size(2) == T && lse.is_contiguous(),
                      "causal_attention: `lse` must be a contiguous float32 [B, H, T] tensor on q's device");
}
void check_lse(const Tensor& lse, const Tensor& q) { check_lse_of(lse, q.device(), q.size(0), q.size(1), q.size(2)); }
// A packed [B, T, 3*H*D] operand.
void check_packed(const Tensor& qkv, int64_t H) {
    TORCH_CHECK_VALUE(qkv.dim() == 3 && H > 0, "causal_attention_packed expects a [B, T, 3*C] tensor and a positive number of heads");
    TORCH_CHECK(qkv.size(2) / 3 / H * H * 3 == qkv.size(2), "causal_attention_packed: the last axis (", qkv.size(2), ") is not 3 * num_heads * head_dim");
    TORCH_CHECK(qkv.is_cuda(), "causal_attention: tensor is not on a CUDA device (there is no CPU path)");
    TORCH_CHECK_TYPE(qkv.scalar_type() == at::kFloat || qkv.scalar_type() == at::kBFloat16,
                     "causal_attention: dtype must be float32 or bfloat16, the same for all tensors");
}

// A [B, H, T, D] operand as the C ABI takes it.
struct Operand {
    void* ptr;
    ib200_layout lay;
};
Operand operand(const Tensor& t) {
    TORCH_CHECK_VALUE(t.stride(3) == 1, "causal_attention: the head-dim axis must be contiguous");
    return {t.data_ptr(), {t.stride(0), t.stride(1), t.stride(2)}};
}
// In place when the kernels can address the tensor (contiguous rows, 16-byte aligned strides); otherwise the dense copy the
// reference makes with .contiguous().
Tensor dense_or_view(const Tensor& t) {
    const int64_t unit = 16 / t.element_size();
    bool ok = t.stride(3) == 1 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0;
    for (int a = 0; a < 3; ++a) ok = ok && t.stride(a) > 0 && t.stride(a) % unit == 0;
    return ok ? t : t.contiguous();
}
// The same for a packed [B, T, n*H*D] tensor.
Tensor dense_or_packed(const Tensor& t) {
    const int64_t unit = 16 / t.element_size();
    const bool ok = t.stride(2) == 1 && t.stride(0) > 0 && t.stride(1) > 0 && t.stride(0) % unit == 0 && t.stride(1) % unit == 0 &&
                    (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0;
    return ok ? t : t.contiguous();
}
// One third of a packed [B, T, 3, H, D] buffer, as a [B, H, T, D] operand.
Operand packed_operand(const Tensor& p, int which, int64_t C, int64_t D) {
    return {static_cast<char*>(p.data_ptr()) + static_cast<int64_t>(which) * C * p.element_size(), {p.stride(0), D, p.stride(1)}};
}

struct Shape {
    int B, H, T, D, dtype;
};
Shape shape_of(const Tensor& q) {
    return {static_cast<int>(q.size(0)), static_cast<int>(q.size(1)), static_cast<int>(q.size(2)), static_cast<int>(q.size(3)), dtype_code(q)};
}
float scale_of(const std::optional<double>& s, int64_t D) { return static_cast<float>(s ? *s : 1.0 / std::sqrt(static_cast<double>(D))); }

// ---- launches (the caller has made the tensors' device current) ------------------------------------------
void launch_fwd(const Shape& s, const Operand& q, const Operand& k, const Operand& v, const Operand& o, float* lse, float scale, bool causal,
                int math_mode, c10::Device device, int total_heads = 0) {
    size_t bytes = 0;
    check_status(g_abi.workspace_bytes(s.B, s.H, s.T, s.D, s.dtype, IB200_PASS_FWD, &bytes), "ib200_attn_workspace_bytes");
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    Workspace& ws = workspace_of(device.index(), stream);
    std::lock_guard<std::mutex> lock(ws.launching);
    reserve(ws.buf, bytes, device);
    TimingScope timing(false);
    if (total_heads > 0) {
        check_status(g_abi.attn_fwd_chunk(q.ptr, k.ptr, v.ptr, o.ptr, lse, &q.lay, &k.lay, &v.lay, &o.lay, total_heads, s.B, s.H, s.T, s.D, scale, causal,
                                          s.dtype, math_mode, ws.buf.data_ptr(), ws.buf.numel(), reinterpret_cast<ib200_stream_t>(stream)),
                     "ib200_attn_fwd_chunk");
        return;
    }
    check_status(g_abi.attn_fwd(q.ptr, k.ptr, v.ptr, o.ptr, lse, &q.lay, &k.lay, &v.lay, &o.lay, s.B, s.H, s.T, s.D, scale, causal, s.dtype, math_mode,
                                ws.buf.data_ptr(), ws.buf.numel(), reinterpret_cast<ib200_stream_t>(stream)),
                 "ib200_attn_fwd_strided");
}

void launch_bwd(const Shape& s, const Operand& q, const Operand& k, const Operand& v, const Operand& o, const Operand& dO, const float* lse,
                const Operand& dq, const Operand& dk, const Operand& dv, float scale, bool causal, int math_mode, c10::Device device) {
    size_t bytes = 0;
    check_status(g_abi.workspace_bytes(s.B, s.H, s.T, s.D, s.dtype, IB200_PASS_BWD, &bytes), "ib200_attn_workspace_bytes");
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
    Workspace& ws = workspace_of(device.index(), stream);
    std::lock_guard<std::mutex> lock(ws.launching);
    reserve(ws.buf, bytes, device);
    TimingScope timing(true);
    check_status(g_abi.attn_bwd(q.ptr, k.ptr, v.ptr, o.ptr, dO.ptr, lse, dq.ptr, dk.ptr, dv.ptr, &q.lay, &k.lay, &v.lay, &o.lay, &dO.lay, &dq.lay, &dk.lay,
                                &dv.lay, s.B, s.H, s.T, s.D, scale, causal, s.dtype, math_mode, ws.buf.data_ptr(), ws.buf.numel(),
                                reinterpret_cast<ib200_stream_t>(stream)),
                 "ib200_attn_bwd_strided");
}

Tensor empty_lse(const Tensor& q, const Shape& s) { return at::empty({s.B, s.H, s.T}, q.options().dtype(at::kFloat)); }
// A [B, H, T, D] view over [B, T, H, D] memory: `y.transpose(1, 2).reshape(B, T, C)` is then free.
Tensor empty_bthd(const Tensor& q, const Shape& s) {
    const int64_t D = s.D, HD = static_cast<int64_t>(s.H) * D;
    return at::empty_strided({s.B, s.H, s.T, s.D}, {s.T * HD, D, HD, 1}, q.options());
}

// Forward on [B, H, T, D] tensors or views.
std::pair<Tensor, Tensor> attention_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const std::optional<double>& scale, bool causal,
                                            int math_mode, const Tensor& out, const Tensor& lse_, bool bthd, int total_heads = 0) {
    check_inputs({&q_, &k_, &v_});
    const c10::cuda::CUDAGuard guard(q_.device());
    const Tensor q = dense_or_view(q_), k = dense_or_view(k_), v = dense_or_view(v_);
    const Shape s = shape_of(q);
    if (out.defined()) check_like(out, q, "out");
    if (lse_.defined()) check_lse(lse_, q);
    Tensor o = out.defined() ? out : bthd ? empty_bthd(q, s) : at::empty(q.sizes(), q.options());
    Tensor lse = lse_.defined() ? lse_ : empty_lse(q, s);
    launch_fwd(s, operand(q), operand(k), operand(v), operand(o), lse.data_ptr<float>(), scale_of(scale, s.D), causal, math_mode, q.device(), total_heads);
    return {o, lse};
}

struct Grads {
    Tensor dq, dk, dv;
};
Grads attention_backward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& o_, const Tensor& dO_, const Tensor& lse,
                         const std::optional<double>& scale, bool causal, int math_mode, Tensor dq, Tensor dk, Tensor dv) {
    check_inputs({&q_, &k_, &v_, &o_, &dO_});
    const c10::cuda::CUDAGuard guard(q_.device());
    const Tensor q = dense_or_view(q_), k = dense_or_view(k_), v = dense_or_view(v_), o = dense_or_view(o_), dO = dense_or_view(dO_);
    const Shape s = shape_of(q);
    check_lse(lse, q);
    auto output = [&](Tensor& t, const char* name) {
        if (t.defined()) check_like(t, q, name); else t = at::empty(q.sizes(), q.options());
    };
    output(dq, "dq");
    output(dk, "dk");
    output(dv, "dv");
    launch_bwd(s, operand(q), operand(k), operand(v), operand(o), operand(dO), lse.data_ptr<float>(), operand(dq), operand(dk), operand(dv),
               scale_of(scale, s.D), causal, math_mode, q.device());
    return {dq, dk, dv};
}

// ---- autograd nodes ----------------------------------------------------------------
void set_python_error(const StatusError& e) {      // with the GIL
    PyObject* err = PyObject_CallFunction(g_abi.error_class, "is", e.status, e.where);
    if (!err) return;
    PyErr_SetObject(g_abi.error_class, err);
    Py_DECREF(err);
}
// Body of a node: a status becomes a Python exception that the engine carries over to the thread that called backward.
template <class F>
variable_list in_node(F&& f) {
    try {
        return f();
    } catch (const StatusError& e) {
        python_error err;
        {
            pybind11::gil_scoped_acquire gil;
            set_python_error(e);
            err.persist();
        }
        throw err;
    }
}
// The ops have no forward-mode derivative: a dual input must not lose its tangent silently.
void refuse_tangents(std::initializer_list<const Tensor*> ts, const char* op) {
    for (const Tensor* t : ts)
        TORCH_CHECK_NOT_IMPLEMENTED(!t->defined() || !t->_fw_grad(0).defined(), op, ": forward-mode differentiation is not implemented");
}

// The backward node of the fused op: saves q, k, v, out and lse; produces dq, dk, dv.  Plays the role a
// `class AttentionBackward : public Node` has in the reference (src/inferno/gradfn/node.h:23-45).
struct AttentionBackward : torch::autograd::Node {
    SavedVariable q, k, v, o, lse;
    double scale = 0;
    bool causal = true;
    int math_mode = 0;

    variable_list apply(variable_list&& grads) override {
        return in_node([&] { return backward(grads); });
    }
    variable_list backward(const variable_list& grads) {
        if (!grads[0].defined()) return variable_list(3);
        const Tensor tq = q.unpack(), tk = k.unpack(), tv = v.unpack(), to = o.unpack(shared_from_this()), tl = lse.unpack();
        at::AutoDispatchBelowADInplaceOrView below;
        const int64_t B = tq.size(0), H = tq.size(1), T = tq.size(2), D = tq.size(3), step = H * D * tq.element_size();
        auto at_byte = [](const Tensor& t) { return static_cast<const char*>(t.data_ptr()); };
        Tensor dq, dk, dv;
        // slices of one packed [B, T, 3, H, D] buffer get their gradients in one buffer of the same layout
        if (tq.strides() == tk.strides() && tk.strides() == tv.strides() && tq.stride(2) == 3 * H * D && tq.stride(1) == D &&
            at_byte(tk) - at_byte(tq) == step && at_byte(tv) - at_byte(tk) == step) {
            const Tensor g = at::empty({B, T, 3, H, D}, tq.options());
            dq = g.select(2, 0).transpose(1, 2);
            dk = g.select(2, 1).transpose(1, 2);
            dv = g.select(2, 2).transpose(1, 2);
        }
        const Grads r = attention_backward(tq, tk, tv, to, grads[0], tl, scale, causal, math_mode, dq, dk, dv);
        return {r.dq, r.dk, r.dv};
    }
    void release_variables() override {
        q.reset_data(); k.reset_data(); v.reset_data(); o.reset_data(); lse.reset_data();
    }
    std::string name() const override { return "AttentionBackward"; }
};

Tensor causal_attention(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<double>& scale, bool causal, int math_mode, bool bthd,
                        int total_heads) {
    refuse_tangents({&q, &k, &v}, "causal_attention");
    const bool differentiable = torch::autograd::compute_requires_grad(q, k, v);
    Tensor o, lse;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        std::tie(o, lse) = attention_forward(q, k, v, scale, causal, math_mode, Tensor(), Tensor(), bthd, total_heads);
    }
    if (differentiable) {
        auto node = std::shared_ptr<AttentionBackward>(new AttentionBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(q, k, v));
        node->q = SavedVariable(q, false);
        node->k = SavedVariable(k, false);
        node->v = SavedVariable(v, false);
        node->lse = SavedVariable(lse, false);
        node->scale = scale ? *scale : 1.0 / std::sqrt(static_cast<double>(q.size(3)));
        node->causal = causal;
        node->math_mode = math_mode;
        torch::autograd::set_history(o, node);
        node->o = SavedVariable(o, true);
    }
    return o;
}

// The same op on a fused projection output [B, T, 3*C]: one input, one gradient.  Written for three views of the packed
// buffer, autograd would fill a zeroed buffer per view, copy each slice's gradient into it and add the three up (240 of the
// 490 us of a 12-head T = 1024 B = 16 layer); here dq, dk, dv land in their places in the gradient itself.
struct PackedAttentionBackward : torch::autograd::Node {
    SavedVariable qkv, o, lse;      // o: [B, T, C]
    int64_t H = 0;
    float scale = 0;
    int math_mode = 0;

    variable_list apply(variable_list&& grads) override {
        return in_node([&] { return backward(grads); });
    }
    variable_list backward(const variable_list& grads) {
        if (!grads[0].defined()) return variable_list(1);
        const Tensor p_ = qkv.unpack(), o_ = o.unpack(shared_from_this()), tl = lse.unpack();
        at::AutoDispatchBelowADInplaceOrView below;
        // what was saved has passed through the user's saved-tensor hooks, and may come back with other strides, or as something else
        check_packed(p_, H);
        const c10::cuda::CUDAGuard guard(p_.device());
        const int64_t B = p_.size(0), T = p_.size(1), C = p_.size(2) / 3, D = C / H;
        for (const Tensor& t : {o_, grads[0]}) {
            TORCH_CHECK(t.device() == p_.device(), "causal_attention: tensors are on different devices");
            TORCH_CHECK_TYPE(t.scalar_type() == p_.scalar_type(), "causal_attention: dtype must be float32 or bfloat16, the same for all tensors");
            TORCH_CHECK_VALUE(t.dim() == 3 && t.size(0) == B && t.size(1) == T && t.size(2) == C, "causal_attention: the output and its gradient must be [B, T, C]");
        }
        check_lse_of(tl, p_.device(), B, H, T);
        const Tensor p = dense_or_packed(p_), to = dense_or_packed(o_), dy = dense_or_packed(grads[0]);
        const Shape s{static_cast<int>(B), static_cast<int>(H), static_cast<int>(T), static_cast<int>(D), dtype_code(p)};
        Tensor g = at::empty({B, T, 3 * C}, p.options());
        launch_bwd(s, packed_operand(p, 0, C, D), packed_operand(p, 1, C, D), packed_operand(p, 2, C, D), packed_operand(to, 0, C, D),
                   packed_operand(dy, 0, C, D), tl.data_ptr<float>(), packed_operand(g, 0, C, D), packed_operand(g, 1, C, D), packed_operand(g, 2, C, D), scale,
                   true, math_mode, p.device());
        return {g};
    }
    void release_variables() override {
        qkv.reset_data(); o.reset_data(); lse.reset_data();
    }
    std::string name() const override { return "PackedAttentionBackward"; }
};

Tensor causal_attention_packed(const Tensor& qkv, int64_t H, const std::optional<double>& scale, int math_mode, int total_heads) {
    check_packed(qkv, H);
    const int64_t B = qkv.size(0), T = qkv.size(1), C = qkv.size(2) / 3, D = C / H;
    refuse_tangents({&qkv}, "causal_attention");
    const bool differentiable = torch::autograd::compute_requires_grad(qkv);
    Tensor o, lse, p;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        const c10::cuda::CUDAGuard guard(qkv.device());
        p = dense_or_packed(qkv);
        const Shape s{static_cast<int>(B), static_cast<int>(H), static_cast<int>(T), static_cast<int>(D), dtype_code(p)};
        o = at::empty({B, T, C}, p.options());
        lse = at::empty({B, H, T}, p.options().dtype(at::kFloat));
        launch_fwd(s, packed_operand(p, 0, C, D), packed_operand(p, 1, C, D), packed_operand(p, 2, C, D), packed_operand(o, 0, C, D), lse.data_ptr<float>(),
                   scale_of(scale, D), true, math_mode, p.device(), total_heads);
    }
    if (differentiable) {
        auto node = std::shared_ptr<PackedAttentionBackward>(new PackedAttentionBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(qkv));
        node->qkv = SavedVariable(p, false);
        node->lse = SavedVariable(lse, false);
        node->H = H;
        node->scale = scale_of(scale, D);
        node->math_mode = math_mode;
        torch::autograd::set_history(o, node);
        node->o = SavedVariable(o, true);
    }
    return o;
}

// ---- projections -------------------------------------------------------------------
// Shapes first, ahead of any allocation: the kernels get no more than the pointers and M, K, N.
void check_linear_shapes(const Tensor& x, const Tensor& w) {
    TORCH_CHECK_VALUE(w.dim() == 2, "linear: w must be [in, out]");
    TORCH_CHECK_VALUE(x.dim() >= 1 && x.size(-1) == w.size(0), "linear: the last axis of x must be w's first (", w.size(0), "), x is ", x.sizes());
}
void check_same_device(const Tensor& t, const Tensor& x, const char* name) {
    TORCH_CHECK_VALUE(t.device() == x.device(), "linear: ", name, " is on ", t.device(), ", x on ", x.device());
}
void check_bf16_cuda(const Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda(), "linear: ", name, " is not on a CUDA device (there is no CPU path)");
    TORCH_CHECK_TYPE(t.scalar_type() == at::kBFloat16, "linear: ", name, " must be bfloat16");
}

Tensor linear_forward(const Tensor& x, const Tensor& w, const Tensor& bias) {
    check_linear_shapes(x, w);
    const int64_t K = w.size(0), N = w.size(1);
    TORCH_CHECK_VALUE(!bias.defined() || bias.numel() == N, "linear: the bias must have ", N, " elements");
    check_bf16_cuda(x, "x");
    check_bf16_cuda(w, "w");
    check_same_device(w, x, "w");
    if (bias.defined()) check_same_device(bias, x, "the bias");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = x.reshape({-1, K}).contiguous(), wc = w.contiguous();
    Tensor b = bias;
    if (b.defined() && b.scalar_type() != at::kBFloat16) b = b.to(at::kFloat);
    if (b.defined()) b = b.contiguous();
    // the kernel reads a bias in place: a bf16 slice that does not begin on 16 bytes is copied, as it was when every bias became fp32
    if (b.defined() && b.scalar_type() == at::kBFloat16 && (reinterpret_cast<uintptr_t>(b.data_ptr()) & 15u)) b = b.clone();
    auto shape = x.sizes().vec();
    shape.back() = N;
    Tensor y = at::empty(shape, x.options());
    const int M = static_cast<int>(x2.size(0));
    const size_t bytes = g_abi.linear_workspace_bytes(M, static_cast<int>(K), static_cast<int>(N), IB200_PASS_FWD);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    std::unique_lock<std::mutex> lock;
    Tensor scratch;
    if (bytes) {
        Workspace& ws = workspace_of(x.device().index(), stream);
        lock = std::unique_lock<std::mutex>(ws.launching);
        scratch = linear_scratch(ws, bytes, x.device());
    }
    check_status(g_abi.linear_fwd(x2.data_ptr(), wc.data_ptr(), b.defined() ? b.data_ptr() : nullptr, b.defined() ? dtype_code(b) : IB200_DTYPE_F32,
                                  y.data_ptr(), M, static_cast<int>(K), static_cast<int>(N), bytes ? scratch.data_ptr() : nullptr, bytes,
                                  reinterpret_cast<ib200_stream_t>(stream)),
                 "ib200_linear_fwd_ws");
    return y;
}

struct LinearGrads {
    Tensor dx, dw, db;
};
LinearGrads linear_backward(const Tensor& x, const Tensor& w, const Tensor& dy, bool need_dx, bool need_dw, bool need_db, bool db_bf16) {
    check_linear_shapes(x, w);
    const int64_t K = w.size(0), N = w.size(1);
    TORCH_CHECK_VALUE(dy.dim() >= 1 && dy.size(-1) == N && dy.numel() / std::max<int64_t>(N, 1) == x.numel() / std::max<int64_t>(K, 1),
                      "linear: dy must have the rows of x and ", N, " columns, dy is ", dy.sizes(), ", x is ", x.sizes());
    check_bf16_cuda(x, "x");
    check_bf16_cuda(w, "w");
    check_bf16_cuda(dy, "dy");
    check_same_device(w, x, "w");
    check_same_device(dy, x, "dy");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = x.reshape({-1, K}).contiguous(), dy2 = dy.reshape({-1, N}).contiguous(), wc = w.contiguous();
    const int M = static_cast<int>(x2.size(0));
    LinearGrads g;
    if (need_dx) g.dx = at::empty(x.sizes(), x.options());
    if (need_dw) g.dw = at::empty({K, N}, x.options());
    if (need_db) g.db = at::empty({N}, x.options().dtype(db_bf16 ? at::kBFloat16 : at::kFloat));
    const size_t bytes = g_abi.linear_workspace_bytes(M, static_cast<int>(K), static_cast<int>(N), IB200_PASS_BWD);
    cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    Workspace& ws = workspace_of(x.device().index(), stream);
    std::lock_guard<std::mutex> lock(ws.launching);
    const Tensor scratch = linear_scratch(ws, bytes, x.device());
    auto ptr = [](const Tensor& t) -> void* { return t.defined() ? t.data_ptr() : nullptr; };
    check_status(g_abi.linear_bwd(x2.data_ptr(), wc.data_ptr(), dy2.data_ptr(), ptr(g.dx), ptr(g.dw), ptr(g.db), db_bf16 ? IB200_DTYPE_BF16 : IB200_DTYPE_F32, M,
                                  static_cast<int>(K), static_cast<int>(N), scratch.data_ptr(), bytes,
                                  reinterpret_cast<ib200_stream_t>(stream)),
                 "ib200_linear_bwd_ws");
    return g;
}

struct LinearBackward : torch::autograd::Node {
    SavedVariable x, w;
    bool has_bias = false;
    at::ScalarType bias_type = at::kFloat;

    variable_list apply(variable_list&& grads) override {
        return in_node([&] { return backward(grads); });
    }
    variable_list backward(const variable_list& grads) {
        variable_list out(3);
        if (!grads[0].defined()) return out;
        const Tensor tx = x.unpack(), tw = w.unpack();
        at::AutoDispatchBelowADInplaceOrView below;
        LinearGrads g = linear_backward(tx, tw, grads[0], task_should_compute_output(0), task_should_compute_output(1),
                                        has_bias && task_should_compute_output(2), bias_type == at::kBFloat16);
        out[0] = g.dx;
        out[1] = g.dw;
        if (g.db.defined()) out[2] = g.db.to(bias_type);      // fp32 and bf16 come in the right type
        return out;
    }
    void release_variables() override { x.reset_data(); w.reset_data(); }
    std::string name() const override { return "LinearBackward"; }
};

Tensor linear(const Tensor& x, const Tensor& w, const Tensor& bias) {
    refuse_tangents({&x, &w, &bias}, "linear");
    const bool differentiable = torch::autograd::compute_requires_grad(x, w, bias);
    Tensor y;
    {
        at::AutoDispatchBelowADInplaceOrView below;
        y = linear_forward(x, w, bias);
    }
    if (differentiable) {
        auto node = std::shared_ptr<LinearBackward>(new LinearBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(x, w, bias));
        node->x = SavedVariable(x, false);
        node->w = SavedVariable(w, false);
        node->has_bias = bias.defined();
        if (bias.defined()) node->bias_type = bias.scalar_type();
        torch::autograd::set_history(y, node);
    }
    return y;
}

// ---- Python boundary ---------------------------------------------------------------
// Plain METH_FASTCALL functions: positional arguments, None for an absent tensor or the default scale.
const Tensor& arg_tensor(PyObject* o) {
    TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a torch.Tensor, got ", Py_TYPE(o)->tp_name);
    return THPVariable_Unpack(o);
}
Tensor arg_opt_tensor(PyObject* o) { return o == Py_None ? Tensor() : arg_tensor(o); }
std::optional<double> arg_scale(PyObject* o) {
    if (o == Py_None) return std::nullopt;
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) throw python_error();
    return d;
}
int64_t arg_int(PyObject* o) {
    const long long v = PyLong_AsLongLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}
// None (0): the call is the whole problem; otherwise the heads of the problem that it is a part of.
int arg_total_heads(PyObject* o) {
    if (o == Py_None) return 0;
    const int64_t n = arg_int(o);
    TORCH_CHECK_VALUE(n > 0 && n <= 0x7fffffff, "causal_attention: total_heads must be a positive number of heads, got ", n);
    return static_cast<int>(n);
}
bool arg_bool(PyObject* o) {
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
void want(Py_ssize_t got, Py_ssize_t n) {
    TORCH_CHECK_TYPE(got == n, "expected ", n, " arguments, got ", got);
}
PyObject* wrap(const Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}
PyObject* wrap_tuple(std::initializer_list<const Tensor*> ts) {
    PyObject* out = PyTuple_New(static_cast<Py_ssize_t>(ts.size()));
    if (!out) throw python_error();
    Py_ssize_t i = 0;
    for (const Tensor* t : ts) PyTuple_SET_ITEM(out, i++, wrap(*t));
    return out;
}

template <class F>
PyObject* guarded(F&& f) {
    HANDLE_TH_ERRORS
    try {
        return f();
    } catch (const StatusError& e) {
        set_python_error(e);
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 2);
        const char* path = PyUnicode_AsUTF8(a[0]);
        if (!path) throw python_error();
        void* so = dlopen(path, RTLD_NOW | RTLD_LOCAL);
        TORCH_CHECK(so, "cannot load ", path, ": ", dlerror());
        auto get = [&](auto& fn, const char* name) {
            fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(so, name));
            TORCH_CHECK(fn, path, " does not export ", name);
        };
        get(g_abi.workspace_bytes, "ib200_attn_workspace_bytes");
        get(g_abi.attn_fwd, "ib200_attn_fwd_strided");
        get(g_abi.attn_fwd_chunk, "ib200_attn_fwd_chunk");
        get(g_abi.attn_bwd, "ib200_attn_bwd_strided");
        get(g_abi.linear_workspace_bytes, "ib200_linear_workspace_bytes");
        get(g_abi.linear_fwd, "ib200_linear_fwd_ws");
        get(g_abi.linear_bwd, "ib200_linear_bwd_ws");
        get(g_abi.set_timing_events, "ib200_attn_set_timing_events");
        get(g_abi.status_string, "ib200_status_string");
        Py_INCREF(a[1]);
        Py_XDECREF(g_abi.error_class);
        g_abi.error_class = a[1];
        Py_RETURN_NONE;
    });
}

// (q, k, v, scale, causal, math_mode, out, lse, total_heads) -> (o, lse)
PyObject* py_attention_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 9);
        const Tensor &q = arg_tensor(a[0]), &k = arg_tensor(a[1]), &v = arg_tensor(a[2]);
        const auto scale = arg_scale(a[3]);
        const bool causal = arg_bool(a[4]);
        const int math_mode = static_cast<int>(arg_int(a[5]));
        const Tensor out = arg_opt_tensor(a[6]), lse = arg_opt_tensor(a[7]);
        const int total_heads = arg_total_heads(a[8]);
        std::pair<Tensor, Tensor> r;
        {
            pybind11::gil_scoped_release nogil;
            at::AutoDispatchBelowADInplaceOrView below;
            r = attention_forward(q, k, v, scale, causal, math_mode, out, lse, false, total_heads);
        }
        return wrap_tuple({&r.first, &r.second});
    });
}

// (q, k, v, o, dO, lse, scale, causal, math_mode, dq, dk, dv) -> (dq, dk, dv)
PyObject* py_attention_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 12);
        const Tensor &q = arg_tensor(a[0]), &k = arg_tensor(a[1]), &v = arg_tensor(a[2]), &o = arg_tensor(a[3]), &dO = arg_tensor(a[4]), &lse = arg_tensor(a[5]);
        const auto scale = arg_scale(a[6]);
        const bool causal = arg_bool(a[7]);
        const int math_mode = static_cast<int>(arg_int(a[8]));
        const Tensor dq = arg_opt_tensor(a[9]), dk = arg_opt_tensor(a[10]), dv = arg_opt_tensor(a[11]);
        Grads g;
        {
            pybind11::gil_scoped_release nogil;
            at::AutoDispatchBelowADInplaceOrView below;
            g = attention_backward(q, k, v, o, dO, lse, scale, causal, math_mode, dq, dk, dv);
        }
        return wrap_tuple({&g.dq, &g.dk, &g.dv});
    });
}

// (q, k, v, scale, causal, math_mode, bthd_out, total_heads) -> y, differentiable
PyObject* py_causal_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 8);
        const Tensor &q = arg_tensor(a[0]), &k = arg_tensor(a[1]), &v = arg_tensor(a[2]);
        const auto scale = arg_scale(a[3]);
        const bool causal = arg_bool(a[4]);
        const int math_mode = static_cast<int>(arg_int(a[5]));
        const bool bthd = arg_bool(a[6]);
        const int total_heads = arg_total_heads(a[7]);
        Tensor y;
        {
            pybind11::gil_scoped_release nogil;
            y = causal_attention(q, k, v, scale, causal, math_mode, bthd, total_heads);
        }
        return wrap(y);
    });
}

// (qkv, num_heads, scale, math_mode, total_heads) -> y, differentiable
PyObject* py_causal_attention_packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 5);
        const Tensor& qkv = arg_tensor(a[0]);
        const int64_t H = arg_int(a[1]);
        const auto scale = arg_scale(a[2]);
        const int math_mode = static_cast<int>(arg_int(a[3]));
        const int total_heads = arg_total_heads(a[4]);
        Tensor y;
        {
            pybind11::gil_scoped_release nogil;
            y = causal_attention_packed(qkv, H, scale, math_mode, total_heads);
        }
        return wrap(y);
    });
}

// (x, w, bias) -> y; the differentiable form and the plain one
PyObject* py_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 3);
        const Tensor &x = arg_tensor(a[0]), &w = arg_tensor(a[1]);
        const Tensor bias = arg_opt_tensor(a[2]);
        Tensor y;
        {
            pybind11::gil_scoped_release nogil;
            y = linear(x, w, bias);
        }
        return wrap(y);
    });
}
PyObject* py_linear_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 3);
        const Tensor &x = arg_tensor(a[0]), &w = arg_tensor(a[1]);
        const Tensor bias = arg_opt_tensor(a[2]);
        Tensor y;
        {
            pybind11::gil_scoped_release nogil;
            at::AutoDispatchBelowADInplaceOrView below;
            y = linear_forward(x, w, bias);
        }
        return wrap(y);
    });
}
// (x, w, dy, need_dx, need_dw, need_db) -> (dx, dw, db)
PyObject* py_linear_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 6);
        const Tensor &x = arg_tensor(a[0]), &w = arg_tensor(a[1]), &dy = arg_tensor(a[2]);
        const bool need_dx = arg_bool(a[3]), need_dw = arg_bool(a[4]), need_db = arg_bool(a[5]);
        LinearGrads g;
        {
            pybind11::gil_scoped_release nogil;
            at::AutoDispatchBelowADInplaceOrView below;
            g = linear_backward(x, w, dy, need_dx, need_dw, need_db, false);
        }
        return wrap_tuple({&g.dx, &g.dw, &g.db});
    });
}

// () -> {(device index, stream handle): workspace tensor}
PyObject* py_workspaces(PyObject*, PyObject* const*, Py_ssize_t) {
    return guarded([&]() -> PyObject* {
        std::vector<std::pair<std::pair<int, int64_t>, Tensor>> list;
        {
            // A launch holds its entry's lock without the GIL and may come to need it there (to free a buffer that Python has seen, or
            // to allocate under a Python dispatch mode), so nobody waits for that lock with the GIL in hand.
            pybind11::gil_scoped_release nogil;
            std::lock_guard<std::mutex> lock(g_ws_mutex);
            for (const auto& [key, ws] : workspace_table()) {
                std::lock_guard<std::mutex> launching(ws->launching);
                if (ws->buf.defined()) list.emplace_back(key, ws->buf);
            }
        }
        PyObject* out = PyDict_New();
        if (!out) throw python_error();
        for (const auto& [key, buf] : list) {
            PyObject* k = Py_BuildValue("(iL)", key.first, static_cast<long long>(key.second));
            PyObject* v = wrap(buf);
            if (k && v) PyDict_SetItem(out, k, v);
            Py_XDECREF(k);
            Py_XDECREF(v);
        }
        return out;
    });
}

// ([(start, stop), ...] forward, the same for backward): CUDA event handles, consumed one pair per attention call in call order
PyObject* py_queue_timing_events(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return guarded([&]() -> PyObject* {
        want(n, 2);
        std::deque<std::pair<cudaEvent_t, cudaEvent_t>> queues[2];      // filled first: reading a sequence may run Python code, which must not happen under the lock
        for (int i = 0; i < 2; ++i) {
            auto& q = queues[i];
            PyObject* seq = PySequence_Fast(a[i], "expected a sequence of event pairs");
            if (!seq) throw python_error();
            for (Py_ssize_t j = 0; j < PySequence_Fast_GET_SIZE(seq); ++j) {
                unsigned long long e0 = 0, e1 = 0;
                if (!PyArg_ParseTuple(PySequence_Fast_GET_ITEM(seq, j), "KK", &e0, &e1)) {
                    Py_DECREF(seq);
                    throw python_error();
                }
                q.emplace_back(reinterpret_cast<cudaEvent_t>(e0), reinterpret_cast<cudaEvent_t>(e1));
            }
            Py_DECREF(seq);
        }
        std::lock_guard<std::mutex> lock(g_timing.m);
        g_timing.fwd.swap(queues[0]);
        g_timing.bwd.swap(queues[1]);
        g_timing.any = !g_timing.fwd.empty() || !g_timing.bwd.empty();
        Py_RETURN_NONE;
    });
}

#define IB200_PY(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_##name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {IB200_PY(bind),
                           IB200_PY(attention_forward),
                           IB200_PY(attention_backward),
                           IB200_PY(causal_attention),
                           IB200_PY(causal_attention_packed),
                           IB200_PY(linear),
                           IB200_PY(linear_forward),
                           IB200_PY(linear_backward),
                           IB200_PY(workspaces),
                           IB200_PY(queue_timing_events),
                           {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_host_ops", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_ops() {
    PyObject* m = PyModule_Create(&g_module);
    // the torch whose classes this module was compiled against
    if (m && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) {
        Py_DECREF(m);
        return nullptr;
    }
    return m;
}

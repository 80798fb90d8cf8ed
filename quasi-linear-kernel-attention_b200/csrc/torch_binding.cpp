// The operators on torch tensors: argument checks, workspaces and outputs from torch's caching allocator, the current stream,
// and the autograd nodes, over the C ABI of include/qlka.h (whose functions are looked up in the library that qlka_native.py
// names). A call through ctypes and Python's autograd spends 20 us (a training step of attention 500 us and more) on the host,
// more than the kernels of a short sequence take.
//
// Checks and messages follow the reference's host code (Weighted_Laplace_Sum/csrc/binding.cpp:66-79,
// Weighted_Abs_Sum/csrc/binding.cpp:69-84, :251-262, :387-392).
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>

#include <dlfcn.h>

#include "../../include/qlka.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;

struct Api {
#define QLKA_FN(name) decltype(&::name) name = nullptr
    QLKA_FN(qlka_status_string);
    QLKA_FN(qlka_last_cuda_error);
    QLKA_FN(qlka_laplace_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_laplace_sum_forward);
    QLKA_FN(qlka_laplace_backward_workspace_bytes);
    QLKA_FN(qlka_weighted_laplace_sum_backward);
    QLKA_FN(qlka_abs_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_abs_sum_forward);
    QLKA_FN(qlka_abs_backward_workspace_bytes);
    QLKA_FN(qlka_weighted_abs_sum_backward);
    QLKA_FN(qlka_sgn_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_sgn_sum_forward);
    QLKA_FN(qlka_attention_workspace_bytes);
    QLKA_FN(qlka_attention_forward);
    QLKA_FN(qlka_attention_backward_workspace_bytes);
    QLKA_FN(qlka_attention_backward);
    QLKA_FN(qlka_linear_workspace_bytes);
    QLKA_FN(qlka_split_rows);
    QLKA_FN(qlka_split_heads);
    QLKA_FN(qlka_linear_qkv);
    QLKA_FN(qlka_linear_gelu);
    QLKA_FN(qlka_linear_residual);
    QLKA_FN(qlka_linear_error);
#undef QLKA_FN
} api;

void load(const std::string& path) {
    void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(h, "cannot load ", path, ": ", dlerror());
#define QLKA_FN(name)                                                       \
    api.name = reinterpret_cast<decltype(api.name)>(dlsym(h, #name));      \
    TORCH_CHECK(api.name, path, " has no ", #name)
    QLKA_FN(qlka_status_string);
    QLKA_FN(qlka_last_cuda_error);
    QLKA_FN(qlka_laplace_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_laplace_sum_forward);
    QLKA_FN(qlka_laplace_backward_workspace_bytes);
    QLKA_FN(qlka_weighted_laplace_sum_backward);
    QLKA_FN(qlka_abs_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_abs_sum_forward);
    QLKA_FN(qlka_abs_backward_workspace_bytes);
    QLKA_FN(qlka_weighted_abs_sum_backward);
    QLKA_FN(qlka_sgn_forward_workspace_bytes);
    QLKA_FN(qlka_weighted_sgn_sum_forward);
    QLKA_FN(qlka_attention_workspace_bytes);
    QLKA_FN(qlka_attention_forward);
    QLKA_FN(qlka_attention_backward_workspace_bytes);
    QLKA_FN(qlka_attention_backward);
    QLKA_FN(qlka_linear_workspace_bytes);
    QLKA_FN(qlka_split_rows);
    QLKA_FN(qlka_split_heads);
    QLKA_FN(qlka_linear_qkv);
    QLKA_FN(qlka_linear_gelu);
    QLKA_FN(qlka_linear_residual);
    QLKA_FN(qlka_linear_error);
#undef QLKA_FN
}

void check_status(const int st) {
    if (st == QLKA_OK) return;
    if (st == QLKA_ERR_CUDA) TORCH_CHECK(false, api.qlka_status_string(st), " (cudaError ", api.qlka_last_cuda_error(), ")");
    TORCH_CHECK(false, api.qlka_status_string(st));
}

qlka_stream_t current_stream() { return reinterpret_cast<qlka_stream_t>(at::cuda::getCurrentCUDAStream().stream()); }

struct Dims { int P, D, N, M, C; };

Dims check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, const char* names) {
    TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda(), names, " must be CUDA tensors");
    TORCH_CHECK(q.device() == k.device() && q.device() == v.device(), names, " must be on one device");
    TORCH_CHECK(q.scalar_type() == at::kFloat && k.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat, names, " must be float32");
    TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, names, " must be 3D");
    TORCH_CHECK(q.size(0) == k.size(0) && q.size(0) == v.size(0), "batch size must match");
    TORCH_CHECK(q.size(1) == k.size(1), "q and k must have the same feature dimension");
    TORCH_CHECK(k.size(2) == v.size(1), "k and v must have the same length");
    TORCH_CHECK(q.is_contiguous() && k.is_contiguous() && v.is_contiguous(), names, " must be contiguous");
    auto fits = [](const int64_t x) { TORCH_CHECK(x <= INT_MAX, "P*D*max(N,M) must fit int32 (cub sort offsets)"); return (int)x; };
    return {fits(q.size(0)), fits(q.size(1)), fits(k.size(2)), fits(q.size(2)), fits(v.size(2))};
}

void check_like(const Tensor& t, const char* name, const at::IntArrayRef shape, const Tensor& q) {
    TORCH_CHECK(t.is_cuda() && t.device() == q.device(), name, " must be on q's CUDA device");
    TORCH_CHECK(t.scalar_type() == at::kFloat, name, " must be float32");
    TORCH_CHECK(t.sizes() == shape, name, " must have shape ", shape);
    TORCH_CHECK(t.is_contiguous(), name, " must be contiguous");
}

// The row matrices must start on a 16-byte boundary; a contiguous view at an odd storage offset is copied once instead of being
// refused, as the reference accepts any contiguous tensor.
Tensor aligned(const Tensor& t) {
    return (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) == 0 ? t : t.clone(at::MemoryFormat::Contiguous);
}

const float* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr<float>() : nullptr; }
float* out_ptr(const Tensor& t) { return t.defined() ? t.mutable_data_ptr<float>() : nullptr; }

Tensor floats(const at::IntArrayRef shape, const Tensor& like) {
    return at::detail::empty_cuda(shape, at::kFloat, like.device(), std::nullopt);
}

// call(workspace, bytes) with a workspace of the size that `size` gives for these dimensions. Where the device has not that much left, the call is
// offered less and less: most take some, and go over their heads in pieces. What none takes is the allocator's error.
template <class Size, class... Args, class Call>
void with_workspace(const Tensor& like, Call call, Size size, Args... dims) {
    size_t bytes = 0;
    check_status(size(dims..., &bytes));
    std::exception_ptr refused;
    for (const int sixteenths : {16, 15, 14, 12, 8, 4, 2, 1}) {
        const size_t have = bytes / 16 * sixteenths + (sixteenths == 16 ? bytes % 16 : 0);
        Tensor ws;
        try {
            ws = at::detail::empty_cuda({(int64_t)std::max<size_t>(have, 256)}, at::kByte, like.device(), std::nullopt);
        } catch (const c10::OutOfMemoryError&) {
            if (!refused) refused = std::current_exception();
            continue;
        }
        const int st = call(ws.mutable_data_ptr(), have);
        if (refused && st == QLKA_ERR_WORKSPACE) break;
        return check_status(st);
    }
    std::rethrow_exception(refused);
}

// ------------------------------------------------------------------ operators
std::tuple<Tensor, Tensor> laplace_forward(const Tensor& q, const Tensor& k, const Tensor& v_) {
    const Dims d = check_qkv(q, k, v_, "q, k and v");
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor v = aligned(v_);
    Tensor out_w = floats({d.P, d.M, d.C}, q), out_u = floats({d.P, d.M}, q);
    with_workspace(q, [&](void* ws, size_t bytes) {
        return api.qlka_weighted_laplace_sum_forward(ptr(q), ptr(k), ptr(v), out_ptr(out_w), out_ptr(out_u), ws, bytes, d.P, d.D, d.N, d.M, d.C, current_stream());
    }, api.qlka_laplace_forward_workspace_bytes, d.P, d.D, d.N, d.M, d.C);
    return {out_w, out_u};
}

template <class Size, class Call>
std::tuple<Tensor, Tensor, Tensor> backward(Size size, Call call, const Tensor& q, const Tensor& k, const Tensor& v_, const Tensor& g_w_, const Tensor& g_u) {
    const Dims d = check_qkv(q, k, v_, "q, k, and v");
    check_like(g_w_, "g_w", {d.P, d.M, d.C}, q);
    if (g_u.defined()) check_like(g_u, "g_u", {d.P, d.M}, q);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor v = aligned(v_), g_w = aligned(g_w_);
    Tensor gq = floats({d.P, d.D, d.M}, q), gk = floats({d.P, d.D, d.N}, q), gv = floats({d.P, d.N, d.C}, q);
    with_workspace(q, [&](void* ws, size_t bytes) {
        return call(ptr(q), ptr(k), ptr(v), ptr(g_w), ptr(g_u), out_ptr(gq), out_ptr(gk), out_ptr(gv), ws, bytes, d.P, d.D, d.N, d.M, d.C, current_stream());
    }, size, d.P, d.D, d.N, d.M, d.C);
    return {gq, gk, gv};
}

std::tuple<Tensor, Tensor, Tensor> laplace_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_w, const std::optional<Tensor>& g_u) {
    return backward(api.qlka_laplace_backward_workspace_bytes, api.qlka_weighted_laplace_sum_backward, q, k, v, g_w, g_u.value_or(Tensor()));
}

std::tuple<Tensor, Tensor, Tensor> abs_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_w, const std::optional<Tensor>& g_u) {
    return backward(api.qlka_abs_backward_workspace_bytes, api.qlka_weighted_abs_sum_backward, q, k, v, g_w, g_u.value_or(Tensor()));
}

std::tuple<Tensor, std::optional<Tensor>> abs_forward(const Tensor& q, const Tensor& k, const Tensor& v_, const bool full, const int64_t path) {
    const Dims d = check_qkv(q, k, v_, "q, k, and v");
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor v = aligned(v_);
    Tensor out_w = floats({d.P, d.M, d.C}, q), out_u;
    if (full) out_u = floats({d.P, d.M}, q);
    with_workspace(q, [&](void* ws, size_t bytes) {
        return api.qlka_weighted_abs_sum_forward(ptr(q), ptr(k), ptr(v), out_ptr(out_w), out_ptr(out_u), ws, bytes, d.P, d.D, d.N, d.M, d.C, (int)path, current_stream());
    }, api.qlka_abs_forward_workspace_bytes, d.P, d.D, d.N, d.M, d.C);
    return {out_w, full ? std::optional<Tensor>(out_u) : std::nullopt};
}

Tensor sgn_forward(const Tensor& q, const Tensor& k, const Tensor& v_, const Tensor& g_) {
    const Dims d = check_qkv(q, k, v_, "q, k, and v");
    check_like(g_, "g", {d.P, d.M, d.C}, q);
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor v = aligned(v_), g = aligned(g_);
    Tensor out = floats({d.P, d.D, d.M}, q);
    with_workspace(q, [&](void* ws, size_t bytes) {
        return api.qlka_weighted_sgn_sum_forward(ptr(q), ptr(k), ptr(v), ptr(g), out_ptr(out), ws, bytes, d.P, d.D, d.N, d.M, d.C, current_stream());
    }, api.qlka_sgn_forward_workspace_bytes, d.P, d.D, d.N, d.M, d.C);
    return out;
}

// ------------------------------------------------------------------ autograd of the operators
class LaplaceSum : public torch::autograd::Function<LaplaceSum> {
public:
    static tensor_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v) {
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({q, k, v});
        auto [w, u] = laplace_forward(q, k, v);
        return {w, u};
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        if (!g[0].defined() && !g[1].defined()) return {Tensor(), Tensor(), Tensor()};
        const auto s = ctx->get_saved_variables();
        const Tensor g_w = g[0].defined() ? g[0].contiguous() : at::zeros({s[0].size(0), s[0].size(2), s[2].size(2)}, s[0].options());
        auto [gq, gk, gv] = ::backward(api.qlka_laplace_backward_workspace_bytes, api.qlka_weighted_laplace_sum_backward, s[0], s[1], s[2],
                                       g_w, g[1].defined() ? g[1].contiguous() : g[1]);
        return {gq, gk, gv};
    }
};

class AbsSum : public torch::autograd::Function<AbsSum> {
public:
    static tensor_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const bool full, const int64_t path) {
        ctx->set_materialize_grads(false);
        ctx->save_for_backward({q, k, v});
        auto [w, u] = abs_forward(q, k, v, full, path);
        if (full) return {w, *u};
        return {w};
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        const bool with_u = g.size() > 1 && g[1].defined();
        if (!g[0].defined() && !with_u) return {Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
        const auto s = ctx->get_saved_variables();
        // (nothing flowed back into the row sums: the native call skips their scalar terms)
        const Tensor g_w = g[0].defined() ? g[0].contiguous() : at::zeros({s[0].size(0), s[0].size(2), s[2].size(2)}, s[0].options());
        auto [gq, gk, gv] = ::backward(api.qlka_abs_backward_workspace_bytes, api.qlka_weighted_abs_sum_backward, s[0], s[1], s[2],
                                       g_w, with_u ? g[1].contiguous() : Tensor());
        return {gq, gk, gv, Tensor(), Tensor()};
    }
};

// Whether a call has to go through its autograd node. Forward-mode tangents do too: the nodes have no rule for them and say so.
bool wants_grad(const Tensor& q, const Tensor& k, const Tensor& v) {
    auto dual = [](const Tensor& t) { return t._fw_grad(/*level=*/0).defined(); };
    return (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) || dual(q) || dual(k) || dual(v);
}

std::tuple<Tensor, Tensor> laplace_sum(const Tensor& q, const Tensor& k, const Tensor& v) {
    if (!wants_grad(q, k, v)) return laplace_forward(q, k, v);
    auto out = LaplaceSum::apply(q, k, v);
    return {out[0], out[1]};
}

std::vector<Tensor> abs_sum(const Tensor& q, const Tensor& k, const Tensor& v, const bool full, const int64_t path) {
    if (!wants_grad(q, k, v)) {
        auto [w, u] = abs_forward(q, k, v, full, path);
        if (full) return {w, *u};
        return {w};
    }
    return AbsSum::apply(q, k, v, full, path);
}

// ------------------------------------------------------------------ attention on (B, H, S, D)
struct AttnDims { int B, H, S, D, C; };

AttnDims check_attention(const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& keep) {
    TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda(), "q, k, and v must be CUDA tensors");
    TORCH_CHECK(q.device() == k.device() && q.device() == v.device(), "q, k, and v must be on one device");
    TORCH_CHECK(q.scalar_type() == at::kFloat && k.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat, "q, k, and v must be float32");
    TORCH_CHECK(q.dim() == 4 && k.sizes() == q.sizes() && v.dim() == 4 && v.sizes().slice(0, 3) == q.sizes().slice(0, 3),
                "expected q, k (B, H, S, D) and v (B, H, S, Dv)");
    if (keep) TORCH_CHECK(keep->dim() == 2 && keep->size(0) == q.size(0) && keep->size(1) == q.size(2), "keep must be (B, S)");
    for (const int64_t x : {q.size(0), q.size(1), q.size(2), q.size(3), v.size(3)}) TORCH_CHECK(x <= INT_MAX, "P*D*max(N,M) must fit int32 (cub sort offsets)");
    return {(int)q.size(0), (int)q.size(1), (int)q.size(2), (int)q.size(3), (int)v.size(3)};
}

Tensor keep_floats(const std::optional<Tensor>& keep, const Tensor& q) {
    return keep ? keep->to(q.device(), at::kFloat).contiguous() : Tensor();
}

Tensor attention_forward(const int64_t kind, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& keep, const double tau, const AttnDims& d, Tensor* den) {
    Tensor out = floats({d.B, d.H, d.S, d.C}, q);
    if (den) *den = floats({d.B, d.H, d.S}, q);
    with_workspace(q, [&](void* ws, size_t bytes) {
        return api.qlka_attention_forward((int)kind, ptr(q), ptr(k), ptr(v), ptr(keep), (float)tau, out_ptr(out), den ? out_ptr(*den) : nullptr,
                                          ws, bytes, d.B, d.H, d.S, d.D, d.C, current_stream());
    }, api.qlka_attention_workspace_bytes, (int)kind, d.B, d.H, d.S, d.D, d.C, (int)keep.defined());
    return out;
}

// The output's version when the forward pass ended, without its memory.
struct OutputVersion : torch::CustomClassHolder {
    c10::VariableVersion counter;
    const uint32_t       at;
    explicit OutputVersion(const Tensor& out) : counter(out.unsafeGetTensorImpl()->version_counter()), at(counter.current_version()) {}
    bool changed() const { return counter.current_version() != at; }
};

class Attention : public torch::autograd::Function<Attention> {
public:
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const std::optional<Tensor>& mask, const int64_t kind, const double tau) {
        const Tensor keep = mask.value_or(Tensor());
        const AttnDims d{(int)q.size(0), (int)q.size(1), (int)q.size(2), (int)q.size(3), (int)v.size(3)};
        Tensor den;
        Tensor out = attention_forward(kind, q, k, v, keep, tau, d, &den);
        // The gradient needs the output, but a caller may change it in place, as after any division. So it is saved with a version of
        // its own, which no such change fails on, and computed again by the backward pass if there was one.
        ctx->save_for_backward({q, k, v, keep, out.variable_data(), den});
        ctx->saved_data["out"]  = c10::IValue::make_capsule(c10::make_intrusive<OutputVersion>(out));
        ctx->saved_data["kind"] = kind;
        ctx->saved_data["tau"]  = tau;
        return out;
    }
    static tensor_list backward(AutogradContext* ctx, tensor_list g) {
        const auto s = ctx->get_saved_variables();
        // (hooks on saved tensors may hand back other tensors: any strides, any place)
        const int kind = (int)ctx->saved_data["kind"].toInt();
        const AttnDims d = check_attention(s[0], s[1], s[2], s[3].defined() ? std::optional<Tensor>(s[3]) : std::nullopt);
        const c10::cuda::CUDAGuard guard(s[0].device());
        const Tensor q = s[0].contiguous(), k = s[1].contiguous(), v = aligned(s[2].contiguous()), keep = s[3].defined() ? s[3].contiguous() : s[3];
        const Tensor saved_out = aligned(s[4].contiguous()), den = s[5].contiguous();
        if (keep.defined()) check_like(keep, "keep", {d.B, d.S}, q);
        check_like(saved_out, "the saved output", {d.B, d.H, d.S, d.C}, q);
        check_like(den, "the saved row sums", {d.B, d.H, d.S}, q);
        const Tensor grad = aligned(g[0].contiguous());
        const double tau = ctx->saved_data["tau"].toDouble();
        const bool   changed = static_cast<const OutputVersion*>(ctx->saved_data["out"].toCapsule().get())->changed();
        const Tensor out = changed ? attention_forward(kind, q, k, v, keep, tau, d, nullptr) : saved_out;
        Tensor gq = floats(q.sizes(), q), gk = floats(k.sizes(), q), gv = floats(v.sizes(), q);
        with_workspace(q, [&](void* ws, size_t bytes) {
            return api.qlka_attention_backward(kind, ptr(q), ptr(k), ptr(v), ptr(keep), (float)tau, ptr(out), ptr(den), ptr(grad),
                                               out_ptr(gq), out_ptr(gk), out_ptr(gv), ws, bytes, d.B, d.H, d.S, d.D, d.C, current_stream());
        }, api.qlka_attention_backward_workspace_bytes, kind, d.B, d.H, d.S, d.D, d.C, (int)keep.defined());
        return {gq, gk, gv, Tensor(), Tensor(), Tensor()};
    }
};

// The attention, differentiable where an input asks for it. None where a gradient is wanted that has no single native call.
std::optional<Tensor> attention(const int64_t kind, const Tensor& q_, const Tensor& k_, const Tensor& v_, const double tau, const std::optional<Tensor>& keep_) {
    const AttnDims d = check_attention(q_, k_, v_, keep_);
    const c10::cuda::CUDAGuard guard(q_.device());
    const bool grad = wants_grad(q_, k_, v_);
    if (grad) {
        size_t bytes = 0;
        const int st = api.qlka_attention_backward_workspace_bytes((int)kind, d.B, d.H, d.S, d.D, d.C, (int)keep_.has_value(), &bytes);
        if (st == QLKA_ERR_UNSUPPORTED) return std::nullopt;
        check_status(st);
    }
    const Tensor q = q_.contiguous(), k = k_.contiguous(), v = aligned(v_.contiguous()), keep = keep_floats(keep_, q_);
    if (!grad) return attention_forward(kind, q, k, v, keep, tau, d, nullptr);
    return Attention::apply(q, k, v, keep.defined() ? std::optional<Tensor>(keep) : std::nullopt, kind, tau);
}

// ------------------------------------------------------------------ linear layers of the encoder (inference)
void check_matrix(const Tensor& t, const char* name, const at::IntArrayRef shape, const Tensor& like) {
    TORCH_CHECK(t.is_cuda() && t.device() == like.device() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.sizes() == shape,
                name, " must be a contiguous float32 CUDA tensor of shape ", shape, " on the input's device");
}

Tensor parts_of(const int64_t rows, const int64_t K, const Tensor& like) { return at::detail::empty_cuda({3, rows, K}, at::kBFloat16, like.device(), std::nullopt); }

Tensor split_rows(const Tensor& x, const Tensor& ln_weight, const Tensor& ln_bias, const double eps) {
    const int64_t rows = x.size(0), K = x.size(1);
    check_matrix(x, "x", {rows, K}, x);
    check_matrix(ln_weight, "ln_weight", {K}, x);
    check_matrix(ln_bias, "ln_bias", {K}, x);
    const c10::cuda::CUDAGuard guard(x.device());
    Tensor parts = parts_of(rows, K, x);
    check_status(api.qlka_split_rows(ptr(x), ptr(ln_weight), ptr(ln_bias), (float)eps, parts.mutable_data_ptr(), (int)rows, (int)K, current_stream()));
    return parts;
}

Tensor split_heads(const Tensor& o) {
    const int64_t B = o.size(0), H = o.size(1), S = o.size(2), D = o.size(3);
    check_matrix(o, "o", {B, H, S, D}, o);
    const c10::cuda::CUDAGuard guard(o.device());
    Tensor parts = parts_of(B * S, H * D, o);
    check_status(api.qlka_split_heads(ptr(o), parts.mutable_data_ptr(), (int)B, (int)H, (int)S, (int)D, current_stream()));
    return parts;
}

struct Layer { int M, N, K; Tensor ws; size_t bytes; };
Layer layer(const Tensor& parts, const Tensor& weight, const Tensor& bias) {
    TORCH_CHECK(parts.is_cuda() && parts.scalar_type() == at::kBFloat16 && parts.is_contiguous() && parts.dim() == 3 && parts.size(0) == 3, "parts must come from split_rows or split_heads");
    const int64_t M = parts.size(1), K = parts.size(2), N = weight.size(0);
    check_matrix(weight, "weight", {N, K}, parts);
    check_matrix(bias, "bias", {N}, parts);
    Layer l{(int)M, (int)N, (int)K, Tensor(), api.qlka_linear_workspace_bytes((int)N, (int)K)};
    l.ws = at::detail::empty_cuda({(int64_t)l.bytes}, at::kByte, parts.device(), std::nullopt);
    return l;
}

std::tuple<Tensor, Tensor, Tensor> linear_qkv(const Tensor& parts, const Tensor& weight, const Tensor& bias, const Tensor& table, const int64_t B, const int64_t S, const int64_t H) {
    const c10::cuda::CUDAGuard guard(parts.device());
    const Layer l = layer(parts, weight, bias);
    TORCH_CHECK(l.M == B * S && l.N == 3 * H * 64, "expected B * S rows and 3 * H * 64 columns");
    check_matrix(table, "table", {S, 32, 2}, parts);
    Tensor q = floats({B, H, S, 64}, parts), k = floats({B, H, S, 64}, parts), v = floats({B, H, S, 64}, parts);
    check_status(api.qlka_linear_qkv(parts.const_data_ptr(), ptr(weight), ptr(bias), ptr(table), out_ptr(q), out_ptr(k), out_ptr(v),
                                     l.ws.mutable_data_ptr(), l.bytes, (int)B, (int)S, (int)H, l.K, current_stream()));
    return {q, k, v};
}

Tensor linear_gelu(const Tensor& parts, const Tensor& weight, const Tensor& bias) {
    const c10::cuda::CUDAGuard guard(parts.device());
    const Layer l = layer(parts, weight, bias);
    Tensor out = parts_of(l.M, l.N, parts);
    check_status(api.qlka_linear_gelu(parts.const_data_ptr(), ptr(weight), ptr(bias), out.mutable_data_ptr(), l.ws.mutable_data_ptr(), l.bytes, l.M, l.N, l.K, current_stream()));
    return out;
}

void linear_residual(const Tensor& parts, const Tensor& weight, const Tensor& bias, const Tensor& x) {
    const c10::cuda::CUDAGuard guard(parts.device());
    const Layer l = layer(parts, weight, bias);
    check_matrix(x, "x", {l.M, l.N}, parts);
    check_status(api.qlka_linear_residual(parts.const_data_ptr(), ptr(weight), ptr(bias), out_ptr(x), l.ws.mutable_data_ptr(), l.bytes, l.M, l.N, l.K, current_stream()));
}

int linear_error() {
    int e = 0;
    check_status(api.qlka_linear_error(&e));
    return e;
}

}  // namespace

// Every call that enqueues work lets go of Python's lock: a launch can wait for room in its stream's queue, and other threads drive
// other streams and GPUs.
PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    using Unlocked = py::call_guard<py::gil_scoped_release>;
    m.def("load", &load);
    m.def("laplace_forward", &laplace_forward, Unlocked());
    m.def("laplace_backward", &laplace_backward, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("g_w"), py::arg("g_u") = py::none(), Unlocked());
    m.def("laplace_sum", &laplace_sum, Unlocked());
    m.def("abs_forward", &abs_forward, Unlocked());
    m.def("abs_backward", &abs_backward, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("g_w"), py::arg("g_u") = py::none(), Unlocked());
    m.def("abs_sum", &abs_sum, Unlocked());
    m.def("sgn_forward", &sgn_forward, Unlocked());
    m.def("attention", &attention, Unlocked());
    m.def("split_rows", &split_rows, Unlocked());
    m.def("split_heads", &split_heads, Unlocked());
    m.def("linear_qkv", &linear_qkv, Unlocked());
    m.def("linear_gelu", &linear_gelu, Unlocked());
    m.def("linear_residual", &linear_residual, Unlocked());
    m.def("linear_error", &linear_error, Unlocked());
}

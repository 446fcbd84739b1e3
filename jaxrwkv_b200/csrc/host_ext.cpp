// Native host path of the operators: argument checks, result allocation, the autograd nodes and the calls into
// libb200wkv.so without the Python interpreter in between.
//
// A call through torch.autograd.Function in Python costs 80-100 us forward and 350 us for a forward and backward,
// a ctypes call of a decoding step 30 us: more than most kernels behind them.  The same work from C++ costs a
// few microseconds per call.  Every function here returns None when it is handed something out of the ordinary
// (arguments that are no plain tensors or carry a tangent, a functorch transform, a dispatch mode or a tracer in force,
// shapes or types that do not fit); the Python functions that call them then take their own path, which handles vmap
// and raises the errors.
#include <torch/csrc/python_headers.h>

#include <array>
#include <functional>
#include <memory>
#include <unordered_map>

#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "../../include/b200wkv.h"
#include "host_calls.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

PyObject* g_error_class = nullptr;   // jaxrwkv_b200._lib.B200WKVError

[[noreturn]] void raise(const std::string& msg) {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(g_error_class ? g_error_class : PyExc_RuntimeError, msg.c_str());
    python_error e;
    e.persist();
    throw e;
}
void check(int status) {
    if (status != B200WKV_OK)
        raise(std::string("b200wkv: ") + b200wkv_strerror(status) + " (status " + std::to_string(status) + ")");
}

void cuda_check(cudaError_t e) {
    if (e != cudaSuccess) raise(std::string("b200wkv: ") + cudaGetErrorString(e));
}

const void* in(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* out(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }
Tensor bytes(size_t n, const Tensor& like) { return fresh({(int64_t)n}, at::kByte, like); }
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? B200WKV_F32 : B200WKV_BF16; }
cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// The plain case: no functorch transform, no dispatch mode, nothing that records a trace.
bool plain_mode() {
    static const c10::DispatchKeySet special({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::Tracer});
    return (c10::impl::tls_local_dispatch_key_set().included_ & special).empty() && !c10::impl::dispatch_mode_enabled();
}
// A dual tensor of forward-mode differentiation: what runs below the dispatcher would drop its tangent without a word.
bool has_tangent(const Tensor& t) {
    // (the general look takes a lock; most tensors have no autograd record, or one without any tangent that is no view's)
    const auto* const meta = torch::autograd::impl::get_autograd_meta(t);
    return meta != nullptr && (meta->fw_grad_ != nullptr || meta->is_view_) && t._fw_grad(/*level=*/0).defined();
}
// One floating type the kernels know, one CUDA device, contiguous enough to be made so by contiguous().
bool same_kind(const Tensor* t, int n) {
    const auto type = t[0].scalar_type();
    if (type != at::kFloat && type != at::kBFloat16) return false;
    for (int i = 0; i < n; ++i)
        if (!t[i].is_cuda() || t[i].scalar_type() != type || t[i].device() != t[0].device() || t[i].layout() != at::kStrided ||
            t[i].numel() == 0)
            return false;
    return true;
}
bool any_grad(const Tensor* t, int n) {
    if (!at::GradMode::is_enabled()) return false;
    for (int i = 0; i < n; ++i)
        if (t[i].requires_grad()) return true;
    return false;
}
bool any_grad_defined(const Tensor* t, int n) {
    for (int i = 0; i < n; ++i)
        if (t[i].defined() && any_grad(t + i, 1)) return true;
    return false;
}
bool sizes_are(const Tensor& t, at::IntArrayRef lead, std::initializer_list<int64_t> tail) {
    if (t.dim() != (int64_t)(lead.size() + tail.size())) return false;
    size_t i = 0;
    for (int64_t d : lead)
        if (t.size(i++) != d) return false;
    for (int64_t d : tail)
        if (t.size(i++) != d) return false;
    return true;
}

// `length` as (lead) 32-bit words and `new_starts` as (lead, T) bytes; both may be shared by leading axes.
struct Flags {
    Tensor length, starts;
    Flags(const Tensor& len, const Tensor& ns, at::IntArrayRef lead, int64_t T, const Tensor& like) {
        length = len;
        if (!(len.scalar_type() == at::kInt && len.device() == like.device() && len.sizes() == lead && len.is_contiguous()))
            length = len.to(like.device()).expand(lead).to(at::kInt).contiguous();
        std::vector<int64_t> shape(lead.begin(), lead.end());
        shape.push_back(T);
        starts = ns;
        if (!((ns.scalar_type() == at::kByte || ns.scalar_type() == at::kBool) && ns.device() == like.device() &&
              ns.sizes() == at::IntArrayRef(shape) && ns.is_contiguous())) {
            starts = ns.to(like.device());
            if (starts.scalar_type() != at::kBool) starts = starts.to(at::kByte);
            starts = starts.expand(shape).contiguous();
        }
    }
};

// Dense and where the widest accesses fit: a contiguous view may begin anywhere.
bool on_16_bytes(const Tensor& t) { return (uintptr_t)in(t) % 16 == 0; }
Tensor dense(const Tensor& t) {
    const Tensor c = t.contiguous();
    return on_16_bytes(c) ? c : c.clone(at::MemoryFormat::Contiguous);
}
// A cotangent as the kernels read it (autograd hands in slices of larger ones, such as a concatenation's); an undefined one stays
// undefined (the kernels take NULL for zero).
Tensor cotangent(const Tensor& g, const Tensor& like) {
    return !g.defined() ? g : dense(g.scalar_type() == like.scalar_type() ? g : g.to(like.scalar_type()));
}

// What stands for an optional operand that is not there: an autograd node's arguments have to be defined.
Tensor nothing(const Tensor& like) { return fresh({0}, like.scalar_type(), like); }
Tensor if_any(const Tensor& t) { return t.defined() && t.numel() > 0 ? t : Tensor(); }

// Gradients asked for with create_graph=True: the values are right, differentiating them again is an error.
struct Refuse : public torch::autograd::Function<Refuse> {
    static variable_list forward(AutogradContext* ctx, at::TensorList from, const std::function<variable_list()>& compute, std::string name) {
        ctx->saved_data["name"] = name;
        return compute();
    }
    static variable_list backward(AutogradContext* ctx, variable_list) {
        raise(ctx->saved_data["name"].toStringRef() + ": second-order differentiation is not supported");
    }
};
variable_list once_differentiable(const char* name, const variable_list& saved, const variable_list& grads,
                                  const std::function<variable_list()>& compute) {
    if (!at::GradMode::is_enabled()) return compute();
    variable_list from;                           // a node's inputs have to be defined
    for (const variable_list* l : {&saved, &grads})
        for (const Tensor& t : *l)
            if (t.defined()) from.push_back(t);
    return Refuse::apply(at::TensorList(from), compute, std::string(name));
}
template <class Op>
variable_list gradients_of(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    return once_differentiable(Op::kName, saved, grads, [&]() { return Op::gradients(saved, grads); });
}

// ------------------------------------------------------------------------------------------------- RWKV-7
// Streams (lead, T, H, N), state (lead, H, N, N), any number of leading batch axes.
// `n` bytes, or an undefined tensor where the device has no room for them
static Tensor bytes_if_room(size_t n, const Tensor& like) {
    try {
        return bytes(n, like);
    } catch (const c10::OutOfMemoryError&) {
        return Tensor();
    }
}
// What a forward call wants beside its results: a workspace until it is enqueued, and, where asked for, what its backward reads.  Without
// room for the one or the other (up to 2 GiB; 16 and 20 KB per 16 tokens and head in fp32) there are kernels that need less.
struct Wkv7Room {
    Tensor workspace, residual;
    size_t residual_bytes = 0;
    Wkv7Room(const Tensor& like, int B, int T, int H, int N, bool keep) {
        const int code = dtype_code(like);
        const bool known = N == 64 && B > 0 && T > 0 && H > 0;       // (the call says what is wrong with others)
        const size_t n = known && T > 1 ? b200wkv::wkv7_workspace_bytes(code, B, T, H, keep) : 0;
        if (n != 0) workspace = bytes_if_room(n, like);
        if (!keep) return;
        const auto fits = [&](size_t size) {
            residual_bytes = size;
            return (residual = bytes_if_room(size, like)).defined();
        };
        const size_t least = b200wkv7_residual_min_bytes(code, B, T, H, N);
        if (known && fits(b200wkv::wkv7_kept_bytes(code, B, T, H, workspace.defined()))) return;
        workspace.reset();
        if (known && fits(b200wkv::wkv7_kept_bytes(code, B, T, H, false))) return;
        residual_bytes = least;
        residual = bytes(least, like);
    }
    void* ws() const { return workspace.defined() ? workspace.mutable_data_ptr() : nullptr; }
};
static Tensor wkv7_bwd_workspace(const Tensor& like, int B, int T, int H, const Tensor& residual) {
    const size_t n = b200wkv::wkv7_bwd_workspace_bytes(dtype_code(like), B, T, H, (size_t)residual.numel());
    return n != 0 ? bytes_if_room(n, like) : Tensor();               // (without it a sequence is walked in longer runs)
}

struct Wkv7 {
    static constexpr const char* kName = "wkv7";
    static constexpr int kIn = 7;                 // r w k v a b s

    static bool fits(const Tensor* t) {
        if (!same_kind(t, kIn) || t[2].dim() < 3) return false;
        for (int i : {0, 1, 3, 4, 5})
            if (!t[i].sizes().equals(t[2].sizes())) return false;
        const int64_t H = t[2].size(-2), N = t[2].size(-1);
        return sizes_are(t[6], t[2].sizes().slice(0, t[2].dim() - 3), {H, N, N});
    }
    static std::pair<Tensor, Tensor> forward(const Tensor* t, const Tensor& length, const Tensor& starts, Tensor* residual) {
        const Tensor& k = t[2];
        const c10::cuda::CUDAGuard guard(k.device());
        const auto lead = k.sizes().slice(0, k.dim() - 3);
        const int T = (int)k.size(-3), H = (int)k.size(-2), N = (int)k.size(-1), B = (int)c10::multiply_integers(lead);
        const Flags f(length, starts, lead, T, k);
        Tensor c[kIn];
        for (int i = 0; i < kIn; ++i) c[i] = t[i].contiguous();
        Tensor y = fresh_like(k), s_out = fresh_like(t[6]);
        const Wkv7Room room(k, B, T, H, N, residual != nullptr);
        if (residual) *residual = room.residual;
        check(b200wkv::wkv7_fwd(stream_of(k), dtype_code(k), B, T, H, N, in(c[1]), in(c[0]), in(c[2]), in(c[3]), in(c[4]), in(c[5]),
                           in(c[6]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), out(y), out(s_out),
                           out(room.residual), room.residual_bytes, 0, room.ws()));
        return {s_out, y};
    }
    // saved: the seven operands, length, new_starts, residual; grads: of the returned state and of the output
    static variable_list gradients(const variable_list& saved, const variable_list& grads) {
        const Tensor& k = saved[2];
        const c10::cuda::CUDAGuard guard(k.device());
        const auto lead = k.sizes().slice(0, k.dim() - 3);
        const int T = (int)k.size(-3), H = (int)k.size(-2), N = (int)k.size(-1), B = (int)c10::multiply_integers(lead);
        const Flags f(saved[7], saved[8], lead, T, k);
        const Tensor &res = saved[9], gs = cotangent(grads[0], k), gy = cotangent(grads[1], k);
        Tensor c[kIn], g[kIn];
        for (int i = 0; i < kIn; ++i) {
            c[i] = saved[i].contiguous();
            g[i] = fresh_like(saved[i]);
        }
        const Tensor ws = wkv7_bwd_workspace(k, B, T, H, res);
        check(b200wkv::wkv7_bwd(stream_of(k), dtype_code(k), B, T, H, N, in(c[1]), in(c[0]), in(c[2]), in(c[3]), in(c[4]), in(c[5]),
                                in(c[6]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), in(gy), in(gs), out(res),
                                (size_t)res.numel(), out(g[1]), out(g[0]), out(g[2]), out(g[3]), out(g[4]), out(g[5]), out(g[6]), 0, out(ws)));
        return {g[0], g[1], g[2], g[3], g[4], g[5], g[6]};
    }
};

struct Wkv7Node : public torch::autograd::Function<Wkv7Node> {
    static variable_list forward(AutogradContext* ctx, const Tensor& r, const Tensor& w, const Tensor& k, const Tensor& v,
                                 const Tensor& a, const Tensor& b, const Tensor& s, const Tensor& length, const Tensor& starts) {
        const Tensor t[] = {r, w, k, v, a, b, s};
        Tensor residual;
        auto [s_out, y] = Wkv7::forward(t, length, starts, &residual);
        ctx->save_for_backward({r, w, k, v, a, b, s, length, starts, residual});
        ctx->set_materialize_grads(false);
        return {s_out, y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list g = gradients_of<Wkv7>(ctx, grads);
        g.resize(9);
        return g;
    }
};

// ------------------------------------------------------------------------------------------------- RWKV-5 / 5.2 / 6
struct Wkv6Versioned {
    static constexpr int kIn = 6;                 // r k v w u s
    struct Dims {
        at::IntArrayRef lead;
        int B, T, H, N;
        explicit Dims(const Tensor& k) : lead(k.sizes().slice(0, k.dim() - 3)) {
            B = (int)c10::multiply_integers(lead);
            T = (int)k.size(-3); H = (int)k.size(-2); N = (int)k.size(-1);
        }
    };
    static bool fits(bool per_token, const Tensor* t) {
        if (!same_kind(t, kIn) || t[1].dim() < 3) return false;
        const Dims d(t[1]);
        const auto shared = [&](const Tensor& x) { return x.dim() == 3 && x.size(0) == d.H && (x.size(1) == d.N || x.size(1) == 1) && x.size(2) == 1; };
        return t[0].sizes().equals(t[1].sizes()) && t[2].sizes().equals(t[1].sizes()) && shared(t[4]) &&
               (per_token ? sizes_are(t[3], d.lead, {d.T, d.H, d.N, 1}) : shared(t[3])) && sizes_are(t[5], d.lead, {d.H, d.N, d.N});
    }
    // a per-head constant (H, N or 1, 1) as the dense (H, N) array the kernels read
    static Tensor dense_hn(const Tensor& x, const Dims& d) { return x.flatten(1).expand({d.H, d.N}).contiguous(); }
    static void operands(bool per_token, const Tensor* t, const Dims& d, Tensor* c) {
        for (int i : {0, 1, 2, 5}) c[i] = t[i].contiguous();
        c[3] = per_token ? t[3].contiguous() : dense_hn(t[3], d);
        c[4] = dense_hn(t[4], d);
    }
    static std::pair<Tensor, Tensor> forward(bool per_token, const Tensor* t, const Tensor& length, const Tensor& starts,
                                             Tensor* residual) {
        const Tensor& k = t[1];
        const c10::cuda::CUDAGuard guard(k.device());
        const Dims d(k);
        const Flags f(length, starts, d.lead, d.T, k);
        Tensor c[kIn];
        operands(per_token, t, d, c);
        Tensor y = fresh_like(k), s_out = fresh_like(t[5]);
        const size_t rbytes = residual ? b200wkv6_residual_bytes(dtype_code(k), d.B, d.T, d.H, d.N) : 0;
        if (residual) *residual = bytes(rbytes, k);
        // a constant decay (5, 5.2) without gradients: the arithmetic of a training call, with room for the states between its runs
        const size_t wbytes = residual || d.N != 64 ? 0 : b200wkv::wkv6_workspace_bytes(dtype_code(k), per_token, d.B, d.T, d.H);
        const Tensor scratch = wbytes ? bytes(wbytes, k) : Tensor();
        check(b200wkv::wkv6_fwd(stream_of(k), dtype_code(k), per_token ? 6 : 5, d.B, d.T, d.H, d.N, in(c[0]), in(c[1]), in(c[2]),
                                in(c[3]), in(c[4]), in(c[5]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), out(y),
                                out(s_out), residual ? out(*residual) : nullptr, rbytes, 0, wbytes ? out(scratch) : nullptr));
        return {s_out, y};
    }
    static variable_list gradients(bool per_token, const variable_list& saved, const variable_list& grads) {
        const Tensor &k = saved[1], &w = saved[3], &u = saved[4];
        const c10::cuda::CUDAGuard guard(k.device());
        const Dims d(k);
        const Flags f(saved[6], saved[7], d.lead, d.T, k);
        const Tensor &res = saved[8], gs = cotangent(grads[0], k), gy = cotangent(grads[1], k);
        Tensor c[kIn];
        operands(per_token, saved.data(), d, c);
        Tensor gr = fresh_like(k), gk = fresh_like(k), gv = fresh_like(k), gs0 = fresh_like(saved[5]);
        Tensor gw = per_token ? fresh_like(w) : fresh({d.B, d.H, d.N}, at::kFloat, k);
        Tensor gu = fresh({d.B, d.H, d.N}, at::kFloat, k);
        check(b200wkv6_bwd(stream_of(k), dtype_code(k), per_token ? 6 : 5, d.B, d.T, d.H, d.N, in(c[0]), in(c[1]), in(c[2]),
                           in(c[3]), in(c[4]), in(c[5]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), in(gy), in(gs),
                           out(res), (size_t)res.numel(), out(gr), out(gk), out(gv), out(gw), out(gu), out(gs0), 0));
        // gradients of the shared operands: summed over the batch, and over the channels of a per-head constant
        if (u.size(1) == d.N && (per_token || w.size(1) == d.N)) {
            const Tensor du = fresh_like(u), dw = per_token ? gw : fresh_like(w);
            check(b200wkv::wkv6_parameter_grads(stream_of(k), dtype_code(k), d.B, d.H * d.N, per_token ? nullptr : (const float*)in(gw), (const float*)in(gu),
                                                per_token ? nullptr : out(dw), out(du)));
            return {gr, gk, gv, dw, du, gs0};
        }
        const auto shared = [&](const Tensor& g, const Tensor& p) {
            return (p.size(1) == 1 ? g.sum(at::IntArrayRef{0, 2}) : g.sum(0)).to(p.scalar_type()).view(p.sizes());
        };
        if (!per_token) gw = shared(gw, w);
        return {gr, gk, gv, gw, shared(gu, u), gs0};
    }
};
template <bool kPerToken>
struct Wkv6 {
    static constexpr const char* kName = "wkv6";
    static variable_list gradients(const variable_list& saved, const variable_list& grads) {
        return Wkv6Versioned::gradients(kPerToken, saved, grads);
    }
};
template <bool kPerToken>
struct Wkv6Node : public torch::autograd::Function<Wkv6Node<kPerToken>> {
    static variable_list forward(AutogradContext* ctx, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
                                 const Tensor& u, const Tensor& s, const Tensor& length, const Tensor& starts) {
        const Tensor t[] = {r, k, v, w, u, s};
        Tensor residual;
        auto [s_out, y] = Wkv6Versioned::forward(kPerToken, t, length, starts, &residual);
        ctx->save_for_backward({r, k, v, w, u, s, length, starts, residual});
        ctx->set_materialize_grads(false);
        return {s_out, y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list g = gradients_of<Wkv6<kPerToken>>(ctx, grads);
        g.resize(8);
        return g;
    }
};

// ------------------------------------------------------------------------------------------------- RWKV-4
// k, v (lead, T, C), parameters (C), state (lead, 3, C).  With r (lead, T, C) the result is r * wkv, as the model takes it.
struct Wkv4 {
    static constexpr const char* kName = "wkv4";
    struct Dims {
        at::IntArrayRef lead;
        int B, T, C;
        explicit Dims(const Tensor& k) : lead(k.sizes().slice(0, k.dim() - 2)) {
            B = (int)c10::multiply_integers(lead);
            T = (int)k.size(-2); C = (int)k.size(-1);
        }
    };
    // t: k v w u s [r]
    static bool fits(const Tensor* t, bool with_r) {
        if (!same_kind(t, with_r ? 6 : 5) || t[0].dim() < 2) return false;
        const Dims d(t[0]);
        return t[1].sizes().equals(t[0].sizes()) && sizes_are(t[2], {}, {d.C}) && sizes_are(t[3], {}, {d.C}) &&
               sizes_are(t[4], d.lead, {3, d.C}) && (!with_r || t[5].sizes().equals(t[0].sizes()));
    }
    static std::pair<Tensor, Tensor> forward(const Tensor* t, const Tensor& length, const Tensor& starts, Tensor* residual) {
        const Tensor& k = t[0];
        const c10::cuda::CUDAGuard guard(k.device());
        const Dims d(k);
        const Flags f(length, starts, d.lead, d.T, k);
        Tensor c[6];
        for (int i = 0; i < 6; ++i) c[i] = t[i].defined() ? t[i].contiguous() : t[i];
        Tensor y = fresh_like(k), s_out = fresh_like(t[4]);
        if (residual) *residual = bytes(b200wkv4_residual_bytes(dtype_code(k), d.B, d.T, d.C), k);
        check(b200wkv::wkv4_fwd(stream_of(k), dtype_code(k), d.B, d.T, d.C, true, in(c[2]), in(c[3]), in(c[5]), in(c[0]), in(c[1]), in(c[4]),
                                (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), out(s_out), out(y),
                                residual ? out(*residual) : nullptr));
        return {s_out, y};
    }
    // saved: k v w u s r length new_starts residual
    static variable_list gradients(const variable_list& saved, const variable_list& grads) {
        const Tensor &k = saved[0], r = if_any(saved[5]);
        const bool with_r = r.defined();
        const c10::cuda::CUDAGuard guard(k.device());
        const Dims d(k);
        const Flags f(saved[6], saved[7], d.lead, d.T, k);
        const Tensor gs = cotangent(grads[0], k), gy = cotangent(grads[1], k), rc = with_r ? r.contiguous() : Tensor();
        Tensor c[4], g[6];
        for (int i = 0; i < 4; ++i) c[i] = saved[i].contiguous();
        for (int i = 0; i < 5; ++i) g[i] = fresh_like(saved[i]);
        if (with_r) g[5] = fresh_like(r);
        const Tensor sums = fresh({2, d.B, d.C}, at::kFloat, k);
        float* gw = (float*)out(sums);
        float* gu = gw + (size_t)d.B * d.C;
        check(b200wkv::wkv4_bwd(stream_of(k), dtype_code(k), d.B, d.T, d.C, true, in(c[2]), in(c[3]), in(rc), in(c[0]), in(c[1]), in(gy),
                                (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), in(gs), in(saved[8]), gw, gu, out(g[5]),
                                out(g[0]), out(g[1]), out(g[4])));
        check(b200wkv::wkv4_parameter_grads(stream_of(k), dtype_code(k), d.B, d.C, in(c[2]), gw, gu, out(g[2]), out(g[3])));
        return {g[0], g[1], g[2], g[3], g[4], g[5]};
    }
};
struct Wkv4Node : public torch::autograd::Function<Wkv4Node> {
    static variable_list forward(AutogradContext* ctx, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u,
                                 const Tensor& s, const Tensor& r, const Tensor& length, const Tensor& starts) {
        const Tensor t[] = {k, v, w, u, s, if_any(r)};
        Tensor residual;
        auto [s_out, y] = Wkv4::forward(t, length, starts, &residual);
        ctx->save_for_backward({k, v, w, u, s, r, length, starts, residual});
        ctx->set_materialize_grads(false);
        return {s_out, y};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        variable_list g = gradients_of<Wkv4>(ctx, grads);
        g.resize(8);
        return g;
    }
};

// ------------------------------------------------------------------------------------------------- decoding
// One token on layer `layer` of the packed state (B, L, 2 + N, H N), in place.  An undefined tensor when it does not fit.
Tensor step_packed(const Tensor* t /* r w k v a b */, const Tensor& state, int64_t layer, const Tensor& starts, const Tensor& length) {
    if (!same_kind(t, 6) || t[0].dim() < 3 || state.dim() != 4 || state.scalar_type() != t[0].scalar_type() || !state.is_contiguous() ||
        state.device() != t[0].device())
        return Tensor();
    const int64_t B = t[0].size(0), H = t[0].size(-2), N = t[0].size(-1);
    if (t[0].numel() != B * H * N || state.size(0) != B || state.size(2) != 2 + N || state.size(3) != H * N || layer < 0 ||
        layer >= state.size(1))
        return Tensor();
    for (int i = 1; i < 6; ++i)
        if (!t[i].sizes().equals(t[0].sizes())) return Tensor();
    const c10::cuda::CUDAGuard guard(state.device());
    Tensor c[6], len = length, ns = starts;
    for (int i = 0; i < 6; ++i) c[i] = t[i].contiguous();
    if (len.defined()) len = len.to(state.device()).expand({B}).to(at::kInt).contiguous();
    if (ns.defined()) {
        if (ns.numel() != B) return Tensor();
        ns = ns.to(state.device());
        if (ns.scalar_type() != at::kBool) ns = ns.to(at::kByte);
        ns = ns.contiguous();
    }
    Tensor y = fresh_like(t[0]);
    char* block = (char*)out(state) + (layer * state.stride(1) + 2 * state.stride(2)) * state.element_size();
    check(b200wkv7_step_inplace(stream_of(state), dtype_code(state), (int)B, (int)H, (int)N, in(c[1]), in(c[0]), in(c[2]), in(c[3]),
                                in(c[4]), in(c[5]), block, state.stride(0), (const uint32_t*)in(len), (const uint8_t*)in(ns), out(y)));
    return y;
}

// ------------------------------------------------------------------------------------------------- matrix products
// The framework's GEMM library with the choice of its kernel made once per shape: at::mm makes it anew on every call, 10 us
// of host time each, and a layer has 36 products.  Row-major operands; every pointer on a 16-byte boundary.
class Gemm {
    static constexpr size_t kWorkspace = 32 << 20;
    static constexpr size_t kPlans = 512;             // per host thread; then the table starts over
    struct Plan {
        cublasLtMatmulDesc_t op = nullptr;
        cublasLtMatrixLayout_t a = nullptr, b = nullptr, c = nullptr;
        cublasLtMatmulAlgo_t algo;
        ~Plan() {
            if (a) cublasLtMatrixLayoutDestroy(a);
            if (b) cublasLtMatrixLayoutDestroy(b);
            if (c) cublasLtMatrixLayoutDestroy(c);
            if (op) cublasLtMatmulDescDestroy(op);
        }
    };
    typedef std::array<int64_t, 6> Key;               // device, m, n, k, form, type
    struct Hash {
        size_t operator()(const Key& k) const {
            size_t h = 0;
            for (int64_t x : k) h = h * 1000003 + (size_t)x;
            return h;
        }
    };
    Tensor workspace_;
    cudaStream_t stream_;
    cublasLtHandle_t handle_;
    bool bf16_, tf32_;
    int64_t device_;

    static cublasLtHandle_t handle(int device) {
        thread_local int current = -1;                // an autograd thread may not have made the device's context current yet
        if (current != device) {
            cuda_check(cudaSetDevice(device));
            current = device;
        }
        return at::cuda::getCurrentCUDABlasLtHandle();
    }
    static void ok(cublasStatus_t s) {
        if (s != CUBLAS_STATUS_SUCCESS) raise("b200wkv: matrix product failed (cublasLt status " + std::to_string((int)s) + ")");
    }
    std::shared_ptr<Plan> make(int64_t m, int64_t n, int64_t k, bool ta, bool tb) const {
        auto p = std::make_shared<Plan>();
        const cudaDataType_t type = bf16_ ? CUDA_R_16BF : CUDA_R_32F;
        ok(cublasLtMatmulDescCreate(&p->op, tf32_ ? CUBLAS_COMPUTE_32F_FAST_TF32 : CUBLAS_COMPUTE_32F, CUDA_R_32F));
        // the library is column-major: C^T = B^T A^T, so its first operand is B and its second A
        const cublasOperation_t first = tb ? CUBLAS_OP_T : CUBLAS_OP_N, second = ta ? CUBLAS_OP_T : CUBLAS_OP_N;
        ok(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSA, &first, sizeof(first)));
        ok(cublasLtMatmulDescSetAttribute(p->op, CUBLASLT_MATMUL_DESC_TRANSB, &second, sizeof(second)));
        ok(cublasLtMatrixLayoutCreate(&p->a, type, tb ? k : n, tb ? n : k, tb ? k : n));
        ok(cublasLtMatrixLayoutCreate(&p->b, type, ta ? m : k, ta ? k : m, ta ? m : k));
        ok(cublasLtMatrixLayoutCreate(&p->c, type, n, m, n));
        cublasLtMatmulPreference_t pref;
        ok(cublasLtMatmulPreferenceCreate(&pref));
        const size_t ws = kWorkspace;
        const uint32_t align = 16;
        cublasLtMatmulPreferenceSetAttribute(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &ws, sizeof(ws));
        for (auto a : {CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES,
                       CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES})
            cublasLtMatmulPreferenceSetAttribute(pref, a, &align, sizeof(align));
        cublasLtMatmulHeuristicResult_t found;
        int n_found = 0;
        const cublasStatus_t s = cublasLtMatmulAlgoGetHeuristic(handle_, p->op, p->a, p->b, p->c, p->c, pref, 1, &found, &n_found);
        cublasLtMatmulPreferenceDestroy(pref);
        ok(s);
        if (n_found < 1) ok(CUBLAS_STATUS_NOT_SUPPORTED);
        p->algo = found.algo;
        return p;
    }
    void run(int64_t m, int64_t n, int64_t k, bool ta, bool tb, const void* A, const void* B, void* C, bool add) const {
        thread_local std::unordered_map<Key, std::shared_ptr<Plan>, Hash> plans;
        const Key key{device_, m, n, k, ta * 2 + tb, bf16_ * 2 + tf32_};
        auto it = plans.find(key);
        if (it == plans.end()) {
            if (plans.size() >= kPlans) plans.clear();
            it = plans.emplace(key, make(m, n, k, ta, tb)).first;
        }
        const Plan& p = *it->second;
        const float alpha = 1.f, beta = add ? 1.f : 0.f;
        ok(cublasLtMatmul(handle_, p.op, &alpha, B, p.a, A, p.b, &beta, C, p.c, C, p.c, &p.algo, out(workspace_), kWorkspace, stream_));
    }

   public:
    Gemm(const Tensor& like, cudaStream_t st)
        : workspace_(bytes(kWorkspace, like)), stream_(st), handle_(handle(like.device().index())),
          bf16_(like.scalar_type() == at::kBFloat16), tf32_(!bf16_ && at::globalContext().allowTF32CuBLAS()), device_(like.device().index()) {}
    // C (m, n) = A (m, k) B (k, n)
    void nn(int64_t m, int64_t n, int64_t k, const void* A, const void* B, void* C) const { run(m, n, k, false, false, A, B, C, false); }
    // C (m, n) [+]= A (m, k) B^T, B (n, k)
    void nt(int64_t m, int64_t n, int64_t k, const void* A, const void* B, void* C, bool add = false) const { run(m, n, k, false, true, A, B, C, add); }
    // C (m, n) = A^T B, A (k, m), B (k, n)
    void tn(int64_t m, int64_t n, int64_t k, const void* A, const void* B, void* C) const { run(m, n, k, true, false, A, B, C, false); }
};

// ------------------------------------------------------------------------------------------------- time mixing
// A whole RWKV-7 time-mixing layer as one node: the token shift, the projections (library GEMMs, as before), the elementwise
// stage in front of the operator, the operator, the elementwise stage behind it.  As separate autograd functions and
// torch ops the host needs 2.6 ms for a forward and backward whatever the size.  Here the intermediates of a pass share one
// allocation, gradients of one tensor that meet from several places are added where a kernel reads or a GEMM
// writes them anyway, the shift's six cotangents are written where its backward kernel reads them, and parameter
// gradients leave one reduction kernel in their final type.
struct Layer {
    static constexpr const char* kName = "time_mixing_seq";
    enum { kMix = 0, kWr = 6, kWk, kWv, kWo, kW1, kW2, kA1, kA2, kV1, kV2, kG1, kG2, kW0, kA0, kV0, kKk, kKa, kRk, kLnW, kLnB, kParams };
    static constexpr int64_t kN = 64;

    struct Dims {
        int64_t B, T, C, H, rows;
        bool first;                    // the first layer: no value mix
        int64_t inner[4];              // widths of the low-rank projections w, a, v, g
        Dims(const Tensor& x, const Tensor* p, int64_t H_, bool first_)
            : B(x.size(0)), T(x.size(1)), C(x.size(2)), H(H_), rows(B * T), first(first_),
              inner{p[kW1].size(1), p[kA1].size(1), first_ ? 0 : p[kV1].size(1), p[kG1].size(1)} {}
    };
    static constexpr float kEps = 64e-5f;

    // One allocation cut into pieces of whole 256-byte lines.
    struct Slab {
        Tensor t;
        int64_t esz, used = 0;
        static int64_t padded(int64_t n, int64_t esz) { return (n * esz + 255) / 256 * 256; }
        Slab(const Tensor& like, std::initializer_list<int64_t> pieces) : esz(like.element_size()) {
            int64_t n = 0;
            for (int64_t p : pieces) n += padded(p, esz);
            t = bytes((size_t)n, like);
        }
        Slab(const Tensor& given, int64_t element) : t(given), esz(element) {}
        void* take(int64_t n) {
            void* p = (char*)out(t) + used;
            used += padded(n, esz);
            return p;
        }
    };
    // The forward's intermediates, all in one slab: streams of (rows, C) and the low-rank hidden rows.
    struct Inter {
        void *mixed, *r, *k, *wl, *al, *vl, *g, *w, *kp, *vp, *ai, *bi, *y, *xo, *hidden[4];
        static Slab make(const Tensor& x, const Dims& d) {
            const int64_t n = d.rows * d.C;
            return Slab(x, {6 * n, n, n, n, n, n, n, n, n, n, n, n, n, n, d.rows * d.inner[0], d.rows * d.inner[1], d.rows * d.inner[2],
                            d.rows * d.inner[3]});
        }
        Inter(Slab s, const Dims& d) {
            const int64_t n = d.rows * d.C;
            mixed = s.take(6 * n);
            for (void** p : {&r, &k, &wl, &al, &vl, &g, &w, &kp, &vp, &ai, &bi, &y, &xo}) *p = s.take(n);
            for (int i = 0; i < 4; ++i) hidden[i] = s.take(d.rows * d.inner[i]);
        }
    };
    static void* at(void* p, int64_t elements, const Tensor& x) { return (char*)p + elements * x.element_size(); }

    // rows `first`.. of every sequence's (1 + N, C) state block as a dense array, and back (no copy where they are dense)
    static const void* dense_rows(const Tensor& state, int64_t first, int64_t n, Tensor& room, cudaStream_t st) {
        const int64_t C = state.size(2), e = state.element_size(), pitch = state.size(1) * C * e;
        const char* src = (const char*)in(state) + first * C * e;
        if (state.size(0) == 1) return src;
        room = fresh({state.size(0), n, C}, state.scalar_type(), state);
        cuda_check(cudaMemcpy2DAsync(out(room), n * C * e, src, pitch, n * C * e, state.size(0), cudaMemcpyDeviceToDevice, st));
        return in(room);
    }
    struct Landing {                   // where a kernel writes a dense array that belongs into rows of a state
        Tensor state, room;
        int64_t first, n;
        void* p;
        Landing(const Tensor& s, int64_t first_, int64_t n_) : state(s), first(first_), n(n_) {
            if (s.size(0) > 1) room = fresh({s.size(0), n, s.size(2)}, s.scalar_type(), s);
            p = room.defined() ? out(room) : place();
        }
        void* place() const { return (char*)out(state) + first * state.size(2) * state.element_size(); }
        void finish(cudaStream_t st) const {
            if (!room.defined()) return;
            const int64_t row = state.size(2) * state.element_size();
            cuda_check(cudaMemcpy2DAsync(place(), state.size(1) * row, in(room), n * row, n * row, state.size(0), cudaMemcpyDeviceToDevice, st));
        }
    };

    static bool fits(const Tensor& x, const Tensor& state, const Tensor& v_first, const Tensor* p, int64_t H, int64_t S, bool first) {
        if (x.dim() != 3 || state.dim() != 3 || S != kN || H < 1 || H > 128) return false;
        const int64_t B = x.size(0), C = x.size(2);
        const Tensor t[] = {x, state, v_first};
        if (C != H * S || B > 65535 || x.size(0) * x.size(1) > 2147483647 / 8 || !same_kind(t, 3) || !sizes_are(state, {}, {B, 1 + S, C}) ||
            !v_first.sizes().equals(x.sizes()))
            return false;
        for (const Tensor* t : {&x, &v_first})        // (the state's rows are made dense below)
            if (t->is_contiguous() && !on_16_bytes(*t)) return false;
        for (int i = 0; i < kParams; ++i) {
            if (first && (i == kV0 || i == kV1 || i == kV2)) continue;
            if (!p[i].defined() || p[i].scalar_type() != x.scalar_type() || p[i].device() != x.device() || !p[i].is_contiguous() ||
                (uintptr_t)in(p[i]) % 16 != 0)
                return false;
            if (i >= kWr && i <= kWo) {
                if (!sizes_are(p[i], {}, {C, C})) return false;
            } else if (i >= kW1 && i <= kG2) {
                if (p[i].dim() != 2 || p[i].numel() == 0) return false;
                const bool down = (i - kW1) % 2 == 0;
                if (p[i].size(down ? 0 : 1) != C || p[i].size(down ? 1 : 0) != p[down ? i + 1 : i - 1].size(down ? 0 : 1)) return false;
            } else if (p[i].numel() != C) {
                return false;
            }
        }
        return true;
    }

    struct Kept {                      // what the backward needs beside the parameters
        Tensor x, state, v_first, v, slab, length, starts, residual;
        Tensor rows[2];                // the state's first row and the others, where they had to be made dense
    };

    // returns (out (B, T, C), new_state)
    static std::pair<Tensor, Tensor> forward(const Dims& d, const Tensor& x_, const Tensor& state_, const Tensor& v_first, const Tensor* p,
                                             const Tensor& length, const Tensor& starts, bool residual, Kept& kept) {
        const c10::cuda::CUDAGuard guard(x_.device());
        const cudaStream_t st = stream_of(x_);
        const int code = dtype_code(x_), B = (int)d.B, T = (int)d.T, C = (int)d.C, H = (int)d.H;
        const Flags f(length, starts, {d.B}, d.T, x_);
        const Tensor x = x_.contiguous(), state = dense(state_);
        kept = {x, state, d.first ? Tensor() : v_first.contiguous(), fresh({d.B, d.T, d.C}, x.scalar_type(), x), Inter::make(x, d).t, f.length,
                f.starts, Tensor(), {}};
        const Inter q(Slab(kept.slab, x.element_size()), d);
        Gemm gemm(x, st);
        Tensor new_state = fresh_like(state), o = fresh({d.B, d.T, d.C}, x.scalar_type(), x);
        const void* prev = dense_rows(state, 0, 1, kept.rows[0], st);
        const void* s0 = dense_rows(state, 1, kN, kept.rows[1], st);
        const Landing shift_row(new_state, 0, 1), s_out(new_state, 1, kN);
        const void* mix[6];
        for (int i = 0; i < 6; ++i) mix[i] = in(p[kMix + i]);
        check(b200wkv::token_shift_fwd(st, code, B, T, C, 6, in(x), prev, mix, (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), q.mixed,
                                       shift_row.p));
        shift_row.finish(st);
        void* m[6];                    // the inputs of r, w, k, v, a, g
        for (int i = 0; i < 6; ++i) m[i] = at(q.mixed, i * d.rows * d.C, x);
        void* const v = out(kept.v);
        gemm.nt(d.rows, d.C, d.C, m[0], in(p[kWr]), q.r);
        gemm.nt(d.rows, d.C, d.C, m[2], in(p[kWk]), q.k);
        gemm.nt(d.rows, d.C, d.C, m[3], in(p[kWv]), v);
        const auto lora = [&](int which, int down, void* input, int act, void* to) {
            gemm.nn(d.rows, d.inner[which], d.C, input, in(p[down]), q.hidden[which]);
            if (act) check(b200wkv::activation(st, code, act, d.rows * d.inner[which], q.hidden[which], nullptr));
            gemm.nn(d.rows, d.C, d.inner[which], q.hidden[which], in(p[down + 1]), to);
        };
        lora(0, kW1, m[1], b200wkv::kTanh, q.wl);
        lora(1, kA1, m[4], 0, q.al);
        if (!d.first) lora(2, kV1, m[3], 0, q.vl);
        lora(3, kG1, m[5], b200wkv::kSigmoid, q.g);
        check(b200wkv7_mix_pre_fwd(st, code, d.rows, H, (int)kN, !d.first, q.k, q.wl, q.al, v, in(kept.v_first), d.first ? nullptr : q.vl, in(p[kW0]),
                                   in(p[kA0]), in(p[kV0]), in(p[kKk]), in(p[kKa]), q.w, q.kp, q.vp, q.ai, q.bi));
        const Wkv7Room room(x, B, T, H, (int)kN, residual);
        kept.residual = room.residual;
        check(b200wkv::wkv7_fwd(st, code, B, T, H, (int)kN, q.w, q.r, q.kp, q.vp, q.ai, q.bi, s0, (const uint32_t*)in(f.length),
                           (const uint8_t*)in(f.starts), q.y, s_out.p, out(kept.residual), room.residual_bytes, 0, room.ws()));
        s_out.finish(st);
        check(b200wkv7_mix_post_fwd(st, code, d.rows, H, (int)kN, kEps, q.y, q.r, q.kp, q.vp, q.g, in(p[kLnW]), in(p[kLnB]), in(p[kRk]), q.xo));
        gemm.nt(d.rows, d.C, d.C, q.xo, in(p[kWo]), out(o));
        return {o, new_state};
    }

    // grads: of out, new_state and (first layer) v.  Returns gradients of x, state, v_first and the parameters;
    // `wanted` says which of them anybody asked for.
    static variable_list gradients(const Dims& d, const Kept& kept, const Tensor* p, const variable_list& grads, const std::vector<bool>& wanted) {
        const Tensor& x = kept.x;
        const c10::cuda::CUDAGuard guard(x.device());
        const cudaStream_t st = stream_of(x);
        const int code = dtype_code(x), B = (int)d.B, T = (int)d.T, C = (int)d.C, H = (int)d.H;
        const int64_t n = d.rows * d.C, widest = std::max(std::max(d.inner[0], d.inner[1]), std::max(d.inner[2], d.inner[3]));
        const Inter q(Slab(kept.slab, x.element_size()), d);
        Gemm gemm(x, st);
        variable_list g(3 + kParams);
        const auto want = [&](int i) { return (bool)wanted[3 + i]; };
        // d W of y = input W (or input W^T where the weight is kept transposed): a sum over the rows
        const auto weight = [&](int i, int64_t a, int64_t b, const void* left, const void* right) {
            if (!want(i)) return;
            g[3 + i] = fresh({a, b}, x.scalar_type(), x);
            gemm.tn(a, b, d.rows, left, right, out(g[3 + i]));
        };
        const Tensor gout = cotangent(grads[0], x), gstate = cotangent(grads[1], x);
        Slab room(x, {6 * n, n, n, n, n, n, n, n, n, n, n, n, n, n, d.rows * widest});
        void* const gmixed = room.take(6 * n);
        void *gxo, *dr, *dkp, *dvp, *dg, *gr, *gw, *gk, *gv, *ga, *gb, *dvl, *dwl;
        for (void** b : {&gxo, &dr, &dkp, &dvp, &dg, &gr, &gw, &gk, &gv, &ga, &gb, &dvl, &dwl}) *b = room.take(n);
        void* const dh = room.take(d.rows * widest);
        void* m[6];                    // the inputs of r, w, k, v, a, g, and their cotangents where the shift's backward reads them
        void* gm[6];
        for (int i = 0; i < 6; ++i) {
            m[i] = at(q.mixed, i * n, x);
            gm[i] = at(gmixed, i * n, x);
        }
        const int n_part = b200wkv7_mix_partial_rows(d.rows, H, (int)kN), tiles = (T + B200WKV_SHIFT_TILE - 1) / B200WKV_SHIFT_TILE;
        const Tensor partial = fresh({(int64_t)n_part * 8 + d.B * tiles * 6, d.C}, at::kFloat, x);
        float* const part_pre = (float*)out(partial);
        float* const part_post = part_pre + (size_t)n_part * 5 * d.C;
        float* const part_mix = part_post + (size_t)n_part * 3 * d.C;

        gemm.nn(d.rows, d.C, d.C, in(gout), in(p[kWo]), gxo);
        weight(kWo, d.C, d.C, in(gout), q.xo);
        void* const dy = gm[0];        // gmixed is room until its parts are written, last of all
        check(b200wkv7_mix_post_bwd(st, code, d.rows, H, (int)kN, kEps, q.y, q.r, q.kp, q.vp, q.g, in(p[kLnW]), in(p[kLnB]), in(p[kRk]), gxo, dy, dr,
                                    dkp, dvp, dg, part_post));
        Tensor copies[2];
        const auto kept_rows = [&](int i) { return kept.rows[i].defined() ? in(kept.rows[i]) : at((void*)in(kept.state), i * d.C, x); };
        const void *s0 = kept_rows(1), *prev = kept_rows(0);
        const void* gs = dense_rows(gstate, 1, kN, copies[1], st);
        if (wanted[1]) g[1] = fresh_like(kept.state);
        const Tensor state_room = wanted[1] ? g[1] : fresh_like(kept.state);
        const Landing gprev(state_room, 0, 1), gs0(state_room, 1, kN);
        const Tensor ws = wkv7_bwd_workspace(x, B, T, H, kept.residual);
        check(b200wkv::wkv7_bwd(st, code, B, T, H, (int)kN, q.w, q.r, q.kp, q.vp, q.ai, q.bi, s0, (const uint32_t*)in(kept.length),
                                (const uint8_t*)in(kept.starts), dy, gs, out(kept.residual), (size_t)kept.residual.numel(), gw, gr, gk, gv, ga, gb, gs0.p, 0,
                                out(ws)));
        if (wanted[1]) gs0.finish(st);
        // r, k' and v' also feed the stage behind the operator: its shares (dr, dkp, dvp) are added where the next kernel reads
        // anyway (gr in place)
        const Tensor gv_out = d.first ? cotangent(grads[2], x) : Tensor();
        void *const dk = gxo, *const dal = gm[1], *const dv = gm[2];
        if (!d.first && wanted[2]) g[2] = fresh({d.B, d.T, d.C}, x.scalar_type(), x);
        void* const dvf = d.first ? nullptr : g[2].defined() ? out(g[2]) : gm[3];
        check(b200wkv::wkv7_mix_pre_bwd(st, code, (int)d.rows, C, !d.first, q.k, q.wl, q.al, in(kept.v), in(kept.v_first), q.vl, in(p[kW0]), in(p[kA0]),
                                        in(p[kV0]), in(p[kKk]), in(p[kKa]), gw, gk, gv, ga, gb, dk, dwl, dal, dv, dvf, dvl, part_pre,
                                        {dkp, dvp, in(gv_out), dr, gr}));
        // dal and dv lie in parts of gmixed that the products below fill: the products that read them come first
        const auto lora = [&](int which, int down, const void* up_grad, const void* input, void* into, int act, bool add) {
            weight(down + 1, d.inner[which], d.C, q.hidden[which], up_grad);
            gemm.nt(d.rows, d.inner[which], d.C, up_grad, in(p[down + 1]), dh);
            if (act) check(b200wkv::activation(st, code, act, d.rows * d.inner[which], dh, q.hidden[which]));
            weight(down, d.C, d.inner[which], input, dh);
            gemm.nt(d.rows, d.C, d.inner[which], dh, in(p[down]), into, add);
        };
        lora(1, kA1, dal, m[4], gm[4], 0, false);
        weight(kWv, d.C, d.C, dv, m[3]);
        gemm.nn(d.rows, d.C, d.C, dv, in(p[kWv]), gm[3]);
        if (!d.first) lora(2, kV1, dvl, m[3], gm[3], 0, true);
        weight(kWr, d.C, d.C, gr, m[0]);
        gemm.nn(d.rows, d.C, d.C, gr, in(p[kWr]), gm[0]);
        weight(kWk, d.C, d.C, dk, m[2]);
        gemm.nn(d.rows, d.C, d.C, dk, in(p[kWk]), gm[2]);
        lora(0, kW1, dwl, m[1], gm[1], b200wkv::kTanh, false);
        lora(3, kG1, dg, m[5], gm[5], b200wkv::kSigmoid, false);

        const Tensor gx = fresh({d.B, d.T, d.C}, x.scalar_type(), x);
        const void* mix[6];
        for (int i = 0; i < 6; ++i) mix[i] = in(p[kMix + i]);
        const void* gstate0 = dense_rows(gstate, 0, 1, copies[0], st);
        check(b200wkv::token_shift_bwd(st, code, B, T, C, 6, in(x), prev, mix, (const uint32_t*)in(kept.length), (const uint8_t*)in(kept.starts), gmixed,
                                       gstate0, out(gx), gprev.p, part_mix));
        if (wanted[0]) g[0] = gx;
        if (wanted[1]) gprev.finish(st);
        // parameter gradients: column sums of the kernels' partial rows
        const Tensor sums = fresh({14, d.C}, x.scalar_type(), x);
        check(b200wkv::column_sums(st, code, {{part_mix, B * tiles, 6 * C}, {part_pre, n_part, 5 * C}, {part_post, n_part, 3 * C}}, out(sums)));
        const int order[14] = {kMix, kMix + 1, kMix + 2, kMix + 3, kMix + 4, kMix + 5, kW0, kA0, kV0, kKk, kKa, kLnW, kLnB, kRk};
        for (int i = 0; i < 14; ++i)
            if (want(order[i]) && p[order[i]].defined()) g[3 + order[i]] = sums[i].view(p[order[i]].sizes());
        return g;
    }
};

struct LayerNode : public torch::autograd::Function<LayerNode> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& state, const Tensor& v_first, at::TensorList params,
                                 const Tensor& length, const Tensor& starts, int64_t H, bool first) {
        const Layer::Dims d(x, params.data(), H, first);
        Layer::Kept k;
        auto [o, new_state] = Layer::forward(d, x, state, v_first, params.data(), length, starts, true, k);
        variable_list keep(params.begin(), params.end());
        for (const Tensor& t : {k.x, k.state, k.v_first, k.v, k.slab, k.length, k.starts, k.residual, k.rows[0], k.rows[1]}) keep.push_back(t);
        ctx->saved_data["H"] = H;
        ctx->saved_data["first"] = first;
        ctx->save_for_backward(keep);
        if (first) return {o, new_state, k.v};
        return {o, new_state};
    }
    static variable_list backward(AutogradContext* ctx, variable_list grads) {
        const variable_list saved = ctx->get_saved_variables();
        const bool first = ctx->saved_data["first"].toBool();
        const Tensor* s = saved.data() + Layer::kParams;
        const Layer::Kept k{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], {s[8], s[9]}};
        const Layer::Dims d(k.x, saved.data(), ctx->saved_data["H"].toInt(), first);
        std::vector<bool> wanted(3 + Layer::kParams);
        for (int j = 0; j < 3 + Layer::kParams; ++j) wanted[j] = ctx->needs_input_grad(j);
        variable_list g = once_differentiable(Layer::kName, saved, grads, [&]() { return Layer::gradients(d, k, saved.data(), grads, wanted); });
        g.resize(3 + Layer::kParams + 4);
        return g;
    }
};

// ------------------------------------------------------------------------------------------------- Python
bool take(PyObject* const* args, int n, Tensor* to, bool look_for_tangents = true) {
    for (int i = 0; i < n; ++i) {
        if (!THPVariable_CheckExact(args[i])) return false;
        to[i] = THPVariable_Unpack(args[i]);
        if (look_for_tangents && has_tangent(to[i])) return false;
    }
    return plain_mode();
}
PyObject* pair(const Tensor& a, const Tensor& b) {
    THPObjectPtr t(PyTuple_New(2));
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t.get(), 0, THPVariable_Wrap(a));
    PyTuple_SET_ITEM(t.get(), 1, THPVariable_Wrap(b));
    return t.release();
}

PyObject* py_wkv7(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    Tensor t[9], s_out, y;
    if (n != 9 || !take(args, 9, t) || !Wkv7::fits(t)) Py_RETURN_NONE;
    {
        pybind11::gil_scoped_release no_gil;
        if (any_grad(t, 7)) {
            variable_list o = Wkv7Node::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8]);
            s_out = o[0]; y = o[1];
        } else {
            std::tie(s_out, y) = Wkv7::forward(t, t[7], t[8], nullptr);
        }
    }
    return pair(s_out, y);
    END_HANDLE_TH_ERRORS
}

PyObject* py_wkv6(PyObject*, PyObject* const* args, Py_ssize_t n) {   // (per_token, r, k, v, w, u, s, length, new_starts)
    HANDLE_TH_ERRORS
    Tensor t[8], s_out, y;
    if (n != 9) Py_RETURN_NONE;
    const bool per_token = args[0] == Py_True;
    if (!take(args + 1, 8, t) || !Wkv6Versioned::fits(per_token, t)) Py_RETURN_NONE;
    {
        pybind11::gil_scoped_release no_gil;
        if (any_grad(t, 6)) {
            variable_list o = per_token ? Wkv6Node<true>::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7])
                                        : Wkv6Node<false>::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]);
            s_out = o[0]; y = o[1];
        } else {
            std::tie(s_out, y) = Wkv6Versioned::forward(per_token, t, t[6], t[7], nullptr);
        }
    }
    return pair(s_out, y);
    END_HANDLE_TH_ERRORS
}

PyObject* py_wkv4(PyObject*, PyObject* const* args, Py_ssize_t n) {   // (r or None, k, v, w, u, s, length, new_starts)
    HANDLE_TH_ERRORS
    Tensor t[8], s_out, y;   // k v w u s r length new_starts
    if (n != 8 || !take(args + 1, 5, t) || !take(args + 6, 2, t + 6)) Py_RETURN_NONE;
    if (args[0] != Py_None && !take(args, 1, t + 5)) Py_RETURN_NONE;
    const bool with_r = t[5].defined();
    if (!Wkv4::fits(t, with_r)) Py_RETURN_NONE;
    {
        pybind11::gil_scoped_release no_gil;
        if (any_grad(t, with_r ? 6 : 5)) {
            variable_list o = Wkv4Node::apply(t[0], t[1], t[2], t[3], t[4], with_r ? t[5] : nothing(t[0]), t[6], t[7]);
            s_out = o[0]; y = o[1];
        } else {
            std::tie(s_out, y) = Wkv4::forward(t, t[6], t[7], nullptr);
        }
    }
    return pair(s_out, y);
    END_HANDLE_TH_ERRORS
}

// (x, state, v_first, att, length, new_starts, H, S, layer_id) -> (out, new_state, v_first)
PyObject* py_time_mixing(PyObject*, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    static const char* const kNames[Layer::kParams] = {"x_r", "x_w", "x_k", "x_v", "x_a", "x_g", "receptance", "key", "value", "output",
                                                       "w1", "w2", "a1", "a2", "v1", "v2", "g1", "g2", "w0", "a0", "v0", "k_k", "k_a", "r_k",
                                                       "ln_x", "ln_x"};
    Tensor t[3], flags[2], p[Layer::kParams];
    if (n != 9 || !take(args, 3, t) || !PyDict_CheckExact(args[3]) || !take(args + 4, 2, flags) || at::autocast::is_autocast_enabled(at::kCUDA))
        Py_RETURN_NONE;
    for (int i = 6; i < 9; ++i)
        if (!PyLong_CheckExact(args[i])) Py_RETURN_NONE;
    const int64_t H = PyLong_AsLongLong(args[6]), S = PyLong_AsLongLong(args[7]);
    const bool first = PyLong_AsLongLong(args[8]) == 0;
    for (int i = 0; i < Layer::kParams; ++i) {
        if (first && (i == Layer::kV0 || i == Layer::kV1 || i == Layer::kV2)) continue;      // not used by the first layer
        PyObject* item = PyDict_GetItemString(args[3], kNames[i]);
        if (item && ((i >= Layer::kWr && i <= Layer::kWo) || i >= Layer::kLnW))
            item = PyDict_CheckExact(item) ? PyDict_GetItemString(item, i == Layer::kLnB ? "bias" : "weight") : nullptr;
        if (!item || !take(&item, 1, &p[i])) Py_RETURN_NONE;
    }
    if (!Layer::fits(t[0], t[1], t[2], p, H, S, first)) Py_RETURN_NONE;
    Tensor o, new_state, v;
    {
        pybind11::gil_scoped_release no_gil;
        const Tensor vf = first ? Tensor() : t[2];
        if (any_grad(t, first ? 2 : 3) || any_grad_defined(p, Layer::kParams)) {
            for (Tensor& q : p)
                if (!q.defined()) q = nothing(t[0]);      // the first layer's v0, v1, v2
            variable_list r = LayerNode::apply(t[0], t[1], first ? nothing(t[0]) : vf, at::TensorList(p, Layer::kParams), flags[0], flags[1], H, first);
            o = r[0]; new_state = r[1];
            if (first) v = r[2];
        } else {
            const at::AutoGradMode no_grad(false);
            const Layer::Dims d(t[0], p, H, first);
            Layer::Kept k;
            std::tie(o, new_state) = Layer::forward(d, t[0], t[1], vf, p, flags[0], flags[1], false, k);
            v = k.v;
        }
    }
    THPObjectPtr tuple(PyTuple_New(3));
    if (!tuple) throw python_error();
    PyTuple_SET_ITEM(tuple.get(), 0, THPVariable_Wrap(o));
    PyTuple_SET_ITEM(tuple.get(), 1, THPVariable_Wrap(new_state));
    if (!first) Py_INCREF(args[2]);
    PyTuple_SET_ITEM(tuple.get(), 2, first ? THPVariable_Wrap(v) : args[2]);
    return tuple.release();
    END_HANDLE_TH_ERRORS
}

PyObject* py_step_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {   // (r, w, k, v, a, b, state, layer, new_starts, length)
    HANDLE_TH_ERRORS
    // (no autograd bookkeeping here nor in the Python function behind: the look for tangents, 0.15 us of a call's 4.5, is left out)
    Tensor t[7], starts, length, y;
    if (n != 10 || !take(args, 7, t, false) || !PyLong_CheckExact(args[7])) Py_RETURN_NONE;
    if (args[8] != Py_None && !take(args + 8, 1, &starts, false)) Py_RETURN_NONE;
    if (args[9] != Py_None && !take(args + 9, 1, &length, false)) Py_RETURN_NONE;
    const int64_t layer = PyLong_AsLongLong(args[7]);
    if (layer == -1 && PyErr_Occurred()) throw python_error();
    {
        pybind11::gil_scoped_release no_gil;
        y = step_packed(t, t[6], layer, starts, length);
    }
    if (!y.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

PyObject* py_set_error_class(PyObject*, PyObject* cls) {
    Py_INCREF(cls);
    Py_XSETREF(g_error_class, cls);
    Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"wkv7", (PyCFunction)(void (*)(void))py_wkv7, METH_FASTCALL, nullptr},
    {"wkv6", (PyCFunction)(void (*)(void))py_wkv6, METH_FASTCALL, nullptr},
    {"wkv4", (PyCFunction)(void (*)(void))py_wkv4, METH_FASTCALL, nullptr},
    {"time_mixing", (PyCFunction)(void (*)(void))py_time_mixing, METH_FASTCALL, nullptr},
    {"step_packed", (PyCFunction)(void (*)(void))py_step_packed, METH_FASTCALL, nullptr},
    {"set_error_class", py_set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_b200wkv_host", "native host path of the WKV operators", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200wkv_host(void) { return PyModule_Create(&kModule); }

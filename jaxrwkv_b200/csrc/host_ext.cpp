// Native host path of the operators: argument checks, result allocation, the autograd nodes and the calls into
// libb200wkv.so without the Python interpreter in between.
//
// A call through torch.autograd.Function in Python costs 80-100 us forward and 350 us for a forward and backward,
// a ctypes call of a decoding step 30 us: more than most kernels behind them.  The same work from C++ costs a
// few microseconds per call.  Every function here returns None when it is handed something out of the ordinary
// (arguments that are no plain tensors, a functorch transform or a dispatch mode in force, shapes or types that do
// not fit); the Python functions that call them then take their own path, which handles vmap and raises the errors.
#include <torch/csrc/python_headers.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/object_ptr.h>

#include <ATen/ATen.h>
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

const void* in(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* out(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
    return at::detail::empty_cuda(sizes, type, like.device(), std::nullopt);
}
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }
Tensor bytes(size_t n, const Tensor& like) { return fresh({(int64_t)n}, at::kByte, like); }
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? B200WKV_F32 : B200WKV_BF16; }
cudaStream_t stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

// The plain case: no functorch transform, no dispatch mode.
bool plain_mode() {
    return !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
           !c10::impl::dispatch_mode_enabled();
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

// A cotangent as the kernels read it; an absent one (undefined, or the empty stand-in of gradients_of) is undefined: the
// kernels take NULL for zero.
Tensor cotangent(const Tensor& g, const Tensor& like) {
    return !g.defined() || g.numel() == 0 ? Tensor() : (g.scalar_type() == like.scalar_type() ? g : g.to(like.scalar_type())).contiguous();
}

// Gradients asked for with create_graph=True: the values are right, differentiating them again is an error.
template <class Op>
struct NoSecondOrder : public torch::autograd::Function<NoSecondOrder<Op>> {
    static variable_list forward(AutogradContext*, at::TensorList saved, at::TensorList grads) {
        return Op::gradients(variable_list(saved.begin(), saved.end()), variable_list(grads.begin(), grads.end()));
    }
    static variable_list backward(AutogradContext*, variable_list) {
        raise(std::string(Op::kName) + ": second-order differentiation is not supported");
    }
};
template <class Op>
variable_list gradients_of(AutogradContext* ctx, const variable_list& grads) {
    const variable_list saved = ctx->get_saved_variables();
    if (!at::GradMode::is_enabled()) return Op::gradients(saved, grads);
    variable_list given = grads;                  // a node's inputs have to be defined
    for (Tensor& g : given)
        if (!g.defined()) g = fresh({0}, saved[0].scalar_type(), saved[0]);
    return NoSecondOrder<Op>::apply(at::TensorList(saved), at::TensorList(given));
}

// ------------------------------------------------------------------------------------------------- RWKV-7
// Streams (lead, T, H, N), state (lead, H, N, N), any number of leading batch axes.
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
        const size_t rbytes = residual ? b200wkv7_residual_bytes(dtype_code(k), B, T, H, N) : 0;
        if (residual) *residual = bytes(rbytes, k);
        check(b200wkv7_fwd(stream_of(k), dtype_code(k), B, T, H, N, in(c[1]), in(c[0]), in(c[2]), in(c[3]), in(c[4]), in(c[5]),
                           in(c[6]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), out(y), out(s_out),
                           residual ? out(*residual) : nullptr, rbytes, 0));
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
        check(b200wkv7_bwd(stream_of(k), dtype_code(k), B, T, H, N, in(c[1]), in(c[0]), in(c[2]), in(c[3]), in(c[4]), in(c[5]),
                           in(c[6]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), in(gy), in(gs), out(res),
                           (size_t)res.numel(), out(g[1]), out(g[0]), out(g[2]), out(g[3]), out(g[4]), out(g[5]), out(g[6]), 0));
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
        check(b200wkv6_fwd(stream_of(k), dtype_code(k), per_token ? 6 : 5, d.B, d.T, d.H, d.N, in(c[0]), in(c[1]), in(c[2]),
                           in(c[3]), in(c[4]), in(c[5]), (const uint32_t*)in(f.length), (const uint8_t*)in(f.starts), out(y),
                           out(s_out), residual ? out(*residual) : nullptr, rbytes, 0));
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
    // saved: k v w u s r length new_starts residual (r may be undefined)
    static variable_list gradients(const variable_list& saved, const variable_list& grads) {
        const Tensor &k = saved[0], &r = saved[5];
        const bool with_r = r.defined() && r.numel() > 0;
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
        const Tensor t[] = {k, v, w, u, s, r};
        Tensor residual;
        auto [s_out, y] = Wkv4::forward(t, length, starts, &residual);
        ctx->save_for_backward({k, v, w, u, s, r.defined() ? r : fresh({0}, k.scalar_type(), k), length, starts, residual});
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

// ------------------------------------------------------------------------------------------------- Python
bool take(PyObject* const* args, int n, Tensor* to) {
    for (int i = 0; i < n; ++i) {
        if (!THPVariable_CheckExact(args[i])) return false;
        to[i] = THPVariable_Unpack(args[i]);
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
        // a constant decay (5, 5.2) without gradients also asks for a residual: the kernels of that call compute in fp32
        if (any_grad(t, 6)) {
            variable_list o = per_token ? Wkv6Node<true>::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7])
                                        : Wkv6Node<false>::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]);
            s_out = o[0]; y = o[1];
        } else {
            Tensor residual;
            std::tie(s_out, y) = Wkv6Versioned::forward(per_token, t, t[6], t[7], per_token ? nullptr : &residual);
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
            variable_list o = Wkv4Node::apply(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7]);
            s_out = o[0]; y = o[1];
        } else {
            std::tie(s_out, y) = Wkv4::forward(t, t[6], t[7], nullptr);
        }
    }
    return pair(s_out, y);
    END_HANDLE_TH_ERRORS
}

PyObject* py_step_packed(PyObject*, PyObject* const* args, Py_ssize_t n) {   // (r, w, k, v, a, b, state, layer, new_starts, length)
    HANDLE_TH_ERRORS
    Tensor t[7], starts, length, y;
    if (n != 10 || !take(args, 7, t) || !PyLong_CheckExact(args[7])) Py_RETURN_NONE;
    if (args[8] != Py_None && !take(args + 8, 1, &starts)) Py_RETURN_NONE;
    if (args[9] != Py_None && !take(args + 9, 1, &length)) Py_RETURN_NONE;
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
    {"step_packed", (PyCFunction)(void (*)(void))py_step_packed, METH_FASTCALL, nullptr},
    {"set_error_class", py_set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_b200wkv_host", "native host path of the WKV operators", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b200wkv_host(void) { return PyModule_Create(&kModule); }

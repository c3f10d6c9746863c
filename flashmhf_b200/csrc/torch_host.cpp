// Host path between torch tensors and the C ABI: argument checks, layout decisions, output and scratch allocation and
// the autograd functions, in C++.
//
// Why here and not in Python: a decode-shaped call, or a short training step, lasts some tens of microseconds on the
// GPU, and what a call costs the interpreter (attribute look-ups, ctypes structs, torch.empty, autograd.Function in both
// directions) was more than that: 20 us for a forward call whose checks had been remembered, about 200 us for forward +
// backward of the operator, 660 us for forward + backward of a layer.  Through this file a call costs its allocations
// and its launches.
//
// The C-ABI library itself stays free of torch types: its entry points are taken from the handle that
// flashmhf_b200/_lib.py has loaded (bind()), so one copy of the library serves ctypes callers and this module.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <cmath>
#include <optional>

#include "../../include/flashmhf.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct Api {
    decltype(&flashmhf_strerror) strerror = nullptr;
    decltype(&flashmhf_last_cuda_error) last_cuda_error = nullptr;
    decltype(&flashmhf_forward) forward = nullptr, forward_chained = nullptr;
    decltype(&flashmhf_backward) backward = nullptr;
    decltype(&flashmhf_forward_workspace_bytes) forward_ws = nullptr;
    decltype(&flashmhf_backward_workspace_bytes) backward_ws = nullptr;
    decltype(&flashmhf_prologue_forward) prologue_forward = nullptr;
    decltype(&flashmhf_prologue_backward_workspace_bytes) prologue_backward_ws = nullptr;
    decltype(&flashmhf_prologue_backward) prologue_backward = nullptr;
    decltype(&flashmhf_lm_rope) lm_rope = nullptr;
    decltype(&flashmhf_lm_rmsnorm_forward) rmsnorm_forward = nullptr;
    decltype(&flashmhf_lm_rmsnorm_backward_workspace_bytes) rmsnorm_backward_ws = nullptr;
    decltype(&flashmhf_lm_rmsnorm_backward) rmsnorm_backward = nullptr;
    PyObject *error_type = nullptr;  // flashmhf_b200._lib.FlashMHFError(status, message)
};
Api api;

void bind(uintptr_t handle, py::object error_type) {
    void *h = reinterpret_cast<void *>(handle);
    auto get = [h](auto &fn, const char *name) {
        void *p = dlsym(h, name);
        if (!p) throw std::runtime_error(std::string("the C-ABI library lacks ") + name);
        fn = reinterpret_cast<std::decay_t<decltype(fn)>>(p);
    };
    get(api.strerror, "flashmhf_strerror");
    get(api.last_cuda_error, "flashmhf_last_cuda_error");
    get(api.forward, "flashmhf_forward");
    get(api.forward_chained, "flashmhf_forward_chained");
    get(api.backward, "flashmhf_backward");
    get(api.forward_ws, "flashmhf_forward_workspace_bytes");
    get(api.backward_ws, "flashmhf_backward_workspace_bytes");
    get(api.prologue_forward, "flashmhf_prologue_forward");
    get(api.prologue_backward_ws, "flashmhf_prologue_backward_workspace_bytes");
    get(api.prologue_backward, "flashmhf_prologue_backward");
    get(api.lm_rope, "flashmhf_lm_rope");
    get(api.rmsnorm_forward, "flashmhf_lm_rmsnorm_forward");
    get(api.rmsnorm_backward_ws, "flashmhf_lm_rmsnorm_backward_workspace_bytes");
    get(api.rmsnorm_backward, "flashmhf_lm_rmsnorm_backward");
    Py_XDECREF(api.error_type);
    api.error_type = error_type.release().ptr();
}

// Raises FlashMHFError for a non-zero status (from a backward thread too: autograd carries the Python error across).
void check(int status) {
    if (status == FLASHMHF_OK) return;
    std::string msg = api.strerror(status);
    if (status == FLASHMHF_ERR_CUDA) msg += std::string(": ") + api.last_cuda_error();
    py::gil_scoped_acquire gil;
    PyObject *args = Py_BuildValue("(is)", status, msg.c_str());
    PyObject *exc = PyObject_CallObject(api.error_type, args);
    Py_XDECREF(args);
    if (exc) {
        PyErr_SetObject(api.error_type, exc);
        Py_DECREF(exc);
    }
    python_error err;
    err.persist();
    throw std::move(err);
}

void *current_stream(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

struct Shape {
    int64_t B, H, S, Dh, Hk, E, De;
};

std::string dims_text(const Tensor &t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + ")";
}

Shape validate(const Tensor &Q, const Tensor &K, const Tensor &U, const Tensor &V, const Tensor &R) {
    if (Q.dim() != 4 || K.dim() != 4 || R.dim() != 4)
        throw py::value_error("expected Q [B,H,S,d_h], K/U/V [H_kuv,E,d_e,d_h], R [B,H,S,E]");
    const Shape s{Q.size(0), Q.size(1), Q.size(2), Q.size(3), K.size(0), K.size(1), K.size(2)};
    if (s.De % 64 != 0) throw py::value_error("Expert dimension " + std::to_string(s.De) + " must be divisible by 64");
    if (U.sizes() != K.sizes() || V.sizes() != K.sizes() || K.size(3) != s.Dh)
        throw py::value_error("K/U/V shapes must agree and end in d_h=" + std::to_string(s.Dh) + ": " + dims_text(K) + ", " +
                              dims_text(U) + ", " + dims_text(V));
    if (s.Hk < 1 || s.H % s.Hk != 0)
        throw py::value_error("num_heads " + std::to_string(s.H) + " must be a multiple of num_kuv_heads " + std::to_string(s.Hk));
    if (R.size(0) != s.B || R.size(1) != s.H || R.size(2) != s.S || R.size(3) != s.E)
        throw py::value_error("R must be (" + std::to_string(s.B) + ", " + std::to_string(s.H) + ", " + std::to_string(s.S) + ", " +
                              std::to_string(s.E) + "), got " + dims_text(R));
    if (s.Dh != 64 && s.Dh != 96 && s.Dh != 128)
        throw py::value_error("head_dim " + std::to_string(s.Dh) + " not supported (64, 96 or 128)");
    const auto dt = Q.scalar_type();
    if ((dt != at::kBFloat16 && dt != at::kFloat) || K.scalar_type() != dt || U.scalar_type() != dt || V.scalar_type() != dt)
        throw py::type_error(std::string("flash_mhf expects Q, K, U, V all in torch.bfloat16 (or all float32 for the check mode), got Q=") +
                             c10::toString(dt) + ", K=" + c10::toString(K.scalar_type()) + ", V=" + c10::toString(V.scalar_type()) +
                             ", U=" + c10::toString(U.scalar_type()));
    const auto dev = Q.device();
    if (!Q.is_cuda() || K.device() != dev || U.device() != dev || V.device() != dev || R.device() != dev)
        throw py::value_error("flash_mhf runs on CUDA tensors of one device; there is no CPU path");
    return s;
}

flashmhf_scaling scaling_of(double hs, double us, double fs) {
    for (double v : {hs, us, fs})
        if (v == 0.0 || !std::isfinite(v)) throw py::value_error("scaling constants must be finite and non-zero");
    return flashmhf_scaling{(float)hs, (float)us, (float)fs};
}

flashmhf_dims dims_of(const Shape &s, at::ScalarType dt) {
    return flashmhf_dims{(int32_t)s.B, (int32_t)s.H, (int32_t)s.S, (int32_t)s.Dh, (int32_t)s.Hk, (int32_t)s.E, (int32_t)s.De,
                         dt == at::kBFloat16 ? FLASHMHF_BF16 : FLASHMHF_F32_CHECK};
}

// Can the library address this tensor in place? (unit inner stride, 16-byte aligned outer strides, E and d_e collapse)
bool in_place_ok(const Tensor &t, bool is_weight) {
    const auto st = t.strides();
    const auto sz = t.sizes();
    if (st[3] != 1 && sz[3] != 1) return false;
    if (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) return false;
    if (t.scalar_type() == at::kBFloat16)
        for (int i = 0; i < 3; ++i)
            if (sz[i] > 1 && (st[i] % 8 != 0 || st[i] <= 0)) return false;
    return !(is_weight && sz[1] > 1 && st[1] != sz[2] * st[2]);
}
Tensor addressable(const Tensor &t, bool is_weight) { return in_place_ok(t, is_weight) ? t : t.contiguous(); }

// R as the kernels read it: fp32, unit inner stride, 4-byte aligned (any outer strides).
Tensor routing(const Tensor &R) {
    Tensor r = R.scalar_type() == at::kFloat ? R : R.to(at::kFloat);
    return (r.stride(3) == 1 || r.size(3) == 1) ? r : r.contiguous();
}

flashmhf_tensor view4(const Tensor &t) {
    const auto s = t.strides();
    return flashmhf_tensor{t.data_ptr(), {s[0], s[1], s[2]}};
}
// A decode-shaped tensor [B,H,1,X] as [1,H,B,X]: a permutation, no copy, so that the B token rows of a head share tiles.
flashmhf_tensor tokens_as_sequence(const flashmhf_tensor &t) { return flashmhf_tensor{t.ptr, {t.stride[2], t.stride[1], t.stride[0]}}; }

Tensor scratch(const std::optional<Tensor> &given, size_t nbytes, const Tensor &like) {
    if (!given) return at::empty({(int64_t)nbytes}, like.options().dtype(at::kByte));
    const Tensor &w = *given;
    if (w.device() != like.device() || w.scalar_type() != at::kByte || w.numel() < (int64_t)nbytes ||
        (reinterpret_cast<uintptr_t>(w.data_ptr()) & 255u))
        throw py::value_error("workspace must be a 256-byte aligned uint8 tensor of at least " + std::to_string(nbytes) + " bytes on " +
                              like.device().str());
    return w;
}

// ------------------------------------------------------------------------------------------------ operator
Tensor forward_checked(const Shape &s, const Tensor &Q0, const Tensor &K0, const Tensor &U0, const Tensor &V0, const Tensor &R0,
                       const std::optional<Tensor> &out, const flashmhf_scaling &sc, bool chained,
                       const std::optional<Tensor> &workspace) {
    c10::cuda::CUDAGuard guard(Q0.device());
    const Tensor Q = addressable(Q0, false), K = addressable(K0, true), U = addressable(U0, true), V = addressable(V0, true), R = routing(R0);
    Tensor O = out ? *out : at::empty_like(Q);   // keeps Q's memory layout ([B,H,S,d] or [B,S,H,d])
    flashmhf_fwd_params p{};
    p.d = dims_of(s, Q.scalar_type());
    p.Q = view4(Q); p.K = view4(K); p.U = view4(U); p.V = view4(V); p.R = view4(R); p.O = view4(O);
    p.scale = sc;
    if (s.S == 1 && s.B > 1) {
        p.Q = tokens_as_sequence(p.Q); p.R = tokens_as_sequence(p.R); p.O = tokens_as_sequence(p.O);
        p.d.B = 1;
        p.d.S = (int32_t)s.B;
    }
    Tensor ws;
    p.workspace_bytes = api.forward_ws(&p.d);
    if (p.workspace_bytes) {
        ws = scratch(workspace, p.workspace_bytes, Q);
        p.workspace = ws.data_ptr();
    }
    check((chained ? api.forward_chained : api.forward)(&p, current_stream(Q)));
    return O;
}

Tensor op_forward(const Tensor &Q, const Tensor &K, const Tensor &U, const Tensor &V, const Tensor &R, const std::optional<Tensor> &out,
                  double hs, double us, double fs, bool chained, const std::optional<Tensor> &workspace) {
    at::AutoGradMode no_grad(false);
    const Shape s = validate(Q, K, U, V, R);
    return forward_checked(s, Q, K, U, V, R, out, scaling_of(hs, us, fs), chained, workspace);
}

struct Grads {
    Tensor dQ, dK, dU, dV, dR;
};
Grads backward_checked(const Shape &s, const Tensor &Q0, const Tensor &K0, const Tensor &U0, const Tensor &V0, const Tensor &R0,
                       const Tensor &dO0, const flashmhf_scaling &sc, uint32_t parts, const Tensor *weight_grads) {
    c10::cuda::CUDAGuard guard(Q0.device());
    const Tensor Q = addressable(Q0, false), K = addressable(K0, true), U = addressable(U0, true), V = addressable(V0, true), R = routing(R0);
    const Tensor dO = addressable(dO0.scalar_type() == Q.scalar_type() ? dO0 : dO0.to(Q.scalar_type()), false);
    const bool inputs = parts & FLASHMHF_BWD_INPUTS, weights = parts & FLASHMHF_BWD_WEIGHTS;
    Grads g;
    flashmhf_bwd_params p{};
    p.d = dims_of(s, Q.scalar_type());
    p.Q = view4(Q); p.K = view4(K); p.U = view4(U); p.V = view4(V); p.R = view4(R); p.dO = view4(dO);
    p.scale = sc;
    p.parts = parts;
    if (inputs) {
        g.dQ = at::empty_like(Q);   // keeps Q's memory layout
        g.dR = at::empty({s.B, s.H, s.S, s.E}, Q.options().dtype(at::kFloat));
        p.dQ = view4(g.dQ); p.dR = view4(g.dR);
    }
    Tensor ws;
    if (weights) {
        if (weight_grads) {
            g.dK = weight_grads[0]; g.dU = weight_grads[1]; g.dV = weight_grads[2];
        } else {
            // in the weights' own memory layout (a layer passes strided views of [I, H_kuv*d_h] parameters: their gradients
            // then need no re-layout copy); the fp32 check kernels write contiguous outputs
            const auto fmt = Q.scalar_type() == at::kBFloat16 ? at::MemoryFormat::Preserve : at::MemoryFormat::Contiguous;
            g.dK = at::empty_like(K, K.options(), fmt);
            g.dU = at::empty_like(U, U.options(), fmt);
            g.dV = at::empty_like(V, V.options(), fmt);
        }
        p.dK = view4(g.dK); p.dU = view4(g.dU); p.dV = view4(g.dV);
        p.workspace_bytes = api.backward_ws(&p.d);
        ws = at::empty({(int64_t)std::max<size_t>(p.workspace_bytes, 1)}, Q.options().dtype(at::kByte));
        p.workspace = ws.data_ptr();
    }
    check(api.backward(&p, current_stream(Q)));
    return g;
}

// parts: 0 everything, else the FLASHMHF_BWD_* mask
py::tuple op_backward(const Tensor &Q, const Tensor &K, const Tensor &U, const Tensor &V, const Tensor &R, const Tensor &dO, double hs,
                      double us, double fs, uint32_t parts, const std::optional<std::vector<Tensor>> &weight_grads) {
    at::AutoGradMode no_grad(false);
    const Shape s = validate(Q, K, U, V, R);
    if (parts == 0) parts = FLASHMHF_BWD_INPUTS | FLASHMHF_BWD_WEIGHTS;
    const flashmhf_scaling sc = scaling_of(hs, us, fs);
    if (weight_grads && (parts & FLASHMHF_BWD_WEIGHTS)) {
        const Tensor *w[3] = {&K, &U, &V};
        if (weight_grads->size() != 3) throw py::value_error("weight_grads must be (dK, dU, dV)");
        for (int i = 0; i < 3; ++i) {
            const Tensor &g = (*weight_grads)[i];
            if (g.sizes() != w[i]->sizes() || g.scalar_type() != w[i]->scalar_type() || g.device() != w[i]->device())
                throw py::value_error("weight_grads must match K, U, V in shape, dtype and device");
        }
    }
    const Grads g = backward_checked(s, Q, K, U, V, R, dO, sc, parts, weight_grads ? weight_grads->data() : nullptr);
    auto some = [](const Tensor &t) -> py::object { return t.defined() ? py::cast(t) : py::none(); };
    return py::make_tuple(some(g.dQ), some(g.dK), some(g.dU), some(g.dV), some(g.dR));
}

struct OpFunction : public torch::autograd::Function<OpFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &Q, const Tensor &K, const Tensor &U, const Tensor &V, const Tensor &R,
                          double hs, double us, double fs) {
        const Shape s = validate(Q, K, U, V, R);
        Tensor O = forward_checked(s, Q, K, U, V, R, std::nullopt, scaling_of(hs, us, fs), false, std::nullopt);
        ctx->save_for_backward({Q, K, U, V, R});
        ctx->saved_data["scale"] = std::vector<double>{hs, us, fs};
        return O;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const std::vector<double> sc = ctx->saved_data["scale"].toDoubleVector();
        const Tensor &Q = sv[0], &K = sv[1], &U = sv[2], &V = sv[3], &R = sv[4];
        if (!grads[0].defined()) return variable_list(8);
        uint32_t parts = 0;   // a gradient nobody asked for (frozen weights, or inputs that are data) is not computed
        if (ctx->needs_input_grad(0) || ctx->needs_input_grad(4)) parts |= FLASHMHF_BWD_INPUTS;
        if (ctx->needs_input_grad(1) || ctx->needs_input_grad(2) || ctx->needs_input_grad(3)) parts |= FLASHMHF_BWD_WEIGHTS;
        if (!parts) return variable_list(8);
        const Shape s{Q.size(0), Q.size(1), Q.size(2), Q.size(3), K.size(0), K.size(1), K.size(2)};
        Grads g = backward_checked(s, Q, K, U, V, R, grads[0], flashmhf_scaling{(float)sc[0], (float)sc[1], (float)sc[2]}, parts, nullptr);
        if (g.dR.defined() && R.scalar_type() != at::kFloat) g.dR = g.dR.to(R.scalar_type());
        return {g.dQ, g.dK, g.dU, g.dV, g.dR, Tensor(), Tensor(), Tensor()};
    }
};

Tensor flash_mhf(const Tensor &Q, const Tensor &K, const Tensor &U, const Tensor &V, const Tensor &R, double hs, double us, double fs) {
    return OpFunction::apply(Q, K, U, V, R, hs, us, fs);
}

// ------------------------------------------------------------------------------------------------ prologue
struct Prologue {
    Tensor x, w, r;   // projected activations [B,S,H*d_h]; norm weight and router as contiguous fp32 (w undefined: no RMSNorm)
    int64_t B, S, H, Dh, E;
    double eps;
};
Prologue prologue_args(const Tensor &x_proj, const std::optional<Tensor> &q_norm, const Tensor &router, double eps) {
    if (x_proj.scalar_type() != at::kBFloat16 || !x_proj.is_cuda())
        throw py::type_error("fused_prologue expects a CUDA bfloat16 activation tensor");
    if (x_proj.dim() != 3 || router.dim() != 3) throw py::value_error("expected activations [B,S,H*d_h] and a router [H,d_h,E]");
    Prologue a;
    a.H = router.size(0); a.Dh = router.size(1); a.E = router.size(2);
    a.B = x_proj.size(0); a.S = x_proj.size(1);
    if (x_proj.size(2) != a.H * a.Dh)
        throw py::value_error("hidden size " + std::to_string(x_proj.size(2)) + " != H*d_h = " + std::to_string(a.H) + "*" + std::to_string(a.Dh));
    if ((a.Dh != 64 && a.Dh != 96 && a.Dh != 128) || a.E > 32)
        throw py::value_error("fused_prologue supports d_h in {64, 96, 128} and at most 32 sub-networks");
    a.eps = eps;
    a.x = x_proj.contiguous();
    if (q_norm) a.w = q_norm->detach().to(at::kFloat).contiguous();
    a.r = router.detach().to(at::kFloat).contiguous();
    return a;
}
flashmhf_prologue_params prologue_params(const Prologue &a) {
    flashmhf_prologue_params p{};
    p.B = (int32_t)a.B; p.S = (int32_t)a.S; p.H = (int32_t)a.H; p.Dh = (int32_t)a.Dh; p.E = (int32_t)a.E;
    p.eps = (float)a.eps;
    p.X = a.x.data_ptr();
    p.x_token_stride = a.H * a.Dh;
    p.norm_weight = a.w.defined() ? a.w.data_ptr<float>() : nullptr;
    p.router = a.r.data_ptr<float>();
    return p;
}
// Q [B,S,H*d_h] in the activations' own layout (the activations themselves without RMSNorm) and R [B,H,S,E]
std::pair<Tensor, Tensor> run_prologue(const Prologue &a) {
    c10::cuda::CUDAGuard guard(a.x.device());
    Tensor q = a.w.defined() ? at::empty_like(a.x) : a.x;
    Tensor R = at::empty({a.B, a.H, a.S, a.E}, a.x.options().dtype(at::kFloat));
    flashmhf_prologue_params p = prologue_params(a);
    p.Q = q.data_ptr();
    p.R = R.data_ptr<float>();
    check(api.prologue_forward(&p, current_stream(a.x)));
    return {q, R};
}
struct PrologueGrads {
    Tensor dX, d_router, d_norm;
};
// dQ [B,H,S,d_h] with a unit inner stride, dR [B,H,S,E] contiguous fp32
PrologueGrads run_prologue_backward(const Prologue &a, const Tensor &dQ, const Tensor &dR) {
    c10::cuda::CUDAGuard guard(a.x.device());
    PrologueGrads g{at::empty_like(a.x), at::empty_like(a.r), a.w.defined() ? at::empty_like(a.w) : Tensor()};
    flashmhf_prologue_bwd_params p{};
    p.fwd = prologue_params(a);
    p.dQ = dQ.data_ptr();
    for (int i = 0; i < 3; ++i) p.dq_stride[i] = dQ.stride(i);
    p.dR = dR.data_ptr<float>();
    p.dX = g.dX.data_ptr();
    p.d_router = g.d_router.data_ptr<float>();
    p.d_norm_weight = g.d_norm.defined() ? g.d_norm.data_ptr<float>() : nullptr;
    p.workspace_bytes = api.prologue_backward_ws(&p.fwd);
    Tensor ws = at::empty({(int64_t)p.workspace_bytes}, a.x.options().dtype(at::kByte));
    p.workspace = ws.data_ptr();
    check(api.prologue_backward(&p, current_stream(a.x)));
    return g;
}
Tensor heads_view(const Tensor &t, int64_t H, int64_t Dh) {   // [B,S,H*d_h] memory as a [B,H,S,d_h] view
    return t.view({t.size(0), t.size(1), H, Dh}).transpose(1, 2);
}

struct PrologueFunction : public torch::autograd::Function<PrologueFunction> {
    static variable_list forward(AutogradContext *ctx, const Tensor &x_proj, const std::optional<Tensor> &q_norm, const Tensor &router,
                                 double eps) {
        const Prologue a = prologue_args(x_proj, q_norm, router, eps);
        auto [q, R] = run_prologue(a);
        ctx->save_for_backward({a.x, a.w, a.r});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["router_dtype"] = (int64_t)router.scalar_type();
        ctx->saved_data["norm_dtype"] = q_norm ? (int64_t)q_norm->scalar_type() : (int64_t)-1;
        return {heads_view(q, a.H, a.Dh), R};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        Prologue a{sv[0], sv[1], sv[2], sv[0].size(0), sv[0].size(1), sv[2].size(0), sv[2].size(1), sv[2].size(2),
                   ctx->saved_data["eps"].toDouble()};
        Tensor dQ = grads[0], dR = grads[1];
        if (!dQ.defined()) dQ = at::zeros({a.B, a.H, a.S, a.Dh}, a.x.options());
        if (!dR.defined()) dR = at::zeros({a.B, a.H, a.S, a.E}, a.x.options().dtype(at::kFloat));
        dQ = dQ.to(at::kBFloat16);
        if (dQ.stride(3) != 1) dQ = dQ.contiguous();
        PrologueGrads g = run_prologue_backward(a, dQ, dR.to(at::kFloat).contiguous());
        const int64_t nd = ctx->saved_data["norm_dtype"].toInt();
        if (nd >= 0) g.d_norm = g.d_norm.to((at::ScalarType)nd);
        return {g.dX, g.d_norm, g.d_router.to((at::ScalarType)ctx->saved_data["router_dtype"].toInt()), Tensor()};
    }
};
std::pair<Tensor, Tensor> fused_prologue(const Tensor &x_proj, const std::optional<Tensor> &q_norm, const Tensor &router, double eps) {
    variable_list o = PrologueFunction::apply(x_proj, q_norm, router, eps);
    return {o[0], o[1]};
}

// ------------------------------------------------------------------------------------------------ layer
// [I, H_kuv*d_h] parameter -> [H_kuv, E, d_e, d_h] strided view the operator reads in place (no copy)
Tensor expert_view(const Tensor &w, int64_t Hkuv, int64_t E) {
    const int64_t I = w.size(0), dh = w.size(1) / Hkuv;
    return w.view({E, I / E, Hkuv, dh}).permute({2, 0, 1, 3});
}

// Prologue and operator as one autograd node: projected activations [B,S,H*d_h] -> O [B,S,H*d_h].
struct LayerCoreFunction : public torch::autograd::Function<LayerCoreFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x_proj, const std::optional<Tensor> &q_norm, const Tensor &router,
                          const Tensor &gate, const Tensor &up, const Tensor &down, int64_t Hkuv, double eps, double hs, double us, double fs) {
        const Prologue a = prologue_args(x_proj, q_norm, router, eps);
        auto [q, R] = run_prologue(a);
        const Tensor Q = heads_view(q, a.H, a.Dh);
        const Tensor K = expert_view(gate, Hkuv, a.E), U = expert_view(up, Hkuv, a.E), V = expert_view(down, Hkuv, a.E);
        const Shape s = validate(Q, K, U, V, R);
        const Tensor O = forward_checked(s, Q, K, U, V, R, std::nullopt, scaling_of(hs, us, fs), false, std::nullopt);
        ctx->save_for_backward({a.x, a.w, a.r, q, R, gate, up, down});
        ctx->saved_data["k"] = std::vector<double>{eps, hs, us, fs};
        ctx->saved_data["i"] = std::vector<int64_t>{Hkuv, (int64_t)router.scalar_type(), q_norm ? (int64_t)q_norm->scalar_type() : (int64_t)-1};
        return O.transpose(1, 2).reshape({a.B, a.S, a.H * a.Dh});   // no copy: O has Q's layout
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        variable_list out(11);
        if (!grads[0].defined()) return out;
        const variable_list sv = ctx->get_saved_variables();
        const std::vector<double> k = ctx->saved_data["k"].toDoubleVector();
        const std::vector<int64_t> n = ctx->saved_data["i"].toIntVector();
        const Prologue a{sv[0], sv[1], sv[2], sv[0].size(0), sv[0].size(1), sv[2].size(0), sv[2].size(1), sv[2].size(2), k[0]};
        const Tensor Q = heads_view(sv[3], a.H, a.Dh), &R = sv[4];
        const Tensor K = expert_view(sv[5], n[0], a.E), U = expert_view(sv[6], n[0], a.E), V = expert_view(sv[7], n[0], a.E);
        uint32_t parts = 0;
        const int nt = a.w.defined() ? 6 : 5;   // tensor arguments present: x, (norm weight), router, then the three weights
        for (int i = 0; i < nt; ++i)
            if (ctx->needs_input_grad(i)) parts |= i < nt - 3 ? FLASHMHF_BWD_INPUTS : FLASHMHF_BWD_WEIGHTS;
        if (!parts) return out;
        const Shape s{a.B, a.H, a.S, a.Dh, n[0], a.E, K.size(2)};
        const Tensor dO = grads[0].reshape({a.B, a.S, a.H, a.Dh}).transpose(1, 2);
        const Grads g = backward_checked(s, Q, K, U, V, R, dO, flashmhf_scaling{(float)k[1], (float)k[2], (float)k[3]}, parts, nullptr);
        if (parts & FLASHMHF_BWD_INPUTS) {
            PrologueGrads pg = run_prologue_backward(a, g.dQ, g.dR);
            out[0] = pg.dX;
            if (pg.d_norm.defined()) out[1] = pg.d_norm.to((at::ScalarType)n[2]);
            out[2] = pg.d_router.to((at::ScalarType)n[1]);
        }
        if (parts & FLASHMHF_BWD_WEIGHTS) {
            auto param = [&](const Tensor &d, const Tensor &w) { return d.permute({1, 2, 0, 3}).reshape(w.sizes()); };
            out[3] = param(g.dK, sv[5]);
            out[4] = param(g.dU, sv[6]);
            out[5] = param(g.dV, sv[7]);
        }
        return out;
    }
};

Tensor mhffn_layer(const Tensor &x, const std::optional<Tensor> &w1, const std::optional<Tensor> &b1, const std::optional<Tensor> &q_norm,
                   const Tensor &router, const Tensor &gate, const Tensor &up, const Tensor &down, const std::optional<Tensor> &w2,
                   const std::optional<Tensor> &b2, int64_t Hkuv, double eps, double hs, double us, double fs) {
    const Tensor q_lin = w1 ? at::linear(x, *w1, b1) : x;
    const Tensor O = LayerCoreFunction::apply(q_lin, q_norm, router, gate, up, down, Hkuv, eps, hs, us, fs);
    return w2 ? at::linear(O, *w2, b2) : O;
}

// ------------------------------------------------------------------------------------------------ LM helpers
Tensor run_rope(const Tensor &x, const Tensor &cos_t, const Tensor &sin_t, bool transpose) {
    c10::cuda::CUDAGuard guard(x.device());
    Tensor y = at::empty_like(x);
    const int64_t B = x.size(0), S = x.size(1), nh = x.size(2), hd = x.size(3);
    check(api.lm_rope(x.data_ptr(), y.data_ptr(), cos_t.data_ptr<float>(), sin_t.data_ptr<float>(), B * S, (int32_t)S, (int32_t)nh,
                      (int32_t)hd, nh * hd, nh * hd, transpose ? 1 : 0, current_stream(x)));
    return y;
}
struct RotaryFunction : public torch::autograd::Function<RotaryFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x, const Tensor &cos_t, const Tensor &sin_t) {
        ctx->save_for_backward({cos_t, sin_t});
        return run_rope(x.contiguous(), cos_t, sin_t, false);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        return {run_rope(grads[0].contiguous(), sv[0], sv[1], true), Tensor(), Tensor()};
    }
};
Tensor rotary(const Tensor &x, const Tensor &cos_t, const Tensor &sin_t) { return RotaryFunction::apply(x, cos_t, sin_t); }

struct RMSNormFunction : public torch::autograd::Function<RMSNormFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x0, const Tensor &weight, double eps) {
        const Tensor x = x0.contiguous(), w = weight.detach().to(at::kFloat).contiguous();
        c10::cuda::CUDAGuard guard(x.device());
        Tensor y = at::empty_like(x);
        const int64_t n = x.size(-1);
        check(api.rmsnorm_forward(x.data_ptr(), w.data_ptr<float>(), y.data_ptr(), x.numel() / n, (int32_t)n, (float)eps, current_stream(x)));
        ctx->save_for_backward({x, w});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["dtype"] = (int64_t)weight.scalar_type();
        return y;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Tensor &x = sv[0], &w = sv[1];
        const Tensor g = grads[0].contiguous();
        c10::cuda::CUDAGuard guard(x.device());
        Tensor dx = at::empty_like(x), dw = at::empty_like(w);
        const int64_t n = x.size(-1), rows = x.numel() / n;
        const size_t nbytes = api.rmsnorm_backward_ws(rows, (int32_t)n);
        Tensor ws = at::empty({(int64_t)nbytes}, x.options().dtype(at::kByte));
        check(api.rmsnorm_backward(x.data_ptr(), w.data_ptr<float>(), g.data_ptr(), dx.data_ptr(), dw.data_ptr<float>(), ws.data_ptr(),
                                   nbytes, rows, (int32_t)n, (float)ctx->saved_data["eps"].toDouble(), current_stream(x)));
        return {dx, dw.to((at::ScalarType)ctx->saved_data["dtype"].toInt()), Tensor()};
    }
};
Tensor rmsnorm(const Tensor &x, const Tensor &weight, double eps) { return RMSNormFunction::apply(x, weight, eps); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("op_forward", torch::wrap_pybind_function(op_forward));
    m.def("op_backward", torch::wrap_pybind_function(op_backward));
    m.def("flash_mhf", torch::wrap_pybind_function(flash_mhf));
    m.def("fused_prologue", torch::wrap_pybind_function(fused_prologue));
    m.def("mhffn_layer", torch::wrap_pybind_function(mhffn_layer));
    m.def("rotary", torch::wrap_pybind_function(rotary));
    m.def("rmsnorm", torch::wrap_pybind_function(rmsnorm));
}

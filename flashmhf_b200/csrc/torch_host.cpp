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
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
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
    decltype(&flashmhf_backward) backward = nullptr, backward_inputs = nullptr;
    decltype(&flashmhf_forward_workspace_bytes) forward_ws = nullptr;
    decltype(&flashmhf_backward_workspace_bytes) backward_ws = nullptr, backward_inputs_ws = nullptr;
    decltype(&flashmhf_prologue_forward_dtype) prologue_forward = nullptr;
    decltype(&flashmhf_prologue_backward_workspace_bytes) prologue_backward_ws = nullptr;
    decltype(&flashmhf_prologue_backward_dtype) prologue_backward = nullptr;
    decltype(&flashmhf_lm_rope) lm_rope = nullptr;
    decltype(&flashmhf_lm_rmsnorm_forward_dtype) rmsnorm_forward = nullptr;
    decltype(&flashmhf_lm_rmsnorm_backward_workspace_bytes) rmsnorm_backward_ws = nullptr;
    decltype(&flashmhf_lm_rmsnorm_backward_dtype) rmsnorm_backward = nullptr;
    decltype(&flashmhf_lm_rope_pair) lm_rope_pair = nullptr;
    decltype(&flashmhf_lm_add_rmsnorm_forward) add_rmsnorm_forward = nullptr;
    decltype(&flashmhf_lm_add_rmsnorm_backward) add_rmsnorm_backward = nullptr;
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
    get(api.backward_inputs, "flashmhf_backward_inputs");
    get(api.forward_ws, "flashmhf_forward_workspace_bytes");
    get(api.backward_ws, "flashmhf_backward_workspace_bytes");
    get(api.backward_inputs_ws, "flashmhf_backward_inputs_workspace_bytes");
    get(api.prologue_forward, "flashmhf_prologue_forward_dtype");
    get(api.prologue_backward_ws, "flashmhf_prologue_backward_workspace_bytes");
    get(api.prologue_backward, "flashmhf_prologue_backward_dtype");
    get(api.lm_rope, "flashmhf_lm_rope");
    get(api.rmsnorm_forward, "flashmhf_lm_rmsnorm_forward_dtype");
    get(api.rmsnorm_backward_ws, "flashmhf_lm_rmsnorm_backward_workspace_bytes");
    get(api.rmsnorm_backward, "flashmhf_lm_rmsnorm_backward_dtype");
    get(api.lm_rope_pair, "flashmhf_lm_rope_pair");
    get(api.add_rmsnorm_forward, "flashmhf_lm_add_rmsnorm_forward");
    get(api.add_rmsnorm_backward, "flashmhf_lm_add_rmsnorm_backward");
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

bool has_tangent(const Tensor &t) { return t.defined() && t._fw_grad(/*level=*/0).defined(); }

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
// The call itself, from addresses and strides: how much scratch it needs, and the launch.
void as_sequence(flashmhf_fwd_params &p) {
    if (p.d.S == 1 && p.d.B > 1) {
        p.Q = tokens_as_sequence(p.Q); p.R = tokens_as_sequence(p.R); p.O = tokens_as_sequence(p.O);
        p.d.S = p.d.B;
        p.d.B = 1;
    }
    p.workspace_bytes = api.forward_ws(&p.d);
}
void launch_forward(flashmhf_fwd_params &p, const Tensor &like, bool chained, const std::optional<Tensor> &workspace) {
    as_sequence(p);
    Tensor ws;
    if (p.workspace_bytes) {
        ws = scratch(workspace, p.workspace_bytes, like);
        p.workspace = ws.data_ptr();
    }
    check((chained ? api.forward_chained : api.forward)(&p, current_stream(like)));
}

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
    launch_forward(p, Q, chained, workspace);
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
    }
    p.workspace_bytes = weights ? api.backward_ws(&p.d) : api.backward_inputs_ws(&p.d);
    if (p.workspace_bytes) {
        ws = at::empty({(int64_t)p.workspace_bytes}, Q.options().dtype(at::kByte));
        p.workspace = ws.data_ptr();
    }
    check((weights ? api.backward : api.backward_inputs)(&p, current_stream(Q)));
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
    Tensor x, w, r;   // projected activations [B,S,H*d_h]; norm weight (undefined: no RMSNorm) and router, both bf16 or both fp32
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
    for (const Tensor *t : {&router, q_norm ? &*q_norm : &router})
        if (t->device() != x_proj.device()) throw py::value_error("router and norm weight must be on the activations' device, " + x_proj.device().str());
    if (q_norm && q_norm->numel() != a.H * a.Dh)
        throw py::value_error("norm weight must have " + std::to_string(a.H) + "*" + std::to_string(a.Dh) + " values, got " + dims_text(*q_norm));
    a.eps = eps;
    a.x = x_proj.contiguous();
    // bf16 parameters are read as they are; any other mix goes in as fp32
    const bool bf16 = router.scalar_type() == at::kBFloat16 && (!q_norm || q_norm->scalar_type() == at::kBFloat16);
    const auto dt = bf16 ? at::kBFloat16 : at::kFloat;
    if (q_norm) a.w = q_norm->detach().to(dt).contiguous();
    a.r = router.detach().to(dt).contiguous();
    return a;
}
flashmhf_prologue_params prologue_params(const Prologue &a) {
    flashmhf_prologue_params p{};
    p.B = (int32_t)a.B; p.S = (int32_t)a.S; p.H = (int32_t)a.H; p.Dh = (int32_t)a.Dh; p.E = (int32_t)a.E;
    p.eps = (float)a.eps;
    p.X = a.x.data_ptr();
    p.x_token_stride = a.H * a.Dh;
    p.norm_weight = a.w.defined() ? static_cast<const float *>(a.w.data_ptr()) : nullptr;   // in the type dtype_code(a.r) names
    p.router = static_cast<const float *>(a.r.data_ptr());
    return p;
}
int32_t dtype_code(const Tensor &param) { return param.scalar_type() == at::kBFloat16 ? FLASHMHF_BF16 : FLASHMHF_F32_CHECK; }
// Q [B,S,H*d_h] in the activations' own layout (the activations themselves without RMSNorm) and R [B,H,S,E]
void launch_prologue(const Prologue &a, void *q, void *R) {
    flashmhf_prologue_params p = prologue_params(a);
    p.Q = q;
    p.R = static_cast<float *>(R);
    check(api.prologue_forward(&p, dtype_code(a.r), current_stream(a.x)));
}
std::pair<Tensor, Tensor> run_prologue(const Prologue &a) {
    c10::cuda::CUDAGuard guard(a.x.device());
    Tensor q = a.w.defined() ? at::empty_like(a.x) : a.x;
    Tensor R = at::empty({a.B, a.H, a.S, a.E}, a.x.options().dtype(at::kFloat));
    launch_prologue(a, q.data_ptr(), R.data_ptr());
    return {q, R};
}
struct PrologueGrads {
    Tensor dX, d_router, d_norm;
};
// dQ [B,H,S,d_h] bf16 with a unit inner stride, dR [B,H,S,E] contiguous fp32
PrologueGrads run_prologue_backward(const Prologue &a, const void *dQ, const int64_t *dq_stride, const float *dR) {
    c10::cuda::CUDAGuard guard(a.x.device());
    PrologueGrads g{at::empty_like(a.x), at::empty_like(a.r), a.w.defined() ? at::empty_like(a.w) : Tensor()};
    flashmhf_prologue_bwd_params p{};
    p.fwd = prologue_params(a);
    p.dQ = dQ;
    for (int i = 0; i < 3; ++i) p.dq_stride[i] = dq_stride[i];
    p.dR = dR;
    p.dX = g.dX.data_ptr();
    p.d_router = static_cast<float *>(g.d_router.data_ptr());
    p.d_norm_weight = g.d_norm.defined() ? static_cast<float *>(g.d_norm.data_ptr()) : nullptr;
    p.workspace_bytes = api.prologue_backward_ws(&p.fwd);
    Tensor ws = at::empty({(int64_t)p.workspace_bytes}, a.x.options().dtype(at::kByte));
    p.workspace = ws.data_ptr();
    check(api.prologue_backward(&p, dtype_code(a.r), current_stream(a.x)));
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
        auto rows = [](const Tensor &t) { return t.defined() ? t.contiguous() : t; };   // (a hook may have given back another layout)
        Prologue a{rows(sv[0]), rows(sv[1]), rows(sv[2]), sv[0].size(0), sv[0].size(1), sv[2].size(0), sv[2].size(1), sv[2].size(2),
                   ctx->saved_data["eps"].toDouble()};
        Tensor dQ = grads[0], dR = grads[1];
        if (!dQ.defined()) dQ = at::zeros({a.B, a.H, a.S, a.Dh}, a.x.options());
        if (!dR.defined()) dR = at::zeros({a.B, a.H, a.S, a.E}, a.x.options().dtype(at::kFloat));
        dQ = dQ.to(at::kBFloat16);
        if (dQ.stride(3) != 1) dQ = dQ.contiguous();
        dR = dR.to(at::kFloat).contiguous();
        PrologueGrads g = run_prologue_backward(a, dQ.data_ptr(), dQ.strides().data(), dR.data_ptr<float>());
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
// The same view, and the [B,H,S,*] views of activations and routing weights, as addresses and strides only: a torch view
// costs the host about as much as an allocation, and a layer call needs a dozen of them each way.
flashmhf_tensor expert_address(const Tensor &w, int64_t Dh, int64_t De) {
    const int64_t ld = w.stride(0);
    return flashmhf_tensor{w.data_ptr(), {Dh, De * ld, ld}};
}
flashmhf_tensor heads_address(void *p, const Prologue &a) { return flashmhf_tensor{p, {a.S * a.H * a.Dh, a.Dh, a.H * a.Dh}}; }
flashmhf_tensor routing_address(void *p, const Prologue &a) { return flashmhf_tensor{p, {a.H * a.S * a.E, a.S * a.E, a.E}}; }
// Can the operator read this parameter as it lies? (the rule of in_place_ok for the view above)
bool expert_ok(const Tensor &w) {
    return w.dim() == 2 && w.scalar_type() == at::kBFloat16 && w.stride(1) == 1 && w.stride(0) % 8 == 0 && w.stride(0) >= w.size(1) &&
           !(reinterpret_cast<uintptr_t>(w.data_ptr()) & 15u);
}
size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

// The whole layer as one autograd node: projection, prologue, operator, projection.  As separate nodes its backward is a
// dozen small steps of the autograd engine (views, transposes and products of the two linear maps, the prologue, the
// operator), which on short inputs take the host longer than their kernels take the GPU.
Shape layer_shape(const Prologue &a, const Tensor &gate, const Tensor &up, const Tensor &down, int64_t Hkuv) {
    const int64_t I = gate.size(0);
    if (Hkuv < 1 || a.H % Hkuv != 0)
        throw py::value_error("num_heads " + std::to_string(a.H) + " must be a multiple of num_kuv_heads " + std::to_string(Hkuv));
    if (gate.size(1) != Hkuv * a.Dh || up.sizes() != gate.sizes() || down.sizes() != gate.sizes() || I % a.E != 0)
        throw py::value_error("gate, up and down weights must be [E*d_e, H_kuv*d_h], got " + dims_text(gate) + ", " + dims_text(up) + ", " +
                              dims_text(down));
    if ((I / a.E) % 64 != 0) throw py::value_error("Expert dimension " + std::to_string(I / a.E) + " must be divisible by 64");
    if (gate.device() != a.x.device() || up.device() != a.x.device() || down.device() != a.x.device())
        throw py::value_error("flash_mhf runs on CUDA tensors of one device; there is no CPU path");
    return Shape{a.B, a.H, a.S, a.Dh, Hkuv, a.E, I / a.E};
}
// x [B,S,n] times w^T: one product on the flattened rows (at::linear takes more steps to the same call)
Tensor project(const Tensor &x, const Tensor &w, const std::optional<Tensor> &b) {
    if (b || !x.is_contiguous()) return at::linear(x, w, b);
    return at::mm(x.view({x.size(0) * x.size(1), x.size(2)}), w.t()).view({x.size(0), x.size(1), w.size(0)});
}
struct LayerForward {
    Prologue a;
    Tensor q, R, O, y;   // q and R only where they are to be kept for a backward
};
LayerForward layer_forward(const Tensor &x, const std::optional<Tensor> &w1, const std::optional<Tensor> &b1,
                           const std::optional<Tensor> &q_norm, const Tensor &router, const Tensor &gate, const Tensor &up,
                           const Tensor &down, const std::optional<Tensor> &w2, const std::optional<Tensor> &b2, int64_t Hkuv, double eps,
                           double hs, double us, double fs, bool keep) {
    at::AutoDispatchBelowADInplaceOrView below;   // nothing in here is recorded: the caller is the autograd node, or there is none
    c10::cuda::CUDAGuard guard(x.device());
    LayerForward f{prologue_args(w1 ? project(x, *w1, b1) : x, q_norm, router, eps)};
    const Prologue &a = f.a;
    const Shape s = layer_shape(a, gate, up, down, Hkuv);
    f.O = at::empty_like(a.x);
    flashmhf_fwd_params p{};
    p.d = dims_of(s, at::kBFloat16);
    p.scale = scaling_of(hs, us, fs);
    p.K = expert_address(gate, s.Dh, s.De); p.U = expert_address(up, s.Dh, s.De); p.V = expert_address(down, s.Dh, s.De);
    p.O = heads_address(f.O.data_ptr(), a);
    // (chained: the operation directly before the operator is this layer's prologue, which does not write the weights)
    if (keep) {
        std::tie(f.q, f.R) = run_prologue(a);
        p.Q = heads_address(f.q.data_ptr(), a); p.R = routing_address(f.R.data_ptr(), a);
        launch_forward(p, a.x, true, std::nullopt);
    } else {   // Q, R and the operator's scratch in one allocation
        flashmhf_fwd_params need = p;
        as_sequence(need);
        const size_t q_bytes = a.w.defined() ? align256((size_t)a.B * a.S * a.H * a.Dh * 2) : 0, r_bytes = align256((size_t)a.B * a.S * a.H * a.E * 4);
        const Tensor tmp = at::empty({(int64_t)(q_bytes + r_bytes + need.workspace_bytes)}, a.x.options().dtype(at::kByte));
        char *base = static_cast<char *>(tmp.data_ptr());
        void *q = q_bytes ? base : a.x.data_ptr();
        launch_prologue(a, q, base + q_bytes);
        p.Q = heads_address(q, a); p.R = routing_address(base + q_bytes, a);
        as_sequence(p);
        p.workspace = p.workspace_bytes ? base + q_bytes + r_bytes : nullptr;
        check(api.forward_chained(&p, current_stream(a.x)));
    }
    f.y = w2 ? project(f.O, *w2, b2) : f.O;
    return f;
}

struct LayerFunction : public torch::autograd::Function<LayerFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x, const std::optional<Tensor> &w1, const std::optional<Tensor> &b1,
                          const std::optional<Tensor> &q_norm, const Tensor &router, const Tensor &gate, const Tensor &up,
                          const Tensor &down, const std::optional<Tensor> &w2, const std::optional<Tensor> &b2, int64_t Hkuv, double eps,
                          double hs, double us, double fs) {
        const LayerForward f = layer_forward(x, w1, b1, q_norm, router, gate, up, down, w2, b2, Hkuv, eps, hs, us, fs, true);
        const Prologue &a = f.a;
        const Tensor &q = f.q, &R = f.R, &O = f.O;
        ctx->save_for_backward({w1 ? x : Tensor(), w1 ? *w1 : Tensor(), a.x, a.w, a.r, q, R, gate, up, down, w2 ? O : Tensor(),
                                w2 ? *w2 : Tensor()});
        ctx->saved_data["k"] = std::vector<double>{eps, hs, us, fs};
        ctx->saved_data["i"] = std::vector<int64_t>{Hkuv, (int64_t)router.scalar_type(), q_norm ? (int64_t)q_norm->scalar_type() : (int64_t)-1,
                                                    (int64_t)b1.has_value(), (int64_t)b2.has_value()};
        return f.y;
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        variable_list out(15);
        if (!grads[0].defined()) return out;
        const variable_list sv = ctx->get_saved_variables();   // (may run the caller's hooks, and a checkpointed region again)
        std::optional<at::AutoDispatchBelowADInplaceOrView> below;
        if (!at::GradMode::is_enabled()) below.emplace();
        const std::vector<double> k = ctx->saved_data["k"].toDoubleVector();
        const std::vector<int64_t> n = ctx->saved_data["i"].toIntVector();
        // The kernels take these by address, in the layout in which they were saved; what a hook gave back may have another.
        const Tensor &x = sv[0], &w1 = sv[1], &w2 = sv[11];
        auto rows = [](const Tensor &t) { return t.defined() ? t.contiguous() : t; };
        auto weight = [](const Tensor &t) { return expert_ok(t) ? t : t.contiguous(); };
        const Tensor q = rows(sv[5]), R = rows(sv[6]), O = rows(sv[10]);
        const Prologue a{rows(sv[2]), rows(sv[3]), rows(sv[4]), sv[2].size(0), sv[2].size(1), sv[4].size(0), sv[4].size(1), sv[4].size(2), k[0]};
        // which arguments want a gradient (autograd numbers the tensors that were passed)
        const bool given[10] = {true, w1.defined(), n[3] != 0, a.w.defined(), true, true, true, true, w2.defined(), n[4] != 0};
        bool need[10];
        for (int i = 0, edge = 0; i < 10; ++i) need[i] = given[i] && ctx->needs_input_grad(edge++);
        const int64_t T = a.B * a.S, hid = a.H * a.Dh;
        uint32_t parts = 0;
        if (need[0] || need[1] || need[2] || need[3] || need[4]) parts |= FLASHMHF_BWD_INPUTS;
        if (need[5] || need[6] || need[7]) parts |= FLASHMHF_BWD_WEIGHTS;

        Tensor d = grads[0].reshape({T, grads[0].size(2)});
        if (need[8]) out[8] = d.t().mm(O.view({T, hid}));
        if (need[9]) out[9] = d.sum(0);
        if (!parts) return out;
        if (w2.defined()) d = d.mm(w2);
        d = d.contiguous();
        const bool inputs = parts & FLASHMHF_BWD_INPUTS, weights = parts & FLASHMHF_BWD_WEIGHTS;
        const Tensor gate = weight(sv[7]), up = weight(sv[8]), down = weight(sv[9]);
        c10::cuda::CUDAGuard guard(d.device());
        flashmhf_bwd_params p{};
        p.d = dims_of(Shape{a.B, a.H, a.S, a.Dh, n[0], a.E, gate.size(0) / a.E}, at::kBFloat16);
        // dQ, dR and the scratch of the operator live until the prologue's backward has run: one allocation for all three
        const size_t dq_bytes = align256((size_t)T * hid * 2), dr_bytes = align256((size_t)T * a.H * a.E * 4);
        p.workspace_bytes = weights ? api.backward_ws(&p.d) : api.backward_inputs_ws(&p.d);
        const Tensor tmp = at::empty({(int64_t)(dq_bytes + dr_bytes + p.workspace_bytes + 1)}, d.options().dtype(at::kByte));
        char *base = static_cast<char *>(tmp.data_ptr());
        p.Q = heads_address(q.data_ptr(), a); p.dO = heads_address(d.data_ptr(), a); p.R = routing_address(R.data_ptr(), a);
        p.K = expert_address(gate, a.Dh, p.d.De); p.U = expert_address(up, a.Dh, p.d.De); p.V = expert_address(down, a.Dh, p.d.De);
        p.dQ = heads_address(base, a); p.dR = routing_address(base + dq_bytes, a);
        p.workspace = base + dq_bytes + dr_bytes;
        p.scale = flashmhf_scaling{(float)k[1], (float)k[2], (float)k[3]};
        p.parts = parts;
        if (weights) {
            out[5] = at::empty_like(gate); out[6] = at::empty_like(up); out[7] = at::empty_like(down);
            p.dK = expert_address(out[5], a.Dh, p.d.De); p.dU = expert_address(out[6], a.Dh, p.d.De); p.dV = expert_address(out[7], a.Dh, p.d.De);
        }
        check((weights ? api.backward : api.backward_inputs)(&p, current_stream(d)));
        if (inputs) {
            const PrologueGrads pg = run_prologue_backward(a, static_cast<char *>(p.dQ.ptr), p.dQ.stride, static_cast<float *>(p.dR.ptr));
            if (pg.d_norm.defined()) out[3] = pg.d_norm.to((at::ScalarType)n[2]);
            out[4] = pg.d_router.to((at::ScalarType)n[1]);
            if (w1.defined()) {
                const Tensor dp = pg.dX.view({T, hid});
                if (need[1]) out[1] = dp.t().mm(x.reshape({T, x.size(2)}));
                if (need[2]) out[2] = dp.sum(0);
                if (need[0]) out[0] = dp.mm(w1).view(x.sizes());
            } else {
                out[0] = pg.dX;
            }
        }
        return out;
    }
};

Tensor mhffn_layer(const Tensor &x, const std::optional<Tensor> &w1, const std::optional<Tensor> &b1, const std::optional<Tensor> &q_norm,
                   const Tensor &router, const Tensor &gate, const Tensor &up, const Tensor &down, const std::optional<Tensor> &w2,
                   const std::optional<Tensor> &b2, int64_t Hkuv, double eps, double hs, double us, double fs) {
    auto plain = [](const std::optional<Tensor> &t) { return !t || t->scalar_type() == at::kBFloat16; };
    if (x.is_cuda() && x.dim() == 3 && expert_ok(gate) && expert_ok(up) && expert_ok(down) && plain(x) && plain(w1) && plain(b1) && plain(w2) &&
        plain(b2) && !at::autocast::is_autocast_enabled(at::kCUDA)) {
        // (a tangent goes through the node as well, which refuses it: there is no forward-mode derivative)
        const bool grad = at::GradMode::is_enabled();
        auto wants = [grad](const std::optional<Tensor> &t) { return t && ((grad && t->requires_grad()) || has_tangent(*t)); };
        if (wants(x) || wants(w1) || wants(b1) || wants(q_norm) || wants(router) || wants(gate) || wants(up) || wants(down) || wants(w2) || wants(b2))
            return LayerFunction::apply(x, w1, b1, q_norm, router, gate, up, down, w2, b2, Hkuv, eps, hs, us, fs);
        return layer_forward(x, w1, b1, q_norm, router, gate, up, down, w2, b2, Hkuv, eps, hs, us, fs, false).y;
    }
    // other dtypes, autocast, or weights that have to be copied first: torch's own rules for each step
    auto [Q, R] = fused_prologue(w1 ? at::linear(x, *w1, b1) : x, q_norm, router, eps);
    const int64_t E = router.size(2);
    const Tensor O = flash_mhf(Q, expert_view(gate, Hkuv, E), expert_view(up, Hkuv, E), expert_view(down, Hkuv, E), R, hs, us, fs)
                         .transpose(1, 2).reshape({x.size(0), x.size(1), router.size(0) * router.size(1)});
    return w2 ? at::linear(O, *w2, b2) : O;
}

// ------------------------------------------------------------------------------------------------ LM helpers
// The kernels take addresses and trust the sizes: bf16 [B,S,heads,hd] with tables of at least S rows of hd/2, all on one GPU.
void check_rope(const Tensor &x, const Tensor &cos_t, const Tensor &sin_t) {
    if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() != 4) throw py::value_error("rotary embedding expects CUDA bf16 [B,S,heads,head_dim]");
    for (const Tensor &t : {cos_t, sin_t})
        if (t.device() != x.device() || t.scalar_type() != at::kFloat || t.dim() < 1 || !t.is_contiguous() || t.size(-1) * 2 != x.size(3) ||
            t.numel() < x.size(1) * t.size(-1))
            throw py::value_error("rotary tables must be contiguous fp32 [S or more, head_dim/2] on the activations' device");
}
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
        check_rope(x, cos_t, sin_t);
        ctx->save_for_backward({cos_t, sin_t});
        return run_rope(x.contiguous(), cos_t, sin_t, false);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        return {run_rope(grads[0].contiguous(), sv[0], sv[1], true), Tensor(), Tensor()};
    }
};
Tensor rotary(const Tensor &x, const Tensor &cos_t, const Tensor &sin_t) { return RotaryFunction::apply(x, cos_t, sin_t); }

// bf16 [..., n] and a weight of n values on the same GPU
void check_norm(const Tensor &x, const Tensor &weight) {
    if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() < 1) throw py::value_error("RMSNorm expects a CUDA bf16 tensor");
    if (weight.device() != x.device() || weight.numel() != x.size(-1))
        throw py::value_error("RMSNorm weight must have " + std::to_string(x.size(-1)) + " values on " + x.device().str() + ", got " + dims_text(weight));
}
struct RMSNormFunction : public torch::autograd::Function<RMSNormFunction> {
    static Tensor forward(AutogradContext *ctx, const Tensor &x0, const Tensor &weight, double eps) {
        check_norm(x0, weight);
        const Tensor x = x0.contiguous();
        const Tensor w = (weight.scalar_type() == at::kBFloat16 ? weight.detach() : weight.detach().to(at::kFloat)).contiguous();
        c10::cuda::CUDAGuard guard(x.device());
        Tensor y = at::empty_like(x);
        const int64_t n = x.size(-1);
        check(api.rmsnorm_forward(x.data_ptr(), w.data_ptr(), dtype_code(w), y.data_ptr(), x.numel() / n, (int32_t)n, (float)eps, current_stream(x)));
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
        check(api.rmsnorm_backward(x.data_ptr(), w.data_ptr(), dtype_code(w), g.data_ptr(), dx.data_ptr(), dw.data_ptr(),
                                   ws.data_ptr(), nbytes, rows, (int32_t)n, (float)ctx->saved_data["eps"].toDouble(), current_stream(x)));
        return {dx, dw.to((at::ScalarType)ctx->saved_data["dtype"].toInt()), Tensor()};
    }
};
Tensor rmsnorm(const Tensor &x, const Tensor &weight, double eps) { return RMSNormFunction::apply(x, weight, eps); }

void check_rope_pair(const Tensor &q, const Tensor &k, const Tensor &cos_t, const Tensor &sin_t) {
    check_rope(q, cos_t, sin_t);
    check_rope(k, cos_t, sin_t);
    if (k.device() != q.device() || k.size(0) != q.size(0) || k.size(1) != q.size(1)) throw py::value_error("queries and keys must have the same B and S");
}
// queries [B,S,nq,hd] and keys [B,S,nk,hd], both rotated in one launch
variable_list run_rope_pair(const Tensor &q, const Tensor &k, const Tensor &cos_t, const Tensor &sin_t, bool transpose) {
    c10::cuda::CUDAGuard guard(q.device());
    Tensor yq = at::empty_like(q), yk = at::empty_like(k);
    const int64_t B = q.size(0), S = q.size(1);
    check(api.lm_rope_pair(q.data_ptr(), yq.data_ptr(), (int32_t)q.size(2), k.data_ptr(), yk.data_ptr(), (int32_t)k.size(2),
                           cos_t.data_ptr<float>(), sin_t.data_ptr<float>(), B * S, (int32_t)S, (int32_t)q.size(3), transpose ? 1 : 0,
                           current_stream(q)));
    return {yq, yk};
}
struct RotaryPairFunction : public torch::autograd::Function<RotaryPairFunction> {
    static variable_list forward(AutogradContext *ctx, const Tensor &q, const Tensor &k, const Tensor &cos_t, const Tensor &sin_t) {
        check_rope_pair(q, k, cos_t, sin_t);
        ctx->save_for_backward({cos_t, sin_t});
        ctx->saved_data["shape"] = std::vector<int64_t>{q.size(2), k.size(2)};
        return run_rope_pair(q.contiguous(), k.contiguous(), cos_t, sin_t, false);
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        variable_list out(4);
        if (grads[0].defined() && grads[1].defined()) {
            variable_list d = run_rope_pair(grads[0].contiguous(), grads[1].contiguous(), sv[0], sv[1], true);
            out[0] = d[0];
            out[1] = d[1];
        } else {
            for (int i = 0; i < 2; ++i)
                if (grads[i].defined()) out[i] = run_rope(grads[i].contiguous(), sv[0], sv[1], true);
        }
        return out;
    }
};
std::pair<Tensor, Tensor> rotary_pair(const Tensor &q, const Tensor &k, const Tensor &cos_t, const Tensor &sin_t) {
    variable_list o = RotaryPairFunction::apply(q, k, cos_t, sin_t);
    return {o[0], o[1]};
}

// Self-attention of the LM without gradients: projections, rotary embedding, library attention, projection (the steps of
// lm.Attention.forward; a forward pass over a short input waits for the interpreter, not for the GPU).
Tensor lm_attention(const Tensor &x, const Tensor &wq, const Tensor &wk, const Tensor &wv, const Tensor &wo, int64_t nh, int64_t nkv,
                    const Tensor &cos_t, const Tensor &sin_t) {
    for (const Tensor &t : {x, wq, wk, wv, wo}) TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(t), "attention in one call has no forward-mode derivative");
    at::AutoDispatchBelowADInplaceOrView below;
    const int64_t B = x.size(0), S = x.size(1), hd = wq.size(0) / nh;
    auto heads = [&](const Tensor &w, int64_t n) { return project(x, w, std::nullopt).view({B, S, n, hd}); };
    const Tensor q = heads(wq, nh), k = heads(wk, nkv), v = heads(wv, nkv).transpose(1, 2);
    check_rope_pair(q, k, cos_t, sin_t);
    const variable_list r = run_rope_pair(q, k, cos_t, sin_t, false);
    const Tensor o = at::scaled_dot_product_attention(r[0].transpose(1, 2), r[1].transpose(1, 2), v, std::nullopt, 0.0, /*is_causal=*/true,
                                                      std::nullopt, /*enable_gqa=*/nkv != nh);
    return project(o.transpose(1, 2).reshape({B, S, nh * hd}), wo, std::nullopt);
}

// (h + d, RMSNorm(h + d) * weight)
struct AddRMSNormFunction : public torch::autograd::Function<AddRMSNormFunction> {
    static variable_list forward(AutogradContext *ctx, const Tensor &h0, const Tensor &d0, const Tensor &weight, double eps) {
        check_norm(h0, weight);
        if (d0.sizes() != h0.sizes() || d0.scalar_type() != h0.scalar_type() || d0.device() != h0.device())
            throw py::value_error("add_rmsnorm expects two tensors alike, got " + dims_text(h0) + " and " + dims_text(d0));
        const Tensor h = h0.contiguous(), d = d0.contiguous();
        const Tensor w = (weight.scalar_type() == at::kBFloat16 ? weight.detach() : weight.detach().to(at::kFloat)).contiguous();
        c10::cuda::CUDAGuard guard(h.device());
        Tensor sum = at::empty_like(h), y = at::empty_like(h);
        const int64_t n = h.size(-1);
        check(api.add_rmsnorm_forward(h.data_ptr(), d.data_ptr(), w.data_ptr(), dtype_code(w), sum.data_ptr(), y.data_ptr(), h.numel() / n,
                                      (int32_t)n, (float)eps, current_stream(h)));
        ctx->save_for_backward({sum, w});
        ctx->saved_data["eps"] = eps;
        ctx->saved_data["dtype"] = (int64_t)weight.scalar_type();
        return {sum, y};
    }
    static variable_list backward(AutogradContext *ctx, variable_list grads) {
        const variable_list sv = ctx->get_saved_variables();
        const Tensor &sum = sv[0], &w = sv[1];
        if (!grads[1].defined()) return {grads[0], grads[0], Tensor(), Tensor()};
        const Tensor g = grads[1].contiguous(), gh = grads[0].defined() ? grads[0].contiguous() : Tensor();
        c10::cuda::CUDAGuard guard(sum.device());
        Tensor dx = at::empty_like(sum), dw = at::empty_like(w);
        const int64_t n = sum.size(-1), rows = sum.numel() / n;
        const size_t nbytes = api.rmsnorm_backward_ws(rows, (int32_t)n);
        Tensor ws = at::empty({(int64_t)nbytes}, sum.options().dtype(at::kByte));
        check(api.add_rmsnorm_backward(sum.data_ptr(), w.data_ptr(), dtype_code(w), g.data_ptr(), gh.defined() ? gh.data_ptr() : nullptr,
                                       dx.data_ptr(), dw.data_ptr(), ws.data_ptr(), nbytes, rows, (int32_t)n,
                                       (float)ctx->saved_data["eps"].toDouble(), current_stream(sum)));
        return {dx, dx, dw.to((at::ScalarType)ctx->saved_data["dtype"].toInt()), Tensor()};
    }
};
std::pair<Tensor, Tensor> add_rmsnorm(const Tensor &h, const Tensor &d, const Tensor &weight, double eps) {
    variable_list o = AddRMSNormFunction::apply(h, d, weight, eps);
    return {o[0], o[1]};
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("op_forward", torch::wrap_pybind_function(op_forward));
    m.def("op_backward", torch::wrap_pybind_function(op_backward));
    m.def("flash_mhf", torch::wrap_pybind_function(flash_mhf));
    m.def("fused_prologue", torch::wrap_pybind_function(fused_prologue));
    m.def("mhffn_layer", torch::wrap_pybind_function(mhffn_layer));
    m.def("rotary", torch::wrap_pybind_function(rotary));
    m.def("lm_attention", torch::wrap_pybind_function(lm_attention));
    m.def("rotary_pair", torch::wrap_pybind_function(rotary_pair));
    m.def("add_rmsnorm", torch::wrap_pybind_function(add_rmsnorm));
    m.def("rmsnorm", torch::wrap_pybind_function(rmsnorm));
}

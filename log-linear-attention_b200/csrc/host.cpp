// Native host side of the Python package: one call into this module does what a public call needs between its argument checks and its
// kernels - output and scratch allocation, the C-ABI calls, the autograd nodes.
//
// It exists because small calls are bound by the host.  The same work in Python (an autograd.Function, ctypes calls of 20 arguments,
// context managers) took 100 us for a forward, 250 us for a backward and 15 us for a decode step on the box the kernels are timed on,
// several times the kernels of a short sequence.
//
// Every entry returns None when the operands are not the ones it takes (dtypes, devices, shapes); the Python caller then goes its
// general way, which also raises the errors.  The kernels are reached through the C ABI of libllattn.so (include/llattn.h), which is
// loaded from the path that the Python binding uses.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <ATen/cuda/EmptyTensor.h>
#include "../../include/llattn.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

#define LLATTN_FUNCS(F)                                                                                                             \
    F(llattn_mamba2_fwd_workspace_bytes) F(llattn_mamba2_fwd) F(llattn_mamba2_fwd_residual) F(llattn_mamba2_fwd_prompt) F(llattn_mamba2_bwd_workspace_bytes) F(llattn_mamba2_bwd_layer_workspace_bytes) F(llattn_mamba2_bwd_saved) F(llattn_mamba2_bwd_layer)        \
    F(llattn_mamba2_layer_prep_fwd) F(llattn_mamba2_layer_prep_bwd) F(llattn_mamba2_layer_step) F(llattn_gdn_layer_step)            \
    F(llattn_mamba2_prompt_prep) F(llattn_mamba2_prompt_residual) F(llattn_mamba2_prompt_states) F(llattn_mamba2_prompt_tail) F(llattn_mamba2_residual) F(llattn_mixer_prep_fwd)            \
    F(llattn_mixer_prep_bwd) F(llattn_mixer_norm_fwd) F(llattn_mixer_norm_bwd) F(llattn_gdn_prompt_prep)                             \
    F(llattn_gdn_fwd_workspace_bytes) F(llattn_gdn_fwd_keep_workspace_bytes) F(llattn_gdn_fwd) F(llattn_gdn_fwd_keep)                \
    F(llattn_gdn_prompt) F(llattn_gdn_prompt_scratch_bytes) F(llattn_gdn_bwd_workspace_bytes) F(llattn_gdn_bwd)                      \
    F(llattn_gdn_bwd_kept_workspace_bytes) F(llattn_gdn_bwd_kept_bf16dv) F(llattn_gdn_bwd_kept_normed) F(llattn_gdn_grad_out) F(llattn_workspace_status) F(llattn_clear)

struct Library {
#define LLATTN_MEMBER(name) decltype(&::name) name = nullptr;
    LLATTN_FUNCS(LLATTN_MEMBER)
#undef LLATTN_MEMBER
} lib;

void bind(const std::string& path) {
    void* so = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(so, "cannot load ", path, ": ", dlerror());
#define LLATTN_BIND(name)                                                   \
    lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(so, #name));      \
    TORCH_CHECK(lib.name, path, " has no " #name);
    LLATTN_FUNCS(LLATTN_BIND)
#undef LLATTN_BIND
}

void check(int rc, const char* what) {
    if (rc == 0) return;
    TORCH_CHECK_VALUE(rc > 0, what, ": unsupported arguments (code ", rc, ")");
    TORCH_CHECK(false, what, ": CUDA error ", rc);
}

// ------------------------------------------------------------------------------------------ small helpers
inline bool is(const Tensor& t, at::ScalarType s) { return t.defined() && t.is_cuda() && t.scalar_type() == s; }
inline bool bf16(const Tensor& t) { return is(t, at::kBFloat16); }
inline bool f32(const Tensor& t) { return t.defined() && t.scalar_type() == at::kFloat; }
// a parameter: fp32 or bf16 on the device, or absent
inline bool param(const Tensor& t) { return !t.defined() || (t.is_cuda() && (t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16)); }
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
// contiguous, and where the kernels' 16-byte accesses can start: a contiguous view into a larger tensor may start anywhere
inline bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
inline Tensor contiguous(const Tensor& t) {
    if (!t.defined()) return t;
    const Tensor c = t.contiguous();
    return aligned(c) ? c : c.clone();
}
// what a node saved; hooks may hand back any tensor of the same values
inline variable_list saved(AutogradContext* ctx) {
    variable_list s = ctx->get_saved_variables();
    for (Tensor& t : s)
        if (t.defined() && !(t.is_contiguous() && aligned(t))) t = contiguous(t);
    return s;
}
using Maybe = std::optional<Tensor>;     // a tensor that may be absent: autograd functions take no undefined tensors
inline Tensor of(const Maybe& t) { return t.has_value() ? *t : Tensor(); }
inline Tensor empty(at::IntArrayRef size, at::ScalarType dt, const Tensor& like) {
    return at::detail::empty_cuda(size, dt, like.device(), std::nullopt);        // behind the dispatcher: 1 us less a tensor
}
inline Tensor contiguous_like(const Tensor& t) { return empty(t.sizes(), t.scalar_type(), t); }
inline Tensor zeros(int64_t n, const Tensor& like, void* stream) {
    const Tensor t = empty({n}, at::kFloat, like);
    check(lib.llattn_clear(t.data_ptr(), n * sizeof(float), stream), "llattn_clear");
    return t;
}
inline bool wants_grad(std::initializer_list<Tensor> ts) {
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor& t : ts)
        if (t.defined() && t.requires_grad()) return true;
    return false;
}
// A forward-mode derivative on an operand: the nodes have none to hand on, so such calls go the general way, whose autograd function says so.
inline bool has_tangent(std::initializer_list<Tensor> ts) {
    for (const Tensor& t : ts)
        if (t.defined() && t._fw_grad(0).defined()) return true;
    return false;
}
inline bool same_device(std::initializer_list<Tensor> ts) {
    const Tensor* first = nullptr;
    for (const Tensor& t : ts) {
        if (!t.defined()) continue;
        if (first && t.device() != first->device()) return false;
        first = &t;
    }
    return true;
}
inline bool native_set(std::initializer_list<Tensor> ts) { return same_device(ts) && !has_tangent(ts); }
inline int ceil_log2(int64_t x) {
    int l = 0;
    while ((int64_t(1) << l) < x) ++l;
    return l;
}
inline int bit_length(int64_t x) {
    int l = 0;
    while (x) {
        ++l;
        x >>= 1;
    }
    return l;
}
void check_status(const Tensor& ws, void* stream, const char* what) {
    int status = -1;
    check(lib.llattn_workspace_status(ws.data_ptr(), &status, stream), "llattn_workspace_status");
    TORCH_CHECK(status == 0, what, ": a kernel gave up on a bounded wait (status word set); the outputs are not valid");
}
// the current stream of t's device, which the guard makes the current one
struct On {
    c10::cuda::CUDAGuard guard;
    void* stream;
    explicit On(const Tensor& t) : guard(t.device()), stream(at::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

// ------------------------------------------------------------------------------------------ Mamba-2 chunkwise kernels
bool mamba2_shape(int64_t T, int64_t H, int64_t G, int64_t N, int64_t P, int64_t L) {
    return T > 0 && T % 64 == 0 && T <= 524288 && G > 0 && H % G == 0 && (N == 64 || N == 128) && P == 64 && L <= 32 && L >= 7 + ceil_log2(T / 64);
}
struct Scan {
    Tensor o, g_cum, ws;
};
// contiguous operands of the checked shape
Scan mamba2_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& l, void* stream, bool status) {
    const int B = k.size(0), T = k.size(1), G = k.size(2), K = k.size(3), H = v.size(2), V = v.size(3), L = l.size(3);
    Scan s;
    s.o = contiguous_like(v);
    s.g_cum = contiguous_like(g);
    const size_t n = lib.llattn_mamba2_fwd_workspace_bytes(B, T, H, G, K, V, L);
    s.ws = empty({(int64_t)std::max<size_t>(n, 256)}, at::kByte, q);
    check(lib.llattn_mamba2_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), l.data_ptr(), s.o.data_ptr(), fptr(s.g_cum), s.ws.data_ptr(),
                                s.ws.numel(), B, T, H, G, K, V, L, stream),
          "llattn_mamba2_fwd");
    if (status) check_status(s.ws, stream, "llattn_mamba2_fwd");
    return s;
}
// the same with y = o + D x in the place of o
Scan mamba2_fwd_residual(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& l, const Tensor& x, const Tensor& D,
                         void* stream, bool status) {
    const int B = k.size(0), T = k.size(1), G = k.size(2), K = k.size(3), H = v.size(2), V = v.size(3), L = l.size(3);
    Scan s;
    s.o = empty(x.sizes(), f32(D) ? at::kFloat : at::kBFloat16, x);
    s.g_cum = contiguous_like(g);
    const size_t n = lib.llattn_mamba2_fwd_workspace_bytes(B, T, H, G, K, V, L);
    s.ws = empty({(int64_t)std::max<size_t>(n, 256)}, at::kByte, q);
    const int rc = lib.llattn_mamba2_fwd_residual(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), l.data_ptr(), x.data_ptr(), D.data_ptr(),
                                                  s.o.data_ptr(), f32(D), T, fptr(s.g_cum), s.ws.data_ptr(), s.ws.numel(), B, T, H, G, K, V, L, stream);
    if (rc == LLATTN_ERR_UNSUPPORTED_SHAPE) {
        const Tensor y = s.o, D32 = D.to(at::kFloat);
        s = mamba2_fwd(q, k, v, g, l, stream, status);
        check(lib.llattn_mamba2_residual(s.o.data_ptr(), x.data_ptr(), fptr(D32), y.data_ptr(), f32(D), (long)B * T * H, H, V, stream),
              "llattn_mamba2_residual");
        s.o = y;
        return s;
    }
    check(rc, "llattn_mamba2_fwd_residual");
    if (status) check_status(s.ws, stream, "llattn_mamba2_fwd_residual");
    return s;
}
struct ScanGrads {
    Tensor dq, dk, dv, dg, dl;       // dl fp32
};
ScanGrads mamba2_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_cum, const Tensor& l, const Tensor& d_o, const Tensor& fws,
                     void* stream, bool status, bool layer) {
    const int B = k.size(0), T = k.size(1), G = k.size(2), K = k.size(3), H = v.size(2), V = v.size(3), L = l.size(3);
    ScanGrads r;
    const Tensor qk = empty({2, B, T, G, K}, at::kBFloat16, q);      // side by side: one conversion pass writes both
    r.dq = qk.select(0, 0);
    r.dk = qk.select(0, 1);
    r.dv = contiguous_like(v);
    r.dg = contiguous_like(g_cum);
    r.dl = empty(l.sizes(), at::kFloat, l);
    const size_t n = (layer ? lib.llattn_mamba2_bwd_layer_workspace_bytes : lib.llattn_mamba2_bwd_workspace_bytes)(B, T, H, G, K, V, L);
    const Tensor ws = empty({(int64_t)std::max<size_t>(n, 256)}, at::kByte, q);
    const auto bwd = layer ? lib.llattn_mamba2_bwd_layer : lib.llattn_mamba2_bwd_saved;
    check(bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g_cum), l.data_ptr(), d_o.data_ptr(), r.dq.data_ptr(), r.dk.data_ptr(), r.dv.data_ptr(),
              fptr(r.dg), fptr(r.dl), ws.data_ptr(), ws.numel(), ptr(fws), fws.defined() ? fws.numel() : 0, B, T, H, G, K, V, L, stream),
          "llattn_mamba2_bwd_saved");
    if (status) check_status(ws, stream, "llattn_mamba2_bwd_saved");
    return r;
}

// ---- hattention_kernel, Mamba-2 structure
struct Mamba2Kernel : torch::autograd::Function<Mamba2Kernel> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& l, bool keep,
                          bool status, bool layer) {
        On on(q);
        const Tensor q_ = contiguous(q), k_ = contiguous(k), v_ = contiguous(v), g_ = contiguous(g), l_ = contiguous(l);
        Scan s = mamba2_fwd(q_, k_, v_, g_, l_, on.stream, status);
        if (ctx) {
            ctx->save_for_backward({q_, k_, v_, s.g_cum, l_, keep ? s.ws : Tensor()});
            ctx->saved_data["status"] = status;
            ctx->saved_data["layer"] = layer;
        }
        return s.o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list d) {
        const auto s = saved(ctx);
        On on(s[0]);
        ScanGrads r = mamba2_bwd(s[0], s[1], s[2], s[3], s[4], contiguous(d[0].to(at::kBFloat16)), s[5], on.stream,
                                 ctx->saved_data["status"].toBool(), ctx->saved_data["layer"].toBool());
        return {r.dq, r.dk, r.dv, r.dg, r.dl.to(at::kBFloat16), Tensor(), Tensor(), Tensor()};
    }
};

py::object hattention_mamba2(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& l, bool keep, bool status, bool layer) {
    if (!bf16(q) || !bf16(k) || !bf16(v) || !is(g, at::kFloat) || !bf16(l) || k.dim() != 4 || v.dim() != 4 || l.dim() != 4 || q.sizes() != k.sizes() ||
        !native_set({q, k, v, g, l}))
        return py::none();
    const int64_t B = k.size(0), T = k.size(1), H = v.size(2), L = l.size(3);
    if (v.size(0) != B || v.size(1) != T || g.sizes() != at::IntArrayRef({B, T, H}) || l.sizes() != at::IntArrayRef({B, T, H, L}) ||
        !mamba2_shape(T, H, k.size(2), k.size(3), v.size(3), L))
        return py::none();
    py::gil_scoped_release nogil;
    Tensor o = wants_grad({q, k, v, g, l}) ? Mamba2Kernel::apply(q, k, v, g, l, keep, status, layer)
                                             : Mamba2Kernel::forward(nullptr, q, k, v, g, l, false, status, layer);
    py::gil_scoped_acquire gil;
    return py::cast(o);
}

// ---- the layer call: preparation, chunkwise kernels, D residual
struct Mamba2Layer : torch::autograd::Function<Mamba2Layer> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm, const Tensor& dl,
                          const Tensor& Lp, const Maybe& D, const Maybe& bias, int64_t mode, bool keep, bool status) {
        On on(x);
        const int B = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), L = dl.size(3);
        const Tensor x_ = contiguous(x), dt_ = contiguous(dt), dl_ = contiguous(dl), A_ = contiguous(A.to(at::kFloat)), Lp_ = contiguous(Lp),
                     D_ = contiguous(of(D)), b_ = contiguous(of(bias)), q = contiguous(Cm), k = contiguous(Bm);
        const Tensor v = contiguous_like(x_), g = empty({B, T, H}, at::kFloat, x), lam = contiguous_like(dl_);
        check(lib.llattn_mamba2_layer_prep_fwd(x_.data_ptr(), dt_.data_ptr(), ptr(b_), f32(b_), fptr(A_), dl_.data_ptr(), Lp_.data_ptr(), f32(Lp_),
                                               v.data_ptr(), fptr(g), lam.data_ptr(), (long)B * T * H, H, P, L, (int)mode, on.stream),
              "llattn_mamba2_layer_prep_fwd");
        const Scan s = D_.defined() ? mamba2_fwd_residual(q, k, v, g, lam, x_, D_, on.stream, status) : mamba2_fwd(q, k, v, g, lam, on.stream, status);
        const Tensor& y = s.o;
        if (ctx) {
            ctx->save_for_backward({x_, dt_, A_, k, q, dl_, Lp_, D_, b_, v, s.g_cum, lam, keep ? s.ws : Tensor()});
            ctx->saved_data["mode"] = mode;
            ctx->saved_data["status"] = status;
            ctx->saved_data["A"] = (int64_t)A.scalar_type();
        }
        return y;
    }
    static variable_list backward(AutogradContext* ctx, variable_list d) {
        const auto s = saved(ctx);
        const Tensor &x = s[0], &dt = s[1], &A = s[2], &k = s[3], &q = s[4], &dl = s[5], &Lp = s[6], &D = s[7], &bias = s[8], &v = s[9], &g_cum = s[10],
                     &lam = s[11], &ws = s[12];
        On on(x);
        const int B = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), L = dl.size(3);
        const Tensor dy = contiguous(d[0].to(at::kBFloat16));
        ScanGrads r = mamba2_bwd(q, k, v, g_cum, lam, dy, ws, on.stream, ctx->saved_data["status"].toBool(), true);
        const Tensor dx = contiguous_like(x), ddt = contiguous_like(dt), ddl = contiguous_like(dl);
        const Tensor acc = zeros(3 * H + (int64_t)H * L, x, on.stream);
        float* a = fptr(acc);
        check(lib.llattn_mamba2_layer_prep_bwd(x.data_ptr(), dt.data_ptr(), ptr(bias), f32(bias), fptr(A), dl.data_ptr(), Lp.data_ptr(), f32(Lp), ptr(D),
                                               f32(D), r.dv.data_ptr(), fptr(r.dg), fptr(r.dl), dy.data_ptr(), dx.data_ptr(), ddt.data_ptr(), ddl.data_ptr(),
                                               a, a + H, a + 3 * H, a + 2 * H, (long)B * T * H, H, P, L, (int)ctx->saved_data["mode"].toInt(), on.stream),
              "llattn_mamba2_layer_prep_bwd");
        // one conversion for all parameters that are kept in bf16
        const at::ScalarType A_dt = (at::ScalarType)ctx->saved_data["A"].toInt();
        Tensor half;
        auto part = [&](int64_t at0, int64_t n, at::ScalarType t) {
            if (t == at::kFloat) return acc.narrow(0, at0, n);
            if (!half.defined()) half = acc.to(at::kBFloat16);
            return t == at::kBFloat16 ? half.narrow(0, at0, n) : acc.narrow(0, at0, n).to(t);
        };
        return {dx, ddt, part(0, H, A_dt), r.dk, r.dq, ddl, part(3 * H, (int64_t)H * L, Lp.scalar_type()).view({H, L}),
                D.defined() ? part(2 * H, H, D.scalar_type()) : Tensor(), bias.defined() ? part(H, H, bias.scalar_type()) : Tensor(), Tensor(), Tensor(),
                Tensor()};
    }
};

bool layer_operands(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm, const Tensor& dl, const Tensor& Lp,
                    const Tensor& D, const Tensor& bias) {
    if (!bf16(x) || !bf16(dt) || !bf16(Bm) || !bf16(Cm) || !bf16(dl) || !A.is_cuda() || !A.is_floating_point() || !param(Lp) || !param(D) || !param(bias) ||
        x.dim() != 4 || Bm.dim() != 4 || dl.dim() != 4 || Lp.dim() != 2 || Cm.sizes() != Bm.sizes() || !native_set({x, dt, A, Bm, Cm, dl, Lp, D, bias}))
        return false;
    const int64_t B = x.size(0), T = x.size(1), H = x.size(2), L = dl.size(3);
    return dt.sizes() == at::IntArrayRef({B, T, H}) && A.sizes() == at::IntArrayRef({H}) && Bm.size(0) == B && Bm.size(1) == T &&
           dl.sizes() == at::IntArrayRef({B, T, H, L}) && Lp.sizes() == at::IntArrayRef({H, L}) && (!D.defined() || D.sizes() == at::IntArrayRef({H})) &&
           (!bias.defined() || bias.sizes() == at::IntArrayRef({H})) && x.size(3) == 64 && Bm.size(2) > 0 && H % Bm.size(2) == 0 &&
           (Bm.size(3) == 64 || Bm.size(3) == 128) && L <= 32 && B * T * H < (int64_t(1) << 28);
}

py::object mamba2_layer(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm, const Tensor& dl, const Tensor& Lp,
                        const Maybe& D_, const Maybe& bias_, int64_t mode, bool keep, bool status) {
    const Tensor D = of(D_), bias = of(bias_);
    if (!layer_operands(x, dt, A, Bm, Cm, dl, Lp, D, bias) || !mamba2_shape(x.size(1), x.size(2), Bm.size(2), Bm.size(3), x.size(3), dl.size(3)))
        return py::none();
    py::gil_scoped_release nogil;
    Tensor y = wants_grad({x, dt, A, Bm, Cm, dl, Lp, D, bias}) ? Mamba2Layer::apply(x, dt, A, Bm, Cm, dl, Lp, D_, bias_, mode, keep, status)
                                                              : Mamba2Layer::forward(nullptr, x, dt, A, Bm, Cm, dl, Lp, D_, bias_, mode, false, status);
    py::gil_scoped_acquire gil;
    return py::cast(y);
}

// ---- a prompt of any length: outputs and level states (level-major), after its T0 whole-chunk tokens and the n < 64 behind them
struct Prompt {
    int B, T0, n, H, G, N, P, L;
    Prompt(int B, int T, int H, int G, int N, int P, int L) : B(B), T0(T / 64 * 64), n(T % 64), H(H), G(G), N(N), P(P), L(L) {}
    int T() const { return T0 + n; }
    bool takes() const { return T() > 0 && L >= 1 + bit_length(T() - 1) && (T0 == 0 || mamba2_shape(T0, H, G, N, P, L)); }
    // several sequences with tails: the tensors hold the whole chunks of all of them first, then the tails
    bool split() const { return B > 1 && n > 0 && T0 > 0; }
    Tensor parts(const Tensor& t) const {
        if (!split()) return t;
        return at::cat({t.narrow(1, 0, T0).reshape({-1}), t.narrow(1, T0, n).reshape({-1})});
    }
    // tensors of B T() tokens, split; x as it is and D, or neither.  (y, states (B,H,L,N,P))
    std::pair<Tensor, Tensor> run(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& lam, const Tensor& x, const Tensor& D,
                                  void* stream, bool status) const {
        const bool y32 = f32(D);
        const Tensor y = empty({B, T(), H, P}, y32 ? at::kFloat : at::kBFloat16, v), states = empty({B, H, L, N, P}, at::kFloat, v);
        const Tensor part = n > 0 && T0 > 0 ? empty({B, n, H, P}, at::kFloat, v) : Tensor();
        int rc = 0;
        if (T0 > 0) {
            const Tensor g_cum = empty({B, T0, H}, at::kFloat, v);
            const size_t bytes = std::max<size_t>(lib.llattn_mamba2_fwd_workspace_bytes(B, T0, H, G, N, P, L), 256);
            const Tensor ws = empty({(int64_t)bytes}, at::kByte, v);
            rc = lib.llattn_mamba2_fwd_prompt(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), lam.data_ptr(), ptr(x), ptr(D), y.data_ptr(), y32, n,
                                              fptr(part), fptr(states), L, fptr(g_cum), ws.data_ptr(), bytes, B, T0, H, G, N, P, L, stream);
            if (rc == 0 && status) check_status(ws, stream, "llattn_mamba2_fwd_prompt");
            if (rc != LLATTN_ERR_UNSUPPORTED_SHAPE || !D.defined()) {
                check(rc, "llattn_mamba2_fwd_prompt");
                return {y, states};
            }
            const Tensor o = empty({B, T0, H, P}, at::kBFloat16, v);
            check(lib.llattn_mamba2_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), lam.data_ptr(), o.data_ptr(), fptr(g_cum), ws.data_ptr(), bytes, B,
                                        T0, H, G, N, P, L, stream),
                  "llattn_mamba2_fwd");
            if (status) check_status(ws, stream, "llattn_mamba2_fwd");
            check(lib.llattn_mamba2_prompt_residual(o.data_ptr(), x.data_ptr(), ptr(D), y.data_ptr(), y32, B, T0, n, H, P, stream),
                  "llattn_mamba2_prompt_residual");
            check(lib.llattn_mamba2_prompt_states(k.data_ptr(), v.data_ptr(), fptr(g), fptr(states), ws.data_ptr(), bytes, B, T0, n, H, G, N, P, L, stream),
                  "llattn_mamba2_prompt_states");
        }
        if (n > 0)
            check(lib.llattn_mamba2_prompt_tail(q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), lam.data_ptr(), ptr(x), ptr(D), y32, y.data_ptr(),
                                                fptr(states), L, fptr(part), B, T0, n, H, G, N, P, L, stream),
                  "llattn_mamba2_prompt_tail");
        return {y, states};
    }
};

py::object mamba2_prompt(const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm, const Tensor& dl, const Tensor& Lp,
                         const Maybe& D_, const Maybe& bias_, int64_t mode, bool status) {
    const Tensor D = of(D_), bias = of(bias_);
    if (!layer_operands(x, dt, A, Bm, Cm, dl, Lp, D, bias) || wants_grad({x, dt, A, Bm, Cm, dl, Lp, D, bias})) return py::none();
    const Prompt p(x.size(0), x.size(1), x.size(2), Bm.size(2), Bm.size(3), x.size(3), dl.size(3));
    if (!p.takes()) return py::none();
    std::pair<Tensor, Tensor> r;
    {
        py::gil_scoped_release nogil;
        at::NoGradGuard no_grad;
        On on(x);
        const Tensor x_ = contiguous(x), dt_ = contiguous(dt), dl_ = contiguous(dl), A_ = contiguous(A.to(at::kFloat)), Lp_ = contiguous(Lp),
                     D_c = contiguous(D), b_ = contiguous(bias);
        Tensor q = contiguous(Cm), k = contiguous(Bm), qs, ks;
        const Tensor v = contiguous_like(x_), g = empty(dt_.sizes(), at::kFloat, x), lam = contiguous_like(dl_);
        if (p.split()) {
            qs = contiguous_like(q);
            ks = contiguous_like(q);
        }
        check(lib.llattn_mamba2_prompt_prep(x_.data_ptr(), dt_.data_ptr(), ptr(b_), f32(b_), fptr(A_), dl_.data_ptr(), Lp_.data_ptr(), f32(Lp_),
                                            q.data_ptr(), k.data_ptr(), v.data_ptr(), fptr(g), lam.data_ptr(), ptr(qs), ptr(ks), p.B, p.T0, p.n, p.H, p.G,
                                            p.N, p.P, p.L, (int)mode, on.stream),
              "llattn_mamba2_prompt_prep");
        if (p.split()) {
            q = qs;
            k = ks;
        }
        r = p.run(q, k, v, g, lam, D_c.defined() ? x_ : Tensor(), D_c, on.stream, status);
        r.second = r.second.permute({0, 1, 3, 4, 2});
    }
    return py::make_tuple(r.first, r.second);
}

// hattention_prefill, Mamba-2 structure, on the scan's own operands: (o, level-major states) or None
py::object mamba2_prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& l, bool status) {
    if (!bf16(q) || !bf16(k) || !bf16(v) || !is(g, at::kFloat) || !bf16(l) || k.dim() != 4 || v.dim() != 4 || l.dim() != 4 || q.sizes() != k.sizes() ||
        !same_device({q, k, v, g, l}))
        return py::none();
    const int64_t B = k.size(0), T = k.size(1), G = k.size(2), N = k.size(3), H = v.size(2), P = v.size(3), L = l.size(3);
    if (B < 1 || v.size(0) != B || v.size(1) != T || g.sizes() != at::IntArrayRef({B, T, H}) || l.sizes() != at::IntArrayRef({B, T, H, L}) || G < 1 ||
        H % G != 0 || (N != 64 && N != 128) || P != 64 || L > 32 || T > 600000 || B * T * H >= (int64_t(1) << 28))
        return py::none();
    const Prompt p(B, T, H, G, N, P, L);
    if (!p.takes()) return py::none();
    std::pair<Tensor, Tensor> r;
    {
        py::gil_scoped_release nogil;
        at::NoGradGuard no_grad;
        On on(q);
        r = p.run(p.parts(contiguous(q)), p.parts(contiguous(k)), p.parts(contiguous(v)), p.parts(contiguous(g)), p.parts(contiguous(l)), Tensor(), Tensor(),
                  on.stream, status);
        r.second = r.second.permute({0, 1, 3, 4, 2});
    }
    return py::make_tuple(r.first, r.second);
}

// ---- the mixer between its projections
struct Mixer : torch::autograd::Function<Mixer> {
    static Tensor forward(AutogradContext* ctx, const Tensor& zx, const Tensor& cw, const Maybe& cb, const Tensor& bias, const Tensor& A, const Tensor& Lp,
                          const Tensor& D, const Tensor& nw, double eps, int64_t G, int64_t mode, bool keep, bool status) {
        On on(zx);
        const int B = zx.size(0), T = zx.size(1), W = zx.size(2), H = Lp.size(0), L = Lp.size(1), dim = H * 64, N = (W - 2 * dim - H - H * L) / (2 * G);
        const Tensor z = contiguous(zx), cw_ = contiguous(cw), cb_ = contiguous(of(cb)), b_ = contiguous(bias), A_ = contiguous(A.to(at::kFloat)),
                     Lp_ = contiguous(Lp), D_ = contiguous(D), nw_ = contiguous(nw);
        const Tensor x = empty({B, T, H, 64}, at::kBFloat16, zx), v = contiguous_like(x), k = empty({B, T, G, N}, at::kBFloat16, zx), q = contiguous_like(k);
        const Tensor g = empty({B, T, H}, at::kFloat, zx), lam = empty({B, T, H, L}, at::kBFloat16, zx);
        check(lib.llattn_mixer_prep_fwd(z.data_ptr(), cw_.data_ptr(), f32(cw_), ptr(cb_), f32(cb_), ptr(b_), f32(b_), fptr(A_), Lp_.data_ptr(), f32(Lp_),
                                        x.data_ptr(), v.data_ptr(), k.data_ptr(), q.data_ptr(), fptr(g), lam.data_ptr(), B, T, H, (int)G, N, L, (int)mode,
                                        on.stream),
              "llattn_mixer_prep_fwd");
        Scan s = mamba2_fwd(q, k, v, g, lam, on.stream, status);
        const Tensor out = empty({B, T, dim}, at::kBFloat16, zx), rstd = empty({B, T}, at::kFloat, zx);
        check(lib.llattn_mixer_norm_fwd(s.o.data_ptr(), x.data_ptr(), ptr(D_), f32(D_), z.data_ptr(), W, nw_.data_ptr(), f32(nw_), out.data_ptr(),
                                        fptr(rstd), (long)B * T, H, (float)eps, on.stream),
              "llattn_mixer_norm_fwd");
        if (ctx) {
            ctx->save_for_backward({z, cw_, cb_, b_, A_, Lp_, D_, nw_, x, v, k, q, s.g_cum, lam, s.o, rstd, keep ? s.ws : Tensor()});
            ctx->saved_data["mode"] = mode;
            ctx->saved_data["status"] = status;
            ctx->saved_data["A"] = (int64_t)A.scalar_type();
        }
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list d) {
        const auto s = saved(ctx);
        const Tensor &z = s[0], &cw = s[1], &cb = s[2], &bias = s[3], &A = s[4], &Lp = s[5], &D = s[6], &nw = s[7], &x = s[8], &v = s[9], &k = s[10],
                     &q = s[11], &g_cum = s[12], &lam = s[13], &o = s[14], &rstd = s[15], &ws = s[16];
        On on(z);
        const int B = z.size(0), T = z.size(1), W = z.size(2), H = Lp.size(0), L = Lp.size(1), dim = H * 64, G = k.size(2), N = k.size(3);
        const Tensor dn = contiguous(d[0].to(at::kBFloat16));
        const Tensor dzx = contiguous_like(z), dy = empty(x.sizes(), at::kBFloat16, x);
        // sums over tokens: conv taps and bias, norm weight, A, dt_bias, D, L
        const int64_t ch = dim + 2 * G * N, at_b = ch * 4, at_n = ch * 5, at_A = at_n + dim, at_dt = at_A + H, at_D = at_dt + H, at_L = at_D + H;
        const Tensor acc = zeros(at_L + (int64_t)H * L, z, on.stream);
        float* a = fptr(acc);
        check(lib.llattn_mixer_norm_bwd(o.data_ptr(), x.data_ptr(), ptr(D), f32(D), z.data_ptr(), W, nw.data_ptr(), f32(nw), dn.data_ptr(), fptr(rstd),
                                        dy.data_ptr(), dzx.data_ptr(), a + at_n, a + at_D, (long)B * T, H, on.stream),
              "llattn_mixer_norm_bwd");
        ScanGrads r = mamba2_bwd(q, k, v, g_cum, lam, dy, ws, on.stream, ctx->saved_data["status"].toBool(), true);
        check(lib.llattn_mixer_prep_bwd(z.data_ptr(), cw.data_ptr(), f32(cw), ptr(cb), f32(cb), ptr(bias), f32(bias), fptr(A), Lp.data_ptr(), f32(Lp), ptr(D),
                                        f32(D), r.dv.data_ptr(), dy.data_ptr(), r.dq.data_ptr(), r.dk.data_ptr(), fptr(r.dg), fptr(r.dl), dzx.data_ptr(), a,
                                        a + at_b, a + at_A, a + at_dt, a + at_L, B, T, H, G, N, L, (int)ctx->saved_data["mode"].toInt(), on.stream),
              "llattn_mixer_prep_bwd");
        const at::ScalarType A_dt = (at::ScalarType)ctx->saved_data["A"].toInt();
        Tensor half;
        auto part = [&](int64_t at0, at::IntArrayRef size, at::ScalarType t) {
            int64_t n = 1;
            for (int64_t e : size) n *= e;
            if (t == at::kFloat) return acc.narrow(0, at0, n).view(size);
            if (!half.defined()) half = acc.to(at::kBFloat16);
            return t == at::kBFloat16 ? half.narrow(0, at0, n).view(size) : acc.narrow(0, at0, n).view(size).to(t);
        };
        auto grad = [&](const Tensor& p, int64_t at0) { return p.defined() ? part(at0, p.sizes(), p.scalar_type()) : Tensor(); };
        return {dzx, grad(cw, 0), grad(cb, at_b), grad(bias, at_dt), part(at_A, {H}, A_dt), grad(Lp, at_L), grad(D, at_D), grad(nw, at_n), Tensor(), Tensor(),
                Tensor(), Tensor(), Tensor()};
    }
};

// zxbcdtdl (B,T,W) with the widths already checked -> the normed output (B,T,H 64), or None
py::object mamba2_mixer(const Tensor& zx, const Tensor& cw, const Maybe& cb_, const Tensor& bias, const Tensor& A, const Tensor& Lp,
                        const Tensor& D, const Tensor& nw, double eps, int64_t G, int64_t mode, bool keep, bool status) {
    const Tensor cb = of(cb_);
    if (!bf16(zx) || !param(cw) || !param(cb) || !param(bias) || !param(Lp) || !param(D) || !param(nw) || !A.is_cuda() || !A.is_floating_point() ||
        zx.dim() != 3 || Lp.dim() != 2 || !native_set({zx, cw, cb, bias, A, Lp, D, nw}))
        return py::none();
    const int64_t T = zx.size(1), H = Lp.size(0), L = Lp.size(1), dim = H * 64, rest = zx.size(2) - 2 * dim - H - H * L;
    if (G <= 0 || rest <= 0 || rest % (2 * G) != 0) return py::none();
    const int64_t N = rest / (2 * G), ch = dim + 2 * G * N;
    if (!mamba2_shape(T, H, G, N, 64, L) || H > 128 || cw.sizes() != at::IntArrayRef({ch, 4}) || (cb.defined() && cb.sizes() != at::IntArrayRef({ch})) ||
        nw.sizes() != at::IntArrayRef({dim}) || zx.size(0) * T * H >= (int64_t(1) << 28))
        return py::none();
    py::gil_scoped_release nogil;
    Tensor y = wants_grad({zx, cw, cb, bias, A, Lp, D, nw}) ? Mixer::apply(zx, cw, cb_, bias, A, Lp, D, nw, eps, G, mode, keep, status)
                                                           : Mixer::forward(nullptr, zx, cw, cb_, bias, A, Lp, D, nw, eps, G, mode, false, status);
    py::gil_scoped_acquire gil;
    return py::cast(y);
}

// ------------------------------------------------------------------------------------------ Gated DeltaNet
constexpr int GDN_K = 128, GDN_V_MAX = 384;      // key width of the kernels; widest value head

struct GdnInputs {
    Tensor qn, kn, v, b, g, l;       // one row per part of a value head
    int B, T, H, G, K, V, L;         // of the caller's tensors (T and L as padded)
    // A value head is `rep` heads of `width` columns that share q, k, beta, g and lambda: the delta rule acts on every value column
    // independently.  The kernels take 64 or 128 columns a head; all parts run in one launch.
    int rep, width;
    int heads() const { return H * rep; }
    void split() {
        width = V % 128 == 0 ? 128 : 64;
        rep = V / width;
    }
};

// l2norm of q and k, lambda times its factor, the parts of wide heads, split into T0 tokens of whole chunks and n others where several sequences
// have both; what none of these changes is used as it is
GdnInputs gdn_prepare(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g, const Tensor& l, int T0, int n, double scale,
                      double lam_mul, void* stream) {
    GdnInputs a;
    a.B = q.size(0);
    a.T = T0 + n;
    a.G = q.size(2);
    a.K = q.size(3);
    a.H = v.size(2);
    a.V = v.size(3);
    a.L = l.size(3);
    a.split();
    const int B = a.B, H = a.heads(), T = a.T, L = a.L;
    const bool split = B > 1 && T0 > 0 && n > 0, own = split || a.rep > 1, own_l = own || lam_mul != 0.0;
    a.qn = empty({B, T, H, GDN_K}, at::kBFloat16, q);
    a.kn = contiguous_like(a.qn);
    a.v = split ? empty({B, T, H, a.width}, at::kBFloat16, q) : v;
    a.b = own ? empty({B, T, H}, at::kBFloat16, q) : b;
    a.g = own ? empty({B, T, H}, at::kFloat, q) : g;
    a.l = own_l ? empty({B, T, H, L}, at::kBFloat16, q) : l;
    check(lib.llattn_gdn_prompt_prep(q.data_ptr(), k.data_ptr(), v.data_ptr(), b.data_ptr(), fptr(g), l.data_ptr(), a.qn.data_ptr(), a.kn.data_ptr(),
                                     split ? a.v.data_ptr() : nullptr, own ? a.b.data_ptr() : nullptr, own ? fptr(a.g) : nullptr,
                                     own_l ? a.l.data_ptr() : nullptr, B, T0, n, a.H, a.G, a.K, GDN_K, a.V, a.rep, L, (float)scale, (float)lam_mul, stream),
          "llattn_gdn_prompt_prep");
    return a;
}

bool gdn_operands(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g, const Tensor& l) {
    if (!bf16(q) || !bf16(k) || !bf16(v) || !bf16(b) || !is(g, at::kFloat) || !bf16(l) || q.dim() != 4 || v.dim() != 4 || l.dim() != 4 ||
        q.sizes() != k.sizes() || !same_device({q, k, v, b, g, l}))
        return false;
    const int64_t B = q.size(0), T = q.size(1), G = q.size(2), K = q.size(3), H = v.size(2), V = v.size(3), L = l.size(3);
    return v.size(0) == B && v.size(1) == T && b.sizes() == at::IntArrayRef({B, T, H}) && g.sizes() == at::IntArrayRef({B, T, H}) &&
           l.sizes() == at::IntArrayRef({B, T, H, L}) && T > 0 && G > 0 && H % G == 0 && K <= GDN_K && K % 8 == 0 && V > 0 && V % 64 == 0 && V <= GDN_V_MAX &&
           L <= 32 && B * T * H < (int64_t(1) << 28);
}

struct GdnKernel : torch::autograd::Function<GdnKernel> {
    static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g, const Tensor& l,
                          double scale, double lam_mul, int64_t keep_bytes, bool status) {
        On on(q);
        const Tensor q_ = contiguous(q), k_ = contiguous(k), v_ = contiguous(v), b_ = contiguous(b), g_ = contiguous(g), l_ = contiguous(l);
        const int T = q.size(1);
        GdnInputs a = gdn_prepare(q_, k_, v_, b_, g_, l_, T, 0, scale, lam_mul, on.stream);
        const int B = a.B, H = a.heads(), V = a.width;
        const size_t keep_need = lib.llattn_gdn_fwd_keep_workspace_bytes(B, T, H, GDN_K, V, a.L);
        const bool keep = ctx != nullptr && (int64_t)keep_need <= keep_bytes;
        const Tensor g_cum = contiguous_like(a.g), Aw = empty({B, T, H, 64}, at::kBFloat16, q), Au = contiguous_like(Aw);
        const size_t bytes = keep ? keep_need : lib.llattn_gdn_fwd_workspace_bytes(B, T, H, GDN_K, V, a.L);
        const Tensor ws = empty({(int64_t)bytes}, at::kByte, q), o = contiguous_like(v_);
        check((keep ? lib.llattn_gdn_fwd_keep : lib.llattn_gdn_fwd)(a.qn.data_ptr(), a.kn.data_ptr(), a.v.data_ptr(), a.b.data_ptr(), fptr(a.g), a.l.data_ptr(),
                                                                   o.data_ptr(), fptr(g_cum), Aw.data_ptr(), Au.data_ptr(), ws.data_ptr(), bytes, B, T, H,
                                                                   GDN_K, V, a.L, on.stream),
              "llattn_gdn_fwd");
        if (status) check_status(ws, on.stream, "llattn_gdn_fwd");
        if (ctx) {
            variable_list save = {q_, k_, v_, a.b, g_cum, a.l, Aw, Au};
            if (keep) save.insert(save.end(), {a.qn, a.kn, ws});
            ctx->save_for_backward(save);
            ctx->saved_data["scale"] = scale;
            ctx->saved_data["lam_mul"] = lam_mul;
            ctx->saved_data["status"] = status;
        }
        return o;
    }
    static variable_list backward(AutogradContext* ctx, variable_list d) {
        const auto s = saved(ctx);
        On on(s[0]);
        const Tensor &q = s[0], &k = s[1], &v = s[2], &b = s[3], &g_cum = s[4], &l = s[5], &Aw = s[6], &Au = s[7];
        const bool kept = s.size() > 8, status = ctx->saved_data["status"].toBool();
        const double scale = ctx->saved_data["scale"].toDouble(), lam_mul = ctx->saved_data["lam_mul"].toDouble();
        GdnInputs a;
        a.B = q.size(0);
        a.T = q.size(1);
        a.H = q.size(2);
        a.K = q.size(3);
        a.V = v.size(3);
        a.L = l.size(3);
        a.split();
        const int B = a.B, T = a.T, H = a.heads(), V = a.width;
        Tensor qn, kn;
        if (kept) {
            qn = s[8];
            kn = s[9];
        } else {
            qn = empty({B, T, H, GDN_K}, at::kBFloat16, q);
            kn = contiguous_like(qn);
            check(lib.llattn_gdn_prompt_prep(q.data_ptr(), k.data_ptr(), nullptr, nullptr, nullptr, nullptr, qn.data_ptr(), kn.data_ptr(), nullptr, nullptr,
                                             nullptr, nullptr, B, T, 0, a.H, a.H, a.K, GDN_K, a.V, a.rep, a.L, (float)scale, 0.f, on.stream),
                  "llattn_gdn_prompt_prep");
        }
        const Tensor d_o = contiguous(d[0].to(at::kBFloat16));
        // fp32 gradients of what the parts of a head share; dg is handed on as it is where a head has one part
        const int64_t rows = (int64_t)B * T * a.H, prows = rows * a.rep;
        const Tensor gq = empty({B, T, a.H, a.K}, at::kBFloat16, q), gk = contiguous_like(gq);
        const Tensor dgp = empty({B, T, H}, at::kFloat, q), dlb = empty({prows * (a.L + 1)}, at::kFloat, q);
        float *dl = fptr(dlb), *db = dl + prows * a.L;
        const size_t bytes = (kept ? lib.llattn_gdn_bwd_kept_workspace_bytes : lib.llattn_gdn_bwd_workspace_bytes)(B, T, H, GDN_K, V, a.L);
        const Tensor ws = empty({(int64_t)bytes}, at::kByte, q);
        Tensor dv = empty(v.sizes(), kept ? at::kBFloat16 : at::kFloat, q);
        // heads of one part and full width: the kernels take the backward of the normalisation along
        bool normed = kept && a.rep == 1 && a.K == GDN_K;
        if (normed) {
            const Tensor& fws = s[10];
            const int rc = lib.llattn_gdn_bwd_kept_normed(qn.data_ptr(), kn.data_ptr(), q.data_ptr(), k.data_ptr(), (float)scale, v.data_ptr(), b.data_ptr(),
                                                          fptr(g_cum), l.data_ptr(), Aw.data_ptr(), Au.data_ptr(), d_o.data_ptr(), gq.data_ptr(),
                                                          gk.data_ptr(), dv.data_ptr(), db, fptr(dgp), dl, fws.data_ptr(), fws.numel(), ws.data_ptr(),
                                                          bytes, B, T, H, GDN_K, V, a.L, on.stream);
            normed = rc != LLATTN_ERR_UNSUPPORTED_SHAPE;
            if (normed) check(rc, "llattn_gdn_bwd_kept_normed");
        }
        Tensor dqk;
        float *dq = nullptr, *dk = nullptr;
        if (!normed) {
            dqk = empty({2 * prows * GDN_K}, at::kFloat, q);
            dq = fptr(dqk);
            dk = dq + prows * GDN_K;
            if (kept) {
                const Tensor& fws = s[10];
                check(lib.llattn_gdn_bwd_kept_bf16dv(qn.data_ptr(), kn.data_ptr(), v.data_ptr(), b.data_ptr(), fptr(g_cum), l.data_ptr(), Aw.data_ptr(),
                                                     Au.data_ptr(), d_o.data_ptr(), dq, dk, dv.data_ptr(), db, fptr(dgp), dl, fws.data_ptr(), fws.numel(),
                                                     ws.data_ptr(), bytes, B, T, H, GDN_K, V, a.L, on.stream),
                      "llattn_gdn_bwd_kept_bf16dv");
            } else {
                check(lib.llattn_gdn_bwd(qn.data_ptr(), kn.data_ptr(), v.data_ptr(), b.data_ptr(), fptr(g_cum), l.data_ptr(), Aw.data_ptr(), Au.data_ptr(),
                                         d_o.data_ptr(), dq, dk, fptr(dv), db, fptr(dgp), dl, ws.data_ptr(), bytes, B, T, H, GDN_K, V, a.L, on.stream),
                      "llattn_gdn_bwd");
                dv = dv.to(at::kBFloat16);
            }
        }
        if (status) check_status(ws, on.stream, "llattn_gdn_bwd");
        const Tensor gb = empty({B, T, a.H}, at::kBFloat16, q), gl = empty({B, T, a.H, a.L}, at::kBFloat16, q);
        const Tensor gg = a.rep > 1 ? empty({B, T, a.H}, at::kFloat, q) : dgp;
        check(lib.llattn_gdn_grad_out(normed ? nullptr : q.data_ptr(), k.data_ptr(), dq, dk, db, dl, a.rep > 1 ? fptr(dgp) : nullptr, gq.data_ptr(),
                                      gk.data_ptr(), gb.data_ptr(), gl.data_ptr(), fptr(gg), rows, a.rep, a.K, GDN_K, a.L, (float)scale, (float)lam_mul, on.stream),
              "llattn_gdn_grad_out");
        return {gq, gk, dv, gb, gg, gl, Tensor(), Tensor(), Tensor(), Tensor()};
    }
};

// hattention_kernel, delta-rule structure: l2norm of q (scaled) and k, lambda times lam_mul unless that is 0
py::object hattention_gdn(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g, const Tensor& l, double scale, double lam_mul,
                          int64_t keep_bytes, bool status) {
    if (!gdn_operands(q, k, v, b, g, l) || has_tangent({q, k, v, b, g, l})) return py::none();
    const int64_t T = q.size(1);
    if (T % 64 != 0 || T > 16384 || l.size(3) < 7 + ceil_log2(T / 64)) return py::none();
    const bool grad = wants_grad({q, k, v, b, g, l});
    if (grad && q.size(2) != v.size(2)) return py::none();
    py::gil_scoped_release nogil;
    Tensor o = grad ? GdnKernel::apply(q, k, v, b, g, l, scale, lam_mul, keep_bytes, status)
                    : GdnKernel::forward(nullptr, q, k, v, b, g, l, scale, lam_mul, 0, status);
    py::gil_scoped_acquire gil;
    return py::cast(o);
}

// a prompt of any length -> (o, level-major states) or None
py::object gdn_prompt(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g, const Tensor& l, double scale, double lam_mul,
                      bool status) {
    if (!gdn_operands(q, k, v, b, g, l)) return py::none();
    const int T = q.size(1), L = l.size(3), T0 = T / 64 * 64, n = T % 64;
    if (T0 > 16384 || L < 1 + bit_length(T - 1)) return py::none();
    Tensor o, states;
    {
        py::gil_scoped_release nogil;
        at::NoGradGuard no_grad;
        On on(q);
        GdnInputs a = gdn_prepare(contiguous(q), contiguous(k), contiguous(v), contiguous(b), contiguous(g), contiguous(l), T0, n, scale, lam_mul,
                                  on.stream);
        const int B = a.B, H = a.heads(), K = a.K, V = a.width;
        states = empty({B, a.H, L, K, a.V}, at::kFloat, q);
        o = empty({B, T, a.H, a.V}, at::kBFloat16, q);
        Tensor chunks = o, g_cum, Aw, Au, ws, scratch;
        size_t bytes = 0, more = 0;
        if (T0 > 0) {
            if (n > 0 && B > 1) chunks = empty({B, T0, a.H, a.V}, at::kBFloat16, q);
            g_cum = empty({B, T0, H}, at::kFloat, q);
            Aw = empty({B, T0, H, 64}, at::kBFloat16, q);
            Au = contiguous_like(Aw);
            bytes = lib.llattn_gdn_fwd_workspace_bytes(B, T0, H, GDN_K, V, L);
            ws = empty({(int64_t)bytes}, at::kByte, q);
        }
        if (n > 0) {
            more = lib.llattn_gdn_prompt_scratch_bytes(B, T0, n, H, a.rep, V);
            scratch = empty({(int64_t)more}, at::kByte, q);
        }
        check(lib.llattn_gdn_prompt(a.qn.data_ptr(), a.kn.data_ptr(), a.v.data_ptr(), a.b.data_ptr(), fptr(a.g), a.l.data_ptr(), chunks.data_ptr(),
                                    o.data_ptr(), fptr(g_cum), ptr(Aw), ptr(Au), fptr(states), K, a.rep, L, ptr(scratch), more, ptr(ws), bytes, B, T0, n, H,
                                    GDN_K, V, L, on.stream),
              "llattn_gdn_prompt");
        if (status && T0 > 0) check_status(ws, on.stream, "llattn_gdn_prompt");
        if (chunks.data_ptr() != o.data_ptr()) o.narrow(1, 0, T0).copy_(chunks);
        states = states.permute({0, 1, 3, 4, 2});
    }
    return py::make_tuple(o, states);
}

// ------------------------------------------------------------------------------------------ decode steps
// Runs the cascade on the token counts (a list of ints, updated in place): the levels that hold tokens before it, as bits, and the
// level that receives the merged ones.  The new token is counted.
struct Cascade {
    unsigned live = 0;
    int carry = 0;
};
Cascade cascade(const py::list& counts, int64_t L) {
    TORCH_CHECK_VALUE((int64_t)counts.size() == L && L <= 32, "one token count per level");
    Cascade c;
    int64_t n[32];
    for (int64_t i = 0; i < L; ++i) {
        n[i] = PyLong_AsLongLong(PyList_GET_ITEM(counts.ptr(), i));
        if (n[i] != 0) c.live |= 1u << i;
    }
    int level = 0;
    while (n[level] == (int64_t(1) << level)) {
        TORCH_CHECK_VALUE(level + 1 < L, "more tokens than the levels can hold");
        n[level + 1] += n[level];
        n[level] = 0;
        ++level;
    }
    TORCH_CHECK_VALUE(n[level] < (int64_t(1) << level), "more tokens in a level than it holds");
    c.carry = level;
    n[0] += 1;
    for (int64_t i = 0; i <= std::min<int64_t>(level, L - 1); ++i) PyList_SetItem(counts.ptr(), i, PyLong_FromLongLong(n[i]));
    return c;
}
bool level_major(const Tensor& s) {
    if (!is(s, at::kFloat) || s.dim() != 5 || !aligned(s)) return false;
    const int64_t H = s.size(1), K = s.size(2), V = s.size(3), L = s.size(4);
    const auto st = s.strides();
    return V % 16 == 0 && st[0] == H * L * K * V && st[1] == L * K * V && st[2] == V && st[3] == 1 && st[4] == K * V;
}

// hselective_state_update on a level-major state: y, or None (nothing done)
py::object mamba2_step(const Tensor& states, const py::list& counts, const Tensor& x, const Tensor& dt, const Tensor& A, const Tensor& Bm, const Tensor& Cm,
                       const Tensor& dl, const Tensor& Lp, const Maybe& D_, const Maybe& bias_, int64_t mode, bool softplus) {
    const Tensor D = of(D_), bias = of(bias_);
    if (!bf16(x) || !bf16(dt) || !bf16(Bm) || !bf16(Cm) || !bf16(dl) || !A.is_cuda() || !A.is_floating_point() || !param(Lp) || !param(D) || !param(bias) ||
        x.dim() != 3 || Bm.dim() != 3 || dl.dim() != 3 || !level_major(states) || wants_grad({x, dt, A, Bm, Cm, dl, Lp, D, bias}) ||
        !native_set({states, x, dt, A, Bm, Cm, dl, Lp, D, bias}))
        return py::none();
    const int64_t B = x.size(0), H = x.size(1), V = x.size(2), G = Bm.size(1), K = Bm.size(2), L = dl.size(2);
    if (states.sizes() != at::IntArrayRef({B, H, K, V, L}) || dt.sizes() != at::IntArrayRef({B, H}) || A.sizes() != at::IntArrayRef({H}) || G <= 0 || H % G != 0 ||
        Bm.size(0) != B || Cm.sizes() != Bm.sizes() || dl.sizes() != at::IntArrayRef({B, H, L}) || Lp.sizes() != at::IntArrayRef({H, L}) ||
        (D.defined() && D.sizes() != at::IntArrayRef({H})) || (bias.defined() && bias.sizes() != at::IntArrayRef({H})) || V > 256 || K > 1024)
        return py::none();
    const Tensor q = contiguous(Cm), k = contiguous(Bm), x_ = contiguous(x), dt_ = contiguous(dt), dl_ = contiguous(dl), Lp_ = contiguous(Lp),
                 A_ = contiguous(A.to(at::kFloat)), D_c = contiguous(D), b_ = contiguous(bias);
    const Tensor y = empty({B, H, V}, f32(D_c) ? at::kFloat : at::kBFloat16, x);
    const Cascade c = cascade(counts, L);
    const int dev = x.device().index();
    check(lib.llattn_mamba2_layer_step(fptr(states), q.data_ptr(), k.data_ptr(), x_.data_ptr(), dt_.data_ptr(), nullptr, dl_.data_ptr(), Lp_.data_ptr(),
                                       f32(Lp_), ptr(D_c), f32(D_c), ptr(b_), f32(b_), fptr(A_), y.data_ptr(), B, H, G, K, V, L, c.live, c.carry, (int)mode,
                                       softplus, dev, at::cuda::getCurrentCUDAStream(dev).stream()),
          "llattn_mamba2_layer_step");
    return py::cast(y);
}

// the one-token call of chunk_h_gated_delta_rule (a token dimension of one in every operand): o (B,1,H,V), or None (nothing done)
py::object gdn_step(const Tensor& states, const py::list& counts, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& b, const Tensor& g,
                    const Tensor& l, double scale, double lam_mul) {
    if (!bf16(q) || !bf16(k) || !bf16(v) || !bf16(b) || !is(g, at::kFloat) || !bf16(l) || q.dim() != 4 || v.dim() != 4 || l.dim() != 4 ||
        q.sizes() != k.sizes() || !level_major(states) || !native_set({states, q, k, v, b, g, l}))
        return py::none();
    const int64_t B = q.size(0), G = q.size(2), K = q.size(3), H = v.size(2), V = v.size(3), L = l.size(3);
    if (q.size(1) != 1 || v.size(0) != B || v.size(1) != 1 || b.sizes() != at::IntArrayRef({B, 1, H}) || g.sizes() != b.sizes() ||
        l.sizes() != at::IntArrayRef({B, 1, H, L}) || states.sizes() != at::IntArrayRef({B, H, K, V, L}) || G <= 0 || H % G != 0 || K > 256)
        return py::none();
    const Tensor q_ = contiguous(q), k_ = contiguous(k), v_ = contiguous(v), b_ = contiguous(b), g_ = contiguous(g), l_ = contiguous(l);
    const Tensor o = empty({B, 1, H, V}, at::kBFloat16, q);
    const Cascade c = cascade(counts, L);
    const int dev = q.device().index();
    check(lib.llattn_gdn_layer_step(fptr(states), q_.data_ptr(), k_.data_ptr(), v_.data_ptr(), b_.data_ptr(), fptr(g_), l_.data_ptr(), o.data_ptr(), B, H, G, K,
                                    V, L, c.live, c.carry, 1, (float)scale, (float)lam_mul, dev, at::cuda::getCurrentCUDAStream(dev).stream()),
          "llattn_gdn_layer_step");
    return py::cast(o);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.def("bind", &bind);
    m.def("hattention_mamba2", &hattention_mamba2);
    m.def("mamba2_layer", &mamba2_layer);
    m.def("mamba2_prompt", &mamba2_prompt);
    m.def("mamba2_prefill", &mamba2_prefill);
    m.def("mamba2_mixer", &mamba2_mixer);
    m.def("mamba2_step", &mamba2_step);
    m.def("hattention_gdn", &hattention_gdn);
    m.def("gdn_prompt", &gdn_prompt);
    m.def("gdn_step", &gdn_step);
}

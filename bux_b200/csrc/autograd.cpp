// The layers' differentiable ops as C++ autograd functions: RMSNorm, per-head norm + RoPE, gated
// activation, bf16 linear and attention. They are the Python functions of ops/functional.py (which
// run for what needs Python: kernel checks, gradients kept in a buffer of the parameter, weights on
// their way from other GPUs, replayed attention) with the same kernels, casts and saved tensors. What
// they take out is the interpreter: a forward and backward of a small op waited for it, not for
// the GPU (forward + backward of an RMSNorm of 16 rows 103 us of host time, 67 now; of a linear 130, 79;
// of an elementwise product of PyTorch's own, which is mostly the hand-over to the backward thread, 61).
#include <torch/csrc/autograd/custom_function.h>
#include <torch/library.h>

#include <atomic>

#include "bindings.h"
#include "gemm_sm100.h"

namespace bux_ops {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

namespace {

std::atomic<int64_t> launched{0};   // kernels launched here (the wrappers of ops/kernels.py count their own)

OptTensor f32(const OptTensor& t) {
  if (!t.has_value() || !t->defined()) return std::nullopt;
  return t->to(at::kFloat).contiguous();
}
OptTensor opt(const Tensor& t) { return t.defined() ? OptTensor(t) : std::nullopt; }
Tensor val(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
Tensor fp32_like(const Tensor& t, at::IntArrayRef shape) { return at::empty(shape, t.options().dtype(at::kFloat)); }

// ------------------------------------------------------------------ RMSNorm
struct RMSNorm : torch::autograd::Function<RMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& w, double eps) {
    TORCH_CHECK(x.dim() > 0 && x.size(-1) > 0, "rmsnorm: rows of at least one element");
    const Tensor xc = x.contiguous();
    Tensor y = at::empty(xc.sizes(), xc.options()), rstd = fp32_like(xc, {xc.numel() / xc.size(-1)});
    rmsnorm_fwd(xc, f32(w), y, rstd, eps);
    launched += 1;
    ctx->save_for_backward({xc, val(w), rstd});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &rstd = saved[2];
    Tensor dx = at::empty(x.sizes(), x.options()), dw;
    if (w.defined()) dw = fp32_like(x, {x.size(-1)});
    rmsnorm_bwd(x, f32(opt(w)), g[0].contiguous(), rstd, dx, opt(dw));
    launched += 1;
    return {dx, w.defined() ? dw.to(w.scalar_type()) : Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------ norm + RoPE
// x as the kernel walks it: itself where it can be read in place (a column slice of a fused projection),
// else a copy. `contiguous()` is no test of that: it returns x itself whatever the strides of its
// dimensions of size 1 are, and wherever x starts.
Tensor walkable(const Tensor& x) {
  return token_stride(x) >= 0 ? x : x.clone(at::MemoryFormat::Contiguous);
}

struct NormRope : torch::autograd::Function<NormRope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& w, const Tensor& cos, const Tensor& sin, double eps) {
    TORCH_CHECK(x.dim() >= 3 && x.size(-1) > 0 && x.size(-2) > 0, "norm_rope: x is [..., tokens, heads, D], of at least one head");
    const Tensor xc = walkable(x);
    const int64_t d = xc.size(-1), h = xc.size(-2), tokens = xc.numel() / (h * d);
    const Tensor c = cos.reshape({-1, d / 2}).to(at::kFloat).contiguous(), s = sin.reshape({-1, d / 2}).to(at::kFloat).contiguous();
    const OptTensor wf = f32(w);
    Tensor y = at::empty(xc.sizes(), xc.options()), rstd;
    if (wf.has_value()) rstd = fp32_like(xc, {tokens * h});
    norm_rope(false, xc, wf, c, s, y, opt(rstd), std::nullopt, std::nullopt, tokens, h, d, token_stride(xc), h * d, eps);
    launched += 1;
    ctx->save_for_backward({xc, val(w), c, s, rstd});
    ctx->saved_data["eps"] = eps;
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1], &c = saved[2], &s = saved[3], &rstd = saved[4];
    const int64_t d = x.size(-1), h = x.size(-2), tokens = x.numel() / (h * d);
    Tensor dx = at::empty(x.sizes(), x.options()), dw;
    if (w.defined()) dw = at::zeros({d}, x.options().dtype(at::kFloat));
    const Tensor xc = walkable(x);   // a hook on saved tensors may have given x back with other strides
    norm_rope(true, xc, f32(opt(w)), c, s, dx, opt(rstd), walkable(g[0].contiguous()), opt(dw), tokens, h, d, token_stride(xc), h * d,
              ctx->saved_data["eps"].toDouble());
    launched += 1;
    return {dx, w.defined() ? dw.to(w.scalar_type()) : Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------ gated activation
struct Glu : torch::autograd::Function<Glu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& h, const OptTensor& row_scale, int64_t kind, double limit, double up_offset) {
    const Tensor hc = h.contiguous();
    const OptTensor rs = f32(row_scale);
    auto shape = hc.sizes().vec();
    shape.back() /= 2;
    Tensor out = at::empty(shape, hc.options());
    glu_fwd(hc, out, rs, kind, limit, up_offset);
    launched += 1;
    ctx->save_for_backward({hc, val(rs)});
    ctx->saved_data["kind"] = kind; ctx->saved_data["limit"] = limit; ctx->saved_data["up_offset"] = up_offset;
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &h = saved[0], &rs = saved[1];
    Tensor dh = at::empty(h.sizes(), h.options()), drs;
    if (rs.defined()) drs = at::empty(rs.sizes(), rs.options());
    glu_bwd(h, g[0].contiguous(), dh, opt(rs), opt(drs), ctx->saved_data["kind"].toInt(), ctx->saved_data["limit"].toDouble(),
            ctx->saved_data["up_offset"].toDouble());
    launched += 1;
    return {dh, drs, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------ linear
// C = A · B^T in bf16 (operands as `gemm` takes them), of the given shape.
Tensor product(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, at::IntArrayRef shape, const Tensor& status) {
  const int64_t m = a.size(a_mn ? 1 : 0), k = a.size(a_mn ? 0 : 1), n = b.size(b_mn ? 1 : 0);
  const Tensor out = at::empty(shape, a.options().dtype(at::kBFloat16));
  Tensor c = out.view({m, n});
  gemm(a, b, c, std::nullopt, std::nullopt, std::nullopt, status, bux::KIND_BF16, bux::MODE_DENSE, m, n, k, k, 1, a_mn, b_mn,
       bux::OUT_BF16, 0, 0, std::nullopt, 0, 0, 0, false, false);
  launched += 1;
  return out;
}

struct Linear : torch::autograd::Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const Tensor& status) {
    const Tensor x2 = x.reshape({-1, x.size(-1)}).contiguous();
    auto shape = x.sizes().vec();
    ctx->saved_data["shape"] = shape;
    ctx->saved_data["status"] = status;
    ctx->save_for_backward({x2, w});
    shape.back() = w.size(0);
    return product(x2, w, false, false, shape, status);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &x2 = saved[0], &w = saved[1];
    const Tensor status = ctx->saved_data["status"].toTensor();
    const Tensor dy = g[0].reshape({-1, g[0].size(-1)}).contiguous();
    Tensor dx, dw;
    if (ctx->needs_input_grad(0)) dx = product(dy, w, false, true, ctx->saved_data["shape"].toIntVector(), status);
    if (ctx->needs_input_grad(1)) dw = product(dy, x2, true, true, w.sizes(), status);
    return {dx, dw, Tensor()};
  }
};

// ------------------------------------------------------------------ attention
struct Attention : torch::autograd::Function<Attention> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_, const Tensor& k_, const Tensor& v_, const OptTensor& sinks,
                        const OptTensor& row_lo, const OptTensor& key_hi, const Tensor& status, bool causal, int64_t window, double scale) {
    const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
    const OptTensor sk = f32(sinks);
    Tensor o = at::empty(q.sizes(), q.options()), lse = fp32_like(q, {q.size(0), q.size(2), q.size(1)});
    attn_fwd(q, k, v, o, lse, sk, status, scale, causal, window, row_lo);
    launched += 1;
    ctx->save_for_backward({q, k, v, o, lse, val(sk), val(row_lo), val(key_hi)});
    ctx->saved_data["status"] = status; ctx->saved_data["causal"] = causal; ctx->saved_data["window"] = window;
    ctx->saved_data["scale"] = scale;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &sk = s[5];
    Tensor dq = at::zeros(q.sizes(), q.options().dtype(at::kFloat)), dk = at::empty(k.sizes(), k.options()), dv = at::empty(v.sizes(), v.options());
    Tensor delta = fp32_like(q, {q.size(0), q.size(2), q.size(1)}), dsk;
    if (sk.defined()) dsk = at::zeros_like(sk);
    attn_bwd(q, k, v, s[3], g[0].contiguous(), s[4], dq, dk, dv, delta, opt(sk), opt(dsk), ctx->saved_data["status"].toTensor(),
             ctx->saved_data["scale"].toDouble(), ctx->saved_data["causal"].toBool(), ctx->saved_data["window"].toInt(), opt(s[6]), opt(s[7]),
             std::nullopt);
    launched += 2;
    return {dq.to(q.scalar_type()), dk, dv, dsk, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor ad_rmsnorm(const Tensor& x, const OptTensor& w, double eps) { return RMSNorm::apply(x, w, eps); }
Tensor ad_norm_rope(const Tensor& x, const OptTensor& w, const Tensor& cos, const Tensor& sin, double eps) {
  return NormRope::apply(x, w, cos, sin, eps);
}
Tensor ad_glu(const Tensor& h, const OptTensor& row_scale, int64_t kind, double limit, double up_offset) {
  return Glu::apply(h, row_scale, kind, limit, up_offset);
}
Tensor ad_linear(const Tensor& x, const Tensor& w, const Tensor& status) { return Linear::apply(x, w, status); }
Tensor ad_attention(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& sinks, const OptTensor& row_lo,
                    const OptTensor& key_hi, const Tensor& status, bool causal, int64_t window, double scale) {
  return Attention::apply(q, k, v, sinks, row_lo, key_hi, status, causal, window, scale);
}
int64_t native_launches() { return launched.load(); }

}  // namespace
}  // namespace bux_ops

TORCH_LIBRARY_FRAGMENT(bux_b200, m) {
  using namespace bux_ops;
  m.def("ad_rmsnorm(Tensor x, Tensor? w, float eps) -> Tensor", &ad_rmsnorm);
  m.def("ad_norm_rope(Tensor x, Tensor? w, Tensor cos, Tensor sin, float eps) -> Tensor", &ad_norm_rope);
  m.def("ad_glu(Tensor h, Tensor? row_scale, int kind, float limit, float up_offset) -> Tensor", &ad_glu);
  m.def("ad_linear(Tensor x, Tensor w, Tensor status) -> Tensor", &ad_linear);
  m.def("ad_attention(Tensor q, Tensor k, Tensor v, Tensor? sinks, Tensor? row_lo, Tensor? key_hi, Tensor status, bool causal, int window, float scale) -> Tensor", &ad_attention);
  m.def("native_launches() -> int", &native_launches);
}

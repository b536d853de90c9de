// The checked wrappers of bindings.cpp that other C++ code of the library calls.
#pragma once
#include <ATen/ATen.h>

namespace bux_ops {

using at::Tensor;

void gemm(const Tensor& a, const Tensor& b, Tensor& c, const std::optional<Tensor>& sfa, const std::optional<Tensor>& sfb,
          const std::optional<Tensor>& group_offsets, const std::optional<Tensor>& status, int64_t kind, int64_t mode, int64_t M,
          int64_t N, int64_t K, int64_t k_total, int64_t groups, bool a_mn, bool b_mn, int64_t out_kind, int64_t bn, int64_t sms,
          const std::optional<Tensor>& wait_flags, int64_t wait_epoch, int64_t wait_rows, int64_t m_rotate, bool wait_on_k, bool wait_on_n,
          const std::optional<Tensor>& scratch = std::nullopt);
void rmsnorm_fwd(const Tensor& x, const std::optional<Tensor>& w, Tensor& y, Tensor& rstd, double eps);
void rmsnorm_bwd(const Tensor& x, const std::optional<Tensor>& w, const Tensor& dy, const Tensor& rstd, Tensor& dx, const std::optional<Tensor>& dw,
                 const std::optional<Tensor>& scratch = std::nullopt);
// Elements between tokens of x [..., T, H, D] when heads are dense and the leading dimensions collapse
// into one (a column slice of a fused projection), x starts on 16 bytes and every token too; else -1.
int64_t token_stride(const Tensor& x);
void norm_rope(bool bwd, const Tensor& x, const std::optional<Tensor>& w, const Tensor& cos, const Tensor& sin, Tensor& y,
               const std::optional<Tensor>& rstd, const std::optional<Tensor>& dy, const std::optional<Tensor>& dw, int64_t tokens,
               int64_t heads, int64_t D, int64_t stride_x, int64_t stride_y, double eps);
void glu_fwd(const Tensor& h, Tensor& out, const std::optional<Tensor>& row_scale, int64_t kind, double limit, double up_offset);
void glu_bwd(const Tensor& h, const Tensor& dout, Tensor& dh, const std::optional<Tensor>& row_scale, const std::optional<Tensor>& d_row_scale,
             int64_t kind, double limit, double up_offset);
void attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, Tensor& o, Tensor& lse, const std::optional<Tensor>& sinks,
              const std::optional<Tensor>& status, double scale, bool causal, int64_t window, const std::optional<Tensor>& row_lo);
void attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& d_o, const Tensor& lse, Tensor& dq,
              Tensor& dk, Tensor& dv, Tensor& delta, const std::optional<Tensor>& sinks, const std::optional<Tensor>& dsinks,
              const std::optional<Tensor>& status, double scale, bool causal, int64_t window, const std::optional<Tensor>& row_lo,
              const std::optional<Tensor>& key_hi, const std::optional<Tensor>& phase_cycles);

}  // namespace bux_ops

// The per-layer operations around the scan: depthwise convolution + SiLU, RMSNorm with and without the residual add, and
// the two kernels of a decode step.
#include "host.h"

namespace mb200_host {
namespace {

// The filter of `width` channels, (width, d_conv).
Tensor filter(const Tensor& weight, int64_t width) {
  numel_is(weight, width * weight.size(-1), "the filter");
  return f32(weight).view({width, weight.size(-1)});
}

struct ConvBackward : public torch::autograd::Node {
  Saved x, w, b;
  at::ScalarType tx, tw, tb;
  std::vector<int64_t> w_shape;
  std::string name() const override { return "CausalConv1dSiluBackward"; }
  void release_variables() override { x.reset(); w.reset(); b.reset(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(3);
    if (!grads[0].defined()) return out;
    const BelowAutograd guard_ad;
    const Tensor xs = x.get(), w32 = w.get(), b32 = b.get();
    const c10::cuda::CUDAGuard guard(xs.device());
    const Tensor dy = rows(grads[0], xs.scalar_type());
    const int64_t B = xs.size(0), L = xs.size(1), W = xs.size(2), K = w32.size(1);
    const Tensor dx = empty({B, L, W}, xs.scalar_type(), xs), acc = empty({W * K + W}, at::kFloat, xs);
    zero_fill(acc);
    const Tensor dw = alias(acc, 0, w_shape), db = b32.defined() ? alias(acc, W * K, {W}) : Tensor();
    check(mb200_conv1d_silu_bwd(ptr(xs), fptr(w32), fptr(b32), ptr(dy), ptr(dx), fptr(dw), fptr(db), B, L, W, int(K), st(xs, 0), st(xs, 1),
                                st(dy, 0), st(dy, 1), st(dx, 0), st(dx, 1), dtype_code(xs.scalar_type()), cuda_stream()),
          "mb200_conv1d_silu_bwd");
    out[0] = like(dx, tx);
    out[1] = like(dw, tw);
    if (db.defined()) out[2] = like(db, tb);
    return out;
  }
};

}  // namespace

Tensor conv1d_silu(const Tensor& x, const Tensor& weight, const OptTensor& bias_) {
  const Tensor& bias = value(bias_);
  require_cuda(x, weight, bias);
  refuse_tangents(x, weight, bias);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor y, xs, w32, b32;
  {
    const BelowAutograd guard_ad;
    xs = rows(x, act_dtype(x));
    w32 = filter(weight, xs.size(2));
    b32 = f32(bias);
    numel_is(b32, xs.size(2), "the bias");
    const int64_t B = xs.size(0), L = xs.size(1), W = xs.size(2), K = w32.size(1);
    y = empty({B, L, W}, xs.scalar_type(), xs);
    check(mb200_conv1d_silu_fwd(ptr(xs), fptr(w32), fptr(b32), ptr(y), B, L, W, int(K), st(xs, 0), st(xs, 1), st(y, 0), st(y, 1),
                                dtype_code(xs.scalar_type()), cuda_stream()),
          "mb200_conv1d_silu_fwd");
  }
  if (wants_grad(x, weight, bias)) {
    auto node = new_node<ConvBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, weight, bias));
    node->x.save(xs); node->w.save(w32); node->b.save(b32);
    node->tx = type_of(x); node->tw = type_of(weight); node->tb = type_of(bias);
    node->w_shape = weight.sizes().vec();
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ------------------------------------------------------------------------------------------------------ norms
namespace {

// (rows, D) view of a tensor for the row-wise kernels.
Tensor row_view(const Tensor& t, at::ScalarType dt) {
  Tensor r = t.reshape({-1, t.size(-1)});
  if (r.scalar_type() != dt) r = r.to(dt);
  return r.stride(-1) == 1 ? r : r.contiguous();
}

struct RmsNormBackward : public torch::autograd::Node {
  Saved x, w, rstd;
  std::vector<int64_t> shape;
  at::ScalarType tx, tw;
  std::string name() const override { return "RMSNormBackward"; }
  void release_variables() override { x.reset(); w.reset(); rstd.reset(); }
  variable_list apply(variable_list&& grads) override {
    variable_list out(2);
    if (!grads[0].defined()) return out;
    const BelowAutograd guard_ad;
    const Tensor x2 = x.get(), w32 = w.get(), rs = rstd.get();
    const c10::cuda::CUDAGuard guard(x2.device());
    const int64_t n = x2.size(0), D = x2.size(1);
    const Tensor dy = row_view(grads[0], x2.scalar_type()), dx = empty({n, D}, x2.scalar_type(), x2);
    Tensor dw;
    if (w32.defined()) {
      dw = empty({D}, at::kFloat, x2);
      zero_fill(dw);
    }
    check(mb200_rmsnorm_bwd(ptr(x2), fptr(w32), fptr(rs), ptr(dy), ptr(dx), fptr(dw), n, D, st(x2, 0), st(dy, 0), st(dx, 0),
                            dtype_code(x2.scalar_type()), cuda_stream()),
          "mb200_rmsnorm_bwd");
    out[0] = like(dx.view(shape), tx);
    if (dw.defined()) out[1] = like(dw, tw);
    return out;
  }
};

struct AddRmsNormBackward : public torch::autograd::Node {
  Saved s, w, rstd;
  std::vector<int64_t> shape;
  at::ScalarType tx, tr, tw;
  bool has_residual = false;
  std::string name() const override { return "AddRMSNormBackward"; }
  void release_variables() override { s.reset(); w.reset(); rstd.reset(); }
  variable_list apply(variable_list&& grads) override {                    // d y, d s -> x, residual, weight
    variable_list out(3);
    const BelowAutograd guard_ad;
    const Tensor sum = s.get(shared_from_this()), w32 = w.get(), rs = rstd.get();
    const c10::cuda::CUDAGuard guard(sum.device());
    const Tensor s2 = sum.view({-1, sum.size(-1)});
    const int64_t n = s2.size(0), D = s2.size(1);
    const auto ts = s2.scalar_type();
    Tensor ds;
    if (grads[0].defined()) {
      auto ty = grads[0].scalar_type();
      if (ty != at::kBFloat16 || ts == at::kBFloat16) ty = ts == at::kBFloat16 ? at::kBFloat16 : at::kFloat;
      const Tensor dy = row_view(grads[0], ty), dr = grads[1].defined() ? row_view(grads[1], ts) : Tensor();
      ds = empty({n, D}, ts, s2);
      Tensor dw;
      if (w32.defined()) {
        dw = empty({D}, at::kFloat, s2);
        zero_fill(dw);
      }
      // a bfloat16 x beside a float32 stream: its gradient leaves the kernel rounded, without a cast of its own
      Tensor dx;
      int rc = MB200_EUNSUPPORTED;
      if (ts == at::kFloat && tx == at::kBFloat16) {
        dx = empty(shape, at::kBFloat16, s2);
        rc = mb200_add_rmsnorm_bwd_both(ptr(s2), fptr(w32), fptr(rs), ptr(dy), ptr(dr), ptr(ds), ptr(dx), fptr(dw), n, D, st(s2, 0), st(dy, 0),
                                        st(dr, 0), st(ds, 0), dtype_code(ts), dtype_code(ty), cuda_stream());
      }
      if (rc == MB200_EUNSUPPORTED) {
        dx = Tensor();
        rc = mb200_add_rmsnorm_bwd(ptr(s2), fptr(w32), fptr(rs), ptr(dy), ptr(dr), ptr(ds), fptr(dw), n, D, st(s2, 0), st(dy, 0), st(dr, 0),
                                   st(ds, 0), dtype_code(ts), dtype_code(ty), cuda_stream());
      }
      check(rc, "mb200_add_rmsnorm_bwd");
      out[0] = dx;
      if (dw.defined()) out[2] = like(dw, tw);
      ds = ds.view(shape);
    } else {
      ds = grads[1];                                                       // only the sum was used further on
      if (!ds.defined()) return out;
      if (w32.defined() && task_should_compute_output(2)) {                // which the weight has no part in
        out[2] = empty(w32.sizes(), tw, s2);
        zero_fill(out[2]);
      }
    }
    if (!out[0].defined()) out[0] = like(ds, tx);
    if (has_residual) out[1] = like(ds, tr);
    return out;
  }
};

constexpr const char* kNeedCuda = "mamba_b200 kernels need CUDA tensors; there is no CPU path";

}  // namespace

Tensor rms_norm(const Tensor& x, const OptTensor& weight_, double eps) {
  const Tensor& weight = value(weight_);
  TORCH_CHECK(x.is_cuda(), kNeedCuda);
  refuse_tangents(x, weight);
  const c10::cuda::CUDAGuard guard(x.device());
  const bool grad = wants_grad(x, weight);
  Tensor y, x2, w32, rstd;
  {
    const BelowAutograd guard_ad;
    const auto dt = act_dtype(x);
    x2 = row_view(x, dt);
    const int64_t n = x2.size(0), D = x2.size(1);
    y = empty(x.sizes(), dt, x);
    if (grad) rstd = empty({n}, at::kFloat, x);
    int rc = MB200_EUNSUPPORTED;
    if (!grad && weight.defined() && weight.scalar_type() == at::kBFloat16 && weight.is_contiguous())
      rc = mb200_rmsnorm_fwd_typed(ptr(x2), ptr(weight), MB200_BF16, ptr(y), nullptr, n, D, st(x2, 0), D, float(eps), dtype_code(dt), cuda_stream());
    if (rc == MB200_EUNSUPPORTED) {
      w32 = f32(weight);
      rc = mb200_rmsnorm_fwd(ptr(x2), fptr(w32), ptr(y), fptr(rstd), n, D, st(x2, 0), D, float(eps), dtype_code(dt), cuda_stream());
    }
    check(rc, "mb200_rmsnorm_fwd");
  }
  if (grad) {
    auto node = new_node<RmsNormBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, weight));
    node->x.save(x2); node->w.save(w32); node->rstd.save(rstd);
    node->shape = x.sizes().vec();
    node->tx = type_of(x); node->tw = type_of(weight);
    torch::autograd::set_history(y, node);
  }
  return y;
}

std::tuple<Tensor, Tensor> add_rms_norm(const Tensor& x, const OptTensor& residual_, const OptTensor& weight_, double eps) {
  const Tensor &residual = value(residual_), &weight = value(weight_);
  TORCH_CHECK(x.is_cuda(), kNeedCuda);
  refuse_tangents(x, residual, weight);
  const c10::cuda::CUDAGuard guard(x.device());
  // the sum has the type `x + residual` would give; under autocast y comes out in the autocast dtype, which is what the
  // projection that consumes it would cast it to anyway
  const auto ts = residual.defined() ? c10::promoteTypes(x.scalar_type(), residual.scalar_type()) : x.scalar_type();
  auto ty = at::autocast::is_autocast_enabled(at::kCUDA) ? at::autocast::get_autocast_dtype(at::kCUDA) : ts;
  if (ty != at::kBFloat16) ty = at::kFloat;
  Tensor y, s, w32, rstd;
  {
    const BelowAutograd guard_ad;
    act_dtype(x, residual);
    const Tensor x2 = row_view(x, x.scalar_type()), r2 = residual.defined() ? row_view(residual, ts) : Tensor();
    w32 = f32(weight);
    const int64_t n = x2.size(0), D = x2.size(1);
    s = empty(x.sizes(), ts, x);
    y = empty(x.sizes(), ty, x);
    rstd = empty({n}, at::kFloat, x);
    check(mb200_add_rmsnorm_fwd(ptr(x2), ptr(r2), fptr(w32), ptr(s), ptr(y), fptr(rstd), n, D, st(x2, 0), st(r2, 0), D, D, float(eps),
                                dtype_code(x2.scalar_type()), dtype_code(ts), dtype_code(ty), cuda_stream()),
          "mb200_add_rmsnorm_fwd");
  }
  if (wants_grad(x, residual, weight)) {
    auto node = new_node<AddRmsNormBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, residual, weight));
    node->shape = x.sizes().vec();
    node->tx = type_of(x); node->tr = type_of(residual); node->tw = type_of(weight);
    node->has_residual = residual.defined();
    variable_list outs{y, s};
    torch::autograd::set_history(outs, node);
    node->s.save(s, true); node->w.save(w32); node->rstd.save(rstd);
  }
  return {y, s};
}

void selftest_queue_conversions(int64_t n) {
  Convert conv;
  for (int64_t i = 0; i < n; ++i) conv.add(nullptr, at::kFloat, nullptr, at::kFloat, 0, 0, 0, 0, 0);
}

// ---------------------------------------------------------------------------------------------- the last residual add
namespace {

struct AddResidualBackward : public torch::autograd::Node {
  at::ScalarType tx;
  std::string name() const override { return "AddResidualBackward"; }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return variable_list(2);
    const BelowAutograd guard_ad;
    const c10::cuda::CUDAGuard guard(grads[0].device());
    Convert conv;
    const Tensor g = grads[0].is_contiguous() ? grads[0] : grads[0].contiguous();
    const Tensor dx = g.scalar_type() == at::kFloat ? conv.cast(g, tx) : like(g, tx);
    conv.run();
    return {dx, grads[0]};
  }
};

}  // namespace

// x + residual at the end of a stack: a bfloat16 mixer output on a float32 stream in one vectorised pass.
Tensor add_residual(const Tensor& x, const Tensor& residual) {
  const bool ours = x.is_cuda() && residual.is_cuda() && x.sizes() == residual.sizes() && x.is_contiguous() && residual.is_contiguous() &&
                    x.scalar_type() == at::kBFloat16 && residual.scalar_type() == at::kFloat && !has_tangent(x) && !has_tangent(residual);
  if (!ours) return at::add(x, residual);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor s;
  {
    const BelowAutograd guard_ad;
    s = empty(x.sizes(), at::kFloat, x);
    const int64_t n = s.numel();
    Convert conv;
    conv.add(ptr(x), at::kBFloat16, ptr(s), at::kFloat, 1, n, n, n, n, MB200_CONVERT_ADD).factor = fptr(residual);
    conv.run();
  }
  if (wants_grad(x, residual)) {
    auto node = new_node<AddResidualBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(x, residual));
    node->tx = type_of(x);
    torch::autograd::set_history(s, node);
  }
  return s;
}

}  // namespace mb200_host

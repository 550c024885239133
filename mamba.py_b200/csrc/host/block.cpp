// The inside of a Mamba block as ONE autograd node.
//
// Written as separate nodes, autograd glues a block's backward together with copies: a `cat` of the gradients of the two halves
// of xz (the whole (B, L, 2 ED) tensor again), a `cat` for the split of the x_proj output, an add of the two gradients that
// reach the conv output, casts of every parameter and of its gradient.  Here the backward writes dz and the conv's dx straight
// into the two halves of d(xz), dB and dC straight into d(x_proj output), adds the second gradient of the conv output in the
// epilogue of the GEMM that produces it, and prepares all parameters (and finishes all their gradients) in one launch.
#include "scan.h"

namespace mb200_host {
namespace {

// Up to 12 element-wise jobs in one launch (mb200_convert).
struct Convert {
  mb200_convert_job jobs[12];
  int n = 0;
  mb200_convert_job& add(const void* src, at::ScalarType st, void* dst, at::ScalarType dt, int64_t rows, int64_t cols, int64_t src_cols,
                         int64_t src_stride, int64_t dst_stride, int op = MB200_CONVERT_COPY) {
    mb200_convert_job& j = jobs[n++];
    j = mb200_convert_job{src, dst, nullptr, rows, cols, src_cols, src_stride, dst_stride, dtype_code(st), dtype_code(dt), op};
    return j;
  }
  // a dense copy of `src` in another type
  Tensor cast(const Tensor& src, at::ScalarType dt) {
    const Tensor dst = empty(src.sizes(), dt, src);
    add(ptr(src), src.scalar_type(), ptr(dst), dt, 1, src.numel(), src.numel(), src.numel(), src.numel());
    return dst;
  }
  void run() {
    if (n) check(mb200_convert(jobs, n, cuda_stream()), "mb200_convert");
    n = 0;
  }
};

bool convertible(at::ScalarType d) { return d == at::kFloat || d == at::kBFloat16; }

// The GEMMs below run in the type their operands have.
using NoAutocast = c10::impl::ExcludeDispatchKeyGuard;

// A parameter the conversion kernel reads directly; anything that is neither float32 nor bfloat16 becomes float32 first.
Tensor param(const Tensor& t) {
  if (!t.defined()) return t;
  return (convertible(t.scalar_type()) ? t : t.to(at::kFloat)).contiguous();
}

// The right-to-left convolution of the second direction is the same kernel with the rows taken backwards.
struct Backwards {
  int64_t sign, skip;
  Backwards(const Tensor& t, bool reverse) : sign(reverse ? -1 : 1), skip(reverse && t.size(1) > 0 ? t.size(1) - 1 : 0) {}
  void* row0(const Tensor& t) const { return static_cast<char*>(t.data_ptr()) + skip * t.stride(1) * t.element_size(); }
  int64_t step(const Tensor& t) const { return sign * t.stride(1); }
};

void conv_forward(const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& y, bool reverse) {
  const Backwards d(x, reverse);
  check(mb200_conv1d_silu_fwd(d.row0(x), fptr(w), fptr(b), d.row0(y), x.size(0), x.size(1), x.size(2), int(w.size(1)), x.stride(0),
                              d.step(x), y.stride(0), d.step(y), dtype_code(x.scalar_type()), cuda_stream()),
        "mb200_conv1d_silu_fwd");
}
void conv_backward(const Tensor& x, const Tensor& w, const Tensor& b, const Tensor& dy, const Tensor& dx, float* dw, float* db, bool reverse) {
  const Backwards d(x, reverse);
  check(mb200_conv1d_silu_bwd(d.row0(x), fptr(w), fptr(b), d.row0(dy), d.row0(dx), dw, db, x.size(0), x.size(1), x.size(2), int(w.size(1)),
                              x.stride(0), d.step(x), dy.stride(0), d.step(dy), dx.stride(0), d.step(dx), dtype_code(x.scalar_type()),
                              cuda_stream()),
        "mb200_conv1d_silu_bwd");
}

enum { kXz, kConvW, kConvB, kXproj, kDtW, kDtB, kALog, kD, kParams };

struct InnerBackward : public torch::autograd::Node {
  Saved xz, xc, dbc, delta, A, D, bias, carries, P, cw, cb, Wx, Wdt;
  int64_t R = 0, Rp = 0, N = 0, S = 1;
  bool reverse = false;
  at::ScalarType types[kParams];
  std::vector<int64_t> cw_shape;

  std::string name() const override { return "MambaInnerBackward"; }
  void release_variables() override {
    for (Saved* s : {&xz, &xc, &dbc, &delta, &A, &D, &bias, &carries, &P, &cw, &cb, &Wx, &Wdt}) s->reset();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(kParams);
    if (!grads[0].defined()) return out;
    const BelowAutograd guard_ad;
    const NoAutocast no_autocast(c10::DispatchKey::AutocastCUDA);
    const Tensor xz_ = xz.get(), xc_ = xc.get(), dbc_ = dbc.get(), A_ = A.get(), Wx_ = Wx.get(), Wdt_ = Wdt.get(), cw_ = cw.get(),
                 cb_ = cb.get();
    const c10::cuda::CUDAGuard guard(xz_.device());
    const auto dt = xc_.scalar_type();
    const int64_t B = xc_.size(0), L = xc_.size(1), W = xc_.size(2), T = B * L, cols = Rp + 2 * N, K = cw_.size(1);
    Tensor dy = rows(grads[0], dt);
    if ((reverse || S > 1) && !tensor_map_ok(dy)) dy = dy.contiguous();
    const Tensor dxz = empty({B, L, 2 * W}, dt, xz_);
    const ScanArgs a{xc_, delta.get(), A_, dbc_.narrow(2, Rp, N), dbc_.narrow(2, Rp + N, N), D.get(), xz_.narrow(2, W, W), bias.get(),
                     Tensor(), reverse};
    ScanGrads g = scan_backward(a, S, dy, carries.get(), P.get(), false, dxz.narrow(2, W, W), W * K + W);
    Convert conv;
    const Tensor d_dbc = empty({T, cols}, dt, xz_), dd2 = g.dd.view({T, W}), xc2 = xc_.view({T, W}), dx2 = g.dx.view({T, W});
    const int64_t es = d_dbc.element_size();
    auto col = [&](int64_t c) { return static_cast<char*>(d_dbc.data_ptr()) + c * es; };
    conv.add(ptr(g.dB), at::kFloat, col(Rp), dt, T, N, N, N, cols);         // float32 accumulators -> activation dtype, in place
    conv.add(ptr(g.dC), at::kFloat, col(Rp + N), dt, T, N, N, N, cols);
    conv.run();
    Tensor d_dt = d_dbc.narrow(1, 0, Rp);
    at::mm_out(d_dt, dd2, Wdt_);                                            // through dt_proj
    const Tensor dWdt = at::mm(dd2.t(), dbc_.view({T, cols}).narrow(1, 0, Rp));          // (W, Rp)
    const Tensor dWx = at::mm(d_dbc.t(), xc2);                              // (Rp + 2 N, W)
    Tensor dxc = dx2;
    at::addmm_out(dxc, dx2, d_dbc, Wx_);                                    // + the gradient through x_proj, in the GEMM's epilogue
    float* dcw = fptr(g.extra);
    float* dcb = dcw + W * K;
    conv_backward(xz_.narrow(2, 0, W), cw_, cb_, dxc.view({B, L, W}), dxz.narrow(2, 0, W), dcw, cb_.defined() ? dcb : nullptr, reverse);

    out[kXz] = dxz;
    at::ScalarType kt[kParams];                                            // what the conversion writes; anything else is cast after it
    for (int i = 0; i < kParams; ++i) kt[i] = convertible(types[i]) ? types[i] : at::kFloat;
    auto dense = [&](int i, const float* src, at::IntArrayRef shape) {
      out[i] = empty(shape, kt[i], xz_);
      const int64_t n = out[i].numel();
      conv.add(src, at::kFloat, ptr(out[i]), kt[i], 1, n, n, n, n);
    };
    dense(kConvW, dcw, cw_shape);
    if (cb_.defined()) dense(kConvB, dcb, {W});
    dense(kDtB, fptr(g.dbias), {W});
    dense(kD, fptr(g.dD), {W});
    out[kALog] = empty({W, N}, kt[kALog], xz_);                             // d A_log = dA * A
    conv.add(ptr(g.dA), at::kFloat, ptr(out[kALog]), kt[kALog], 1, W * N, W * N, W * N, W * N, MB200_CONVERT_MUL).factor = fptr(A_);
    out[kXproj] = empty({R + 2 * N, W}, kt[kXproj], xz_);
    char* wx = static_cast<char*>(ptr(out[kXproj]));
    conv.add(ptr(dWx), dt, wx, kt[kXproj], R, W, W, W, W);
    conv.add(static_cast<char*>(ptr(dWx)) + Rp * W * dWx.element_size(), dt, wx + R * W * out[kXproj].element_size(), kt[kXproj], 2 * N, W,
             W, W, W);
    out[kDtW] = empty({W, R}, kt[kDtW], xz_);
    conv.add(ptr(dWdt), dt, ptr(out[kDtW]), kt[kDtW], W, R, R, Rp, R);
    conv.run();
    for (int i = kConvW; i < kParams; ++i)
      if (out[i].defined()) out[i] = like(out[i], types[i]);
    return out;
  }
};

}  // namespace

// Everything between in_proj and out_proj of MambaBlock.forward (mambapy/mamba.py:214-231): conv1d + SiLU, x_proj, dt_proj and the
// fused scan with softplus(delta + bias) and the gate inside.  With `reverse`, the second direction of the bidirectional block
// (mambapy/vim.py:228-261): the convolution and the scan walk the sequence from its end, everything else is per timestep.
Tensor inner(const Tensor& xz, const Tensor& conv_w, const OptTensor& conv_b_, const Tensor& xproj_w, const Tensor& dt_w, const Tensor& dt_b,
             const Tensor& A_log, const Tensor& D, int64_t R, int64_t N, bool reverse) {
  const Tensor& conv_b = value(conv_b_);
  require_cuda(xz, conv_w, conv_b, xproj_w, dt_w, dt_b, A_log, D);
  const c10::cuda::CUDAGuard guard(xz.device());
  const bool grad = wants_grad(xz, conv_w, conv_b, xproj_w, dt_w, dt_b, A_log, D);
  const auto dt = act_dtype(xz);
  ScanArgs a;
  ScanOut o;
  Tensor cw, cb, dbc, Wx, Wdt, xzs;
  int64_t S = 1, Rp = 0;
  {
    const BelowAutograd guard_ad;
    const NoAutocast no_autocast(c10::DispatchKey::AutocastCUDA);
    xzs = rows(xz, dt);
    const int64_t B = xzs.size(0), L = xzs.size(1), W = xzs.size(2) / 2, K = conv_w.size(-1), T = B * L;
    // dt_rank rounded up to a multiple of 16 bytes: the dt, B and C columns of the x_proj output and the K of the dt_proj GEMM
    // then sit on the grid that TMA and the tensor-core GEMMs want; the extra weights are zero
    const int64_t v = 16 / xzs.element_size();
    Rp = (R + v - 1) / v * v;
    const int64_t cols = Rp + 2 * N;
    Convert conv;
    const Tensor wx = param(xproj_w), wdt = param(dt_w), alog = param(A_log);
    a.A = empty({W, N}, at::kFloat, xzs);
    conv.add(ptr(alog), alog.scalar_type(), ptr(a.A), at::kFloat, 1, W * N, W * N, W * N, W * N, MB200_CONVERT_NEG_EXP);
    Wx = wx;
    Wdt = wdt;
    if (Rp != R || wx.scalar_type() != dt) {
      Wx = empty({cols, W}, dt, xzs);
      char* d = static_cast<char*>(ptr(Wx));
      conv.add(ptr(wx), wx.scalar_type(), d, dt, R, W, W, W, W);
      if (Rp != R) conv.add(nullptr, dt, d + R * W * Wx.element_size(), dt, Rp - R, W, 0, W, W);
      conv.add(static_cast<char*>(ptr(wx)) + R * W * wx.element_size(), wx.scalar_type(), d + Rp * W * Wx.element_size(), dt, 2 * N, W, W, W, W);
    }
    if (Rp != R || wdt.scalar_type() != dt) {
      Wdt = empty({W, Rp}, dt, xzs);
      conv.add(ptr(wdt), wdt.scalar_type(), ptr(Wdt), dt, W, Rp, R, R, Rp);
    }
    auto f32_param = [&](const Tensor& t) {
      const Tensor p = param(t);
      return (!p.defined() || p.scalar_type() == at::kFloat) ? p.detach() : conv.cast(p, at::kFloat);
    };
    cw = f32_param(conv_w).view({W, K});
    cb = conv_b.defined() ? f32_param(conv_b) : Tensor();
    a.D = f32_param(D);
    a.bias = f32_param(dt_b);
    conv.run();
    a.z = xzs.narrow(2, W, W);
    a.x = empty({B, L, W}, dt, xzs);
    conv_forward(xzs.narrow(2, 0, W), cw, cb, a.x, reverse);
    const Tensor dbc2 = at::mm(a.x.view({T, W}), Wx.t());
    a.delta = at::mm(dbc2.narrow(1, 0, Rp), Wdt.t()).view({B, L, W});       // bias and softplus happen in the kernel
    dbc = dbc2.view({B, L, cols});
    a.B = dbc.narrow(2, Rp, N);
    a.C = dbc.narrow(2, Rp + N, N);
    a.reverse = reverse;
    S = reverse ? 1 : cuttable(a, pick_pieces(B, L, W, grad), grad, false);
    if (!scan_forward(a, S, false, grad, o)) {
      TORCH_CHECK(!reverse, "mamba_b200: these tensors cannot be scanned in reverse");
      S = 1;
      scan_forward(a, 1, false, grad, o);
    }
  }
  if (grad) {
    auto node = new_node<InnerBackward>();
    const Tensor* in[kParams] = {&xz, &conv_w, &conv_b, &xproj_w, &dt_w, &dt_b, &A_log, &D};
    for (int i = 0; i < kParams; ++i) node->types[i] = type_of(*in[i]);
    node->set_next_edges(torch::autograd::collect_next_edges(xz, conv_w, conv_b, xproj_w, dt_w, dt_b, A_log, D));
    node->xz.save(xzs); node->xc.save(a.x); node->dbc.save(dbc); node->delta.save(a.delta); node->A.save(a.A); node->D.save(a.D);
    node->bias.save(a.bias); node->carries.save(o.carries); node->P.save(o.P); node->cw.save(cw); node->cb.save(cb); node->Wx.save(Wx);
    node->Wdt.save(Wdt);
    node->R = R; node->Rp = Rp; node->N = N; node->S = S; node->reverse = reverse;
    node->cw_shape = conv_w.sizes().vec();
    torch::autograd::set_history(o.y, node);
  }
  return o.y;
}

// Whether `inner` can scan in reverse: the kernels' reverse direction exists for d_state 16 and activations on the 16-byte grid.
bool inner_reversible(const Tensor& xz, int64_t N) {
  return N == 16 && xz.is_cuda() && convertible(xz.scalar_type()) && xz.is_contiguous() &&
         reinterpret_cast<uintptr_t>(xz.data_ptr()) % 16 == 0 && xz.size(2) / 2 * xz.element_size() % 16 == 0;
}

}  // namespace mb200_host

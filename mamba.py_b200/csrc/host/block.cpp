// A Mamba block -- projections, and one or both directions between them -- as ONE autograd node.
//
// Written as separate nodes, autograd glues a block's backward together with copies: a `cat` of the gradients of the two halves
// of xz (the whole (B, L, 2 ED) tensor again), a `cat` for the split of the x_proj output, an add of the two gradients that
// reach the conv output, casts of every parameter and of its gradient.  Here the backward writes dz and the conv's dx straight
// into the two halves of d(xz), dB and dC straight into d(x_proj output), adds the second gradient of the conv output in the
// epilogue of the GEMM that produces it, and prepares all parameters (and finishes all their gradients) in one launch.  For a
// small model the launches and the host work around them are all that counts: 57 launches and 1660 us of host time for a
// training step of two 64-wide layers with one node per operation.
#include "scan.h"

namespace mb200_host {
namespace {

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

enum { kConvW, kConvB, kXproj, kDtW, kDtB, kALog, kD, kDirParams };

int64_t padded_rank(int64_t R, at::ScalarType dt) {
  // dt_rank rounded up to a multiple of 16 bytes: the dt, B and C columns of the x_proj output and the K of the dt_proj GEMM
  // then sit on the grid that TMA and the tensor-core GEMMs want; the extra weights are zero
  const int64_t v = dt == at::kFloat ? 4 : 8;
  return (R + v - 1) / v * v;
}

// One direction of a block between the projections (mambapy/mamba.py:214-231): conv1d + SiLU, x_proj, dt_proj and the fused
// scan with softplus(delta + bias) and the gate inside.  With `reverse`, the second direction of the bidirectional block
// (mambapy/vim.py:228-261): the convolution and the scan walk the sequence from its end, everything else is per timestep.
struct Direction {
  bool reverse = false;
  int64_t S = 1;
  Tensor xc, dbc, delta, carries, P;                        // what the forward leaves for the backward
  Tensor A, D, bias, cw, cb, Wx, Wdt;                       // the parameters as the kernels take them
  Tensor y;

  // Queues the parameters' conversions, the projections' into the given places if there are any.
  void prepare(Convert& conv, const Tensor* p, at::ScalarType dt, int64_t W, int64_t R, int64_t N, const Tensor& wx_at, const Tensor& wdt_at) {
    const int64_t Rp = padded_rank(R, dt), K = p[kConvW].size(-1);
    const Tensor wx = param(p[kXproj]), wdt = param(p[kDtW]), alog = param(p[kALog]);
    keep = {wx, wdt, alog};
    A = empty({W, N}, at::kFloat, wx);
    conv.add(ptr(alog), alog.scalar_type(), ptr(A), at::kFloat, 1, W * N, W * N, W * N, W * N, MB200_CONVERT_NEG_EXP);
    if (Rp != R || wx_at.defined()) {
      Wx = wx_at.defined() ? wx_at : empty({Rp + 2 * N, W}, dt, wx);
      char* d = static_cast<char*>(ptr(Wx));
      const int64_t es = Wx.element_size();
      conv.add(ptr(wx), wx.scalar_type(), d, dt, 1, R * W, R * W, R * W, R * W);
      conv.add(nullptr, dt, d + R * W * es, dt, 1, (Rp - R) * W, 0, 0, 0);
      conv.add(static_cast<char*>(ptr(wx)) + R * W * wx.element_size(), wx.scalar_type(), d + Rp * W * es, dt, 1, 2 * N * W, 2 * N * W, 2 * N * W,
               2 * N * W);
      Wdt = wdt_at.defined() ? wdt_at : empty({W, Rp}, dt, wx);
      conv.add(ptr(wdt), wdt.scalar_type(), ptr(Wdt), dt, W, Rp, R, R, Rp);
    } else {
      Wx = conv.cast(wx, dt);
      Wdt = conv.cast(wdt, dt);
    }
    auto f32_param = [&](const Tensor& t) {
      if (!t.defined()) return Tensor();
      keep.push_back(param(t));
      return conv.cast(keep.back(), at::kFloat);
    };
    cw = alias(f32_param(p[kConvW]), 0, {W, K});
    cb = f32_param(p[kConvB]);
    D = f32_param(p[kD]);
    bias = f32_param(p[kDtB]);
  }

  void release() { keep.clear(); }                          // once the conversions have been launched
  // The scan of xc, delta and dbc (B, L, Rp + 2 N), which the projections have filled.
  void scan(const Tensor& xz, int64_t Rp, int64_t N, bool grad) {
    const int64_t B = xz.size(0), L = xz.size(1), W = xz.size(2) / 2;
    ScanArgs a{xc, delta, A, columns(dbc, Rp, N), columns(dbc, Rp + N, N), D, columns(xz, W, W), bias, Tensor(), reverse};
    S = reverse ? 1 : cuttable(a, pick_pieces(B, L, W, grad), grad, false);
    ScanOut o;
    if (!scan_forward(a, S, false, grad, o)) {
      TORCH_CHECK(!reverse, "mamba_b200: these tensors cannot be scanned in reverse");
      S = 1;
      scan_forward(a, 1, false, grad, o);
    }
    y = o.y;
    carries = o.carries;
    P = o.P;
  }

  ScanGrads scan_back(const Tensor& xz, Tensor dy, const ScanSinks& to, int64_t Rp, int64_t N) const {
    const int64_t W = xc.size(2);
    if ((reverse || S > 1) && !tensor_map_ok(dy)) dy = dy.contiguous();
    const ScanArgs a{xc, delta, A, columns(dbc, Rp, N), columns(dbc, Rp + N, N), D, columns(xz, W, W), bias, Tensor(), reverse};
    return scan_backward(a, S, dy, carries, P, false, to);
  }

  // The convolution's backward into dxz (B, L, 2 W); the parameters' gradients into out[kDirParams], of types kt, by way of the jobs
  // queued in `finish`, whose sources stay alive in `alive`.
  void finish_back(const Tensor& xz, const ScanGrads& g, const Partials& dWx, const Partials& dWdt, const Tensor& dxz, int64_t R, int64_t N,
                   const at::ScalarType* kt, const std::vector<int64_t>& cw_shape, Tensor* out, Convert& finish, std::vector<Tensor>& alive) const {
    const int64_t W = xc.size(2), Rp = padded_rank(R, xc.scalar_type()), K = cw.size(1);
    float *dcw = fptr(g.extra), *dcb = dcw + W * K;
    conv_backward(columns(xz, 0, W), cw, cb, g.dx, columns(dxz, 0, W), dcw, cb.defined() ? dcb : nullptr, reverse);

    auto dense = [&](int i, const Tensor& src, int64_t offset, at::IntArrayRef shape) {
      if (kt[i] == at::kFloat) {
        out[i] = alias(src, offset, shape);
        return;
      }
      out[i] = empty(shape, kt[i], xz);
      const int64_t n = out[i].numel();
      finish.add(fptr(src) + offset, at::kFloat, ptr(out[i]), kt[i], 1, n, n, n, n);
    };
    dense(kConvW, g.extra, 0, cw_shape);
    if (cb.defined()) dense(kConvB, g.extra, W * K, {W});
    dense(kDtB, g.dbias, 0, {W});
    dense(kD, g.dD, 0, {W});
    out[kALog] = empty({W, N}, kt[kALog], xz);                               // d A_log = dA * A
    finish.add(ptr(g.dA), at::kFloat, ptr(out[kALog]), kt[kALog], 1, W * N, W * N, W * N, W * N, MB200_CONVERT_MUL).factor = fptr(A);
    if (Rp == R) {
      out[kXproj] = finish.settle(dWx, kt[kXproj]);
      out[kDtW] = finish.settle(dWdt, kt[kDtW]);
    } else {
      out[kXproj] = empty({R + 2 * N, W}, kt[kXproj], xz);
      char* wx = static_cast<char*>(ptr(out[kXproj]));
      finish.rows_of(dWx, 0, R, wx, kt[kXproj]);
      finish.rows_of(dWx, Rp, 2 * N, wx + R * W * out[kXproj].element_size(), kt[kXproj]);
      out[kDtW] = empty({W, R}, kt[kDtW], xz);
      mb200_convert_job& j = finish.add(ptr(dWdt.t), dWdt.t.scalar_type(), ptr(out[kDtW]), kt[kDtW], W, R, R, Rp, R);
      j.slices = dWdt.slices;
      j.slice_stride = W * Rp;
    }
    alive.insert(alive.end(), {dWx.t, dWdt.t, g.dA, g.extra});
  }

 private:
  std::vector<Tensor> keep;                                 // sources of the queued conversions
};

// Both directions go through every projection together: their operands lie one behind the other in one tensor each, and two products
// of one shape are one launch.  Whatever walks from one direction to the next does so inside these tensors, which the backward keeps
// whole: two tensors saved apart need not come back side by side (saved-tensor hooks hand out copies).
struct Joint {
  Tensor xc, delta, dbc;                                    // (n, B * L, W), (n, B * L, W), (n, B * L, cols)
  Tensor Wx, Wdt;                                           // (n, cols, W), (n, W, Rp), without the n for one direction

  // A direction's part of the activations.
  void share(Direction& d, int64_t i, int64_t B, int64_t L) const {
    const int64_t T = B * L, W = xc.size(2), cols = dbc.size(2);
    d.xc = alias(xc, i * T * W, {B, L, W});
    d.delta = alias(delta, i * T * W, {B, L, W});
    d.dbc = alias(dbc, i * T * cols, {B, L, cols});
  }
};

void directions_forward(std::vector<Direction>& dirs, Joint& j, const Tensor& xz, int64_t R, int64_t N, bool grad) {
  const auto dt = xz.scalar_type();
  const int64_t n = int64_t(dirs.size()), B = xz.size(0), L = xz.size(1), W = xz.size(2) / 2, T = B * L, Rp = padded_rank(R, dt), cols = Rp + 2 * N;
  j.xc = empty({n, T, W}, dt, xz);
  j.delta = empty({n, T, W}, dt, xz);
  j.dbc = empty({n, T, cols}, dt, xz);
  for (int64_t i = 0; i < n; ++i) {
    Direction& d = dirs[i];
    j.share(d, i, B, L);
    conv_forward(columns(xz, 0, W), d.cw, d.cb, d.xc, d.reverse);
  }
  const Tensor xc0 = alias(j.xc, 0, {T, W}), dbc0 = alias(j.dbc, 0, {T, cols});
  Products mm;
  mm.each(n, dbc0, T * cols, xc0, T * W, transposed(alias(j.Wx, 0, {cols, W})), cols * W, 1.f, 0.f);
  mm.run();
  mm.each(n, alias(j.delta, 0, {T, W}), T * W, columns(dbc0, 0, Rp), T * cols, transposed(alias(j.Wdt, 0, {W, Rp})), W * Rp, 1.f, 0.f);
  mm.run();                                                                  // bias and softplus happen in the kernel
  for (Direction& d : dirs) d.scan(xz, Rp, N, grad);
}

// d(xz) of direction i into dxz[i]; out and kt hold kDirParams entries per direction.
void directions_backward(const std::vector<Direction>& dirs, const Joint& j, const Tensor& xz, const Tensor& dy, const std::vector<Tensor>& dxz, int64_t R, int64_t N,
                         const at::ScalarType* kt, const std::vector<std::vector<int64_t>>& cw_shape, Tensor* out, Convert& finish,
                         std::vector<Tensor>& alive) {
  const auto dt = xz.scalar_type();
  const int64_t n = int64_t(dirs.size()), B = xz.size(0), L = xz.size(1), W = xz.size(2) / 2, T = B * L, Rp = padded_rank(R, dt), cols = Rp + 2 * N;
  const Tensor dx = empty({n, T, W}, dt, xz), dd = empty({n, T, W}, dt, xz), d_dbc = empty({n, T, cols}, dt, xz);
  std::vector<ScanGrads> g;
  Convert acc;
  for (int64_t i = 0; i < n; ++i) {
    const ScanSinks to{columns(dxz[i], W, W), alias(dx, i * T * W, {B, L, W}), alias(dd, i * T * W, {B, L, W}), W * dirs[i].cw.size(1) + W};
    g.push_back(dirs[i].scan_back(xz, dy, to, Rp, N));
    char* row = static_cast<char*>(d_dbc.data_ptr()) + i * T * cols * d_dbc.element_size();
    acc.add(ptr(g[i].dB), at::kFloat, row + Rp * d_dbc.element_size(), dt, T, N, N, N, cols);   // float32 accumulators -> activation dtype
    acc.add(ptr(g[i].dC), at::kFloat, row + (Rp + N) * d_dbc.element_size(), dt, T, N, N, N, cols);
  }
  acc.run();
  const Tensor d0 = alias(d_dbc, 0, {T, cols}), dd0 = alias(dd, 0, {T, W}), dx0 = alias(dx, 0, {T, W}), xc0 = alias(j.xc, 0, {T, W}),
               dbc0 = alias(j.dbc, 0, {T, cols}), Wx0 = alias(j.Wx, 0, {cols, W}), Wdt0 = alias(j.Wdt, 0, {W, Rp});
  Products mm;
  mm.each(n, columns(d0, 0, Rp), T * cols, dd0, T * W, Wdt0, W * Rp, 1.f, 0.f);          // through dt_proj
  const auto dWdt = mm.tall(n, dd0, T * W, columns(dbc0, 0, Rp), T * cols, kt[kDtW], 1.f);      // (W, Rp)
  mm.run();
  const auto dWx = mm.tall(n, d0, T * cols, xc0, T * W, kt[kXproj], 1.f);                       // (Rp + 2 N, W)
  mm.each(n, dx0, T * W, d0, T * cols, Wx0, cols * W, 1.f, 1.f);      // + the gradient through x_proj, in the GEMM's epilogue
  mm.run();
  for (int64_t i = 0; i < n; ++i)
    dirs[i].finish_back(xz, g[i], dWx[i], dWdt[i], dxz[i], R, N, kt + i * kDirParams, cw_shape[i], out + i * kDirParams, finish, alive);
}

enum { kX, kInW, kOutW, kBlockInputs };                     // then kDirParams per direction

struct BlockBackward : public torch::autograd::Node {
  struct SavedDirection {
    Saved carries, P, A, D, bias, cw, cb;
    bool reverse;
    int64_t S;
    std::vector<int64_t> cw_shape;
    template <typename F> void each(F f) {
      for (Saved* s : {&carries, &P, &A, &D, &bias, &cw, &cb}) f(*s);
    }
    void save(const Direction& d) {
      carries.save(d.carries); P.save(d.P); A.save(d.A); D.save(d.D); bias.save(d.bias); cw.save(d.cw); cb.save(d.cb);
      reverse = d.reverse; S = d.S;
    }
    Direction get() const {
      Direction d;
      d.reverse = reverse; d.S = S;
      d.carries = carries.get(); d.P = P.get(); d.A = A.get(); d.D = D.get(); d.bias = bias.get(); d.cw = cw.get(); d.cb = cb.get();
      return d;
    }
  };
  Saved x, in_w, out_w, xz, y, xc, delta, dbc, Wx, Wdt;
  std::vector<SavedDirection> dirs;
  std::vector<at::ScalarType> types;
  std::vector<int64_t> x_shape;
  int64_t R = 0, N = 0;
  float scale = 1.f;

  std::string name() const override { return "MambaBlockBackward"; }
  void release_variables() override {
    for (Saved* s : {&x, &in_w, &out_w, &xz, &y, &xc, &delta, &dbc, &Wx, &Wdt}) s->reset();
    for (auto& d : dirs) d.each([](Saved& s) { s.reset(); });
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(types.size());
    if (!grads[0].defined()) return out;
    const BelowAutograd guard_ad;
    const NoAutocast no_autocast(c10::DispatchKey::AutocastCUDA);
    const Tensor xz_ = xz.get();
    const c10::cuda::CUDAGuard guard(xz_.device());
    const auto dt = xz_.scalar_type();
    const int64_t B = xz_.size(0), L = xz_.size(1), W = xz_.size(2) / 2, T = B * L;
    std::vector<at::ScalarType> kt;                                        // what the conversion writes; anything else is cast after it
    for (auto t : types) kt.push_back(convertible(t) ? t : at::kFloat);
    Convert finish;
    Products mm;
    std::vector<Tensor> alive;
    Tensor dy = rows(grads[0], dt);
    if (out_w.defined) {
      const Tensor w = out_w.get(), s2 = alias(y.get().contiguous(), 0, {T, W}), d2 = dy.reshape({T, w.size(0)});
      const Tensor ds = empty({T, W}, dt, xz_);
      mm.into(ds, d2, w, scale, 0.f);
      dy = alias(ds, 0, {B, L, W});
      if (task_should_compute_output(kOutW)) {
        const Partials dw = mm.tall(d2, s2, kt[kOutW], scale);
        out[kOutW] = finish.settle(dw, kt[kOutW]);
        alive.push_back(dw.t);
      }
      mm.run();
    }
    std::vector<Direction> ds;
    std::vector<Tensor> each;
    std::vector<std::vector<int64_t>> cw_shape;
    const Joint joint{xc.get().contiguous(), delta.get().contiguous(), dbc.get().contiguous(), Wx.get().contiguous(), Wdt.get().contiguous()};
    for (const SavedDirection& d : dirs) {
      ds.push_back(d.get());
      joint.share(ds.back(), int64_t(ds.size()) - 1, B, L);
      each.push_back(empty({B, L, 2 * W}, dt, xz_));
      cw_shape.push_back(d.cw_shape);
    }
    directions_backward(ds, joint, xz_, dy, each, R, N, kt.data() + kBlockInputs, cw_shape, out.data() + kBlockInputs, finish, alive);
    const Tensor dxz = each[0];
    if (each.size() > 1) dxz.add_(each[1]);
    if (in_w.defined) {
      const Tensor w = in_w.get(), x2 = x.get(), d2 = alias(dxz, 0, {T, 2 * W});
      if (task_should_compute_output(kInW)) {
        const Partials dw = mm.tall(d2, x2, kt[kInW], 1.f);
        out[kInW] = finish.settle(dw, kt[kInW]);
        alive.push_back(dw.t);
      }
      if (task_should_compute_output(kX)) {
        alive.push_back(alias(mm.of(d2, w), 0, x_shape));
        out[kX] = finish.cast(alive.back(), kt[kX]);
      }
    } else {
      out[kX] = dxz;
    }
    mm.run();
    finish.run();
    for (size_t i = 0; i < out.size(); ++i)
      if (out[i].defined()) out[i] = like(out[i], types[i]);
    return out;
  }
};

}  // namespace

// x: the block's input (B, L, d_model), or with in_w undefined its xz (B, L, 2 W).  params: conv weight, conv bias, x_proj weight,
// dt_proj weight and bias, A_log, D of one direction or of both.  Returns out_proj of the (summed, with `halve` averaged) scans, or
// with out_w undefined the scan itself.
Tensor block(const Tensor& x, const OptTensor& in_w_, const OptTensor& out_w_, const std::vector<OptTensor>& params, int64_t R, int64_t N,
             bool halve) {
  const Tensor &in_w = value(in_w_), &out_w = value(out_w_);
  TORCH_CHECK_VALUE(params.size() == kDirParams || params.size() == 2 * kDirParams, "a block has 7 parameters per direction");
  std::vector<Tensor> in{x, in_w, out_w};
  for (const auto& p : params) in.push_back(value(p));
  bool grad = false;
  for (const Tensor& t : in) {
    require_cuda(t);
    refuse_tangents(t);
    grad = grad || wants_grad(t);
  }
  const c10::cuda::CUDAGuard guard(x.device());
  const size_t nd = params.size() / kDirParams;
  const int64_t width = in[kBlockInputs + kDtW].defined() && in[kBlockInputs + kDtW].dim() == 2 ? in[kBlockInputs + kDtW].size(0) : -1;
  TORCH_CHECK(x.dim() == 3, "mamba_b200: a block takes (B, L, width) activations, got ", x.sizes());
  if (in_w.defined()) shape_is(in_w, {2 * width, x.size(2)}, "in_proj.weight");
  else shape_is(x, {x.size(0), x.size(1), 2 * width}, "the in_proj output");
  if (out_w.defined()) TORCH_CHECK(out_w.dim() == 2 && out_w.size(1) == width, "mamba_b200: out_proj.weight should take ", width, " features, got ", out_w.sizes());
  for (size_t i = 0; i < nd; ++i) {
    const Tensor* p = in.data() + kBlockInputs + i * kDirParams;
    for (int k : {kConvW, kXproj, kDtW, kDtB, kALog, kD}) TORCH_CHECK(p[k].defined(), "mamba_b200: a block needs every parameter but the conv bias");
    numel_is(p[kConvW], width * p[kConvW].size(-1), "conv1d.weight");
    numel_is(p[kConvB], width, "conv1d.bias");
    shape_is(p[kXproj], {R + 2 * N, width}, "x_proj.weight");
    shape_is(p[kDtW], {width, R}, "dt_proj.weight");
    numel_is(p[kDtB], width, "dt_proj.bias");
    shape_is(p[kALog], {width, N}, "A_log");
    numel_is(p[kD], width, "D");
  }
  std::vector<Direction> dirs(nd);
  Joint joint;
  Tensor x2, wi, wo, xz, s, out;
  const float scale = halve ? 0.5f : 1.f;
  {
    const auto dt = in_w.defined() && at::autocast::is_autocast_enabled(at::kCUDA) ? at::autocast::get_autocast_dtype(at::kCUDA) : x.scalar_type();
    TORCH_CHECK_TYPE(convertible(dt), "mamba_b200 kernels take float32 or bfloat16 activations, got ", dt);
    const BelowAutograd guard_ad;
    const NoAutocast no_autocast(c10::DispatchKey::AutocastCUDA);
    const int64_t B = x.size(0), L = x.size(1), T = B * L, W = in[kBlockInputs + kDtW].size(0);
    Convert conv;
    const Tensor pi = param(in_w), po = param(out_w), px = rows(x, x.scalar_type());
    Tensor xr;                                                               // stays alive until the conversions have been launched
    if (pi.defined()) {
      xr = px.reshape({T, px.size(2)});
      x2 = xr.is_contiguous() && convertible(xr.scalar_type()) ? conv.cast(xr, dt) : xr.to(dt);
      wi = conv.cast(pi, dt);
    } else {
      xz = rows(px, dt);
      if (nd > 1 && !tensor_map_ok(xz)) xz = xz.contiguous();
    }
    wo = conv.cast(po, dt);
    const int64_t Rp = padded_rank(R, dt), cols = Rp + 2 * N;
    if (nd > 1) {
      joint.Wx = empty({int64_t(nd), cols, W}, dt, x);
      joint.Wdt = empty({int64_t(nd), W, Rp}, dt, x);
    }
    for (size_t i = 0; i < nd; ++i) {
      dirs[i].reverse = i == 1;
      dirs[i].prepare(conv, in.data() + kBlockInputs + i * kDirParams, dt, W, R, N, nd > 1 ? alias(joint.Wx, i * cols * W, {cols, W}) : Tensor(),
                      nd > 1 ? alias(joint.Wdt, i * W * Rp, {W, Rp}) : Tensor());
    }
    if (nd == 1) {
      joint.Wx = dirs[0].Wx;
      joint.Wdt = dirs[0].Wdt;
    }
    conv.run();
    Products mm;
    if (wi.defined()) xz = alias(mm.of(x2, transposed(wi)), 0, {B, L, 2 * W});
    mm.run();
    for (auto& d : dirs) d.release();
    directions_forward(dirs, joint, xz, R, N, grad);
    s = nd == 1 ? dirs[0].y : dirs[0].y + dirs[1].y;
    if (wo.defined()) {
      const Tensor o = empty({T, wo.size(0)}, dt, xz);
      mm.into(o, alias(s, 0, {T, W}), transposed(wo), scale, 0.f);
      mm.run();
      out = alias(o, 0, {B, L, wo.size(0)});
    } else {
      out = s;
    }
  }
  if (grad) {
    auto node = new_node<BlockBackward>();
    torch::autograd::edge_list edges;
    for (const Tensor& t : in) {
      node->types.push_back(type_of(t));
      edges.push_back(t.defined() && t.requires_grad() ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge());
    }
    node->set_next_edges(std::move(edges));
    if (wi.defined()) { node->x.save(x2); node->in_w.save(wi); }
    if (wo.defined()) { node->out_w.save(wo); node->y.save(s); }
    node->xz.save(xz);
    node->xc.save(joint.xc); node->delta.save(joint.delta); node->dbc.save(joint.dbc); node->Wx.save(joint.Wx); node->Wdt.save(joint.Wdt);
    node->dirs.resize(nd);
    for (size_t i = 0; i < nd; ++i) {
      node->dirs[i].save(dirs[i]);
      node->dirs[i].cw_shape = in[kBlockInputs + i * kDirParams + kConvW].sizes().vec();
    }
    node->x_shape = x.sizes().vec();
    node->R = R; node->N = N; node->scale = scale;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// Whether a direction can run in reverse on these activations: the kernels' reverse exists for d_state 16 on the 16-byte grid.
bool reversible(int64_t W, int64_t N, at::ScalarType dt) { return N == 16 && convertible(dt) && W * (dt == at::kFloat ? 4 : 2) % 16 == 0; }

}  // namespace mb200_host

// selective_scan_fn and pscan: forward launches and their autograd nodes.
#include "scan.h"
#include <cmath>
#include <cstdlib>

namespace mb200_host {

void check_status(const char* what) {
  static const bool on = [] {
    const char* v = std::getenv("MB200_CHECK_STATUS");
    return v && *v && std::string(v) != "0";
  }();
  if (!on) return;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing(at::cuda::getCurrentCUDAStream(), &capturing));
  if (capturing != cudaStreamCaptureStatusNone) return;
  const int s = mb200_device_status();
  TORCH_CHECK(s == 0, what, ": a bounded wait inside the kernel gave up (device status ", s, "); its outputs are invalid");
}

namespace {

// What enters the pieces of a cut sequence (a.h0, the gradient carries) has one entry a piece.
int launch_forward(const ScanArgs& a, ScanOut& o, bool want_last, bool want_carries, int64_t pieces = 1, int64_t piece_len = 0) {
  const int64_t B = a.batch(), L = a.length(), W = a.width(), N = a.states(), chunk = mb200_sscan_chunk();
  o.y = empty({B, L, W}, a.x.scalar_type(), a.x);
  if (want_last) o.hT = empty({B, W, N}, at::kFloat, a.x);
  if (want_carries) o.carries = empty({B, (L + chunk - 1) / chunk, W, N}, at::kFloat, a.x);
  const int rc = mb200_sscan_fwd_pieces(ptr(a.x), ptr(a.delta), ptr(a.z), fptr(a.A), ptr(a.B), ptr(a.C), fptr(a.D), fptr(a.bias), fptr(a.h0),
                                 ptr(o.y), fptr(o.hT), fptr(o.carries), B, L, W, int(N), st(a.x, 0), st(a.x, 1), st(a.delta, 0),
                                 st(a.delta, 1), st(a.z, 0), st(a.z, 1), st(a.B, 0), st(a.B, 1), st(a.C, 0), st(a.C, 1), st(o.y, 0),
                                 st(o.y, 1), a.code(), a.flags(), pieces, piece_len, cuda_stream());
  if (rc != MB200_EUNSUPPORTED) {
    check(rc, "mb200_sscan_fwd");
    check_status("mb200_sscan_fwd");
  }
  return rc;
}

int64_t piece_length(int64_t L, int64_t S) { return (L + 16 * S - 1) / (16 * S) * 16; }

// Rows cut into S pieces: carry pass, fold, full pass (the protocol of split.py).  False when these tensors cannot be cut.
bool split_forward(const ScanArgs& a, int64_t S, bool want_last, bool want_carries, ScanOut& o) {
  const int64_t B = a.batch(), L = a.length(), W = a.width(), N = a.states(), len = piece_length(L, S);
  const Tensor PS = empty({2, B, S, W, N}, at::kFloat, a.x);
  float *P = fptr(PS), *St = P + B * S * W * N;
  const int rc = mb200_sscan_fwd_carry_pieces(ptr(a.x), ptr(a.delta), fptr(a.A), ptr(a.B), fptr(a.bias), St, P, B, L, W, int(N), st(a.x, 0),
                                              st(a.x, 1), st(a.delta, 0), st(a.delta, 1), st(a.B, 0), st(a.B, 1), a.code(), a.flags(), S, len,
                                              cuda_stream());
  if (rc == MB200_EUNSUPPORTED) return false;
  check(rc, "mb200_sscan_fwd_carry");
  check_status("mb200_sscan_fwd_carry");
  ScanArgs s = a;
  s.h0 = empty({B, S, W, N}, at::kFloat, a.x);
  check(mb200_carry_fold_range(P, St, fptr(a.h0), fptr(s.h0), B, S, W * N, 0, int(S), 0, cuda_stream()), "mb200_carry_fold_range");
  if (launch_forward(s, o, want_last, want_carries, S, len) == MB200_EUNSUPPORTED) return false;
  o.P = alias(PS, 0, {B, S, W, N});
  return true;
}

ScanGrads launch_backward(const ScanArgs& a, const Tensor& dy, const Tensor& carries, const Tensor& g_in, bool want_g_out, const ScanSinks& to,
                          int64_t pieces = 1, int64_t piece_len = 0) {
  const int64_t B = a.batch(), L = a.length(), W = a.width(), N = a.states();
  ScanGrads g;
  const auto dt = a.x.scalar_type();
  auto sink = [&](const Tensor& t) { return t.defined() ? t : empty({B, L, W}, dt, a.x); };
  const int64_t extra = to.extra;
  g.dx = sink(to.dx);
  g.dd = sink(to.dd);
  if (a.z.defined()) g.dz = sink(to.dz);
  // every buffer the kernel accumulates into comes out of ONE zero-filled allocation
  const int64_t nBC = B * L * N, nA = W * N;
  const Tensor acc = empty({2 * nBC + nA + 2 * W + extra}, at::kFloat, a.x);
  zero_fill(acc);
  g.dB = alias(acc, 0, {B, L, N});
  g.dC = alias(acc, nBC, {B, L, N});
  g.dA = alias(acc, 2 * nBC, {W, N});
  g.dD = alias(acc, 2 * nBC + nA, {W});
  if (a.bias.defined()) g.dbias = alias(acc, 2 * nBC + nA + W, {W});
  if (extra) g.extra = alias(acc, 2 * nBC + nA + 2 * W, {extra});
  if (want_g_out) g.g_out = empty({B, W, N}, at::kFloat, a.x);
  check(mb200_sscan_bwd_pieces(ptr(a.x), ptr(a.delta), ptr(a.z), fptr(a.A), ptr(a.B), ptr(a.C), fptr(a.D), fptr(a.bias), ptr(dy), fptr(carries),
                        fptr(g_in), ptr(g.dx), ptr(g.dd), ptr(g.dz), fptr(g.dB), fptr(g.dC), fptr(g.dA), fptr(g.dD), fptr(g.dbias),
                        fptr(g.g_out), B, L, W, int(N), st(a.x, 0), st(a.x, 1), st(a.delta, 0), st(a.delta, 1), st(a.z, 0), st(a.z, 1),
                        st(a.B, 0), st(a.B, 1), st(a.C, 0), st(a.C, 1), st(dy, 0), st(dy, 1), st(g.dx, 0), st(g.dx, 1), st(g.dd, 0),
                        st(g.dd, 1), st(g.dz, 0), st(g.dz, 1), a.code(), a.flags(), pieces, piece_len, cuda_stream()),
        "mb200_sscan_bwd");
  check_status("mb200_sscan_bwd");
  return g;
}

ScanGrads split_backward(const ScanArgs& a, int64_t S, const Tensor& dy, const Tensor& carries, const Tensor& P, bool want_g_out,
                         const ScanSinks& to) {
  const int64_t B = a.batch(), L = a.length(), W = a.width(), N = a.states(), len = piece_length(L, S);
  const Tensor G = empty({B, S, W, N}, at::kFloat, a.x), g_in = empty({B, S, W, N}, at::kFloat, a.x);
  check(mb200_sscan_bwd_carry_pieces(ptr(a.delta), ptr(a.z), ptr(dy), ptr(a.C), fptr(a.A), fptr(a.bias), fptr(G), B, L, W, int(N),
                                     st(a.delta, 0), st(a.delta, 1), st(a.z, 0), st(a.z, 1), st(dy, 0), st(dy, 1), st(a.C, 0), st(a.C, 1),
                                     a.code(), a.flags(), S, len, cuda_stream()),
        "mb200_sscan_bwd_carry");
  check_status("mb200_sscan_bwd_carry");
  check(mb200_carry_fold_range(fptr(P), fptr(G), nullptr, fptr(g_in), B, S, W * N, 0, int(S), 1, cuda_stream()), "mb200_carry_fold_range");
  return launch_backward(a, dy, carries, g_in, want_g_out, to, S, len);
}

}  // namespace

bool tensor_map_ok(const Tensor& t) {
  const int64_t es = t.element_size();
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && t.stride(0) * es % 16 == 0 && t.stride(1) * es % 16 == 0;
}
bool tensor_maps_ok(const ScanArgs& a) {
  for (const Tensor* t : {&a.x, &a.delta, &a.z})
    if (t->defined() && !tensor_map_ok(*t)) return false;
  return a.width() * a.x.element_size() % 16 == 0;
}

int64_t cuttable(const ScanArgs& a, int64_t S, bool grad, bool want_last) {
  if (S == 1 || (tensor_maps_ok(a) && tensor_map_ok(a.B) && tensor_map_ok(a.C) && (!grad || a.states() == 16))) return S;
  if (a.h0.defined() || want_last) return 1;
  int64_t even = 1;
  while (2 * even <= S && a.length() % (32 * even) == 0) even *= 2;
  for (const Tensor* t : {&a.x, &a.delta, &a.z, &a.B, &a.C})
    if (t->defined() && a.batch() > 1 && t->stride(0) != a.length() * t->stride(1)) return 1;
  return even;
}

bool scan_forward(const ScanArgs& a, int64_t S, bool want_last, bool want_carries, ScanOut& o) {
  return S > 1 ? split_forward(a, S, want_last, want_carries, o) : launch_forward(a, o, want_last, want_carries) == MB200_OK;
}
ScanGrads scan_backward(const ScanArgs& a, int64_t S, const Tensor& dy, const Tensor& carries, const Tensor& P, bool want_g_out,
                        const ScanSinks& to) {
  return S > 1 ? split_backward(a, S, dy, carries, P, want_g_out, to) : launch_backward(a, dy, carries, Tensor(), want_g_out, to);
}

namespace {

// B and C are slices of the x_proj output, whose width dt_rank + 2 N often leaves them off the 16-byte grid a tensor map
// needs.  They are 2 N values a token: copying them onto the grid costs a few microseconds and keeps the fused kernels'
// tensor-map path, which is two to three times faster than the path for arbitrary alignment.
void align_bc(ScanArgs& a) {
  if (a.length() == 0 || a.batch() == 0 || !tensor_maps_ok(a) || (tensor_map_ok(a.B) && tensor_map_ok(a.C))) return;
  const int64_t N = a.B.size(2), es = a.B.element_size();
  const bool side_by_side = a.B.strides() == a.C.strides() &&
                            static_cast<char*>(a.C.data_ptr()) - static_cast<char*>(a.B.data_ptr()) == N * es && a.B.stride(1) >= 2 * N;
  if (side_by_side) {                                                   // one copy for both
    const Tensor bc = a.B.as_strided({a.B.size(0), a.B.size(1), 2 * N}, a.B.strides()).contiguous();
    a.B = bc.narrow(2, 0, N);
    a.C = bc.narrow(2, N, N);
  } else {
    a.B = a.B.clone(at::MemoryFormat::Contiguous);
    a.C = a.C.clone(at::MemoryFormat::Contiguous);
  }
}

enum { kX, kDelta, kA, kB, kC, kD, kZ, kBias, kH0, kInputs };

struct ScanBackward : public torch::autograd::Node {
  Saved x, delta, A, B, C, D, z, bias, carries, P;
  at::ScalarType types[kInputs];
  bool given[kInputs];
  bool reverse = false, flipped = false;
  int64_t subshards = 1;

  std::string name() const override { return "SelectiveScanBackward"; }
  void release_variables() override {
    for (Saved* s : {&x, &delta, &A, &B, &C, &D, &z, &bias, &carries, &P}) s->reset();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(kInputs);
    if (!grads[0].defined()) return out;
    const BelowAutograd guard_ad;
    ScanArgs a{x.get(), delta.get(), A.get(), B.get(), C.get(), D.get(), z.get(), bias.get(), Tensor(), reverse};
    const c10::cuda::CUDAGuard guard(a.x.device());
    Tensor dy = rows(flipped ? grads[0].flip(1) : grads[0], a.x.scalar_type());
    // the in-kernel reverse backward and uneven pieces exist on the tensor-map path only; an upstream gradient that is an
    // offset or narrow view of something wider is copied to a dense tensor first
    if ((reverse || subshards > 1) && !tensor_map_ok(dy)) dy = dy.contiguous();
    ScanGrads g = scan_backward(a, subshards, dy, carries.get(), P.get(), given[kH0]);
    if (flipped)
      for (Tensor* t : {&g.dx, &g.dd, &g.dz, &g.dB, &g.dC})
        if (t->defined()) *t = t->flip(1);
    Tensor all[kInputs] = {g.dx, g.dd, g.dA, g.dB, g.dC, g.dD, g.dz, g.dbias, g.g_out};
    Convert conv;                                                      // casts to the inputs' types, all in one launch
    for (int i = 0; i < kInputs; ++i) {
      if (!given[i] || !all[i].defined() || !task_should_compute_output(i)) continue;
      const bool ours = all[i].is_contiguous() && convertible(types[i]) && convertible(all[i].scalar_type());
      out[i] = ours ? conv.cast(all[i], types[i]) : like(all[i], types[i]);
    }
    conv.run();
    return out;
  }
};

}  // namespace

// How many pieces to cut each row into, from a model of the time: the fused kernels have batch * ceil(width / 32) independent
// work items a piece (a CTA owns one, three fit an SM), and one CTA alone on an SM runs much faster than one of three.
// Measured, us for 2048 timesteps with 1 / 2 / 3 CTAs on every SM of 148, means of both types and of A as initialised and as trained:
// forward 82 / 123 / 174 with saved states, 79 / 121 / 170 without (81 / 119 / 169 and 79 / 116 / 164 for A as initialised, 82 / 126 / 179 and
// 80 / 125 / 177 as trained), 112 and 105 with one 48-channel CTA on every SM; backward 279 / 378 / 538; forward carry pass 55 / 87 / 125
// (49 / 78 / 110, 60 / 96 / 140), reverse one 62 / 94 / 135.  Of these, filling the pipeline takes as long as some 10 timesteps.  A carry pass and
// a fold add 4 us of launches on the GPU and 12 of host time, which is what short calls wait for (with 12 for a training step's two of them
// the picks lost 10 to 40 % below 256 steps).  Over 44 cases of 3840 steps (1 to 16 rows 64 to 5120 wide, both types, training and inference) the count picked takes
// 1.9 % longer than the best one on average and 8.8 % at most; where it differs from what the times of earlier kernels picked (2.4 % of
// shapes) it is 0.7 % faster on average, between 17 % faster and 13 % slower.
int64_t pick_pieces(int64_t batch, int64_t length, int64_t width, bool grad) {
  constexpr double kFill = 10, kFwdSaving[] = {0, 82, 123, 174}, kFwd[] = {0, 79, 121, 170}, kBwd[] = {0, 279, 378, 538},
                   kFwdCarry[] = {0, 55, 87, 125}, kBwdCarry[] = {0, 62, 94, 135}, kFwdWide[] = {105, 112};
  const double items = double(batch) * double((width + 31) / 32);
  const double sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  auto passes = [&](double ctas, const double (&t)[4]) {                 // of 2048 timesteps on the longest SM
    const int per_sm = int(std::ceil(ctas / sms)), full = per_sm / 3, rest = per_sm % 3;
    return full * t[3] + t[rest];
  };
  int64_t best = 1;
  double best_us = 0;
  for (int64_t S = 1; S <= 24 && (S == 1 || length / S >= 64); ++S) {
    const double len = double(S == 1 ? length : (length + 16 * S - 1) / (16 * S) * 16);
    if (S > 1 && (S - 1) * len >= length) continue;
    const bool wide = items * S > sms && double(batch) * double((width + 47) / 48) * S <= sms;      // one 48-channel CTA per SM instead
    double all = (wide ? kFwdWide[grad] : passes(items * S, grad ? kFwdSaving : kFwd)) + (grad ? passes(items * S, kBwd) : 0);
    if (S > 1) all += passes(items * (S - 1), kFwdCarry) + (grad ? passes(items * (S - 1), kBwdCarry) : 0);
    const double us = all * (len + kFill) / (2048 + kFill) + (S > 1 ? (grad ? 24 : 12) : 0);
    if (S == 1 || us < best_us) {
      best = S;
      best_us = us;
    }
  }
  return best;
}

py::object selective_scan(const Tensor& x, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D_,
                          const OptTensor& z_, const OptTensor& bias_, const OptTensor& h0_, bool return_last_state, bool reverse,
                          std::optional<int64_t> subshards) {
  const Tensor &D = value(D_), &z = value(z_), &bias = value(bias_), &h0 = value(h0_);
  Tensor y, hT;
  {
    py::gil_scoped_release no_gil;
    require_cuda(x, delta, A, B, C, D, z, bias, h0);
    refuse_tangents(x, delta, A, B, C, D, z, bias, h0);
    const c10::cuda::CUDAGuard guard(x.device());
    const auto dt = act_dtype(x, delta, z, B, C);
    const bool grad = wants_grad(x, delta, A, B, C, D, z, bias, h0);
    ScanOut o;
    ScanArgs a;
    bool flipped = false;
    int64_t S;
    {
      const BelowAutograd guard_ad;
      a = ScanArgs{rows(x, dt), rows(delta, dt), f32(A), rows(B, dt), rows(C, dt), f32(D), rows(z, dt), f32(bias), f32(h0), reverse};
      const int64_t L = a.length();
      // Few batch rows: cut every row into S consecutive pieces that run side by side.
      align_bc(a);
      S = subshards.value_or(0) ? *subshards : pick_pieces(a.batch(), L, a.width(), grad);
      if (reverse || S < 1 || (subshards.value_or(0) && L % (16 * S)) || L == 0) S = 1;
      S = cuttable(a, S, grad, return_last_state);
      // the reverse backward exists for d_state 16 on the tensor-map path; otherwise do what the reference does
      // (mambapy/vim.py:228-261): scan the flipped sequence, flip back
      flipped = reverse && grad && a.states() != 16;
      if (!flipped && !scan_forward(a, S, return_last_state, grad, o)) {
        flipped = reverse;
        S = 1;
        if (!reverse) scan_forward(a, 1, return_last_state, grad, o);
      }
      if (flipped) {
        for (Tensor* t : {&a.x, &a.delta, &a.z, &a.B, &a.C})
          if (t->defined()) *t = t->flip(1);
        a.reverse = false;
        scan_forward(a, 1, return_last_state, grad, o);
        o.y = o.y.flip(1);
      }
    }
    y = o.y;
    hT = o.hT;
    if (grad) {
      auto node = new_node<ScanBackward>();
      const Tensor* in[kInputs] = {&x, &delta, &A, &B, &C, &D, &z, &bias, &h0};
      for (int i = 0; i < kInputs; ++i) {
        node->given[i] = in[i]->defined();
        node->types[i] = type_of(*in[i]);
      }
      node->set_next_edges(torch::autograd::collect_next_edges(x, delta, A, B, C, D, z, bias, h0));
      node->x.save(a.x); node->delta.save(a.delta); node->A.save(a.A); node->B.save(a.B); node->C.save(a.C); node->D.save(a.D);
      node->z.save(a.z); node->bias.save(a.bias); node->carries.save(o.carries); node->P.save(o.P);
      node->reverse = a.reverse; node->flipped = flipped; node->subshards = S;
      torch::autograd::set_history(y, node);
    }
  }
  if (return_last_state) return py::make_tuple(y, hT);
  return py::cast(y);
}

// ------------------------------------------------------------------------------------------------------ pscan
namespace {

// (B, L, D, N) tensor whose (D, N) block is dense; copies only if it is not.
Tensor dense_dn(const Tensor& t) {
  return (t.stride(3) == 1 && (t.size(2) == 1 || t.stride(2) == t.size(3))) ? t : t.contiguous();
}
Tensor pscan_workspace(int64_t B, int64_t nseg, int64_t DN, const Tensor& on) {
  return nseg > 1 ? empty({2 * B * nseg * DN}, at::kFloat, on) : Tensor();
}

struct PScanBackward : public torch::autograd::Node {
  Saved A, H;
  std::string name() const override { return "PScanBackward"; }
  void release_variables() override { A.reset(); H.reset(); }
  variable_list apply(variable_list&& grads) override {
    if (!grads[0].defined()) return variable_list(2);
    const BelowAutograd guard_ad;
    const Tensor h0 = H.get(shared_from_this());
    const c10::cuda::CUDAGuard guard(h0.device());
    const Tensor a = dense_dn(A.get()), h = dense_dn(h0), g = dense_dn(like(grads[0], h0.scalar_type()));
    const int64_t B = h.size(0), L = h.size(1), DN = h.size(2) * h.size(3);
    const Tensor gA = empty(h.sizes(), h.scalar_type(), h), gX = empty(h.sizes(), h.scalar_type(), h);
    const int nseg = L > 0 ? mb200_pscan_segments(B, L, DN) : 1;
    const Tensor ws = pscan_workspace(B, nseg, DN, h);
    check(mb200_pscan_bwd(ptr(a), ptr(h), ptr(g), ptr(gA), ptr(gX), B, L, DN, a.stride(0), a.stride(1), h.stride(0), h.stride(1),
                          g.stride(0), g.stride(1), gA.stride(0), gA.stride(1), gX.stride(0), gX.stride(1), nullptr, fptr(ws), nseg,
                          dtype_code(h.scalar_type()), cuda_stream()),
          "mb200_pscan_bwd");
    return {gA, gX};
  }
};

}  // namespace

Tensor pscan(const Tensor& A, const Tensor& X) {
  require_cuda(A, X);
  refuse_tangents(A, X);
  TORCH_CHECK_VALUE(A.dim() == 4 && A.sizes() == X.sizes(), "pscan expects two (B, L, D, N) tensors, got ", A.sizes(), " and ", X.sizes());
  TORCH_CHECK_TYPE(A.scalar_type() == X.scalar_type(), "A_in and X_in must have the same dtype");
  act_dtype(X);
  const c10::cuda::CUDAGuard guard(X.device());
  const int64_t B = X.size(0), L = X.size(1), DN = X.size(2) * X.size(3);
  Tensor H;
  {
    const BelowAutograd guard_ad;
    const Tensor a = dense_dn(A), x = dense_dn(X);
    H = empty(X.sizes(), X.scalar_type(), X);
    const int nseg = L > 0 ? mb200_pscan_segments(B, L, DN) : 1;
    const Tensor ws = pscan_workspace(B, nseg, DN, X);
    check(mb200_pscan_fwd(ptr(a), ptr(x), ptr(H), B, L, DN, a.stride(0), a.stride(1), x.stride(0), x.stride(1), H.stride(0), H.stride(1),
                          nullptr, nullptr, fptr(ws), nseg, dtype_code(X.scalar_type()), cuda_stream()),
          "mb200_pscan_fwd");
  }
  if (wants_grad(A, X)) {
    auto node = new_node<PScanBackward>();
    node->set_next_edges(torch::autograd::collect_next_edges(A, X));
    node->A.save(A);
    torch::autograd::set_history(H, node);
    node->H.save(H, true);
  }
  return H;
}

}  // namespace mb200_host

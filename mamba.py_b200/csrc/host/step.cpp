// Decode steps: the state update, the conv window, and the whole block.
#include <algorithm>
#include <mutex>
#include <unordered_map>
#include "host.h"

namespace mb200_host {
namespace {

bool small_type(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16; }

// A small parameter as the kernels read it: contiguous, float32 or bfloat16 as the model has it.
Tensor small_param(const Tensor& t) {
  if (!t.defined()) return t;
  const Tensor r = small_type(t) ? t : t.to(at::kFloat);
  return r.is_contiguous() ? r : r.contiguous();
}
int code_of(const Tensor& t) { return t.defined() ? dtype_code(t.scalar_type()) : MB200_F32; }

struct StateStep {
  Tensor y, h;
};

StateStep state_step(const Tensor& x, const Tensor& h, const Tensor& delta, const Tensor& A_, bool log_A, const Tensor& B, const Tensor& C,
                     const Tensor& D_, const Tensor& z, const Tensor& bias_, bool inplace) {
  const auto dt = act_dtype(x, delta, z, B, C);
  const Tensor xs = rows(x, dt), ds = rows(delta, dt), zs = rows(z, dt), Bs = rows(B, dt), Cs = rows(C, dt);
  const Tensor A = small_param(A_), D = small_param(D_), bias = small_param(bias_), h32 = f32(h);
  const int64_t n = xs.size(0), W = xs.size(1), N = A.size(1);
  StateStep o;
  if (inplace) {
    TORCH_CHECK_VALUE(h.defined() && h32.data_ptr() == h.data_ptr(), "inplace=True needs a float32 contiguous state tensor");
    o.h = h;
  } else {
    o.h = empty({n, W, N}, at::kFloat, xs);
  }
  o.y = empty({n, W}, dt, xs);
  check(mb200_ssm_step_params(ptr(xs), ptr(ds), ptr(zs), ptr(A), code_of(A), log_A, ptr(Bs), ptr(Cs), ptr(D), code_of(D), ptr(bias),
                              code_of(bias), fptr(h32), fptr(o.h), ptr(o.y), n, W, int(N), st(xs, 0), st(ds, 0), st(zs, 0), st(Bs, 0),
                              st(Cs, 0), st(o.y, 0), dtype_code(dt), bias.defined() ? MB200_DELTA_SOFTPLUS : 0, cuda_stream()),
        "mb200_ssm_step");
  return o;
}

struct WindowStep {
  Tensor xc, window;
};

WindowStep window_step(const Tensor& x, const Tensor& inputs, const Tensor& weight, const Tensor& bias_, bool inplace,
                       const mb200_convert_job* jobs = nullptr, int n_jobs = 0) {
  const auto dt = act_dtype(x);
  const Tensor xs = rows(x, dt), win = inputs.to(dt).contiguous(), w = small_param(weight), bias = small_param(bias_);
  const int64_t n = xs.size(0), W = xs.size(1);
  numel_is(w, W * w.size(-1), "the filter");
  numel_is(bias, W, "the bias");
  TORCH_CHECK(win.numel() >= n * W * (w.size(-1) - 1), "mamba_b200: the window holds fewer than ", n, " rows of ", W, " channels");
  WindowStep o;
  o.xc = empty({n, W}, dt, xs);
  if (inplace) {
    TORCH_CHECK_VALUE(win.data_ptr() == inputs.data_ptr(), "inplace=True needs a contiguous window of the activation dtype");
    o.window = inputs;
  } else {
    o.window = empty(win.sizes(), dt, xs);
  }
  check(mb200_conv_step_convert(ptr(xs), ptr(win), ptr(w), code_of(w), ptr(bias), code_of(bias), ptr(o.xc), ptr(o.window), n, W,
                                int(w.size(-1)), st(xs, 0), dtype_code(dt), jobs, n_jobs, cuda_stream()),
        "mb200_conv_step");
  return o;
}

// ---- barrier counters of the one-launch step -----------------------------------------------------------------------
// A launch leaves its counters fit for the next one on the same stream, so a stream keeps its own.  At most kMaxStreams are
// kept; a stream beyond them, a stream that is being captured into a graph (whose replays may run anywhere), and a stream that
// torch did not make (destroyed, its handle may come back for another stream while its last launch still runs) gets counters of its
// own for the one call, cleared on the stream.  A launch that gave up at a barrier spoils its counters; once
// somebody has read its status word, none from before are used again.
constexpr size_t kMaxStreams = 64;

Tensor barrier_counters(const Tensor& on) {
  static std::mutex mutex;
  static std::unordered_map<uint64_t, Tensor> kept;
  static unsigned give_ups = 0;
  const auto s = at::cuda::getCurrentCUDAStream();
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing(s, &capturing));
  const uint64_t key = (uint64_t(s.device_index()) << 56) ^ uint64_t(s.id());
  std::lock_guard<std::mutex> lock(mutex);
  if (const unsigned now = mb200_block_step_give_ups(); now != give_ups) {
    kept.clear();
    give_ups = now;
  }
  const bool foreign = s.stream() && reinterpret_cast<intptr_t>(s.stream()) == s.id();        // torch's own have numbers for ids
  const bool keep = capturing == cudaStreamCaptureStatusNone && !foreign;
  if (keep) {
    const auto it = kept.find(key);
    if (it != kept.end()) return it->second;
  }
  const Tensor t = at::empty({mb200_block_step_barrier_bytes()}, on.options().dtype(at::kByte));
  C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), s));
  if (keep && kept.size() < kMaxStreams) kept.emplace(key, t);
  return t;
}

}  // namespace

void selftest_block_step_give_up(const Tensor& on) {
  const c10::cuda::CUDAGuard guard(on.device());
  check(mb200_selftest_block_step_give_up(ptr(barrier_counters(on)), cuda_stream()), "mb200_selftest_block_step_give_up");
}

std::tuple<Tensor, Tensor> ssm_step(const Tensor& x, const OptTensor& h, const Tensor& delta, const Tensor& A, const Tensor& B,
                                    const Tensor& C, const OptTensor& D, const OptTensor& z, const OptTensor& bias, bool inplace) {
  require_cuda(x, delta, A, B, C, value(D), value(z), value(bias), value(h));
  const c10::cuda::CUDAGuard guard(x.device());
  const BelowAutograd guard_ad;
  const StateStep o = state_step(x, value(h), delta, A, false, B, C, value(D), value(z), value(bias), inplace);
  return {o.y, o.h};
}

std::tuple<Tensor, Tensor> conv_step(const Tensor& x, const Tensor& inputs, const Tensor& weight, const OptTensor& bias, bool inplace) {
  require_cuda(x, inputs, weight, value(bias));
  const c10::cuda::CUDAGuard guard(x.device());
  const BelowAutograd guard_ad;
  const WindowStep o = window_step(x, inputs, weight, value(bias), inplace);
  return {o.xc, o.window};
}

// Whether so few tokens that the one launch is the better way.  It reads the activations of all tokens from shared memory again for
// every output row, where the library's bfloat16 kernels use the tensor cores; the float32 ones take longer nearly everywhere.  us a
// layer, weights from HBM, called from Python / inside a CUDA graph, one launch : library:
//               256 wide             768 wide             1536 wide            2560 wide
//   float32  1  14/16 : 40/16        21/23 : 42/29        32/31 : 55/39         61/59 : 71/55
//            2  15/16 : 40/22        22/23 : 59/47        38/37 : 105/92        73/72 : 149/139
//            4  15/17 : 40/28        25/27 : 65/54        43/42 : 114/101       90/88 : 131/117
//            8  17/19 : 43/34        33/33 : 81/69        61/59 : 109/92        128/126 : 164/146
//   bfloat16 1  15/17 : 49/19        21/22 : 50/24        28/28 : 52/31         51/50 : 58/44
//            2  16/18 : 49/16        23/25 : 51/24        35/35 : 53/30         67/66 : 58/43
//            4  17/19 : 50/16        31/33 : 51/23        51/50 : 53/30         107/105 : 56/43
//            8  21/22 : 50/19        47/48 : 51/23        84/84 : 52/30         184/183 : 57/44
// One token 4096 wide 106/104 : 113/96 in float32, 77/79 : 86/71 in bfloat16.
// So up to 8 tokens in float32, and in bfloat16 as long as the tokens the kernel is built for (1, 2, 4, 8) times the inner width are
// at most 8192 values.  Beyond that a call from Python still gains a little here and there (4 x 1536 51 : 53, 8 x 768 47 : 51, 8 x 1024 42 : 51),
// but only host time: the GPU is busy for twice as long (8 x 1024 in a graph 43 : 26).
static constexpr int64_t kOneLaunchTokens = 8, kOneLaunchValuesBf16 = 8192;
static bool takes_one_launch(int64_t tokens, int64_t d_model, int64_t width, at::ScalarType dt) {
  if (tokens < 1 || tokens > kOneLaunchTokens) return false;
  const int64_t built = tokens <= 2 ? tokens : tokens <= 4 ? 4 : 8;
  return dt == at::kFloat || (dt == at::kBFloat16 && built * std::max(d_model, width) <= kOneLaunchValuesBf16);
}

// One decode step of a block (mambapy/mamba.py:351-414) -> (output (B, D), state, window), with fresh cache tensors.
// A few tokens go through one cooperative launch (block_step.cu) when every weight has the activations' type and nothing wants
// a gradient; otherwise the projections are library GEMMs with the two step kernels between them.
std::tuple<Tensor, Tensor, Tensor> block_step(const Tensor& x, const OptTensor& h_, const Tensor& inputs, const Tensor& in_w,
                                              const OptTensor& in_b_, const Tensor& conv_w, const OptTensor& conv_b_, const Tensor& xproj_w,
                                              const Tensor& dt_w, const Tensor& dt_b, const Tensor& A_log, const Tensor& D,
                                              const Tensor& out_w, const OptTensor& out_b_, int64_t R, int64_t N) {
  const Tensor &h = value(h_), &in_b = value(in_b_), &conv_b = value(conv_b_), &out_b = value(out_b_);
  require_cuda(x, h, inputs, in_w, in_b, conv_w, conv_b, xproj_w, dt_w, dt_b, A_log, D, out_w, out_b);
  const c10::cuda::CUDAGuard guard(x.device());
  const auto dt = x.scalar_type();
  TORCH_CHECK(x.dim() == 2 && dt_w.dim() == 2 && out_w.dim() == 2, "mamba_b200: a step takes (B, d_model) activations and matrices as weights");
  const int64_t B = x.size(0), Dm = x.size(1), W = dt_w.size(0), K = conv_w.size(-1);
  shape_is(in_w, {2 * W, Dm}, "in_proj.weight");
  numel_is(in_b, 2 * W, "in_proj.bias");
  numel_is(conv_w, W * K, "conv1d.weight");
  numel_is(conv_b, W, "conv1d.bias");
  shape_is(xproj_w, {R + 2 * N, W}, "x_proj.weight");
  shape_is(dt_w, {W, R}, "dt_proj.weight");
  numel_is(dt_b, W, "dt_proj.bias");
  shape_is(A_log, {W, N}, "A_log");
  numel_is(D, W, "D");
  shape_is(out_w, {out_w.size(0), W}, "out_proj.weight");
  numel_is(out_b, out_w.size(0), "out_proj.bias");
  TORCH_CHECK(inputs.numel() >= B * W * (K - 1) && (!h.defined() || h.numel() >= B * W * N), "mamba_b200: the caches hold fewer than ", B,
              " rows of ", W, " channels");
  bool one = out_w.size(0) == Dm && takes_one_launch(B, Dm, W, dt) && !at::autocast::is_autocast_enabled(at::kCUDA) &&
             !wants_grad(x, in_w, in_b, out_w, out_b);
  for (const Tensor* t : {&in_w, &in_b, &xproj_w, &dt_w, &out_w, &out_b})
    one = one && (!t->defined() || (t->scalar_type() == dt && t->is_contiguous()));
  if (one) {
    const BelowAutograd guard_ad;
    const Tensor xs = rows(x, dt), win = inputs.to(dt).contiguous(), h32 = f32(h);
    const Tensor cw = small_param(conv_w), cb = small_param(conv_b), db = small_param(dt_b), al = small_param(A_log), d = small_param(D);
    const Tensor out = empty({B, Dm}, dt, xs), h_new = empty({B, W, N}, at::kFloat, xs), fresh = empty(win.sizes(), dt, xs);
    mb200_block_step_args a{};
    a.x = ptr(xs); a.in_w = ptr(in_w); a.in_b = ptr(in_b); a.conv_in = ptr(win); a.conv_w = ptr(cw); a.conv_b = ptr(cb);
    a.xproj_w = ptr(xproj_w); a.dt_w = ptr(dt_w); a.dt_b = ptr(db); a.A_log = ptr(al); a.D = ptr(d); a.out_w = ptr(out_w); a.out_b = ptr(out_b);
    a.h_in = fptr(h32); a.conv_out = ptr(fresh); a.out = ptr(out); a.h_out = fptr(h_new);
    a.B = B; a.D_model = Dm; a.W = W; a.R = R; a.x_sb = st(xs, 0);
    a.N = int(N); a.d_conv = int(cw.size(-1)); a.dtype = dtype_code(dt);
    a.conv_w_dtype = code_of(cw); a.conv_b_dtype = code_of(cb); a.dt_b_dtype = code_of(db); a.A_log_dtype = code_of(al); a.D_dtype = code_of(d);
    const Tensor scratch = empty({mb200_block_step_scratch_floats(B, W, R, int(N))}, at::kFloat, xs), bars = barrier_counters(xs);
    const int rc = mb200_block_step(&a, fptr(scratch), ptr(bars), cuda_stream());
    if (rc != MB200_EUNSUPPORTED && rc != MB200_ETOOBIG) {
      check(rc, "mb200_block_step");
      check_status("mb200_block_step");
      return {out, h_new, fresh};
    }
  }
  // outside autograd and autocast the projections need nothing of at::linear but the product
  bool direct = convertible(dt) && !at::autocast::is_autocast_enabled(at::kCUDA) && !wants_grad(x, in_w, in_b, out_w, out_b, xproj_w, dt_w);
  for (const Tensor* t : {&in_w, &xproj_w, &dt_w, &out_w}) direct = direct && t->scalar_type() == dt;
  auto project = [&](const Tensor& v, const Tensor& weight, const OptTensor& bias) {
    if (!direct || value(bias).defined()) return at::linear(v, weight, bias);
    const BelowAutograd guard_ad;
    return product(v, transposed(weight));
  };
  const Tensor xz = project(x, in_w, in_b_);
  WindowStep w;
  // the exponentials of A_log and the casts are worth doing once as soon as enough rows share them
  const bool once = B >= 32 && small_type(A_log) && small_type(D) && small_type(dt_b) && A_log.is_contiguous() && D.is_contiguous() &&
                    dt_b.is_contiguous();
  Tensor A = A_log, Df = D, bf = dt_b;
  {
    const BelowAutograd guard_ad;
    Convert conv;
    if (once) {
      A = empty(A_log.sizes(), at::kFloat, A_log);
      const int64_t n = A.numel();
      conv.add(ptr(A_log), A_log.scalar_type(), ptr(A), at::kFloat, 1, n, n, n, n, MB200_CONVERT_NEG_EXP);
      Df = conv.cast(D, at::kFloat);
      bf = conv.cast(dt_b, at::kFloat);
    }
    w = window_step(columns(xz, 0, W), inputs, conv_w, conv_b, false, conv.jobs, conv.n);
  }
  const Tensor dbc = project(w.xc, xproj_w, {});
  const Tensor delta = project(direct ? columns(dbc, 0, R) : dbc.narrow(1, 0, R), dt_w, {});               // bias and softplus happen in the kernel
  StateStep s;
  {
    const BelowAutograd guard_ad;
    // the kernel reads A in 16-byte vectors; a parameter may lie anywhere (one piece of a flat buffer)
    if (!once && reinterpret_cast<uintptr_t>(A.data_ptr()) % 16) A = A.clone(at::MemoryFormat::Contiguous);
    s = state_step(w.xc, h, delta, A, !once, columns(dbc, R, N), columns(dbc, R + N, N), Df, columns(xz, W, W), bf, false);
  }
  return {project(s.y, out_w, out_b_), s.h, w.window};
}

}  // namespace mb200_host

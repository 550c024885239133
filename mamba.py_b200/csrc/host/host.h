// Host side of the package in C++: argument checks, allocations, autograd nodes and kernel launches, so that a call
// costs a few microseconds of host time instead of a few tens.  Device work goes through the C ABI of
// libmamba_b200.so (include/mamba_b200.h) only.
#pragma once
#include <torch/extension.h>
#include <torch/csrc/autograd/forward_grad.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/core/grad_mode.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <optional>
#include "mamba_b200.h"

namespace mb200_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// ---- checks and preparation ------------------------------------------------------------------------------
inline const Tensor& undefined() {
  static const Tensor t;
  return t;
}
inline const Tensor& value(const OptTensor& t) { return t.has_value() ? *t : undefined(); }

template <typename... Ts> void require_cuda(const Ts&... ts) {
  for (const Tensor* t : {&ts...})
    TORCH_CHECK(!t->defined() || t->is_cuda(), "mamba_b200 runs on CUDA tensors only (there is no CPU path)");
}

// Kernels and GEMMs take sizes from one tensor for all: what calling the modules one by one would compare is compared here.
inline void shape_is(const Tensor& t, at::IntArrayRef want, const char* what) {
  TORCH_CHECK(t.sizes() == want, "mamba_b200: ", what, " should be ", want, ", got ", t.sizes());
}
inline void numel_is(const Tensor& t, int64_t want, const char* what) {
  TORCH_CHECK(!t.defined() || t.numel() == want, "mamba_b200: ", what, " should have ", want, " elements, got ", t.numel());
}

inline void check(int rc, const char* what) {
  TORCH_CHECK(rc == MB200_OK, what, " failed: ", mb200_strerror(rc), " (code ", rc, ")");
}

// Activation dtype a kernel runs in: bfloat16 only when EVERY activation tensor is bfloat16, float32 as soon as one of
// them is (under autocast the reference keeps delta in float32 while x, B and C are bfloat16,
// mambapy/mamba.py:264-265; rounding delta to bfloat16 would change the decay).
template <typename... Ts> at::ScalarType act_dtype(const Ts&... ts) {
  bool all_bf16 = true;
  for (const Tensor* t : {&ts...}) {
    if (!t->defined()) continue;
    const auto d = t->scalar_type();
    TORCH_CHECK_TYPE(d == at::kFloat || d == at::kBFloat16, "mamba_b200 kernels take float32 or bfloat16 activations, got ", d);
    all_bf16 = all_bf16 && d == at::kBFloat16;
  }
  return all_bf16 ? at::kBFloat16 : at::kFloat;
}
inline int dtype_code(at::ScalarType d) { return d == at::kBFloat16 ? MB200_BF16 : MB200_F32; }

// Cast to the activation dtype and make the last dimension unit-stride (copies only if needed).
inline Tensor rows(const Tensor& t, at::ScalarType dt) {
  if (!t.defined()) return t;
  Tensor r = t.scalar_type() == dt ? t : t.to(dt);
  return r.stride(-1) == 1 ? r : r.contiguous();
}
inline Tensor f32(const Tensor& t) {
  if (!t.defined()) return t;
  return (t.scalar_type() == at::kFloat && t.is_contiguous()) ? t.detach() : t.detach().to(at::kFloat).contiguous();
}
inline Tensor like(const Tensor& grad, at::ScalarType dt) { return grad.scalar_type() == dt ? grad : grad.to(dt); }

inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
inline int64_t st(const Tensor& t, int d) { return t.defined() ? t.stride(d) : 0; }
// Straight to the caching allocator: the dispatcher's way to the same place costs three times as much.
inline Tensor empty(at::IntArrayRef shape, at::ScalarType dt, const Tensor& on) {
  return at::detail::empty_cuda(shape, dt, on.device(), std::nullopt);
}
// `shape` dense elements of `base`'s storage from element `offset` of it on (a plain alias, not an autograd view).
inline Tensor alias(const Tensor& base, int64_t offset, at::IntArrayRef shape) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
  t.unsafeGetTensorImpl()->set_version_counter(base.unsafeGetTensorImpl()->version_counter());
  t.unsafeGetTensorImpl()->set_storage_offset(base.storage_offset() + offset);
  t.unsafeGetTensorImpl()->set_sizes_contiguous(shape);
  return t;
}
// The same storage under other sizes and strides, the columns [first, first + n) of the last dimension, and a matrix transposed.
inline Tensor strided(const Tensor& base, int64_t offset, at::IntArrayRef shape, at::IntArrayRef strides) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()), base.key_set(), base.dtype());
  t.unsafeGetTensorImpl()->set_version_counter(base.unsafeGetTensorImpl()->version_counter());
  t.unsafeGetTensorImpl()->set_sizes_and_strides(shape, strides, base.storage_offset() + offset);
  return t;
}
inline Tensor columns(const Tensor& t, int64_t first, int64_t n) {
  c10::SmallVector<int64_t, 4> shape(t.sizes().begin(), t.sizes().end());
  shape.back() = n;
  return strided(t, first * t.stride(-1), shape, t.strides());
}
inline Tensor transposed(const Tensor& t) { return strided(t, 0, {t.size(1), t.size(0)}, {t.stride(1), t.stride(0)}); }
// Item i of matrices that lie s elements apart.
inline Tensor item(const Tensor& t, int64_t i, int64_t s) { return i ? strided(t, i * s, t.sizes(), t.strides()) : t; }
inline void zero_fill(const Tensor& t) {
  C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, t.nbytes(), at::cuda::getCurrentCUDAStream()));
}
inline void* cuda_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// With MB200_CHECK_STATUS=1 in the environment every launch of a kernel with bounded waits (the fused scans, the one-launch step)
// is followed by a device synchronisation and a read of the kernels' status word; a wait that gave up then raises.  A stream that
// is being captured into a graph launches nothing yet and is left alone.
void check_status(const char* what);

// The library's own tensor operations record nothing: autograd sees the nodes below only.
using BelowAutograd = at::AutoDispatchBelowADInplaceOrView;

// ---- autograd plumbing ------------------------------------------------------------------------------------
template <typename... Ts> bool wants_grad(const Ts&... ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : {&ts...})
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
// The nodes have no forward-mode derivative.  A tangent that a call would lose is an error, with gradients recorded or not.
inline bool has_tangent(const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); }
template <typename... Ts> void refuse_tangents(const Ts&... ts) {
  if (!torch::autograd::ForwardADLevel::try_get_by_idx(0)) return;
  for (const Tensor* t : {&ts...})
    TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(*t), "mamba_b200: forward-mode automatic differentiation is not implemented");
}
template <typename N> std::shared_ptr<N> new_node() { return std::shared_ptr<N>(new N(), torch::autograd::deleteNode); }

// A tensor kept for the backward; intermediates and inputs alike (version counters are checked on unpacking).
struct Saved {
  SavedVariable v;
  bool defined = false;
  void save(const Tensor& t, bool is_output = false) {
    defined = t.defined();
    if (defined) v = SavedVariable(t, is_output);
  }
  Tensor get(const std::shared_ptr<torch::autograd::Node>& self = nullptr) const { return defined ? v.unpack(self) : Tensor(); }
  void reset() { v.reset_data(); }
};

// A matrix product as it leaves the GEMM: one (rows, cols) matrix, or `slices` float32 ones to be added up.
struct Partials {
  Tensor t;
  int slices;
  int64_t rows, cols;
};
// `tall` is a^T b for two tall matrices of one type (gemm.cpp); `out` is the type wanted if nothing has to be added up.
// Independent products in one place: the small ones are collected and share a launch (run()), the others go to the library at once.
struct Products {
  mb200_product p[4];
  int n = 0;
  at::ScalarType dt;
  bool add(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta);       // false: not a small one
  void into(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta);      // out = alpha * a b + beta * out
  Tensor of(const Tensor& a, const Tensor& b);
  // n products of one shape; item i of an operand lies s* elements behind item i - 1
  void each(int64_t n, const Tensor& out, int64_t so, const Tensor& a, int64_t sa, const Tensor& b, int64_t sb, float alpha, float beta);
  std::vector<Partials> tall(int64_t n, const Tensor& a, int64_t sa, const Tensor& b, int64_t sb, at::ScalarType out, float alpha);
  Partials tall(const Tensor& a, const Tensor& b, at::ScalarType out, float alpha) { return tall(1, a, 0, b, 0, out, alpha)[0]; }
  void run();
};

// Element-wise jobs of one launch (mb200_convert).
struct Convert {
  mb200_convert_job jobs[MB200_CONVERT_MAX_JOBS];
  int n = 0;
  mb200_convert_job& add(const void* src, at::ScalarType st, void* dst, at::ScalarType dt, int64_t rows, int64_t cols, int64_t src_cols,
                         int64_t src_stride, int64_t dst_stride, int op = MB200_CONVERT_COPY) {
    // (not launched when full: a job's source may be a product that has yet to run)
    TORCH_CHECK(n < MB200_CONVERT_MAX_JOBS, "mamba_b200: more than ", int(MB200_CONVERT_MAX_JOBS), " conversions for one launch");
    mb200_convert_job& j = jobs[n++];
    j = mb200_convert_job{src, dst, nullptr, rows, cols, src_cols, src_stride, dst_stride, dtype_code(st), dtype_code(dt), op, 1, 0};
    return j;
  }
  // a dense tensor once more in another type; itself when it has that type already
  Tensor cast(const Tensor& src, at::ScalarType dt) {
    if (!src.defined() || src.scalar_type() == dt) return src;
    const Tensor dst = empty(src.sizes(), dt, src);
    const int64_t m = src.numel();
    add(ptr(src), src.scalar_type(), ptr(dst), dt, 1, m, m, m, m);
    return dst;
  }
  // rows [first, first + rows) of a product into dst
  void rows_of(const Partials& p, int64_t first, int64_t rows, void* dst, at::ScalarType dt);
  Tensor settle(const Partials& p, at::ScalarType dt);
  void run() {
    if (n) check(mb200_convert(jobs, n, cuda_stream()), "mb200_convert");
    n = 0;
  }
};
inline void Convert::rows_of(const Partials& p, int64_t first, int64_t rows, void* dst, at::ScalarType dt) {
  const int64_t n = rows * p.cols;
  mb200_convert_job& j = add(static_cast<char*>(p.t.data_ptr()) + first * p.cols * p.t.element_size(), p.t.scalar_type(), dst, dt, 1, n, n, n, n);
  j.slices = p.slices;
  j.slice_stride = p.rows * p.cols;
}
inline Tensor Convert::settle(const Partials& p, at::ScalarType dt) {
  if (p.slices == 1 && p.t.scalar_type() == dt) return p.t;
  const Tensor dst = empty({p.rows, p.cols}, dt, p.t);
  rows_of(p, 0, p.rows, ptr(dst), dt);
  return dst;
}
inline bool convertible(at::ScalarType d) { return d == at::kFloat || d == at::kBFloat16; }

// What a node remembers of an input whose gradient it returns.
inline at::ScalarType type_of(const Tensor& t) { return t.defined() ? t.scalar_type() : at::kFloat; }

// ---- entry points -------------------------------------------------------------------------------------------
py::object selective_scan(const Tensor& x, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const OptTensor& D,
                          const OptTensor& z, const OptTensor& delta_bias, const OptTensor& h0, bool return_last_state, bool reverse,
                          std::optional<int64_t> subshards);
Tensor pscan(const Tensor& A, const Tensor& X);
Tensor conv1d_silu(const Tensor& x, const Tensor& weight, const OptTensor& bias);
Tensor rms_norm(const Tensor& x, const OptTensor& weight, double eps);
std::tuple<Tensor, Tensor> add_rms_norm(const Tensor& x, const OptTensor& residual, const OptTensor& weight, double eps);
// out = alpha * a b + beta * out, and a b (gemm.cpp)
void product_into(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta);
Tensor product(const Tensor& a, const Tensor& b);
Tensor add_residual(const Tensor& x, const Tensor& residual);
std::tuple<Tensor, Tensor> ssm_step(const Tensor& x, const OptTensor& h, const Tensor& delta, const Tensor& A, const Tensor& B,
                                    const Tensor& C, const OptTensor& D, const OptTensor& z, const OptTensor& delta_bias, bool inplace);
std::tuple<Tensor, Tensor> conv_step(const Tensor& x, const Tensor& inputs, const Tensor& weight, const OptTensor& bias, bool inplace);

Tensor block(const Tensor& x, const OptTensor& in_w, const OptTensor& out_w, const std::vector<OptTensor>& params, int64_t dt_rank,
             int64_t d_state, bool halve);
bool reversible(int64_t width, int64_t d_state, at::ScalarType dt);
std::tuple<Tensor, Tensor, Tensor> block_step(const Tensor& x, const OptTensor& h, const Tensor& inputs, const Tensor& in_w, const OptTensor& in_b,
                                              const Tensor& conv_w, const OptTensor& conv_b, const Tensor& xproj_w, const Tensor& dt_w,
                                              const Tensor& dt_b, const Tensor& A_log, const Tensor& D, const Tensor& out_w,
                                              const OptTensor& out_b, int64_t dt_rank, int64_t d_state);

// Queues `n` empty conversions for one launch, without launching them.
void selftest_queue_conversions(int64_t n);
// Spoils the barrier counters that the current stream keeps for the one-launch step on `on`'s device, as a launch that gave up does.
void selftest_block_step_give_up(const Tensor& on);

int64_t pick_pieces(int64_t batch, int64_t length, int64_t width, bool grad);

}  // namespace mb200_host

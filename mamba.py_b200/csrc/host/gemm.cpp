// The projections' matrix products: the library GEMM that at::mm ends in, without the way there.
//
// at::mm costs 9 us of host time around a launch of 4 (dispatcher, structured-kernel set-up, an output allocation through the
// dispatcher, TensorIterator-style checks); a training step of a small layer has twelve of them.  Here the arguments go straight
// to cuBLAS on torch's handle of the current stream, which carries its workspace and its float32 precision setting.
#include <ATen/Context.h>
#include <cublas_v2.h>
#include <limits>
#include "host.h"

namespace mb200_host {
namespace {

// A 2-d tensor as a column-major operand: `trans` says that its memory, read by columns, is the tensor itself.
struct Operand {
  bool ok, trans;
  int64_t ld;
  explicit Operand(const Tensor& t) {
    const int64_t r = t.size(0), c = t.size(1), s0 = t.stride(0), s1 = t.stride(1);
    if ((s1 == 1 || c == 1) && s0 >= c) {
      ok = true; trans = false; ld = s0;
    } else {
      ok = (s0 == 1 || r == 1) && s1 >= r; trans = true; ld = s1;
    }
    ok = ok && ld <= std::numeric_limits<int>::max() && r > 0 && c > 0 && r <= std::numeric_limits<int>::max() && c <= std::numeric_limits<int>::max();
  }
  cublasOperation_t op() const { return trans ? CUBLAS_OP_T : CUBLAS_OP_N; }
};

// Settings under which at::mm would do something else than the two calls below.
bool plain_settings() {
  auto& ctx = at::globalContext();
  const auto backend = ctx.blasPreferredBackend();
  return (backend == at::BlasBackend::Cublas || backend == at::BlasBackend::Default) && !ctx.deterministicAlgorithms() &&
         ctx.allowBF16ReductionCuBLAS() == at::CuBLASReductionOption::AllowReducedPrecisionWithSplitK;
}

}  // namespace

// out = alpha * a b + beta * out; out has unit-stride rows.
void product_into(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta) {
  const auto dt = out.scalar_type();
  const Operand A(a), B(b), O(out);
  if (!A.ok || !B.ok || !O.ok || O.trans || a.size(1) != b.size(0) || out.size(0) != a.size(0) || out.size(1) != b.size(1) ||
      a.scalar_type() != dt || b.scalar_type() != dt || !convertible(dt) || !plain_settings()) {
    Tensor o = out;
    at::addmm_out(o, o, a, b, beta, alpha);
    return;
  }
  // row-major out is column-major out^T = b^T a^T
  const int m = int(b.size(1)), n = int(a.size(0)), k = int(a.size(1));
  const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
  const cublasStatus_t rc =
      dt == at::kFloat
          ? cublasSgemm(handle, B.op(), A.op(), m, n, k, &alpha, fptr(b), int(B.ld), fptr(a), int(A.ld), &beta, fptr(out), int(O.ld))
          : cublasGemmEx(handle, B.op(), A.op(), m, n, k, &alpha, ptr(b), CUDA_R_16BF, int(B.ld), ptr(a), CUDA_R_16BF, int(A.ld), &beta,
                         ptr(out), CUDA_R_16BF, int(O.ld), CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT_TENSOR_OP);
  TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "mamba_b200: matrix product failed, cuBLAS status ", int(rc));
}

Tensor product(const Tensor& a, const Tensor& b) {
  const Tensor out = empty({a.size(0), b.size(1)}, a.scalar_type(), a);
  product_into(out, a, b, 1.f, 0.f);
  return out;
}

}  // namespace mb200_host

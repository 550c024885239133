// The projections' matrix products: the library GEMM that at::mm ends in, without the way there.
//
// at::mm costs 9 us of host time around a launch of 4 (dispatcher, structured-kernel set-up, an output allocation through the
// dispatcher, TensorIterator-style checks); a training step of a small layer has twelve of them.  Here the arguments go straight
// to cuBLAS on torch's handle of the current stream, which carries its workspace and its float32 precision setting.
#include <ATen/Context.h>
#include <cublas_v2.h>
#include <algorithm>
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

// Tiles of 32 x 32 and terms up to which a product goes through our own kernel.  What that saves is host time, for a product that shares
// a launch and for one alone (a library call takes the host longer than a launch); on the GPU it is never ahead.  Device time of one,
// ours / library, us: float32 (122, 256, 64) 6.3 / 6.3, (64, 64, 256) 10.4 / 8.3, (500, 500, 128) 8.4 / 6.6, (512, 512, 256) 14.5 / 9.2;
// bfloat16, where the library has tensor cores, (122, 256, 64) 6.3 / 4.3, (122, 64, 128) 10.4 / 4.3, (512, 512, 64) 8.4 / 4.3.
// Calls that fall under the rule wait for the host.  us, two layers of 64 channels, 122 tokens, ours / ours where shared / library:
//                            called from Python     inside a CUDA graph, where there is no host work
//   training    float32      506 / 549 / 643        178 / 172 / 197
//               bfloat16     665 / 693 / 691        178 / 156 / 156
//   inference   float32      117 / 156 / 152         68 /  64 /  62
//               bfloat16     159 / 174 / 174         62 /  53 /  51
bool small(int64_t M, int64_t N, int64_t K, at::ScalarType dt) {
  const int64_t tiles = (M + 31) / 32 * ((N + 31) / 32);
  if (dt == at::kFloat) return tiles <= 64 ? K <= 256 : tiles <= 296 && K <= 128;
  return tiles <= 64 && K <= 64;
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

bool Products::add(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta) {
  const int64_t M = a.size(0), N = b.size(1), K = a.size(1);
  if (!small(M, N, K, a.scalar_type()) || out.stride(1) != 1 || b.size(0) != K || out.size(0) != M || out.size(1) != N || a.scalar_type() != b.scalar_type() ||
      !convertible(a.scalar_type()) || !convertible(out.scalar_type()) || (n > 0 && dt != a.scalar_type()))
    return false;
  if (n == 4) run();
  dt = a.scalar_type();
  p[n++] = mb200_product{a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), a.stride(1), b.stride(0), b.stride(1), out.stride(0),
                         alpha, beta, dtype_code(out.scalar_type())};
  return true;
}

void Products::into(const Tensor& out, const Tensor& a, const Tensor& b, float alpha, float beta) {
  if (!add(out, a, b, alpha, beta)) product_into(out, a, b, alpha, beta);
}

Tensor Products::of(const Tensor& a, const Tensor& b) {
  const Tensor out = empty({a.size(0), b.size(1)}, a.scalar_type(), a);
  into(out, a, b, 1.f, 0.f);
  return out;
}

void Products::run() {
  if (n) check(mb200_small_gemm(p, n, dtype_code(dt), cuda_stream()), "mb200_small_gemm");
  n = 0;
}

// The gradient of a weight is a product over all tokens with a small result: at (12608 tokens, 384 x 44) the library picks 12 tiles of
// 64 x 32 and walks all tokens in each, 17.7 us for 11 MB.  Cutting the tokens so that about every SM has a tile, with float32 partial
// sums that the conversion of the gradients adds up on its way, puts the whole chip on it.  At most 16 cuts (the sum reads them all)
// of at least 512 tokens (below that a product is a launch's latency anyway).
std::vector<Partials> Products::tall(int64_t n, const Tensor& a, int64_t sa, const Tensor& b, int64_t sb, at::ScalarType out, float alpha) {
  const auto dt = a.scalar_type();
  const int64_t T = a.size(0), M = a.size(1), N = b.size(1);
  const Operand A(a), B(b);
  const bool own = small(M, N, T, dt) && convertible(dt) && convertible(out);
  const bool ours = A.ok && B.ok && !A.trans && !B.trans && b.size(0) == T && b.scalar_type() == dt && convertible(dt) && convertible(out) && plain_settings();
  std::vector<Partials> res;
  const int64_t tiles = (M + 63) / 64 * ((N + 63) / 64) * n;
  const int64_t sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  int64_t S = tiles ? std::max<int64_t>(1, std::min<int64_t>({16, sms / tiles, T / 512})) : 1;
  if (own || !ours || (S == 1 && n == 1 && dt == at::kFloat)) {
    for (int64_t i = 0; i < n; ++i) {
      const Tensor o = empty({M, N}, own ? out : dt, a);
      into(o, transposed(item(a, i, sa)), item(b, i, sb), alpha, 0.f);
      res.push_back({o, 1, M, N});
    }
    return res;
  }
  for (int64_t s = S; 2 * s > S && S > 1; --s)
    if (T % s == 0) {                                            // equal cuts where the number of tokens has a divisor nearby
      S = s;
      break;
    }
  const int64_t len = T / S, rest = T - len * S;
  const int slices = int(S + (rest > 0));
  const auto ot = slices > 1 ? at::kFloat : out;
  const Tensor o = empty({n * slices * M, N}, ot, a);
  const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
  const cudaDataType_t in_t = dt == at::kFloat ? CUDA_R_32F : CUDA_R_16BF, out_t = ot == at::kFloat ? CUDA_R_32F : CUDA_R_16BF;
  const float beta = 0.f;
  // `count` products of k tokens from element offsets oa, ob on, da and db apart, into slices from `slice` on
  auto run = [&](int64_t oa, int64_t da, int64_t ob, int64_t db, int64_t k, int64_t count, int64_t slice) {
    const char *pa = static_cast<const char*>(a.data_ptr()) + oa * a.element_size(), *pb = static_cast<const char*>(b.data_ptr()) + ob * b.element_size();
    char* po = static_cast<char*>(o.data_ptr()) + slice * M * N * o.element_size();
    const cublasStatus_t rc =
        count == 1 ? cublasGemmEx(handle, CUBLAS_OP_N, CUBLAS_OP_T, int(N), int(M), int(k), &alpha, pb, in_t, int(B.ld), pa, in_t, int(A.ld), &beta,
                                  po, out_t, int(N), CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT)
                   : cublasGemmStridedBatchedEx(handle, CUBLAS_OP_N, CUBLAS_OP_T, int(N), int(M), int(k), &alpha, pb, in_t, int(B.ld), db, pa, in_t,
                                                int(A.ld), da, &beta, po, out_t, int(N), M * N, int(count), CUBLAS_COMPUTE_32F, CUBLAS_GEMM_DEFAULT);
    TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "mamba_b200: matrix product failed, cuBLAS status ", int(rc));
  };
  if (rest == 0 && (n == 1 || (sa == T * A.ld && sb == T * B.ld))) {
    run(0, len * A.ld, 0, len * B.ld, len, n * S, 0);            // cuts of all items are evenly spaced
  } else {
    for (int64_t i = 0; i < n; ++i) {
      run(i * sa, len * A.ld, i * sb, len * B.ld, len, S, i * slices);
      if (rest) run(i * sa + len * S * A.ld, 0, i * sb + len * S * B.ld, 0, rest, 1, i * slices + S);
    }
  }
  for (int64_t i = 0; i < n; ++i)
    res.push_back({slices == 1 ? alias(o, i * M * N, {M, N}) : alias(o, i * slices * M * N, {slices, M, N}), slices, M, N});
  return res;
}

void Products::each(int64_t n, const Tensor& out, int64_t so, const Tensor& a, int64_t sa, const Tensor& b, int64_t sb, float alpha, float beta) {
  const auto dt = out.scalar_type();
  const Operand A(a), B(b), O(out);
  const int64_t M = a.size(0), N = b.size(1), K = a.size(1);
  if (n == 1 || small(M, N, K, dt) || !A.ok || !B.ok || !O.ok || O.trans || b.size(0) != K || out.size(0) != M || out.size(1) != N ||
      a.scalar_type() != dt || b.scalar_type() != dt || !convertible(dt) || !plain_settings()) {
    for (int64_t i = 0; i < n; ++i) into(item(out, i, so), item(a, i, sa), item(b, i, sb), alpha, beta);
    return;
  }
  const cublasHandle_t handle = at::cuda::getCurrentCUDABlasHandle();
  const cudaDataType_t t = dt == at::kFloat ? CUDA_R_32F : CUDA_R_16BF;
  const cublasStatus_t rc = cublasGemmStridedBatchedEx(handle, B.op(), A.op(), int(N), int(M), int(K), &alpha, ptr(b), t, int(B.ld), sb, ptr(a), t,
                                                       int(A.ld), sa, &beta, ptr(out), t, int(O.ld), so, int(n), CUBLAS_COMPUTE_32F,
                                                       CUBLAS_GEMM_DEFAULT);
  TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "mamba_b200: matrix product failed, cuBLAS status ", int(rc));
}

}  // namespace mb200_host

// Small matrix products, several independent ones in one launch.
//
// A training step of a small layer has twelve products of a few hundred by a few hundred.  The library takes about 4.6 us of GPU and
// more than that of host time for each; what they compute is under a microsecond.  Here the products that do not depend on one
// another (a projection's input gradient and its weight gradient) share a launch, and a launch is all the host does.  Bound by
// latency: a CTA owns a 32 x 32 tile and walks K in slabs of 32 through shared memory, the next slab's loads in flight while one is
// multiplied; any strides, so that transposes cost nothing.  float32 multiply-adds for either input type.  Two layers of 64 channels,
// 122 tokens, a training step called from Python: 643 us with the library's products, 506 with these, 8 launches a layer for 12 (inside
// a CUDA graph 197 and 178).
#include "common.cuh"

namespace mb200 {
namespace {

constexpr int kTile = 32, kSlab = 32, kGemmThreads = 128, kMaxProducts = 4;
constexpr int kPitch = kTile + 4;                       // rows of a slab stay 16-byte aligned

struct Products {
  mb200_product p[kMaxProducts];
  int first_block[kMaxProducts + 1];
  int n;
};

// A 32 x 32 slab of a strided matrix, 8 elements a thread, neighbouring threads along the direction with the smaller stride.
template <typename T> struct Slab {
  static constexpr int kEach = kTile * kSlab / kGemmThreads;
  float v[kEach];
  __device__ __forceinline__ static void at(int u, bool along_k, int& t, int& k) {
    const int i = threadIdx.x + u * kGemmThreads;
    t = along_k ? i / kSlab : i % kTile;
    k = along_k ? i % kSlab : i / kTile;
  }
  // element (t, k) at t * ts + k * ks
  __device__ __forceinline__ void load(const T* p, int64_t ts, int64_t ks, int t_left, int k_left, bool along_k) {
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      int t, k;
      at(u, along_k, t, k);
      v[u] = t < t_left && k < k_left ? Elem<T>::to_f(p[t * ts + k * ks]) : 0.f;
    }
  }
  __device__ __forceinline__ void store(float (*s)[kPitch], bool along_k) const {
#pragma unroll
    for (int u = 0; u < kEach; ++u) {
      int t, k;
      at(u, along_k, t, k);
      s[k][t] = v[u];
    }
  }
};

template <typename T>
__global__ void __launch_bounds__(kGemmThreads) small_gemm_kernel(const __grid_constant__ Products all) {
  __shared__ alignas(16) float as[kSlab][kPitch], bs[kSlab][kPitch];
  int q = 0;
  while (q + 1 < all.n && int(blockIdx.x) >= all.first_block[q + 1]) ++q;
  const mb200_product& p = all.p[q];
  const int tiles_n = int((p.N + kTile - 1) / kTile), tile = int(blockIdx.x) - all.first_block[q];
  const int64_t m0 = int64_t(tile / tiles_n) * kTile, n0 = int64_t(tile % tiles_n) * kTile;
  const int m_left = int(min(int64_t(kTile), p.M - m0)), n_left = int(min(int64_t(kTile), p.N - n0));
  const bool a_along_k = p.a_ck <= p.a_rm, b_along_k = p.b_rk <= p.b_cn;
  const T *a = static_cast<const T*>(p.a) + m0 * p.a_rm, *b = static_cast<const T*>(p.b) + n0 * p.b_cn;
  // this thread's outputs: rows ty * 2 + {0, 1}, columns tx * 4 + {0 .. 3}
  const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;
  float acc[2][4] = {};
  Slab<T> av, bv;
  av.load(a, p.a_rm, p.a_ck, m_left, int(min(int64_t(kSlab), p.K)), a_along_k);
  bv.load(b, p.b_cn, p.b_rk, n_left, int(min(int64_t(kSlab), p.K)), b_along_k);
  for (int64_t k0 = 0; k0 < p.K; k0 += kSlab) {
    if (k0) __syncthreads();
    av.store(as, a_along_k);
    bv.store(bs, b_along_k);
    __syncthreads();
    const int64_t next = k0 + kSlab;
    if (next < p.K) {
      const int left = int(min(int64_t(kSlab), p.K - next));
      av.load(a + next * p.a_ck, p.a_rm, p.a_ck, m_left, left, a_along_k);
      bv.load(b + next * p.b_rk, p.b_cn, p.b_rk, n_left, left, b_along_k);
    }
#pragma unroll
    for (int k = 0; k < kSlab; ++k) {
      const float2 x = *reinterpret_cast<const float2*>(&as[k][ty * 2]);
      const float4 y = *reinterpret_cast<const float4*>(&bs[k][tx * 4]);
      acc[0][0] = fmaf(x.x, y.x, acc[0][0]); acc[0][1] = fmaf(x.x, y.y, acc[0][1]);
      acc[0][2] = fmaf(x.x, y.z, acc[0][2]); acc[0][3] = fmaf(x.x, y.w, acc[0][3]);
      acc[1][0] = fmaf(x.y, y.x, acc[1][0]); acc[1][1] = fmaf(x.y, y.y, acc[1][1]);
      acc[1][2] = fmaf(x.y, y.z, acc[1][2]); acc[1][3] = fmaf(x.y, y.w, acc[1][3]);
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = ty * 2 + i, n = tx * 4 + j;
      if (m >= m_left || n >= n_left) continue;
      const int64_t o = (m0 + m) * p.out_rm + n0 + n;
      float v = p.alpha * acc[i][j];
      if (p.out_dtype == MB200_F32) {
        float* d = static_cast<float*>(p.out) + o;
        *d = p.beta != 0.f ? fmaf(p.beta, *d, v) : v;
      } else {
        __nv_bfloat16* d = static_cast<__nv_bfloat16*>(p.out) + o;
        *d = __float2bfloat16_rn(p.beta != 0.f ? fmaf(p.beta, __bfloat162float(*d), v) : v);
      }
    }
}

}  // namespace
}  // namespace mb200

using namespace mb200;

extern "C" int mb200_small_gemm(const mb200_product* products, int n, int dtype, void* stream) {
  if (n < 0 || n > kMaxProducts || (n > 0 && !products)) return MB200_EINVAL;
  if (dtype != MB200_F32 && dtype != MB200_BF16) return MB200_EDTYPE;
  Products all;
  all.n = 0;
  int64_t blocks = 0;
  for (int i = 0; i < n; ++i) {
    const mb200_product& p = products[i];
    if (p.M < 0 || p.N < 0 || p.K < 0) return MB200_EINVAL;
    if (p.out_dtype != MB200_F32 && p.out_dtype != MB200_BF16) return MB200_EDTYPE;
    if (p.M == 0 || p.N == 0) continue;
    if (!p.out || (p.K > 0 && (!p.a || !p.b))) return MB200_EINVAL;
    all.p[all.n] = p;
    all.first_block[all.n++] = int(blocks);
    blocks += (p.M + kTile - 1) / kTile * ((p.N + kTile - 1) / kTile);
    if (blocks > (int64_t(1) << 30)) return MB200_ETOOBIG;
  }
  if (all.n == 0) return MB200_OK;
  all.first_block[all.n] = int(blocks);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == MB200_F32) small_gemm_kernel<float><<<unsigned(blocks), kGemmThreads, 0, st>>>(all);
  else small_gemm_kernel<__nv_bfloat16><<<unsigned(blocks), kGemmThreads, 0, st>>>(all);
  return check_launch();
}

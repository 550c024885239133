// The body of the element-wise jobs (mb200_convert_job), for the launch that does nothing else and for kernels that take a few along.
#pragma once
#include "common.cuh"

namespace mb200 {
namespace {

constexpr int kConvertThreads = 256;
constexpr int kPerThread = 4;

struct Job : mb200_convert_job {
  bool vec;
};
template <int kMax> struct Jobs {
  Job job[kMax];
  int first_block[kMax + 1];             // blocks first_block[i] .. first_block[i + 1] - 1 work on job i
  int n;
};

__device__ __forceinline__ float load_as_float(const void* p, int dtype, int64_t i) {
  return dtype == MB200_F32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}

// Block `block` of the jobs' blocks, kConvertThreads threads.
template <int kMax> __device__ __forceinline__ void convert_block(const Jobs<kMax>& jobs, int block) {
  int k = 0;
  while (k + 1 < jobs.n && block >= jobs.first_block[k + 1]) ++k;
  const Job& j = jobs.job[k];
  const int64_t total = j.rows * j.cols;
  const int64_t base = int64_t(block - jobs.first_block[k]) * kConvertThreads * kPerThread + threadIdx.x;
  const bool small = total < (int64_t(1) << 31);               // 32-bit division is several times cheaper
  auto row_col = [&](int64_t i, int64_t& r, int64_t& c) {
    if (j.rows == 1) { r = 0; c = i; }
    else if (small) { const unsigned q = unsigned(i) / unsigned(j.cols); r = q; c = i - int64_t(q) * j.cols; }
    else { r = i / j.cols; c = i - r * j.cols; }
  };
  // rows on the vector grid: four neighbouring elements a thread
  if (j.vec) {
    const int64_t i = (int64_t(block - jobs.first_block[k]) * kConvertThreads + threadIdx.x) * 4;
    if (i >= total) return;
    int64_t row, c;
    row_col(i, row, c);
    const int64_t from = row * j.src_stride + c, to = row * j.dst_stride + c;
    alignas(16) float f[4];
    if (j.src_dtype == MB200_F32) {
      *reinterpret_cast<float4*>(f) = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(j.src) + from));
    } else {
      const uint2 w = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(j.src) + from));
      f[0] = __uint_as_float(w.x << 16); f[1] = __uint_as_float(w.x & 0xffff0000u);
      f[2] = __uint_as_float(w.y << 16); f[3] = __uint_as_float(w.y & 0xffff0000u);
    }
    if (j.slices > 1) {                                        // float32 partial sums
      const float* p = static_cast<const float*>(j.src) + from;
#pragma unroll 4
      for (int q = 1; q < j.slices; ++q) {
        const float4 g = __ldg(reinterpret_cast<const float4*>(p + q * j.slice_stride));
        f[0] += g.x; f[1] += g.y; f[2] += g.z; f[3] += g.w;
      }
    }
    if (j.op == MB200_CONVERT_NEG_EXP) {
#pragma unroll
      for (int u = 0; u < 4; ++u) f[u] = -expf(f[u]);
    } else if (j.op != MB200_CONVERT_COPY) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(j.factor + i));
      const float gv[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) f[u] = j.op == MB200_CONVERT_MUL ? f[u] * gv[u] : f[u] + gv[u];
    }
    if (j.dst_dtype == MB200_F32) {
      *reinterpret_cast<float4*>(static_cast<float*>(j.dst) + to) = make_float4(f[0], f[1], f[2], f[3]);
    } else {
      const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
      *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(j.dst) + to) =
          make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
    return;
  }
  float v[kPerThread];
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    const int64_t i = base + u * kConvertThreads;
    v[u] = 0.f;
    if (i >= total) continue;
    int64_t r, c;
    row_col(i, r, c);
    if (j.src && c < j.src_cols) v[u] = load_as_float(j.src, j.src_dtype, r * j.src_stride + c);
    for (int q = 1; q < j.slices; ++q)
      if (c < j.src_cols) v[u] += load_as_float(j.src, j.src_dtype, q * j.slice_stride + r * j.src_stride + c);
    if (j.op == MB200_CONVERT_NEG_EXP) v[u] = -expf(v[u]);
    if (j.op == MB200_CONVERT_MUL) v[u] *= j.factor[i];
    if (j.op == MB200_CONVERT_ADD) v[u] += j.factor[i];
  }
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    const int64_t i = base + u * kConvertThreads;
    if (i >= total) continue;
    int64_t r, c;
    row_col(i, r, c);
    const int64_t o = r * j.dst_stride + c;
    if (j.dst_dtype == MB200_F32) static_cast<float*>(j.dst)[o] = v[u];
    else static_cast<__nv_bfloat16*>(j.dst)[o] = __float2bfloat16_rn(v[u]);
  }
}

// Checks the jobs and gives them blocks; MB200_OK and the number of blocks, or an error.
template <int kMax> int collect_jobs(const mb200_convert_job* jobs, int n, Jobs<kMax>& all, int64_t& blocks) {
  if (n < 0 || n > kMax || (n > 0 && !jobs)) return MB200_EINVAL;
  all.n = 0;
  blocks = 0;
  for (int i = 0; i < n; ++i) {
    const mb200_convert_job& j = jobs[i];
    if (j.rows < 0 || j.cols < 0 || j.src_cols > j.cols || (j.slices > 1 && (!j.src || j.src_dtype != MB200_F32))) return MB200_EINVAL;
    if ((j.src && j.src_dtype != MB200_F32 && j.src_dtype != MB200_BF16) || (j.dst_dtype != MB200_F32 && j.dst_dtype != MB200_BF16))
      return MB200_EDTYPE;
    if (j.rows == 0 || j.cols == 0) continue;
    if (!j.dst || ((j.op == MB200_CONVERT_MUL || j.op == MB200_CONVERT_ADD) && !j.factor)) return MB200_EINVAL;
    static_cast<mb200_convert_job&>(all.job[all.n]) = j;
    all.job[all.n].vec = (j.rows == 1 || (j.src_stride % 4 == 0 && j.dst_stride % 4 == 0)) && j.cols % 4 == 0 && j.src && j.src_cols == j.cols && aligned16(j.src) && aligned16(j.dst) && aligned16(j.factor) &&
                           (j.slices <= 1 || j.slice_stride % 4 == 0);
    all.first_block[all.n++] = int(blocks);
    blocks += (j.rows * j.cols + kConvertThreads * kPerThread - 1) / (kConvertThreads * kPerThread);
    if (blocks > (int64_t(1) << 30)) return MB200_ETOOBIG;
  }
  all.first_block[all.n] = int(blocks);
  return MB200_OK;
}

}  // namespace
}  // namespace mb200

// RMSNorm over the last dimension, forward and backward:
//     y = x * rsqrt(mean(x^2) + eps) * weight          (mambapy/mamba.py:416-433; weight absent with muP)
// This is the normalisation in front of every MambaBlock (ResidualBlock.forward, mambapy/mamba.py:111)
// and the optional inner normalisation of delta, B, C.  The reference builds it from five elementwise
// and reduction ops; here a row is read once and written once (HBM streaming).
//
// Mapping (vectorised rows up to 8192 wide): kTPR threads share a row and hold ALL of it in registers, four columns a thread
// in each of kC chunks, so every element is read once and written once; one CTA of 256 threads works on 256 / kTPR rows at a
// time.  A thread sees the same columns in every row it takes, so dweight is a sum in its own registers, and only leaves them
// at the end (shared memory over the CTA's row groups, then one atomic per column and CTA).  All arithmetic is float32
// whatever the I/O type.  Measured on B200: backward with the residual gradient, (16384, 768) float32 stream and bfloat16 dy
// 58 -> 31 us (a shared-memory atomic per element bound it); forward (256, 2560) bfloat16 7.3 -> 3.1 us (one warp per row left
// most of the GPU idle).
// Rows that are wider or off the vector grid go through the row-by-row kernels: one warp per row, read twice, the second time
// out of L1/L2.
#include <initializer_list>
#include "common.cuh"

namespace mb200 {
namespace {

constexpr int kNormThreads = 256;
constexpr int kNormWarps = kNormThreads / 32;

template <typename T, int V> struct alignas(sizeof(T) * V) NVec {
  T v[V];
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
  return v;
}

template <typename T, int V>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_fwd_kernel(const T* __restrict__ x, const float* __restrict__ w, T* __restrict__ y,
                   float* __restrict__ rstd, int64_t rows, int64_t D, int64_t x_rs, int64_t y_rs, float eps) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = int64_t(blockIdx.x) * kNormWarps + (threadIdx.x >> 5);
  const int64_t nwarps = int64_t(gridDim.x) * kNormWarps;
  for (int64_t r = warp; r < rows; r += nwarps) {
    const T* xp = x + r * x_rs;
    T* yp = y + r * y_rs;
    float ss = 0.f;
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      const NVec<T, V> v = *reinterpret_cast<const NVec<T, V>*>(xp + d);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float f = Elem<T>::to_f(v.v[i]);
        ss = fmaf(f, f, ss);
      }
    }
    const float rs = rsqrtf(warp_sum(ss) / float(D) + eps);
    if (rstd && lane == 0) rstd[r] = rs;
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      const NVec<T, V> v = *reinterpret_cast<const NVec<T, V>*>(xp + d);
      NVec<T, V> o;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        float f = Elem<T>::to_f(v.v[i]) * rs;
        if (w) f *= w[d + i];
        o.v[i] = Elem<T>::from_f(f);
      }
      *reinterpret_cast<NVec<T, V>*>(yp + d) = o;
    }
  }
}

// dx = (g - xhat * mean(g * xhat)) * rstd with g = dy * weight, xhat = x * rstd;  dweight = sum_rows dy * xhat.
template <typename T, int V, bool kAccW>
__global__ void __launch_bounds__(kNormThreads)
rmsnorm_bwd_kernel(const T* __restrict__ x, const float* __restrict__ w, const float* __restrict__ rstd,
                   const T* __restrict__ dy, T* __restrict__ dx, float* __restrict__ dw, int64_t rows, int64_t D,
                   int64_t x_rs, int64_t dy_rs, int64_t dx_rs) {
  extern __shared__ float s_dw[];               // [D] when kAccW
  const int lane = threadIdx.x & 31;
  const int64_t warp = int64_t(blockIdx.x) * kNormWarps + (threadIdx.x >> 5);
  const int64_t nwarps = int64_t(gridDim.x) * kNormWarps;
  if constexpr (kAccW) {
    for (int64_t d = threadIdx.x; d < D; d += kNormThreads) s_dw[d] = 0.f;
    __syncthreads();
  }
  for (int64_t r = warp; r < rows; r += nwarps) {
    const T* xp = x + r * x_rs;
    const T* gp = dy + r * dy_rs;
    T* op = dx + r * dx_rs;
    const float rs = rstd[r];
    float dot = 0.f;
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      const NVec<T, V> xv = *reinterpret_cast<const NVec<T, V>*>(xp + d);
      const NVec<T, V> gv = *reinterpret_cast<const NVec<T, V>*>(gp + d);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float xh = Elem<T>::to_f(xv.v[i]) * rs;
        const float gy = Elem<T>::to_f(gv.v[i]);
        if constexpr (kAccW) atomicAdd(&s_dw[d + i], gy * xh);
        dot = fmaf(w ? gy * w[d + i] : gy, xh, dot);
      }
    }
    const float m = warp_sum(dot) / float(D);
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      const NVec<T, V> xv = *reinterpret_cast<const NVec<T, V>*>(xp + d);
      const NVec<T, V> gv = *reinterpret_cast<const NVec<T, V>*>(gp + d);
      NVec<T, V> o;
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float xh = Elem<T>::to_f(xv.v[i]) * rs;
        float g = Elem<T>::to_f(gv.v[i]);
        if (w) g *= w[d + i];
        o.v[i] = Elem<T>::from_f((g - xh * m) * rs);
      }
      *reinterpret_cast<NVec<T, V>*>(op + d) = o;
    }
  }
  if constexpr (kAccW) {
    __syncthreads();
    for (int64_t d = threadIdx.x; d < D; d += kNormThreads) atomicAdd(dw + d, s_dw[d]);
  }
}

// ---- residual add fused with the normalisation that follows it -----------------------------------------
// A stack of blocks computes x_{l+1} = mixer(norm(x_l)) + x_l (mambapy/mamba.py:106-112).  Written per
// layer that is an add kernel (read two tensors, write one) followed by the norm (read one, write one);
// fused, the sum is formed in registers:   s = x + res_in;  res_out = s;  y = s * rsqrt(mean(s^2) + eps) * w.
// x (the previous mixer's output), the residual stream and y may have different element types (under
// autocast the mixer's output and y are bfloat16 while the residual stream stays float32).
template <typename T, int V>
__device__ __forceinline__ void load_vec(const T* p, float (&f)[V]) {
  const NVec<T, V> v = *reinterpret_cast<const NVec<T, V>*>(p);
#pragma unroll
  for (int i = 0; i < V; ++i) f[i] = Elem<T>::to_f(v.v[i]);
}
template <typename T, int V>
__device__ __forceinline__ void store_vec(T* p, const float (&f)[V]) {
  NVec<T, V> v;
#pragma unroll
  for (int i = 0; i < V; ++i) v.v[i] = Elem<T>::from_f(f[i]);
  *reinterpret_cast<NVec<T, V>*>(p) = v;
}

template <typename TX, typename TR, typename TY, int V>
__global__ void __launch_bounds__(kNormThreads)
add_rmsnorm_fwd_kernel(const TX* __restrict__ x, const TR* __restrict__ res_in, const float* __restrict__ w,
                       TR* __restrict__ res_out, TY* __restrict__ y, float* __restrict__ rstd, int64_t rows,
                       int64_t D, int64_t x_rs, int64_t ri_rs, int64_t ro_rs, int64_t y_rs, float eps) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = int64_t(blockIdx.x) * kNormWarps + (threadIdx.x >> 5);
  const int64_t nwarps = int64_t(gridDim.x) * kNormWarps;
  for (int64_t r = warp; r < rows; r += nwarps) {
    float ss = 0.f;
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      float a[V], c[V];
      load_vec<TX, V>(x + r * x_rs + d, a);
      if (res_in) {
        load_vec<TR, V>(res_in + r * ri_rs + d, c);
#pragma unroll
        for (int i = 0; i < V; ++i) a[i] += c[i];
      }
      // the sum is rounded to the residual stream's type BEFORE it is normalised, as the reference's
      // separate add would have rounded it
#pragma unroll
      for (int i = 0; i < V; ++i) { a[i] = Elem<TR>::to_f(Elem<TR>::from_f(a[i])); ss = fmaf(a[i], a[i], ss); }
      store_vec<TR, V>(res_out + r * ro_rs + d, a);
    }
    const float rs = rsqrtf(warp_sum(ss) / float(D) + eps);
    if (rstd && lane == 0) rstd[r] = rs;
    __syncwarp();
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {       // second pass out of L1/L2: this lane's own stores
      float a[V];
      load_vec<TR, V>(res_out + r * ro_rs + d, a);
#pragma unroll
      for (int i = 0; i < V; ++i) a[i] = w ? a[i] * rs * w[d + i] : a[i] * rs;
      store_vec<TY, V>(y + r * y_rs + d, a);
    }
  }
}

// ds = (g - shat * mean(g * shat)) * rstd + dres_out, with g = dy * weight and shat = s * rstd: the gradient of
// the sum s, which is the gradient of both x and res_in.  dweight as in rmsnorm_bwd_kernel.
template <typename TR, typename TY, int V, bool kAccW>
__global__ void __launch_bounds__(kNormThreads)
add_rmsnorm_bwd_kernel(const TR* __restrict__ s, const float* __restrict__ w, const float* __restrict__ rstd,
                       const TY* __restrict__ dy, const TR* __restrict__ dres, TR* __restrict__ ds,
                       float* __restrict__ dw, int64_t rows, int64_t D, int64_t s_rs, int64_t dy_rs,
                       int64_t dr_rs, int64_t ds_rs) {
  extern __shared__ float s_dw[];               // [D] when kAccW
  const int lane = threadIdx.x & 31;
  const int64_t warp = int64_t(blockIdx.x) * kNormWarps + (threadIdx.x >> 5);
  const int64_t nwarps = int64_t(gridDim.x) * kNormWarps;
  if constexpr (kAccW) {
    for (int64_t d = threadIdx.x; d < D; d += kNormThreads) s_dw[d] = 0.f;
    __syncthreads();
  }
  for (int64_t r = warp; r < rows; r += nwarps) {
    const float rs = rstd[r];
    float dot = 0.f;
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      float sv[V], gv[V];
      load_vec<TR, V>(s + r * s_rs + d, sv);
      load_vec<TY, V>(dy + r * dy_rs + d, gv);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float sh = sv[i] * rs;
        if constexpr (kAccW) atomicAdd(&s_dw[d + i], gv[i] * sh);
        dot = fmaf(w ? gv[i] * w[d + i] : gv[i], sh, dot);
      }
    }
    const float m = warp_sum(dot) / float(D);
    for (int64_t d = int64_t(lane) * V; d < D; d += 32 * V) {
      float sv[V], gv[V], o[V];
      load_vec<TR, V>(s + r * s_rs + d, sv);
      load_vec<TY, V>(dy + r * dy_rs + d, gv);
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float g = w ? gv[i] * w[d + i] : gv[i];
        o[i] = (g - sv[i] * rs * m) * rs;
      }
      if (dres) {
        float rv[V];
        load_vec<TR, V>(dres + r * dr_rs + d, rv);
#pragma unroll
        for (int i = 0; i < V; ++i) o[i] += rv[i];
      }
      store_vec<TR, V>(ds + r * ds_rs + d, o);
    }
  }
  if constexpr (kAccW) {
    __syncthreads();
    for (int64_t d = threadIdx.x; d < D; d += kNormThreads) atomicAdd(dw + d, s_dw[d]);
  }
}

// ---- rows held in registers -----------------------------------------------------------------------------
struct NormWeight {
  const void* p;
  int dtype;
  __device__ __forceinline__ float4 at4(int64_t d) const {
    if (!p) return make_float4(1.f, 1.f, 1.f, 1.f);
    if (dtype == MB200_F32) return __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(p) + d));
    float f[4];
    load_vec<__nv_bfloat16, 4>(static_cast<const __nv_bfloat16*>(p) + d, f);
    return make_float4(f[0], f[1], f[2], f[3]);
  }
};

// Sum over the kTPR threads of a row; every thread of the CTA calls it (s_part: one float per warp).
template <int kTPR>
__device__ __forceinline__ float row_sum(float v, float* s_part) {
  v = warp_sum(v);
  if constexpr (kTPR > 32) {
    const int warp = threadIdx.x >> 5, first = warp / (kTPR / 32) * (kTPR / 32);
    __syncthreads();                                     // the previous sum has been read
    if ((threadIdx.x & 31) == 0) s_part[warp] = v;
    __syncthreads();
    v = 0.f;
#pragma unroll
    for (int i = 0; i < kTPR / 32; ++i) v += s_part[first + i];
  }
  return v;
}

// s = x (+ res_in), written to res_out when that is given;  y = s * rsqrt(mean(s^2) + eps) * w.
template <typename TX, typename TR, typename TY, int kTPR, int kC>
__global__ void __launch_bounds__(kNormThreads)
norm_rows_fwd_kernel(const TX* __restrict__ x, const TR* __restrict__ res_in, const NormWeight w, TR* __restrict__ res_out,
                     TY* __restrict__ y, float* __restrict__ rstd, int64_t rows, int64_t D, int64_t x_rs, int64_t ri_rs,
                     int64_t ro_rs, int64_t y_rs, float eps) {
  __shared__ float s_part[kNormWarps];
  constexpr int kRows = kNormThreads / kTPR;
  const int64_t r = int64_t(blockIdx.x) * kRows + threadIdx.x / kTPR;
  const int t = threadIdx.x % kTPR;
  const bool ok = r < rows;
  float v[kC][4], ss = 0.f;
#pragma unroll
  for (int c = 0; c < kC; ++c) {
    const int64_t d = (int64_t(c) * kTPR + t) * 4;
    if (ok && d < D) {
      load_vec<TX, 4>(x + r * x_rs + d, v[c]);
      if (res_in) {
        float q[4];
        load_vec<TR, 4>(res_in + r * ri_rs + d, q);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[c][i] += q[i];
      }
    } else {
      v[c][0] = v[c][1] = v[c][2] = v[c][3] = 0.f;
    }
  }
#pragma unroll
  for (int c = 0; c < kC; ++c)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // the sum is rounded to the residual stream's type BEFORE it is normalised, as the reference's separate add would have
      v[c][i] = Elem<TR>::to_f(Elem<TR>::from_f(v[c][i]));
      ss = fmaf(v[c][i], v[c][i], ss);
    }
  const float rs = rsqrtf(row_sum<kTPR>(ss, s_part) / float(D) + eps);
  if (!ok) return;
  if (rstd && t == 0) rstd[r] = rs;
#pragma unroll
  for (int c = 0; c < kC; ++c) {
    const int64_t d = (int64_t(c) * kTPR + t) * 4;
    if (d >= D) continue;
    if (res_out) store_vec<TR, 4>(res_out + r * ro_rs + d, v[c]);
    const float4 g = w.at4(d);
    const float o[4] = {v[c][0] * rs * g.x, v[c][1] * rs * g.y, v[c][2] * rs * g.z, v[c][3] * rs * g.w};
    store_vec<TY, 4>(y + r * y_rs + d, o);
  }
}

// ds = (g - shat * mean(g * shat)) * rstd (+ dres), g = dy * w, shat = s * rstd;  dw = sum over rows of dy * shat.  ds_bf16, when
// given, is ds once more, dense and rounded: the gradient of a bfloat16 mixer output beside that of the float32 stream.
// The grid is one wave of CTAs, so that the rows they walk are few and the dweight atomics too: as many as fit by registers, 3 per SM
// with up to 3 chunks a thread (compiled for that: 88 registers instead of 80 let only two in, and a grid for three then ran in two
// waves), 2 with 4 and 1 with 8.  Some of these spill 8 to 24 bytes for it (3 chunks of float32: 116 us with the spill against 123 for
// two CTAs per SM at 60000 x 768 with a residual gradient, 30.9 / 28.9 at 16384 x 768 without one, 7.4 / 5.5 at 2048; 4 chunks: 36 against
// 51 for one CTA at 16384 x 1024).  us before / after, 12.6 M elements in float32: 53 / 40 at 768 wide, 46 / 38 at 192, 46 / 34 at 2048,
// 54 / 46 at 5120 (with 3 CTAs per SM forced on 4 chunks 46 and 60 at 2048 and 2560, for 34 and 47).
constexpr int norm_bwd_ctas(int chunks) { return chunks <= 3 ? 3 : chunks == 4 ? 2 : 1; }
template <typename TR, typename TY, int kTPR, int kC>
__global__ void __launch_bounds__(kNormThreads, norm_bwd_ctas(kC))
norm_rows_bwd_kernel(const TR* __restrict__ s, const float* __restrict__ w, const float* __restrict__ rstd,
                     const TY* __restrict__ dy, const TR* __restrict__ dres, TR* __restrict__ ds,
                     __nv_bfloat16* __restrict__ ds_bf16, float* __restrict__ dw,
                     int64_t rows, int64_t D, int64_t s_rs, int64_t dy_rs, int64_t dr_rs, int64_t ds_rs) {
  constexpr int kRows = kNormThreads / kTPR;
  __shared__ float s_part[kNormWarps];
  __shared__ __align__(16) float s_dw[kRows > 1 ? kTPR * kC * 4 : 4];
  const int t = threadIdx.x % kTPR, group = threadIdx.x / kTPR;
  const NormWeight weight{w, MB200_F32};
  float acc[kC][4];
#pragma unroll
  for (int c = 0; c < kC; ++c) acc[c][0] = acc[c][1] = acc[c][2] = acc[c][3] = 0.f;
  for (int64_t r0 = int64_t(blockIdx.x) * kRows; r0 < rows; r0 += int64_t(gridDim.x) * kRows) {
    const int64_t r = r0 + group;
    const bool ok = r < rows;
    const float rs = ok ? rstd[r] : 0.f;
    float sv[kC][4], gv[kC][4], dot = 0.f;
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      const int64_t d = (int64_t(c) * kTPR + t) * 4;
      if (ok && d < D) {
        load_vec<TR, 4>(s + r * s_rs + d, sv[c]);
        load_vec<TY, 4>(dy + r * dy_rs + d, gv[c]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) sv[c][i] = gv[c][i] = 0.f;
      }
    }
    float rv[kC][4];
    if (dres) {
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        const int64_t d = (int64_t(c) * kTPR + t) * 4;
        if (ok && d < D) load_vec<TR, 4>(dres + r * dr_rs + d, rv[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      const int64_t d = (int64_t(c) * kTPR + t) * 4;
      const float4 g4 = d < D ? weight.at4(d) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float wv[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sv[c][i] *= rs;
        acc[c][i] = fmaf(gv[c][i], sv[c][i], acc[c][i]);
        gv[c][i] *= wv[i];
        dot = fmaf(gv[c][i], sv[c][i], dot);
      }
    }
    const float m = row_sum<kTPR>(dot, s_part) / float(D);
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      const int64_t d = (int64_t(c) * kTPR + t) * 4;
      if (!ok || d >= D) continue;
      float o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = (gv[c][i] - sv[c][i] * m) * rs + (dres ? rv[c][i] : 0.f);
      store_vec<TR, 4>(ds + r * ds_rs + d, o);
      if (ds_bf16) store_vec<__nv_bfloat16, 4>(ds_bf16 + r * D + d, o);
    }
  }
  if (!dw) return;
  if constexpr (kRows > 1) {
    for (int g = 0; g < kRows; ++g) {                      // the row groups take turns: no atomics in shared memory
      __syncthreads();
      if (group == g) {
#pragma unroll
        for (int c = 0; c < kC; ++c)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float* a = s_dw + (c * kTPR + t) * 4 + i;
            *a = g ? *a + acc[c][i] : acc[c][i];
          }
      }
    }
    __syncthreads();
    for (int64_t d = threadIdx.x; d < D; d += kNormThreads) atomicAdd(dw + d, s_dw[d]);
  } else {
#pragma unroll
    for (int c = 0; c < kC; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t d = (int64_t(c) * kTPR + t) * 4 + i;
        if (d < D) atomicAdd(dw + d, acc[c][i]);
      }
  }
}

// Runs go(threads per row, chunks) with the smallest row layout that holds D columns; false: D needs the row-by-row kernels.
template <int kTPR, int kC> struct RowLayout {};
template <typename F> bool with_row_layout(int64_t D, F&& go) {
  if (D <= 128) go(RowLayout<32, 1>{});
  else if (D <= 256) go(RowLayout<32, 2>{});
  else if (D <= 512) go(RowLayout<64, 2>{});
  else if (D <= 768) go(RowLayout<64, 3>{});
  else if (D <= 1024) go(RowLayout<64, 4>{});
  else if (D <= 2048) go(RowLayout<128, 4>{});
  else if (D <= 4096) go(RowLayout<256, 4>{});
  else if (D <= 8192) go(RowLayout<256, 8>{});
  else return false;
  return true;
}

template <typename TX, typename TR, typename TY>
bool rows_fwd(const void* x, const void* res_in, NormWeight w, void* res_out, void* y, float* rstd, int64_t rows, int64_t D, int64_t x_rs,
              int64_t ri_rs, int64_t ro_rs, int64_t y_rs, float eps, cudaStream_t st) {
  return with_row_layout(D, [&]<int kTPR, int kC>(RowLayout<kTPR, kC>) {
    const int64_t grid = (rows + kNormThreads / kTPR - 1) / (kNormThreads / kTPR);
    norm_rows_fwd_kernel<TX, TR, TY, kTPR, kC><<<unsigned(grid), kNormThreads, 0, st>>>(
        (const TX*)x, (const TR*)res_in, w, (TR*)res_out, (TY*)y, rstd, rows, D, x_rs, ri_rs, ro_rs, y_rs, eps);
  });
}
template <typename TR, typename TY>
bool rows_bwd(const void* s, const float* w, const float* rstd, const void* dy, const void* dres, void* ds, void* ds_bf16, float* dw, int64_t rows, int64_t D,
              int64_t s_rs, int64_t dy_rs, int64_t dr_rs, int64_t ds_rs, cudaStream_t st) {
  return with_row_layout(D, [&]<int kTPR, int kC>(RowLayout<kTPR, kC>) {
    constexpr int kRows = kNormThreads / kTPR;
    const int64_t want = (rows + kRows - 1) / kRows, cap = int64_t(sm_count()) * norm_bwd_ctas(kC);
    norm_rows_bwd_kernel<TR, TY, kTPR, kC><<<unsigned(want < cap ? want : cap), kNormThreads, 0, st>>>(
        (const TR*)s, w, rstd, (const TY*)dy, (const TR*)dres, (TR*)ds, (__nv_bfloat16*)ds_bf16, dw, rows, D, s_rs, dy_rs, dr_rs, ds_rs);
  });
}

int norm_grid(int64_t rows) {
  const int64_t want = (rows + kNormWarps - 1) / kNormWarps;
  const int64_t cap = int64_t(sm_count()) * 8;                    // 8 CTAs of 256 threads per SM
  return int(want < cap ? (want > 0 ? want : 1) : cap);
}

}  // namespace
}  // namespace mb200

using namespace mb200;

static int norm_vec(int64_t D, int es, std::initializer_list<const void*> ptrs, std::initializer_list<int64_t> strides) {
  const int v = 16 / es;
  if (D % v) return 1;
  for (const void* p : ptrs) if (!aligned16(p)) return 1;
  for (int64_t s : strides) if (s % v) return 1;
  return v;
}

// Four columns a thread: every pointer on a 16-byte boundary, every row stride a multiple of 8 elements.
static bool rows_vec(int64_t D, std::initializer_list<const void*> ptrs, std::initializer_list<int64_t> strides) {
  if (D % 4) return false;
  for (const void* p : ptrs) if (!aligned16(p)) return false;
  for (int64_t s : strides) if (s % 8) return false;
  return true;
}

extern "C" int mb200_rmsnorm_fwd(const void* x, const float* weight, void* y, float* rstd, int64_t rows,
                                 int64_t D, int64_t x_rs, int64_t y_rs, float eps, int dtype, void* stream) {
  return mb200_rmsnorm_fwd_typed(x, weight, MB200_F32, y, rstd, rows, D, x_rs, y_rs, eps, dtype, stream);
}

extern "C" int mb200_rmsnorm_fwd_typed(const void* x, const void* weight_, int w_dtype, void* y, float* rstd, int64_t rows,
                                       int64_t D, int64_t x_rs, int64_t y_rs, float eps, int dtype, void* stream) {
  if (rows < 0 || D < 0) return MB200_EINVAL;
  if ((dtype != MB200_F32 && dtype != MB200_BF16) || (w_dtype != MB200_F32 && w_dtype != MB200_BF16)) return MB200_EDTYPE;
  const NormWeight nw{weight_, w_dtype};
  if (rows > 0 && D > 0 && x && y && rows_vec(D, {x, y, weight_}, {x_rs, y_rs})) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    using bf = __nv_bfloat16;
    if (dtype == MB200_F32 ? rows_fwd<float, float, float>(x, nullptr, nw, nullptr, y, rstd, rows, D, x_rs, 0, 0, y_rs, eps, s)
                           : rows_fwd<bf, bf, bf>(x, nullptr, nw, nullptr, y, rstd, rows, D, x_rs, 0, 0, y_rs, eps, s))
      return check_launch();
  }
  if (weight_ && w_dtype != MB200_F32) return MB200_EUNSUPPORTED;          // the row-by-row kernels read a float32 weight
  const float* weight = static_cast<const float*>(weight_);
  if (rows == 0 || D == 0) return MB200_OK;
  if (!x || !y) return MB200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int es = dtype == MB200_F32 ? 4 : 2;
  const int v = norm_vec(D, es, {x, y}, {x_rs, y_rs});
  const int grid = norm_grid(rows);
#define MB200_NORM_FWD(TT, VV) \
  rmsnorm_fwd_kernel<TT, VV><<<grid, kNormThreads, 0, st>>>((const TT*)x, weight, (TT*)y, rstd, rows, D, x_rs, y_rs, eps)
  if (dtype == MB200_F32) { if (v > 1) MB200_NORM_FWD(float, 4); else MB200_NORM_FWD(float, 1); }
  else { if (v > 1) MB200_NORM_FWD(__nv_bfloat16, 8); else MB200_NORM_FWD(__nv_bfloat16, 1); }
#undef MB200_NORM_FWD
  return check_launch();
}

extern "C" int mb200_rmsnorm_bwd(const void* x, const float* weight, const float* rstd, const void* dy, void* dx,
                                 float* dweight, int64_t rows, int64_t D, int64_t x_rs, int64_t dy_rs,
                                 int64_t dx_rs, int dtype, void* stream) {
  if (rows < 0 || D < 0) return MB200_EINVAL;
  if (dtype != MB200_F32 && dtype != MB200_BF16) return MB200_EDTYPE;
  if (rows == 0 || D == 0) return MB200_OK;
  if (!x || !rstd || !dy || !dx) return MB200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int es = dtype == MB200_F32 ? 4 : 2;
  if (rows_vec(D, {x, dy, (const void*)dx, weight}, {x_rs, dy_rs, dx_rs})) {
    using bf = __nv_bfloat16;
    if (dtype == MB200_F32 ? rows_bwd<float, float>(x, weight, rstd, dy, nullptr, dx, nullptr, dweight, rows, D, x_rs, dy_rs, 0, dx_rs, st)
                           : rows_bwd<bf, bf>(x, weight, rstd, dy, nullptr, dx, nullptr, dweight, rows, D, x_rs, dy_rs, 0, dx_rs, st))
      return check_launch();
  }
  const int v = norm_vec(D, es, {x, dy, (const void*)dx}, {x_rs, dy_rs, dx_rs});
  if (dweight && D > 12288) return MB200_ETOOBIG;                    // the CTA's dweight buffer is D floats of static-limit shared memory
  const int grid = norm_grid(rows);
  const size_t smem = dweight ? size_t(D) * sizeof(float) : 0;
#define MB200_NORM_BWD(TT, VV)                                                                             \
  {                                                                                                        \
    if (dweight)                                                                                           \
      rmsnorm_bwd_kernel<TT, VV, true><<<grid, kNormThreads, smem, st>>>((const TT*)x, weight, rstd,      \
          (const TT*)dy, (TT*)dx, dweight, rows, D, x_rs, dy_rs, dx_rs);                                   \
    else                                                                                                   \
      rmsnorm_bwd_kernel<TT, VV, false><<<grid, kNormThreads, 0, st>>>((const TT*)x, weight, rstd,        \
          (const TT*)dy, (TT*)dx, dweight, rows, D, x_rs, dy_rs, dx_rs);                                   \
  }
  if (dtype == MB200_F32) { if (v > 1) MB200_NORM_BWD(float, 4) else MB200_NORM_BWD(float, 1) }
  else { if (v > 1) MB200_NORM_BWD(__nv_bfloat16, 8) else MB200_NORM_BWD(__nv_bfloat16, 1) }
#undef MB200_NORM_BWD
  return check_launch();
}

// Element-type triple of the fused add + norm: (x, residual stream, y), each MB200_F32 or MB200_BF16.
template <typename TX, typename TR, typename TY>
static int add_norm_fwd_launch(const void* x, const void* res_in, const float* weight, void* res_out, void* y,
                               float* rstd, int64_t rows, int64_t D, int64_t x_rs, int64_t ri_rs, int64_t ro_rs,
                               int64_t y_rs, float eps, bool vec, cudaStream_t st) {
  if (vec && aligned16(weight) &&
      rows_fwd<TX, TR, TY>(x, res_in, NormWeight{weight, MB200_F32}, res_out, y, rstd, rows, D, x_rs, ri_rs, ro_rs, y_rs, eps, st))
    return check_launch();
  const int grid = norm_grid(rows);
  if (vec)
    add_rmsnorm_fwd_kernel<TX, TR, TY, 4><<<grid, kNormThreads, 0, st>>>((const TX*)x, (const TR*)res_in, weight,
        (TR*)res_out, (TY*)y, rstd, rows, D, x_rs, ri_rs, ro_rs, y_rs, eps);
  else
    add_rmsnorm_fwd_kernel<TX, TR, TY, 1><<<grid, kNormThreads, 0, st>>>((const TX*)x, (const TR*)res_in, weight,
        (TR*)res_out, (TY*)y, rstd, rows, D, x_rs, ri_rs, ro_rs, y_rs, eps);
  return check_launch();
}

extern "C" int mb200_add_rmsnorm_fwd(const void* x, const void* res_in, const float* weight, void* res_out, void* y,
                                     float* rstd, int64_t rows, int64_t D, int64_t x_rs, int64_t ri_rs, int64_t ro_rs,
                                     int64_t y_rs, float eps, int dtype_x, int dtype_res, int dtype_y, void* stream) {
  if (rows < 0 || D < 0) return MB200_EINVAL;
  for (int dt : {dtype_x, dtype_res, dtype_y})
    if (dt != MB200_F32 && dt != MB200_BF16) return MB200_EDTYPE;
  if (rows == 0 || D == 0) return MB200_OK;
  if (!x || !res_out || !y) return MB200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // 4 elements per access: 16 bytes in float32, 8 in bfloat16; every pointer and stride must allow it
  bool vec = D % 4 == 0;
  for (const void* q : {x, res_in, (const void*)res_out, (const void*)y}) vec = vec && aligned16(q);
  for (int64_t sd : {x_rs, ri_rs, ro_rs, y_rs}) vec = vec && sd % 8 == 0;
  const int key = dtype_x * 4 + dtype_res * 2 + dtype_y;
#define MB200_ADDNORM(TX, TR, TY) \
  return add_norm_fwd_launch<TX, TR, TY>(x, res_in, weight, res_out, y, rstd, rows, D, x_rs, ri_rs, ro_rs, y_rs, eps, vec, st)
  switch (key) {
    case 0: MB200_ADDNORM(float, float, float);
    case 1: MB200_ADDNORM(float, float, __nv_bfloat16);
    case 4: MB200_ADDNORM(__nv_bfloat16, float, float);
    case 5: MB200_ADDNORM(__nv_bfloat16, float, __nv_bfloat16);
    case 7: MB200_ADDNORM(__nv_bfloat16, __nv_bfloat16, __nv_bfloat16);
    default: return MB200_EUNSUPPORTED;     // a residual stream narrower than what is added to it
  }
#undef MB200_ADDNORM
}

template <typename TR, typename TY>
static int add_norm_bwd_launch(const void* s, const float* weight, const float* rstd, const void* dy, const void* dres,
                               void* ds, void* ds_bf16, float* dweight, int64_t rows, int64_t D, int64_t s_rs, int64_t dy_rs,
                               int64_t dr_rs, int64_t ds_rs, bool vec, cudaStream_t st) {
  if (vec && aligned16(weight) &&
      rows_bwd<TR, TY>(s, weight, rstd, dy, dres, ds, ds_bf16, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs, st))
    return check_launch();
  if (ds_bf16) return MB200_EUNSUPPORTED;
  const int grid = norm_grid(rows);
  const size_t smem = dweight ? size_t(D) * sizeof(float) : 0;
#define MB200_GO(VV, ACC)                                                                                         \
  add_rmsnorm_bwd_kernel<TR, TY, VV, ACC><<<grid, kNormThreads, smem, st>>>((const TR*)s, weight, rstd, (const TY*)dy, \
      (const TR*)dres, (TR*)ds, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs)
  if (vec) { if (dweight) MB200_GO(4, true); else MB200_GO(4, false); }
  else { if (dweight) MB200_GO(1, true); else MB200_GO(1, false); }
#undef MB200_GO
  return check_launch();
}

extern "C" int mb200_add_rmsnorm_bwd_both(const void* s, const float* weight, const float* rstd, const void* dy,
                                     const void* dres, void* ds, void* ds_bf16, float* dweight, int64_t rows, int64_t D,
                                     int64_t s_rs, int64_t dy_rs, int64_t dr_rs, int64_t ds_rs, int dtype_res,
                                     int dtype_y, void* stream) {
  if (rows < 0 || D < 0) return MB200_EINVAL;
  for (int dt : {dtype_res, dtype_y})
    if (dt != MB200_F32 && dt != MB200_BF16) return MB200_EDTYPE;
  if (rows == 0 || D == 0) return MB200_OK;
  if (!s || !rstd || !dy || !ds) return MB200_EINVAL;
  if (dweight && D > 12288) return MB200_ETOOBIG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  bool vec = D % 4 == 0;
  for (const void* q : {s, dy, dres, (const void*)ds, (const void*)ds_bf16}) vec = vec && aligned16(q);
  for (int64_t sd : {s_rs, dy_rs, dr_rs, ds_rs}) vec = vec && sd % 8 == 0;
  if (dtype_res == MB200_F32 && dtype_y == MB200_F32)
    return add_norm_bwd_launch<float, float>(s, weight, rstd, dy, dres, ds, ds_bf16, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs, vec, st);
  if (dtype_res == MB200_F32 && dtype_y == MB200_BF16)
    return add_norm_bwd_launch<float, __nv_bfloat16>(s, weight, rstd, dy, dres, ds, ds_bf16, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs, vec, st);
  if (dtype_res == MB200_BF16 && dtype_y == MB200_BF16)
    return add_norm_bwd_launch<__nv_bfloat16, __nv_bfloat16>(s, weight, rstd, dy, dres, ds, ds_bf16, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs, vec, st);
  return MB200_EUNSUPPORTED;
}

extern "C" int mb200_add_rmsnorm_bwd(const void* s, const float* weight, const float* rstd, const void* dy,
                                     const void* dres, void* ds, float* dweight, int64_t rows, int64_t D,
                                     int64_t s_rs, int64_t dy_rs, int64_t dr_rs, int64_t ds_rs, int dtype_res,
                                     int dtype_y, void* stream) {
  return mb200_add_rmsnorm_bwd_both(s, weight, rstd, dy, dres, ds, nullptr, dweight, rows, D, s_rs, dy_rs, dr_rs, ds_rs, dtype_res, dtype_y,
                                    stream);
}

// One decode step of a whole block (in_proj, conv window, x_proj, dt_proj, state update, gate, out_proj) for a few tokens,
// in ONE cooperative launch.
//
// What bounds it.  With one to eight tokens every projection is a matrix-vector product: the step reads each weight once
// (15 MB for d_model 768 in float32) and does next to nothing with it.  Written as separate kernels it is 7 launches of 2 to
// 8 us each whose weights cannot start moving before the launch in front has drained, and host time of about 50 us for them.
// Here the grid stays resident (one CTA per SM) and walks four phases separated by grid barriers; the weights of the later
// phases are pulled into L2 while the first one runs.
//   1  xz = in_proj(x), one warp per row; the lanes that end up with an x channel shift its window and convolve at once
//   2  dbc = x_proj(xc), one warp per row
//   3  delta = dt_proj(dbc), state update, C-contraction, D skip, gate: a group of lanes per (token, channel)
//   4  out = out_proj(y), one warp per row
// Values between phases are rounded to the activation type, as the separate kernels round them.
#include <atomic>
#include <cstddef>
#include "common.cuh"

namespace mb200 {
namespace {

constexpr int kStepThreads = 512;
constexpr int kStepWarps = kStepThreads / 32;
constexpr int kBarrierSpins = 1 << 22;                 // polls at least 32 ns apart: gives up well within a second

__device__ int g_block_step_status = MB200_DEV_OK;

// Counters of the three barriers, zero when a launch comes to them (the third is cleared behind the next launch's first barrier);
// `poisoned` marks a workspace whose launch gave up.
struct StepBarriers {
  unsigned count[3];
  unsigned poisoned;
};

struct StepParams {
  mb200_block_step_args a;
  StepBarriers* bar;
  float *xc, *z, *dbc, *y;                              // scratch: (B, W), (B, W), (B, R + 2 N), (B, W)
};

// All CTAs of the cooperative grid meet.  False when one of them did not arrive within the limit.
__device__ __forceinline__ bool grid_barrier(StepBarriers* bar, int k) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned* c = &bar->count[k];
    __threadfence();
    atomicAdd(c, 1u);
    ok = 0;
    for (int i = 0; i < kBarrierSpins; ++i) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c) : "memory");
      if (v >= gridDim.x) { ok = 1; break; }
      __nanosleep(32);
    }
    if (!ok) {
      atomicExch(&bar->poisoned, 1u);
      atomicExch(&g_block_step_status, MB200_DEV_WAIT_TIMEOUT);
    }
  }
  __syncthreads();
  return ok != 0;
}

__device__ __forceinline__ float ldf(const void* p, int dtype, int64_t i) {
  return dtype == MB200_F32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
template <typename T> __device__ __forceinline__ float rounded(float v) { return Elem<T>::to_f(Elem<T>::from_f(v)); }

// acc[b] += w[row, :] . x[b, :] over this lane's share of the row; x is float32 with row stride xs (shared or global memory).
template <typename T, int kB>
__device__ __forceinline__ void dot_row(const T* __restrict__ w, const float* x, int64_t xs, int64_t K, int lane, float (&acc)[kB]) {
  constexpr int V = Elem<T>::kVec, kUn = 4;
  int64_t k = int64_t(lane) * V;
  for (; k + (kUn - 1) * 32 * V < K; k += kUn * 32 * V) {
    Vec16<T> wv[kUn];
#pragma unroll
    for (int u = 0; u < kUn; ++u) wv[u] = ldg16(w + k + u * 32 * V);
#pragma unroll
    for (int u = 0; u < kUn; ++u)
#pragma unroll
      for (int b = 0; b < kB; ++b)
#pragma unroll
        for (int i = 0; i < V; i += 4) {
          const float4 xv = *reinterpret_cast<const float4*>(x + b * xs + k + u * 32 * V + i);
          acc[b] = fmaf(Elem<T>::to_f(wv[u].v[i]), xv.x, acc[b]);
          acc[b] = fmaf(Elem<T>::to_f(wv[u].v[i + 1]), xv.y, acc[b]);
          acc[b] = fmaf(Elem<T>::to_f(wv[u].v[i + 2]), xv.z, acc[b]);
          acc[b] = fmaf(Elem<T>::to_f(wv[u].v[i + 3]), xv.w, acc[b]);
        }
  }
  for (; k < K; k += 32 * V) {
    const Vec16<T> wv = ldg16(w + k);
#pragma unroll
    for (int b = 0; b < kB; ++b)
#pragma unroll
      for (int i = 0; i < V; ++i) acc[b] = fmaf(Elem<T>::to_f(wv.v[i]), x[b * xs + k + i], acc[b]);
  }
#pragma unroll
  for (int b = 0; b < kB; ++b)
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) acc[b] += __shfl_xor_sync(0xffffffffu, acc[b], s);
}

__device__ __forceinline__ void prefetch_l2(const void* base, int64_t bytes, int64_t tid, int64_t n) {
  for (int64_t o = tid * 128; o < bytes; o += n * 128)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(base) + o));
}

template <typename T, int N, int kB>
__global__ void __launch_bounds__(kStepThreads, 1) block_step_kernel(const StepParams p) {
  const mb200_block_step_args& a = p.a;
  extern __shared__ __align__(16) float s_x[];            // (kB, max(D, W)) float32
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t B = a.B, D = a.D_model, W = a.W, R = a.R, cols = R + 2 * N;
  // Neighbouring rows go to different SMs: a phase with fewer rows than warps, or a few more, then loads all SMs alike, and not the first
  // third of them.  us a launch, rows in blocks / spread: 76 / 61 at 6 tokens 1024 wide in float32, 20.6 / 13.4 at 3 x 256 in bfloat16,
  // 172 / 153 at 8 x 2048, 191 / 180 at 1 x 2560 (four layers, bfloat16), 16.1 / 15.2 at 1 x 768.
  const int64_t gwarp = int64_t(warp) * gridDim.x + blockIdx.x, nwarps = int64_t(gridDim.x) * kStepWarps;
  if (*reinterpret_cast<volatile unsigned*>(&p.bar->poisoned)) {
    if (threadIdx.x == 0) atomicExch(&g_block_step_status, MB200_DEV_WAIT_TIMEOUT);
    return;
  }
  auto stage = [&](const float* src, int64_t len) {       // (B, len) of the scratch into shared memory, missing tokens as zeros
    for (int64_t i = threadIdx.x; i < kB * len; i += kStepThreads) s_x[i] = i < B * len ? __ldcg(src + i) : 0.f;
    __syncthreads();
  };

  // ---- 1: in_proj, conv window, convolution
  for (int64_t i = threadIdx.x; i < kB * D; i += kStepThreads) {
    const int64_t b = i / D, d = i - b * D;
    s_x[i] = b < B ? Elem<T>::to_f(static_cast<const T*>(a.x)[b * a.x_sb + d]) : 0.f;
  }
  __syncthreads();
  // (with four rows a warp and more every SM is busy, and rows that follow each other in memory stream better: 108.5 / 109.8 at 1 x 2560, float32)
  const bool many = 2 * W >= 4 * nwarps;
  for (int64_t r = many ? int64_t(blockIdx.x) * kStepWarps + warp : gwarp; r < 2 * W; r += nwarps) {
    float acc[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) acc[b] = 0.f;
    dot_row<T, kB>(static_cast<const T*>(a.in_w) + r * D, s_x, D, D, lane, acc);
    float mine = 0.f;
#pragma unroll
    for (int b = 0; b < kB; ++b)
      if (lane == b) mine = acc[b];
    if (lane < B) {
      const float v = rounded<T>(mine + (a.in_b ? Elem<T>::to_f(static_cast<const T*>(a.in_b)[r]) : 0.f));
      if (r >= W) {
        p.z[lane * W + r - W] = v;
      } else {
        const int K = a.d_conv;
        const T* win = static_cast<const T*>(a.conv_in) + (lane * W + r) * (K - 1);
        T* out = static_cast<T*>(a.conv_out) + (lane * W + r) * (K - 1);
        float c = a.conv_b ? ldf(a.conv_b, a.conv_b_dtype, r) : 0.f;
        for (int k = 0; k < K - 1; ++k) {
          const float wv = Elem<T>::to_f(win[k]);
          c = fmaf(ldf(a.conv_w, a.conv_w_dtype, r * K + k), wv, c);
          if (k > 0) out[k - 1] = win[k];
        }
        c = fmaf(ldf(a.conv_w, a.conv_w_dtype, r * K + K - 1), v, c);
        if (K > 1) out[K - 2] = Elem<T>::from_f(v);
        p.xc[lane * W + r] = rounded<T>(c * sigmoidf(c));
      }
    }
  }
  {                                                       // what the later phases read, while others finish this one
    const int64_t t = int64_t(blockIdx.x) * kStepThreads + threadIdx.x, n = int64_t(gridDim.x) * kStepThreads;
    prefetch_l2(a.xproj_w, cols * W * sizeof(T), t, n);
    prefetch_l2(a.dt_w, W * R * sizeof(T), t, n);
    prefetch_l2(a.out_w, D * W * sizeof(T), t, n);
  }
  if (!grid_barrier(p.bar, 0)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) p.bar->count[2] = 0;        // nobody is near the third barrier yet

  // ---- 2: x_proj
  if (int64_t(blockIdx.x) < cols) stage(p.xc, W);            // CTAs without a row go straight to the barrier
  for (int64_t r = gwarp; r < cols; r += nwarps) {
    float acc[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) acc[b] = 0.f;
    dot_row<T, kB>(static_cast<const T*>(a.xproj_w) + r * W, s_x, W, W, lane, acc);
    float mine = 0.f;
#pragma unroll
    for (int b = 0; b < kB; ++b)
      if (lane == b) mine = acc[b];
    if (lane < B) p.dbc[lane * cols + r] = rounded<T>(mine);
  }
  if (!grid_barrier(p.bar, 1)) return;

  // ---- 3: dt_proj, state update, gate; kG lanes per (token, channel), kSt states a lane
  {
    constexpr int kG = N < 32 ? N : 32, kSt = N / kG, kPerWarp = 32 / kG;
    const int g = lane / kG, gl = lane % kG;
    const int64_t items = B * W;
    for (int64_t i0 = gwarp * kPerWarp; i0 < items; i0 += nwarps * kPerWarp) {
      const int64_t i = i0 + g < items ? i0 + g : items - 1;             // a group past the end repeats the last item
      const bool ok = i0 + g < items;
      const int64_t b = i / W, e = i - b * W;
      float h[kSt], A[kSt];
#pragma unroll
      for (int s = 0; s < kSt; ++s) {
        h[s] = a.h_in ? __ldcs(a.h_in + (b * W + e) * N + gl * kSt + s) : 0.f;
        A[s] = ldf(a.A_log, a.A_log_dtype, e * N + gl * kSt + s);
      }
      const float* row = p.dbc + b * cols;
      float dv = 0.f;
      for (int64_t r = gl; r < R; r += kG) dv = fmaf(Elem<T>::to_f(static_cast<const T*>(a.dt_w)[e * R + r]), __ldcg(row + r), dv);
#pragma unroll
      for (int s = kG / 2; s >= 1; s >>= 1) dv += __shfl_xor_sync(0xffffffffu, dv, s, kG);
      dv = softplus_fast(rounded<T>(dv) + ldf(a.dt_b, a.dt_b_dtype, e));
      const float xv = __ldcg(p.xc + b * W + e), dx = dv * xv;
      float yv = 0.f;
#pragma unroll
      for (int s = 0; s < kSt; ++s) {
        const int n = gl * kSt + s;
        const float dec = ex2f(dv * (-expf(A[s])) * kLog2e);
        h[s] = fmaf(dec, h[s], dx * __ldcg(row + R + n));
        yv = fmaf(h[s], __ldcg(row + R + N + n), yv);
        if (ok) __stcs(a.h_out + (b * W + e) * N + n, h[s]);
      }
#pragma unroll
      for (int s = kG / 2; s >= 1; s >>= 1) yv += __shfl_xor_sync(0xffffffffu, yv, s, kG);
      if (ok && gl == 0) {
        yv = fmaf(ldf(a.D, a.D_dtype, e), xv, yv);
        const float zv = __ldcg(p.z + b * W + e);
        p.y[b * W + e] = rounded<T>(yv * zv * sigmoid_fast(zv));
      }
    }
  }
  if (!grid_barrier(p.bar, 2)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) p.bar->count[0] = p.bar->count[1] = 0;

  // ---- 4: out_proj
  if (int64_t(blockIdx.x) >= D) return;
  stage(p.y, W);
  for (int64_t r = gwarp; r < D; r += nwarps) {
    float acc[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) acc[b] = 0.f;
    dot_row<T, kB>(static_cast<const T*>(a.out_w) + r * W, s_x, W, W, lane, acc);
    float mine = 0.f;
#pragma unroll
    for (int b = 0; b < kB; ++b)
      if (lane == b) mine = acc[b];
    if (lane < B)
      static_cast<T*>(a.out)[lane * D + r] = Elem<T>::from_f(mine + (a.out_b ? Elem<T>::to_f(static_cast<const T*>(a.out_b)[r]) : 0.f));
  }
}

template <typename T, int N, int kB>
int block_step_launch(StepParams& p, cudaStream_t st) {
  auto k = block_step_kernel<T, N, kB>;
  const int64_t len = p.a.D_model > p.a.W ? p.a.D_model : p.a.W;
  const int smem = int(kB * len * 4);
  // 48 KB are there without asking, for the kernel's own few static bytes (a barrier's answer) as well
  if (smem > 47 * 1024 && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return MB200_ELAUNCH;
  void* args[] = {&p};
  if (cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(unsigned(sm_count())), dim3(kStepThreads), args, size_t(smem), st) ==
      cudaSuccess)
    return MB200_OK;
  (void)cudaGetLastError();                              // not for the next launch to find
  return MB200_ELAUNCH;
}

template <typename T, int N>
int block_step_batch(StepParams& p, cudaStream_t st) {
  if (p.a.B == 1) return block_step_launch<T, N, 1>(p, st);
  if (p.a.B == 2) return block_step_launch<T, N, 2>(p, st);
  if (p.a.B <= 4) return block_step_launch<T, N, 4>(p, st);
  return block_step_launch<T, N, 8>(p, st);
}
template <typename T>
int block_step_states(StepParams& p, cudaStream_t st) {
  switch (p.a.N) {
    case 8: return block_step_batch<T, 8>(p, st);
    case 16: return block_step_batch<T, 16>(p, st);
    case 32: return block_step_batch<T, 32>(p, st);
    case 64: return block_step_batch<T, 64>(p, st);
    default: return MB200_ENSTATE;
  }
}

}  // namespace
}  // namespace mb200

using namespace mb200;

static std::atomic<unsigned> g_block_step_give_ups{0};

// Reads and clears the status word of the step kernel.  Synchronises the device.
int mb200_block_step_device_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_block_step_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) {
    cudaMemcpyToSymbol(g_block_step_status, &zero, sizeof(int));
    g_block_step_give_ups.fetch_add(1);
  }
  return v;
}
extern "C" unsigned mb200_block_step_give_ups(void) { return g_block_step_give_ups.load(); }
extern "C" int mb200_selftest_block_step_give_up(void* barriers, void* stream) {
  if (!barriers) return MB200_EINVAL;
  char* word = static_cast<char*>(barriers) + offsetof(StepBarriers, poisoned);
  return cudaMemsetAsync(word, 1, sizeof(unsigned), static_cast<cudaStream_t>(stream)) == cudaSuccess ? MB200_OK : MB200_ELAUNCH;
}

extern "C" int64_t mb200_block_step_scratch_floats(int64_t B, int64_t W, int64_t R, int N) { return B * (3 * W + R + 2 * N); }
extern "C" int mb200_block_step_barrier_bytes(void) { return int(sizeof(StepBarriers)); }

extern "C" int mb200_block_step(const mb200_block_step_args* args, float* scratch, void* barriers, void* stream) {
  if (!args || !scratch || !barriers) return MB200_EINVAL;
  const mb200_block_step_args& a = *args;
  if (a.B < 1 || a.D_model < 1 || a.W < 1 || a.R < 1 || a.d_conv < 1) return MB200_EINVAL;
  if (a.dtype != MB200_F32 && a.dtype != MB200_BF16) return MB200_EDTYPE;
  for (int d : {a.conv_w_dtype, a.conv_b_dtype, a.dt_b_dtype, a.A_log_dtype, a.D_dtype})
    if (d != MB200_F32 && d != MB200_BF16) return MB200_EDTYPE;
  if (!a.x || !a.in_w || !a.conv_w || !a.xproj_w || !a.dt_w || !a.dt_b || !a.A_log || !a.D || !a.out_w || !a.h_out || !a.out ||
      (a.d_conv > 1 && (!a.conv_in || !a.conv_out)))
    return MB200_EINVAL;
  // 16-byte weight rows; the activations of all tokens fit shared memory
  const int64_t v = a.dtype == MB200_F32 ? 4 : 8, len = a.D_model > a.W ? a.D_model : a.W, slots = a.B <= 2 ? a.B : a.B <= 4 ? 4 : 8;
  if (a.B > 8 || a.d_conv > 8 || slots * len * 4 > 200 * 1024) return MB200_ETOOBIG;       // the filter as in mb200_conv_step
  if (a.D_model % v || a.W % v || !aligned16(a.in_w) || !aligned16(a.xproj_w) || !aligned16(a.out_w)) return MB200_EUNSUPPORTED;
  StepParams p;
  p.a = a;
  p.bar = static_cast<StepBarriers*>(barriers);
  p.xc = scratch;
  p.z = p.xc + a.B * a.W;
  p.y = p.z + a.B * a.W;
  p.dbc = p.y + a.B * a.W;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return a.dtype == MB200_F32 ? block_step_states<float>(p, st) : block_step_states<__nv_bfloat16>(p, st);
}

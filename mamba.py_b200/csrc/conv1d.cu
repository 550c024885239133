// Depthwise causal conv1d + SiLU on (B, L, ED) tensors, forward and backward, for d_conv = 4:
//     y[b,t,e] = silu( bias[e] + sum_k w[e,k] * x[b, t-3+k, e] ),   x[b, t<0, e] = 0.
// This is the step in front of the selective scan in MambaBlock.forward (mambapy/mamba.py:217-221),
// done there as transpose -> nn.Conv1d(padding=3) -> slice -> transpose -> F.silu.  Here it runs in the
// (B, L, ED) layout the block already has: one read of x and one write of y (HBM-bound streaming).
//
// Mapping: a thread owns a vector of V channels and walks a chunk of `chunk` timesteps with the
// 4-wide window of each channel in registers; a warp covers 32 neighbouring vectors of one chunk, so
// it reads whole contiguous rows.  Chunks are short: the tensors are only (B, L, ED), and HBM bandwidth
// needs tens of thousands of independent loads in flight, which only many short chunks provide; the
// 3-step halo each chunk re-reads comes out of L2.  For the backward the host picks the chunk length
// (a multiple of 4) so that the warps fill the GPU in whole waves.  Loads of a group of timesteps
// are issued together, ahead of the arithmetic.
// The backward walks a chunk with two windows (x and d(pre), both behind), recomputing the
// pre-activation; the 4 warps of a CTA take 4 consecutive chunks of the same channels and add their
// sums for dw and dbias in shared memory first, so global memory sees one atomic per CTA and value.
#include <initializer_list>
#include <type_traits>
#include "common.cuh"

namespace mb200 {
namespace {

constexpr int kConvK = 4;
constexpr int kConvThreads = 256;
// Forward chunks (compile time: the loop over one is fully unrolled).  The longer one saves halo and CTAs, the shorter one has half
// the latency, so 64 steps are taken where they put fewer CTAs on the busiest SM (beyond the three that an SM holds, in whole waves)
// and fewer steps, added over its warps that have a chunk.  us with 32 / 64 steps, bfloat16: 8 x 300 x 1536 (2 CTAs or 1, which has 5
// warps with work) 8.9 / 7.5, 42 x 265 x 512 (3 / 2) 12.7 / 9.1, 4 x 777 x 2048 (2 / 1) 9.1 / 8.2, 8 x 2048 x 1536 (6 / 3) 23.4 / 22.5, but
// 8 x 1003 x 1536 (3 / 2) 12.8 / 14.0, 64 x 197 x 384 (2 / 2) 8.8 / 8.3, 1 x 98 x 512 (1 / 1) 3.8 / 5.4.  Over 100 shapes of 33 to 8192
// steps, both types, this takes 0.3 % longer than the better one on average and 10 % at most (by waves of CTAs alone 2.3 and 43).
constexpr int kConvChunkFwd[2] = {32, 64};
// Timesteps whose loads are in flight together.  Forward 8 (with 3 CTAs of 256 threads per SM): 29.5 us on the 130m layer
// against 33.8 for 4.  Backward 4 (with 4 CTAs of 128 threads): 60 us; 6 and 8 need more registers than 16 warps per SM leave
// and measured 71 and 75, walking backwards with CTAs of 256 threads 69.
constexpr int kConvGroup = 8, kConvGroupBwd = 4;
constexpr int kConvBwdThreads = 128;

static_assert(kConvChunkFwd[0] % kConvGroup == 0 && kConvChunkFwd[1] % kConvGroup == 0, "a chunk is a whole number of groups");

template <typename T, int V> struct alignas(sizeof(T) * V) CVec {
  T v[V];
};
template <typename T, int V>
__device__ __forceinline__ CVec<T, V> cload(const T* p, bool ok) {
  CVec<T, V> r;
  if (!ok) {
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = Elem<T>::from_f(0.f);
  } else if constexpr (sizeof(T) * V == 16) {
    *reinterpret_cast<uint4*>(&r) = __ldg(reinterpret_cast<const uint4*>(p));
  } else if constexpr (sizeof(T) * V == 8) {
    *reinterpret_cast<uint2*>(&r) = __ldg(reinterpret_cast<const uint2*>(p));
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = __ldg(p + i);
  }
  return r;
}
template <typename T, int V>
__device__ __forceinline__ void cstore(T* p, const CVec<T, V>& r) {
  if constexpr (sizeof(T) * V == 16) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(&r);
  else if constexpr (sizeof(T) * V == 8) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(&r);
  else {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = r.v[i];
  }
}

// W channels of float arithmetic in one value: W = 2 uses the packed f32x2 instructions (one issue
// slot for two channels; these kernels would otherwise be bound by instruction issue, not by HBM).
template <int W> struct Pk;
template <> struct Pk<1> {
  float v;
  __device__ __forceinline__ static Pk splat(float a) { return {a}; }
  __device__ __forceinline__ static Pk load(const float* p, int stride) { return {p[0]}; }
  __device__ __forceinline__ float sum() const { return v; }
};
template <> struct Pk<2> {
  float2 v;
  __device__ __forceinline__ static Pk splat(float a) { return {make_float2(a, a)}; }
  __device__ __forceinline__ static Pk load(const float* p, int stride) { return {make_float2(p[0], p[stride])}; }
};
__device__ __forceinline__ Pk<1> pfma(Pk<1> a, Pk<1> b, Pk<1> c) { return {fmaf(a.v, b.v, c.v)}; }
__device__ __forceinline__ Pk<1> pmul(Pk<1> a, Pk<1> b) { return {a.v * b.v}; }
__device__ __forceinline__ Pk<1> padd(Pk<1> a, Pk<1> b) { return {a.v + b.v}; }
__device__ __forceinline__ Pk<1> psigmoid(Pk<1> a) { return {sigmoid_fast(a.v)}; }
__device__ __forceinline__ Pk<2> pfma(Pk<2> a, Pk<2> b, Pk<2> c) { return {__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ Pk<2> pmul(Pk<2> a, Pk<2> b) { return {__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ Pk<2> padd(Pk<2> a, Pk<2> b) { return {__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ Pk<2> psigmoid(Pk<2> a) {
  const float2 m = __fmul2_rn(a.v, make_float2(-kLog2e, -kLog2e));
  const float2 d = __fadd2_rn(make_float2(ex2f(m.x), ex2f(m.y)), make_float2(1.f, 1.f));
  return {make_float2(rcpf(d.x), rcpf(d.y))};
}
// V raw elements <-> V/W packs
template <typename T, int V, int W>
__device__ __forceinline__ void unpack(const CVec<T, V>& r, Pk<W> (&o)[V / W]) {
#pragma unroll
  for (int i = 0; i < V / W; ++i) {
    if constexpr (W == 1) o[i].v = Elem<T>::to_f(r.v[i]);
    else o[i].v = pair_f(&r.v[2 * i]);
  }
}
template <typename T, int V, int W>
__device__ __forceinline__ CVec<T, V> pack(const Pk<W> (&o)[V / W]) {
  CVec<T, V> r;
#pragma unroll
  for (int i = 0; i < V / W; ++i) {
    if constexpr (W == 1) r.v[i] = Elem<T>::from_f(o[i].v);
    else if constexpr (sizeof(T) == 2) {
      *reinterpret_cast<__nv_bfloat162*>(&r.v[2 * i]) = __floats2bfloat162_rn(o[i].v.x, o[i].v.y);
    } else { r.v[2 * i] = o[i].v.x; r.v[2 * i + 1] = o[i].v.y; }
  }
  return r;
}

// grid: x = ceil(nvec / 32) channel groups, y = ceil(nchunk / 8), z = batch; warp w of a CTA takes chunk 8*y + w
template <typename T, int V, int kChunkLen>
__global__ void __launch_bounds__(kConvThreads, 3)
conv1d_silu_fwd_kernel(const T* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       T* __restrict__ y, int64_t L, int64_t ED, int64_t x_sb, int64_t x_sl,
                       int64_t y_sb, int64_t y_sl) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t e = (int64_t(blockIdx.x) * 32 + lane) * V;
  const int64_t t0 = (int64_t(blockIdx.y) * (kConvThreads / 32) + warp) * kChunkLen;
  if (e >= ED || t0 >= L) return;
  const int64_t b = blockIdx.z;
  constexpr int W = (V % 2 == 0) ? 2 : 1, P = V / W;
  using F = Pk<W>;
  F wk[P][kConvK], bv[P], win[P][kConvK - 1];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    bv[i] = bias ? F::load(bias + e + W * i, 1) : F::splat(0.f);
#pragma unroll
    for (int k = 0; k < kConvK; ++k) wk[i][k] = F::load(w + (e + W * i) * kConvK + k, kConvK);
  }
  const T* xp = x + b * x_sb + e + t0 * x_sl;
  T* yp = y + b * y_sb + e + t0 * y_sl;
#pragma unroll
  for (int k = 0; k < kConvK - 1; ++k) {                  // x[t0-3 .. t0-1]
    F xv[P];
    unpack<T, V, W>(cload<T, V>(xp + (k - (kConvK - 1)) * x_sl, t0 > 0), xv);
#pragma unroll
    for (int i = 0; i < P; ++i) win[i][k] = xv[i];
  }
  // Whole chunks (all but a row's last) test nothing; their loop is fully unrolled, so that the compiler hoists the loads of later
  // groups over the arithmetic of earlier ones (28.1 -> 25.4 us, see above, together with moving pointers).
  auto group = [&](auto whole, int left) {
    CVec<T, V> v[kConvGroup];
#pragma unroll
    for (int j = 0; j < kConvGroup; ++j) {
      v[j] = cload<T, V>(xp, decltype(whole)::value || j < left);
      xp += x_sl;
    }
#pragma unroll
    for (int j = 0; j < kConvGroup; ++j) {
      F xn[P], o[P];
      unpack<T, V, W>(v[j], xn);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        F acc = pfma(wk[i][0], win[i][0], bv[i]);
        acc = pfma(wk[i][1], win[i][1], acc);
        acc = pfma(wk[i][2], win[i][2], acc);
        acc = pfma(wk[i][3], xn[i], acc);
        win[i][0] = win[i][1]; win[i][1] = win[i][2]; win[i][2] = xn[i];
        o[i] = pmul(acc, psigmoid(acc));
      }
      if (decltype(whole)::value || j < left) cstore<T, V>(yp, pack<T, V, W>(o));
      yp += y_sl;
    }
  };
  const int left = int(min64(L - t0, kChunkLen));
  // A row's last chunk takes 1, 2, 4 or (of 64 steps) 6 or 8 groups with bounds, unrolled as well.  One group at a time leaves 8 rows in
  // flight and always all of them issues loads that read nothing; us so / so / by what is left, bfloat16: 64 x 31 x 1536
  // 10.1 / 6.5 / 6.2, 64 x 7 x 1536 4.3 / 6.0 / 3.5, 64 x 127 x 768 9.1 / 7.6 / 7.5, 8 x 2041 x 1536 27.0 / 23.6 / 22.3.  (33 to 48 steps in 8 groups
  // instead of 6: 23 x 289 x 378 5.1 us for 4.3.)
  auto groups = [&](auto count, auto whole) {
#pragma unroll
    for (int g = 0; g < decltype(count)::value; ++g) group(whole, left - g * kConvGroup);
  };
  using All = std::integral_constant<int, kChunkLen / kConvGroup>;
  if (left == kChunkLen) groups(All{}, std::true_type{});
  else if (left <= kConvGroup) groups(std::integral_constant<int, 1>{}, std::false_type{});
  else if (left <= 2 * kConvGroup) groups(std::integral_constant<int, 2>{}, std::false_type{});
  else if (kChunkLen == 4 * kConvGroup || left <= 4 * kConvGroup) groups(std::integral_constant<int, 4>{}, std::false_type{});
  else if (left <= 6 * kConvGroup) groups(std::integral_constant<int, 6>{}, std::false_type{});
  else groups(All{}, std::false_type{});
}

// dx[t] = sum_k w[k] * dpre[t+3-k];  dw[k] = sum_{b,t} dpre[t] * x[t-3+k];  dbias = sum dpre;
// dpre[t] = dy[t] * silu'(pre[t]),  pre recomputed from x.
// kLong: chunks long enough to pay for code of their own, which short ones spend more time fetching than running.
//   bfloat16, four channels: the next group's loads are in flight during a group's arithmetic (kAhead), and groups inside the chunk
//   test nothing (kWhole): 8 x 2048 x 1536 41.8 -> 37.7 us, 64 x 1024 x 2048 207 -> 177 against neither; with the loop unrolled by two
//   instead of handing the loaded group on, 72 bytes spilled and 41.6 and 202.  One channel a thread has kWhole alone (84.6 -> 83.2).
//   float32, four channels, has no registers for loads ahead (70 us for 56) and no use for kWhole: whole loads without bounds alone.
// Short ones without any of it: 64 x 31 x 1536 16.0 -> 15.0 us in bfloat16, 17.0 -> 15.4 in float32.
template <typename T, int V, bool kLong>
__global__ void __launch_bounds__(kConvBwdThreads, 4)
conv1d_silu_bwd_kernel(const T* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                       const T* __restrict__ dy, T* __restrict__ dx, float* __restrict__ dw,
                       float* __restrict__ dbias, int64_t L, int64_t ED, int64_t x_sb, int64_t x_sl,
                       int64_t dy_sb, int64_t dy_sl, int64_t dx_sb, int64_t dx_sl, int chunk) {
  constexpr bool kAhead = kLong && sizeof(T) == 2 && V > 1, kWhole = kLong && (sizeof(T) == 2 || V == 1);
  __shared__ float s_acc[32 * V * (kConvK + 1)];          // per channel of the CTA: dw[0..3], dbias
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 32 * V * (kConvK + 1); i += kConvBwdThreads) s_acc[i] = 0.f;
  __syncthreads();
  const int64_t e = (int64_t(blockIdx.x) * 32 + lane) * V;
  const int64_t t0 = (int64_t(blockIdx.y) * (kConvBwdThreads / 32) + warp) * chunk;
  const int64_t t1 = min64(L, t0 + chunk);
  const int64_t b = blockIdx.z;
  if (e < ED && t0 < L) {
    constexpr int W = (V % 2 == 0) ? 2 : 1, P = V / W;
    using F = Pk<W>;
    F wk[P][kConvK], bv[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      bv[i] = bias ? F::load(bias + e + W * i, 1) : F::splat(0.f);
#pragma unroll
      for (int k = 0; k < kConvK; ++k) wk[i][k] = F::load(w + (e + W * i) * kConvK + k, kConvK);
    }
    // Two and a half times the instructions of the arithmetic went into bounds, row addresses and shifting the windows: 47 -> 42 us on
    // 8 x 2048 x 1536 in bfloat16, 16.2 -> 14.6 on 64 x 197 x 384.
    // Time is walked forwards in groups of kConvGroupBwd steps whose loads go out together; dx trails by three steps, because
    // dx[t-3] needs dpre[t-3 .. t].  The windows hold four steps, as many as a group, so that every slot is known at compile time.
    constexpr int kG = kConvGroupBwd, kH = kConvK - 1;
    static_assert(kG == kConvK, "window slots repeat with the groups");
    F xw[P][kG], dw_[P][kG], dwacc[P][kConvK], dbacc[P];
#pragma unroll
    for (int i = 0; i < P; ++i) {
      dbacc[i] = F::splat(0.f);
#pragma unroll
      for (int k = 0; k < kConvK; ++k) dwacc[i][k] = F::splat(0.f);
#pragma unroll
      for (int k = 0; k < kG; ++k) dw_[i][k] = F::splat(0.f);
    }
    const T* xg = x + b * x_sb + e + t0 * x_sl;
    const T* gg = dy + b * dy_sb + e + t0 * dy_sl;
    T* og = dx + b * dx_sb + e + (t0 - kH) * dx_sl;
#pragma unroll
    for (int k = 0; k < kH; ++k) {                         // x[t0-3 .. t0-1]
      F xv[P];
      unpack<T, V, W>(cload<T, V>(xg + (k - kH) * x_sl, t0 > 0), xv);
#pragma unroll
      for (int i = 0; i < P; ++i) xw[i][k + 1] = xv[i];
    }
    const F one = F::splat(1.f), mone = F::splat(-1.f);
    struct Group { CVec<T, V> x[kG], g[kG]; };
    // Steps counted from t0: `own` of them belong to the chunk.  The three behind them only produce dpre for the chunk's last
    // outputs: their own dx, dw belong to the next chunk.  (x, dy read as 0 past the end of the row.)
    const int own = int(t1 - t0), end = int(min64(L, t1 + kH) - t0);
    auto fetch = [&](int s0, Group& q) {
      if (kLong && !kAhead && s0 + kG <= end) {
#pragma unroll
        for (int j = 0; j < kG; ++j) {
          q.x[j] = cload<T, V>(xg, true);
          q.g[j] = cload<T, V>(gg, true);
          xg += x_sl; gg += dy_sl;
        }
      } else {
#pragma unroll
        for (int j = 0; j < kG; ++j) {
          q.x[j] = cload<T, V>(xg, s0 + j < end);
          q.g[j] = cload<T, V>(gg, s0 + j < end);
          xg += x_sl; gg += dy_sl;
        }
      }
    };
    auto group = [&](auto inside, int s0, const Group& q) {
      constexpr bool kIn = decltype(inside)::value;        // every step and every output of the group belongs to the chunk
#pragma unroll
      for (int j = 0; j < kG; ++j) {
        F g[P], xn[P], o[P];
        unpack<T, V, W>(q.g[j], g);
        unpack<T, V, W>(q.x[j], xn);
#pragma unroll
        for (int i = 0; i < P; ++i) {
          xw[i][j] = xn[i];
          F pre = bv[i];
#pragma unroll
          for (int k = 0; k < kConvK; ++k) pre = pfma(wk[i][k], xw[i][(j + 1 + k) % kG], pre);
          const F sg = psigmoid(pre);
          // dpre = dy * s * (1 + pre * (1 - s));  dy is 0 past the end
          const F dp = pmul(pmul(g[i], sg), pfma(pre, pfma(sg, mone, one), one));
          dw_[i][j] = dp;
          // dx[t-3] = w3*dpre[t-3] + w2*dpre[t-2] + w1*dpre[t-1] + w0*dpre[t]
          F acc = pmul(wk[i][0], dp);
#pragma unroll
          for (int k = 1; k < kConvK; ++k) acc = pfma(wk[i][k], dw_[i][(j + kG - k) % kG], acc);
          o[i] = acc;
          if (kIn || s0 + j < own) {
            dbacc[i] = padd(dbacc[i], dp);
#pragma unroll
            for (int k = 0; k < kConvK; ++k) dwacc[i][k] = pfma(dp, xw[i][(j + 1 + k) % kG], dwacc[i][k]);
          }
        }
        if (kIn || (s0 + j >= kH && s0 + j - kH < own)) cstore<T, V>(og, pack<T, V, W>(o));
        og += dx_sl;
      }
    };
    auto run = [&](int s0, const Group& q) {
      if (kWhole && s0 >= kH && s0 + kG <= own) group(std::true_type{}, s0, q);
      else group(std::false_type{}, s0, q);
    };
    if constexpr (kAhead) {
      Group q, next;
      fetch(0, q);
#pragma unroll 1
      for (int s0 = 0; s0 < own + kH; s0 += kG) {
        fetch(s0 + kG, next);
        run(s0, q);
        q = next;
      }
    } else {
#pragma unroll 1
      for (int s0 = 0; s0 < own + kH; s0 += kG) {
        Group q;
        fetch(s0, q);
        run(s0, q);
      }
    }
#pragma unroll
    for (int i = 0; i < P; ++i) {
#pragma unroll
      for (int u = 0; u < W; ++u) {
        float* a = s_acc + (lane * V + i * W + u) * (kConvK + 1);
#pragma unroll
        for (int k = 0; k < kConvK; ++k) {
          float val;
          if constexpr (W == 1) val = dwacc[i][k].v; else val = u ? dwacc[i][k].v.y : dwacc[i][k].v.x;
          atomicAdd(a + k, val);
        }
        float dbv;
        if constexpr (W == 1) dbv = dbacc[i].v; else dbv = u ? dbacc[i].v.y : dbacc[i].v.x;
        atomicAdd(a + kConvK, dbv);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * V * (kConvK + 1); i += kConvBwdThreads) {
    const int64_t ch = int64_t(blockIdx.x) * 32 * V + i / (kConvK + 1);
    const int k = i % (kConvK + 1);
    if (ch >= ED) continue;
    if (k < kConvK) atomicAdd(dw + ch * kConvK + k, s_acc[i]);
    else if (dbias) atomicAdd(dbias + ch, s_acc[i]);
  }
}

}  // namespace
}  // namespace mb200

using namespace mb200;

// Chunk length (multiple of 4 in [16, 256]) that minimises waves x (chunk + halo): `cols` warps per
// (row, chunk), `warps_per_sm` resident warps per SM.
static int pick_conv_chunk(int64_t B, int64_t L, int64_t cols, int warps_per_sm) {
  const double cap = double(sm_count()) * warps_per_sm;
  int best = 32;
  double best_cost = 1e300;
  for (int c = 16; c <= 256; c += 4) {
    const double warps = double(cols) * double((L + c - 1) / c) * double(B);
    const double waves = warps <= cap ? 1.0 : double(int64_t((warps + cap - 1) / cap));
    // a wave that is not full still runs for a whole chunk; very few warps cannot keep HBM busy
    const double fill = warps < cap ? cap / (warps > 1 ? warps : 1) : 1.0;
    const double cost = waves * (c + 3) * (fill > 4 ? fill / 4 : 1.0);
    if (cost < best_cost) { best_cost = cost; best = c; }
  }
  return best;
}

static bool conv_vec_ok(int64_t ED, int kv, std::initializer_list<const void*> ptrs,
                        std::initializer_list<int64_t> strides) {
  if (ED % kv) return false;
  for (const void* p : ptrs) if (!aligned16(p)) return false;
  for (int64_t s : strides) if (s % kv) return false;
  return true;
}

extern "C" int mb200_conv1d_silu_fwd(const void* x, const float* w, const float* bias, void* y,
                                     int64_t B, int64_t L, int64_t ED, int K, int64_t x_sb, int64_t x_sl,
                                     int64_t y_sb, int64_t y_sl, int dtype, void* stream) {
  if (B < 0 || L < 0 || ED < 0) return MB200_EINVAL;
  if (K != kConvK) return MB200_ETOOBIG;
  if (dtype != MB200_F32 && dtype != MB200_BF16) return MB200_EDTYPE;
  if (B == 0 || L == 0 || ED == 0) return MB200_OK;
  if (!x || !w || !y) return MB200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int kv = 4;                                      // 4 channels per thread: 8-byte (bf16) or 16-byte (f32) accesses
  const bool vec = conv_vec_ok(ED, kv, {x, y}, {x_sb, x_sl, y_sb, y_sl});
  const int v = vec ? kv : 1;
  const int64_t cols = (ED + 32 * int64_t(v) - 1) / (32 * int64_t(v));
  const int64_t sms = sm_count();
  int64_t ngroup = 0, best = 0, best_rounds = 0;
  bool longer = false;
  for (int k = 0; k < 2; ++k) {
    constexpr int64_t kWarps = kConvThreads / 32, kResident = 3;
    const int64_t chunk = kConvChunkFwd[k], chunks = (L + chunk - 1) / chunk, groups = (chunks + kWarps - 1) / kWarps;
    if (k == 0 && groups > 65535) return MB200_ETOOBIG;
    const int64_t ctas = cols * groups * B, per_sm = (ctas + sms - 1) / sms, full = min64(chunks, kWarps);
    const int64_t rounds = per_sm <= kResident ? per_sm : (per_sm + kResident - 1) / kResident * kResident;
    // in a last round of no more than `cols` CTAs all are a row's last
    const int64_t last = rounds == per_sm && ctas - (rounds - 1) * sms <= cols ? chunks - (groups - 1) * kWarps : full;
    const int64_t cost = ((rounds - 1) * full + last) * (chunk + kConvK - 1);
    if (k == 0 || (rounds < best_rounds && cost < best)) { best = cost; best_rounds = rounds; ngroup = groups; longer = k == 1; }
  }
  if (B > 65535) return MB200_ETOOBIG;
  const dim3 grid(static_cast<unsigned>(cols), static_cast<unsigned>(ngroup), static_cast<unsigned>(B));
#define MB200_CONV_FWD(TT, VV) do { \
    if (longer) conv1d_silu_fwd_kernel<TT, VV, kConvChunkFwd[1]><<<grid, kConvThreads, 0, st>>>((const TT*)x, w, bias, (TT*)y, L, ED, x_sb, x_sl, y_sb, y_sl); \
    else conv1d_silu_fwd_kernel<TT, VV, kConvChunkFwd[0]><<<grid, kConvThreads, 0, st>>>((const TT*)x, w, bias, (TT*)y, L, ED, x_sb, x_sl, y_sb, y_sl); \
  } while (0)
  if (dtype == MB200_F32) { if (vec) MB200_CONV_FWD(float, 4); else MB200_CONV_FWD(float, 1); }
  else { if (vec) MB200_CONV_FWD(__nv_bfloat16, 4); else MB200_CONV_FWD(__nv_bfloat16, 1); }
#undef MB200_CONV_FWD
  return check_launch();
}

extern "C" int mb200_conv1d_silu_bwd(const void* x, const float* w, const float* bias, const void* dy,
                                     void* dx, float* dw, float* dbias, int64_t B, int64_t L, int64_t ED,
                                     int K, int64_t x_sb, int64_t x_sl, int64_t dy_sb, int64_t dy_sl,
                                     int64_t dx_sb, int64_t dx_sl, int dtype, void* stream) {
  if (B < 0 || L < 0 || ED < 0) return MB200_EINVAL;
  if (K != kConvK) return MB200_ETOOBIG;
  if (dtype != MB200_F32 && dtype != MB200_BF16) return MB200_EDTYPE;
  if (B == 0 || L == 0 || ED == 0) return MB200_OK;
  if (!x || !w || !dy || !dx || !dw) return MB200_EINVAL;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int kv = 4;                                      // 4 channels per thread: 8-byte (bf16) or 16-byte (f32) accesses
  const bool vec = conv_vec_ok(ED, kv, {x, dy, (const void*)dx}, {x_sb, x_sl, dy_sb, dy_sl, dx_sb, dx_sl});
  const int v = vec ? kv : 1;
  const int64_t cols = (ED + 32 * int64_t(v) - 1) / (32 * int64_t(v));
  const int chunk = pick_conv_chunk(B, L, cols, 16);
  const int64_t nchunk = (L + chunk - 1) / chunk;
  const int64_t ngroup = (nchunk + kConvBwdThreads / 32 - 1) / (kConvBwdThreads / 32);
  if (B > 65535 || ngroup > 65535) return MB200_ETOOBIG;
  const dim3 grid(static_cast<unsigned>(cols), static_cast<unsigned>(ngroup), static_cast<unsigned>(B));
#define MB200_CONV_BWD(TT, VV) do { \
    if (longer) conv1d_silu_bwd_kernel<TT, VV, true><<<grid, kConvBwdThreads, 0, st>>>((const TT*)x, w, bias, (const TT*)dy, (TT*)dx, dw, dbias, L, ED, x_sb, x_sl, dy_sb, dy_sl, dx_sb, dx_sl, chunk); \
    else conv1d_silu_bwd_kernel<TT, VV, false><<<grid, kConvBwdThreads, 0, st>>>((const TT*)x, w, bias, (const TT*)dy, (TT*)dx, dw, dbias, L, ED, x_sb, x_sl, dy_sb, dy_sl, dx_sb, dx_sl, chunk); \
  } while (0)
  // us as a short / long chunk: bfloat16 20.0 / 20.9 at 8 x 900 x 1536 (chunks of 40), 21.9 / 22.1 at 8 x 1003 x 1536 (44), 26.4 / 25.1 at
  // 8 x 1200 x 1536 (52); float32 24.0 / 25.2 at 64 x 127 x 768 (24), 24.8 / 23.4 at 1 x 1777 x 5120 (32), 34.6 / 31.4 at 8 x 1003 x 1536 (44).
  const bool longer = chunk >= (dtype == MB200_F32 ? 32 : 48);
  if (dtype == MB200_F32) { if (vec) MB200_CONV_BWD(float, 4); else MB200_CONV_BWD(float, 1); }
  else { if (vec) MB200_CONV_BWD(__nv_bfloat16, 4); else MB200_CONV_BWD(__nv_bfloat16, 1); }
#undef MB200_CONV_BWD
  return check_launch();
}

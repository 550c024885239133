// Fused selective scan, backward, d_state 16 on tensors a tensor map can describe (sscan_bwd_generic.cuh: every other
// case).  One pass over x, delta, z, dy, B, C that writes dx, ddelta, dz and accumulates dB, dC, dA, dD; hidden states
// are recomputed chunk by chunk from the states the forward saved every kChunk (8) timesteps.
//
// What bounds it.  Per state element a timestep owes 12 FP32 operations and one and a half exponentials, and every
// (t, n) owes two sums over all channels (dB, dC): the kernel is bound by instruction issue and the register file's
// read ports, with the MUFU and shared-memory pipes close behind, and not by HBM.  So nothing is handed between warps.
//
// Structure: ONE WARP is one CTA and owns 32 channels of one batch row (or of one piece of it), walking time backwards.
// Lane = (channel group cg, state quad q): a thread owns 4 states of 4 channels, as two PAIRS of neighbouring channels.
//   - Packed f32x2 arithmetic runs over the channel pair: delta, delta * x and dy' of a pair come out of shared memory as
//     ready operands, sums over states need no horizontal add, and products for dB and dC are summed over the thread's
//     own four channels before anything crosses lanes.
//   - Lane 0 issues TMA loads (x, delta, z, dy boxes; the saved states as one bulk copy) kStages chunks ahead.
//   - Once per (t, channel) the lane that owns the channel evaluates softplus, the gate and its derivative and leaves
//     the operands in the warp's shared memory.
//   - A chunk is walked as two halves of four steps with the states AND the decays of a half in registers, so a decay is
//     evaluated one and a half times instead of twice.
//   - Per step, two transposing butterflies: over q (dx, ddelta, dz need sums over states; lane q ends up with its own
//     channel's three sums) and over cg (dB, dC; every lane ends up with one (which, n) and adds it to global memory).
//   - Lane pairs read the same channel operands: a 16-byte shared load whose neighbouring lanes share an address costs 2
//     cycles of the shared-memory pipe, one with 4 or 8 alternating addresses 4 (measured).
#pragma once
#include "scan_math.cuh"
#include "sscan.cuh"
#include "tma.cuh"

namespace mb200 {

constexpr int kWN = 16;                       // d_state
constexpr int kWCh = 32;                      // channels per warp
#ifndef MB200_PART
#define MB200_PART 2
#endif
#ifndef MB200_PARTU
#define MB200_PARTU 1
#endif
constexpr int kPart = MB200_PART, kPartUnroll = MB200_PARTU;   // steps whose states and decays are in registers together

struct Bwd16Maps {
  CUtensorMap x, d, z, dy, dx, dd, dz;
};

template <typename T> struct Bwd16Smem {
  static constexpr int kStages = 2;
  static constexpr int kBox = kChunk * kWCh * int(sizeof(T));               // one raw x / delta / z / dy box
  static constexpr int kSaved = 4 * kBox;                                    // the chunk's saved states [32][16]
  static constexpr int kStageBytes = 4 * kBox + kWCh * kWN * 4;
  static constexpr int kOp = kStages * kStageBytes;                          // float4 [8][32]: {delta, partner's; delta x, partner's}
  static constexpr int kDy = kOp + kChunk * 32 * 16;                         // float2 [8][32]: {dy', partner's}
  static constexpr int kOwn = kDy + kChunk * 32 * 8;                         // float2 [8][32]: {x, d gate * dy}
  static constexpr int kBC = kOwn + kChunk * 32 * 8;                         // float2 [8][2][16]: B, C, each value twice
  static constexpr int kOut = kBC + kChunk * 32 * 8;                         // T [3][8][32]: dx, ddelta, dz boxes on their way out
  static constexpr int kMid = kOut + 3 * kBox;                               // float4 [3][8][32]: states entering steps 2, 4, 6
  static constexpr int kBars = kMid + 3 * 8 * 32 * 16 / 2;
  static constexpr int kBytes = kBars + kStages * 8;
};

namespace {
__device__ int g_bwd16_status = MB200_DEV_OK;                                // one word per translation unit
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// Box in shared memory -> element coordinates (c, l, b) of the mapped tensor; what lies outside the tensor is not written.
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int c, int l, int b) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(c), "r"(l), "r"(b), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void red_add(float* addr, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v));          // no clobber: later loads may move ahead of it
}
// One round of a transposing butterfly: of the pair (lo, hi) this lane keeps `hi` if its bit is set, else `lo`, and adds its
// partner's copy of the same value.
__device__ __forceinline__ float fold_pair(float lo, float hi, bool bit, int mask) {
  const float keep = bit ? hi : lo, send = bit ? lo : hi;
  return keep + __shfl_xor_sync(0xffffffffu, send, mask);
}

// kCarryOnly is the reverse carry pass of a split backward: gc <- a[t] * (dy'[t] * C[t] + gc), which also returns the
// piece's decay product exp(A * sum delta).  It reads no x, no B and no saved states.
template <typename T, bool kRev, bool kSoftplus, bool kHasZ, bool kCarryOnly>
__global__ void __launch_bounds__(32)
sscan_bwd16_kernel(const __grid_constant__ Bwd16Maps maps, const SscanBwdParams p) {
  using S = Bwd16Smem<T>;
  constexpr int kStages = S::kStages, N = kWN;
  extern __shared__ __align__(128) unsigned char smem[];
  float4* s_op = reinterpret_cast<float4*>(smem + S::kOp);
  float2* s_dy = reinterpret_cast<float2*>(smem + S::kDy);
  float2* s_own = reinterpret_cast<float2*>(smem + S::kOwn);
  float2* s_bc = reinterpret_cast<float2*>(smem + S::kBC);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBars);

  const int lane = threadIdx.x, q = (lane >> 1) & 3, cg = (lane & 1) | (lane >> 3) << 1;
  const int64_t b = blockIdx.y, pc = int64_t(blockIdx.z) + p.piece0, e0 = int64_t(blockIdx.x) * kWCh;
  const int cols_ok = int(min64(kWCh, p.ED - e0));
  const int64_t t_lo = pc * p.piece_len, t_hi = min64(p.L, t_lo + p.piece_len);
  const int nch = int((t_hi - t_lo + kChunk - 1) / kChunk);
  const int64_t chunks_all = (p.L + kChunk - 1) / kChunk;
  // Chunks are taken in the opposite order of the scan being differentiated (kRev: it ran from t = L-1 down to 0); step s
  // of a chunk in the scan's own order is its row `row(s)`.  Saved states are indexed by time chunk.
  auto chunk_t0 = [&](int j) { return t_lo + int64_t(kRev ? j : nch - 1 - j) * kChunk; };
  auto row = [](int s) { return kRev ? kChunk - 1 - s : s; };
  // Channels (inside the warp's 32) of this lane's two pair slots.  The order depends on q so that the butterfly over q
  // needs no selects: slot 0's first channel is the one this lane owns, its second the partner's (lane ^ 2), and slot 1
  // is slot 0 of lane ^ 4.
  auto chan = [&](int slot, int k) { return 2 * ((slot ^ (q >> 1)) * 8 + cg) + (k ^ (q & 1)); };
  const int own = chan(0, 0);
  const int64_t e_own = e0 + own;
  const bool own_ok = own < cols_ok;

  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < kStages; ++i) mbar_init(&bars[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  auto stage_ptr = [&](int j) { return smem + (j % kStages) * S::kStageBytes; };
  const uint32_t saved_bytes = uint32_t(cols_ok) * N * 4;
  auto issue = [&](int j) {                                                  // lane 0
    unsigned char* st = stage_ptr(j);
    uint64_t* bar = &bars[j % kStages];
    const int t0 = int(chunk_t0(j));
    constexpr int boxes = (kCarryOnly ? 2 : 3) + (kHasZ ? 1 : 0);
    mbar_expect_tx(bar, uint32_t(boxes * S::kBox) + (kCarryOnly ? 0 : saved_bytes));
    if constexpr (!kCarryOnly) tma_load_3d(st, &maps.x, int(e0), t0, int(b), bar);
    tma_load_3d(st + S::kBox, &maps.d, int(e0), t0, int(b), bar);
    if constexpr (kHasZ) tma_load_3d(st + 2 * S::kBox, &maps.z, int(e0), t0, int(b), bar);
    tma_load_3d(st + 3 * S::kBox, &maps.dy, int(e0), t0, int(b), bar);
    if constexpr (!kCarryOnly)
      bulk_load(st + S::kSaved, p.carries + ((b * chunks_all + t0 / kChunk) * p.ED + e0) * N, saved_bytes, bar);
  };
  if (lane == 0)
    for (int j = 0; j < kStages && j < nch; ++j) issue(j);

  // B and C rows of a chunk: any alignment, through registers one chunk ahead
  const T* gB = static_cast<const T*>(p.Bm) + b * p.b_sb;
  const T* gC = static_cast<const T*>(p.Cm) + b * p.c_sb;
  const T* gBC = (lane < N) ? gB + lane : gC + (lane - N);
  const int64_t bc_sl = (lane < N) ? p.b_sl : p.c_sl;
  T bc[kChunk];
  auto fetch_bc = [&](int j) {
    const int64_t t0 = chunk_t0(j);
    const int rows_ok = int(min64(kChunk, t_hi - t0));
#pragma unroll
    for (int r = 0; r < kChunk; ++r) bc[r] = r < rows_ok ? __ldg(gBC + (t0 + r) * bc_sl) : Elem<T>::from_f(0.f);
  };
  fetch_bc(0);

  // ---- this thread's states: [slot][state], packed over the slot's two channels
  f2 A2[2][4], gc[2][4], dA[2][4];
#pragma unroll
  for (int sl = 0; sl < 2; ++sl) {
    float a[2][4], g[2][4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = chan(sl, k);
      const int64_t o = (e0 + c) * N + 4 * q;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        a[k][n] = c < cols_ok ? p.A[o + n] * kLog2e : 0.f;
        g[k][n] = (c < cols_ok && p.g_in) ? p.g_in[b * p.ED * N + o + n] : 0.f;
      }
      // carries of the pieces on the far side, folded towards this one (g_in enters the last piece)
      if (!kCarryOnly && p.pieces > 1 && c < cols_ok) {
        for (int64_t r = kRev ? 0 : p.pieces - 1; r != pc; r += kRev ? 1 : -1) {
          const int64_t w = (b * p.pieces + r) * p.ED * N + o;
#pragma unroll
          for (int n = 0; n < 4; ++n) g[k][n] = fmaf(p.piece_P[w + n], g[k][n], p.piece_G[w + n]);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      A2[sl][n] = pk(a[0][n], a[1][n]);
      gc[sl][n] = pk(g[0][n], g[1][n]);
      dA[sl][n] = 0ull;
    }
  }
  const float bias = (kSoftplus && own_ok) ? p.delta_bias[e_own] : 0.f;
  const float Dv = (own_ok && p.D) ? p.D[e_own] : 0.f;
  float dD = 0.f, dbias = 0.f, dsum = 0.f, dcomp = 0.f;
  float* gred = nullptr;
  if constexpr (!kCarryOnly) {
    // the (which, n) this lane's butterfly ends with
    const int n = 4 * q + ((lane >> 3) & 1) * 2 + (lane & 1);
    gred = ((lane >> 4) ? p.dC : p.dB) + b * p.L * N + n;
  }

  for (int j = 0; j < nch; ++j) {
    const int64_t t0 = chunk_t0(j);
    const int rows_ok = int(min64(kChunk, t_hi - t0));
#pragma unroll
    for (int r = 0; r < kChunk; ++r) s_bc[r * 32 + lane] = make_float2(Elem<T>::to_f(bc[r]), Elem<T>::to_f(bc[r]));
    if (j + 1 < nch) fetch_bc(j + 1);
    if (!mbar_wait(&bars[j % kStages], (j / kStages) & 1)) {
      atomicExch(&g_bwd16_status, MB200_DEV_WAIT_TIMEOUT);
      return;
    }
    // ---- operands of the chunk, by the lanes that own the channels
    {
      const T* st = reinterpret_cast<const T*>(stage_ptr(j)) + own;
      float dgrp = 0.f;
#pragma unroll
      for (int r = 0; r < kChunk; ++r) {
        const float xv = kCarryOnly ? 0.f : Elem<T>::to_f(st[r * kWCh]);
        float dv = Elem<T>::to_f(st[(kChunk + r) * kWCh]);
        const float dyv = Elem<T>::to_f(st[(3 * kChunk + r) * kWCh]);
        if constexpr (kSoftplus) dv = softplus_sel(dv + bias);
        if (r >= rows_ok) dv = 0.f;                                          // past the end of the sequence: no step
        float dyg = dyv, fz = 0.f;
        if constexpr (kHasZ) {
          const float zv = Elem<T>::to_f(st[(2 * kChunk + r) * kWCh]);
          const float sg = sigmoid_fast(zv), ds = dyv * sg;
          dyg = ds * zv;
          fz = ds * fmaf(zv, 1.f - sg, 1.f);
        }
        const float dx = dv * xv;
        s_op[r * 32 + lane] = make_float4(dv, __shfl_xor_sync(0xffffffffu, dv, 2), dx, kCarryOnly ? 0.f : __shfl_xor_sync(0xffffffffu, dx, 2));
        s_dy[r * 32 + lane] = make_float2(dyg, __shfl_xor_sync(0xffffffffu, dyg, 2));
        if constexpr (!kCarryOnly) s_own[r * 32 + lane] = make_float2(xv, fz);
        if constexpr (kCarryOnly) dgrp += dv;
      }
      if constexpr (kCarryOnly) {                                            // L can be 10^5, and it feeds an exponent
        const float yk = dgrp - dcomp, tk = dsum + yk;
        dcomp = (tk - dsum) - yk;
        dsum = tk;
      }
    }
    f2 h0[2][4];
    if constexpr (!kCarryOnly) {
      const float4* sv = reinterpret_cast<const float4*>(stage_ptr(j) + S::kSaved);
#pragma unroll
      for (int sl = 0; sl < 2; ++sl) {
        // past the last channel shared memory holds whatever was there before: no state
        float4 u = sv[chan(sl, 0) * 4 + q], v = sv[chan(sl, 1) * 4 + q];
        if (chan(sl, 0) >= cols_ok) u = make_float4(0.f, 0.f, 0.f, 0.f);
        if (chan(sl, 1) >= cols_ok) v = make_float4(0.f, 0.f, 0.f, 0.f);
        h0[sl][0] = pk(u.x, v.x); h0[sl][1] = pk(u.y, v.y); h0[sl][2] = pk(u.z, v.z); h0[sl][3] = pk(u.w, v.w);
      }
    }
    __syncwarp();                                                            // operands are visible, the raw stage is free
    if (lane == 0 && j + kStages < nch) issue(j + kStages);

    // packed operands of row r
    struct Four { f2 v[4]; };
    auto load_bc = [&](int r, int which) {
      const ulonglong2* s = reinterpret_cast<const ulonglong2*>(s_bc + r * 32 + which * N + 4 * q);
      const ulonglong2 a = s[0], c = s[1];
      return Four{{a.x, a.y, c.x, c.y}};
    };
    auto load_op = [&](int r, int sl) { return *reinterpret_cast<const ulonglong2*>(s_op + r * 32 + (lane ^ (4 * sl))); };
    auto load_dy = [&](int r, int sl) { return *reinterpret_cast<const f2*>(s_dy + r * 32 + (lane ^ (4 * sl))); };
    auto decay = [&](f2 d2, int sl, f2 (&a)[4]) {
#pragma unroll
      for (int n = 0; n < 4; ++n) a[n] = pex2(pmul(d2, A2[sl][n]));
    };
    if constexpr (kCarryOnly) {
#pragma unroll
      for (int s = kChunk - 1; s >= 0; --s) {
        const int r = row(s);
        const Four C4 = load_bc(r, 1);
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
          f2 a[4];
          const f2 dy2 = load_dy(r, sl);
          decay(load_op(r, sl).x, sl, a);
#pragma unroll
          for (int n = 0; n < 4; ++n) gc[sl][n] = pmul(a[n], pfma(dy2, C4.v[n], gc[sl][n]));
        }
      }
    } else {
      // one forward step: h <- a h + (delta x) B, the product last so that delta x is the operand that repeats
      auto forward = [&](int s, f2 (&h)[2][4], f2 (&a)[2][4]) {
        const int r = row(s);
        const Four B4 = load_bc(r, 0);
#pragma unroll
        for (int sl = 0; sl < 2; ++sl) {
          const ulonglong2 o = load_op(r, sl);
          decay(o.x, sl, a[sl]);
#pragma unroll
          for (int n = 0; n < 4; ++n) h[sl][n] = pfma(o.y, B4.v[n], pmul(a[sl][n], h[sl][n]));
        }
      };
      T* out = reinterpret_cast<T*>(smem + S::kOut) + own;
      ulonglong2* mid = reinterpret_cast<ulonglong2*>(smem + S::kMid) + lane;
      {
        f2 h[2][4], a[2][4];
#pragma unroll
        for (int sl = 0; sl < 2; ++sl)
#pragma unroll
          for (int n = 0; n < 4; ++n) h[sl][n] = h0[sl][n];
#pragma unroll
        for (int s = 0; s < kChunk - kPart; ++s) {
          forward(s, h, a);
          if (s % kPart == kPart - 1) {
#pragma unroll
            for (int sl = 0; sl < 2; ++sl)
#pragma unroll
              for (int n = 0; n < 4; n += 2) mid[(s / kPart * 4 + sl * 2 + n / 2) * 32] = make_ulonglong2(h[sl][n], h[sl][n + 1]);
          }
        }
      }
      // the boxes of the previous chunk have left shared memory before new values are put there
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      __syncwarp();
#pragma unroll kPartUnroll
      for (int part = kChunk / kPart - 1; part >= 0; --part) {
        f2 hin[2][4], hh[kPart][2][4], aa[kPart][2][4];
#pragma unroll
        for (int sl = 0; sl < 2; ++sl)
#pragma unroll
          for (int n = 0; n < 4; n += 2) {
            const ulonglong2 m = mid[((part > 0 ? part - 1 : 0) * 4 + sl * 2 + n / 2) * 32];
            hin[sl][n] = part > 0 ? m.x : h0[sl][n];
            hin[sl][n + 1] = part > 0 ? m.y : h0[sl][n + 1];
          }
#pragma unroll
        for (int i = 0; i < kPart; ++i) {
#pragma unroll
          for (int sl = 0; sl < 2; ++sl)
#pragma unroll
            for (int n = 0; n < 4; ++n) hh[i][sl][n] = i ? hh[i ? i - 1 : 0][sl][n] : hin[sl][n];
          forward(part * kPart + i, hh[i], aa[i]);
        }
        float* pred = gred + (t0 + row(part * kPart)) * N;
#pragma unroll
        for (int i = kPart - 1; i >= 0; --i) {
          const int r = row(part * kPart + i), ri = kRev ? -i : i;           // row, and rows from the part's first
          const Four B4 = load_bc(r, 0), C4 = load_bc(r, 1);
          f2 dB2[4], dC2[4], ys[2], gB[2], wA[2];
          float d_own = 0.f, dy_own = 0.f;
#pragma unroll
          for (int sl = 0; sl < 2; ++sl) {
            const ulonglong2 o = load_op(r, sl);
            const f2 dy2 = load_dy(r, sl);
            if (sl == 0) { d_own = lo(o.x); dy_own = lo(dy2); }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
              const f2 hc = hh[i][sl][n], hp = i ? hh[i ? i - 1 : 0][sl][n] : hin[sl][n];
              const f2 g = pfma(dy2, C4.v[n], gc[sl][n]);
              dC2[n] = sl ? pfma(dy2, hc, dC2[n]) : pmul(dy2, hc);
              dB2[n] = sl ? pfma(o.y, g, dB2[n]) : pmul(o.y, g);
              if (kHasZ) ys[sl] = n ? pfma(hc, C4.v[n], ys[sl]) : pmul(hc, C4.v[n]);
              gB[sl] = n ? pfma(g, B4.v[n], gB[sl]) : pmul(g, B4.v[n]);
              gc[sl][n] = pmul(aa[i][sl][n], g);
              const f2 w = pmul(gc[sl][n], hp);
              dA[sl][n] = pfma(o.x, w, dA[sl][n]);
              wA[sl] = n ? pfma(w, A2[sl][n], wA[sl]) : pmul(w, A2[sl][n]);
            }
          }
          // dB, dC: sums over the 8 channel groups; lane bits 4, 3, 0 pick which, n / 2, n % 2
          {
            float u[4];
#pragma unroll
            for (int n = 0; n < 4; ++n) u[n] = fold_pair(lo(dB2[n]) + hi(dB2[n]), lo(dC2[n]) + hi(dC2[n]), (lane & 16) != 0, 16);
            const float v0 = fold_pair(u[0], u[2], (lane & 8) != 0, 8), v1 = fold_pair(u[1], u[3], (lane & 8) != 0, 8);
            const float tot = fold_pair(v0, v1, (lane & 1) != 0, 1);
            if (r < rows_ok) red_add(pred + ri * N, tot);
          }
          // sums over the four state quads: lane q ends with the channel it owns
          auto over_q = [&](const f2 (&v)[2]) {
            const f2 t = padd(v[0], pk(__shfl_xor_sync(0xffffffffu, lo(v[1]), 4), __shfl_xor_sync(0xffffffffu, hi(v[1]), 4)));
            return lo(t) + __shfl_xor_sync(0xffffffffu, hi(t), 2);
          };
          const float ysum = kHasZ ? over_q(ys) : 0.f, gBs = over_q(gB), wAs = over_q(wA);
          const float2 xf = s_own[r * 32 + lane];                            // {x, d gate * dy}
          // d softplus = sigmoid(raw) = 1 - exp(-softplus(raw)); series where the difference cancels
          float spg = 1.f;
          if constexpr (kSoftplus) {
            const float ser = d_own * (1.f - d_own * (0.5f - d_own * (1.f / 6.f))), ful = 1.f - __expf(-d_own);
            spg = d_own < 1e-2f ? ser : ful;
          }
          // channels and rows outside the tensor contribute zeros to the sums
          const float dxv = fmaf(dy_own, Dv, d_own * gBs);
          const float ddv = fmaf(xf.x, gBs, wAs * (1.f / kLog2e)) * spg;
          dD = fmaf(dy_own, xf.x, dD);
          dbias += ddv;
          out[r * kWCh] = Elem<T>::from_f(dxv);
          out[(kChunk + r) * kWCh] = Elem<T>::from_f(ddv);
          if constexpr (kHasZ) out[(2 * kChunk + r) * kWCh] = Elem<T>::from_f(xf.y * fmaf(Dv, xf.x, ysum));
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        const unsigned char* o = smem + S::kOut;
        tma_store_3d(&maps.dx, o, int(e0), int(t0), int(b));
        tma_store_3d(&maps.dd, o + S::kBox, int(e0), int(t0), int(b));
        if constexpr (kHasZ) tma_store_3d(&maps.dz, o + 2 * S::kBox, int(e0), int(t0), int(b));
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    }
    __syncwarp();                                                            // the operand arrays may be rewritten
  }

  if constexpr (kCarryOnly) {
    // hand the sum of delta of every channel to the lanes that hold its states
    reinterpret_cast<float*>(s_own)[own] = dsum;
    __syncwarp();
#pragma unroll
    for (int sl = 0; sl < 2; ++sl)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = chan(sl, k);
        if (c >= cols_ok) continue;
        const float sd = reinterpret_cast<const float*>(s_own)[c];
        const int64_t w = (b * p.pieces + pc) * p.ED * N + (e0 + c) * N + 4 * q;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          p.piece_P[w + n] = ex2f((k ? hi(A2[sl][n]) : lo(A2[sl][n])) * sd);
          p.piece_G[w + n] = k ? hi(gc[sl][n]) : lo(gc[sl][n]);
        }
      }
  } else {
    const bool first = pc == (kRev ? p.pieces - 1 : 0);                      // nothing precedes this piece: its carry leaves
#pragma unroll
    for (int sl = 0; sl < 2; ++sl)
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int c = chan(sl, k);
        if (c >= cols_ok) continue;
        const int64_t o = (e0 + c) * N + 4 * q;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          red_add(p.dA + o + n, k ? hi(dA[sl][n]) : lo(dA[sl][n]));
          if (p.g_out && first) p.g_out[b * p.ED * N + o + n] = k ? hi(gc[sl][n]) : lo(gc[sl][n]);
        }
      }
    if (own_ok) {
      if (p.dD) red_add(p.dD + e_own, dD);
      if (p.ddelta_bias) red_add(p.ddelta_bias + e_own, dbias);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
}

}  // namespace mb200

// Fused selective scan, backward.  One pass over x, delta, z, B, C, dy (read once) that writes
// dx, ddelta, dz and accumulates dB, dC, dA, dD; the hidden states are recomputed chunk by chunk
// from the states the forward saved every kChunk (8) timesteps.
//
// The kernel is bound by shared-memory traffic, instruction issue and the latency of each warp's
// dependent chain, not by HBM, so the recurrences run on warps that do nothing else (tensor-map
// path, d_state 16; the register-staged kernel in sscan_bwd_generic.cuh covers every other case).
//
// A CTA of 256 threads owns 32 channels of one batch row and walks time BACKWARDS in tiles of 16
// (two saved states per tile):
//   - warp 4 issues TMA loads of the raw x, delta, z, dy, B, C boxes a few tiles ahead into a
//     shared-memory ring and converts each landed tile into float32 operands
//     ({softplus(delta+bias), delta*x}, its derivative, dy*silu(z), that of silu, B, C; double-buffered).
//   - warps 0-3 (consumers; a thread owns 2 states of 2 neighbouring channels) recompute the 8 states of a
//     chunk forwards from its saved state into registers and walk them backwards:
//     g[t] = dy'[t] C[t] + a[t+1] g[t+1],  da = g h[t-1].  Operands of the walk are fetched two
//     timesteps ahead.  Per timestep a thread leaves its partial sums over states (for y, dx, ddelta; two
//     lanes add theirs first) and its products for dB, dC, already added over its two channels, in shared
//     memory, in windows of 2 timesteps.
//     Why 2 x 2: what goes through shared memory is what bounds the kernel.  Of its 4 elements a thread hands
//     over 8 products and 3 sums (4 states of a channel), 4 and 3 (2 x 2, with three shuffles) or 2 and 12; and
//     B and C of a state pair are then short loads of two addresses (side by side, so that the reverse walk takes one),
//     delta and delta*x 16-byte loads that two lanes share.
//     44.6 -> 34.8 wavefronts per 128 elements and 610 -> 544 us on 8 x 2048 x 1536 in bfloat16, together with
//     what follows (526 with index arithmetic out of the loops); without the shuffles (twice the sums) 587.
//   - warps 5 and 7 finish alternate windows: sum the 4 partials of each channel, form dx, ddelta,
//     dz (and the running sums for dD and d(delta_bias)), store them.  delta, dy' and the derivatives of
//     softplus and silu come from the operand tile: the converter has their exponentials in hand, and these
//     two warps were what the consumers waited for (614 us with the derivatives evaluated here).
//   - warp 6 sums the dB, dC products of each window over the CTA's 16 channel pairs and adds the
//     result to global memory with vector atomics.
//   - Hand-off through CTA-local mbarriers; every wait is bounded (see mbar_wait).  A barrier's
//     round trip through the busy shared-memory pipe costs a few hundred cycles, so the consumers
//     ask for a window's buffer with a non-blocking test before the arithmetic of the window and
//     only block if the answer was "not yet".
#include "sscan_bwd_generic.cuh"
#include "tma.cuh"

namespace mb200 {
namespace {

constexpr int kBN = 16;                      // d_state of this path
constexpr int kBTE = 32;                     // channels per CTA
constexpr int kBTile = 2 * kChunk;           // timesteps per tile (two saved states per tile)
constexpr int kHalf = kChunk;                // states kept in registers at a time
constexpr int kBWin = 2;                     // timesteps per reduction window
constexpr int kWinsPerTile = kBTile / kBWin;
constexpr int kBwdThreads = 256;
constexpr int kNpPlane = kBN / 4 * kBTE;     // one kind of partial sum of a timestep: floats [state quad][channel]
constexpr int kNpStep = 3 * kNpPlane;        // for y, dx, ddelta
constexpr int kEpStep = kBN / 2 * kBTE / 2;  // dB, dC products of a timestep: float4 [state pair][channel pair]

__device__ int g_bwd_status = MB200_DEV_OK;

template <typename T> struct alignas(sizeof(T) * 2) Vec2 {
  T v[2];
};

struct BwdMaps {
  CUtensorMap x, d, z, dy, B, C;
};

template <typename T> struct TmaBwdSmem {
  static constexpr int kStages = sizeof(T) == 2 ? 6 : 3;
  static constexpr int kActBytes = kBTile * kBTE * int(sizeof(T));
  static constexpr int kBcBytes = kBTile * kBN * int(sizeof(T));
  static constexpr int kStageBytes = 4 * kActBytes + 2 * kBcBytes;       // x, delta, z, dy, B, C
  static constexpr int kRaw = 0;
  static constexpr int kOp = kRaw + kStages * kStageBytes;                // float4 [2][16][16]
  static constexpr int kAux = kOp + 2 * kBTile * kBTE * 8;                // float4 [2][16][16]
  static constexpr int kDyp = kAux + 2 * kBTile * kBTE * 8;               // float  [2][16][32]
  static constexpr int kBC = kDyp + 2 * kBTile * kBTE * 4;                // float4 [2][16][8]
  static constexpr int kNp = kBC + 4 * kBTile * kBN * 4;                   // float  [2][kBWin][3][4][32]
  static constexpr int kEp = kNp + 2 * kBWin * kNpStep * 4;                  // float4 [2][kBWin][8][16]
  static constexpr int kD = kEp + 2 * kBWin * kEpStep * 16;               // float [32]
  static constexpr int kBias = kD + kBTE * 4;
  static constexpr int kBars = kBias + kBTE * 4;                          // 2*kStages + 8 mbarriers
  static constexpr int kBytes = kBars + (2 * kStages + 8) * 8;
};

__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// The softplus option and the presence of the gate are template parameters too: as run-time flags they
// cost the converter and finishing warps (the busiest ones) branches and selects, 6 % of the launch.
// (Without a gate the sum for y, which only dz needs, is still formed and handed over: 501 us for 525 on 8 x 2048 x 1536 in bfloat16.)
// Saved states that lie next to a channel's others instead of two by two are 8-byte loads 64 bytes apart: 556 us there for 525, 138 for 134
// on 3 x 1003 x 1000.
template <typename T, bool kRev, bool kSoftplus, bool kHasZ>
__global__ void __launch_bounds__(kBwdThreads, 3)
sscan_bwd_tma_kernel(const __grid_constant__ BwdMaps maps, const SscanBwdParams p) {
  using S = TmaBwdSmem<T>;
  constexpr int kStages = S::kStages, kAhead = S::kStages - 2;
  constexpr int N = kBN;

  extern __shared__ __align__(128) unsigned char smem_raw[];
  float4* s_op = reinterpret_cast<float4*>(smem_raw + S::kOp);      // {delta, delta, delta*x, delta*x} of a channel pair
  float4* s_aux = reinterpret_cast<float4*>(smem_raw + S::kAux);    // {d softplus x 2, dy d(silu z)/dz x 2} of a channel pair
  float* s_dyp = reinterpret_cast<float*>(smem_raw + S::kDyp);
  float4* s_BC = reinterpret_cast<float4*>(smem_raw + S::kBC);      // {B, B, C, C} of a state pair
  float* s_np = reinterpret_cast<float*>(smem_raw + S::kNp);
  float4* s_ep = reinterpret_cast<float4*>(smem_raw + S::kEp);
  float* s_D = reinterpret_cast<float*>(smem_raw + S::kD);
  float* s_bias = reinterpret_cast<float*>(smem_raw + S::kBias);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + S::kBars);
  uint64_t* raw_full = bars;                      // [kStages] copy landed
  uint64_t* raw_free = bars + kStages;            // [kStages] warps 4, 5, 7 are done with the stage
  uint64_t* op_full = bars + 2 * kStages;         // [2] operands committed (warp 4)
  uint64_t* op_empty = op_full + 2;               // [2] consumers are done with the operand buffer
  uint64_t* win_full = op_full + 4;               // [2] consumers filled a window of partials
  uint64_t* win_empty = op_full + 6;              // [2] finishing warps drained it

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t e0 = int64_t(blockIdx.x) * kBTE;
  // times fit 32 bits on this path; what is 64-bit in the loops costs the recurrence warps spills
  const int64_t b = blockIdx.y;
  const int pc = int(blockIdx.z), t_lo = int(pc * p.piece_len), t_hi = int(min64(p.L, t_lo + p.piece_len));
  const int cols_ok = int(min64(kBTE, p.ED - e0));
  constexpr bool softplus = kSoftplus;
  constexpr bool has_z = kHasZ;
  const int ntiles = (t_hi - t_lo + kBTile - 1) / kBTile;
  // Direction of the scan being differentiated (MB200_REVERSE: it ran from t = L-1 down to 0).  Tiles
  // are taken in the opposite order of that scan: iteration j works on the tile that starts at
  // tile_t0(j); step s of a tile in the scan's own order is its row `row(s)`.  Saved states are
  // indexed by time chunk: entry c is the state entering chunk c in the scan direction.
  constexpr bool rev = kRev;
  auto tile_t0 = [&](int j) { return t_lo + (rev ? j : ntiles - 1 - j) * kBTile; };
  auto row = [](int s) { return rev ? kBTile - 1 - s : s; };

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < kStages; ++i) { mbar_init(&raw_full[i], 1); mbar_init(&raw_free[i], 96); }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mbar_init(&op_full[i], 32); mbar_init(&op_empty[i], 128 + 64);
      mbar_init(&win_full[i], 128); mbar_init(&win_empty[i], 64);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < kBTE; i += kBwdThreads) {
    const bool ok = i < cols_ok;
    s_D[i] = (ok && p.D) ? p.D[e0 + i] : 0.f;
    s_bias[i] = (ok && softplus) ? p.delta_bias[e0 + i] : 0.f;
  }
  __syncthreads();
  auto fail = [&]() { atomicExch(&g_bwd_status, MB200_DEV_WAIT_TIMEOUT); };

  // The recurrence warps need far more registers than the others: hand 24 registers per thread of
  // warps 4-7 over to warps 0-3 (the kernel is compiled for 80; 128 * 56 + 128 * 104 = 256 * 80).  112 / 48 is no slower with three CTAs on
  // an SM (524 us for 523 on 8 x 2048 x 1536) but 4 % with one (292 for 280); 120 / 40 spills.
  if (warp < 4) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  }
  if (warp < 4) {
    // ================================================================== consumers
    // A thread owns the states n0, n0 + 1 of the channels c0, c0 + 1; the two lanes of a channel pair are neighbours.
    const int sp = 2 * warp + (lane & 1), cp = lane >> 1;             // state pair 0..7, channel pair 0..15
    const int n0 = 2 * sp, c0 = 2 * cp;
    const int64_t e = e0 + c0;
    const bool ok0 = e < p.ED, ok1 = e + 1 < p.ED;
    float2 A2[2], gc[2], dAacc[2];                                    // [state]{channel}
    {
      const float* A0 = p.A + e * N + n0;
      const float* g0 = p.g_in ? p.g_in + ((b * p.pieces + pc) * p.ED + e) * N + n0 : nullptr;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        A2[k] = make_float2(ok0 ? A0[k] * kLog2e : 0.f, ok1 ? A0[N + k] * kLog2e : 0.f);
        gc[k] = make_float2(ok0 && g0 ? g0[k] : 0.f, ok1 && g0 ? g0[N + k] : 0.f);
        dAacc[k] = make_float2(0.f, 0.f);
      }
    }
    // slot of this channel pair in the rows of the operand tile (even and odd rows are swizzled differently)
    const int op_off0 = swz(0, cp), op_off1 = swz(1, cp);
    const int npo = warp * kBTE + lane;
    // sum over the 4 states of both lanes of a channel pair: the even lane gets the first channel's, the odd one the second's
    auto lanes_sum = [&](float2 v) {
      const float give = (lane & 1) ? v.x : v.y, keep = (lane & 1) ? v.y : v.x;
      return keep + __shfl_xor_sync(0xffffffffu, give, 1);
    };
    float4* const epo = s_ep + sp * 16 + (cp ^ ((sp & 1) * 4));
    const int nchunks = int((p.L + kHalf - 1) / kHalf);
    // saved states of a chunk as [state]{channel}
    struct Pair { float2 v[2]; };
    const bool paired = (p.flags & MB200_PAIRED_STATES) != 0, wide = paired && ok1 && !(p.ED & 1);
    const float* carry_base = p.carries + b * nchunks * p.ED * N + state_pair(paired, p.ED, N, e, sp);
    auto load_carry = [&](int c) {
      Pair r;
      r.v[0] = r.v[1] = make_float2(0.f, 0.f);
      const float* src = carry_base + c * p.ED * N;
      if (c < nchunks) {
        if (wide) {
          const float4 q = *reinterpret_cast<const float4*>(src);
          r.v[0] = make_float2(q.x, q.z); r.v[1] = make_float2(q.y, q.w);
        } else {
          if (ok0) { const float2 q = *reinterpret_cast<const float2*>(src); r.v[0].x = q.x; r.v[1].x = q.y; }
          if (ok1) { const float2 q = *reinterpret_cast<const float2*>(src + (paired ? 2 : N)); r.v[0].y = q.x; r.v[1].y = q.y; }
        }
      }
      return r;
    };
    // Chunks are taken from the end of the scan to its start; the state entering the next one is fetched a chunk ahead.
    const int c_lo = t_lo / kHalf, nch = 2 * ntiles;
    auto chunk_at = [&](int k) { return c_lo + (rev ? k : nch - 1 - k); };
    Pair carry_next = load_carry(chunk_at(0));

#pragma unroll 1
    for (int k8 = 0; k8 < nch; ++k8) {
      const int j = k8 >> 1, buf = j & 1, second = k8 & 1;   // tile, its operand buffer, second chunk taken from it
      const Pair hin = carry_next;                           // state entering the chunk
      if (k8 + 1 < nch) carry_next = load_carry(chunk_at(k8 + 1));
      if (!second && !mbar_wait(&op_full[buf], (j >> 1) & 1)) { fail(); return; }
      // rows of the chunk: step i of the scan is row `rw(i)`
      const int r0 = buf * kBTile + ((second != 0) == rev ? kHalf : 0);
      auto rw = [](int i) { return rev ? kHalf - 1 - i : i; };
      const float4* op0 = s_op + r0 * (kBTE / 2) + op_off0;
      const float4* op1 = s_op + r0 * (kBTE / 2) + op_off1;
      const float* dyp = s_dyp + r0 * kBTE + c0;
      const float4* sBC = s_BC + r0 * (N / 2) + sp;

      // states after each step of the chunk, in registers
      float2 hh[kHalf][2];
      {
        float2 h[2] = {hin.v[0], hin.v[1]};
#pragma unroll
        for (int i = 0; i < kHalf; ++i) {
          const int r = rw(i);
          const float4 o = ((r & 1) ? op1 : op0)[r * (kBTE / 2)];
          const float2 Bp = *reinterpret_cast<const float2*>(sBC + r * (N / 2));
          const float2 dt = make_float2(o.x, o.y), dtx = make_float2(o.z, o.w);
          const float2 e0v = __fmul2_rn(dt, A2[0]), e1v = __fmul2_rn(dt, A2[1]);
          const float2 a0 = make_float2(ex2f(e0v.x), ex2f(e0v.y)), a1 = make_float2(ex2f(e1v.x), ex2f(e1v.y));
          h[0] = __ffma2_rn(a0, h[0], __fmul2_rn(dtx, make_float2(Bp.x, Bp.x)));
          h[1] = __ffma2_rn(a1, h[1], __fmul2_rn(dtx, make_float2(Bp.y, Bp.y)));
          hh[i][0] = h[0]; hh[i][1] = h[1];
        }
      }
      // operands of the reverse walk are fetched two timesteps ahead, so that their trip through the
      // shared-memory pipe overlaps the previous timestep's arithmetic, stores and barrier traffic
      struct Opnd { float4 o; float2 dy; float4 bc; };
      auto fetch = [&](int i) {
        const int rr = rw(i);
        Opnd r;
        r.o = ((rr & 1) ? op1 : op0)[rr * (kBTE / 2)];
        r.dy = *reinterpret_cast<const float2*>(dyp + rr * kBTE);
        r.bc = sBC[rr * (N / 2)];
        return r;
      };
      Opnd nx = fetch(kHalf - 1), nx2 = fetch(kHalf - 2);
#pragma unroll
      for (int wi = kHalf / kBWin - 1; wi >= 0; --wi) {
        // Windows are taken from the chunk's end, the two buffers in turn.  A chunk has four, so that buffer and parity are
        // known here (the first wait for each buffer, parity 1 of a new barrier, returns at once).
        const int wb = (kHalf / kBWin - 1 - wi) & 1, wpar = ((kHalf / kBWin - 1 - wi) >> 1) ^ 1;
        static_assert(kHalf / kBWin == 4, "buffers and parities repeat every chunk");
        // asked now, needed only before the first store of the window
        const bool slot_free = mbar_test(&win_empty[wb], wpar);
        float* np = s_np + wb * kBWin * kNpStep;
        float4* ep = epo + wb * kBWin * kEpStep;
#pragma unroll
        for (int ti = kBWin - 1; ti >= 0; --ti) {
          const int i = wi * kBWin + ti;                    // index inside the chunk
          const Opnd cu = nx;
          nx = nx2;
          if (i > 1) nx2 = fetch(i - 2);
          const float2 dt = make_float2(cu.o.x, cu.o.y), dtx = make_float2(cu.o.z, cu.o.w), dy2 = cu.dy;
          const float2 Bv[2] = {make_float2(cu.bc.x, cu.bc.x), make_float2(cu.bc.y, cu.bc.y)};
          const float2 Cv[2] = {make_float2(cu.bc.z, cu.bc.z), make_float2(cu.bc.w, cu.bc.w)};
          float2 ysum, gBs, wAs;                                            // {channel}
          float dB[2], dC[2];                                               // [state], over the two channels
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const float2 hcur = hh[i][k], hprev = i ? hh[i - 1][k] : hin.v[k];
            const float2 g = __ffma2_rn(dy2, Cv[k], gc[k]);
            ysum = k ? __ffma2_rn(hcur, Cv[k], ysum) : __fmul2_rn(hcur, Cv[k]);
            dC[k] = fmaf(dy2.y, hcur.y, dy2.x * hcur.x);
            dB[k] = fmaf(g.y, dtx.y, g.x * dtx.x);
            gBs = k ? __ffma2_rn(g, Bv[k], gBs) : __fmul2_rn(g, Bv[k]);
            const float2 ev = __fmul2_rn(dt, A2[k]);
            gc[k] = __fmul2_rn(make_float2(ex2f(ev.x), ex2f(ev.y)), g);
            const float2 w = __fmul2_rn(gc[k], hprev);
            dAacc[k] = __ffma2_rn(w, dt, dAacc[k]);
            wAs = k ? __ffma2_rn(w, A2[k], wAs) : __fmul2_rn(w, A2[k]);
          }
          const float s0 = lanes_sum(ysum), s1 = lanes_sum(gBs), s2 = lanes_sum(wAs);
          if (ti == kBWin - 1 && !slot_free && !mbar_wait(&win_empty[wb], wpar)) { fail(); return; }
          np[ti * kNpStep + npo] = s0;
          np[ti * kNpStep + kNpPlane + npo] = s1;
          np[ti * kNpStep + 2 * kNpPlane + npo] = s2;
          ep[ti * kEpStep] = make_float4(dB[0], dB[1], dC[0], dC[1]);
        }
        mbar_arrive(&win_full[wb]);
      }
      if (second) mbar_arrive(&op_empty[buf]);
    }
    const bool leaves = p.g_out && pc == (rev ? p.pieces - 1 : 0);   // the carry that leaves the scan's first timestep
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!(c ? ok1 : ok0)) continue;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        atomicAdd(p.dA + (e + c) * N + n0 + k, c ? dAacc[k].y : dAacc[k].x);
        if (leaves) p.g_out[(b * p.ED + e + c) * N + n0 + k] = c ? gc[k].y : gc[k].x;
      }
    }
    return;
  }
  auto stage_ptr = [&](int j) { return smem_raw + S::kRaw + int(j % kStages) * S::kStageBytes; };
  // Window wl (0..7, in processing order) of a tile covers its steps 14 - 2 wl and 15 - 2 wl in scan order: from window to
  // window, across tiles too, time moves by two rows, and the pointers below by a constant.  (Products of row and stride
  // for every window were 4 of 112 instructions per warp and timestep: 541 -> 529 us.  The finishing warps' loop is not unrolled: 568.)
  auto win_row = [&](int wl, int ti) { return row(kBTile - kBWin * (wl + 1) + ti); };

  if (warp == 4) {
    // ================================================================== loader + converter
    const uint32_t stage_tx = uint32_t((has_z ? 4 : 3) * S::kActBytes + 2 * S::kBcBytes);
    auto issue = [&](int j) -> bool {                       // lane 0 only
      const int r = int(j % kStages);
      if (j >= kStages && !mbar_wait(&raw_free[r], int((j / kStages - 1) & 1))) return false;
      unsigned char* st = stage_ptr(j);
      const int t0 = int(tile_t0(j));
      mbar_expect_tx(&raw_full[r], stage_tx);
      tma_load_3d(st, &maps.x, int(e0), t0, int(b), &raw_full[r]);
      tma_load_3d(st + S::kActBytes, &maps.d, int(e0), t0, int(b), &raw_full[r]);
      if (has_z) tma_load_3d(st + 2 * S::kActBytes, &maps.z, int(e0), t0, int(b), &raw_full[r]);
      tma_load_3d(st + 3 * S::kActBytes, &maps.dy, int(e0), t0, int(b), &raw_full[r]);
      tma_load_3d(st + 4 * S::kActBytes, &maps.B, 0, t0, int(b), &raw_full[r]);
      tma_load_3d(st + 4 * S::kActBytes + S::kBcBytes, &maps.C, 0, t0, int(b), &raw_full[r]);
      return true;
    };
    if (lane == 0) {
      for (int j = 0; j < kAhead && j < ntiles; ++j)
        if (!issue(j)) { fail(); return; }
    }
    for (int j = 0; j < ntiles; ++j) {
      const int buf = int(j & 1);
      const int rows_ok = min(kBTile, t_hi - tile_t0(j));
      if (j >= 2 && !mbar_wait(&op_empty[buf], int(((j - 2) >> 1) & 1))) { fail(); return; }
      if (!mbar_wait(&raw_full[j % kStages], int((j / kStages) & 1))) { fail(); return; }
      const unsigned char* st = stage_ptr(j);
      const T* rx = reinterpret_cast<const T*>(st);
      const T* rd = reinterpret_cast<const T*>(st + S::kActBytes);
      const T* rz = reinterpret_cast<const T*>(st + 2 * S::kActBytes);
      const T* rdy = reinterpret_cast<const T*>(st + 3 * S::kActBytes);
      float4* tile = s_op + buf * kBTile * (kBTE / 2);
      float4* auxt = s_aux + buf * kBTile * (kBTE / 2);
      float* dyt = s_dyp + buf * kBTile * kBTE;
      const float4 bq = *reinterpret_cast<const float4*>(s_bias + (lane & 7) * 4);   // this lane's 4 channels
      const float bias4[4] = {bq.x, bq.y, bq.z, bq.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = lane + 32 * i;
        const int rr = v >> 3, cc = (v & 7) * 4;
        const Vec4<T> xv = *reinterpret_cast<const Vec4<T>*>(rx + rr * kBTE + cc);
        const Vec4<T> dv4 = *reinterpret_cast<const Vec4<T>*>(rd + rr * kBTE + cc);
        const Vec4<T> yv4 = *reinterpret_cast<const Vec4<T>*>(rdy + rr * kBTE + cc);
        Vec4<T> zv4 = yv4;
        if (has_z) zv4 = *reinterpret_cast<const Vec4<T>*>(rz + rr * kBTE + cc);
        float2 o[4], sg[2], dq[2];
        float dyo[4];
#pragma unroll
        for (int k = 0; k < 4; k += 2) {                   // two channels at a time (packed arithmetic)
          float2 dv = pair_f(&dv4.v[k]);
          sg[k / 2] = dq[k / 2] = make_float2(0.f, 0.f);
          if (softplus) dv = softplus_sigmoid_fast2(__fadd2_rn(dv, make_float2(bias4[k], bias4[k + 1])), sg[k / 2]);
          if (rr >= rows_ok) dv = make_float2(0.f, 0.f);
          const float2 dx2 = __fmul2_rn(dv, pair_f(&xv.v[k]));
          o[k] = dv;
          o[k + 1] = dx2;
          float2 g = pair_f(&yv4.v[k]);
          if (has_z) {
            // silu(z) = z s, its derivative s (1 + z (1 - s))
            const float2 zf = pair_f(&zv4.v[k]), s = sigmoid_fast2(zf);
            const float2 one = make_float2(1.f, 1.f), mone = make_float2(-1.f, -1.f);
            const float2 gs = __fmul2_rn(g, s);
            dq[k / 2] = __fmul2_rn(gs, __ffma2_rn(zf, __ffma2_rn(s, mone, one), one));
            g = __fmul2_rn(gs, zf);
          }
          dyo[k] = g.x;
          dyo[k + 1] = g.y;
        }
        tile[rr * (kBTE / 2) + swz(rr, cc >> 1)] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
        tile[rr * (kBTE / 2) + swz(rr, (cc >> 1) + 1)] = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
        if (softplus || has_z) {
          auxt[rr * (kBTE / 2) + swz(rr, cc >> 1)] = make_float4(sg[0].x, sg[0].y, dq[0].x, dq[0].y);
          auxt[rr * (kBTE / 2) + swz(rr, (cc >> 1) + 1)] = make_float4(sg[1].x, sg[1].y, dq[1].x, dq[1].y);
        }
        *reinterpret_cast<float4*>(dyt + rr * kBTE + cc) = make_float4(dyo[0], dyo[1], dyo[2], dyo[3]);
      }
      const T* rB = reinterpret_cast<const T*>(st + 4 * S::kActBytes);      // B box then C box
      float2* dst = reinterpret_cast<float2*>(s_BC + buf * kBTile * (N / 2));
      constexpr int kBcVecs = kBTile * N / 4;                                // 64
#pragma unroll
      for (int i = 0; i < 2 * kBcVecs / 32; ++i) {
        const int v = lane + 32 * i, q = v % kBcVecs;                        // four states of one row of B, then of C
        const Vec4<T> r4 = *reinterpret_cast<const Vec4<T>*>(rB + v * 4);
        dst[4 * q + (v >= kBcVecs)] = make_float2(Elem<T>::to_f(r4.v[0]), Elem<T>::to_f(r4.v[1]));
        dst[4 * q + 2 + (v >= kBcVecs)] = make_float2(Elem<T>::to_f(r4.v[2]), Elem<T>::to_f(r4.v[3]));
      }
      mbar_arrive(&op_full[buf]);
      mbar_arrive(&raw_free[j % kStages]);
      if (lane == 0 && j + kAhead < ntiles && !issue(j + kAhead)) { fail(); return; }
    }
    return;
  }

  if (warp == 6) {
    // ================================================================== dB, dC: sums over channels
    // A lane owns one row of products (timestep of the window, state pair) and one half of the CTA's 16 channel pairs: it adds
    // its 8 float4 {dB, dB, dC, dC}.  The lanes of a quarter-warp start at different channel pairs, which keeps their loads out of
    // each other's banks.  Neighbouring lanes then swap halves, so that each holds four consecutive states of dB or of dC and
    // sends them to global memory with one vector atomic.
    const int hf = lane >> 4, r = lane & 15, ti = r >> 3, which = r & 1;
    int t = tile_t0(0) + win_row(0, ti);
    float* gptr = (which ? p.dC : p.dB) + (b * p.L + t) * N + 4 * ((r & 7) >> 1);
    for (int j = 0; j < ntiles; ++j) {
#pragma unroll 1
      for (int wl = 0; wl < kWinsPerTile; ++wl) {
        const int wseq = j * kWinsPerTile + wl;
        const int wb = wseq & 1;
        if (!mbar_wait(&win_full[wb], (wseq >> 1) & 1)) { fail(); return; }
        const float4* rowp = s_ep + wb * kBWin * kEpStep + r * 16 + hf * 8;
        float2 acc0 = make_float2(0.f, 0.f), acc1 = acc0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = rowp[c ^ (r & 7)];
          acc0 = __fadd2_rn(acc0, make_float2(v.x, v.y));
          acc1 = __fadd2_rn(acc1, make_float2(v.z, v.w));
        }
        mbar_arrive(&win_empty[wb]);
        const float2 give = which ? acc0 : acc1;
        const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, give.x, 1), __shfl_xor_sync(0xffffffffu, give.y, 1));
        const float2 lo = which ? got : acc0, hi = which ? acc1 : got;
        if (t < t_hi) red_add_v4(gptr, lo.x, lo.y, hi.x, hi.y);
        t += rev ? kBWin : -kBWin;
        gptr += (rev ? kBWin : -kBWin) * N;
      }
    }
    return;
  }

  // ==================================================================== warps 5, 7: dx, ddelta, dz
  {
    const int par = (warp == 5) ? 0 : 1;                 // parity of the windows this warp finishes
    const int ti = lane >> 4, c0 = (lane & 15) * 2;
    int t = tile_t0(0) + win_row(par, ti);
    T* odx = static_cast<T*>(p.dx) + b * p.dx_sb + e0 + c0 + t * p.dx_sl;
    T* odd = static_cast<T*>(p.ddelta) + b * p.dd_sb + e0 + c0 + t * p.dd_sl;
    T* odz = has_z ? static_cast<T*>(p.dz) + b * p.dz_sb + e0 + c0 + t * p.dz_sl : nullptr;
    constexpr int kMove = rev ? 2 * kBWin : -2 * kBWin;   // rows between two windows of this warp
    const float* const np = s_np + (par * kBWin + ti) * kNpStep + c0;
    const int row0 = win_row(par, ti), swz0 = swz(row0, c0 >> 1);     // all rows of a lane have one parity
    const float2 Dv = make_float2(s_D[c0], s_D[c0 + 1]);
    float2 dDacc = make_float2(0.f, 0.f), dbacc = dDacc;
    for (int j = 0; j < ntiles; ++j) {
      if (!mbar_wait(&raw_full[j % kStages], int((j / kStages) & 1))) { fail(); return; }
      const T* rx = reinterpret_cast<const T*>(stage_ptr(j)) + row0 * kBTE + c0;
      // delta, dy' and the derivatives come from the operand tile the consumers are reading (still held: this warp
      // is one of the arrivals the converter waits for before it reuses the buffer)
      const int buf = int(j & 1);
      const float4* opt = s_op + (buf * kBTile + row0) * (kBTE / 2) + swz0;
      const float4* auxt = s_aux + (buf * kBTile + row0) * (kBTE / 2) + swz0;
      const float* dyt = s_dyp + (buf * kBTile + row0) * kBTE + c0;
#pragma unroll 1
      for (int wk = 0; wk < kWinsPerTile / 2; ++wk) {
        if (!mbar_wait(&win_full[par], wk & 1)) { fail(); return; }
        const int tt = wk * kMove;                       // row inside the tile, from row0
        float2 sums[3];                                  // of y, dx, ddelta, over the 4 state quads of both channels
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          float2 q[kBN / 4];
#pragma unroll
          for (int k = 0; k < kBN / 4; ++k) q[k] = *reinterpret_cast<const float2*>(np + v * kNpPlane + k * kBTE);
#pragma unroll
          for (int w = kBN / 8; w > 0; w /= 2)
#pragma unroll
            for (int k = 0; k < w; ++k) q[k] = __fadd2_rn(q[k], q[k + w]);
          sums[v] = q[0];
        }
        mbar_arrive(&win_empty[par]);
        if (t < t_hi && c0 < cols_ok) {
          const Vec2<T> xv = *reinterpret_cast<const Vec2<T>*>(rx + tt * kBTE);
          const float2 dv = *reinterpret_cast<const float2*>(opt + tt * (kBTE / 2));
          const float2 dyg2 = *reinterpret_cast<const float2*>(dyt + tt * kBTE);
          float4 aux = make_float4(0.f, 0.f, 0.f, 0.f);
          if (softplus || has_z) aux = auxt[tt * (kBTE / 2)];
          Vec2<T> ox, od, oz;
          const float2 xf = pair_f(&xv.v[0]), gB = sums[1];
          if (has_z) pair_to(&oz.v[0], __fmul2_rn(make_float2(aux.z, aux.w), __ffma2_rn(Dv, xf, sums[0])));
          pair_to(&ox.v[0], __ffma2_rn(dyg2, Dv, __fmul2_rn(dv, gB)));
          float2 dd = __ffma2_rn(xf, gB, __fmul2_rn(sums[2], make_float2(1.f / kLog2e, 1.f / kLog2e)));
          if (softplus) dd = __fmul2_rn(dd, make_float2(aux.x, aux.y));
          dDacc = __ffma2_rn(dyg2, xf, dDacc);               // of channels past the end: never added up
          dbacc = __fadd2_rn(dbacc, dd);
          pair_to(&od.v[0], dd);
          if (c0 + 2 <= cols_ok) {
            *reinterpret_cast<Vec2<T>*>(odx) = ox;
            *reinterpret_cast<Vec2<T>*>(odd) = od;
            if (has_z) *reinterpret_cast<Vec2<T>*>(odz) = oz;
          } else {
            *odx = ox.v[0];
            *odd = od.v[0];
            if (has_z) *odz = oz.v[0];
          }
        }
        t += kMove;
        odx += kMove * p.dx_sl;
        odd += kMove * p.dd_sl;
        if (has_z) odz += kMove * p.dz_sl;
      }
      mbar_arrive(&op_empty[buf]);
      mbar_arrive(&raw_free[j % kStages]);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (c0 + k < cols_ok) {
        if (p.dD) atomicAdd(p.dD + e0 + c0 + k, k ? dDacc.y : dDacc.x);
        if (p.ddelta_bias) atomicAdd(p.ddelta_bias + e0 + c0 + k, k ? dbacc.y : dbacc.x);
      }
    }
  }
}

}  // namespace
}  // namespace mb200

namespace mb200 {
namespace {

template <typename T>
int bwd_tma_launch(const SscanBwdParams& p, cudaStream_t st) {
  using S = TmaBwdSmem<T>;
  constexpr bool bf = sizeof(T) == 2;
  BwdMaps m;
  bool ok = tma_encode(&m.x, p.x, bf, p.B, p.L, p.ED, p.x_sb, p.x_sl, kBTE, kBTile) &&
            tma_encode(&m.d, p.delta, bf, p.B, p.L, p.ED, p.d_sb, p.d_sl, kBTE, kBTile) &&
            tma_encode(&m.dy, p.dy, bf, p.B, p.L, p.ED, p.dy_sb, p.dy_sl, kBTE, kBTile) &&
            tma_encode(&m.B, p.Bm, bf, p.B, p.L, kBN, p.b_sb, p.b_sl, kBN, kBTile) &&
            tma_encode(&m.C, p.Cm, bf, p.B, p.L, kBN, p.c_sb, p.c_sl, kBN, kBTile);
  if (ok && p.z) ok = tma_encode(&m.z, p.z, bf, p.B, p.L, p.ED, p.z_sb, p.z_sl, kBTE, kBTile);
  else if (ok) m.z = m.x;
  if (!ok) return 1;                                   // caller falls back to the generic path
  const bool rv = (p.flags & MB200_REVERSE) != 0, sp = (p.flags & MB200_DELTA_SOFTPLUS) != 0, hz = p.z != nullptr;
  void (*k)(const BwdMaps, const SscanBwdParams) = nullptr;
#define MB200_BWD_PICK(R, S, Z) if (rv == R && sp == S && hz == Z) k = sscan_bwd_tma_kernel<T, R, S, Z>;
  MB200_BWD_PICK(false, false, false) MB200_BWD_PICK(false, false, true)
  MB200_BWD_PICK(false, true, false) MB200_BWD_PICK(false, true, true)
  MB200_BWD_PICK(true, false, false) MB200_BWD_PICK(true, false, true)
  MB200_BWD_PICK(true, true, false) MB200_BWD_PICK(true, true, true)
#undef MB200_BWD_PICK
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes) != cudaSuccess)
    return MB200_ELAUNCH;
  dim3 grid(unsigned((p.ED + kBTE - 1) / kBTE), unsigned(p.B), unsigned(p.pieces));
  k<<<grid, kBwdThreads, S::kBytes, st>>>(m, p);
  return check_launch();
}

bool bwd_tma_path_ok(const SscanBwdParams& p, int N, int es) {
  if (N != kBN || p.L >= (int64_t(1) << 31) || p.ED >= (int64_t(1) << 31)) return false;
  bool ok = tma_compatible(p.x, p.x_sb, p.x_sl, p.ED, es, kBTE) &&
            tma_compatible(p.delta, p.d_sb, p.d_sl, p.ED, es, kBTE) &&
            tma_compatible(p.dy, p.dy_sb, p.dy_sl, p.ED, es, kBTE) &&
            tma_compatible(p.Bm, p.b_sb, p.b_sl, N, es, N) &&
            tma_compatible(p.Cm, p.c_sb, p.c_sl, N, es, N);
  if (p.z) ok = ok && tma_compatible(p.z, p.z_sb, p.z_sl, p.ED, es, kBTE) && aligned16(p.dz) &&
                (p.dz_sl * es) % 16 == 0 && (p.dz_sb * es) % 16 == 0;
  ok = ok && aligned16(p.dx) && aligned16(p.ddelta) && (p.dx_sl * es) % 16 == 0 && (p.dx_sb * es) % 16 == 0 &&
       (p.dd_sl * es) % 16 == 0 && (p.dd_sb * es) % 16 == 0 && aligned16(p.dB) && aligned16(p.dC);
  return ok && tma_encoder() != nullptr;
}

}  // namespace
}  // namespace mb200

using namespace mb200;

// Reads (and clears) the device-side status word of the backward kernel.  Synchronises the device.
int mb200_bwd_device_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_bwd_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_bwd_status, &zero, sizeof(int));
  return v;
}

extern "C" int mb200_sscan_bwd_pieces(const void* x, const void* delta, const void* z, const float* A,
                               const void* Bm, const void* Cm, const float* D,
                               const float* delta_bias, const void* dy, const float* carries,
                               const float* g_in, void* dx, void* ddelta, void* dz, float* dB,
                               float* dC, float* dA, float* dD, float* ddelta_bias, float* g_out,
                               int64_t B, int64_t L, int64_t ED, int N,
                               int64_t x_sb, int64_t x_sl, int64_t d_sb, int64_t d_sl,
                               int64_t z_sb, int64_t z_sl, int64_t b_sb, int64_t b_sl,
                               int64_t c_sb, int64_t c_sl, int64_t dy_sb, int64_t dy_sl,
                               int64_t dx_sb, int64_t dx_sl, int64_t dd_sb, int64_t dd_sl,
                               int64_t dz_sb, int64_t dz_sl, int dtype, int flags, int64_t pieces, int64_t piece_len,
                               void* stream) {
  if (B < 0 || L < 0 || ED < 0) return MB200_EINVAL;
  if (dtype != MB200_F32 && dtype != MB200_BF16) return MB200_EDTYPE;
  if (N != 8 && N != 16 && N != 32 && N != 64) return MB200_ENSTATE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (B == 0 || ED == 0) return MB200_OK;
  if (L == 0) {                                   // nothing to differentiate; the carry passes through
    if (g_out) {
      if (g_in) cudaMemcpyAsync(g_out, g_in, sizeof(float) * B * ED * N, cudaMemcpyDeviceToDevice, st);
      else cudaMemsetAsync(g_out, 0, sizeof(float) * B * ED * N, st);
    }
    return check_launch();
  }
  if (!x || !delta || !A || !Bm || !Cm || !dy || !carries || !dx || !ddelta || !dB || !dC || !dA)
    return MB200_EINVAL;
  if (z && !dz) return MB200_EINVAL;
  if ((flags & MB200_DELTA_SOFTPLUS) && !delta_bias) return MB200_EINVAL;
  if (B > 65535 || pieces > 65535) return MB200_ETOOBIG;
  if (!pieces_ok(pieces, piece_len, L)) return MB200_EINVAL;
  if (!aligned16(carries) || !aligned16(g_in) || !aligned16(g_out)) return MB200_EALIGN;
  SscanBwdParams p;
  p.x = x; p.delta = delta; p.z = z; p.Bm = Bm; p.Cm = Cm; p.dy = dy; p.A = A; p.D = D;
  p.delta_bias = delta_bias; p.carries = carries; p.g_in = g_in;
  p.dx = dx; p.ddelta = ddelta; p.dz = dz; p.dB = dB; p.dC = dC; p.dA = dA; p.dD = dD;
  p.ddelta_bias = ddelta_bias; p.g_out = g_out;
  p.B = B; p.L = L; p.ED = ED;
  p.x_sb = x_sb; p.x_sl = x_sl; p.d_sb = d_sb; p.d_sl = d_sl; p.z_sb = z_sb; p.z_sl = z_sl;
  p.b_sb = b_sb; p.b_sl = b_sl; p.c_sb = c_sb; p.c_sl = c_sl; p.dy_sb = dy_sb; p.dy_sl = dy_sl;
  p.dx_sb = dx_sb; p.dx_sl = dx_sl; p.dd_sb = dd_sb; p.dd_sl = dd_sl; p.dz_sb = dz_sb; p.dz_sl = dz_sl;
  p.flags = flags;
  if (pieces > 1) { p.pieces = pieces; p.piece_len = piece_len; }
  const int es = dtype == MB200_F32 ? 4 : 2;
  if (bwd_tma_path_ok(p, N, es)) {
    const int rc = dtype == MB200_F32 ? bwd_tma_launch<float>(p, st) : bwd_tma_launch<__nv_bfloat16>(p, st);
    if (rc <= 0) return rc;
  }
  if (pieces > 1) {                                // as extra batch rows, where the strides allow it
    if (g_out || !pieces_as_rows(B, L, pieces, piece_len, {x_sb, d_sb, z ? z_sb : L * z_sl, b_sb, c_sb, dy_sb, dx_sb, dd_sb, z ? dz_sb : L * dz_sl},
                                 {x_sl, d_sl, z_sl, b_sl, c_sl, dy_sl, dx_sl, dd_sl, dz_sl}))
      return MB200_EUNSUPPORTED;
    const int64_t n = piece_len;
    return mb200_sscan_bwd(x, delta, z, A, Bm, Cm, D, delta_bias, dy, carries, g_in, dx, ddelta, dz, dB, dC, dA, dD, ddelta_bias, nullptr,
                           B * pieces, n, ED, N, n * x_sl, x_sl, n * d_sl, d_sl, n * z_sl, z_sl, n * b_sl, b_sl, n * c_sl, c_sl, n * dy_sl,
                           dy_sl, n * dx_sl, dx_sl, n * dd_sl, dd_sl, n * dz_sl, dz_sl, dtype, flags, stream);
  }
  if (flags & MB200_REVERSE) return MB200_EUNSUPPORTED;   // the reverse direction exists on the tensor-map path only
  const int kv = dtype == MB200_F32 ? 4 : 8;
  bool vec = ED % kv == 0;
  for (const void* q : {x, delta, z, Bm, Cm, dy, (const void*)dx, (const void*)ddelta, (const void*)dz})
    vec = vec && aligned16(q);
  for (int64_t s : {x_sb, x_sl, d_sb, d_sl, b_sb, b_sl, c_sb, c_sl, dy_sb, dy_sl, dx_sb, dx_sl, dd_sb, dd_sl})
    vec = vec && s % kv == 0;
  if (z) vec = vec && z_sb % kv == 0 && z_sl % kv == 0 && dz_sb % kv == 0 && dz_sl % kv == 0;
  return dtype == MB200_F32 ? bwd_generic_launch_t<float>(p, N, vec, st)
                            : bwd_generic_launch_t<__nv_bfloat16>(p, N, vec, st);
}

extern "C" int mb200_sscan_bwd(const void* x, const void* delta, const void* z, const float* A,
                               const void* Bm, const void* Cm, const float* D,
                               const float* delta_bias, const void* dy, const float* carries,
                               const float* g_in, void* dx, void* ddelta, void* dz, float* dB,
                               float* dC, float* dA, float* dD, float* ddelta_bias, float* g_out,
                               int64_t B, int64_t L, int64_t ED, int N,
                               int64_t x_sb, int64_t x_sl, int64_t d_sb, int64_t d_sl,
                               int64_t z_sb, int64_t z_sl, int64_t b_sb, int64_t b_sl,
                               int64_t c_sb, int64_t c_sl, int64_t dy_sb, int64_t dy_sl,
                               int64_t dx_sb, int64_t dx_sl, int64_t dd_sb, int64_t dd_sl,
                               int64_t dz_sb, int64_t dz_sl, int dtype, int flags, void* stream) {
  return mb200_sscan_bwd_pieces(x, delta, z, A, Bm, Cm, D, delta_bias, dy, carries, g_in, dx, ddelta, dz, dB, dC, dA, dD, ddelta_bias, g_out,
                                B, L, ED, N, x_sb, x_sl, d_sb, d_sl, z_sb, z_sl, b_sb, b_sl, c_sb, c_sl, dy_sb, dy_sl, dx_sb, dx_sl,
                                dd_sb, dd_sl, dz_sb, dz_sl, dtype, flags, 1, 0, stream);
}

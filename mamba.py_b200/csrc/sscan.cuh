// Geometry and parameter blocks shared by the fused selective-scan kernels.
#pragma once
#include <initializer_list>
#include "common.cuh"
#include "tile.cuh"

namespace mb200 {

// Timesteps between two saved states.  The backward kernels keep the states of one chunk in
// registers while they walk it in reverse (kChunk * 4 floats per thread), which fixes this at 8:
// the saved states cost kChunk times less memory than the full state tensor the reference keeps.
constexpr int kChunk = 8;

// A thread owns 4 states of one channel, so N/4 lanes share a channel and a 128-thread CTA
// covers 128/(N/4) channels.  kTT is the number of timesteps staged per shared-memory tile.
template <int N> struct SscanGeom {
  static_assert(N % 4 == 0 && N >= 8 && N <= 64, "d_state must be 8, 16, 32 or 64");
  static constexpr int kLPE = N / 4;                       // lanes per channel
  static constexpr int kTE = kThreadsPerCta / kLPE;        // channels per CTA
  static constexpr int kTT = (N == 16 || N == 32) ? 32 : 16;   // timesteps per tile (fits 48 KB static smem)
};

// The operand tile holds one float2 {delta, delta*x} per (timestep, channel).  Two channels share
// a 16-byte slot; slot s of row t is stored at physical slot swz(t, s).  The XOR spreads the
// slots that one quarter-warp of the commit writes together (and odd/even rows) over different
// banks, so the commit's 128-bit stores and the hot loop's 64-bit loads are conflict free.
__device__ __forceinline__ int swz(int t, int s) {
  return s ^ ((s >> 3) & 1) ^ ((t & 1) << 1);
}
// float2 index of channel column c in row t of a tile that is `te` channels wide
__device__ __forceinline__ int op_index(int t, int c, int te) {
  return t * te + swz(t, c >> 1) * 2 + (c & 1);
}

// four consecutive channels of one timestep, moved with one 8- or 16-byte access
template <typename T> struct alignas(sizeof(T) * 4) Vec4 {
  T v[4];
};

// Sum of the kLPE partial sums the lanes of one channel left in shared memory.
template <int kLPE>
__device__ __forceinline__ float sum_lanes(const float* p) {
  if constexpr (kLPE == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return v.x + v.y;
  } else {
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < kLPE; l += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + l);
      s += (v.x + v.y) + (v.z + v.w);
    }
    return s;
  }
}

// Commit the fetched B and C tiles (kTT-or-kChunk rows of N values) to shared memory as float32.
template <typename T, int N, int KVB, typename Regs>
__device__ __forceinline__ void commit_bc(const Regs& rB, const Regs& rC, float* sB, float* sC, int tid) {
  using Map = typename Regs::Map;
#pragma unroll
  for (int i = 0; i < Map::kPerThread; ++i) {
    if (!Map::owns(i, tid)) continue;
    const int rr = Map::row(i, tid), cc = Map::col(i, tid);
    float* db = sB + rr * N + cc;
    float* dc = sC + rr * N + cc;
    if constexpr (KVB % 4 == 0) {
#pragma unroll
      for (int k = 0; k < KVB; k += 4) {
        *reinterpret_cast<float4*>(db + k) =
            make_float4(Elem<T>::to_f(rB.r[i].v[k]), Elem<T>::to_f(rB.r[i].v[k + 1]),
                        Elem<T>::to_f(rB.r[i].v[k + 2]), Elem<T>::to_f(rB.r[i].v[k + 3]));
        *reinterpret_cast<float4*>(dc + k) =
            make_float4(Elem<T>::to_f(rC.r[i].v[k]), Elem<T>::to_f(rC.r[i].v[k + 1]),
                        Elem<T>::to_f(rC.r[i].v[k + 2]), Elem<T>::to_f(rC.r[i].v[k + 3]));
      }
    } else {
#pragma unroll
      for (int k = 0; k < KVB; ++k) {
        db[k] = Elem<T>::to_f(rB.r[i].v[k]);
        dc[k] = Elem<T>::to_f(rC.r[i].v[k]);
      }
    }
  }
}

// Where the saved state {2k, 2k+1} of channel e lies inside an entry of ED x N floats: next to the channel's other states, or
// (MB200_PAIRED_STATES) next to the same pair of the neighbouring channels.
__host__ __device__ __forceinline__ int64_t state_pair(bool paired, int64_t ED, int N, int64_t e, int k) {
  return paired ? (k * ED + e) * 2 : e * N + 2 * k;
}
// Four consecutive states from 4q on.
__device__ __forceinline__ void store_states(float* entry, bool paired, int64_t ED, int N, int64_t e, int q, float4 h) {
  if (paired) {
    *reinterpret_cast<float2*>(entry + state_pair(true, ED, N, e, 2 * q)) = make_float2(h.x, h.y);
    *reinterpret_cast<float2*>(entry + state_pair(true, ED, N, e, 2 * q + 1)) = make_float2(h.z, h.w);
  } else {
    *reinterpret_cast<float4*>(entry + e * N + 4 * q) = h;
  }
}
__device__ __forceinline__ float4 load_states(const float* entry, bool paired, int64_t ED, int N, int64_t e, int q) {
  if (!paired) return *reinterpret_cast<const float4*>(entry + e * N + 4 * q);
  const float2 lo = *reinterpret_cast<const float2*>(entry + state_pair(true, ED, N, e, 2 * q));
  const float2 hi = *reinterpret_cast<const float2*>(entry + state_pair(true, ED, N, e, 2 * q + 1));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

struct SscanFwdParams {
  const void *x, *delta, *z, *Bm, *Cm;
  const float *A, *D, *delta_bias, *h0;
  void* y;
  float *hT, *carries;
  float* pT = nullptr;         // (B, ED, N) decay product of the whole span; written by the state-only pass
  int64_t B, L, ED;
  int64_t x_sb, x_sl, d_sb, d_sl, z_sb, z_sl, b_sb, b_sl, c_sb, c_sl, y_sb, y_sl;
  int flags;
  // A sequence cut into `pieces` spans of piece_len timesteps (a multiple of 16; the last may be shorter) that are scanned
  // side by side: h0, and the state and decay product of the passes without y, are then (B, pieces, ED, N).  A launch
  // covers launch_pieces of them from piece0.
  int64_t pieces = 1, piece_len = int64_t(1) << 40, piece0 = 0, launch_pieces = 1;
};

struct SscanBwdParams {
  const void *x, *delta, *z, *Bm, *Cm, *dy;
  const float *A, *D, *delta_bias, *carries, *g_in;
  void *dx, *ddelta, *dz;
  float *dB, *dC, *dA, *dD, *ddelta_bias, *g_out;
  int64_t B, L, ED;
  int64_t x_sb, x_sl, d_sb, d_sl, z_sb, z_sl, b_sb, b_sl, c_sb, c_sl, dy_sb, dy_sl;
  int64_t dx_sb, dx_sl, dd_sb, dd_sl, dz_sb, dz_sl;
  int flags;
  int64_t pieces = 1, piece_len = int64_t(1) << 40;      // as in the forward; g_in is then (B, pieces, ED, N)
};

}  // namespace mb200

// Pieces of a sequence: their length is a multiple of the kernels' 16-step tiles and each holds at least one timestep.
namespace mb200 {
inline bool pieces_ok(int64_t pieces, int64_t piece_len, int64_t L) {
  return pieces == 1 || (pieces > 1 && piece_len > 0 && piece_len % 16 == 0 && (pieces - 1) * piece_len < L);
}
// Whether (B, pieces) can be read as one batch dimension: even pieces, and batch strides that continue the rows.
inline bool pieces_as_rows(int64_t B, int64_t L, int64_t pieces, int64_t piece_len, std::initializer_list<int64_t> sb,
                           std::initializer_list<int64_t> sl) {
  if (pieces * piece_len != L || B * pieces > 65535) return false;
  auto l = sl.begin();
  for (int64_t s : sb)
    if (B > 1 && s != L * *l++) return false;
  return true;
}
}  // namespace mb200

// Internal flag (never part of the public flags): run the forward kernel as the reverse carry pass.
namespace mb200 { constexpr int kFlagCarryPass = 1 << 16; }
int mb200_fwd_tma_try(const mb200::SscanFwdParams& p, int N, int dtype, cudaStream_t st);

// Device-side status words of the kernels that contain bounded waits (host functions; each reads
// and clears its kernel's word, synchronising the device).
int mb200_fwd_device_status();
int mb200_bwd_device_status();
int mb200_block_step_device_status();

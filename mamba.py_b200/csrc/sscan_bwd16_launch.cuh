// Instantiation and launch of the d_state 16 backward for one element type (included by one source per type).
#pragma once
#include "sscan_bwd16.cuh"

namespace mb200 {
namespace {

template <typename T>
int bwd16_launch(const SscanBwdParams& p, bool carry_only, cudaStream_t st) {
  using S = Bwd16Smem<T>;
  constexpr bool bf = sizeof(T) == 2;
  constexpr int es = int(sizeof(T));
  auto fits = [&](const void* q, int64_t sb, int64_t sl) { return tma_compatible(q, sb, sl, p.ED, es, kWCh); };
  if (p.L >= (int64_t(1) << 31) || p.ED >= (int64_t(1) << 31) || !tma_encoder()) return 1;
  if (!fits(p.x, p.x_sb, p.x_sl) || !fits(p.delta, p.d_sb, p.d_sl) || !fits(p.dy, p.dy_sb, p.dy_sl) || (p.z && !fits(p.z, p.z_sb, p.z_sl)))
    return 1;
  Bwd16Maps m;
  auto encode = [&](CUtensorMap* map, const void* q, int64_t sb, int64_t sl) {
    return tma_encode(map, q, bf, p.B, p.L, p.ED, sb, sl, kWCh, kChunk);
  };
  if (!encode(&m.x, p.x, p.x_sb, p.x_sl) || !encode(&m.d, p.delta, p.d_sb, p.d_sl) || !encode(&m.dy, p.dy, p.dy_sb, p.dy_sl)) return 1;
  if (p.z) {
    if (!encode(&m.z, p.z, p.z_sb, p.z_sl)) return 1;
  } else {
    m.z = m.x;
  }
  if (!carry_only) {
    if (!fits(p.dx, p.dx_sb, p.dx_sl) || !fits(p.ddelta, p.dd_sb, p.dd_sl) || (p.z && !fits(p.dz, p.dz_sb, p.dz_sl))) return 1;
    if (!encode(&m.dx, p.dx, p.dx_sb, p.dx_sl) || !encode(&m.dd, p.ddelta, p.dd_sb, p.dd_sl)) return 1;
    if (p.z && !encode(&m.dz, p.dz, p.dz_sb, p.dz_sl)) return 1;
  }
  const bool rv = (p.flags & MB200_REVERSE) != 0, sp = (p.flags & MB200_DELTA_SOFTPLUS) != 0, hz = p.z != nullptr;
  void (*k)(const Bwd16Maps, const SscanBwdParams) = nullptr;
#define MB200_PICK(R, SP, Z)                                                                              \
  if (rv == R && sp == SP && hz == Z)                                                                     \
    k = carry_only ? sscan_bwd16_kernel<T, R, SP, Z, true> : sscan_bwd16_kernel<T, R, SP, Z, false>;
  MB200_PICK(false, false, false) MB200_PICK(false, false, true) MB200_PICK(false, true, false) MB200_PICK(false, true, true)
  MB200_PICK(true, false, false) MB200_PICK(true, false, true) MB200_PICK(true, true, false) MB200_PICK(true, true, true)
#undef MB200_PICK
  static_assert(S::kBytes <= 48 * 1024, "no opt-in to large shared memory needed");
  cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  const dim3 grid(unsigned((p.ED + kWCh - 1) / kWCh), unsigned(p.B), unsigned(p.launch_pieces));
  k<<<grid, 32, S::kBytes, st>>>(m, p);
  return check_launch();
}

// Reads and clears this translation unit's status word.  Synchronises the device.
int bwd16_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_bwd16_status, sizeof(int)) != cudaSuccess) return -1;
  if (v) cudaMemcpyToSymbol(g_bwd16_status, &zero, sizeof(int));
  return v;
}

}  // namespace
}  // namespace mb200

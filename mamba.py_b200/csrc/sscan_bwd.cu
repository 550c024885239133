// Entry points of the fused selective scan backward.  Kernels: sscan_bwd16.cuh (d_state 16, tensors a tensor map can describe),
// sscan_bwd_generic.cuh (everything else).
#include "sscan_bwd_generic.cuh"

using namespace mb200;

// Reads (and clears) the device-side status words of the backward kernels.  Synchronises the device.
int mb200_bwd_device_status() {
  const int a = bwd16_status_f32(), b = bwd16_status_bf16();
  return a ? a : b;
}

extern "C" int mb200_sscan_bwd_split(const void* x, const void* delta, const void* z, const float* A,
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
                               float* ws, void* stream) {
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
  if (pieces < 1 || (pieces > 1 && (!ws || !aligned16(ws) || piece_len < kChunk || piece_len % kChunk || (pieces - 1) * piece_len >= L)))
    return MB200_EINVAL;
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
  const int es = dtype == MB200_F32 ? 4 : 2;
  if (N == 16) {
    auto launch = [&](const SscanBwdParams& q, bool carry_only) {
      return dtype == MB200_F32 ? bwd16_launch_f32(q, carry_only, st) : bwd16_launch_bf16(q, carry_only, st);
    };
    p.pieces = p.launch_pieces = pieces;
    if (pieces > 1) {
      p.piece_len = piece_len;
      p.piece_P = ws;
      p.piece_G = ws + B * pieces * ED * N;
      // the piece at the scan's start is left out of the carry pass: its carry feeds nothing
      SscanBwdParams c = p;
      c.launch_pieces = pieces - 1;
      c.piece0 = (flags & MB200_REVERSE) ? 0 : 1;
      const int rc = launch(c, true);
      if (rc < 0) return rc;
      if (rc == 1) p.pieces = p.launch_pieces = 1;             // not for these tensors: one span
    }
    const int rc = launch(p, false);
    if (rc <= 0) return rc;
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
  return mb200_sscan_bwd_split(x, delta, z, A, Bm, Cm, D, delta_bias, dy, carries, g_in, dx, ddelta, dz, dB, dC, dA, dD, ddelta_bias, g_out,
                               B, L, ED, N, x_sb, x_sl, d_sb, d_sl, z_sb, z_sl, b_sb, b_sl, c_sb, c_sl, dy_sb, dy_sl, dx_sb, dx_sl,
                               dd_sb, dd_sl, dz_sb, dz_sl, dtype, flags, 1, 0, nullptr, stream);
}

// The fused scan on prepared tensors: forward and backward with the choice between one launch and rows cut into pieces.
#pragma once
#include "host.h"

namespace mb200_host {

// The tensors of a scan as the kernels take them: one activation dtype, unit-stride last dimension, float32 parameters.
struct ScanArgs {
  Tensor x, delta, A, B, C, D, z, bias, h0;
  bool reverse = false;
  int flags() const { return (bias.defined() ? MB200_DELTA_SOFTPLUS : 0) | (reverse ? MB200_REVERSE : 0) | MB200_PAIRED_STATES; }
  int code() const { return dtype_code(x.scalar_type()); }
  int64_t batch() const { return x.size(0); }
  int64_t length() const { return x.size(1); }
  int64_t width() const { return x.size(2); }
  int64_t states() const { return A.size(1); }
};
struct ScanOut {
  Tensor y, hT, carries, P;
};
struct ScanGrads {
  Tensor dx, dd, dz, dB, dC, dA, dD, dbias, g_out;
  Tensor extra;                        // zero-filled float32 asked for along with the accumulators
};

// 16-byte aligned base and byte strides: what a tiled tensor map of a (B, L, C) tensor needs.
bool tensor_map_ok(const Tensor& t);
bool tensor_maps_ok(const ScanArgs& a);

// The number of pieces these tensors can be cut into, at most S: any number when every pass takes the tensor-map path, a power of
// two that divides the sequence when the pieces have to be read as extra batch rows.
int64_t cuttable(const ScanArgs& a, int64_t S, bool grad, bool want_last);

// S consecutive pieces per row; S = 1 is the single launch.  False (S = 1 only) when the kernels cannot scan these tensors
// in reverse.
bool scan_forward(const ScanArgs& a, int64_t S, bool want_last, bool want_carries, ScanOut& o);
// Where a caller wants gradients written (dz may be a strided view), and how many zeroed floats behind the accumulators.
struct ScanSinks {
  Tensor dz, dx, dd;
  int64_t extra = 0;
};
ScanGrads scan_backward(const ScanArgs& a, int64_t S, const Tensor& dy, const Tensor& carries, const Tensor& P, bool want_g_out,
                        const ScanSinks& to = {});

}  // namespace mb200_host

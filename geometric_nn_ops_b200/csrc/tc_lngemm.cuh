// LayerNorm fused into the projection GEMMs of the triangle multiplicative update (16-bit dtypes, 128 channels).
//
//   ln_gate_in   x -> z = LayerNorm(x) normalised in shared memory, then both halves of
//                a | b = (z Wp^T + bp) * sigmoid(z Wg^T + bg) * mask, channel-major; z and the row statistics are
//                written out for the output gate and the backward pass.
//   ln_gate_out  t (channel-major) -> u = LayerNorm over channels, normalised in shared memory in the layout the
//                contraction left it in (the MMA reads it as an MN-major operand, so nothing is transposed), then
//                out = (u Wo^T + bo) * sigmoid(z Wgo^T + bgo); u is kept channel-major for the backward pass.
//   gate_in_bwd  z, da, db -> dP, dG of both halves and the input weights' gradients (no LayerNorm: the same kernel shape with
//                resident weights).
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {

// Does pixel px of planes of [pitch, pitch] pixels that hold [n, n] lie beyond them?  (n = 0: nothing does)
__device__ __forceinline__ bool pad_pixel(long long px, int n, int pitch) {
  if (n == 0) return false;
  const long long plane = (long long)pitch * pitch;
  const int p = (int)(px % plane);
  return p / pitch >= n || p % pitch >= n;
}
// 1 / sqrt(var + eps) of pixel px.  A pad's variance is zero, and with eps = 0 its infinity, times its zeros, would reach every
// pixel through the contraction: 0 there, so that a pad is normalised to the bias as with any other eps.
__device__ __forceinline__ float pixel_rstd(float var, float eps, long long px, int n, int pitch) {
  const float rs = 1.0f / sqrtf(var + eps);
  return isinf(rs) && pad_pixel(px, n, pitch) ? 0.0f : rs;
}

struct LnGateIn {
  int dtype;                 // TRI_BF16 / TRI_F16
  long long M, plane;        // pixels in all; pixels per batch entry (channel-plane stride of a / b)
  float eps;
  const void* x;             // [M, 128]
  int n = 0, pitch = 0;      // n > 0: planes of [pitch, pitch] pixels hold [n, n]; x is zero beyond
  bool own_pitch = false;    // x is [n, n, 128] and the mask [n, n] (one batch entry), not [M, 128] and [M]
  const void* gamma;         // [128] or null
  const void* beta;          // [128] or null
  const void* wcat;          // [512, 128]: rows [Wp_a; Wg_a; Wp_b; Wg_b]
  const float* bias_cat;     // [512] in the same row order, or null
  const void* mask;          // [M] in the input dtype, or null
  void* z;                   // [M, 128]
  float* mean;               // [M]
  float* rstd;               // [M]
  void* a_cm;                // [B, 128, plane]
  void* b_cm;
  bool first = false;        // no kernel of this call came before: launched plainly
  int* err;                  // device status word (zeroed by the caller)
};

bool ln_gate_in_supported(int dtype, long long M, long long plane);
int ln_gate_in(cudaStream_t st, const LnGateIn& p);

struct LnGateOut {
  int dtype;                 // TRI_BF16 / TRI_F16
  long long M;               // pixels (one batch entry: the channel planes of t are M pixels apart)
  float eps;
  const void* t_cm;          // [128, M]
  const void* z;             // [M, 128]
  const void* gamma;         // [128] or null
  const void* beta;          // [128] or null
  const void* w_out;         // [128, 128], rows = output channel
  const void* w_gate;        // [128, 128]
  const float* bias_out;     // [256]: output bias, gate bias; or null
  void* u_cm;                // [128, M] or null (inference: nothing to keep)
  float* mean;               // [M]
  float* rstd;               // [M]
  void* out;                 // [M, 128]
  const void* residual = nullptr;   // [M, 128], added to the (rounded) result, or null
  int n = 0, pitch = 0;      // n > 0: the pixels [pitch, pitch] hold [n, n], t is zero beyond
  bool own_pitch = false;    // out is [n, n, 128] (no residual) and not [M, 128]
  bool first = false;        // as above
  int* err;
};

// One batch entry, 64-pixel groups aligned: M a multiple of 64.
bool ln_gate_out_supported(int dtype, long long M, long long plane);
int ln_gate_out(cudaStream_t st, const LnGateOut& p);

// Input gate backward: dP, dG of both halves from the recomputed projections of z and the gradients of a and b, and their
// products with z summed over the pixels.
struct GateInBwd {
  int dtype;                 // fp32: TF32 products
  long long M;               // pixels (one batch entry)
  const void* z;             // [M, 128]
  const void* wcat;          // [512, 128]: rows [Wp_a; Wg_a; Wp_b; Wg_b]
  const float* bias_cat;     // [512] or null
  const void* mask;          // [M] or null
  const void* da_cm;         // [128, M]
  const void* db_cm;
  void* dpg;                 // [512, M]: rows [dP_a; dG_a; dP_b; dG_b]
  float* partial;            // [gate_in_bwd_parts][512, 128]: parts of dPG z, or null
  bool first = false;        // as above
  int* err;
};
bool gate_in_bwd_supported(int dtype, long long M, long long plane);
int gate_in_bwd_parts(int dtype, long long M);   // one for every two SMs at most
int gate_in_bwd(cudaStream_t st, const GateInBwd& p);

}  // namespace tc
}  // namespace tri

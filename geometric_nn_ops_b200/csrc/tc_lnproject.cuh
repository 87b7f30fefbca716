// LayerNorm + q | k | v projection + per-head pair bias in one kernel (16-bit types, 128 channels).
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {

struct LnProject {
  int dtype;                 // TRI_BF16 / TRI_F16
  long long M, plane;        // pixels in all; per batch entry of the head-major bias
  int n_out, heads;          // columns of q | k | v (0: none), heads
  float eps;
  const void* z;             // [M, 128]
  const void* gamma;         // [128] or null
  const void* beta;          // [128] or null
  const void* w_qkv;         // [n_out, 128]
  const void* w_bias;        // [heads, 128]
  void* qkv;                 // [M, n_out]
  void* bias;                // [M / plane][heads][plane]
  int* err;                  // 256 bytes: the status (see leave_status)
};

bool ln_project_supported(int dtype, long long M, int n_out, int heads);
int ln_project(cudaStream_t st, const LnProject& p);

}  // namespace tc
}  // namespace tri

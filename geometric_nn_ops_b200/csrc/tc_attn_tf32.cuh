// fp32 triangle attention with TF32 products on the tensor cores (tc_attn_tf32.cu).
#pragma once

#include "common.cuh"

namespace tri {
namespace tc {

bool attn_tf32_supported(const TriAttnDesc* d, int is_bwd);
size_t attn_tf32_ws_bytes(const TriAttnDesc* d, int is_bwd);
int attn_tf32_forward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, void* o, float* stats,
                      void* ws, size_t ws_size, cudaStream_t st);
int attn_tf32_backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, const void* o,
                       const float* stats, const void* d_o, void* dq, void* dk, void* dv, float* dbias, void* ws, size_t ws_size, cudaStream_t st);

// the additive key-mask terms of a call (see mask_terms_kernel); `flags` [B][S][H]: cleared, and the terms times log2(e) follow
int launch_mask_terms(const TriAttnDesc* d, const uint8_t* mask, float* out, int* err, int* flags, cudaStream_t st);

}  // namespace tc
}  // namespace tri

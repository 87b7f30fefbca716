// fp32 triangle attention with TF32 products on the tensor cores (tc_attn_tf32.cu).
#pragma once

#include "common.cuh"

namespace tri {
namespace tc {

bool attn_tf32_supported(const TriAttnDesc* d, int is_bwd);
size_t attn_tf32_ws_bytes(const TriAttnDesc* d, int is_bwd);
// the workspace has room for what the call needs, a copy of a bias that starts off a 16-byte boundary included
bool attn_tf32_has_room(const TriAttnDesc* d, const void* bias, size_t ws_size, int is_bwd);
int attn_tf32_forward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, void* o, float* stats,
                      void* ws, size_t ws_size, cudaStream_t st);
int attn_tf32_backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, const void* o,
                       const float* stats, const void* d_o, void* dq, void* dk, void* dv, float* dbias, void* ws, size_t ws_size, cudaStream_t st);

// The row chunks of a dbias pass (64 queries x 128 keys per CTA) on `slots` CTAs at a time, the bytes of their partial sums
// (none for one chunk), and their sum in fixed order.
int dbias_row_chunks(const TriAttnDesc* d, int slots);
size_t dbias_partial_bytes(const TriAttnDesc* d, int slots);
int launch_sum_partials(const float* partial, int chunks, long long n, float* out, cudaStream_t st);

}  // namespace tc
}  // namespace tri

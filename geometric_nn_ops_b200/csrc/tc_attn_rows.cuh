// Forward triangle attention that shares a pair-bias tile between three rows (tc_attn_rows.cu).
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {

// rank-5 map over a [B, S, N, H, D] tensor given its (batch, row, residue, head) strides; a box is `rows` residues of
// `width` channels (32 or 64), zero beyond D
int qkv_tile_map(CUtensorMap* out, const void* p, const TriAttnDesc* d, const int64_t* st, int rows, int width);

// its offsets are 32-bit: rows of statistics, and O in 16-byte pieces
bool attn_fwd_rows_fits(const TriAttnDesc* d);
// Boxes: tq 128 queries, tk and tv 64 keys of 32 channels; fp32: operands rounded to TF32, tv in the swizzle with 32-byte atoms,
// more than 64 residues.  tbias: 128 queries x 64 keys (fp32: x 32), or null.  mask_terms: made by
// launch_mask_terms, which clears *err, or null.  `first`: no kernel
// of the call came before.
int attn_fwd_rows(const TriAttnDesc* d, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap* tbias,
                  bool bias_batched, const uint8_t* mask, const float* mask_terms, void* o, float* stats, int* err, bool first, cudaStream_t st);

// The additive key-mask terms of a call, [B][S][N rounded up to 128], for kernels so long that a launch does not show (see
// launch_dependent); the shorter ones make them on the way.
bool wants_mask_terms(const TriAttnDesc* d);
int launch_mask_terms(const TriAttnDesc* d, const uint8_t* mask, float* out, int* err, cudaStream_t st);

}  // namespace tc
}  // namespace tri

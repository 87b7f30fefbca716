// Forward triangle attention that shares a pair-bias tile between three rows (tc_attn_rows.cu).
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {

// rank-5 map over a [B, S, N, H, D] tensor given its (batch, row, residue, head) strides; a box is `rows` residues of
// `width` channels (32 or 64), zero beyond D
int qkv_tile_map(CUtensorMap* out, const void* p, const TriAttnDesc* d, const int64_t* st, int rows, int width);

// its offsets are 32-bit: rows of statistics, and O in units of 8 elements
bool attn_fwd_rows_fits(const TriAttnDesc* d);
// tbias: map over the bias with boxes of 128 queries x 64 keys, or null.  mask_terms: [B][S][npad] additive key-mask
// terms (0, -1e9, -inf beyond N).
int attn_fwd_rows(const TriAttnDesc* d, const void* q, const void* k, const void* v, const CUtensorMap* tbias,
                  bool bias_batched, void* o, float* stats, const float* mask_terms, int* err, cudaStream_t st);

}  // namespace tc
}  // namespace tri

// Triangle attention outside the tcgen05 path: fp32 operands, and every shape that the tcgen05 kernels do not take.
//
// Flash-style, with the additive pair bias and the key mask fused in, fp32 accumulation everywhere.  fp32 inputs at matmul
// precision "ieee" are multiplied exactly on the CUDA cores; with precision tf32 the operands of each product are rounded
// to TF32 and multiplied by the warp-level matrix instructions.
//
// Math follows triangle_attention_torch
// (geometric_nn_ops_torch/triangle/_reference/triangle_attention.py:28-44):
//   logits = (q*scale).k + bias + mask_bias,  mask_bias = 1e9*(mask-1)
// with the mask term added last, so a fully masked row degenerates to a uniform
// softmax exactly as the reference's does (_masking.py:13-42).
// The backward recomputes P from the saved statistics; dbias is summed over the rows in chunks, each in a fixed order (no
// atomics, deterministic).
#include <algorithm>
#include <mutex>

#include "attn_simt_kernels.cuh"

namespace tri {
namespace simt {

int forward_f32(const AttnArgs& a, cudaStream_t st);
int forward_tf32(const AttnArgs& a, cudaStream_t st);
int forward_bf16(const AttnArgs& a, cudaStream_t st);
int forward_f16(const AttnArgs& a, cudaStream_t st);
int backward_f32(const AttnArgs& a, float* part, cudaStream_t st);
int backward_tf32(const AttnArgs& a, float* part, cudaStream_t st);
int backward_bf16(const AttnArgs& a, float* part, cudaStream_t st);
int backward_f16(const AttnArgs& a, float* part, cudaStream_t st);

namespace {

// A tile of dbias is one CTA's, however many rows there are: with few tiles the rows are split into chunks until some
// 900 CTAs (two waves of three per SM) are there, at four rows or more per chunk.
int dbias_chunks(const TriAttnDesc* d) {
  const int tile_n = d->D <= 32 ? 64 : 32;
  const long long tiles = ceil_div(d->n_res, 64) * ceil_div(d->n_res, tile_n) * d->B * d->H;
  return (int)std::max(1LL, std::min(900 / tiles, (long long)d->n_seq / 4));
}
size_t delta_bytes(const TriAttnDesc* d) { return align_up((size_t)d->B * d->n_seq * d->H * d->n_res * sizeof(float)); }

// four elements of each row of these tensors at once: 16 (8) bytes, aligned
bool rows_of_four(const TriAttnDesc* d, const void* p, const int64_t* st) {
  const int e = d->dtype == TRI_F32 ? 4 : 2;
  return p == nullptr || ((reinterpret_cast<uintptr_t>(p) % (4 * e)) == 0 && d->D % 4 == 0 && st[0] % 4 == 0 && st[1] % 4 == 0 &&
                          st[2] % 4 == 0 && st[3] % 4 == 0);
}

AttnArgs make_args(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask) {
  AttnArgs a{};
  a.d = *d; a.q = q; a.k = k; a.v = v; a.bias = bias; a.mask = mask; a.chunks = 1; a.chunk_rows = d->n_seq;
  a.vec = rows_of_four(d, q, d->q_st) && rows_of_four(d, k, d->k_st) && rows_of_four(d, v, d->v_st);
  const int e = d->dtype == TRI_F32 ? 4 : 2;
  a.pair_bias = reinterpret_cast<uintptr_t>(bias) % (2 * e) == 0 && d->bias_st[0] % 2 == 0 && d->bias_st[1] % 2 == 0 && d->bias_st[2] % 2 == 0;
  return a;
}

int backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, const void* o,
             const float* lse, const void* d_o, void* dq, void* dk, void* dv, float* dbias, float* delta, float* part, int chunks,
             cudaStream_t st) {
  AttnArgs a = make_args(d, q, k, v, bias, mask);
  a.o = const_cast<void*>(o); a.lse = const_cast<float*>(lse); a.d_o = d_o; a.dq = dq; a.dk = dk; a.dv = dv; a.dbias = dbias; a.delta = delta;
  a.vec = a.vec && rows_of_four(d, d_o, d->do_st);
  a.vec_out = rows_of_four(d, o, d->o_st) && rows_of_four(d, dq, d->dq_st) && rows_of_four(d, dk, d->dk_st) && rows_of_four(d, dv, d->dv_st);
  a.chunk_rows = (d->n_seq + chunks - 1) / chunks;
  a.chunks = (d->n_seq + a.chunk_rows - 1) / a.chunk_rows;
  if (d->dtype == TRI_BF16) return backward_bf16(a, part, st);
  if (d->dtype == TRI_F16) return backward_f16(a, part, st);
  return d->precision == TRI_PREC_TF32 ? backward_tf32(a, part, st) : backward_f32(a, part, st);
}

}  // namespace

size_t attn_ws_bytes(const TriAttnDesc* d, int is_bwd) {
  if (!is_bwd) return 256;
  const int chunks = dbias_chunks(d);
  return delta_bytes(d) + 256 + (chunks > 1 ? align_up((size_t)chunks * d->B * d->H * d->n_res * d->n_res * sizeof(float)) : 0);
}

int attn_forward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
                 const uint8_t* mask, void* o, float* lse, cudaStream_t st) {
  AttnArgs a = make_args(d, q, k, v, bias, mask);
  a.o = o; a.lse = lse;
  a.vec_out = rows_of_four(d, o, d->o_st);
  if (d->dtype == TRI_BF16) return forward_bf16(a, st);
  if (d->dtype == TRI_F16) return forward_f16(a, st);
  return d->precision == TRI_PREC_TF32 ? forward_tf32(a, st) : forward_f32(a, st);
}

int attn_backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
                  const uint8_t* mask, const void* o, const float* lse, const void* d_o, void* dq, void* dk,
                  void* dv, float* dbias, void* ws, size_t ws_size, cudaStream_t st) {
  if (ws_size < attn_ws_bytes(d, 1)) return fail(TRI_ERR_WORKSPACE, "attention backward workspace too small");
  float* delta = (float*)ws;
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + delta_bytes(d) + 256);
  return backward(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, delta, part, dbias_chunks(d), st);
}

// ---------------------------------------------------------------------------------------------
// Backward without any caller- or library-allocated scratch.
//
// Some callers cannot hand this library a workspace: code running where device allocation is
// forbidden or impossible (a real-time serving loop with a frozen memory pool, a plugin host that
// gives operators no allocator, a process already at its memory limit).  For them the one scratch
// buffer the backward needs, delta[b,s,h,i] = sum_d dO*O, lives in this file-scope device array.
// Every GPU that loads the library carries these 4 MiB until the process exits.
//
// The array's name is only a host-side handle.  Its device address is looked up once per device, with
// that device current, through cudaGetSymbolAddress, and that address is what the kernels get.
// ---------------------------------------------------------------------------------------------
constexpr size_t kStaticDeltaFloats = size_t(1) << 20;  // B * n_seq * H * n_res may not exceed this
static __device__ __align__(256) float g_static_delta[kStaticDeltaFloats];

size_t attn_static_scratch_rows() { return kStaticDeltaFloats; }

int attn_backward_static(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
                         const uint8_t* mask, const void* o, const float* lse, const void* d_o, void* dq, void* dk,
                         void* dv, float* dbias, cudaStream_t st) {
  const size_t rows = (size_t)d->B * d->n_seq * d->H * d->n_res;
  if (rows > kStaticDeltaFloats)
    return fail(TRI_ERR_UNSUPPORTED,
                "B*n_seq*H*n_res = %zu exceeds the built-in scratch of %zu rows; use tri_attn_bwd with a workspace",
                rows, kStaticDeltaFloats);
  constexpr int kMaxDevices = 64;
  static float* device_ptr[kMaxDevices] = {};
  static std::mutex mu;
  int dev = 0;
  TRI_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(TRI_ERR_UNSUPPORTED, "device index %d out of range", dev);
  float* delta = nullptr;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (device_ptr[dev] == nullptr) {
      void* p = nullptr;
      TRI_CUDA_OK(cudaGetSymbolAddress(&p, g_static_delta));  // first call on this device: set-up
      device_ptr[dev] = static_cast<float*>(p);
    }
    delta = device_ptr[dev];
  }
  // delta is written in full by the first kernel before anything reads it: nothing to clear.
  return backward(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, delta, nullptr, 1, st);
}

}  // namespace simt
}  // namespace tri

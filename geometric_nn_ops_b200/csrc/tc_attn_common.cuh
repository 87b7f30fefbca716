// Small device helpers shared by the tensor-core attention kernels.
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kMaskSentinel = 1e9f;

// byte offset of 16-byte chunk `g` (0..15, 8 elements each) of row r inside a [128 x 128] two-block SW128 tile
__device__ __forceinline__ int sw128_chunk(int r, int g) {
  return (g >> 3) * 16384 + r * 128 + (((g & 7) ^ (r & 7)) << 4);
}

// the additive term of a key: 0 where it is kept, -1e9 where it is masked, -inf beyond the row
__device__ __forceinline__ float mask_term(uint32_t kept, bool in) { return !in ? -INFINITY : kept != 0 ? 0.0f : -kMaskSentinel; }

template <typename T> struct ElemIsBf16 { static constexpr bool value = false; };
template <> struct ElemIsBf16<__nv_bfloat16> { static constexpr bool value = true; };

// tcgen05.wait::ld that the registers of two loads pass through, so that no use of them can move above it
__device__ __forceinline__ void ld_wait8x2(uint32_t (&v)[8], uint32_t (&w)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(w[0]),
                 "+r"(w[1]), "+r"(w[2]), "+r"(w[3]), "+r"(w[4]), "+r"(w[5]), "+r"(w[6]), "+r"(w[7])::"memory");
}

// three-input maximum (one instruction on sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float2 pair(uint32_t lo, uint32_t hi) { return make_float2(__uint_as_float(lo), __uint_as_float(hi)); }
__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }

// a pair plus the 16-bit pair of a word, as two additions that widen their operand on the way
template <typename T> __device__ __forceinline__ float2 add_wide(float2 x, uint32_t w) {
  if constexpr (ElemIsBf16<T>::value)
    asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; add.rn.f32.bf16 %0, lo, %0; add.rn.f32.bf16 %1, hi, %1; }" : "+f"(x.x), "+f"(x.y) : "r"(w));
  else
    asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; add.rn.f32.f16 %0, lo, %0; add.rn.f32.f16 %1, hi, %1; }" : "+f"(x.x), "+f"(x.y) : "r"(w));
  return x;
}

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  union { uint4 u; T h[8]; } pk;
  pk.u = v;
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = to_f32(pk.h[i]);
}

// byte offset of 16-byte chunk g (0..7) of row r inside a one-block SW128 tile (rows of 64 16-bit elements)
__device__ __forceinline__ int sw128_chunk1(int r, int g) { return r * 128 + ((g ^ (r & 7)) << 4); }

}  // namespace
}  // namespace tc
}  // namespace tri

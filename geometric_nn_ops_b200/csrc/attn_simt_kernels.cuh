// Kernels of the fp32-operand triangle attention, forward and backward: exact fp32 on the CUDA cores, or TF32 products
// on the warp-level matrix instructions where the caller allows them.  Included by one .cu file per operand type.
//
// All kernels have one form.  A CTA of four warps owns a tile of 64 * MB "m" rows (queries, or keys in the dK / dV
// kernel), 16 * MB per warp, and walks over "n" tiles of 8 * NB rows, double-buffered by cp.async.  A product over the head
// dim (`rows_product`, both operands read as rows) leaves a [16 MB x 8 NB] tile of logits or of dP in registers, and a
// product over the n rows (`cols_product`) takes such a tile as its left operand.  Both come in two versions that share the
// register layout of mma.m16n8k8's accumulator -- thread (r = lane / 4, c = lane % 4) holds rows r, r + 8 and columns
// 2c, 2c + 1 of each 16 x 8 block -- so that the softmax between them is written once:
//   TF32   mma.sync on operands rounded to TF32 in shared memory.  The order of the contraction is free, so the slots are
//          given out such that a fragment is one 16-byte load per row and the accumulators of the first product are the
//          left operand of the second without a shuffle.
//   exact  4 MB x 2 NB-column register tiles of FMAs: 2 MB + 2 NB 16-byte loads feed 16 MB NB of them.
//
// What bounded the kernels that these replace (scalar shared loads, 4 x 4 outputs per thread, dbias on N^2 / 4096 * H CTAs
// whatever the number of rows) was the shared-memory pipe, and for dbias an idle chip.  What bounds these is instruction
// issue: about half of the slots at 12 warps per SM (168 registers per thread; the 32-wide tiles are compiled for three CTAs),
// of which the matrix instructions are a small part; in the exact kernels the FMAs are.  At 256 x 256 x 4 heads x 32 with
// TF32 (exact): forward 0.66 -> 0.13 ms (0.65 -> 0.34), dK and dV 1.11 -> 0.22 (0.55), dQ 0.85 -> 0.17 (0.40), dbias
// 5.6 -> 0.23 (0.40), delta 0.072 -> 0.025.
#pragma once

#include "attn_simt.cuh"
#include "common.cuh"

namespace tri {
namespace simt {

constexpr int kWarps = 4, kCta = 32 * kWarps;
constexpr float kLog2E = 1.4426950408889634f;

// The reference's torch path accumulates in fp32 for every 16/32-bit dtype and takes the sentinel of
// that accumulate dtype (triangle_attention.py:28,40 of its _reference package): 1e9.
constexpr float kSentinel = 1e9f;

struct AttnArgs {
  TriAttnDesc d;
  const void *q, *k, *v, *bias;
  const uint8_t* mask;
  void* o;
  float* lse;                 // [2][B, S, H, N]: maximum and log of the sum
  const void* d_o;
  void *dq, *dk, *dv;
  float *dbias, *delta;       // dbias: [chunks][B, H, N, N]
  int chunks, chunk_rows;     // dbias: row chunks
  int vec;                    // four elements of q, k, v, dO rows can be read at once
  int vec_out;                // ... of the outputs written at once
  int pair_bias;              // bias rows start on pairs
};

namespace {

__device__ __forceinline__ long long off4(const int64_t* st, int b, int s, int i, int h) {
  return b * st[0] + s * st[1] + i * st[2] + h * st[3];
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float4 ld_shared4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void st_shared4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// e^x.  With TF32 products the argument has ten bits anyway and the result is rounded to ten: base-2 hardware exponential.
template <bool TF32>
__device__ __forceinline__ float exp_of(float x) {
  if constexpr (TF32) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * kLog2E));
    return y;
  } else {
    return expf(x);
  }
}

// Tiles hold rows of DB floats in 16-byte chunks, the chunk index XORed with swz(row).  For rows 0..7 this is a bijection
// (a column of chunks is free of bank conflicts), it differs in bit 2 between rows 2i and 2i + 1 (the fragments of a
// product over the head dim read 4 consecutive chunks of two neighbouring rows), and in bits 1-2 among rows of one parity
// (those of a product over the rows read two chunks of four such rows).
__device__ __forceinline__ uint32_t swz(int row) { return (uint32_t)((row & 6) ^ ((row & 1) * 5)); }
template <int DB>
__device__ __forceinline__ uint32_t chunk_at(uint32_t tile, int row, int chunk) {
  return tile + row * (DB * 4) + (((uint32_t)chunk ^ swz(row)) << 4);
}

template <typename T>
__device__ __forceinline__ float4 load4(const T* p, int valid, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (sizeof(T) == 2) {
    if (vec) {
      union { uint2 u; T h[4]; } pk;
      pk.u = *reinterpret_cast<const uint2*>(p);
      return make_float4(to_f32(pk.h[0]), to_f32(pk.h[1]), to_f32(pk.h[2]), to_f32(pk.h[3]));
    }
  } else {
    if (vec) return *reinterpret_cast<const float4*>(p);
  }
  v.x = to_f32(p[0]);
  if (valid > 1) v.y = to_f32(p[1]);
  if (valid > 2) v.z = to_f32(p[2]);
  if (valid > 3) v.w = to_f32(p[3]);
  return v;
}

// Rows row0 .. row0 + ROWS - 1 of one (b, s, h) slice, zero beyond n rows and D columns.  fp32 goes by cp.async and is scaled
// and rounded in place by the same threads once it is there (`settle`); 16-bit operands are converted on the way.
template <typename T, int DB, int ROWS>
__device__ __forceinline__ void fetch(uint32_t tile, const T* base, long long stride, int row0, int n, int D, bool vec, float mul) {
  for (int i = threadIdx.x; i < ROWS * (DB / 4); i += kCta) {
    const int row = i / (DB / 4), ch = i % (DB / 4), valid = row0 + row < n ? D - ch * 4 : 0;
    const T* src = base + (valid > 0 ? (row0 + row) * stride + ch * 4 : 0);
    const uint32_t dst = chunk_at<DB>(tile, row, ch);
    if constexpr (sizeof(T) == 4) {
      if (vec) {
        cp_async16(dst, src, valid > 0 ? 16 : 0);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) cp_async4(dst + 4 * e, e < valid ? src + e : base, e < valid ? 4 : 0);
      }
    } else {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (valid > 0) v = load4(src, valid, vec);
      st_shared4(dst, make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul));
    }
  }
}
template <typename T, int DB, int ROWS, bool TF32, bool SCALED>
__device__ __forceinline__ void settle(uint32_t tile, float mul) {
  if constexpr (sizeof(T) == 4 && (TF32 || SCALED)) {
    for (int i = threadIdx.x; i < ROWS * (DB / 4); i += kCta) {
      const uint32_t a = chunk_at<DB>(tile, i / (DB / 4), i % (DB / 4));
      float4 v = ld_shared4(a);
      if constexpr (SCALED) v = make_float4(v.x * mul, v.y * mul, v.z * mul, v.w * mul);
      if constexpr (TF32) v = make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
      st_shared4(a, v);
    }
  }
}

__device__ __forceinline__ void mma_tf32(float (&c)[4], float a0, float a1, float a2, float a3, float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)),
                 "r"(__float_as_uint(b0)), "r"(__float_as_uint(b1)));
}

// acc[m][n] += sum_d A[m][d] B[n][d]; A: this warp's 16 MB rows of its tile
template <int DB, int MB, int NB, bool TF32>
__device__ __forceinline__ void rows_product(float (&acc)[MB][NB][4], uint32_t A, uint32_t B) {
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3, m0 = (threadIdx.x >> 5) * 16 * MB;
  if constexpr (TF32) {
#pragma unroll
    for (int t = 0; t < DB / 16; ++t) {
      float4 lo[MB], hi[MB];
#pragma unroll
      for (int mb = 0; mb < MB; ++mb) {
        lo[mb] = ld_shared4(chunk_at<DB>(A, m0 + mb * 16 + r, t * 4 + c));
        hi[mb] = ld_shared4(chunk_at<DB>(A, m0 + mb * 16 + r + 8, t * 4 + c));
      }
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const float4 b = ld_shared4(chunk_at<DB>(B, nb * 8 + r, t * 4 + c));
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) mma_tf32(acc[mb][nb], lo[mb].x, hi[mb].x, lo[mb].y, hi[mb].y, b.x, b.y);
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) mma_tf32(acc[mb][nb], lo[mb].z, hi[mb].z, lo[mb].w, hi[mb].w, b.z, b.w);
      }
    }
  } else {
#pragma unroll 1
    for (int ch = 0; ch < DB / 4; ++ch) {
      float4 a[2 * MB];
#pragma unroll
      for (int i = 0; i < 2 * MB; ++i) a[i] = ld_shared4(chunk_at<DB>(A, m0 + i * 8 + r, ch));
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float4 b = ld_shared4(chunk_at<DB>(B, nb * 8 + 2 * c + e, ch));
#pragma unroll
          for (int i = 0; i < 2 * MB; ++i) {
            float& x = acc[i >> 1][nb][(i & 1) * 2 + e];
            x = fmaf(a[i].x, b.x, x); x = fmaf(a[i].y, b.y, x); x = fmaf(a[i].z, b.z, x); x = fmaf(a[i].w, b.w, x);
          }
        }
    }
  }
}

// acc[m][d] += sum_n P[m][n] B[n][d].  Element (g, e, x) of a row's accumulators is column 32 g + 8 c + 4 e + x.
// `stage`: this warp's 16 MB x 8 NB floats of shared memory (exact products only).
template <int DB, int MB, int NB, bool TF32>
__device__ __forceinline__ void cols_product(float (&acc)[MB][DB / 32][4][4], const float (&p)[MB][NB][4], uint32_t B, uint32_t stage) {
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  if constexpr (TF32) {
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      float a[MB][4];
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i) a[mb][i] = round_tf32(p[mb][nb][i]);
#pragma unroll
      for (int g = 0; g < DB / 32; ++g) {
        const float4 b0 = ld_shared4(chunk_at<DB>(B, nb * 8 + 2 * c, g * 8 + r)), b1 = ld_shared4(chunk_at<DB>(B, nb * 8 + 2 * c + 1, g * 8 + r));
#pragma unroll
        for (int mb = 0; mb < MB; ++mb) {
          mma_tf32(acc[mb][g][0], a[mb][0], a[mb][2], a[mb][1], a[mb][3], b0.x, b1.x);
          mma_tf32(acc[mb][g][1], a[mb][0], a[mb][2], a[mb][1], a[mb][3], b0.y, b1.y);
          mma_tf32(acc[mb][g][2], a[mb][0], a[mb][2], a[mb][1], a[mb][3], b0.z, b1.z);
          mma_tf32(acc[mb][g][3], a[mb][0], a[mb][2], a[mb][1], a[mb][3], b0.w, b1.w);
        }
      }
    }
  } else {
    constexpr int W = NB * 32;   // bytes of a staged row; its 16-byte chunks are XORed with the row
    __syncwarp();
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int hi = 0; hi < 2; ++hi)
          asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(stage + (mb * 16 + hi * 8 + r) * W + (((nb * 2 + (c >> 1)) ^ r) << 4) + (c & 1) * 8),
                       "f"(p[mb][nb][hi * 2]), "f"(p[mb][nb][hi * 2 + 1]) : "memory");
    __syncwarp();
#pragma unroll 1
    for (int ch = 0; ch < NB * 2; ++ch) {
      float a[2 * MB][4];
#pragma unroll
      for (int i = 0; i < 2 * MB; ++i) {
        const float4 v = ld_shared4(stage + (i * 8 + r) * W + ((ch ^ r) << 4));
        a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int g = 0; g < DB / 32; ++g)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float4 b = ld_shared4(chunk_at<DB>(B, ch * 4 + j, g * 8 + 2 * c + e));
#pragma unroll
            for (int i = 0; i < 2 * MB; ++i) {
              const int q = (i & 1) * 2 + e;
              acc[i >> 1][g][0][q] = fmaf(a[i][j], b.x, acc[i >> 1][g][0][q]);
              acc[i >> 1][g][1][q] = fmaf(a[i][j], b.y, acc[i >> 1][g][1][q]);
              acc[i >> 1][g][2][q] = fmaf(a[i][j], b.z, acc[i >> 1][g][2][q]);
              acc[i >> 1][g][3][q] = fmaf(a[i][j], b.w, acc[i >> 1][g][3][q]);
            }
          }
    }
  }
}

// s = bias (ADD: s += bias) of this warp's rows (queries) and NB * 8 keys from k0, zero where there is none.  A tile inside the
// plane whose rows start on pairs is read without a test per element (rows beyond the last query repeat it: nothing of them is
// kept).  TF32 products start from the bias.  Exact ones start from zero and take it afterwards, in one rounding, as the
// reference does: a sum that starts from it rounds every term beside it (errors four to eight times larger from a bias of 10 on).
template <typename T, int MB, int NB, bool ADD>
__device__ __forceinline__ void bias_tile(float (&s)[MB][NB][4], const T* bias, long long row_st, int q0, int k0, int n, bool pairs) {
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const bool fast = bias != nullptr && pairs && k0 + NB * 8 <= n;
  auto put = [](float& x, float v) { x = ADD ? x + v : v; };
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const T* row = bias + (bias != nullptr ? min(q0 + mb * 16 + hi * 8 + r, n - 1) * row_st + k0 + 2 * c : 0);
      if (fast) {
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          if constexpr (sizeof(T) == 4) {
            const float2 v = __ldg(reinterpret_cast<const float2*>(row + nb * 8));
            put(s[mb][nb][hi * 2], v.x);
            put(s[mb][nb][hi * 2 + 1], v.y);
          } else {
            union { uint32_t u; T h[2]; } v;
            v.u = __ldg(reinterpret_cast<const uint32_t*>(row + nb * 8));
            put(s[mb][nb][hi * 2], to_f32(v.h[0]));
            put(s[mb][nb][hi * 2 + 1], to_f32(v.h[1]));
          }
        }
      } else {
        const int left = bias != nullptr ? n - k0 - 2 * c : 0;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          put(s[mb][nb][hi * 2], nb * 8 < left ? to_f32(row[nb * 8]) : 0.f);
          put(s[mb][nb][hi * 2 + 1], nb * 8 + 1 < left ? to_f32(row[nb * 8 + 1]) : 0.f);
        }
      }
    }
}
// ... with the keys as this warp's rows and NB * 8 queries from q0
template <typename T, int MB, int NB, bool ADD>
__device__ __forceinline__ void bias_tile_t(float (&s)[MB][NB][4], const T* bias, long long row_st, int key0, int q0, int n) {
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const T* col = bias + (bias != nullptr ? (q0 + 2 * c) * row_st + key0 + r : 0);
  const bool fast = bias != nullptr && key0 + 16 * MB <= n && q0 + NB * 8 <= n;
#pragma unroll
  for (int nb = 0; nb < NB; ++nb, col += 8 * row_st)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const T* at = col + e * row_st;
#pragma unroll
      for (int i = 0; i < 2 * MB; ++i) {
        const bool live = fast || (bias != nullptr && key0 + r + i * 8 < n && q0 + nb * 8 + 2 * c + e < n);
        const float v = live ? to_f32(__ldg(at + i * 8)) : 0.f;
        float& x = s[i >> 1][nb][(i & 1) * 2 + e];
        x = ADD ? x + v : v;
      }
    }
}

// out[row][d] = acc * mul for this thread's rows and columns
template <typename T, int DB, int MB>
__device__ __forceinline__ void store_rows(T* out, long long stride, int row0, int n, int D, bool vec, const float (&acc)[MB][DB / 32][4][4],
                                           const float (&mul)[MB][2]) {
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int row = row0 + mb * 16 + hi * 8 + r;
      if (row >= n) continue;
      T* dst = out + row * stride;
#pragma unroll
      for (int g = 0; g < DB / 32; ++g)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int dd = g * 32 + 8 * c + 4 * e;
          float v[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) v[x] = acc[mb][g][x][hi * 2 + e] * mul[mb][hi];
          if (vec && dd < D) {
            if constexpr (sizeof(T) == 4) {
              *reinterpret_cast<float4*>(dst + dd) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
              union { uint2 u; T h[4]; } pk;
#pragma unroll
              for (int x = 0; x < 4; ++x) pk.h[x] = from_f32<T>(v[x]);
              *reinterpret_cast<uint2*>(dst + dd) = pk.u;
            }
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x)
              if (dd + x < D) dst[dd + x] = from_f32<T>(v[x]);
          }
        }
    }
}

// which (b, s, h) slice and m tile a CTA has: tiles run fastest, so that neighbours share the slice's n rows in L2
struct Slice { int b, s, h, m0; };
__device__ __forceinline__ Slice slice_of(const TriAttnDesc& d, int m_tile) {
  const int tiles = (d.n_res + m_tile - 1) / m_tile;
  Slice x;
  int z = blockIdx.x / tiles;
  x.m0 = (blockIdx.x - z * tiles) * m_tile;
  x.h = z % d.H; z /= d.H;
  x.s = z % d.n_seq; x.b = z / d.n_seq;
  return x;
}

// The mask term of key kj: 1e9 * (float(mask) - 1), +0.0 when kept; -inf beyond the last key.
__device__ __forceinline__ float mask_term(const uint8_t* mask_row, int kj, int n) {
  return kj >= n ? -INFINITY : (mask_row == nullptr || mask_row[kj] ? 0.f : -kSentinel);
}

template <int DB, int MB, int NB, bool TF32>
constexpr int fwd_smem() {
  return (64 * MB * DB + 4 * 8 * NB * DB + 2 * 8 * NB + (TF32 ? 0 : kWarps * 16 * MB * 8 * NB)) * 4;
}
template <typename T, int DB, int MB, int NB, bool TF32>
__global__ void __launch_bounds__(kCta, DB == 32 ? 3 : 1) attn_fwd_kernel(const AttnArgs a) {
  extern __shared__ __align__(128) float sm[];
  constexpr int NT = 8 * NB;
  const TriAttnDesc& d = a.d;
  const Slice z = slice_of(d, 64 * MB);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane & 3, n = d.n_res, D = d.D;
  const uint32_t sQ = smem_addr(sm), sK = sQ + 64 * MB * DB * 4, sV = sK + 2 * NT * DB * 4, stage0 = sV + 2 * NT * DB * 4;
  float* sM = sm + 64 * MB * DB + 4 * NT * DB;                   // [2][NT] mask terms
  const uint32_t stage = stage0 + 2 * NT * 4 + warp * (16 * MB * NT * 4);
  const T* q = static_cast<const T*>(a.q) + off4(d.q_st, z.b, z.s, 0, z.h);
  const T* k = static_cast<const T*>(a.k) + off4(d.k_st, z.b, z.s, 0, z.h);
  const T* v = static_cast<const T*>(a.v) + off4(d.v_st, z.b, z.s, 0, z.h);
  const T* bias = a.bias == nullptr ? nullptr : static_cast<const T*>(a.bias) + z.b * d.bias_st[0] + z.h * d.bias_st[1];
  const uint8_t* mask = a.mask == nullptr ? nullptr : a.mask + z.b * d.mask_st[0] + z.s * d.mask_st[1];
  const bool vec = a.vec != 0;
  auto issue = [&](int k0, int b) {
    fetch<T, DB, NT>(sK + b * NT * DB * 4, k, d.k_st[2], k0, n, D, vec, 1.f);
    fetch<T, DB, NT>(sV + b * NT * DB * 4, v, d.v_st[2], k0, n, D, vec, 1.f);
    cp_commit();
    if (threadIdx.x < NT) sM[b * NT + threadIdx.x] = mask_term(mask, k0 + threadIdx.x, n);
  };
  fetch<T, DB, 64 * MB>(sQ, q, d.q_st[2], z.m0, n, D, vec, d.scale);
  issue(0, 0);
  float acc[MB][DB / 32][4][4] = {}, m[MB][2], l[MB][2];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb) { m[mb][0] = m[mb][1] = -INFINITY; l[mb][0] = l[mb][1] = 0.f; }
  for (int k0 = 0, b = 0; k0 < n; k0 += NT, b ^= 1) {
    const uint32_t tK = sK + b * NT * DB * 4, tV = sV + b * NT * DB * 4;
    cp_wait();
    if (k0 == 0) settle<T, DB, 64 * MB, TF32, true>(sQ, d.scale);
    settle<T, DB, NT, TF32, false>(tK, 1.f);
    settle<T, DB, NT, TF32, false>(tV, 1.f);
    __syncthreads();
    if (k0 + NT < n) issue(k0 + NT, b ^ 1);
    float s[MB][NB][4] = {};
    if constexpr (TF32) bias_tile<T, MB, NB, false>(s, bias, d.bias_st[2], z.m0 + warp * 16 * MB, k0, n, a.pair_bias != 0);
    rows_product<DB, MB, NB, TF32>(s, sQ, tK);
    if constexpr (!TF32) bias_tile<T, MB, NB, true>(s, bias, d.bias_st[2], z.m0 + warp * 16 * MB, k0, n, a.pair_bias != 0);
    float mn[MB][2];
#pragma unroll
    for (int mb = 0; mb < MB; ++mb) mn[mb][0] = m[mb][0], mn[mb][1] = m[mb][1];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const float2 t = *reinterpret_cast<const float2*>(sM + b * NT + nb * 8 + 2 * c);
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          s[mb][nb][i] += i & 1 ? t.y : t.x;
          mn[mb][i >> 1] = fmaxf(mn[mb][i >> 1], s[mb][nb][i]);
        }
    }
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int hi = 0; hi < 2; ++hi) {
        float x = mn[mb][hi];
        x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
        x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
        x = fmaxf(x, -3.402823466e38f);   // no key with a finite logit yet: P = exp(-inf), not exp(-inf + inf)
        const float alpha = exp_of<TF32>(m[mb][hi] - x);
        m[mb][hi] = x;
        float sum = 0.f;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float& y = s[mb][nb][hi * 2 + e];
            y = exp_of<TF32>(y - x);
            sum += y;
          }
        l[mb][hi] = l[mb][hi] * alpha + sum;
#pragma unroll
        for (int g = 0; g < DB / 32; ++g)
#pragma unroll
          for (int x4 = 0; x4 < 4; ++x4) { acc[mb][g][x4][hi * 2] *= alpha; acc[mb][g][x4][hi * 2 + 1] *= alpha; }
      }
    cols_product<DB, MB, NB, TF32>(acc, s, tV, stage);
  }
  const int row0 = z.m0 + warp * 16 * MB;
  float inv[MB][2];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      float x = l[mb][hi];
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      inv[mb][hi] = 1.0f / x;
      const int qi = row0 + mb * 16 + hi * 8 + (lane >> 2);
      if (c == 0 && qi < n) {
        const long long row = (((long long)z.b * d.n_seq + z.s) * d.H + z.h) * n + qi;
        a.lse[row] = m[mb][hi];
        a.lse[(long long)d.B * d.n_seq * d.H * n + row] = logf(x);
      }
    }
  store_rows<T, DB, MB>(static_cast<T*>(a.o) + off4(d.o_st, z.b, z.s, 0, z.h), d.o_st[2], row0, n, D, a.vec_out != 0, acc, inv);
}

// ---------------------------------------------------------------------------------------------------- backward

// delta[b,s,h,i] = sum_d dO * O: eight lanes per row
template <typename T>
__global__ void __launch_bounds__(256) attn_delta_kernel(const AttnArgs a) {
  const TriAttnDesc& d = a.d;
  const long long row = (blockIdx.x * 256LL + threadIdx.x) >> 3;
  const bool live = row < (long long)d.B * d.n_seq * d.H * d.n_res;
  float acc = 0.f;
  if (live) {
    const int i = row % d.n_res;
    long long z = row / d.n_res;
    const int h = z % d.H; z /= d.H;
    const int s = z % d.n_seq, b = z / d.n_seq;
    const T* o = static_cast<const T*>(a.o) + off4(d.o_st, b, s, i, h);
    const T* g = static_cast<const T*>(a.d_o) + off4(d.do_st, b, s, i, h);
    const bool vec = a.vec != 0 && a.vec_out != 0;
    for (int dd = (threadIdx.x & 7) * 4; dd < d.D; dd += 32) {
      const float4 x = load4(o + dd, d.D - dd, vec), y = load4(g + dd, d.D - dd, vec);
      acc = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, acc))));
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (live && (threadIdx.x & 7) == 0) a.delta[row] = acc;
}

// P = exp((S - m) - log l) and dS = P (dP - delta); the two statistics stay separate because m + log l would round log l
// away when m is the -1e9 of a fully masked row.
template <bool TF32>
__device__ __forceinline__ float p_of(float s, float m, float ll) { return exp_of<TF32>((s - m) - ll); }

template <int DB, int MB, int NB, bool TF32>
constexpr int dkdv_smem() {
  return (2 * 64 * MB * DB + 4 * 8 * NB * DB + 2 * 3 * 8 * NB + (TF32 ? 0 : kWarps * 16 * MB * 8 * NB)) * 4;
}
// m rows: keys; n rows: queries (the tile of logits is transposed)
template <typename T, int DB, int MB, int NB, bool TF32>
__global__ void __launch_bounds__(kCta, DB == 32 ? 3 : 1) attn_bwd_dkdv_kernel(const AttnArgs a) {
  extern __shared__ __align__(128) float sm[];
  constexpr int NT = 8 * NB;
  const TriAttnDesc& d = a.d;
  const Slice z = slice_of(d, 64 * MB);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3, n = d.n_res, D = d.D;
  const uint32_t sK = smem_addr(sm), sV = sK + 64 * MB * DB * 4, sQ = sV + 64 * MB * DB * 4, sG = sQ + 2 * NT * DB * 4;
  float* sS = sm + 2 * 64 * MB * DB + 4 * NT * DB;               // [2][3][NT]: m, log l, delta of the queries
  const uint32_t stat0 = sG + 2 * NT * DB * 4, stage = stat0 + 6 * NT * 4 + warp * (16 * MB * NT * 4);
  const T* q = static_cast<const T*>(a.q) + off4(d.q_st, z.b, z.s, 0, z.h);
  const T* g = static_cast<const T*>(a.d_o) + off4(d.do_st, z.b, z.s, 0, z.h);
  const T* bias = a.bias == nullptr ? nullptr : static_cast<const T*>(a.bias) + z.b * d.bias_st[0] + z.h * d.bias_st[1];
  const uint8_t* mask = a.mask == nullptr ? nullptr : a.mask + z.b * d.mask_st[0] + z.s * d.mask_st[1];
  const long long row0 = (((long long)z.b * d.n_seq + z.s) * d.H + z.h) * n, rows = (long long)d.B * d.n_seq * d.H * n;
  const bool vec = a.vec != 0;
  auto issue = [&](int q0, int b) {
    fetch<T, DB, NT>(sQ + b * NT * DB * 4, q, d.q_st[2], q0, n, D, vec, d.scale);
    fetch<T, DB, NT>(sG + b * NT * DB * 4, g, d.do_st[2], q0, n, D, vec, 1.f);
    for (int i = threadIdx.x; i < 3 * NT; i += kCta) {
      const int which = i / NT, qi = q0 + i % NT;
      const float* src = which == 2 ? a.delta : a.lse + which * rows;
      cp_async4(stat0 + (b * 3 * NT + i) * 4, src + row0 + (qi < n ? qi : 0), qi < n ? 4 : 0);
    }
    cp_commit();
  };
  fetch<T, DB, 64 * MB>(sK, static_cast<const T*>(a.k) + off4(d.k_st, z.b, z.s, 0, z.h), d.k_st[2], z.m0, n, D, vec, 1.f);
  fetch<T, DB, 64 * MB>(sV, static_cast<const T*>(a.v) + off4(d.v_st, z.b, z.s, 0, z.h), d.v_st[2], z.m0, n, D, vec, 1.f);
  issue(0, 0);
  const int key0 = z.m0 + warp * 16 * MB;
  float term[MB][2];                                               // mask terms of this thread's keys
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) term[mb][hi] = mask_term(mask, key0 + mb * 16 + hi * 8 + r, n);
  float acc_k[MB][DB / 32][4][4] = {}, acc_v[MB][DB / 32][4][4] = {};
  for (int q0 = 0, b = 0; q0 < n; q0 += NT, b ^= 1) {
    const uint32_t tQ = sQ + b * NT * DB * 4, tG = sG + b * NT * DB * 4;
    cp_wait();
    if (q0 == 0) { settle<T, DB, 64 * MB, TF32, false>(sK, 1.f); settle<T, DB, 64 * MB, TF32, false>(sV, 1.f); }
    settle<T, DB, NT, TF32, true>(tQ, d.scale);
    settle<T, DB, NT, TF32, false>(tG, 1.f);
    __syncthreads();
    if (q0 + NT < n) issue(q0 + NT, b ^ 1);
    const float* st = sS + b * 3 * NT + 2 * c;
    float s[MB][NB][4] = {}, dp[MB][NB][4] = {};
    if constexpr (TF32) bias_tile_t<T, MB, NB, false>(s, bias, d.bias_st[2], key0, q0, n);
    rows_product<DB, MB, NB, TF32>(s, sK, tQ);
    if constexpr (!TF32) bias_tile_t<T, MB, NB, true>(s, bias, d.bias_st[2], key0, q0, n);
    auto minus_delta = [&] {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const float2 dl = *reinterpret_cast<const float2*>(st + 2 * NT + nb * 8);
#pragma unroll
        for (int mb = 0; mb < MB; ++mb)
#pragma unroll
          for (int i = 0; i < 4; ++i) dp[mb][nb][i] -= i & 1 ? dl.y : dl.x;
      }
    };
    if constexpr (TF32) minus_delta();
    rows_product<DB, MB, NB, TF32>(dp, sV, tG);
    if constexpr (!TF32) minus_delta();
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const float2 mx = *reinterpret_cast<const float2*>(st + nb * 8), ll = *reinterpret_cast<const float2*>(st + NT + nb * 8);
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float p = p_of<TF32>(s[mb][nb][i] + term[mb][i >> 1], i & 1 ? mx.y : mx.x, i & 1 ? ll.y : ll.x);
          s[mb][nb][i] = p;
          dp[mb][nb][i] *= p;
        }
    }
    cols_product<DB, MB, NB, TF32>(acc_v, s, tG, stage);    // dV[k] += sum_q P[q,k] dO[q]
    cols_product<DB, MB, NB, TF32>(acc_k, dp, tQ, stage);   // dK[k] += sum_q dS[q,k] (scale q)
  }
  float one[MB][2];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb) one[mb][0] = one[mb][1] = 1.f;
  store_rows<T, DB, MB>(static_cast<T*>(a.dk) + off4(d.dk_st, z.b, z.s, 0, z.h), d.dk_st[2], key0, n, D, a.vec_out != 0, acc_k, one);
  store_rows<T, DB, MB>(static_cast<T*>(a.dv) + off4(d.dv_st, z.b, z.s, 0, z.h), d.dv_st[2], key0, n, D, a.vec_out != 0, acc_v, one);
}

// this thread's rows' statistics: maximum, log of the sum, delta
template <int MB>
__device__ __forceinline__ void row_stats(const AttnArgs& a, long long row0, long long rows, int q0, int n, float (&mx)[MB][2], float (&ll)[MB][2],
                                          float (&dl)[MB][2]) {
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int qi = q0 + mb * 16 + hi * 8 + ((threadIdx.x & 31) >> 2);
      const long long at = row0 + (qi < n ? qi : 0);
      mx[mb][hi] = a.lse[at]; ll[mb][hi] = a.lse[rows + at]; dl[mb][hi] = a.delta[at];
    }
}

template <int DB, int MB, int NB, bool TF32>
constexpr int dq_smem() {
  return (2 * 64 * MB * DB + 4 * 8 * NB * DB + 2 * 8 * NB + (TF32 ? 0 : kWarps * 16 * MB * 8 * NB)) * 4;
}
template <typename T, int DB, int MB, int NB, bool TF32>
__global__ void __launch_bounds__(kCta, DB == 32 ? 3 : 1) attn_bwd_dq_kernel(const AttnArgs a) {
  extern __shared__ __align__(128) float sm[];
  constexpr int NT = 8 * NB;
  const TriAttnDesc& d = a.d;
  const Slice z = slice_of(d, 64 * MB);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = lane & 3, n = d.n_res, D = d.D;
  const uint32_t sQ = smem_addr(sm), sG = sQ + 64 * MB * DB * 4, sK = sG + 64 * MB * DB * 4, sV = sK + 2 * NT * DB * 4;
  float* sM = sm + 2 * 64 * MB * DB + 4 * NT * DB;
  const uint32_t stage = sV + 2 * NT * DB * 4 + 2 * NT * 4 + warp * (16 * MB * NT * 4);
  const T* k = static_cast<const T*>(a.k) + off4(d.k_st, z.b, z.s, 0, z.h);
  const T* v = static_cast<const T*>(a.v) + off4(d.v_st, z.b, z.s, 0, z.h);
  const T* bias = a.bias == nullptr ? nullptr : static_cast<const T*>(a.bias) + z.b * d.bias_st[0] + z.h * d.bias_st[1];
  const uint8_t* mask = a.mask == nullptr ? nullptr : a.mask + z.b * d.mask_st[0] + z.s * d.mask_st[1];
  const bool vec = a.vec != 0;
  auto issue = [&](int k0, int b) {
    fetch<T, DB, NT>(sK + b * NT * DB * 4, k, d.k_st[2], k0, n, D, vec, 1.f);
    fetch<T, DB, NT>(sV + b * NT * DB * 4, v, d.v_st[2], k0, n, D, vec, 1.f);
    cp_commit();
    if (threadIdx.x < NT) sM[b * NT + threadIdx.x] = mask_term(mask, k0 + threadIdx.x, n);
  };
  fetch<T, DB, 64 * MB>(sQ, static_cast<const T*>(a.q) + off4(d.q_st, z.b, z.s, 0, z.h), d.q_st[2], z.m0, n, D, vec, d.scale);
  fetch<T, DB, 64 * MB>(sG, static_cast<const T*>(a.d_o) + off4(d.do_st, z.b, z.s, 0, z.h), d.do_st[2], z.m0, n, D, vec, 1.f);
  issue(0, 0);
  const int q0 = z.m0 + warp * 16 * MB;
  float mx[MB][2], ll[MB][2], dl[MB][2];
  row_stats<MB>(a, (((long long)z.b * d.n_seq + z.s) * d.H + z.h) * n, (long long)d.B * d.n_seq * d.H * n, q0, n, mx, ll, dl);
  float acc[MB][DB / 32][4][4] = {};
  for (int k0 = 0, b = 0; k0 < n; k0 += NT, b ^= 1) {
    const uint32_t tK = sK + b * NT * DB * 4, tV = sV + b * NT * DB * 4;
    cp_wait();
    if (k0 == 0) { settle<T, DB, 64 * MB, TF32, true>(sQ, d.scale); settle<T, DB, 64 * MB, TF32, false>(sG, 1.f); }
    settle<T, DB, NT, TF32, false>(tK, 1.f);
    settle<T, DB, NT, TF32, false>(tV, 1.f);
    __syncthreads();
    if (k0 + NT < n) issue(k0 + NT, b ^ 1);
    float s[MB][NB][4] = {}, dp[MB][NB][4] = {};
    if constexpr (TF32) bias_tile<T, MB, NB, false>(s, bias, d.bias_st[2], q0, k0, n, a.pair_bias != 0);
    rows_product<DB, MB, NB, TF32>(s, sQ, tK);
    if constexpr (!TF32) bias_tile<T, MB, NB, true>(s, bias, d.bias_st[2], q0, k0, n, a.pair_bias != 0);
    auto minus_delta = [&] {
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int i = 0; i < 4; ++i) dp[mb][nb][i] -= dl[mb][i >> 1];
    };
    if constexpr (TF32) minus_delta();
    rows_product<DB, MB, NB, TF32>(dp, sG, tV);
    if constexpr (!TF32) minus_delta();
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const float2 t = *reinterpret_cast<const float2*>(sM + b * NT + nb * 8 + 2 * c);
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i) dp[mb][nb][i] *= p_of<TF32>(s[mb][nb][i] + (i & 1 ? t.y : t.x), mx[mb][i >> 1], ll[mb][i >> 1]);
    }
    cols_product<DB, MB, NB, TF32>(acc, dp, tK, stage);     // dQ[q] += sum_k dS[q,k] K[k]
  }
  float mul[MB][2];
#pragma unroll
  for (int mb = 0; mb < MB; ++mb) mul[mb][0] = mul[mb][1] = d.scale;
  store_rows<T, DB, MB>(static_cast<T*>(a.dq) + off4(d.dq_st, z.b, z.s, 0, z.h), d.dq_st[2], q0, n, D, a.vec_out != 0, acc, mul);
}

// dbias[b,h,i,j] = sum over the rows s of dS, in order.  A CTA has one tile of the plane and `chunk_rows` rows; the chunks'
// partial sums are added in order afterwards (dbias_reduce_kernel), so the result does not depend on the schedule.
template <int DB, int MB, int NB>
constexpr int dbias_smem() {
  return 2 * (2 * 64 * MB * DB + 2 * 8 * NB * DB + 8 * NB) * 4;
}
template <typename T, int DB, int MB, int NB, bool TF32>
__global__ void __launch_bounds__(kCta, DB == 32 ? 3 : 1) attn_bwd_dbias_kernel(const AttnArgs a) {
  extern __shared__ __align__(128) float sm[];
  constexpr int MT = 64 * MB, NT = 8 * NB, kStage = (2 * MT * DB + 2 * NT * DB) * 4;
  const TriAttnDesc& d = a.d;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3, n = d.n_res, D = d.D;
  const int tiles_m = (n + MT - 1) / MT, tiles_n = (n + NT - 1) / NT;
  // rows chunks run slowest: the CTAs that run together read the same rows
  int x = blockIdx.x;
  const int nt = x % tiles_n; x /= tiles_n;
  const int mt = x % tiles_m; x /= tiles_m;
  const int h = x % d.H; x /= d.H;
  const int b = x % d.B, chunk = x / d.B;
  const int m0 = mt * MT, k0 = nt * NT, q0 = m0 + warp * 16 * MB;
  const int s_begin = chunk * a.chunk_rows, s_end = min(s_begin + a.chunk_rows, d.n_seq);
  const uint32_t base = smem_addr(sm);
  float* sM = sm + 2 * kStage / 4;                                // [2][NT]
  const T* bias = a.bias == nullptr ? nullptr : static_cast<const T*>(a.bias) + b * d.bias_st[0] + h * d.bias_st[1];
  const bool vec = a.vec != 0;
  const long long rows = (long long)d.B * d.n_seq * d.H * n;
  auto issue = [&](int s, int buf) {
    const uint32_t t = base + buf * kStage;
    fetch<T, DB, MT>(t, static_cast<const T*>(a.q) + off4(d.q_st, b, s, 0, h), d.q_st[2], m0, n, D, vec, d.scale);
    fetch<T, DB, MT>(t + MT * DB * 4, static_cast<const T*>(a.d_o) + off4(d.do_st, b, s, 0, h), d.do_st[2], m0, n, D, vec, 1.f);
    fetch<T, DB, NT>(t + 2 * MT * DB * 4, static_cast<const T*>(a.k) + off4(d.k_st, b, s, 0, h), d.k_st[2], k0, n, D, vec, 1.f);
    fetch<T, DB, NT>(t + (2 * MT + NT) * DB * 4, static_cast<const T*>(a.v) + off4(d.v_st, b, s, 0, h), d.v_st[2], k0, n, D, vec, 1.f);
    cp_commit();
    if (threadIdx.x < NT)
      sM[buf * NT + threadIdx.x] = mask_term(a.mask == nullptr ? nullptr : a.mask + b * d.mask_st[0] + s * d.mask_st[1], k0 + threadIdx.x, n);
  };
  float acc[MB][NB][4] = {}, bt[MB][NB][4], mx[MB][2], ll[MB][2], dl[MB][2];
  bias_tile<T, MB, NB, false>(bt, bias, d.bias_st[2], q0, k0, n, a.pair_bias != 0);
  if (s_begin < s_end) issue(s_begin, 0);
  for (int s = s_begin, buf = 0; s < s_end; ++s, buf ^= 1) {
    const uint32_t tQ = base + buf * kStage, tG = tQ + MT * DB * 4, tK = tG + MT * DB * 4, tV = tK + NT * DB * 4;
    row_stats<MB>(a, (((long long)b * d.n_seq + s) * d.H + h) * n, rows, q0, n, mx, ll, dl);
    cp_wait();
    settle<T, DB, MT, TF32, true>(tQ, d.scale);
    settle<T, DB, MT, TF32, false>(tG, 1.f);
    settle<T, DB, NT, TF32, false>(tK, 1.f);
    settle<T, DB, NT, TF32, false>(tV, 1.f);
    __syncthreads();
    if (s + 1 < s_end) issue(s + 1, buf ^ 1);
    float p[MB][NB][4], dp[MB][NB][4];
#pragma unroll
    for (int mb = 0; mb < MB; ++mb)
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int i = 0; i < 4; ++i) { p[mb][nb][i] = TF32 ? bt[mb][nb][i] : 0.f; dp[mb][nb][i] = TF32 ? -dl[mb][i >> 1] : 0.f; }
    rows_product<DB, MB, NB, TF32>(p, tQ, tK);
    rows_product<DB, MB, NB, TF32>(dp, tG, tV);
    if constexpr (!TF32) {
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
          for (int i = 0; i < 4; ++i) { p[mb][nb][i] += bt[mb][nb][i]; dp[mb][nb][i] -= dl[mb][i >> 1]; }
    }
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      const float2 t = *reinterpret_cast<const float2*>(sM + buf * NT + nb * 8 + 2 * c);
#pragma unroll
      for (int mb = 0; mb < MB; ++mb)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          acc[mb][nb][i] = fmaf(p_of<TF32>(p[mb][nb][i] + (i & 1 ? t.y : t.x), mx[mb][i >> 1], ll[mb][i >> 1]), dp[mb][nb][i], acc[mb][nb][i]);
    }
  }
  float* out = a.dbias + (((long long)chunk * d.B + b) * d.H + h) * n * (long long)n;
  const bool pairs = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(a.dbias) & 7) == 0;
#pragma unroll
  for (int mb = 0; mb < MB; ++mb)
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
      const int qi = q0 + mb * 16 + hi * 8 + r;
      if (qi >= n) continue;
      float* row = out + (long long)qi * n + k0 + 2 * c;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int left = n - (k0 + nb * 8 + 2 * c);
        if (left >= 2 && pairs) {
          *reinterpret_cast<float2*>(row + nb * 8) = make_float2(acc[mb][nb][hi * 2], acc[mb][nb][hi * 2 + 1]);
        } else {
          if (left >= 1) row[nb * 8] = acc[mb][nb][hi * 2];
          if (left >= 2) row[nb * 8 + 1] = acc[mb][nb][hi * 2 + 1];
        }
      }
    }
}

__global__ void __launch_bounds__(256) dbias_reduce_kernel(const float* __restrict__ part, float* __restrict__ out, long long n, int chunks) {
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= n) return;
  float s = part[i];
  for (int c = 1; c < chunks; ++c) s += part[c * n + i];
  out[i] = s;
}

// ---------------------------------------------------------------------------------------------------- launches

template <typename K>
int start(K kern, long long ctas, size_t smem, cudaStream_t st, const AttnArgs& a) {
  if (smem > 48 * 1024) TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<(unsigned)ctas, kCta, smem, st>>>(a);
  TRI_LAUNCH_OK();
  return 0;
}
inline long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }

template <typename T, int DB, int MB, int NB, bool TF32>
int forward_launch(const AttnArgs& a, cudaStream_t st) {
  const TriAttnDesc& d = a.d;
  const double pairs = (double)d.B * d.n_seq * d.H * d.n_res * (double)d.n_res;
  KernelTimer kt("simt_attn_fwd", st, 4.0 * pairs * d.D, 4.0 * sizeof(T) * d.B * d.n_seq * (double)d.n_res * d.H * d.D);
  return start(attn_fwd_kernel<T, DB, MB, NB, TF32>, ceil_div(d.n_res, 64 * MB) * d.B * d.n_seq * d.H, fwd_smem<DB, MB, NB, TF32>(), st, a);
}

template <typename T, int DB, int MB, int NB, int NBB, bool TF32>
int backward_launch(AttnArgs a, float* part, cudaStream_t st) {
  const TriAttnDesc& d = a.d;
  const long long slices = (long long)d.B * d.n_seq * d.H, rows = slices * d.n_res;
  const double pairs = (double)rows * d.n_res, tensor_bytes = sizeof(T) * (double)d.B * d.n_seq * d.n_res * d.H * d.D;
  {
    KernelTimer kt("simt_attn_delta", st, 0.0, 2.0 * tensor_bytes);
    attn_delta_kernel<T><<<(unsigned)ceil_div(rows, 32), 256, 0, st>>>(a);
    TRI_LAUNCH_OK();
  }
  {
    KernelTimer kt("simt_attn_bwd_dkdv", st, 8.0 * pairs * d.D, 6.0 * tensor_bytes);
    TRI_TRY(start(attn_bwd_dkdv_kernel<T, DB, MB, NB, TF32>, ceil_div(d.n_res, 64 * MB) * slices, dkdv_smem<DB, MB, NB, TF32>(), st, a));
  }
  {
    KernelTimer kt("simt_attn_bwd_dq", st, 2.0 * pairs * d.D, 5.0 * tensor_bytes);
    TRI_TRY(start(attn_bwd_dq_kernel<T, DB, MB, NB, TF32>, ceil_div(d.n_res, 64 * MB) * slices, dq_smem<DB, MB, NB, TF32>(), st, a));
  }
  if (a.dbias != nullptr) {
    float* out = a.dbias;
    const long long plane = (long long)d.B * d.H * d.n_res * (long long)d.n_res;
    if (a.chunks > 1) a.dbias = part;
    KernelTimer kt("simt_attn_bwd_dbias", st, 0.0, 4.0 * tensor_bytes);
    TRI_TRY(start(attn_bwd_dbias_kernel<T, DB, 1, NBB, TF32>,
                  ceil_div(d.n_res, 64) * ceil_div(d.n_res, 8 * NBB) * d.B * d.H * a.chunks, dbias_smem<DB, 1, NBB>(), st, a));
    if (a.chunks > 1) {
      dbias_reduce_kernel<<<(unsigned)ceil_div(plane, 256), 256, 0, st>>>(part, out, plane, a.chunks);
      TRI_LAUNCH_OK();
    }
  }
  return 0;
}

}  // namespace

// Tiles by head dim.  Up to 32, where the accumulators are few, two 16-row blocks per warp share each fragment of the n rows
// (fewer shared loads per product) unless that would leave half of the last m tile empty; 16-bit operands come here only in
// small or odd shapes and have the one-block form alone.
template <typename T, bool TF32>
int forward_any(const AttnArgs& a, cudaStream_t st) {
  if (a.d.D <= 32) {
    if constexpr (sizeof(T) == 4)
      if (ceil_div(a.d.n_res, 64) % 2 == 0) return forward_launch<T, 32, 2, 8, TF32>(a, st);
    return forward_launch<T, 32, 1, 8, TF32>(a, st);
  }
  return a.d.D <= 64 ? forward_launch<T, 64, 1, 8, TF32>(a, st) : forward_launch<T, 128, 1, 4, TF32>(a, st);
}
template <typename T, bool TF32>
int backward_any(const AttnArgs& a, float* part, cudaStream_t st) {
  if (a.d.D <= 32) {
    if constexpr (sizeof(T) == 4)
      if (ceil_div(a.d.n_res, 64) % 2 == 0) return backward_launch<T, 32, 2, 4, 8, TF32>(a, part, st);
    return backward_launch<T, 32, 1, 8, 8, TF32>(a, part, st);
  }
  return a.d.D <= 64 ? backward_launch<T, 64, 1, 8, 4, TF32>(a, part, st) : backward_launch<T, 128, 1, 4, 4, TF32>(a, part, st);
}

}  // namespace simt
}  // namespace tri

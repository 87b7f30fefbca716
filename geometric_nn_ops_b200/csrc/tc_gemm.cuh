// Persistent, warp-specialised tcgen05 GEMM:  D[m, n] = sum_k A(m, k) * B(n, k), fp32 accumulation in TMEM.
//
//   warp 0      TMA producer: fills a ring of shared-memory stages (128-byte swizzle) with operand tiles
//   warp 1      MMA issuer:   tcgen05.mma from the stages into one of two TMEM accumulators
//   warps 2..9  epilogue:     two groups of four warps (each group covers the 128 TMEM lanes and takes every
//                             other 32 of the accumulator columns): tcgen05.ld, fused epilogue, 16/32-byte stores
//
// A tile is 128 (M) x BN (N); K advances 128 bytes per stage (64 bf16/fp16 or 32 fp32 elements).  Each
// operand may be K-major (K contiguous in global memory) or MN-major (M or N contiguous); the second form
// is what the transposed contractions and the weight-gradient GEMMs need, and costs nothing: only the TMA
// box shape and the MMA descriptors differ.  Two K "segments" with their own tensor maps can feed the
// same tile, either into the same accumulator columns (a sum of two products) or into the second half
// of them (two products side by side); the fused gate epilogues use that.  With split_k the batch index
// selects a K range instead of a batch entry (weight gradients over all pixels).
//
// The input-gate GEMMs run TRANSPOSED (weights are the M operand, pixels the N operand), so that a thread
// owns one channel and its registers hold consecutive pixels: the channel-major a / b / dPG tensors are
// then written and read with plain contiguous vector accesses instead of 2-byte scatters.
//
// All waits are bounded (see tc_common.cuh); a timeout lands in *args.err and the kernel drains.
#pragma once

#include "tc_common.cuh"

namespace tri {
namespace tc {

enum Epilogue {
  EPI_STORE = 0,         // out0[batch][m][n] = acc (+ bias0[n])
  EPI_GATE_IN = 1,       // transposed: rows = channels of one half (tile_m = a or b), cols [P(128 px) | G(128 px)]:
                         //   half-plane[c][px] = (P+bp)*sigmoid(G+bg)*mask[px]
  EPI_GATE_OUT = 2,      // rows = pixels, cols [y(128) | g(128)]: out0[m][c] = (y+b)*sigmoid(g+b)
  EPI_GATE_OUT_BWD = 3,  // same cols, aux = d_out: out0 = d_out*sig, out1 = d_out*(y+b)*sig*(1-sig)
  EPI_GATE_IN_BWD = 4,   // transposed like GATE_IN; aux2/aux3 = channel-major d(a), d(b); aux = mask;
                         //   d = d(half)[c][px]*mask;  out0 is channel-major [512][M]:
                         //   row half*256+c = d*sig(G),  row half*256+128+c = d*P*sig*(1-sig)
  EPI_GATE_MUL = 5,      // out0[m][n] = aux[m][n] * sigmoid(acc); aux alone comes from the kernels before
  EPI_LN_BWD = 6,        // rows of 128 channels: acc = d(LayerNorm(x)); dx = rstd (gamma acc - mean(gamma acc) - xhat mean(gamma acc xhat)),
                         //   and per CTA the sums over rows of acc xhat and acc
  EPI_LN_BWD_T = 7       // the same with the 128 channels as rows and pixels as columns; x and dx [128][N]
};
constexpr bool epi_is_ln(int epi) { return epi == EPI_LN_BWD || epi == EPI_LN_BWD_T; }

constexpr int kBM = 128;
constexpr int kStageA = kBM * 128;  // bytes
// warp 0 producer, warp 1 MMA, then the epilogue warps: 16 for the gate epilogues, whose per-element arithmetic (sigmoid,
// products) is latency-bound with fewer warps per scheduler, 8 for the plain store.  (Gate-in backward on 8 warps with the
// gradients fetched a tile ahead into registers: 0.381 ms per launch at 768 x 768 pixels against 0.365.)
constexpr int gemm_epi_warps(int epi) { return epi == EPI_STORE || epi == EPI_GATE_MUL ? 8 : 16; }
constexpr int gemm_threads(int epi) { return 64 + 32 * gemm_epi_warps(epi); }
// Operand stages and x tiles.  EPI_LN_BWD has ten (fp32: twenty) blocks of K per tile, and stages are worth more than a second x
// tile (768 x 768 pixels, bf16: 215 us per launch with four and two, 206 with five and one); EPI_LN_BWD_T has two (four), and it is
// the other way round (191 us with five and one, 137 with four and two; fp32 at 512 x 512 116 with four and one, 91 with two and two).
constexpr int gemm_stages(int epi, int bn, int es) {
  return epi == EPI_LN_BWD_T ? (es == 2 ? 4 : 2) : bn == 256 ? 4 : !epi_is_ln(epi) ? 6 : es == 2 ? 5 : 4;
}
constexpr int gemm_x_tiles(int epi) { return epi == EPI_LN_BWD_T ? 2 : 1; }
// (x tiles, partial sums; gamma, or the totals of 16 warps' columns and the tiles' pixels' statistics)
constexpr int gemm_extra(int epi, int es) {
  const int nx = gemm_x_tiles(epi);
  return !epi_is_ln(epi) ? 0 : nx * 128 * 128 * es + 2 * 4 * 128 * 8 + (epi == EPI_LN_BWD ? 512 : 16 * 256 + nx * 2 * 512);
}


struct GemmArgs {
  int M, N;                  // output extent of one batch entry
  int kblocks0, kblocks1;    // K blocks (of 128 bytes) in segment 0 / segment 1 (0 = no second segment)
  int seg1_col;              // accumulator column where segment 1 lands (0 = add to segment 0's columns)
  int seg1_n;                // N extent of segment 1's MMA (columns), segment 0 uses bn0
  int bn0;                   // N extent of segment 0's MMA: the columns from one tile to the next, up to the kernel's BN
  int batches, tiles_m, tiles_n;
  int split_k;               // batch index selects K range [batch*kblocks0, ...) instead of a batch entry
  int a_tile_batch;          // the M-tile index is A's batch coordinate (rows 0..127 of plane tile_m)
  int a_mn[2], b_mn[2];      // per segment: operand is MN-major
  uint32_t idesc[2];
  // epilogue
  void* out0;
  void* out1;
  long long ld_out, batch_out;   // elements
  const float* bias0;            // per output column (EPI_STORE) / per accumulator column or row (gates)
  const void* aux;               // mask (GATE_IN*) or d_out (GATE_OUT_BWD), in the input dtype
  const void* aux2;              // GATE_IN_BWD: channel-major gradient of the a half
  const void* aux3;              //              ... of the b half
  long long plane;               // GATE_IN(_BWD): pixels per batch entry; channel-major plane stride
  bool wide;                     // out0, out1, aux2, aux3 and the peers' buffers start on 32-byte boundaries
  // GATE_IN with peer_world > 0: channel c of half tm goes to GPU c / peer_cs, into its buffer
  // [2 * peer_batches][peer_cs][peer_world][plane] at (tm * peer_batches + batch, c % peer_cs, peer_rank)
  void* peer_out[16];
  int peer_world, peer_rank, peer_cs, peer_batches;
  // LN_BWD
  CUtensorMap tmX, tmDx;         // tiles of 128 rows x 128 bytes
  const void* gamma;             // [128] in the input dtype, or null
  const float *mean, *rstd;      // [M]
  float *sum_g, *sum_b;          // [CTAs][128]
  int* err;
};

template <typename T> struct ElemTraits;
template <> struct ElemTraits<__nv_bfloat16> { static constexpr int kind = KIND_BF16; };
template <> struct ElemTraits<__half> { static constexpr int kind = KIND_F16; };
template <> struct ElemTraits<float> { static constexpr int kind = KIND_TF32; };

__device__ __forceinline__ float fast_sigmoid(float x) {
  return rcp_approx(1.0f + ex2_approx(-1.4426950408889634f * x));
}

// sigmoid(x + b) of two values, x from the accumulator and nb2 = -b log2e: packed fp32x2 arithmetic around the two MUFU
// pairs.  (A quotient by __fdividef costs several instructions of range handling, which the denominator 1 + 2^y, at
// least one, does not need.)
__device__ __forceinline__ float2 sigmoid2(float2 x, float2 nb2 = make_float2(0.f, 0.f)) {
  const float2 t = __ffma2_rn(x, make_float2(-1.4426950408889634f, -1.4426950408889634f), nb2);
  const float2 den = __fadd2_rn(make_float2(ex2_approx(t.x), ex2_approx(t.y)), make_float2(1.0f, 1.0f));
  return make_float2(rcp_approx(den.x), rcp_approx(den.y));
}

// 8 consecutive elements <-> registers, with 16-byte (16-bit types) or 2 x 16-byte (fp32) accesses
template <typename T> __device__ __forceinline__ void load8(const T* p, float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    union { uint4 u; T h[8]; } pk;
    pk.u = *reinterpret_cast<const uint4*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_f32(pk.h[i]);
  }
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float* v) {
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack2<T>(v[0], v[1]), pack2<T>(v[2], v[3]), pack2<T>(v[4], v[5]), pack2<T>(v[6], v[7]));
  }
}

// The same 8 elements as raw 16-byte words: issued early, converted when used, so that a tile's global loads
// are all in flight before its arithmetic (the epilogue warps are too few to hide one load after another).
template <typename T> struct Raw8 { uint4 w[sizeof(T) == 4 ? 2 : 1]; };
template <typename T> __device__ __forceinline__ Raw8<T> ldraw8(const T* p) {
  Raw8<T> r;
  r.w[0] = __ldg(reinterpret_cast<const uint4*>(p));
  if constexpr (sizeof(T) == 4) r.w[1] = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  return r;
}
template <typename T> __device__ __forceinline__ void cvtraw8(const Raw8<T>& r, float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    v[0] = __uint_as_float(r.w[0].x); v[1] = __uint_as_float(r.w[0].y); v[2] = __uint_as_float(r.w[0].z); v[3] = __uint_as_float(r.w[0].w);
    v[4] = __uint_as_float(r.w[1].x); v[5] = __uint_as_float(r.w[1].y); v[6] = __uint_as_float(r.w[1].z); v[7] = __uint_as_float(r.w[1].w);
  } else {
    union { uint4 u; T h[8]; } pk;
    pk.u = r.w[0];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_f32(pk.h[i]);
  }
}

// the same as four packed pairs
template <typename T> __device__ __forceinline__ void cvtraw8p(const Raw8<T>& r, float2 (&v)[4]) {
  const uint4 a = r.w[0];
  if constexpr (sizeof(T) == 4) {
    const uint4 b = r.w[1];
    v[0] = make_float2(__uint_as_float(a.x), __uint_as_float(a.y)); v[1] = make_float2(__uint_as_float(a.z), __uint_as_float(a.w));
    v[2] = make_float2(__uint_as_float(b.x), __uint_as_float(b.y)); v[3] = make_float2(__uint_as_float(b.z), __uint_as_float(b.w));
  } else {
    v[0] = unpack2<T>(a.x); v[1] = unpack2<T>(a.y); v[2] = unpack2<T>(a.z); v[3] = unpack2<T>(a.w);
  }
}

// 32-byte accesses (16 values of a 16-bit type) for the channel-major tensors of the transposed gate GEMMs: a lane
// then reads or writes whole 32-byte sectors of its channel row instead of two half sectors in two requests.
template <typename T> __device__ __forceinline__ void ldraw16(const T* p, Raw8<T>& lo, Raw8<T>& hi) {
  static_assert(sizeof(T) == 2, "16-bit types");
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(lo.w[0].x), "=r"(lo.w[0].y), "=r"(lo.w[0].z), "=r"(lo.w[0].w), "=r"(hi.w[0].x), "=r"(hi.w[0].y),
                 "=r"(hi.w[0].z), "=r"(hi.w[0].w)
               : "l"(p));
}
// the i-th pair of eight values, and stores of eight and sixteen
template <typename T> __device__ __forceinline__ void putraw8(Raw8<T>& r, int i, float2 v) {
  if constexpr (sizeof(T) == 4) {
    uint4& w = r.w[i >> 1];
    if (i & 1) { w.z = __float_as_uint(v.x); w.w = __float_as_uint(v.y); }
    else { w.x = __float_as_uint(v.x); w.y = __float_as_uint(v.y); }
  } else {
    const uint32_t k = pack2<T>(v.x, v.y);
    if (i == 0) r.w[0].x = k; else if (i == 1) r.w[0].y = k; else if (i == 2) r.w[0].z = k; else r.w[0].w = k;
  }
}
template <typename T> __device__ __forceinline__ void straw8(T* p, const Raw8<T>& r) {
  reinterpret_cast<uint4*>(p)[0] = r.w[0];
  if constexpr (sizeof(T) == 4) reinterpret_cast<uint4*>(p)[1] = r.w[1];
}
template <typename T> __device__ __forceinline__ void straw16(T* p, const Raw8<T>& lo, const Raw8<T>& hi) {
  static_assert(sizeof(T) == 2, "16-bit types");
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.w[0].x), "r"(lo.w[0].y), "r"(lo.w[0].z),
               "r"(lo.w[0].w), "r"(hi.w[0].x), "r"(hi.w[0].y), "r"(hi.w[0].z), "r"(hi.w[0].w)
               : "memory");
}
template <typename T> __device__ __forceinline__ void store16(T* p, const float* v) {
  static_assert(sizeof(T) == 2, "16-bit types");
  uint32_t w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = pack2<T>(v[2 * i], v[2 * i + 1]);
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
               "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// One step of the transposition of 4 x 4 pieces of 16 bytes over four lanes: piece p of lane l meets piece p ^ B of lane l ^ B.
template <int B>
__device__ __forceinline__ void swap_pieces(uint32_t (&w)[16], int lane) {
  const bool up = (lane & B) != 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    if (p & B) continue;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint32_t &lo = w[4 * p + e], &hi = w[4 * (p | B) + e];
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, B);
      if (up) lo = got;
      else hi = got;
    }
  }
}

// 16 channels of this lane's pixel m (channels c ..) into rows of 128 floats; lanes are consecutive pixels, M a multiple of four
__device__ __forceinline__ void store_rows4(float* out, const float (&v)[16], int m, int M, int c, int lane) {
  uint32_t w[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(v[e]);
  swap_pieces<1>(w, lane);
  swap_pieces<2>(w, lane);
  if (m >= M) return;
  uint4* dst = reinterpret_cast<uint4*>(out + (long long)(m & ~3) * 128 + c) + (lane & 3);
#pragma unroll
  for (int q = 0; q < 4; ++q) dst[q * 32] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}
// pieces that were read from rows m & ~3 .. (one of four lanes' columns each) into 16 channels of this lane's row
template <typename T>
__device__ __forceinline__ void swap_rows(Raw8<T>& a, Raw8<T>& b, int lane) {
  if constexpr (sizeof(T) == 4) {
    uint32_t w[16] = {a.w[0].x, a.w[0].y, a.w[0].z, a.w[0].w, a.w[1].x, a.w[1].y, a.w[1].z, a.w[1].w,
                      b.w[0].x, b.w[0].y, b.w[0].z, b.w[0].w, b.w[1].x, b.w[1].y, b.w[1].z, b.w[1].w};
    swap_pieces<1>(w, lane);
    swap_pieces<2>(w, lane);
    a.w[0] = make_uint4(w[0], w[1], w[2], w[3]); a.w[1] = make_uint4(w[4], w[5], w[6], w[7]);
    b.w[0] = make_uint4(w[8], w[9], w[10], w[11]); b.w[1] = make_uint4(w[12], w[13], w[14], w[15]);
  }
}

// 32 columns of this lane's row, rows `ld` apart, all four rows of a lane group valid or none: the lanes exchange their 16-byte
// pieces, so that a request covers 64 bytes of eight rows
template <typename TOUT>
__device__ __forceinline__ void store_rows32(TOUT* dst, const float (&v)[32], long long ld, bool valid, int lane) {
  constexpr int E = 16 / sizeof(TOUT), H = sizeof(TOUT) / 2;   // elements of a piece; groups of four pieces
  TOUT* at = dst + (lane & 3) * (E - ld);
#pragma unroll
  for (int h = 0; h < H; ++h) {
    uint32_t w[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      if constexpr (sizeof(TOUT) == 4) w[e] = __float_as_uint(v[h * 16 + e]);
      else w[e] = pack2<TOUT>(v[2 * e], v[2 * e + 1]);
    }
    swap_pieces<1>(w, lane);
    swap_pieces<2>(w, lane);
    if (valid) {
#pragma unroll
      for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(at + q * ld + h * 4 * E) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    }
  }
}

template <typename TOUT>
__device__ __forceinline__ void store_row32(TOUT* dst, const float (&v)[32], int valid, bool vec_ok) {
  if (valid >= 32 && vec_ok) {
    if constexpr (sizeof(TOUT) == 2) {
      if ((reinterpret_cast<uintptr_t>(dst) & 31) == 0) {   // whole 32-byte sectors per request
        store16<TOUT>(dst, &v[0]);
        store16<TOUT>(dst + 16, &v[16]);
        return;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) store8<TOUT>(dst + 8 * i, &v[8 * i]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (vec_ok && i * 8 + 8 <= valid) {
        store8<TOUT>(dst + 8 * i, &v[8 * i]);
      } else {
#pragma unroll
        for (int e = i * 8; e < i * 8 + 8; ++e)
          if (e < valid) dst[e] = from_f32<TOUT>(v[e]);
      }
    }
  }
}

// two 32-column loads (columns c0.. and c1..) with one wait
__device__ __forceinline__ void ld32x2_f(uint32_t t0, uint32_t t1, float (&a)[32], float (&b)[32]) {
  uint32_t ra[32], rb[32];
  tmem_ld_32x32(t0, ra);
  tmem_ld_32x32(t1, rb);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) { a[i] = __uint_as_float(ra[i]); b[i] = __uint_as_float(rb[i]); }
}
// two 16-column loads with one wait
__device__ __forceinline__ void ld16x2_f(uint32_t t0, uint32_t t1, float (&a)[16], float (&b)[16]) {
  uint32_t ra[16], rb[16];
  tmem_ld_32x16(t0, ra);
  tmem_ld_32x16(t1, rb);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) { a[i] = __uint_as_float(ra[i]); b[i] = __uint_as_float(rb[i]); }
}
__device__ __forceinline__ void ld32_f(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  tmem_ld_32x32(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// where the gate-in epilogue writes channel `row` of half `tm`, batch entry `bb`, pixel `pix`: this GPU's
// channel-major output, or (row-sharded runs) the exchange buffer of the GPU that owns the channel
template <typename TOUT>
__device__ __forceinline__ TOUT* gate_in_dst(const GemmArgs& g, int tm, long long bb, int row, long long pix) {
  if (g.peer_world > 0) {
    const int w = row / g.peer_cs, cl = row - w * g.peer_cs;
    return reinterpret_cast<TOUT*>(g.peer_out[w]) +
           ((((long long)tm * g.peer_batches + bb) * g.peer_cs + cl) * g.peer_world + g.peer_rank) * g.plane + pix;
  }
  return reinterpret_cast<TOUT*>(tm == 0 ? g.out0 : g.out1) + (bb * 128 + row) * g.plane + pix;
}

// sums over the 32 lanes of a warp of 32 values each: lane l gets value l's (31 exchanges)
__device__ __forceinline__ float sum_lanes32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// Epilogue EPI_LN_BWD, 16 warps: thread = row (pixel) of the tile, 32 of its 128 channels; a row's four threads meet through
// shared memory.  dx replaces x in its tile and leaves by TMA.  The sums over rows (the LayerNorm's weight gradients) go across
// the lanes of a warp, tile by tile, and across warps at the end.  No early return: the warps meet on named barriers.
// At 768 x 768 pixels, bf16: 206 us per launch for 7 tensors (161 at the copy rate), against 145 + 93 for the product and a kernel of
// its own with dz between them; fp32 (TF32) at 512 x 512 181 against 140 + 66.
template <typename T>
__device__ __forceinline__ void ln_bwd_rows(const GemmArgs& g, uint8_t* sX, float2* s_part, float* s_gamma, uint64_t* tfull, uint64_t* tempty,
                                            uint64_t* xfull, uint64_t* xempty, uint32_t tmem_base, int total, int warp, int lane) {
  constexpr int ES = sizeof(T), PIECES = 32 * ES / 16;          // 16-byte pieces of a thread's channels
  const int quarter = warp & 3, grp = (warp - 2) >> 2, row = quarter * 32 + lane, t = (warp - 2) * 32 + lane;
  if (t < 128) s_gamma[t] = g.gamma ? to_f32(static_cast<const T*>(g.gamma)[t]) : 1.f;
  named_barrier(5, 512);
  // this thread's pieces: its sub-tile of 128-byte rows, swizzled by the row
  const uint32_t xa = smem_u32(sX) + (ES == 2 ? grp >> 1 : grp) * 16384 + row * 128, piece0 = ES == 2 ? (grp & 1) * 4 : 0, sw = row & 7;
  float acc_g = 0.f, acc_b = 0.f;
  int acc = 0, i = 0;
  uint32_t acc_phase = 0;
  for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++i) {
    const int m = tile * kBM + row;
    float mu = 0.f, rs = 0.f;
    if (m < g.M) { mu = g.mean[m]; rs = g.rstd[m]; }
    mbar_wait(xfull, i & 1, g.err, 7);
    mbar_wait(&tfull[acc], acc_phase, g.err, 4);
    tc_fence_after_sync();
    float v[32], xh[32];
    ld32_f(tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * 128 + grp * 32, v);
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&tempty[acc]);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const uint4 raw = lds128(xa + (((piece0 + p) ^ sw) << 4));
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (ES == 2) {
          const float2 x = unpack2<T>(w[e]);
          xh[p * 8 + 2 * e] = (x.x - mu) * rs;
          xh[p * 8 + 2 * e + 1] = (x.y - mu) * rs;
        } else {
          xh[p * 4 + e] = (__uint_as_float(w[e]) - mu) * rs;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
      const float4 gm = *reinterpret_cast<const float4*>(s_gamma + grp * 32 + c);
      const float k[4] = {gm.x, gm.y, gm.z, gm.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float d = v[c + e] * k[e];
        s1 += d;
        s2 = fmaf(d, xh[c + e], s2);
      }
    }
    float2* part = s_part + (i & 1) * 512;     // (the set of two tiles ago: every warp has met the others since it was read)
    part[grp * 128 + row] = make_float2(s1, s2);
    named_barrier(1 + quarter, 128);
    s1 = s2 = 0.f;
#pragma unroll
    for (int q = 0; q < 4; ++q) { const float2 p = part[q * 128 + row]; s1 += p.x; s2 += p.y; }
    s1 *= 1.0f / 128;
    s2 *= 1.0f / 128;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      uint32_t w[4];
      auto dx = [&](int c) { return rs * (v[c] * s_gamma[grp * 32 + c] - s1 - xh[c] * s2); };
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if constexpr (ES == 2) w[e] = pack2<T>(dx(p * 8 + 2 * e), dx(p * 8 + 2 * e + 1));
        else w[e] = __float_as_uint(dx(p * 4 + e));
      }
      sts128(xa + (((piece0 + p) ^ sw) << 4), w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async_smem();
    named_barrier(5, 512);
    if (t == 0) {
      for (int c = 0; c < ES; ++c) tma_store_3d(&g.tmDx, sX + c * 16384, c * (128 / ES), tile * kBM, 0);
      bulk_commit_group();
      bulk_wait_group_read0();
      mbar_arrive(xempty);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 32; ++c) xh[c] *= v[c];
    acc_g += sum_lanes32(xh, lane);
    acc_b += sum_lanes32(v, lane);
    acc ^= 1;
    if (acc == 0) acc_phase ^= 1;
  }
  // channel grp 32 + lane of this warp's quarter of the rows
  named_barrier(5, 512);
  s_part[quarter * 128 + grp * 32 + lane] = make_float2(acc_g, acc_b);
  named_barrier(5, 512);
  if (t < 128) {
    float2 s = s_part[t];
    for (int q = 1; q < 4; ++q) { const float2 p = s_part[q * 128 + t]; s.x += p.x; s.y += p.y; }
    g.sum_g[blockIdx.x * 128 + t] = s.x;
    g.sum_b[blockIdx.x * 128 + t] = s.y;
  }
  if (t == 0) bulk_wait_group0();
}

// Epilogue EPI_LN_BWD_T: thread = channel, 32 of the tile's 128 pixels.  Here the sums over channels go across the lanes of a warp
// and the four warps of a pixel chunk, and the sums over pixels stay in the thread.  xhat is formed twice: its registers would not
// fit beside the accumulators and the sums under way.  No early return, as above.
// At 768 x 768 pixels, bf16: 137 us per launch for 3 tensors (69 at the copy rate), against 55 + 117 with du between two kernels;
// fp32 (TF32) at 512 x 512 91 against 47 + 101.
template <typename T>
__device__ __forceinline__ void ln_bwd_cols(const GemmArgs& g, uint8_t* sX, float2* s_part, float2* s_tot, const float* s_stat, uint64_t* tfull,
                                            uint64_t* tempty, uint64_t* xfull, uint64_t* xempty, uint32_t tmem_base, int total, int warp, int lane) {
  constexpr int ES = sizeof(T), PIECES = 32 * ES / 16, PE = 16 / ES;     // 16-byte pieces of a thread's pixels, elements of one
  constexpr int NX = gemm_x_tiles(EPI_LN_BWD_T), XBYTES = 128 * 128 * ES;
  const int quarter = warp & 3, grp = (warp - 2) >> 2, row = quarter * 32 + lane, t = (warp - 2) * 32 + lane;
  const float gamma = g.gamma ? to_f32(static_cast<const T*>(g.gamma)[row]) : 1.f;
  const uint32_t xa0 = smem_u32(sX) + (ES == 2 ? grp >> 1 : grp) * 16384 + row * 128, piece0 = ES == 2 ? (grp & 1) * 4 : 0, sw = row & 7;
  float2* tot = s_tot + (warp - 2) * 32;
  float acc_g = 0.f, acc_b = 0.f;
  int acc = 0, i = 0;
  uint32_t acc_phase = 0;
  uint32_t xa = xa0;
  const float *s_mu = s_stat + grp * 32, *s_rs = s_mu + 128;
  // xhat of a piece's pixels
  auto hats = [&](int p, float (&xh)[PE]) {
    const uint4 raw = lds128(xa + (((piece0 + p) ^ sw) << 4));
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < PE; e += 4) {
      const float4 mu = *reinterpret_cast<const float4*>(s_mu + p * PE + e), rs = *reinterpret_cast<const float4*>(s_rs + p * PE + e);
      float x[4];
      if constexpr (ES == 2) {
        const float2 a = unpack2<T>(w[e / 2]), b = unpack2<T>(w[e / 2 + 1]);
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = __uint_as_float(w[k]);
      }
      xh[e] = (x[0] - mu.x) * rs.x; xh[e + 1] = (x[1] - mu.y) * rs.y; xh[e + 2] = (x[2] - mu.z) * rs.z; xh[e + 3] = (x[3] - mu.w) * rs.w;
    }
  };
  for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++i) {
    const int b = i % NX;
    xa = xa0 + b * XBYTES;
    s_mu = s_stat + b * 256 + grp * 32;
    s_rs = s_mu + 128;
    mbar_wait(&xfull[b], (i / NX) & 1, g.err, 7);
    mbar_wait(&tfull[acc], acc_phase, g.err, 4);
    tc_fence_after_sync();
    float v[32];
    ld32_f(tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * 128 + grp * 32, v);
    tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive(&tempty[acc]);
    float2 mine;       // this warp's channels' sums for pixel grp 32 + lane
    {
      float a[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) { acc_b += v[c]; a[c] = v[c] * gamma; }
      mine.x = sum_lanes32(a, lane);
    }
    {
      float a[32];
#pragma unroll
      for (int p = 0; p < PIECES; ++p) {
        float xh[PE];
        hats(p, xh);
#pragma unroll
        for (int e = 0; e < PE; ++e) {
          const float d = v[p * PE + e] * xh[e];
          acc_g += d;
          a[p * PE + e] = d * gamma;
        }
      }
      mine.y = sum_lanes32(a, lane);
    }
    float2* part = s_part + (i & 1) * 512 + grp * 32 + lane;     // (the set of two tiles ago: every warp has met the others since it was read)
    part[quarter * 128] = mine;
    named_barrier(1 + grp, 128);
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; ++q) { const float2 p = part[q * 128]; sum.x += p.x; sum.y += p.y; }
    __syncwarp();
    tot[lane] = make_float2(sum.x * (1.0f / 128), sum.y * (1.0f / 128));
    __syncwarp();
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      float xh[PE], o[PE];
      hats(p, xh);
#pragma unroll
      for (int e = 0; e < PE; e += 2) {
        const float4 m = *reinterpret_cast<const float4*>(tot + p * PE + e);    // two pixels
        const float2 rs = *reinterpret_cast<const float2*>(s_rs + p * PE + e);
        o[e] = rs.x * (v[p * PE + e] * gamma - m.x - xh[e] * m.y);
        o[e + 1] = rs.y * (v[p * PE + e + 1] * gamma - m.z - xh[e + 1] * m.w);
      }
      uint32_t w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (ES == 2) w[k] = pack2<T>(o[2 * k], o[2 * k + 1]);
        else w[k] = __float_as_uint(o[k]);
      }
      sts128(xa + (((piece0 + p) ^ sw) << 4), w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async_smem();
    named_barrier(5, 512);
    if (t == 0) {
      for (int c = 0; c < ES; ++c) tma_store_3d(&g.tmDx, sX + b * XBYTES + c * 16384, tile * 128 + c * (128 / ES), 0, 0);
      bulk_commit_group();
      bulk_wait_group_read0();
      mbar_arrive(&xempty[b]);
    }
    __syncwarp();
    acc ^= 1;
    if (acc == 0) acc_phase ^= 1;
  }
  // this thread's channel, its 32 of each tile's pixels
  named_barrier(5, 512);
  s_part[grp * 128 + row] = make_float2(acc_g, acc_b);
  named_barrier(5, 512);
  if (t < 128) {
    float2 s = s_part[t];
    for (int q = 1; q < 4; ++q) { const float2 p = s_part[q * 128 + t]; s.x += p.x; s.y += p.y; }
    g.sum_g[blockIdx.x * 128 + t] = s.x;
    g.sum_b[blockIdx.x * 128 + t] = s.y;
  }
  if (t == 0) bulk_wait_group0();
}

template <typename TIN, typename TOUT, int BN, int EPI, int STAGES>
__global__ void __launch_bounds__(gemm_threads(EPI), 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmB0,
               const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ GemmArgs g) {
  constexpr int ES = sizeof(TIN);
  constexpr int BKE = 128 / ES;        // K elements per stage
  constexpr int UK = 32 / ES;          // K elements per MMA
  constexpr int CE = 128 / ES;         // MN elements per 128-byte chunk (MN-major operands)
  constexpr int STAGE_B = BN * 128;
  // MN-major tiles: 16-bit types use the plain 128-byte swizzle (8-k groups of 1024 bytes); 32-bit
  // types only exist with the 32-byte-atom swizzle (4-k groups of 512 bytes, layout code 1).
  constexpr uint32_t MN_SBO = ES == 4 ? 512 : 1024;
  constexpr uint32_t MN_LAYOUT = ES == 4 ? 1 : 2;
  constexpr int KIND = ElemTraits<TIN>::kind == KIND_TF32 ? KIND_TF32 : KIND_F16;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * kStageA;
  // LN_BWD: the x tile, two sets of partial sums, gamma; LN_BWD_T: ..., 16 warps' totals, the pixels' mean and rstd
  [[maybe_unused]] constexpr int XBYTES = 128 * 128 * ES, NX = gemm_x_tiles(EPI);
  uint8_t* sX = sB + STAGES * STAGE_B;
  [[maybe_unused]] float2* s_part = reinterpret_cast<float2*>(sX + NX * XBYTES);     // [2][4][128]
  [[maybe_unused]] float* s_gamma = reinterpret_cast<float*>(s_part + 2 * 4 * 128);
  [[maybe_unused]] float2* s_tot = s_part + 2 * 4 * 128;
  [[maybe_unused]] float* s_stat = reinterpret_cast<float*>(s_tot + 16 * 32);      // [NX][2][128]
  uint64_t* full = reinterpret_cast<uint64_t*>(sX + gemm_extra(EPI, ES));
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint64_t* tempty = tfull + 2;
  [[maybe_unused]] uint64_t* xfull = tempty + 2;     // [2] x tile landed
  [[maybe_unused]] uint64_t* xempty = xfull + 2;     // [2] ... and its dx has been read by the store
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2 + (epi_is_ln(EPI) ? 4 : 0));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], gemm_epi_warps(EPI)); }
    if constexpr (epi_is_ln(EPI)) {
      for (int b = 0; b < 2; ++b) { mbar_init(&xfull[b], 1); mbar_init(&xempty[b], 1); }
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmA0);
    tma_prefetch_desc(&tmB0);
  }
  if constexpr (EPI == EPI_LN_BWD_T) {   // what a last tile's copies leave unwritten is read beside zeros
    if (threadIdx.x < NX * 256) s_stat[threadIdx.x] = 0.f;
    fence_proxy_async_smem();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 2 * BN);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  if constexpr (EPI == EPI_GATE_MUL) dependent_trigger();   // (the epilogue waits; s and the weights were there before o's call)
  else dependent_enter();

  const int total = g.batches * g.tiles_m * g.tiles_n;
  const int kb_total = g.kblocks0 + g.kblocks1;
  // tile -> (batch, tile_m, tile_n); with a_tile_batch the M tiles (weight blocks) of one pixel tile are
  // adjacent in the schedule so the shared activation tile is still in L2 for the second one
  auto decode = [&](int tile, int& tm, int& tn, int& bz) {
    if (g.a_tile_batch) { tm = tile % g.tiles_m; tn = (tile / g.tiles_m) % g.tiles_n; }
    else { tn = tile % g.tiles_n; tm = (tile / g.tiles_n) % g.tiles_m; }
    bz = tile / (g.tiles_n * g.tiles_m);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    const bool leader = elect_one();
    if (leader) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        int tm, tn, bz;
        decode(tile, tm, tn, bz);
        const int n0 = tn * g.bn0;
        const int zc = g.split_k ? 0 : bz;
        const int koff = g.split_k ? bz * g.kblocks0 * BKE : 0;
        const int am = g.a_tile_batch ? 0 : tm * kBM, az = g.a_tile_batch ? tm : zc;
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, g.err, 1)) { ok = false; break; }
          const int seg = kb >= g.kblocks0 ? 1 : 0;
          const int kk = (seg ? kb - g.kblocks0 : kb) * BKE + koff;
          const CUtensorMap* ma = seg ? &tmA1 : &tmA0;
          const CUtensorMap* mb = seg ? &tmB1 : &tmB0;
          const int bn = seg ? g.seg1_n : g.bn0;
          mbar_expect_tx(&full[stage], kStageA + bn * 128);
          uint8_t* a_dst = sA + stage * kStageA;
          uint8_t* b_dst = sB + stage * STAGE_B;
          if (!g.a_mn[seg]) {
            tma_load_3d(a_dst, ma, &full[stage], kk, am, az);
          } else {
            for (int c = 0; c < kBM / CE; ++c) tma_load_3d(a_dst + c * (BKE * 128), ma, &full[stage], am + c * CE, kk, az);
          }
          if (!g.b_mn[seg]) {
            tma_load_3d(b_dst, mb, &full[stage], kk, n0, zc);
          } else {
            for (int c = 0; c < bn / CE; ++c) tma_load_3d(b_dst + c * (BKE * 128), mb, &full[stage], n0 + c * CE, kk, zc);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if constexpr (epi_is_ln(EPI)) {   // (after the operands: the tile before may still hold the buffer)
          const uint32_t i = (tile - blockIdx.x) / gridDim.x, b = i % NX;
          uint64_t* bar = &xfull[b];
          if (!ok || !mbar_wait(&xempty[b], ((i / NX) & 1) ^ 1, g.err, 6)) break;
          const uint32_t stat = EPI == EPI_LN_BWD_T ? 4 * min(128, g.N - n0) : 0;   // (N is a multiple of four)
          mbar_expect_tx(bar, XBYTES + 2 * stat);
          for (int c = 0; c < ES; ++c)
            tma_load_3d(sX + b * XBYTES + c * 16384, &g.tmX, bar, EPI == EPI_LN_BWD ? c * CE : n0 + c * CE, EPI == EPI_LN_BWD ? tm * kBM : 0, 0);
          if constexpr (EPI == EPI_LN_BWD_T) {
            bulk_load(s_stat + b * 256, g.mean + n0, stat, bar);
            bulk_load(s_stat + b * 256 + 128, g.rstd + n0, stat, bar);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    const bool leader = elect_one();
    if (leader) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      const uint32_t a_base = smem_u32(sA), b_base = smem_u32(sB);
      for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, g.err, 2)) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < kb_total; ++kb) {
          if (!mbar_wait(&full[stage], phase, g.err, 3)) { ok = false; break; }
          tc_fence_after_sync();
          const int seg = kb >= g.kblocks0 ? 1 : 0;
          const int kin = seg ? kb - g.kblocks0 : kb;
          const uint32_t d_addr = tmem_base + acc * BN + (seg ? g.seg1_col : 0);
          const bool fresh = kin == 0 && !(seg == 1 && g.seg1_col == 0);  // first product into these columns
          const uint32_t a_stage = a_base + stage * kStageA, b_stage = b_base + stage * STAGE_B;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t ad = g.a_mn[seg] ? make_smem_desc(a_stage + ks * UK * 128, BKE * 128, MN_SBO, MN_LAYOUT)
                                            : make_smem_desc(a_stage + ks * 32, 16, 1024);
            const uint64_t bd = g.b_mn[seg] ? make_smem_desc(b_stage + ks * UK * 128, BKE * 128, MN_SBO, MN_LAYOUT)
                                            : make_smem_desc(b_stage + ks * 32, 16, 1024);
            umma<KIND>(d_addr, ad, bd, g.idesc[seg], (fresh && ks == 0) ? 0u : 1u);
          }
          umma_commit(&empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (ok) umma_commit(&tfull[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue: groups of 4 warps
    const int quarter = warp & 3;            // the TMEM lane quarter this warp may read
    const int grp = (warp - 2) >> 2;         // column share this warp's group takes (2 or 4 groups)
    constexpr int NGRP = gemm_epi_warps(EPI) / 4;
    constexpr int CPG = 4 / NGRP;            // gate epilogues: 32-pixel (or channel) chunks per group
    const int row = quarter * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    if constexpr (EPI == EPI_GATE_MUL) dependent_wait();
    if constexpr (EPI == EPI_LN_BWD) {
      ln_bwd_rows<TIN>(g, sX, s_part, s_gamma, tfull, tempty, xfull, xempty, tmem_base, total, warp, lane);
    } else if constexpr (EPI == EPI_LN_BWD_T) {
      ln_bwd_cols<TIN>(g, sX, s_part, s_tot, s_stat, tfull, tempty, xfull, xempty, tmem_base, total, warp, lane);
    } else {
    // The backward gate epilogues read a gradient tile from global memory, just before they wait for the product.
    constexpr bool kGradTile = EPI == EPI_GATE_IN_BWD || EPI == EPI_GATE_OUT_BWD;
    auto fetch_grad = [&](int t, Raw8<TIN> (&dst)[CPG][4]) {
      int tm, tn, bz;
      decode(t, tm, tn, bz);
      if constexpr (EPI == EPI_GATE_IN_BWD) {
        const TIN* dplane = reinterpret_cast<const TIN*>(tm == 0 ? g.aux2 : g.aux3);
        const uint32_t t0 = (uint32_t)tn * 128, plane = (uint32_t)g.plane, tb0 = t0 / plane, tp0 = t0 - tb0 * plane;
        const TIN* base = dplane + ((long long)tb0 * 128 + row) * g.plane + tp0;
        const bool wide = sizeof(TIN) == 2 && (g.plane & 15) == 0 && (g.N & 15) == 0 && g.wide;   // 16-pixel groups: aligned, never split
#pragma unroll
        for (int jj = 0; jj < CPG; ++jj)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int off = (grp * CPG + jj) * 32 + u * 8;
            if (t0 + off < (uint32_t)g.N) {
              const TIN* src = base + off;
              for (uint32_t pix = tp0 + off; pix >= plane; pix -= plane) src += 127 * g.plane;   // the next batch entry's plane of this channel
              if constexpr (sizeof(TIN) == 2) {
                if (wide) { if ((u & 1) == 0) ldraw16<TIN>(src, dst[jj][u], dst[jj][u + 1]); }
                else dst[jj][u] = ldraw8<TIN>(src);
              } else {
                dst[jj][u] = ldraw8<TIN>(src);
              }
            }
          }
      } else if constexpr (EPI == EPI_GATE_OUT_BWD) {
        const int m = tm * kBM + row;
        const TIN* dout = reinterpret_cast<const TIN*>(g.aux) + (long long)m * 128;
        const bool wide = (reinterpret_cast<uintptr_t>(g.aux) & 31) == 0;   // (rows of 256 bytes; the caller's tensor may start between)
        if (m < g.M) {
#pragma unroll
          for (int jj = 0; jj < CPG; ++jj)
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
              if constexpr (sizeof(TIN) == 2) {
                const TIN* src = dout + (grp * CPG + jj) * 32 + u * 8;
                if (wide) {
                  ldraw16<TIN>(src, dst[jj][u], dst[jj][u + 1]);
                } else {
                  dst[jj][u] = ldraw8<TIN>(src);
                  dst[jj][u + 1] = ldraw8<TIN>(src + 8);
                }
              } else {
                // (each lane a quarter of four rows' 16 channels: swap_rows gives it its own row's)
                const uint4* src = reinterpret_cast<const uint4*>(dout - (long long)(lane & 3) * 128 + (grp * CPG + jj) * 32 + u * 8) + (lane & 3);
                dst[jj][u].w[0] = __ldg(src); dst[jj][u].w[1] = __ldg(src + 32);
                dst[jj][u + 1].w[0] = __ldg(src + 64); dst[jj][u + 1].w[1] = __ldg(src + 96);
              }
            }
        }
      }
    };
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      int tm, tn, bz;
      decode(tile, tm, tn, bz);
      Raw8<TIN> dpre[CPG][4];
      if constexpr (kGradTile) fetch_grad(tile, dpre);
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull[acc], acc_phase, g.err, 4))) break;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * BN;
      if constexpr (EPI == EPI_STORE || EPI == EPI_GATE_MUL) {
        const int m = tm * kBM + row, n0 = tn * g.bn0, n_end = min(g.N, n0 + g.bn0);
        TOUT* out = reinterpret_cast<TOUT*>(g.out0) + bz * g.batch_out + (long long)m * g.ld_out;
        const bool vec_ok = (g.ld_out * sizeof(TOUT)) % 16 == 0 && (g.batch_out * sizeof(TOUT)) % 16 == 0 && (reinterpret_cast<uintptr_t>(g.out0) & 15) == 0;
#pragma unroll 1
        for (int j = grp; j * 32 < g.bn0; j += NGRP) {   // 32-column chunks
          float v[32];
          ld32_f(t_row + j * 32, v);
          const int n = n0 + j * 32;
          if (g.bias0 != nullptr) {
#pragma unroll
            for (int i = 0; i < 32; ++i) if (n + i < n_end) v[i] += g.bias0[n + i];
          }
          if constexpr (EPI == EPI_GATE_MUL) {   // (N is a multiple of eight)
            const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const TIN*>(g.aux) + (long long)m * g.ld_out + n);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (m >= g.M || n + u * 8 >= n_end) continue;
              const uint4 x = src[u];
              const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 r = __fmul2_rn(unpack2<TIN>(w[i]), sigmoid2(make_float2(v[u * 8 + 2 * i], v[u * 8 + 2 * i + 1])));
                v[u * 8 + 2 * i] = r.x;
                v[u * 8 + 2 * i + 1] = r.y;
              }
            }
          }
          if ((g.M & 3) == 0 && vec_ok && n_end - n >= 32) store_rows32<TOUT>(out + n, v, g.ld_out, m < g.M, lane);
          else if (m < g.M && n < n_end) store_row32<TOUT>(out + n, v, n_end - n, vec_ok);
        }
      } else if constexpr (EPI == EPI_GATE_IN || EPI == EPI_GATE_IN_BWD) {
        // row = channel of half tm; columns: P for pixels n0..n0+127, then G for the same pixels
        const uint32_t n0 = (uint32_t)tn * 128, plane = (uint32_t)g.plane, np0 = n0 % plane;
        const bool wide16 = sizeof(TOUT) == 2 && (g.plane & 15) == 0 && (g.N & 15) == 0 && (g.ld_out & 15) == 0 && g.wide;
        // fp32: 16 pixels of four channels, exchanged between four lanes (64 bytes of eight rows per request, not 16 of 32)
        const bool wide4 = EPI == EPI_GATE_IN && sizeof(TOUT) == 4 && (g.plane & 15) == 0 && (g.N & 15) == 0 && g.peer_world == 0;
        const TIN* mask = reinterpret_cast<const TIN*>(g.aux);
        float bp = 0.f, bg = 0.f;
        if (g.bias0 != nullptr) { bp = g.bias0[tm * 256 + row]; bg = g.bias0[tm * 256 + 128 + row]; }
        const float2 bp2 = make_float2(bp, bp), nbg2 = make_float2(-1.4426950408889634f * bg, -1.4426950408889634f * bg);
        // gate-in: this channel's plane at the tile's first pixel; backward: the dP row (dG lies 128 rows on)
        TOUT* dst0;
        if constexpr (EPI == EPI_GATE_IN) dst0 = gate_in_dst<TOUT>(g, tm, n0 / plane, row, np0);
        else dst0 = reinterpret_cast<TOUT*>(g.out0) + (long long)(tm * 256 + row) * g.ld_out + n0;
#pragma unroll
        for (int jj = 0; jj < CPG; ++jj) {
          const int j = grp * CPG + jj;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {   // 16 pixels at a time keeps the registers of 576 threads within budget
            const uint32_t off = j * 32 + hf * 16;
            float p[16], gt[16];
            ld16x2_f(t_row + off, t_row + 128 + off, p, gt);
            Raw8<TOUT> o0[2], o1[2];   // GATE_IN: gated value; GATE_IN_BWD: dP and dG
#pragma unroll
            for (int uu = 0; uu < 2; ++uu) {
              const uint32_t m8 = n0 + off + uu * 8;   // 8 pixels: same batch entry, all valid or none
              if (m8 >= (uint32_t)g.N) continue;
              float2 mk[4];
              if (mask != nullptr) cvtraw8p<TIN>(ldraw8<TIN>(mask + m8), mk);
              float2 d[4];
              if constexpr (EPI == EPI_GATE_IN_BWD) cvtraw8p<TIN>(dpre[jj][hf * 2 + uu], d);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int e = uu * 8 + 2 * i;
                const float2 pv = __fadd2_rn(make_float2(p[e], p[e + 1]), bp2);
                const float2 sg = sigmoid2(make_float2(gt[e], gt[e + 1]), nbg2);
                if constexpr (EPI == EPI_GATE_IN) {
                  float2 r = __fmul2_rn(pv, sg);
                  if (mask != nullptr) r = __fmul2_rn(r, mk[i]);
                  putraw8(o0[uu], i, r);
                } else {
                  float2 dd = d[i];
                  if (mask != nullptr) dd = __fmul2_rn(dd, mk[i]);
                  const float2 dp = __fmul2_rn(dd, sg);                                           // d * sig
                  const float2 oms = __ffma2_rn(sg, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f));
                  const float2 dg = __fmul2_rn(__fmul2_rn(dp, pv), oms);                          // d * P * sig * (1 - sig)
                  putraw8(o0[uu], i, dp);
                  putraw8(o1[uu], i, dg);
                }
              }
              if (!wide16 && !wide4) {
                TOUT* dst = dst0 + off + uu * 8;
                if constexpr (EPI == EPI_GATE_IN) {
                  if (np0 + off + uu * 8 >= plane) dst = gate_in_dst<TOUT>(g, tm, m8 / plane, row, m8 % plane);
                  straw8<TOUT>(dst, o0[uu]);
                } else {
                  straw8<TOUT>(dst, o0[uu]);
                  straw8<TOUT>(dst + 128 * g.ld_out, o1[uu]);
                }
              }
            }
            if constexpr (sizeof(TOUT) == 4 && EPI == EPI_GATE_IN) {
              if (wide4 && n0 + off < (uint32_t)g.N) {
                TOUT* dst = np0 + off >= plane ? gate_in_dst<TOUT>(g, tm, (n0 + off) / plane, row, (n0 + off) % plane) : dst0 + off;
                swap_rows(o0[0], o0[1], lane);
                uint4* at = reinterpret_cast<uint4*>(dst - (long long)(lane & 3) * g.plane) + (lane & 3);
                const long long step = g.plane / 4;
                at[0] = o0[0].w[0]; at[step] = o0[0].w[1]; at[2 * step] = o0[1].w[0]; at[3 * step] = o0[1].w[1];
              }
            }
            if constexpr (sizeof(TOUT) == 2) {
              if (wide16 && n0 + off < (uint32_t)g.N) {   // one 32-byte store per output row
                TOUT* dst = dst0 + off;
                if constexpr (EPI == EPI_GATE_IN) {
                  if (np0 + off >= plane) dst = gate_in_dst<TOUT>(g, tm, (n0 + off) / plane, row, (n0 + off) % plane);
                  straw16<TOUT>(dst, o0[0], o0[1]);
                } else {
                  straw16<TOUT>(dst, o0[0], o0[1]);
                  straw16<TOUT>(dst + 128 * g.ld_out, o1[0], o1[1]);
                }
              }
            }
          }
        }
      } else {
        // EPI_GATE_OUT / EPI_GATE_OUT_BWD: row = pixel; cols [0,128) = y, [128,256) = gate pre-activation
        const int m = tm * kBM + row;
        TOUT* o0 = reinterpret_cast<TOUT*>(g.out0) + (long long)m * 128;
        TOUT* o1 = reinterpret_cast<TOUT*>(g.out1) + (long long)m * 128;
#pragma unroll
        for (int jj = 0; jj < CPG; ++jj) {
          const int j = grp * CPG + jj;
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            float y[16], gt[16];
            ld16x2_f(t_row + j * 32 + hf * 16, t_row + 128 + j * 32 + hf * 16, y, gt);
            {
              float r0[16], r1[16];
              if constexpr (EPI == EPI_GATE_OUT_BWD && sizeof(TIN) == 4) swap_rows(dpre[jj][hf * 2], dpre[jj][hf * 2 + 1], lane);
#pragma unroll
              for (int uu = 0; uu < 2; ++uu) {
                float2 d[4];
                if constexpr (EPI == EPI_GATE_OUT_BWD) cvtraw8p<TIN>(dpre[jj][hf * 2 + uu], d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const int e = uu * 8 + 2 * i, c = j * 32 + hf * 16 + e;
                  float2 yv = make_float2(y[e], y[e + 1]), gv = make_float2(gt[e], gt[e + 1]);
                  if (g.bias0 != nullptr) {
                    yv = __fadd2_rn(yv, *reinterpret_cast<const float2*>(g.bias0 + c));
                    gv = __fadd2_rn(gv, *reinterpret_cast<const float2*>(g.bias0 + 128 + c));
                  }
                  const float2 sg = sigmoid2(gv);
                  if constexpr (EPI == EPI_GATE_OUT) {
                    const float2 r = __fmul2_rn(yv, sg);
                    r0[e] = r.x; r0[e + 1] = r.y;
                  } else {
                    const float2 dy = __fmul2_rn(d[i], sg);
                    const float2 oms = __ffma2_rn(sg, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f));
                    const float2 dg = __fmul2_rn(__fmul2_rn(dy, yv), oms);
                    r0[e] = dy.x; r0[e + 1] = dy.y;
                    r1[e] = dg.x; r1[e + 1] = dg.y;
                  }
                }
              }
              // 16 channels of this pixel: one 32-byte store for 16-bit outputs (two where the tensors start between).  fp32: four lanes exchange their pieces, so that a request covers 64 bytes of eight rows and not 16 of 32
              if constexpr (sizeof(TOUT) == 2) {
                if (m < g.M) {
                  TOUT* at = o0 + j * 32 + hf * 16;
                  TOUT* at1 = o1 + j * 32 + hf * 16;
                  if (g.wide) {
                    store16<TOUT>(at, r0);
                    if constexpr (EPI == EPI_GATE_OUT_BWD) store16<TOUT>(at1, r1);
                  } else {
                    store8<TOUT>(at, r0);
                    store8<TOUT>(at + 8, r0 + 8);
                    if constexpr (EPI == EPI_GATE_OUT_BWD) { store8<TOUT>(at1, r1); store8<TOUT>(at1 + 8, r1 + 8); }
                  }
                }
              } else {
                store_rows4(reinterpret_cast<float*>(g.out0), r0, m, g.M, j * 32 + hf * 16, lane);
                if constexpr (EPI == EPI_GATE_OUT_BWD) store_rows4(reinterpret_cast<float*>(g.out1), r1, m, g.M, j * 32 + hf * 16, lane);
              }
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
// One GEMM operand: a rank-3 tensor (inner, outer, batch); inner is contiguous.  K-major: inner = K,
// outer = rows (M or N).  MN-major: inner = rows, outer = K.
struct Operand {
  const void* ptr = nullptr;
  bool mn_major = false;
  uint64_t inner = 0, outer = 0, batch = 1;
  uint64_t st_outer = 0, st_batch = 0;  // elements
};

struct GemmPlan {
  Operand a[2], b[2];
  int M = 0, N = 0;
  int K0 = 0, K1 = 0;        // K extent per segment (per split when split_k)
  int seg1_col = 0;
  int batches = 1;
  int split_k = 0;
  int a_tiles = 0;           // > 0: A's batch dimension enumerates this many 128-row M tiles (gate-in GEMMs)
  void* out0 = nullptr;
  void* out1 = nullptr;
  long long ld_out = 0, batch_out = 0;
  const float* bias0 = nullptr;
  const void* aux = nullptr;
  const void* aux2 = nullptr;
  const void* aux3 = nullptr;
  const void *x = nullptr, *gamma = nullptr;   // LN_BWD: x, out0 = dx [M][128]
  const float *mean = nullptr, *rstd = nullptr;
  float *sum_g = nullptr, *sum_b = nullptr;    // [min(tiles, SMs)][128]
  long long plane = 0;
  void* const* peer_out = nullptr;   // GATE_IN: per-rank exchange buffers (see GemmArgs)
  int peer_world = 0, peer_rank = 0, peer_batches = 0;
  bool first = false;                // no kernel of this call came before: launched plainly
  int beside = 0;                    // SMs that the kernel before leaves to this one, which starts beside it
  const char* name = "tc_gemm";
  const char* pair_name = nullptr;   // the timer's name for it on pairs of SMs (null: the same)
  double flops = 0, bytes = 0;
};

// dtype: TRI_F32 (tf32 MMA), TRI_BF16, TRI_F16.  out_f32: EPI_STORE writes fp32 instead of the input dtype.
int launch_gemm(cudaStream_t st, int dtype, int epi, int bn, bool out_f32, const GemmPlan& p, int* err);

// The plain product on pairs of SMs (tc_gemm_pair.cu).  Does it suit, against tiles of 128 x `width`, elements of `es` bytes?  ta, tb: boxes of 128 rows.
bool gemm_pair_fits(const GemmPlan& p, int width, int kblocks, int es);
int launch_gemm_pair(cudaStream_t st, int dtype, const CUtensorMap& ta, const CUtensorMap& tb, const GemmPlan& p, int* err);

}  // namespace tc
}  // namespace tri

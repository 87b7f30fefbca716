// Triangle attention on the tensor cores for fp32 with TF32 products, head dim up to 32 (tcgen05 kind::tf32, TMEM, TMA).
//
// The operands of a product are rounded to TF32 (nearest), as the CUDA-core path does: q, k, v and dO once per call into
// copies in the workspace, P and dS of the backward when they are stored; the forward's P is multiplied as two TF32 terms.
// Everything else is fp32.
//   forward   the row-sharing kernel of tc_attn_rows.cu on the rounded copies
//   dK / dV   one item per (batch, row, head, 128-key block), thread = key: S^T = K Q^T, dP^T = V dO^T per 64-query tile,
//             dV += P^T dO, dK += dS^T Q
//   dQ        one item per 128-query block, thread = query: S = Q K^T, dP = dO V^T per 64-key tile, dQ += dS K
//   dbias     one CTA per (row chunk, batch, head, 64-query block, 128-key block), thread = key, summing dS over its rows
// P and dS replace S and dP in TMEM column by column and are read from there.  The tile that a second product reads across
// its rows is fetched once more: 32-bit operands exist in that form only in the swizzle with 32-byte atoms, which the first
// product cannot read.  dQ is a pass of its own, since dS^T would have to go through shared memory in that form as well.
// Row constants come with the products (TfFactors); the mathematics is that of tc_attn.cu.
//
// What bounds them: the chain of a step (no pipe is above 40 %), and the copies: 100 to 270 MB of rounded operands per direction.
// One training step at N = 256, 4 heads of 32, 785 us on the CUDA cores' path: rounding 34, forward 70, the backward's
// preparation 52, dK / dV 93, dQ 87, dbias 60.  What took the passes there: sums that are stored beside the next item's first step (dK / dV 113 -> 98 us,
// with the copies issued in the order in which their places become free).  Two sets of warps on alternate steps: no difference.
#include <algorithm>
#include <cstdlib>

#include "tc_attn_common.cuh"
#include "tc_attn_rows.cuh"
#include "tc_attn_tf32.cuh"

namespace tri {
namespace tc {

namespace {

constexpr int kTile = 128 * 128, kHalf = 64 * 128;   // bytes of 128 and 64 rows of 32 fp32
constexpr int kThreads = 576;                        // 16 arithmetic warps (four per 32 rows, 16 columns each), MMA, copies
constexpr uint32_t kHiK = desc_hi(1024, 2), kHiMn = desc_hi(512, 1);

// Row constants through the products, as RowFactors in tc_attn.cu: {c1, c2, c3, d1 | d2, d3, 0, 0} of a query, c = -(m + log l) /
// scale and d = -delta in three TF32 terms each, against {1, 1, 1, 0 | 0 ...} of a key for S and {0, 0, 0, 1 | 1, 1, 0, 0} for dP.
// Two planes of 16 bytes per query; rows with |m| > 256 or a value that is not finite are flagged and go without.
struct TfFactors {
  static constexpr int kBlock = 384;          // eight equal rows, read with a row-group stride of 16 bytes
  static constexpr int kBytes = 4 * kBlock;   // S, columns 0-3 | 4-7 | dP, columns 0-3 | 4-7
  static constexpr uint32_t HI_KEY = desc_hi(16, 0), HI_QUERY = desc_hi(128, 0);   // no swizzle
  __device__ static uint32_t key_s(uint32_t at) { return desc_lo(at, kBlock); }
  __device__ static uint32_t key_dp(uint32_t at) { return desc_lo(at + 2 * kBlock, kBlock); }
  __device__ static uint32_t query(uint32_t at, int rows) { return desc_lo(at, rows * 16); }
  __device__ static void fill(uint8_t* key, int tid) {
    if (tid >= kBytes / 16) return;
    const int part = tid / (kBlock / 16);
    reinterpret_cast<float4*>(key)[tid] = part == 0 ? make_float4(1.f, 1.f, 1.f, 0.f) : part == 2 ? make_float4(0.f, 0.f, 0.f, 1.f)
                                        : part == 3 ? make_float4(1.f, 1.f, 0.f, 0.f) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ static bool fits(float m, float c, float d) { return fabsf(m) <= 256.f && fabsf(c) <= 1e30f && fabsf(d) <= 1e30f; }
  __device__ static void pack(float c, float d, float4& lo, float4& hi) {
    lo.x = round_tf32(c); c -= lo.x;
    lo.y = round_tf32(c); c -= lo.y;
    lo.z = round_tf32(c);
    lo.w = round_tf32(d); d -= lo.w;
    hi.x = round_tf32(d); d -= hi.x;
    hi.y = round_tf32(d);
    hi.z = hi.w = 0.f;
  }
};

// ---------------------------------------------------------------------------------------------
// preparation
// ---------------------------------------------------------------------------------------------
struct RoundArgs {
  const float* src[3];
  int64_t st[3][4];     // strides of (batch, row, residue, head)
  float* dst[3];        // [B][S][N][H][D]
  int S, N, H, D;
  unsigned rows;        // B S N H
};
// forward: a row of up to 32 channels by eight lanes; blockIdx.y = tensor
__global__ void __launch_bounds__(256) round_copies_kernel(const RoundArgs a) {
  dependent_trigger();
  const unsigned row = blockIdx.x * 32u + (threadIdx.x >> 3);   // (fewer than 2^31)
  const int c = (threadIdx.x & 7) * 4, t = blockIdx.y;
  if (row >= a.rows || c >= a.D) return;
  unsigned z = row / (unsigned)a.H;
  const unsigned h = row - z * a.H, n = z % (unsigned)a.N;
  z /= (unsigned)a.N;
  const unsigned b = z / (unsigned)a.S, s = z - b * a.S;
  const float4 v = *reinterpret_cast<const float4*>(a.src[t] + b * a.st[t][0] + s * a.st[t][1] + n * a.st[t][2] + h * a.st[t][3] + c);
  *reinterpret_cast<float4*>(a.dst[t] + (long long)row * a.D + c) = make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
}

// backward, in one launch: q, k, v and dO rounded, the row constants as factors and (for flagged rows) as prep = -m | -log l log2e |
// -delta, the key-mask terms (0, -1e9, -inf beyond N; in a second plane times log2(e)), the bias transposed.  A block has a (batch, row,
// head), a warp 32 queries at a time, eight lanes to a row of up to 32 channels; the first blocks transpose a tile of 32 x 32 each.  Bound by
// the bytes: N = 256, 4 heads of 32, 52 us, 48 by the copy rate (with three blocks an SM its
// registers spill: 68), as four kernels 35 + 26 + 3 + 4 and their gaps.
struct PrepareArgs {
  const float *q, *k, *v, *o, *d_o, *stats, *bias;
  float *q_r, *k_r, *v_r, *d_o_r;   // [B][S][N][H][D]
  float* bias_t;
  float4* aug;          // [2][B][S][H][npad]
  float* prep;          // [3][B][S][H][npad]
  float* mask_terms;    // [2][B][S][npad]
  int* large;           // [B][S][H]
  int* err;             // cleared
  const uint8_t* mask;
  int npad, pitch, tiles, transposes;   // tiles of a side of the bias; blocks that transpose
};
__global__ void __launch_bounds__(256, 2) prepare_bwd_kernel(const TriAttnDesc d, const PrepareArgs a) {
  __shared__ float tile[32][33];
  dependent_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = d.n_res;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.err[0] = a.err[1] = 0;
  if ((int)blockIdx.x < a.transposes) {
    unsigned z = blockIdx.x;
    const int k0 = (int)(z % (unsigned)a.tiles) * 32; z /= (unsigned)a.tiles;
    const int q0 = (int)(z % (unsigned)a.tiles) * 32, bh = (int)(z / (unsigned)a.tiles);
    const float* src = a.bias + bh / d.H * d.bias_st[0] + bh % d.H * d.bias_st[1];
    float* dst = a.bias_t + (int64_t)bh * N * a.pitch;
    for (int i = warp; i < 32; i += 8)
      if (q0 + i < N && k0 + lane < N) tile[i][lane] = src[(q0 + i) * d.bias_st[2] + k0 + lane];
    __syncthreads();
    for (int i = warp; i < 32; i += 8)
      if (k0 + i < N && q0 + lane < N) dst[(int64_t)(k0 + i) * a.pitch + q0 + lane] = tile[lane][i];
    return;
  }
  const unsigned row = blockIdx.x - a.transposes, bs = row / (unsigned)d.H, h = row - bs * (unsigned)d.H;
  const unsigned b = bs / (unsigned)d.n_seq, s = bs - b * (unsigned)d.n_seq;
  const long long planes = (long long)d.B * d.n_seq, plane = planes * d.H * a.npad, total = planes * d.H * N;
  if (h == 0) {
    for (int k = threadIdx.x; k < a.npad; k += 256) {
      const float v = mask_term(a.mask != nullptr && k < N ? a.mask[b * d.mask_st[0] + s * d.mask_st[1] + k] : 1u, k < N);
      a.mask_terms[(long long)bs * a.npad + k] = v;
      a.mask_terms[(planes + bs) * a.npad + k] = v * kLog2e;
    }
  }
  const bool on = (lane & 7) * 4 < d.D;
  const int ch = on ? (lane & 7) * 4 : 0;
  const float *qb = a.q + b * d.q_st[0] + s * d.q_st[1] + h * d.q_st[3] + ch, *kb = a.k + b * d.k_st[0] + s * d.k_st[1] + h * d.k_st[3] + ch,
              *vb = a.v + b * d.v_st[0] + s * d.v_st[1] + h * d.v_st[3] + ch, *ob = a.o + b * d.o_st[0] + s * d.o_st[1] + h * d.o_st[3] + ch,
              *gb = a.d_o + b * d.do_st[0] + s * d.do_st[1] + h * d.do_st[3] + ch;
  int flag = 0;
  for (int n0 = warp * 32; n0 < a.npad; n0 += 256) {
    const int i = n0 + lane;   // this lane's query once the sums are there
    const long long at = (long long)row * a.npad + i;
    const bool in = i < N;
    const float m = in ? a.stats[(long long)row * N + i] : 0.f, ll = in ? a.stats[total + (long long)row * N + i] : 0.f;
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      float4 x[2][5];
      float part[2] = {0.f, 0.f};
      bool live[2];
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const int n = n0 + (e + f) * 4 + (lane >> 3);
        live[f] = on && n < N;
        const int64_t r = live[f] ? n : 0;   // (a row that is there in place of one that is not: the loads need no branch)
        x[f][0] = *reinterpret_cast<const float4*>(ob + r * d.o_st[2]);
        x[f][1] = *reinterpret_cast<const float4*>(gb + r * d.do_st[2]);
        x[f][2] = *reinterpret_cast<const float4*>(qb + r * d.q_st[2]);
        x[f][3] = *reinterpret_cast<const float4*>(kb + r * d.k_st[2]);
        x[f][4] = *reinterpret_cast<const float4*>(vb + r * d.v_st[2]);
      }
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const int n = n0 + (e + f) * 4 + (lane >> 3);
        if (!live[f]) continue;
        part[f] = fmaf(x[f][0].x, x[f][1].x, fmaf(x[f][0].y, x[f][1].y, fmaf(x[f][0].z, x[f][1].z, x[f][0].w * x[f][1].w)));
        const long long to = (((long long)bs * N + n) * d.H + h) * d.D + ch;
        float* const dst[4] = {a.d_o_r, a.q_r, a.k_r, a.v_r};
#pragma unroll
        for (int w = 0; w < 4; ++w)
          *reinterpret_cast<float4*>(dst[w] + to) = make_float4(round_tf32(x[f][w + 1].x), round_tf32(x[f][w + 1].y), round_tf32(x[f][w + 1].z), round_tf32(x[f][w + 1].w));
      }
      __syncwarp();
#pragma unroll
      for (int f = 0; f < 2; ++f) {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) part[f] += __shfl_xor_sync(0xffffffffu, part[f], o);
        const float v = __shfl_sync(0xffffffffu, part[f], (lane & 3) * 8);
        if (lane >> 2 == e + f) acc = v;
      }
    }
    const float c = in ? -(m + ll) / d.scale : 0.f;
    const bool fits = TfFactors::fits(m, c, acc);
    if (!fits) flag = 1;
    float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
    if (fits) TfFactors::pack(c, -acc, lo, hi);
    a.aug[at] = lo;
    a.aug[plane + at] = hi;
    a.prep[at] = -m;
    a.prep[plane + at] = -ll * kLog2e;
    a.prep[2 * plane + at] = -acc;
  }
  flag = __syncthreads_or(flag);
  if (threadIdx.x == 0) a.large[row] = flag;
}

// the bias in rows of `pitch`
__global__ void copy_bias_kernel(const float* __restrict__ in, int64_t st_b, int64_t st_h, int64_t st_q, int n, int H, int pitch, float* __restrict__ out) {
  dependent_trigger();
  const int bh = blockIdx.z, b = bh / H, h = bh % H;
  const int q = blockIdx.y * 8 + threadIdx.y, k = blockIdx.x * 32 + threadIdx.x;
  if (q < n && k < n) out[((int64_t)bh * n + q) * pitch + k] = in[b * st_b + h * st_h + q * st_q + k];
}

// ---------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------
struct TfBwdArgs {
  int B, S, N, H, D, npad;
  float scale;
  const float4* aug;
  const float* prep;
  const int* large;
  const float* mask_terms;     // [2][B][S][npad]: natural, times log2(e)
  long long plane, mask_plane; // B S H npad, B S npad
  int bias_b_mul;
  float* out[2];               // dK (dQ), dV; dbias or its row chunks
  int64_t out_st[2][4];
  uint32_t idesc_s, idesc_acc;
  int row_chunks;
  int* err;
};

// what a step's 16 columns of S and dP become: e = S scale log2e + (bias + mask) log2e, P = 2^e, dS = P dP
struct Sixteen { float2 s[8], d[8]; };
__device__ __forceinline__ void load16x2(uint32_t t_s, uint32_t t_d, Sixteen& v) {
  uint32_t a[16], b[16];
  tmem_ld_32x16(t_s, a);
  tmem_ld_32x16(t_d, b);
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]), "+r"(a[8]), "+r"(a[9]), "+r"(a[10]),
                 "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15]), "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]),
                 "+r"(b[5]), "+r"(b[6]), "+r"(b[7]), "+r"(b[8]), "+r"(b[9]), "+r"(b[10]), "+r"(b[11]), "+r"(b[12]), "+r"(b[13]), "+r"(b[14]),
                 "+r"(b[15])::"memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) { v.s[i] = pair(a[2 * i], a[2 * i + 1]); v.d[i] = pair(b[2 * i], b[2 * i + 1]); }
}

// dK / dV (KV) or dQ.  Persistent: a CTA takes items blockIdx.x, blockIdx.x + gridDim.x, ... and treats their tiles of 64 rows as
// one stream c = 0, 1, ...  Shared memory: the item's two stationary tiles (two buffers), per step the two streamed tiles and
// their copies for the second products, the bias tile (two buffers each).
//   in[2]    copies -> MMA            streamed tiles, row constants (an item's first: stationary tiles) of step c
//   late[2]  copies -> MMA            ... the copies for the second products
//   bias[2]  copies -> threads        bias tile, mask terms, statistics of a flagged row
//   s[2]     MMA -> threads, copies   S and dP of step c are in TMEM (and the streamed tiles are free)
//   p[2]     threads -> MMA           ... P and dS have taken their place
//   acc[2]   MMA -> copies, threads   the second products of step c are done
template <bool KV> struct GeoT {
  static constexpr int LATE = (KV ? 2 : 1) * kHalf;           // copies for the second products
  static constexpr int ROWS = KV ? 64 : 128;                  // queries whose constants a step needs
  static constexpr int OFF_A = 0;                             // [2] x two stationary tiles
  static constexpr int OFF_B = OFF_A + 4 * kTile;             // [2] x two streamed tiles
  static constexpr int OFF_L = OFF_B + 4 * kHalf;             // [2]
  static constexpr int OFF_BIAS = OFF_L + 2 * LATE;           // [2] x [128 x 64], two SW128 tiles of 32 columns
  static constexpr int OFF_F = OFF_BIAS + 2 * 32768;          // [2] factors: two planes of ROWS x 16 bytes
  static constexpr int OFF_ST = OFF_F + 2 * ROWS * 32;        // [2] -m, -log l log2e, -delta of ROWS queries
  static constexpr int OFF_M = OFF_ST + 2 * ROWS * 12;        // [2] mask terms: 128 keys (KV) or 64
  static constexpr int OFF_KEY = OFF_M + 2 * 512;
  static constexpr int OFF_BAR = OFF_KEY + TfFactors::kBytes;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
};

template <bool KV, bool HB>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_tf32_kernel(const __grid_constant__ CUtensorMap tmA0, const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB0,
                     const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmL0, const __grid_constant__ CUtensorMap tmL1,
                     const __grid_constant__ CUtensorMap tmBias, const TfBwdArgs a) {
  using G = GeoT<KV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* bar_in = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);
  uint64_t *bar_late = bar_in + 2, *bar_bias = bar_in + 4, *bar_s = bar_in + 6, *bar_p = bar_in + 8, *bar_acc = bar_in + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_in + 12);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blocks = (a.N + 127) / 128, nsteps = (a.N + 63) / 64;
  const long long items = (long long)blocks * a.H * a.S * a.B;
  const int my_items = blockIdx.x < items ? (int)((items - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
  const int total = my_items * nsteps;
  struct Item { int blk, h, s, b; };
  auto item_of = [&](int n) {   // (the item count fits 31 bits)
    unsigned z = blockIdx.x + (unsigned)n * gridDim.x;
    Item it;
    it.blk = (int)(z % (unsigned)blocks); z /= (unsigned)blocks;
    it.h = (int)(z % (unsigned)a.H); z /= (unsigned)a.H;
    it.s = (int)(z % (unsigned)a.S);
    it.b = (int)(z / (unsigned)a.S);
    return it;
  };
  auto row_of = [&](const Item& it) { return ((long long)it.b * a.S + it.s) * a.H + it.h; };
  // the flag of item n, asked for an item ahead of its use (the last one's again beyond it)
  auto flag_of = [&](int n) { return a.large[row_of(item_of(min(n, my_items - 1)))]; };

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_in[i], 1); mbar_init(&bar_late[i], 1); mbar_init(&bar_bias[i], 1); mbar_init(&bar_s[i], 1); mbar_init(&bar_p[i], 16);
      mbar_init(&bar_acc[i], 1);
    }
    mbar_fence_init();
  }
  TfFactors::fill(smem + G::OFF_KEY, tid);
  fence_proxy_async_smem();
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  constexpr uint32_t COL_DP = 64, COL_ACC = 256;   // S / P and dP / dS of even and odd steps at 0 and 128; two sums of 32 columns of
                                                   // even and odd items at 256 and 320
  bool ok = true;

  if (warp == 17) {
    if (lane == 0 && total > 0) {
      // ---------------------------------- copies -------------------------------------------------
      struct Cursor { Item it; int n, j; };
      auto next = [&](Cursor& u) {
        if (++u.j < nsteps) return;
        u.j = 0;
        if (++u.n < my_items) u.it = item_of(u.n);
      };
      Cursor ci{item_of(0), 0, 0}, cb = ci, cl = ci;
      uint32_t flags = flag_of(0) != 0 ? 1u : 0u;   // bit n & 31; ci is ahead of the others by less than an item and three steps
      int flag = flag_of(1);
      auto load_in = [&](int c) {     // (a stationary buffer's last use is two items back, before the step whose S was waited for)
        const Item& it = ci.it;
        if (ci.j == 0 && ci.n > 0) {
          flags = (flags & ~(1u << (ci.n & 31))) | ((flag != 0 ? 1u : 0u) << (ci.n & 31));
          flag = flag_of(ci.n + 1);
        }
        const bool folded = (flags >> (ci.n & 31) & 1u) == 0;
        uint64_t* bar = &bar_in[c & 1];
        uint8_t* dst = smem + G::OFF_B + (c & 1) * 2 * kHalf;
        mbar_expect_tx(bar, 2 * kHalf + (ci.j == 0 ? 2 * kTile : 0) + (folded ? G::ROWS * 32 : 0));
        if (ci.j == 0) {
          uint8_t* st = smem + G::OFF_A + (ci.n & 1) * 2 * kTile;
          tma_load_5d(st, &tmA0, bar, 0, it.h, it.blk * 128, it.s, it.b);
          tma_load_5d(st + kTile, &tmA1, bar, 0, it.h, it.blk * 128, it.s, it.b);
        }
        tma_load_5d(dst, &tmB0, bar, 0, it.h, ci.j * 64, it.s, it.b);
        tma_load_5d(dst + kHalf, &tmB1, bar, 0, it.h, ci.j * 64, it.s, it.b);
        if (folded) {
          const float4* f = a.aug + row_of(it) * a.npad + (KV ? ci.j * 64 : it.blk * 128);
          uint8_t* to = smem + G::OFF_F + (c & 1) * G::ROWS * 32;
          bulk_load(to, f, G::ROWS * 16, bar);
          bulk_load(to + G::ROWS * 16, f + a.plane, G::ROWS * 16, bar);
        }
        next(ci);
      };
      auto load_late = [&](int c) {
        const Item& it = cl.it;
        uint64_t* bar = &bar_late[c & 1];
        uint8_t* dst = smem + G::OFF_L + (c & 1) * G::LATE;
        mbar_expect_tx(bar, G::LATE);
        tma_load_5d(dst, &tmL0, bar, 0, it.h, cl.j * 64, it.s, it.b);
        if (KV) tma_load_5d(dst + kHalf, &tmL1, bar, 0, it.h, cl.j * 64, it.s, it.b);
        next(cl);
      };
      auto load_bias = [&](int c) {
        const Item& it = cb.it;
        const bool folded = (flags >> (cb.n & 31) & 1u) == 0;
        uint64_t* bb = &bar_bias[c & 1];
        mbar_expect_tx(bb, (HB ? 32768 : 0) + (KV ? 512 : 256) + (folded ? 0 : G::ROWS * 12));
        if (HB) {   // KV: the transposed copy, keys x queries; else queries x keys
          uint8_t* to = smem + G::OFF_BIAS + (c & 1) * 32768;
          for (int e = 0; e < 2; ++e) tma_load_4d(to + e * 16384, &tmBias, bb, cb.j * 64 + e * 32, it.blk * 128, it.h, it.b * a.bias_b_mul);
        }
        const float* m = a.mask_terms + (folded ? a.mask_plane : 0) + ((long long)it.b * a.S + it.s) * a.npad;
        bulk_load(smem + G::OFF_M + (c & 1) * 512, m + (KV ? it.blk * 128 : cb.j * 64), KV ? 512 : 256, bb);
        if (!folded) {
          const float* p = a.prep + row_of(it) * a.npad + (KV ? cb.j * 64 : it.blk * 128);
          for (int e = 0; e < 3; ++e) bulk_load(smem + G::OFF_ST + ((c & 1) * 3 + e) * G::ROWS * 4, p + e * a.plane, G::ROWS * 4, bb);
        }
        next(cb);
      };
      for (int c = 0; c < 2 && c < total; ++c) { load_in(c); load_bias(c); load_late(c); }
      // in the order of the events: S(c + 1), P and dS(c), the second products of c
      for (int c = -1; c + 2 < total && ok; ++c) {
        if (c + 3 < total) {
          ok = mbar_wait(&bar_s[(c + 1) & 1], ((c + 1) >> 1) & 1, a.err, 71) && ok;   // its streamed tiles are free
          load_in(c + 3);
        }
        if (c < 0) continue;
        ok = mbar_wait(&bar_p[c & 1], (c >> 1) & 1, a.err, 79) && ok;     // every warp has read its bias
        load_bias(c + 2);
        ok = mbar_wait(&bar_acc[c & 1], (c >> 1) & 1, a.err, 72) && ok;   // its copies are free
        load_late(c + 2);
      }
    }
  } else if (warp == 16) {
    // ------------------------------------ products (the whole warp runs this, one lane issues) ----------
    const bool leader = elect_one();
    const uint32_t a_lo = desc_lo(smem_u32(smem + G::OFF_A), 16), b_lo = desc_lo(smem_u32(smem + G::OFF_B), 16), l_lo = desc_lo(smem_u32(smem + G::OFF_L), kHalf);
    const uint32_t key_s = TfFactors::key_s(smem_u32(smem + G::OFF_KEY)), key_dp = TfFactors::key_dp(smem_u32(smem + G::OFF_KEY));
    const uint32_t f_lo = TfFactors::query(smem_u32(smem + G::OFF_F), G::ROWS);
    int sc = 0, sj = 0, sn = 0;       // step, tile and item of the next scores
    bool folded = total > 0 && flag_of(0) == 0;
    int flag = total > 0 ? flag_of(1) : 0;
    auto issue_scores = [&]() {
      ok = mbar_wait(&bar_in[sc & 1], (sc >> 1) & 1, a.err, 73) && ok;
      tc_fence_after_sync();
      if (leader) {
        const uint32_t t = tmem_base + (sc & 1) * 128, A = a_lo + (sn & 1) * (2 * kTile >> 4), B = b_lo + (sc & 1) * (2 * kHalf >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          umma<KIND_TF32>(t, desc_join(A + ks * 2, kHiK), desc_join(B + ks * 2, kHiK), a.idesc_s, ks > 0);
          umma<KIND_TF32>(t + COL_DP, desc_join(A + (kTile >> 4) + ks * 2, kHiK), desc_join(B + (kHalf >> 4) + ks * 2, kHiK), a.idesc_s, ks > 0);
        }
        if (folded) {
          const uint64_t rows = desc_join(f_lo + (sc & 1) * (G::ROWS * 32 >> 4), TfFactors::HI_QUERY);
          const uint64_t ones = desc_join(key_s, TfFactors::HI_KEY), dones = desc_join(key_dp, TfFactors::HI_KEY);
          umma<KIND_TF32>(t, KV ? ones : rows, KV ? rows : ones, a.idesc_s, 1);
          umma<KIND_TF32>(t + COL_DP, KV ? dones : rows, KV ? rows : dones, a.idesc_s, 1);
        }
        umma_commit(&bar_s[sc & 1]);
      }
      ++sc;
      if (++sj == nsteps) {
        sj = 0;
        ++sn;
        folded = flag == 0;
        flag = flag_of(sn + 1);
      }
    };
    for (int c = 0; c < 2 && c < total; ++c) issue_scores();
    int j = 0, n = 0;
    for (int c = 0; c < total && ok; ++c) {
      ok = mbar_wait(&bar_late[c & 1], (c >> 1) & 1, a.err, 74) && ok;
      ok = mbar_wait(&bar_p[c & 1], (c >> 1) & 1, a.err, 75) && ok;
      tc_fence_after_sync();
      if (leader) {
        const uint32_t t = tmem_base + (c & 1) * 128, acc = tmem_base + COL_ACC + (n & 1) * 64, L = l_lo + (c & 1) * (G::LATE >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          // dK += dS^T Q, dQ += dS K; dV += P^T dO
          umma_ts<KIND_TF32>(acc, t + COL_DP + kk * 8, desc_join(L + kk * 64, kHiMn), a.idesc_acc, j > 0 || kk > 0);
          if (KV) umma_ts<KIND_TF32>(acc + 32, t + kk * 8, desc_join(L + (kHalf >> 4) + kk * 64, kHiMn), a.idesc_acc, j > 0 || kk > 0);
        }
        umma_commit(&bar_acc[c & 1]);
      }
      if (sc < total) issue_scores();    // into the columns that these products read: products of one thread run in order
      if (++j == nsteps) { j = 0; ++n; }
    }
  } else {
    // ------------------------------------ arithmetic: row r of the block, 16 columns -------------------
    const int r = (warp & 3) * 32 + lane, cg = warp >> 2;
    const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    const float2 sc2 = splat(a.scale), l2e2 = splat(kLog2e), scl2 = splat(a.scale * kLog2e);
    const uint32_t bias_a = smem_u32(smem + G::OFF_BIAS) + (cg >> 1) * 16384 + r * 128, chunk0 = (cg & 1) * 4, sw = r & 7;
    // An item's sums, once the products of its last step cl are done; the next item's go to other columns, and the one after
    // that starts when this thread has arrived for a step of the next.
    auto finish = [&](int n, int cl) {
      ok = mbar_wait(&bar_acc[cl & 1], (cl >> 1) & 1, a.err, 78) && ok;
      tc_fence_after_sync();
      const int which = cg >> 1, col = (cg & 1) * 16;     // dK (dQ) or dV, 16 of its channels
      if (KV || which == 0) {
        const Item it = item_of(n);
        uint32_t o[16];
        tmem_ld_32x16(t_row + COL_ACC + (n & 1) * 64 + which * 32 + col, o);
        tmem_ld_wait();
        const int x = it.blk * 128 + r;
        if (x < a.N && ok) {
          const float f = which == 0 ? a.scale : 1.f;
          float* dst = a.out[which] + it.b * a.out_st[which][0] + it.s * a.out_st[which][1] + x * a.out_st[which][2] + it.h * a.out_st[which][3] + col;
#pragma unroll
          for (int g = 0; g < 4; ++g)
            if (col + g * 4 < a.D)
              reinterpret_cast<float4*>(dst)[g] = make_float4(__uint_as_float(o[4 * g]) * f, __uint_as_float(o[4 * g + 1]) * f,
                                                              __uint_as_float(o[4 * g + 2]) * f, __uint_as_float(o[4 * g + 3]) * f);
        }
      }
    };
    int c = 0, flag = total > 0 ? flag_of(0) : 0;
    for (int n = 0; n < my_items && __all_sync(0xffffffffu, ok); ++n) {
      const bool folded = flag == 0;
      flag = flag_of(n + 1);
      for (int j = 0; j < nsteps; ++j, ++c) {
        ok = mbar_wait(&bar_bias[c & 1], (c >> 1) & 1, a.err, 76) && ok;
        ok = mbar_wait(&bar_s[c & 1], (c >> 1) & 1, a.err, 77) && ok;
        tc_fence_after_sync();
        const uint32_t t_s = t_row + (c & 1) * 128 + cg * 16;
        const uint32_t ba = bias_a + (c & 1) * 32768, ma = smem_u32(smem + G::OFF_M) + (c & 1) * 512 + (KV ? r * 4 : cg * 64);
        const uint32_t sa = smem_u32(smem + G::OFF_ST) + (c & 1) * G::ROWS * 12;
        Sixteen v;
        load16x2(t_s, t_s + COL_DP, v);
        uint32_t pw[16], dw[16];
        float mk1 = 0.f;
        if constexpr (KV) mk1 = lds32f(ma);
#pragma unroll
        for (int u = 0; u < 4; ++u) {    // four columns
          float4 bs = make_float4(0.f, 0.f, 0.f, 0.f);
          if constexpr (HB) bs = lds128f(ba + (((chunk0 + u) ^ sw) << 4));
          const float4 mk = KV ? make_float4(mk1, mk1, mk1, mk1) : lds128f(ma + u * 16);
          const float2 b2[2] = {make_float2(bs.x, bs.y), make_float2(bs.z, bs.w)}, m2[2] = {make_float2(mk.x, mk.y), make_float2(mk.z, mk.w)};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int k = u * 2 + i;
            float2 e, d = v.d[k];
            if (folded) {
              e = __ffma2_rn(v.s[k], scl2, __ffma2_rn(b2[i], l2e2, m2[i]));
            } else {
              // statistics per query: this thread's own, or its columns'
              auto stat = [&](int p) {
                const uint32_t at = sa + p * G::ROWS * 4;
                return KV ? make_float2(lds32f(at + (cg * 16 + 2 * k) * 4), lds32f(at + (cg * 16 + 2 * k + 1) * 4)) : splat(lds32f(at + r * 4));
              };
              const float2 x = __fadd2_rn(__ffma2_rn(v.s[k], sc2, m2[i]), b2[i]);
              e = __ffma2_rn(__fadd2_rn(x, stat(0)), l2e2, stat(1));
              d = __fadd2_rn(d, stat(2));
            }
            const float2 p = make_float2(ex2_approx(e.x), ex2_approx(e.y)), ds = __fmul2_rn(p, d);
            if constexpr (KV) { pw[2 * k] = __float_as_uint(round_tf32(p.x)); pw[2 * k + 1] = __float_as_uint(round_tf32(p.y)); }
            dw[2 * k] = __float_as_uint(round_tf32(ds.x)); dw[2 * k + 1] = __float_as_uint(round_tf32(ds.y));
          }
        }
        if constexpr (KV) tmem_st_32x16(t_s, pw);
        tmem_st_32x16(t_s + COL_DP, dw);
        fence_proxy_async_smem();   // (bias, mask terms and statistics have been read: copies write the next ones over them)
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p[c & 1]);
        if (!ok) break;
        if (j == 0 && n > 0) finish(n - 1, c - 1);   // the item before, beside this step's products
      }
      if (!ok) break;
    }
    if (my_items > 0 && ok) finish(my_items - 1, c - 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// dbias: as the 16-bit pass.  The bias of a thread's key and 16 queries and their sums stay in registers.
struct GeoTB {
  static constexpr int NS = 3;                              // row stages
  static constexpr int OFF_F = 2 * kTile + 2 * kHalf;       // factors of 64 queries
  static constexpr int OFF_ST = OFF_F + 2048;               // statistics
  static constexpr int OFF_M = OFF_ST + 768;                // 128 mask terms
  static constexpr int STAGE = 53248;                       // (52 KB: tiles stay 1024-byte aligned)
  static constexpr int OFF_KEY = NS * STAGE;
  static constexpr int OFF_BAR = OFF_KEY + TfFactors::kBytes;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
};
static_assert(GeoTB::OFF_M + 512 <= GeoTB::STAGE, "a stage's parts fit");

__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_dbias_tf32_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                           const __grid_constant__ CUtensorMap tmDO, const float* bias_t, int pitch, const TfBwdArgs a) {
  using G = GeoTB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* bar_in = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);   // [NS]
  uint64_t *bar_s = bar_in + 3, *bar_free = bar_in + 5;                // [2], [4]: row j arrives on bar_free[j & 3]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_in + 9);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qblocks = (a.N + 63) / 64, kblocks = (a.N + 127) / 128;
  unsigned z = blockIdx.x;
  const int k0 = (int)(z % (unsigned)kblocks) * 128; z /= (unsigned)kblocks;
  const int q0 = (int)(z % (unsigned)qblocks) * 64; z /= (unsigned)qblocks;
  const int h = (int)(z % (unsigned)a.H); z /= (unsigned)a.H;
  const int b = (int)(z % (unsigned)a.B), rc = (int)(z / (unsigned)a.B);
  const int per = (a.S + a.row_chunks - 1) / a.row_chunks, s_lo = rc * per, nsteps = max(0, min(a.S, s_lo + per) - s_lo);

  if (tid == 0) {
    for (int i = 0; i < G::NS; ++i) mbar_init(&bar_in[i], 1);
    mbar_init(&bar_s[0], 1); mbar_init(&bar_s[1], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_free[i], 16);
    mbar_fence_init();
  }
  TfFactors::fill(smem + G::OFF_KEY, tid);
  fence_proxy_async_smem();
  if (warp == 0) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  bool ok = true;
  const int* large = a.large + ((long long)b * a.S + s_lo) * a.H + h;   // flags of the rows, H apart

  if (warp == 17) {
    if (lane == 0) {
      auto load_step = [&](int step) {
        const int stg = step % G::NS, s = s_lo + step;
        const long long row0 = (((long long)b * a.S + s) * a.H + h) * (long long)a.npad + q0;
        const bool folded = large[(long long)step * a.H] == 0;
        uint8_t* st = smem + stg * G::STAGE;
        uint64_t* bar = &bar_in[stg];
        mbar_expect_tx(bar, 2 * kTile + 2 * kHalf + (folded ? 2048 : 768) + 512);
        tma_load_5d(st, &tmK, bar, 0, h, k0, s, b);
        tma_load_5d(st + kTile, &tmV, bar, 0, h, k0, s, b);
        tma_load_5d(st + 2 * kTile, &tmQ, bar, 0, h, q0, s, b);
        tma_load_5d(st + 2 * kTile + kHalf, &tmDO, bar, 0, h, q0, s, b);
        if (folded) {
          for (int e = 0; e < 2; ++e) bulk_load(st + G::OFF_F + e * 1024, a.aug + e * a.plane + row0, 1024, bar);
        } else {
          for (int e = 0; e < 3; ++e) bulk_load(st + G::OFF_ST + e * 256, a.prep + e * a.plane + row0, 256, bar);
        }
        bulk_load(st + G::OFF_M, a.mask_terms + (folded ? a.mask_plane : 0) + ((long long)b * a.S + s) * a.npad + k0, 512, bar);
      };
      for (int st = 0; st < G::NS && st < nsteps; ++st) load_step(st);
      for (int j = 0; j + G::NS < nsteps && ok; ++j) {
        ok = mbar_wait(&bar_free[j & 3], (j >> 2) & 1, a.err, 81) && ok;
        load_step(j + G::NS);
      }
    }
  } else if (warp == 16) {
    const bool leader = elect_one();
    const uint32_t base_lo = desc_lo(smem_u32(smem), 16);
    const uint32_t key_s = TfFactors::key_s(smem_u32(smem + G::OFF_KEY)), key_dp = TfFactors::key_dp(smem_u32(smem + G::OFF_KEY));
    const uint32_t f_lo = TfFactors::query(smem_u32(smem + G::OFF_F), 64);
    int flag = nsteps > 0 ? large[0] : 0;
    for (int j = 0; j < nsteps && ok; ++j) {
      const int stg = j % G::NS;
      const bool folded = flag == 0;
      if (j + 1 < nsteps) flag = large[(long long)(j + 1) * a.H];
      if (j >= 2) ok = mbar_wait(&bar_free[(j - 2) & 3], ((j - 2) >> 2) & 1, a.err, 82) && ok;   // TMEM buffer is free
      ok = mbar_wait(&bar_in[stg], (j / G::NS) & 1, a.err, 83) && ok;
      tc_fence_after_sync();
      if (leader) {
        const uint32_t t = tmem_base + (j & 1) * 128, K = base_lo + stg * (G::STAGE >> 4), V = K + (kTile >> 4), Q = V + (kTile >> 4), O = Q + (kHalf >> 4);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma<KIND_TF32>(t, desc_join(K + ks * 2, kHiK), desc_join(Q + ks * 2, kHiK), a.idesc_s, ks > 0);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma<KIND_TF32>(t + 64, desc_join(V + ks * 2, kHiK), desc_join(O + ks * 2, kHiK), a.idesc_s, ks > 0);
        if (folded) {
          const uint64_t rows = desc_join(f_lo + stg * (G::STAGE >> 4), TfFactors::HI_QUERY);
          umma<KIND_TF32>(t, desc_join(key_s, TfFactors::HI_KEY), rows, a.idesc_s, 1);
          umma<KIND_TF32>(t + 64, desc_join(key_dp, TfFactors::HI_KEY), rows, a.idesc_s, 1);
        }
        umma_commit(&bar_s[j & 1]);
      }
    }
  } else {
    const int r = (warp & 3) * 32 + lane, cg = warp >> 2, kj = k0 + r, qc = q0 + cg * 16;
    const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + cg * 16;
    const float2 sc2 = splat(a.scale), l2e2 = splat(kLog2e), scl2 = splat(a.scale * kLog2e);
    float2 acc[8] = {}, bias[8];
    {   // (rows of the transposed copy are whole 16-byte pieces; what lies beyond N is not used)
      const float* src = bias_t + (((long long)b * a.bias_b_mul * a.H + h) * a.N + min(kj, a.N - 1)) * pitch;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (qc + g * 4 < a.N) v = *reinterpret_cast<const float4*>(src + qc + g * 4);
        bias[2 * g] = make_float2(v.x, v.y);
        bias[2 * g + 1] = make_float2(v.z, v.w);
      }
    }
    int flag = nsteps > 0 ? large[0] : 0;
    for (int j = 0; j < nsteps; ++j) {
      const int stg = j % G::NS;
      const bool folded = flag == 0;
      if (j + 1 < nsteps) flag = large[(long long)(j + 1) * a.H];
      ok = mbar_wait(&bar_in[stg], (j / G::NS) & 1, a.err, 83) && ok;
      ok = mbar_wait(&bar_s[j & 1], (j >> 1) & 1, a.err, 84) && ok;
      tc_fence_after_sync();
      const uint32_t at = smem_u32(smem) + stg * G::STAGE;
      const float2 mk = splat(lds32f(at + G::OFF_M + r * 4));
      Sixteen v;
      load16x2(t_row + (j & 1) * 128, t_row + (j & 1) * 128 + 64, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (folded) {
          const float2 e = __ffma2_rn(v.s[k], scl2, __ffma2_rn(bias[k], l2e2, mk));
          acc[k] = __ffma2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), v.d[k], acc[k]);
        } else {
          auto stat = [&](int p) {
            const uint32_t x = at + G::OFF_ST + p * 256 + (cg * 16 + 2 * k) * 4;
            return make_float2(lds32f(x), lds32f(x + 4));
          };
          const float2 x = __fadd2_rn(__ffma2_rn(v.s[k], sc2, mk), bias[k]);
          const float2 e = __ffma2_rn(__fadd2_rn(x, stat(0)), l2e2, stat(1));
          acc[k] = __fadd2_rn(acc[k], __fmul2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), __fadd2_rn(v.d[k], stat(2))));
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_free[j & 3]);
      if (!ok) break;
    }
    if (kj < a.N && ok) {   // a query at a time: lanes are consecutive keys
      float* to = a.out[0] + (long long)rc * a.B * a.H * a.N * a.N + (((long long)b * a.H + h) * a.N + qc) * a.N + kj;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if (qc + i < a.N) to[(long long)i * a.N] = i & 1 ? acc[i >> 1].y : acc[i >> 1].x;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
int pitch_of(const TriAttnDesc* d) { return (d->n_res + 3) / 4 * 4; }
int batches_of(const TriAttnDesc* d) { return d->bias_st[0] != 0 ? d->B : 1; }
size_t tensor_floats(const TriAttnDesc* d) { return (size_t)d->B * d->n_seq * d->n_res * d->H * d->D; }
size_t bias_floats(const TriAttnDesc* d) { return (size_t)batches_of(d) * d->H * d->n_res * pitch_of(d); }
int npad_of(const TriAttnDesc* d) { return (d->n_res + 127) / 128 * 128; }
bool bias_strides_fit(const TriAttnDesc* d) {
  return d->bias_st[0] % 4 == 0 && d->bias_st[1] % 4 == 0 && d->bias_st[2] % 4 == 0 && (d->bias_st[1] != 0 || d->H == 1) && d->bias_st[2] != 0;
}
bool own_bias(const TriAttnDesc* d, const void* bias) { return reinterpret_cast<uintptr_t>(bias) % 16 == 0 && bias_strides_fit(d); }

struct TfWs {
  int* err;
  float *q, *k, *v, *d_o, *bias, *bias_t, *mask, *prep, *part;
  float4* aug;
  int* large;
};
// bias_copy: the bias is not read in place
void carve(Arena& a, const TriAttnDesc* d, int is_bwd, bool bias_copy, TfWs* w) {
  const size_t t = tensor_floats(d), rows = (size_t)d->B * d->n_seq * d->H, np = npad_of(d);
  w->err = a.take<int>(64);
  w->q = a.take<float>(t); w->k = a.take<float>(t); w->v = a.take<float>(t);
  w->bias = a.take<float>(bias_copy ? bias_floats(d) : 0);
  w->mask = a.take<float>((is_bwd ? 2 : wants_mask_terms(d) ? 1 : 0) * (size_t)d->B * d->n_seq * np);
  if (!is_bwd) return;
  w->d_o = a.take<float>(t);
  w->bias_t = a.take<float>(bias_floats(d));
  w->prep = a.take<float>(3 * rows * np);
  w->aug = a.take<float4>(2 * rows * np);
  w->large = a.take<int>(rows);
  w->part = a.take<float>(dbias_partial_bytes(d, sm_count()) / sizeof(float));
}

// boxes of `rows` residues of a rounded copy; `across` for a product that reads it across its rows
int copy_map(CUtensorMap* out, const float* p, const TriAttnDesc* d, int rows, bool across) {
  const uint64_t D = d->D, H = d->H, N = d->n_res, S = d->n_seq;
  const uint64_t dims[5] = {D, H, N, S, (uint64_t)d->B}, str[4] = {D, H * D, N * H * D, S * N * H * D};
  const uint32_t box[5] = {32, 1, (uint32_t)rows, 1, 1};
  return make_tmap(out, p, TRI_F32, 5, dims, str, box, across ? 32 : 128);
}
int bias_tile_map(CUtensorMap* out, const void* p, const TriAttnDesc* d, bool own) {
  const uint64_t N = d->n_res, H = d->H, nb = batches_of(d), pitch = pitch_of(d);
  const uint64_t dims[4] = {N, N, H, nb};
  const uint64_t mine[3] = {(uint64_t)d->bias_st[2], (uint64_t)d->bias_st[1], (uint64_t)d->bias_st[0]}, packed[3] = {pitch, pitch * N, nb > 1 ? pitch * N * H : 0};
  const uint32_t box[4] = {32, 128, 1, 1};
  return make_tmap(out, p, TRI_F32, 4, dims, own ? mine : packed, box, 128);
}
int copy_bias(const TriAttnDesc* d, const void* bias, float* out, cudaStream_t st) {
  copy_bias_kernel<<<dim3(cdiv(d->n_res, 32), cdiv(d->n_res, 8), batches_of(d) * d->H), dim3(32, 8), 0, st>>>(
      static_cast<const float*>(bias), d->bias_st[0], d->bias_st[1], d->bias_st[2], d->n_res, d->H, pitch_of(d), out);
  TRI_LAUNCH_OK();
  return 0;
}

}  // namespace

// Logits from which on TF32 calls come here: below, the rounded copies and the row constants cost more than the CUDA-core path
// (mma.sync) as a whole.  Inference, us there / here: 4 heads of 128, 144, 160, 256 residues (8.4, 12, 16, 67 M) 31 / 29, 51 / 47,
// 63 / 56, 131 / 102; 8 heads of 128, 144 (17, 24 M) 43 / 49, 100 / 86.  Training (both sides on one path): 4 heads of 101, 112,
// 128, 256 (4.1, 5.6, 8.4, 67 M) 115 / 139, 154 / 131, 174 / 132, 785 / 410; 1 head of 176, 200 (5.5, 8 M) 127 / 157, 162 / 157.
constexpr double kMinForward = 2e7, kMinBackward = 5e6;

bool attn_tf32_supported(const TriAttnDesc* d, int is_bwd) {
  const char* forced = getenv("TRI_B200_FORCE_SIMT");
  if (d->dtype != TRI_F32 || d->precision != TRI_PREC_TF32 || (forced != nullptr && forced[0] == '1')) return false;
  if (d->D % 4 != 0 || d->D > 32 || d->n_res <= 64 || d->n_res > 16384 || d->n_seq < 2 || d->n_seq > 65535) return false;
  if ((double)d->B * d->n_seq * d->H * d->n_res * d->n_res < (is_bwd ? kMinBackward : kMinForward)) return false;
  const int64_t* st[8] = {d->q_st, d->k_st, d->v_st, d->o_st, d->do_st, d->dq_st, d->dk_st, d->dv_st};
  for (int i = 0; i < (is_bwd ? 8 : 4); ++i)
    for (int e = 0; e < 4; ++e)
      if (st[i][e] % 4 != 0) return false;
  if ((long long)batches_of(d) * d->H > 65535 || (long long)d->B * d->n_seq * d->H * npad_of(d) >= (1LL << 31)) return false;
  return attn_fwd_rows_fits(d);
}

static size_t ws_bytes(const TriAttnDesc* d, int is_bwd, bool bias_copy) {
  Arena a(nullptr, 0);
  TfWs w;
  carve(a, d, is_bwd, bias_copy, &w);
  return a.off;
}
// (The descriptor does not say where the bias starts: a copy for that reason alone is not counted here.)
size_t attn_tf32_ws_bytes(const TriAttnDesc* d, int is_bwd) { return ws_bytes(d, is_bwd, !bias_strides_fit(d)); }
bool attn_tf32_has_room(const TriAttnDesc* d, const void* bias, size_t ws_size, int is_bwd) {
  return ws_size >= ws_bytes(d, is_bwd, !bias_strides_fit(d) || (bias != nullptr && !own_bias(d, bias)));
}

int attn_tf32_forward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, void* o, float* stats,
                      void* ws, size_t ws_size, cudaStream_t st) {
  Arena ar(ws, ws_size);
  TfWs w;
  carve(ar, d, 0, bias != nullptr && !own_bias(d, bias), &w);
  if (ws == nullptr || !ar.ok()) return fail(TRI_ERR_WORKSPACE, "attention forward workspace too small");
  {
    RoundArgs r;
    const void* src[3] = {q, k, v};
    const int64_t* strides[3] = {d->q_st, d->k_st, d->v_st};
    float* dst[3] = {w.q, w.k, w.v};
    for (int i = 0; i < 3; ++i) {
      r.src[i] = static_cast<const float*>(src[i]);
      r.dst[i] = dst[i];
      for (int e = 0; e < 4; ++e) r.st[i][e] = strides[i][e];
    }
    r.S = d->n_seq; r.N = d->n_res; r.H = d->H; r.D = d->D;
    r.rows = (unsigned)d->B * d->n_seq * d->n_res * d->H;
    KernelTimer kt("tc_attn_round", st, 0.0, 24.0 * tensor_floats(d));
    round_copies_kernel<<<dim3(cdiv(r.rows, 32), 3), 256, 0, st>>>(r);
    TRI_LAUNCH_OK();
  }
  const bool terms = wants_mask_terms(d);
  if (terms) TRI_TRY(launch_mask_terms(d, mask, w.mask, w.err, st));
  CUtensorMap tq, tk, tv, tb;
  TRI_TRY(copy_map(&tq, w.q, d, 128, false));
  TRI_TRY(copy_map(&tk, w.k, d, 64, false));
  TRI_TRY(copy_map(&tv, w.v, d, 64, true));
  if (bias != nullptr) {
    const bool own = own_bias(d, bias);
    if (!own) TRI_TRY(copy_bias(d, bias, w.bias, st));
    TRI_TRY(bias_tile_map(&tb, own ? bias : w.bias, d, own));
  }
  return attn_fwd_rows(d, tq, tk, tv, bias ? &tb : nullptr, d->bias_st[0] != 0, mask, terms ? w.mask : nullptr, o, stats, w.err, false, st);
}

int attn_tf32_backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias, const uint8_t* mask, const void* o,
                       const float* stats, const void* d_o, void* dq, void* dk, void* dv, float* dbias, void* ws, size_t ws_size, cudaStream_t st) {
  Arena ar(ws, ws_size);
  TfWs w;
  carve(ar, d, 1, bias != nullptr && !own_bias(d, bias), &w);
  if (ws == nullptr || !ar.ok()) return fail(TRI_ERR_WORKSPACE, "attention backward workspace too small");
  const int npad = npad_of(d), blocks = npad / 128, nq = cdiv(d->n_res, 64);
  const double pairs = (double)d->B * d->n_seq * d->H * d->n_res * (double)d->n_res, tensor = 4.0 * tensor_floats(d);
  {
    PrepareArgs p;
    p.q = static_cast<const float*>(q); p.k = static_cast<const float*>(k); p.v = static_cast<const float*>(v);
    p.o = static_cast<const float*>(o); p.d_o = static_cast<const float*>(d_o); p.stats = stats; p.bias = static_cast<const float*>(bias);
    p.q_r = w.q; p.k_r = w.k; p.v_r = w.v; p.d_o_r = w.d_o; p.bias_t = w.bias_t; p.aug = w.aug; p.prep = w.prep; p.mask_terms = w.mask;
    p.large = w.large; p.err = w.err; p.mask = mask; p.npad = npad; p.pitch = pitch_of(d);
    p.tiles = cdiv(d->n_res, 32);
    p.transposes = bias != nullptr ? p.tiles * p.tiles * batches_of(d) * d->H : 0;
    const long long planes = (long long)d->B * d->n_seq;
    KernelTimer kt("tc_attn_delta", st, 0.0, 9.0 * tensor);
    prepare_bwd_kernel<<<(unsigned)(p.transposes + planes * d->H), 256, 0, st>>>(*d, p);
    TRI_LAUNCH_OK();
  }
  TfBwdArgs a;
  a.B = d->B; a.S = d->n_seq; a.N = d->n_res; a.H = d->H; a.D = d->D; a.npad = npad; a.scale = d->scale;
  a.aug = w.aug; a.prep = w.prep; a.large = w.large; a.mask_terms = w.mask;
  a.plane = (long long)d->B * d->n_seq * d->H * npad; a.mask_plane = (long long)d->B * d->n_seq * npad;
  a.bias_b_mul = d->bias_st[0] != 0 ? 1 : 0; a.row_chunks = 1; a.err = w.err;
  a.idesc_s = make_idesc(KIND_TF32, 128, 64, false, false);
  a.idesc_acc = make_idesc(KIND_TF32, 128, 32, false, true);
  const long long items = (long long)blocks * d->B * d->n_seq * d->H;
  const unsigned grid = (unsigned)std::min<long long>(items, sm_count());
  CUtensorMap a0, a1, b0, b1, l0, l1, tb;
  // ---- dK, dV: stationary K, V; streamed Q, dO -------------------------------------------------
  if (bias != nullptr) {
    TRI_TRY(bias_tile_map(&tb, w.bias_t, d, false));
  }
  TRI_TRY(copy_map(&a0, w.k, d, 128, false)); TRI_TRY(copy_map(&a1, w.v, d, 128, false));
  TRI_TRY(copy_map(&b0, w.q, d, 64, false)); TRI_TRY(copy_map(&b1, w.d_o, d, 64, false));
  TRI_TRY(copy_map(&l0, w.q, d, 64, true)); TRI_TRY(copy_map(&l1, w.d_o, d, 64, true));
  const CUtensorMap tk = a0, tv = a1, tq = b0, tdo = b1;
  if (bias == nullptr) tb = a0;
  a.out[0] = static_cast<float*>(dk); a.out[1] = static_cast<float*>(dv);
  for (int i = 0; i < 4; ++i) { a.out_st[0][i] = d->dk_st[i]; a.out_st[1][i] = d->dv_st[i]; }
  {
    auto kern = bias ? attn_bwd_tf32_kernel<true, true> : attn_bwd_tf32_kernel<true, false>;
    TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GeoT<true>::SMEM));
    KernelTimer kt("tc_attn_bwd_dkdv", st, 8.0 * pairs * d->D, 6.0 * tensor);
    launch_dependent(us_of_logits(pairs), kern, grid, kThreads, GeoT<true>::SMEM, st, a0, a1, b0, b1, l0, l1, tb, a);
    TRI_LAUNCH_OK();
  }
  // ---- dQ: stationary Q, dO; streamed K, V ------------------------------------------------------
  if (bias != nullptr) {
    const bool own = own_bias(d, bias);
    if (!own) TRI_TRY(copy_bias(d, bias, w.bias, st));
    TRI_TRY(bias_tile_map(&tb, own ? bias : w.bias, d, own));
  }
  TRI_TRY(copy_map(&a0, w.q, d, 128, false)); TRI_TRY(copy_map(&a1, w.d_o, d, 128, false));
  TRI_TRY(copy_map(&b0, w.k, d, 64, false)); TRI_TRY(copy_map(&b1, w.v, d, 64, false));
  TRI_TRY(copy_map(&l0, w.k, d, 64, true));
  a.out[0] = static_cast<float*>(dq);
  for (int i = 0; i < 4; ++i) a.out_st[0][i] = d->dq_st[i];
  {
    auto kern = bias ? attn_bwd_tf32_kernel<false, true> : attn_bwd_tf32_kernel<false, false>;
    TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GeoT<false>::SMEM));
    KernelTimer kt("tc_attn_bwd_dq", st, 6.0 * pairs * d->D, 5.0 * tensor);
    launch_dependent(us_of_logits(pairs), kern, grid, kThreads, GeoT<false>::SMEM, st, a0, a1, b0, b1, l0, l0, tb, a);
    TRI_LAUNCH_OK();
  }
  // ---- dbias ------------------------------------------------------------------------------------
  if (dbias != nullptr) {
    const long long combos = (long long)blocks * nq * d->B * d->H;
    const int chunks = dbias_row_chunks(d, sm_count());
    const long long n = (long long)d->B * d->H * d->n_res * d->n_res;
    a.row_chunks = chunks;
    a.out[0] = chunks > 1 ? w.part : dbias;
    TRI_CUDA_OK(cudaFuncSetAttribute(attn_bwd_dbias_tf32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GeoTB::SMEM));
    KernelTimer kt("tc_attn_bwd_dbias", st, 0.0, 4.0 * tensor);
    launch_dependent(us_of_logits(pairs), attn_bwd_dbias_tf32_kernel, (unsigned)(combos * chunks), kThreads, GeoTB::SMEM, st, tk, tv, tq, tdo, w.bias_t, pitch_of(d), a);
    TRI_LAUNCH_OK();
    if (chunks > 1) TRI_TRY(launch_sum_partials(w.part, chunks, n, dbias, st));
  }
  return 0;
}

}  // namespace tc
}  // namespace tri

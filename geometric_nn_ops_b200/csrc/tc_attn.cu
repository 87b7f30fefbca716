// Tensor-core triangle attention (tcgen05 + TMEM + TMA), bf16 / fp16, head dim up to 64 (tiles of 32 or 64 channels).
//
// All four kernels share one shape: 320 threads, of which warps 0-7 do the elementwise arithmetic (two threads per
// tile row, each owning half of the tile's columns), warp 8 issues every tcgen05.mma and warp 9 every TMA / bulk
// copy.  The three sides meet only on mbarriers, so the serial issue code never sits between the arithmetic warps'
// steps, and score products for the next tile are issued as soon as the accumulators have been read into registers.
// The arithmetic is packed fp32x2 (fma.rn.f32x2 and friends); row constants of the backward come as
// extra channels of the products (RowFactors), and additive key-mask terms (0, -1e9, -inf beyond N) from a small array
// prepared once per call (the forward's copy warp makes them on the way).  With head dim 32 the probabilities (forward) and dS / P^T / dS^T (backward) never touch
// shared memory: they are stored packed into TMEM and read from there as the A operand of the next product, which
// halves the shared-memory traffic that otherwise bounds these kernels.
//
// Forward (head dim up to 32 and three rows or more: tc_attn_rows.cu), per (batch, row, head, 128-query block), per 128-key
// tile:
//   S = Q K^T (TMEM) -> x = scale*S + mask + bias -> running maximum -> P = 2^((x - m) log2e) -> O_half += P V.
//   Each half of the key tile keeps its own maximum, sum and O accumulator (merged at the end); O stays in TMEM
//   and is rescaled only when a maximum grows by more than 8 ln 2.
// Backward: deterministic passes, two with head dim 32 and three otherwise, each recomputing P from the saved statistics (see below).
// Semantics follow triangle_attention_torch (geometric_nn_ops_torch/triangle/_reference/triangle_attention.py:28-44):
// bias and the finite -1e9 key-mask sentinel are added in fp32; keys beyond N_res get -inf.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "tc_attn_common.cuh"
#include "tc_attn_rows.cuh"
#include "tc_attn_tf32.cuh"
#include "tc_paths.cuh"

namespace tri {
namespace tc {

namespace {

struct AttnArgs {
  int B, S, N, H, D;
  float scale;
  void* o;
  int64_t o_st[4];
  float* stats;          // [2][B][S][H][N]: row max, log row sum
  const uint8_t* mask;   // [B][S][N] key masks, or null
  int64_t mask_st[2];
  int bias_b_mul;        // 0 when the bias is broadcast over the batch
  uint32_t idesc_s, idesc_pv;
  int* status;
};

template <int HD> struct Geo {
  static constexpr int RB = HD * 2;                      // bytes per tile row (16-bit elements)
  static constexpr int TILE = 128 * RB;                  // one [128 x HD] tile
  static constexpr uint32_t LAYOUT = RB == 128 ? 2 : 4;  // SWIZZLE_128B or SWIZZLE_64B
  static constexpr uint32_t SBO = 8 * RB;                // 8-row group
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_K = OFF_Q + TILE;             // [2]
  static constexpr int OFF_V = OFF_K + 2 * TILE;         // [2]
  static constexpr int OFF_P = OFF_V + 2 * TILE;         // [2] x [128 x 128] (two SW128 blocks of 64 keys): the bias tile
                                                         // arrives here and each thread overwrites it with its P values
  static constexpr int OFF_MB = OFF_P + 2 * 32768;       // [2] x 128 additive key-mask terms
  static constexpr int OFF_X = OFF_MB + 1024;            // [128][2] floats exchanged when the key halves are merged
  static constexpr int OFF_BAR = OFF_X + 1024;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;      // + alignment slack
};

__global__ void __launch_bounds__(256) mask_terms_kernel(const uint8_t* __restrict__ mask, int64_t st_b, int64_t st_s, int B, int S, int N, int npad,
                                                         float* __restrict__ out, int* err) {
  dependent_trigger();
  const long long idx = blockIdx.x * 256LL + threadIdx.x;
  if (idx == 0) err[0] = err[1] = 0;
  if (idx >= (long long)B * S * npad) return;
  const int k = (int)(idx % npad);
  const long long bs = idx / npad, b = bs / S, s = bs - b * S;
  out[idx] = mask_term(mask != nullptr && k < N ? mask[b * st_b + s * st_s + k] : 1u, k < N);
}

// 320 threads.  Warps 0-7 do the softmax arithmetic: thread (r, hh) owns query row r and the 64-key half hh of each
// 128-key tile, with its own running maximum and sum and its own output accumulator O_hh in TMEM; the halves are
// merged once at the end.  Warp 8 issues the MMAs, warp 9 the TMA copies.  The sides meet on mbarriers:
//   bar_s    MMA -> threads      S = Q K^T of a tile is in TMEM
//   bar_free threads -> MMA, TMA every warp has its logits in registers (next tile's S and K may follow)
//   bar_p    threads -> MMA      P of the tile is in shared memory and O has its final scale (P V may start)
//   bar_pv   MMA -> TMA, threads P V is done: its V stage and P buffer are free and O is current
// The bias tile of step j lands in buffer j & 1 and each thread overwrites its own part with P, so P is double
// buffered at no cost and the threads never wait for P V except to rescale O.
// O stays in TMEM across tiles.  It is rescaled only when a row's maximum grows by more than kRescale, so the
// stored maximum may be stale by up to that much: P <= e^kRescale = 256, and the row sum uses the same maximum.
constexpr float kRescale = 5.545177444f;   // 8 ln 2

template <typename T, int HD, bool HB>
__global__ void __launch_bounds__(320, 2)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmBias,
                   const AttnArgs a) {
  using G = Geo<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem + G::OFF_Q;
  uint8_t* sK = smem + G::OFF_K;
  uint8_t* sV = smem + G::OFF_V;
  uint8_t* sP = smem + G::OFF_P;
  float* sMb = reinterpret_cast<float*>(smem + G::OFF_MB);
  float* sX = reinterpret_cast<float*>(smem + G::OFF_X);   // [128][2]: maximum and sum of key half 1, for the merge
  uint64_t* bar_q = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);
  uint64_t* bar_k = bar_q + 1;      // [2] K tile + mask terms
  uint64_t* bar_v = bar_q + 3;      // [2]
  uint64_t* bar_bias = bar_q + 5;   // [2]
  uint64_t* bar_s = bar_q + 7;
  uint64_t* bar_pv = bar_q + 8;     // [2]: tile c commits to bar_pv[c & 1]
  uint64_t* bar_free = bar_q + 10;  // [4]: tile c arrives on bar_free[c & 3] (the copy warp may lag the threads by up to
                                    // two tiles, so two tiles that share a barrier are never both pending)
  uint64_t* bar_p = bar_q + 14;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_q + 15);
  int* const err = reinterpret_cast<int*>(tmem_slot + 1);   // this CTA's (see leave_status)

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid & 127, hh = (tid >> 7) & 1;
  const int qblocks = (a.N + 127) / 128;
  const int nt = (a.N + 127) / 128;
  // Persistent: this CTA takes work items blockIdx.x, blockIdx.x + gridDim.x, ... (an item = one (batch, row, head,
  // 128-query block)) and treats their key tiles as one stream c = 0, 1, ...: the copy warp runs two tiles ahead
  // across item boundaries, and TMEM, barriers and the pipeline survive from one item to the next.
  const long long items = (long long)qblocks * a.H * a.S * a.B;
  const int my_items = blockIdx.x < items ? (int)((items - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
  const int total = my_items * nt;
  struct Item { int q0, h, s, b; };
  auto item_of = [&](int n) {   // (the item count fits 31 bits: 32-bit divisions)
    unsigned z = blockIdx.x + (unsigned)n * gridDim.x;
    Item it;
    it.q0 = (int)(z % (unsigned)qblocks) * 128; z /= (unsigned)qblocks;
    it.h = (int)(z % (unsigned)a.H); z /= (unsigned)a.H;
    it.s = (int)(z % (unsigned)a.S);
    it.b = (int)(z / (unsigned)a.S);
    return it;
  };

  if (tid == 0) {
    mbar_init(bar_q, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&bar_k[i], 1); mbar_init(&bar_v[i], 1); mbar_init(&bar_bias[i], 1); mbar_init(&bar_pv[i], 1); }
    mbar_init(bar_s, 1); mbar_init(bar_p, 8);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_free[i], 8);
    mbar_fence_init();
    *err = 0;
  }
  if (warp == 0) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  constexpr uint32_t COL_O = 128;   // O_0 at [128, 128 + HD), O_1 at [128 + HD, 128 + 2 HD)
  // With head dim 32 the 256 TMEM columns have room for P itself (two 16-bit values per column) and P V reads it
  // from there, which halves the step's shared-memory traffic.  P is single buffered then: a tile's values are
  // stored once the previous tile's P V is done.
  constexpr bool TMEM_P = HD == 32;
  constexpr uint32_t COL_P = 192;
  bool ok = true;

  if (warp == 9) {
    // ---------------------------------- TMA copies, mask terms -----------------------------------
    // The warp runs together, and gives up together: a lane writes the terms of four keys of a tile, lane 0 issues the copies.
    auto load_q = [&](int n) {
      if (lane != 0) return;
      const Item it = item_of(n);
      mbar_expect_tx(bar_q, G::TILE);
      tma_load_5d(sQ, &tmQ, bar_q, 0, it.h, it.q0, it.s, it.b);
    };
    uint32_t kept[4];
    auto fetch_mask = [&](const Item& it, int t) {   // of key tile t, in time for its load_k
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = t * 128 + lane * 4 + e;
        kept[e] = a.mask != nullptr && k < a.N ? a.mask[it.b * a.mask_st[0] + it.s * a.mask_st[1] + k] : 1u;
      }
    };
    // tile c of the stream: item `it`, key tile t of that item
    auto load_k = [&](int c, const Item& it, int t) {
      const int stg = c & 1, k = t * 128 + lane * 4;
      reinterpret_cast<float4*>(sMb + stg * 128)[lane] = make_float4(mask_term(kept[0], k < a.N), mask_term(kept[1], k + 1 < a.N),
                                                                     mask_term(kept[2], k + 2 < a.N), mask_term(kept[3], k + 3 < a.N));
      __syncwarp();
      if (lane != 0) return;
      mbar_expect_tx(&bar_k[stg], G::TILE);
      tma_load_5d(sK + stg * G::TILE, &tmK, &bar_k[stg], 0, it.h, t * 128, it.s, it.b);
    };
    auto load_v = [&](int c, const Item& it, int t) {
      if (lane != 0) return;
      const int stg = c & 1;
      mbar_expect_tx(&bar_v[stg], G::TILE);
      tma_load_5d(sV + stg * G::TILE, &tmV, &bar_v[stg], 0, it.h, t * 128, it.s, it.b);
    };
    auto load_bias = [&](int c, const Item& it, int t) {
      if (lane != 0) return;
      uint64_t* bb = &bar_bias[c & 1];
      uint8_t* dst = sP + (c & 1) * 32768;
      mbar_expect_tx(bb, 32768);
      tma_load_4d(dst, &tmBias, bb, t * 128, it.q0, it.h, it.b * a.bias_b_mul);
      tma_load_4d(dst + 16384, &tmBias, bb, t * 128 + 64, it.q0, it.h, it.b * a.bias_b_mul);
    };
    // (la_n, la_t): item and key tile of the stream position being loaded, two tiles ahead of the consumers
    int la_n = 0, la_t = 0;
    Item la = item_of(0);
    auto advance = [&]() {
      if (++la_t == nt) { la_t = 0; ++la_n; if (la_n < my_items) la = item_of(la_n); }
    };
    if (total > 0) load_q(0);
    for (int c = 0; c < 2 && c < total; ++c) {
      fetch_mask(la, la_t);
      load_k(c, la, la_t);
      if (HB) load_bias(c, la, la_t);
      load_v(c, la, la_t);
      advance();
    }
    int jt = 0, n_cur = 0;   // key tile and item of stream position c
    for (int c = 0; c < total && ok; ++c) {
      if (c + 2 < total) fetch_mask(la, la_t);
      ok = __all_sync(0xffffffffu, mbar_wait(&bar_free[c & 3], (c >> 2) & 1, err, 16));   // S(c) has been read: its K stage and mask terms are free
      if (++jt == nt) {                                    // ... and it was the item's last use of Q
        jt = 0;
        if (++n_cur < my_items) load_q(n_cur);
      }
      if (c + 2 < total) {
        load_k(c + 2, la, la_t);
        if (HB && TMEM_P) load_bias(c + 2, la, la_t);      // the bias tile has been read too and P does not replace it
        ok = __all_sync(0xffffffffu, mbar_wait(&bar_pv[c & 1], (c >> 1) & 1, err, 15)) && ok;   // P V(c) done: its V stage and P buffer are free
        if (HB && !TMEM_P) load_bias(c + 2, la, la_t);
        load_v(c + 2, la, la_t);
        advance();
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      // ---------------------------------- MMA issue ----------------------------------------------
      constexpr uint32_t HI_KMAJ = desc_hi(G::SBO, G::LAYOUT);
      constexpr uint32_t HI_P = desc_hi(1024, 2);
      const uint32_t q_lo = desc_lo(smem_u32(sQ), 16), k_lo = desc_lo(smem_u32(sK), 16);
      const uint32_t p_lo = desc_lo(smem_u32(sP), 16), vmn_lo = desc_lo(smem_u32(sV), 128 * G::RB);   // V as [n = d, k = key]
      int s_t = 0, s_n = 0;   // key tile and item of the next S product
      auto issue_s = [&](int c) {
        if (s_t == 0) ok = mbar_wait(bar_q, s_n & 1, err, 11) && ok;   // first tile of an item: its Q
        if (++s_t == nt) { s_t = 0; ++s_n; }
        ok = mbar_wait(&bar_k[c & 1], (c >> 1) & 1, err, 12) && ok;
        tc_fence_after_sync();
        const uint32_t so = (c & 1) * (G::TILE >> 4);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma<KIND_F16>(tmem_base, desc_join(q_lo + ks * 2, HI_KMAJ), desc_join(k_lo + so + ks * 2, HI_KMAJ), a.idesc_s, ks > 0);
        umma_commit(bar_s);
      };
      if (total > 0) issue_s(0);
      int j = 0;
      for (int c = 0; c < total && ok; ++c, j = (j + 1 == nt ? 0 : j + 1)) {
        const int stg = c & 1;
        ok = mbar_wait(&bar_free[c & 3], (c >> 2) & 1, err, 16) && ok;   // logits of tile c are in registers
        if (c + 1 < total) issue_s(c + 1);
        ok = mbar_wait(bar_p, c & 1, err, 17) && ok;
        ok = mbar_wait(&bar_v[stg], (c >> 1) & 1, err, 18) && ok;
        tc_fence_after_sync();
        const uint32_t so = stg * (G::TILE >> 4), po = stg * (32768 >> 4);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {   // O_half += P[:, half] V[half]: keys 64 * (kk >> 2) + 16 * (kk & 3) ...
          const uint64_t vd = desc_join(vmn_lo + so + kk * G::RB, HI_KMAJ);
          const uint32_t accf = (j > 0 || (kk & 3) > 0) ? 1u : 0u;
          if constexpr (TMEM_P) umma_ts<KIND_F16>(tmem_base + COL_O + (kk >> 2) * HD, tmem_base + COL_P + kk * 8, vd, a.idesc_pv, accf);
          else umma<KIND_F16>(tmem_base + COL_O + (kk >> 2) * HD, desc_join(p_lo + po + (kk >> 2) * 1024 + (kk & 3) * 2, HI_P), vd, a.idesc_pv, accf);
        }
        umma_commit(&bar_pv[stg]);
      }
    }
  } else {
    // ------------------------------------ softmax warps ------------------------------------------
    const float2 sc2 = splat(a.scale), l2e2 = splat(kLog2e);
    const uint32_t t_o = t_row + COL_O + hh * HD;   // this thread's output accumulator row
    for (int n = 0; n < my_items; ++n) {
      const Item it = item_of(n);
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < nt; ++j) {
        const int c = n * nt + j, stg = c & 1;
        ok = mbar_wait(bar_s, c & 1, err, 13) && ok;
        tc_fence_after_sync();
        ok = mbar_wait(&bar_k[stg], (c >> 1) & 1, err, 12) && ok;   // the tile's mask terms
        if (HB) ok = mbar_wait(&bar_bias[stg], (c >> 1) & 1, err, 14) && ok;
        const uint32_t sPj = smem_u32(sP) + stg * 32768;   // holds the bias tile; with P in shared memory, P when this step is done

        // ---- logits of this thread's 64 keys into registers, their maximum ----------------------------
        float2 x2[32];
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // independent chains
        const uint32_t mb_a = smem_u32(sMb) + stg * 512 + hh * 256;
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          uint32_t rr[32];
          tmem_ld_32x32(t_row + hh * 64 + cc * 32, rr);
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            uint4 raw = make_uint4(0, 0, 0, 0);
            if constexpr (HB) raw = lds128(sPj + sw128_chunk(r, hh * 8 + cc * 4 + u));
            const uint32_t bw[4] = {raw.x, raw.y, raw.z, raw.w};
            const float4 mA = lds128f(mb_a + (cc * 8 + u * 2) * 16), mB = lds128f(mb_a + (cc * 8 + u * 2 + 1) * 16);
            const float2 mk[4] = {make_float2(mA.x, mA.y), make_float2(mA.z, mA.w), make_float2(mB.x, mB.y),
                                  make_float2(mB.z, mB.w)};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float2 v = __ffma2_rn(pair(rr[u * 8 + 2 * i], rr[u * 8 + 2 * i + 1]), sc2, mk[i]);
              if constexpr (HB) v = add_wide<T>(v, bw[i]);   // (head dim 64, 512 x 512 residues, 4 heads: 505 -> 501 us)
              x2[cc * 16 + u * 4 + i] = v;
              mx4[i] = fmax3(mx4[i], v.x, v.y);
            }
          }
        }
        fence_proxy_async_smem();   // the bias tile and mask terms have been read: TMA writes the next ones over them
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_free[c & 3]);

        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        const bool grow = mx > m_run + kRescale;          // (always true on the first tile with a key in range)
        const float m_new = grow ? mx : m_run;
        if (j > 0 && __any_sync(0xffffffffu, grow)) {     // tcgen05.ld / st are warp-wide: rows that keep their maximum scale by 1
          ok = mbar_wait(&bar_pv[(c - 1) & 1], ((c - 1) >> 1) & 1, err, 15) && ok;   // O is current
          tc_fence_after_sync();
          const float alpha = grow ? ex2_approx((m_run - m_new) * kLog2e) : 1.0f;   // m_run = -inf gives 0 (O_hh is 0 then)
          l_run *= alpha;
#pragma unroll
          for (int cc = 0; cc < HD / 16; ++cc) {
            uint32_t o[16];
            tmem_ld_32x16(t_o + cc * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st_32x16(t_o + cc * 16, o);
          }
          tmem_st_wait();
        }
        m_run = m_new;

        // ---- P = 2^((x - m) log2e), its row sum; P rounded to the input dtype -----------------------------
        const float2 nm2 = splat(m_new == -INFINITY ? 0.f : -m_new);   // a half with no key in range yet: P = 2^-inf = 0
        float2 ps2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t pw[32];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 e = __fmul2_rn(__fadd2_rn(x2[g * 4 + i], nm2), l2e2);
            const float2 pp = make_float2(ex2_approx(e.x), ex2_approx(e.y));
            ps2[i & 1] = __fadd2_rn(ps2[i & 1], pp);
            pw[g * 4 + i] = pack2<T>(pp.x, pp.y);
          }
          if constexpr (!TMEM_P)
            sts128(sPj + sw128_chunk(r, hh * 8 + g), pw[g * 4], pw[g * 4 + 1], pw[g * 4 + 2], pw[g * 4 + 3]);
        }
        l_run += (ps2[0].x + ps2[0].y) + (ps2[1].x + ps2[1].y);
        if constexpr (TMEM_P) {
          if (c > 0) ok = mbar_wait(&bar_pv[(c - 1) & 1], ((c - 1) >> 1) & 1, err, 15) && ok;   // the previous P has been read
          tc_fence_after_sync();
#pragma unroll
          for (int cc = 0; cc < 2; ++cc) {   // this thread's query row, its 64 keys as 32 packed columns
            uint32_t w[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = pw[cc * 16 + i];
            tmem_st_32x16(t_row + COL_P + hh * 32 + cc * 16, w);
          }
          tmem_st_wait();
        } else {
          fence_proxy_async_smem();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p);
        if (!ok) break;
      }
      if (!ok) break;

      // ---- merge the two key halves of each row and write O, the row maximum and log row sum -------------
      // Both halves' accumulators sit in this row's TMEM lane; only the maximum and sum of half 1 cross threads.
      // The next item's first P V, which overwrites O, is issued only after every warp has arrived on bar_p
      // for that tile, hence after this.
      const int cl = n * nt + nt - 1;
      ok = mbar_wait(&bar_pv[cl & 1], (cl >> 1) & 1, err, 15) && ok;
      tc_fence_after_sync();
      if (hh == 1) { sX[2 * r] = m_run; sX[2 * r + 1] = l_run; }
      named_barrier(1, 256);
      if (hh == 0) {
        const float m1 = sX[2 * r], l1 = sX[2 * r + 1];
        const float m = fmaxf(m_run, m1);   // finite: key 0 is in range and belongs to half 0
        const float a0 = ex2_approx((m_run - m) * kLog2e), a1 = ex2_approx((m1 - m) * kLog2e);
        const float l = l_run * a0 + l1 * a1;
        const float inv = 1.0f / l, w0 = a0 * inv, w1 = a1 * inv;
        const int qi = it.q0 + r;
        const bool st_ok = qi < a.N && ok;
        T* orow = reinterpret_cast<T*>(a.o) + it.b * a.o_st[0] + it.s * a.o_st[1] + qi * a.o_st[2] + it.h * a.o_st[3];
#pragma unroll
        for (int cc = 0; cc < HD / 16; ++cc) {   // tcgen05.ld is warp-wide: every row loads, valid rows store
          uint32_t o0[16], o1[16];
          tmem_ld_32x16(t_row + COL_O + cc * 16, o0);
          tmem_ld_32x16(t_row + COL_O + HD + cc * 16, o1);
          tmem_ld_wait();
          if (st_ok) {
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              float f[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(o0[g * 8 + i]) * w0 + __uint_as_float(o1[g * 8 + i]) * w1;
              uint4 pk;
              pk.x = pack2<T>(f[0], f[1]); pk.y = pack2<T>(f[2], f[3]);
              pk.z = pack2<T>(f[4], f[5]); pk.w = pack2<T>(f[6], f[7]);
              if (cc * 16 + g * 8 < a.D) reinterpret_cast<uint4*>(orow)[cc * 2 + g] = pk;
            }
          }
        }
        if (st_ok) {
          const long long srow = (((long long)it.b * a.S + it.s) * a.H + it.h) * a.N + qi;
          a.stats[srow] = m;
          a.stats[(long long)a.B * a.S * a.H * a.N + srow] = logf(l);
        }
      }
      tc_fence_before_sync();   // orders this item's TMEM reads before the arrivals that let the next item overwrite O
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
  if (tid == 0) leave_status(a.status, err);
}

// =================================================================================================
// Backward.  Deterministic passes, each recomputing P from the saved statistics (with head dim 32 the first gives dQ too):
//   dK/dV : one CTA per (b, row, head, 128-key block), thread = key.  Per 64-query tile:
//           S^T = K Q^T and dP^T = V dO^T (TMEM), P^T and dS^T packed (TMEM or smem), dV += P^T dO, dK += dS^T Q.
//           The bias is read from a transposed copy so that a thread's queries are contiguous.
//   dQ    : one CTA per (b, row, head, 128-query block), thread = query.  Per 64-key tile:
//           S = Q K^T, dP = dO V^T, dS packed into TMEM, dQ += dS K.
//   dbias : one CTA per (row chunk, b, head, 64-query block, 128-key block) looping over its rows in order and
//           summing dS in registers (no atomics: fixed order), S / dP double buffered in TMEM.
// P = exp((x - m) - log l), dS = P * (dP - delta), delta = sum_d dO*O (attn_prepare_kernel).
// =================================================================================================
struct AttnBwdArgs {
  int B, S, N, H, D;
  float scale;
  const float* stats;    // [2][B][S][H][N]
  const float* delta;    // [B][S][H][N]
  const float* prep;     // [3][B][S][H][npad]: -m, -log l * log2e, -delta, zero in the padding
  long long prep_plane;  // B*S*H*npad
  int npad;              // N rounded up to 128
  const float* mask_terms;   // [2][B][S][npad] additive key-mask terms (0, -1e9, or -inf beyond N); the same times log2(e)
  long long mask_plane;      // B*S*npad
  const uint4* aug;          // [B][S][H][npad] row constants as eight 16-bit factors (see RowFactors)
  const int* large;          // [B][S][H] whether a query of the row goes without them
  const uint8_t* mask;
  int64_t mask_st[2];
  int bias_b_mul;        // 0 when the bias is broadcast over the batch
  void* out0;            // dq (MODE_DQ), dk (dK/dV kernel), dbias fp32 (MODE_DBIAS)
  void* out1;            // dv
  int64_t out0_st[4], out1_st[4];
  uint32_t idesc_a, idesc_b;   // the two MMA shapes of the kernel
  uint32_t idesc_c;            // merged dK/dV + dQ pass: the dQ product (both operands MN-major)
  void* dq_part;               // merged pass: per key block, dS K of that block: [key blocks][B][S][N][H][D] in the input dtype
  long long dq_part_plane;     // elements per key block
  int row_chunks;              // MODE_DBIAS: the row loop is split into this many CTAs, each writing its own partial
  int* err;
};

// Row constants through the products.  With c = -(m + log l) / scale and -delta of a query as further channels of Q and dO,
// against ones for every key, S and dP arrive as (x - m - log l) / scale without bias and mask, and as dP - delta: a logit
// then takes two packed instructions up to the exponential, and no statistics are read beside it.  (As fp32 vectors in shared
// memory they were six of the seven loads of eight logits in the dK/dV pass, and it followed the load pipe: 66 % at N = 768.)
// A factor pair carries 24 bits: three 16-bit terms whose products with the key side's constants add up to the value.
//   query: {c1, c2, c3, d1, d2, d3, 0, 0}     key, for S: {1, 1, 1, 0 ...}     for dP: {0, 0, 0, k1, k2, k3, 0, 0}
// bf16 has fp32's range: k = 1.  fp16 takes delta in steps of 2^-48 up to 31: k = 2^-11, 2^-22, 2^-24.
// A product of 16 channels reads two 16-byte columns per row; the second one of the key side is zero, and the second one of
// the query side is the next eight rows' first (128 bytes of zeros follow the last).
// Rows (batch, row, head) in which a query has |m| > 256, or a value out of range, are flagged, and their CTAs (dbias: steps)
// take differences in natural units instead, as the forward does where logits are large.
struct RowFactors {
  static constexpr int kBlock = 384;            // one 8-row block of equal rows, read with a row-group stride of 16 bytes
  static constexpr int kBytes = 3 * kBlock;     // for S | for dP | zeros
  static constexpr uint32_t HI_KEY = desc_hi(16, 0), HI_QUERY = desc_hi(128, 0);   // no swizzle
  __device__ static uint32_t key_s(uint32_t at) { return desc_lo(at, 2 * kBlock); }
  __device__ static uint32_t key_dp(uint32_t at) { return desc_lo(at + kBlock, kBlock); }
  __device__ static uint32_t query(uint32_t at) { return desc_lo(at, 128); }
  template <typename T> __device__ static void fill(uint8_t* key, int tid) {   // kBytes / 16 threads
    if (tid >= kBytes / 16) return;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (tid < kBlock / 16) { v.x = pack2<T>(1.f, 1.f); v.y = pack2<T>(1.f, 0.f); }
    else if (tid < 2 * kBlock / 16) {
      constexpr bool bf = ElemIsBf16<T>::value;
      v.y = pack2<T>(0.f, bf ? 1.f : 0x1p-11f);
      v.z = pack2<T>(bf ? 1.f : 0x1p-22f, bf ? 1.f : 0x1p-24f);
    }
    reinterpret_cast<uint4*>(key)[tid] = v;
  }
  // the terms of v for factors 1 / s1, 1 / s2, 1 / s3 (powers of two)
  template <typename T> __device__ static void split(float v, float s1, float s2, float s3, float (&t)[3]) {
    t[0] = to_f32(from_f32<T>(v * s1));
    v -= t[0] / s1;
    t[1] = to_f32(from_f32<T>(v * s2));
    v -= t[1] / s2;
    t[2] = to_f32(from_f32<T>(v * s3));
  }
  template <typename T> __device__ static bool fits(float m, float c, float d) {
    constexpr bool bf = ElemIsBf16<T>::value;
    return fabsf(m) <= 256.f && fabsf(c) <= (bf ? 1e30f : 6e4f) && fabsf(d) <= (bf ? 1e30f : 31.f);
  }
  template <typename T> __device__ static uint4 pack(float c, float d) {
    constexpr bool bf = ElemIsBf16<T>::value;
    float a[3], b[3];
    split<T>(c, 1.f, 1.f, 1.f, a);
    split<T>(d, bf ? 1.f : 0x1p11f, bf ? 1.f : 0x1p22f, bf ? 1.f : 0x1p24f, b);
    return make_uint4(pack2<T>(a[0], a[1]), pack2<T>(a[2], b[0]), pack2<T>(b[1], b[2]), 0u);
  }
};

template <int HD> struct GeoC {
  static constexpr int RB = HD * 2;
  static constexpr int TK = 128 * RB;   // K / V tile
  static constexpr int TQ = 64 * RB;    // Q / dO tile
  static constexpr uint32_t LAYOUT = RB == 128 ? 2 : 4;
  static constexpr uint32_t SBO = 8 * RB;
  static constexpr int NQ = 3;                      // query-tile stages: tiles are fetched two steps ahead
  static constexpr int ST = 64 * 16 + 128;          // one stage of row constants: factors of 64 queries and zeros behind them, or
                                                    // (flagged rows) -m, -log l log2e, -delta
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + TK;
  static constexpr int OFF_Q = OFF_V + TK;          // [NQ]
  static constexpr int OFF_DO = OFF_Q + NQ * TQ;    // [NQ]
  static constexpr int OFF_PT = OFF_DO + NQ * TQ;   // [2] x [128 keys x 64 queries] SW128: the transposed bias tile arrives
                                                    // here and each thread overwrites its part with P^T
  static constexpr int OFF_DST = OFF_PT + 2 * 16384;    // [2] x dS^T, same shape
  static constexpr int OFF_ST = OFF_DST + 2 * 16384;    // [NQ] row constants
  static constexpr int OFF_KEY = OFF_ST + NQ * ST;
  static constexpr int OFF_BAR = OFF_KEY + RowFactors::kBytes;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
};

// 320 threads.  Warps 0-7 do the arithmetic: thread (r, hh) owns key r of the block and query half hh of each
// 64-query tile.  Warp 8 issues the MMAs and warp 9 the TMA copies, so none of that serial code sits between the
// arithmetic warps' steps; the sides meet only on mbarriers:
//   bar_s    MMA -> threads      S^T and dP^T of a tile are in TMEM
//   bar_free threads -> MMA      every warp has read them into registers (the next tile's products may start)
//   bar_p    threads -> MMA      P^T and dS^T of the tile are in shared memory (dV, dK products may start)
//   bar_acc  MMA -> TMA, threads those products are done: the tile's stage and its P^T / dS^T buffers are free
// P^T and dS^T are double buffered (P^T over the bias tile it was computed from), so the threads do not wait for
// the dV / dK products of one tile before the arithmetic of the next.
//
// MERGE (head dim 32): the same pass also produces this key block's share of dQ, so that S, the exponentials and dP
// are computed once for dK, dV and dQ instead of once per gradient.  dS^T then goes to shared memory ([128 keys x 64
// queries], the two buffers of a pair of query tiles 16 KB apart) instead of TMEM: dK reads it K-major as before, and
// after every second tile one product dQ_pair[128 queries x D] = dS_pair K reads the pair MN-major (M = queries) with
// K as the MN-major B operand, into the TMEM columns dS^T no longer needs.  The arithmetic warps fetch that
// accumulator one step later and store it, unscaled, as this key block's partial; attn_dq_sum_kernel adds the key
// blocks' partials in fixed order.  A last tile without a partner is paired with a buffer of zeros and has columns of its own.
// The MMA warp runs its code as a whole, so that descriptors stay in uniform registers (a lone lane took 900 clocks to issue a
// tile's products), and dQ is fetched after a tile's arrival on bar_p, beside its products: 1.56 -> 1.45 ms at N = 768.
// Accumulators are read eight queries at a time, the next eight on their way (the wait for a tile's first half had been 600 of
// 4100 clocks), and dQ leaves as 32-byte sectors: 1.45 -> 1.36 ms.  From there on a sustained training step at N = 768 runs at the
// board's power limit (1.8 GHz).  A persistent form (items as one stream) was slower, 1.47 -> 1.58 ms: K and V have no second
// buffer, and the two CTAs of an SM no longer change places.
template <typename T, int HD, bool HB, bool MERGE>
__global__ void __launch_bounds__(320, 2)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmBias, const AttnBwdArgs a) {
  using G = GeoC<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sK = smem + G::OFF_K;
  uint8_t* sV = smem + G::OFF_V;
  uint8_t* sQ = smem + G::OFF_Q;
  uint8_t* sDO = smem + G::OFF_DO;
  uint8_t* sPT = smem + G::OFF_PT;
  uint8_t* sDST = smem + G::OFF_DST;
  uint8_t* sRow = smem + G::OFF_ST;   // [NQ] row constants
  uint64_t* bar_kv = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);
  uint64_t* bar_in = bar_kv + 1;     // [NQ]
  uint64_t* bar_bias = bar_kv + 4;   // [2]
  uint64_t* bar_s = bar_kv + 6;
  uint64_t* bar_acc = bar_kv + 7;    // [4]: tile j commits to bar_acc[j & 3] (the copy warp may lag the MMA warp by up to
                                     // three tiles, so two tiles that share a barrier are never both pending)
  uint64_t* bar_free = bar_kv + 11;
  uint64_t* bar_p = bar_kv + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_kv + 13);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid & 127, hh = (tid >> 7) & 1;
  const int kblocks = (a.N + 127) / 128;
  int z = blockIdx.x;
  const int kvb = z % kblocks; z /= kblocks;
  const int h = z % a.H; z /= a.H;
  const int s = z % a.S;
  const int b = z / a.S;
  const int k0 = kvb * 128;
  const int nsteps = (a.N + 63) / 64;
  const int bias_b = b * a.bias_b_mul;

  if (tid == 0) {
    mbar_init(bar_kv, 1);
    for (int i = 0; i < G::NQ; ++i) mbar_init(&bar_in[i], 1);
    mbar_init(&bar_bias[0], 1); mbar_init(&bar_bias[1], 1); mbar_init(bar_s, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_acc[i], 1);
    mbar_init(bar_free, 8); mbar_init(bar_p, 8);
    mbar_fence_init();
  }
  RowFactors::fill<T>(smem + G::OFF_KEY, tid);
  if (tid >= 288 && tid < 288 + G::NQ * 8) reinterpret_cast<uint4*>(sRow + (tid - 288) / 8 * G::ST + 1024)[(tid - 288) % 8] = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  if (warp == 0) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  const bool folded = a.large[((long long)b * a.S + s) * a.H + h] == 0;   // the row's constants come with the products
  const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  constexpr uint32_t COL_DP = 64, COL_DV = 128, COL_DK = 128 + HD;
  // With head dim 32 the 256 TMEM columns have room for P^T and dS^T themselves (two 16-bit values per column), and
  // the dV / dK products read them from there: half the shared-memory traffic of the step, which is what bounds it.
  // They are single buffered, so a tile's values are stored once the previous tile's products are done.
  constexpr bool TMEM_A = HD == 32;
  constexpr uint32_t COL_PT = 192, COL_DST = 224;
  constexpr uint32_t COL_DQ = COL_DST;   // MERGE: dS^T lives in shared memory and its columns hold the dQ accumulator
  // A last tile without a partner: its product follows its own arrivals on bar_p, behind which the dQ before it may still be read.
  // It goes to the columns of S, which every warp has read (bar_free) and no further product wants.
  constexpr uint32_t COL_DQ_LAST = 0;
  static_assert(!MERGE || TMEM_A, "the merged pass is built for head dim 32");
  bool ok = true;

  if (warp == 9) {
    if (lane == 0) {
      // ---------------------------------- TMA copies ---------------------------------------------
      const long long row0 = (((long long)b * a.S + s) * a.H + h) * (long long)a.npad;
      const float* prep_row = a.prep + row0;
      auto load_step = [&](int step) {
        const int stg = step % G::NQ;
        float* st = reinterpret_cast<float*>(sRow + stg * G::ST);
        mbar_expect_tx(&bar_in[stg], 2 * G::TQ + (folded ? 1024 : 768));
        tma_load_5d(sQ + stg * G::TQ, &tmQ, &bar_in[stg], 0, h, step * 64, s, b);
        tma_load_5d(sDO + stg * G::TQ, &tmDO, &bar_in[stg], 0, h, step * 64, s, b);
        if (folded) {
          bulk_load(st, a.aug + row0 + step * 64, 1024, &bar_in[stg]);
        } else {
          bulk_load(st, prep_row + step * 64, 256, &bar_in[stg]);
          bulk_load(st + 64, prep_row + a.prep_plane + step * 64, 256, &bar_in[stg]);
          bulk_load(st + 128, prep_row + 2 * a.prep_plane + step * 64, 256, &bar_in[stg]);
        }
      };
      auto load_bias = [&](int step) {
        uint64_t* bb = &bar_bias[step & 1];
        mbar_expect_tx(bb, 16384);
        tma_load_4d(sPT + (step & 1) * 16384, &tmBias, bb, step * 64, k0, h, bias_b);   // transposed copy: queries inner
      };
      mbar_expect_tx(bar_kv, 2 * G::TK);
      tma_load_5d(sK, &tmK, bar_kv, 0, h, k0, s, b);
      tma_load_5d(sV, &tmV, bar_kv, 0, h, k0, s, b);
      for (int st = 0; st < G::NQ && st < nsteps; ++st) {
        load_step(st);
        if (HB && st < 2) load_bias(st);
      }
      for (int j = 0; j + 2 < nsteps && ok; ++j) {
        ok = mbar_wait(&bar_acc[j & 3], (j >> 2) & 1, a.err, 39) && ok;   // tile j's dV / dK products are done
        if (HB) load_bias(j + 2);                                         // its P^T buffer is free
        if (j + 3 < nsteps) load_step(j + 3);                             // ... and its Q / dO / statistics stage
      }
    }
  } else if (warp == 8) {
    {
      // ---------------------------------- MMA issue ----------------------------------------------
      // The whole warp runs this code and one lane issues: descriptors stay in uniform registers.
      const bool leader = elect_one();
      // Descriptors are built once: the high word is a constant per operand kind, the low word is
      // (address >> 4) plus the leading-dimension field, so a k-step or a stage only adds to it.
      constexpr uint32_t HI_KMAJ = desc_hi(G::SBO, G::LAYOUT);   // K, V, Q, dO as K-major rows of RB bytes
      constexpr uint32_t HI_PT = desc_hi(1024, 2);               // P^T, dS^T: [128 x 64] SW128
      const uint32_t k_lo = desc_lo(smem_u32(sK), 16), v_lo = desc_lo(smem_u32(sV), 16);
      const uint32_t q_lo = desc_lo(smem_u32(sQ), 16), do_lo = desc_lo(smem_u32(sDO), 16);
      const uint32_t qmn_lo = desc_lo(smem_u32(sQ), 64 * G::RB), domn_lo = desc_lo(smem_u32(sDO), 64 * G::RB);   // MN-major view
      const uint32_t pt_lo = desc_lo(smem_u32(sPT), 16), dst_lo = desc_lo(smem_u32(sDST), 16);
      const uint32_t dsmn_lo = desc_lo(smem_u32(sDST), 16384);      // dS of a tile pair as [m = query, k = key]: MN-major A
      const uint32_t kmn_lo = desc_lo(smem_u32(sK), 128 * G::RB);   // K as [n = d, k = key]: MN-major B
      const uint32_t key_s = RowFactors::key_s(smem_u32(smem + G::OFF_KEY)), key_dp = RowFactors::key_dp(smem_u32(smem + G::OFF_KEY));
      const uint32_t row_lo = RowFactors::query(smem_u32(sRow));
      // S^T = K Q^T and dP^T = V dO^T of one 64-query tile
      auto issue_scores = [&](int step) {
        const int stg = step % G::NQ;
        ok = mbar_wait(&bar_in[stg], (step / G::NQ) & 1, a.err, 32) && ok;
        tc_fence_after_sync();
        const uint32_t so = stg * (G::TQ >> 4);
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks)
            umma<KIND_F16>(tmem_base, desc_join(k_lo + ks * 2, HI_KMAJ), desc_join(q_lo + so + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
#pragma unroll
          for (int ks = 0; ks < HD / 16; ++ks)
            umma<KIND_F16>(tmem_base + COL_DP, desc_join(v_lo + ks * 2, HI_KMAJ), desc_join(do_lo + so + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
          if (folded) {
            const uint64_t rows = desc_join(row_lo + stg * (G::ST >> 4), RowFactors::HI_QUERY);
            umma<KIND_F16>(tmem_base, desc_join(key_s, RowFactors::HI_KEY), rows, a.idesc_a, 1);
            umma<KIND_F16>(tmem_base + COL_DP, desc_join(key_dp, RowFactors::HI_KEY), rows, a.idesc_a, 1);
          }
          umma_commit(bar_s);
        }
      };
      ok = mbar_wait(bar_kv, 0, a.err, 31);
      issue_scores(0);
      for (int j = 0; j < nsteps && ok; ++j) {
        const int qstg = j % G::NQ;
        ok = mbar_wait(bar_free, j & 1, a.err, 37) && ok;
        if (j + 1 < nsteps) issue_scores(j + 1);
        ok = mbar_wait(bar_p, j & 1, a.err, 38) && ok;
        tc_fence_after_sync();
        const uint32_t so = qstg * (G::TQ >> 4), bo = (j & 1) * (16384 >> 4);
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {   // dV += P^T dO   (B = dO as [n = d, k = query]: MN-major)
            const uint64_t bd = desc_join(domn_lo + so + kk * G::RB, HI_KMAJ);
            const uint32_t accf = (j > 0 || kk > 0) ? 1u : 0u;
            if constexpr (TMEM_A) umma_ts<KIND_F16>(tmem_base + COL_DV, tmem_base + COL_PT + kk * 8, bd, a.idesc_b, accf);
            else umma<KIND_F16>(tmem_base + COL_DV, desc_join(pt_lo + bo + kk * 2, HI_PT), bd, a.idesc_b, accf);
          }
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {   // dK += dS^T Q
            const uint64_t bd = desc_join(qmn_lo + so + kk * G::RB, HI_KMAJ);
            const uint32_t accf = (j > 0 || kk > 0) ? 1u : 0u;
            if constexpr (TMEM_A && !MERGE) umma_ts<KIND_F16>(tmem_base + COL_DK, tmem_base + COL_DST + kk * 8, bd, a.idesc_b, accf);
            else umma<KIND_F16>(tmem_base + COL_DK, desc_join(dst_lo + bo + kk * 2, HI_PT), bd, a.idesc_b, accf);
          }
          if constexpr (MERGE) {
            if ((j & 1) || j == nsteps - 1) {   // a pair of query tiles is complete: dQ_pair = dS_pair K (16 keys per product)
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                umma<KIND_F16>(tmem_base + (j & 1 ? COL_DQ : COL_DQ_LAST), desc_join(dsmn_lo + ks * 128, HI_PT), desc_join(kmn_lo + ks * G::RB, HI_KMAJ),
                               a.idesc_c, ks > 0);
            }
          }
          umma_commit(&bar_acc[j & 3]);
        }
      }
    }
  } else {
    // ------------------------------------ arithmetic warps ---------------------------------------
    const int kj = k0 + r;
    float mb = 0.f;
    if (kj >= a.N) mb = -INFINITY;
    else if (a.mask != nullptr) mb = kMaskSentinel * ((a.mask[b * a.mask_st[0] + s * a.mask_st[1] + kj] ? 1.0f : 0.0f) - 1.0f);
    const float2 sc2 = splat(a.scale), mk2 = splat(mb), l2e2 = splat(kLog2e), scl2 = splat(a.scale * kLog2e), mkl2 = splat(mb * kLog2e);
    // MERGE: fetch the dQ accumulator of query-tile pair `pair` (row r = query 128 pair + r, this thread's half of the
    // head dim) and store it, unscaled, as this key block's partial.  tcgen05.ld is warp-wide: every thread loads.
    auto store_dq_pair = [&](int pair, uint32_t col) {
      uint32_t v[16];
      tmem_ld_32x16(t_row + col + hh * 16, v);
      tmem_ld_wait();
      const int qi = pair * 128 + r;
      if (qi < a.N && ok) {
        T* dst = reinterpret_cast<T*>(a.dq_part) + kvb * a.dq_part_plane +
                 ((((long long)b * a.S + s) * a.N + qi) * a.H + h) * a.D + hh * 16;
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = pack2<T>(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        if (a.D == 32) {   // a whole 32-byte sector
          asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
                       "r"(w[5]), "r"(w[6]), "r"(w[7])
                       : "memory");
        } else {
#pragma unroll
          for (int g = 0; g < 2; ++g)
            if (hh * 16 + g * 8 < a.D) reinterpret_cast<uint4*>(dst)[g] = make_uint4(w[g * 4], w[g * 4 + 1], w[g * 4 + 2], w[g * 4 + 3]);
        }
      }
    };

    for (int j = 0; j < nsteps; ++j) {
      const int stg = j & 1, qstg = j % G::NQ;
      ok = mbar_wait(bar_s, j & 1, a.err, 33) && ok;
      tc_fence_after_sync();
      if (!folded) ok = mbar_wait(&bar_in[qstg], (j / G::NQ) & 1, a.err, 32) && ok;   // the tile's row statistics
      if (HB) ok = mbar_wait(&bar_bias[stg], (j >> 1) & 1, a.err, 34) && ok;

      // packed fp32x2 arithmetic: P = 2^((x - m) log2e - log l log2e), dS = P (dP - delta); thread = key, columns = queries.
      // Folded: the accumulators hold (scale q k - m - log l) / scale and dP - delta.
      const uint32_t sPTj = smem_u32(sPT) + stg * 16384;     // holds the transposed bias tile now, P^T when this step is done
      const uint32_t sDSTj = smem_u32(sDST) + stg * 16384;   // (its last readers, tile j-2's products, finished before S^T(j) did)
      const uint32_t st_a = smem_u32(sRow) + qstg * G::ST;   // -m, -log l log2e, -delta of 64 queries, 256 bytes each
      const int c = hh;
      uint32_t pw[16], dw[16];
      // this thread's 32 queries, eight at a time with the next eight's accumulators on their way
      const uint32_t t_s = t_row + hh * 32, t_d = t_row + COL_DP + hh * 32;
      auto eight = [&](auto fold, uint32_t (&rs)[8], uint32_t (&rp)[8], uint32_t (&ns)[8], uint32_t (&np)[8], int u) {
        ld_wait8x2(rs, rp);
        if (u < 3) {
          tmem_ld_32x8(t_s + (u + 1) * 8, ns);
          tmem_ld_32x8(t_d + (u + 1) * 8, np);
        } else {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_free);   // this warp holds its logits: the accumulators can take the next tile
        }
        uint4 raw = make_uint4(0, 0, 0, 0);
        if constexpr (HB) raw = lds128(sPTj + sw128_chunk1(r, c * 4 + u));
        const uint32_t bw[4] = {raw.x, raw.y, raw.z, raw.w};
        if constexpr (fold.value) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 t = HB ? __ffma2_rn(unpack2<T>(bw[i]), l2e2, mkl2) : mkl2;
            const float2 e = __ffma2_rn(pair(rs[2 * i], rs[2 * i + 1]), scl2, t);
            const float2 pp = make_float2(ex2_approx(e.x), ex2_approx(e.y));
            const float2 ds = __fmul2_rn(pp, pair(rp[2 * i], rp[2 * i + 1]));
            pw[u * 4 + i] = pack2<T>(pp.x, pp.y);
            dw[u * 4 + i] = pack2<T>(ds.x, ds.y);
          }
        } else {
          const uint32_t at = st_a + (c * 8 + u * 2) * 16;
          const float4 m0 = lds128f(at), m1 = lds128f(at + 16);
          const float4 l0 = lds128f(at + 256), l1 = lds128f(at + 272);
          const float4 d0 = lds128f(at + 512), d1 = lds128f(at + 528);
          const float2 nm[4] = {make_float2(m0.x, m0.y), make_float2(m0.z, m0.w), make_float2(m1.x, m1.y), make_float2(m1.z, m1.w)};
          const float2 nl[4] = {make_float2(l0.x, l0.y), make_float2(l0.z, l0.w), make_float2(l1.x, l1.y), make_float2(l1.z, l1.w)};
          const float2 nd[4] = {make_float2(d0.x, d0.y), make_float2(d0.z, d0.w), make_float2(d1.x, d1.y), make_float2(d1.z, d1.w)};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 x = __ffma2_rn(pair(rs[2 * i], rs[2 * i + 1]), sc2, mk2);
            if constexpr (HB) x = __fadd2_rn(x, unpack2<T>(bw[i]));
            const float2 e = __ffma2_rn(__fadd2_rn(x, nm[i]), l2e2, nl[i]);
            const float2 pp = make_float2(ex2_approx(e.x), ex2_approx(e.y));
            const float2 ds = __fmul2_rn(pp, __fadd2_rn(pair(rp[2 * i], rp[2 * i + 1]), nd[i]));
            pw[u * 4 + i] = pack2<T>(pp.x, pp.y);
            dw[u * 4 + i] = pack2<T>(ds.x, ds.y);
          }
        }
      };
      auto tile = [&](auto fold) {
        uint32_t sA[8], pA[8], sB[8], pB[8];
        tmem_ld_32x8(t_s, sA);
        tmem_ld_32x8(t_d, pA);
        eight(fold, sA, pA, sB, pB, 0);
        eight(fold, sB, pB, sA, pA, 1);
        eight(fold, sA, pA, sB, pB, 2);
        eight(fold, sB, pB, sA, pA, 3);
      };
      if (folded) tile(std::true_type{});
      else tile(std::false_type{});
      if constexpr (!TMEM_A) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          sts128(sPTj + sw128_chunk1(r, c * 4 + u), pw[u * 4], pw[u * 4 + 1], pw[u * 4 + 2], pw[u * 4 + 3]);
          sts128(sDSTj + sw128_chunk1(r, c * 4 + u), dw[u * 4], dw[u * 4 + 1], dw[u * 4 + 2], dw[u * 4 + 3]);
        }
      }
      if constexpr (TMEM_A) {
        if (j > 0) ok = mbar_wait(&bar_acc[(j - 1) & 3], ((j - 1) >> 2) & 1, a.err, 35) && ok;   // the previous tile's products have read theirs
        tc_fence_after_sync();
        tmem_st_32x16(t_row + COL_PT + hh * 16, pw);    // this thread's key row, its 32 queries as 16 packed columns
        if constexpr (MERGE) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            sts128(sDSTj + sw128_chunk1(r, c * 4 + u), dw[u * 4], dw[u * 4 + 1], dw[u * 4 + 2], dw[u * 4 + 3]);
          if (j == nsteps - 1 && (j & 1) == 0) {   // no partner tile: the pair's second buffer reads as zeros
#pragma unroll
            for (int u = 0; u < 4; ++u)
              sts128(smem_u32(sDST) + 16384 + sw128_chunk1(r, c * 4 + u), 0, 0, 0, 0);
          }
          fence_proxy_async_smem();
        } else {
          tmem_st_32x16(t_row + COL_DST + hh * 16, dw);
        }
        tmem_st_wait();
      } else {
        fence_proxy_async_smem();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
      if (!ok) break;
      // The pair before this tile: its dQ product is done (bar_acc above).  The next one into its columns is that of tile j + 1, which
      // waits for this warp's arrival there; a tile j without a partner has columns of its own.
      if constexpr (MERGE) {
        if (j >= 2 && (j & 1) == 0) store_dq_pair(j / 2 - 1, COL_DQ);
      }
    }
    ok = mbar_wait(&bar_acc[(nsteps - 1) & 3], ((nsteps - 1) >> 2) & 1, a.err, 36) && ok;
    tc_fence_after_sync();
    if constexpr (MERGE) store_dq_pair((nsteps - 1) / 2, nsteps & 1 ? COL_DQ_LAST : COL_DQ);   // the last pair
    {
      const bool st_ok = kj < a.N && ok && hh == 0;
      T* krow = reinterpret_cast<T*>(a.out0) + b * a.out0_st[0] + s * a.out0_st[1] + kj * a.out0_st[2] + h * a.out0_st[3];
      T* vrow = reinterpret_cast<T*>(a.out1) + b * a.out1_st[0] + s * a.out1_st[1] + kj * a.out1_st[2] + h * a.out1_st[3];
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t rk[32], rv[32];
        tmem_ld_32x32(t_row + COL_DK + c * 32, rk);
        tmem_ld_32x32(t_row + COL_DV + c * 32, rv);
        tmem_ld_wait();
        if (st_ok) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            if (c * 32 + g * 8 >= a.D) break;
            uint4 pk;
            pk.x = pack2<T>(__uint_as_float(rk[g * 8 + 0]) * a.scale, __uint_as_float(rk[g * 8 + 1]) * a.scale);
            pk.y = pack2<T>(__uint_as_float(rk[g * 8 + 2]) * a.scale, __uint_as_float(rk[g * 8 + 3]) * a.scale);
            pk.z = pack2<T>(__uint_as_float(rk[g * 8 + 4]) * a.scale, __uint_as_float(rk[g * 8 + 5]) * a.scale);
            pk.w = pack2<T>(__uint_as_float(rk[g * 8 + 6]) * a.scale, __uint_as_float(rk[g * 8 + 7]) * a.scale);
            reinterpret_cast<uint4*>(krow)[c * 4 + g] = pk;
            pk.x = pack2<T>(__uint_as_float(rv[g * 8 + 0]), __uint_as_float(rv[g * 8 + 1]));
            pk.y = pack2<T>(__uint_as_float(rv[g * 8 + 2]), __uint_as_float(rv[g * 8 + 3]));
            pk.z = pack2<T>(__uint_as_float(rv[g * 8 + 4]), __uint_as_float(rv[g * 8 + 5]));
            pk.w = pack2<T>(__uint_as_float(rv[g * 8 + 6]), __uint_as_float(rv[g * 8 + 7]));
            reinterpret_cast<uint4*>(vrow)[c * 4 + g] = pk;
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
}

// ------------------------------------------------------------------------------------------------
// dQ pass: one CTA per (batch, row, head, 128-query block), 64-key tiles.  320 threads: warps 0-7 do the arithmetic
// (thread (r, hh) owns query r and key half hh of each tile), warp 8 issues the MMAs, warp 9 the TMA copies.
//   S = Q K^T, dP = dO V^T (TMEM) -> dS = P (dP - delta) packed into TMEM -> dQ += dS K (A operand read from TMEM).
// Barriers as in the dK/dV pass: bar_s, bar_free, bar_p, and a ring bar_dq[4] for the dQ products.
// ------------------------------------------------------------------------------------------------
template <int HD> struct GeoQ {
  static constexpr int RB = HD * 2;
  static constexpr int TA = 128 * RB;                    // Q / dO tile
  static constexpr int TB = 64 * RB;                     // K / V tile
  static constexpr uint32_t LAYOUT = RB == 128 ? 2 : 4;
  static constexpr uint32_t SBO = 8 * RB;
  static constexpr int NS = 3;                           // K / V stages: tiles are fetched two steps ahead
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = OFF_Q + TA;
  static constexpr int OFF_K = OFF_DO + TA;              // [NS]
  static constexpr int OFF_V = OFF_K + NS * TB;          // [NS]
  static constexpr int OFF_BIAS = OFF_V + NS * TB;       // [2] x [128 queries x 64 keys] SW128
  static constexpr int OFF_MB = OFF_BIAS + 2 * 16384;    // [NS] x 64 additive key-mask terms
  static constexpr int OFF_BAR = OFF_MB + NS * 256;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
};

template <typename T, int HD, bool HB>
__global__ void __launch_bounds__(320, 2)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const __grid_constant__ CUtensorMap tmBias, const AttnBwdArgs a) {
  using G = GeoQ<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sQ = smem + G::OFF_Q;
  uint8_t* sDO = smem + G::OFF_DO;
  uint8_t* sK = smem + G::OFF_K;
  uint8_t* sV = smem + G::OFF_V;
  uint8_t* sBias = smem + G::OFF_BIAS;
  float* sMb = reinterpret_cast<float*>(smem + G::OFF_MB);
  uint64_t* bar_once = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);   // Q + dO
  uint64_t* bar_in = bar_once + 1;    // [NS] K, V and mask terms of a tile
  uint64_t* bar_bias = bar_once + 4;  // [2]
  uint64_t* bar_s = bar_once + 6;
  uint64_t* bar_dq = bar_once + 7;    // [4]: tile j commits to bar_dq[j & 3]
  uint64_t* bar_free = bar_once + 11;
  uint64_t* bar_p = bar_once + 12;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_once + 13);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid & 127, hh = (tid >> 7) & 1;
  const int qblocks = (a.N + 127) / 128;
  int z = blockIdx.x;
  const int qb = z % qblocks; z /= qblocks;
  const int h = z % a.H; z /= a.H;
  const int s = z % a.S;
  const int b = z / a.S;
  const int q0 = qb * 128;
  const int nsteps = (a.N + 63) / 64;
  const int bias_b = b * a.bias_b_mul;

  if (tid == 0) {
    mbar_init(bar_once, 1);
    for (int i = 0; i < G::NS; ++i) mbar_init(&bar_in[i], 1);
    mbar_init(&bar_bias[0], 1); mbar_init(&bar_bias[1], 1); mbar_init(bar_s, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_dq[i], 1);
    mbar_init(bar_free, 8); mbar_init(bar_p, 8);
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  constexpr uint32_t COL_DP = 64, COL_DQ = 128, COL_DS = 128 + HD;   // dS: 64 keys as 32 packed columns
  bool ok = true;

  if (warp == 9) {
    if (lane == 0) {
      // ---------------------------------- TMA copies ---------------------------------------------
      const float* mrow = a.mask_terms + ((long long)b * a.S + s) * a.npad;
      auto load_step = [&](int step) {
        const int stg = step % G::NS;
        mbar_expect_tx(&bar_in[stg], 2 * G::TB + 256);
        tma_load_5d(sK + stg * G::TB, &tmK, &bar_in[stg], 0, h, step * 64, s, b);
        tma_load_5d(sV + stg * G::TB, &tmV, &bar_in[stg], 0, h, step * 64, s, b);
        bulk_load(sMb + stg * 64, mrow + step * 64, 256, &bar_in[stg]);
      };
      auto load_bias = [&](int step) {
        uint64_t* bb = &bar_bias[step & 1];
        mbar_expect_tx(bb, 16384);
        tma_load_4d(sBias + (step & 1) * 16384, &tmBias, bb, step * 64, q0, h, bias_b);
      };
      mbar_expect_tx(bar_once, 2 * G::TA);
      tma_load_5d(sQ, &tmQ, bar_once, 0, h, q0, s, b);
      tma_load_5d(sDO, &tmDO, bar_once, 0, h, q0, s, b);
      for (int st = 0; st < G::NS && st < nsteps; ++st) {
        load_step(st);
        if (HB && st < 2) load_bias(st);
      }
      for (int j = 0; j + 2 < nsteps && ok; ++j) {
        ok = mbar_wait(&bar_dq[j & 3], (j >> 2) & 1, a.err, 26) && ok;   // tile j's dQ product is done
        if (HB) load_bias(j + 2);                                        // (its bias tile was read before that)
        if (j + 3 < nsteps) load_step(j + 3);                            // its K / V stage is free
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      // ---------------------------------- MMA issue ----------------------------------------------
      constexpr uint32_t HI_KMAJ = desc_hi(G::SBO, G::LAYOUT);
      const uint32_t q_lo = desc_lo(smem_u32(sQ), 16), do_lo = desc_lo(smem_u32(sDO), 16);
      const uint32_t k_lo = desc_lo(smem_u32(sK), 16), v_lo = desc_lo(smem_u32(sV), 16);
      const uint32_t kmn_lo = desc_lo(smem_u32(sK), 64 * G::RB);   // K as [n = d, k = key]
      auto issue_scores = [&](int step) {
        const int stg = step % G::NS;
        ok = mbar_wait(&bar_in[stg], (step / G::NS) & 1, a.err, 23) && ok;
        tc_fence_after_sync();
        const uint32_t so = stg * (G::TB >> 4);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma<KIND_F16>(tmem_base, desc_join(q_lo + ks * 2, HI_KMAJ), desc_join(k_lo + so + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma<KIND_F16>(tmem_base + COL_DP, desc_join(do_lo + ks * 2, HI_KMAJ), desc_join(v_lo + so + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
        umma_commit(bar_s);
      };
      ok = mbar_wait(bar_once, 0, a.err, 22);
      issue_scores(0);
      for (int j = 0; j < nsteps && ok; ++j) {
        ok = mbar_wait(bar_free, j & 1, a.err, 28) && ok;
        if (j + 1 < nsteps) issue_scores(j + 1);
        ok = mbar_wait(bar_p, j & 1, a.err, 29) && ok;
        tc_fence_after_sync();
        const uint32_t so = (j % G::NS) * (G::TB >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)   // dQ += dS K   (A = dS from TMEM, B = K as [n = d, k = key]: MN-major)
          umma_ts<KIND_F16>(tmem_base + COL_DQ, tmem_base + COL_DS + kk * 8, desc_join(kmn_lo + so + kk * G::RB, HI_KMAJ), a.idesc_b,
                      (j > 0 || kk > 0) ? 1u : 0u);
        umma_commit(&bar_dq[j & 3]);
      }
    }
  } else {
    // ------------------------------------ arithmetic warps ---------------------------------------
    const int qi = q0 + r;
    const bool q_ok = qi < a.N;
    float m_row = 0.f, l_row = 0.f, d_row = 0.f;
    if (q_ok) {
      const long long plane = (long long)a.B * a.S * a.H * a.N;
      const long long row = (((long long)b * a.S + s) * a.H + h) * a.N + qi;
      m_row = a.stats[row]; l_row = a.stats[plane + row]; d_row = a.delta[row];
    }
    // packed fp32x2 arithmetic: P = 2^((x - m) log2e - log l log2e), dS = P (dP - delta)
    const float2 sc2 = splat(a.scale), nm2 = splat(-m_row), nl2 = splat(-l_row * kLog2e), l2e2 = splat(kLog2e),
                 nd2 = splat(-d_row);

    for (int j = 0; j < nsteps; ++j) {
      const int stg = j & 1, kstg = j % G::NS;
      ok = mbar_wait(bar_s, j & 1, a.err, 24) && ok;
      tc_fence_after_sync();
      ok = mbar_wait(&bar_in[kstg], (j / G::NS) & 1, a.err, 23) && ok;   // the tile's mask terms
      if (HB) ok = mbar_wait(&bar_bias[stg], (j >> 1) & 1, a.err, 25) && ok;
      const uint32_t mb_a = smem_u32(sMb) + kstg * 256 + hh * 128, bias_t = smem_u32(sBias) + stg * 16384;
      uint32_t dw[16];
      // 16 of this thread's 32 columns: dS = P (dP - delta), packed
      auto half = [&](const uint32_t (&rs)[16], const uint32_t (&rp)[16], int h2) {
#pragma unroll
        for (int uu = 0; uu < 2; ++uu) {
          const int u = h2 * 2 + uu;
          uint4 raw = make_uint4(0, 0, 0, 0);
          if constexpr (HB) raw = lds128(bias_t + sw128_chunk1(r, hh * 4 + u));
          const uint32_t bw[4] = {raw.x, raw.y, raw.z, raw.w};
          const float4 mA = lds128f(mb_a + u * 32), mB = lds128f(mb_a + u * 32 + 16);
          const float2 mk[4] = {make_float2(mA.x, mA.y), make_float2(mA.z, mA.w), make_float2(mB.x, mB.y),
                                make_float2(mB.z, mB.w)};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 x = __ffma2_rn(pair(rs[uu * 8 + 2 * i], rs[uu * 8 + 2 * i + 1]), sc2, mk[i]);
            if constexpr (HB) x = __fadd2_rn(x, unpack2<T>(bw[i]));
            const float2 e = __ffma2_rn(__fadd2_rn(x, nm2), l2e2, nl2);
            const float2 p = make_float2(ex2_approx(e.x), ex2_approx(e.y));
            const float2 ds = __fmul2_rn(p, __fadd2_rn(pair(rp[uu * 8 + 2 * i], rp[uu * 8 + 2 * i + 1]), nd2));
            dw[u * 4 + i] = pack2<T>(ds.x, ds.y);
          }
        }
      };
      // the second half's TMEM loads are in flight while the first half is computed
      uint32_t rsA[16], rpA[16], rsB[16], rpB[16];
      tmem_ld_32x16(t_row + hh * 32, rsA);
      tmem_ld_32x16(t_row + COL_DP + hh * 32, rpA);
      tmem_ld_wait();
      tmem_ld_32x16(t_row + hh * 32 + 16, rsB);
      tmem_ld_32x16(t_row + COL_DP + hh * 32 + 16, rpB);
      half(rsA, rpA, 0);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_free);   // this warp holds its logits: the accumulators can take the next tile
      half(rsB, rpB, 1);
      if (j > 0) ok = mbar_wait(&bar_dq[(j - 1) & 3], ((j - 1) >> 2) & 1, a.err, 26) && ok;   // the previous dS has been read
      tc_fence_after_sync();
      tmem_st_32x16(t_row + COL_DS + hh * 16, dw);   // this thread's query row, its 32 keys as 16 packed columns
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
      if (!ok) break;
    }
    ok = mbar_wait(&bar_dq[(nsteps - 1) & 3], ((nsteps - 1) >> 2) & 1, a.err, 27) && ok;
    tc_fence_after_sync();
    {
      // tcgen05.ld is warp-collective: every thread loads, only valid rows store; the halves split the head dim
      const bool st_ok = q_ok && ok;
      T* row = reinterpret_cast<T*>(a.out0) + b * a.out0_st[0] + s * a.out0_st[1] + qi * a.out0_st[2] + h * a.out0_st[3];
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[16];
        tmem_ld_32x16(t_row + COL_DQ + hh * (HD / 2) + c * 16, v);
        tmem_ld_wait();
        if (st_ok) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint4 pk;
            pk.x = pack2<T>(__uint_as_float(v[g * 8 + 0]) * a.scale, __uint_as_float(v[g * 8 + 1]) * a.scale);
            pk.y = pack2<T>(__uint_as_float(v[g * 8 + 2]) * a.scale, __uint_as_float(v[g * 8 + 3]) * a.scale);
            pk.z = pack2<T>(__uint_as_float(v[g * 8 + 4]) * a.scale, __uint_as_float(v[g * 8 + 5]) * a.scale);
            pk.w = pack2<T>(__uint_as_float(v[g * 8 + 6]) * a.scale, __uint_as_float(v[g * 8 + 7]) * a.scale);
            if (hh * (HD / 2) + c * 16 + g * 8 < a.D) reinterpret_cast<uint4*>(row)[(hh * (HD / 2) + c * 16) / 8 + g] = pk;
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
}

// ------------------------------------------------------------------------------------------------
// dbias pass: one CTA per (row chunk, batch, head, 64-query block, 128-key block) looping over the rows of its chunk
// in order and summing dS = P (dP - delta) in registers (no atomics: the sum over rows has a fixed order; the chunks'
// partial sums are added by sum_partials_kernel).  320 threads: warps 0-7 do the arithmetic (thread (r, hh) owns
// key r and query half hh), warp 8 issues the MMAs, warp 9 the TMA copies.  S^T and dP^T are double buffered in TMEM,
// so the products of the next two rows run under the arithmetic of this one.
// Thread = key: what varies over a thread's queries comes with the products (RowFactors), the mask is one value per row and
// the bias, the same for all rows, stays in registers: nothing but the accumulators is read in the loop.
// With thread = query, the bias tile and the rows' mask terms were read for every row: 0.81 -> 0.70 ms at N = 768, 4 heads.
//   bar_s[2]    MMA -> threads        S, dP of a row are in TMEM buffer (row & 1)
//   bar_free[4] threads -> MMA, TMA   the row's accumulators, statistics and mask terms have been read
// ------------------------------------------------------------------------------------------------
template <int HD> struct GeoB {
  static constexpr int RB = HD * 2;
  static constexpr int TA = 128 * RB;                    // K / V tile
  static constexpr int TB = 64 * RB;                     // Q / dO tile
  static constexpr uint32_t LAYOUT = RB == 128 ? 2 : 4;
  static constexpr uint32_t SBO = 8 * RB;
  static constexpr int NS = 3;                           // row stages
  static constexpr int OFF_MASK = 1024 + 128;            // factors of 64 queries and zeros behind them, or (flagged rows)
                                                         // -m, -log l log2e, -delta; then 128 mask terms
  static constexpr int STAT = 2048;                      // (stages stay 1024-byte aligned for the swizzled tiles)
  static constexpr int STAGE = 2 * TA + 2 * TB + STAT;
  static constexpr int OFF_BIAS = NS * STAGE;            // [128 keys x 64 queries] SW128, loaded once
  static constexpr int OFF_KEY = OFF_BIAS + 16384;
  static constexpr int OFF_BAR = OFF_KEY + RowFactors::kBytes;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
};

template <typename T, int HD>
__global__ void __launch_bounds__(320, HD == 32 ? 2 : 1)
attn_bwd_dbias_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                      const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                      const __grid_constant__ CUtensorMap tmBias, const AttnBwdArgs a) {
  using G = GeoB<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sBias = smem + G::OFF_BIAS;
  uint64_t* bar_once = reinterpret_cast<uint64_t*>(smem + G::OFF_BAR);   // bias tile
  uint64_t* bar_in = bar_once + 1;     // [NS]
  uint64_t* bar_s = bar_once + 4;      // [2]
  uint64_t* bar_free = bar_once + 6;   // [4]: row j arrives on bar_free[j & 3]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_once + 10);
  auto stage_k = [&](int stg) { return smem + stg * G::STAGE; };
  auto stage_v = [&](int stg) { return smem + stg * G::STAGE + G::TA; };
  auto stage_q = [&](int stg) { return smem + stg * G::STAGE + 2 * G::TA; };
  auto stage_do = [&](int stg) { return smem + stg * G::STAGE + 2 * G::TA + G::TB; };
  auto stage_stat = [&](int stg) { return reinterpret_cast<float*>(smem + stg * G::STAGE + 2 * G::TA + 2 * G::TB); };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = tid & 127, hh = (tid >> 7) & 1;
  const int qblocks = (a.N + 63) / 64, kblocks = (a.N + 127) / 128;
  int z = blockIdx.x;
  const int kvb = z % kblocks; z /= kblocks;
  const int qb = z % qblocks; z /= qblocks;
  const int h = z % a.H; z /= a.H;
  const int b = z % a.B;
  const int rc = z / a.B;
  const int per = (a.S + a.row_chunks - 1) / a.row_chunks;
  const int s_lo = rc * per;
  const int nsteps = max(0, min(a.S, s_lo + per) - s_lo);
  const int q0 = qb * 64, k0 = kvb * 128;

  if (tid == 0) {
    mbar_init(bar_once, 1);
    for (int i = 0; i < G::NS; ++i) mbar_init(&bar_in[i], 1);
    mbar_init(&bar_s[0], 1); mbar_init(&bar_s[1], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&bar_free[i], 8);
    mbar_fence_init();
  }
  RowFactors::fill<T>(smem + G::OFF_KEY, tid);
  if (tid >= 288 && tid < 288 + G::NS * 8) reinterpret_cast<uint4*>(stage_stat((tid - 288) / 8) + 256)[(tid - 288) % 8] = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  if (warp == 0) tmem_alloc(tmem_slot, 256);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();
  const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
  bool ok = true;
  const int* large = a.large + ((long long)b * a.S + s_lo) * a.H + h;   // flags of the rows, H apart

  if (warp == 9) {
    if (lane == 0) {
      // ---------------------------------- TMA copies ---------------------------------------------
      auto load_step = [&](int step) {
        const int stg = step % G::NS, s = s_lo + step;
        const long long row0 = (((long long)b * a.S + s) * a.H + h) * (long long)a.npad + q0;
        const float* prow = a.prep + row0;
        const bool folded = large[(long long)step * a.H] == 0;
        float* st = stage_stat(stg);
        mbar_expect_tx(&bar_in[stg], 2 * G::TA + 2 * G::TB + (folded ? 1024 : 3 * 256) + 512);
        tma_load_5d(stage_q(stg), &tmQ, &bar_in[stg], 0, h, q0, s, b);
        tma_load_5d(stage_do(stg), &tmDO, &bar_in[stg], 0, h, q0, s, b);
        tma_load_5d(stage_k(stg), &tmK, &bar_in[stg], 0, h, k0, s, b);
        tma_load_5d(stage_v(stg), &tmV, &bar_in[stg], 0, h, k0, s, b);
        if (folded) {
          bulk_load(st, a.aug + row0, 1024, &bar_in[stg]);
        } else {
          bulk_load(st, prow, 256, &bar_in[stg]);
          bulk_load(st + 64, prow + a.prep_plane, 256, &bar_in[stg]);
          bulk_load(st + 128, prow + 2 * a.prep_plane, 256, &bar_in[stg]);
        }
        bulk_load(st + G::OFF_MASK / 4, a.mask_terms + (folded ? a.mask_plane : 0) + ((long long)b * a.S + s) * a.npad + k0, 512, &bar_in[stg]);
      };
      if (nsteps > 0) {   // (a CTA with no rows must not leave a copy in flight)
        mbar_expect_tx(bar_once, 16384);
        tma_load_4d(sBias, &tmBias, bar_once, q0, k0, h, b * a.bias_b_mul);   // transposed copy: queries inner
      }
      for (int st = 0; st < G::NS && st < nsteps; ++st) load_step(st);
      for (int j = 0; j + G::NS < nsteps && ok; ++j) {
        ok = mbar_wait(&bar_free[j & 3], (j >> 2) & 1, a.err, 41) && ok;   // row j has been consumed: its stage is free
        load_step(j + G::NS);
      }
    }
  } else if (warp == 8) {
    if (lane == 0) {
      // ---------------------------------- MMA issue ----------------------------------------------
      constexpr uint32_t HI_KMAJ = desc_hi(G::SBO, G::LAYOUT);
      const uint32_t base_lo = desc_lo(smem_u32(smem), 16);
      const uint32_t key_s = RowFactors::key_s(smem_u32(smem + G::OFF_KEY)), key_dp = RowFactors::key_dp(smem_u32(smem + G::OFF_KEY));
      const uint32_t row_lo = RowFactors::query(smem_u32(stage_stat(0)));
      int flag = nsteps > 0 ? large[0] : 0;
      for (int j = 0; j < nsteps && ok; ++j) {
        const int stg = j % G::NS, buf = j & 1;
        const bool folded = flag == 0;
        if (j + 1 < nsteps) flag = large[(long long)(j + 1) * a.H];
        if (j >= 2) ok = mbar_wait(&bar_free[(j - 2) & 3], ((j - 2) >> 2) & 1, a.err, 42) && ok;   // TMEM buffer is free
        ok = mbar_wait(&bar_in[stg], (j / G::NS) & 1, a.err, 43) && ok;
        tc_fence_after_sync();
        const uint32_t k_lo = base_lo + stg * (G::STAGE >> 4), v_lo = k_lo + (G::TA >> 4), q_lo = v_lo + (G::TA >> 4),
                       do_lo = q_lo + (G::TB >> 4);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma<KIND_F16>(tmem_base + buf * 128, desc_join(k_lo + ks * 2, HI_KMAJ), desc_join(q_lo + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
#pragma unroll
        for (int ks = 0; ks < HD / 16; ++ks)
          umma<KIND_F16>(tmem_base + buf * 128 + 64, desc_join(v_lo + ks * 2, HI_KMAJ), desc_join(do_lo + ks * 2, HI_KMAJ), a.idesc_a, ks > 0);
        if (folded) {
          const uint64_t rows = desc_join(row_lo + stg * (G::STAGE >> 4), RowFactors::HI_QUERY);
          umma<KIND_F16>(tmem_base + buf * 128, desc_join(key_s, RowFactors::HI_KEY), rows, a.idesc_a, 1);
          umma<KIND_F16>(tmem_base + buf * 128 + 64, desc_join(key_dp, RowFactors::HI_KEY), rows, a.idesc_a, 1);
        }
        umma_commit(&bar_s[buf]);
      }
    }
  } else {
    // ------------------------------------ arithmetic warps ---------------------------------------
    float acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.f;
    const float2 sc2 = splat(a.scale), l2e2 = splat(kLog2e), scl2 = splat(a.scale * kLog2e);
    if (nsteps > 0) ok = mbar_wait(bar_once, 0, a.err, 21);
    uint4 bias[4];   // of this thread's key and 32 queries
#pragma unroll
    for (int u = 0; u < 4; ++u) bias[u] = nsteps > 0 ? lds128(smem_u32(sBias) + sw128_chunk1(r, hh * 4 + u)) : make_uint4(0, 0, 0, 0);

    // a row's share of the sum, eight queries at a time with the next eight on their way
    auto add_row = [&](auto fold, int stg, int buf) {
      const uint32_t st_a = smem_u32(stage_stat(stg)), t_s = t_row + buf * 128 + hh * 32;
      const float2 mk2 = splat(lds32f(st_a + G::OFF_MASK + r * 4));   // (in units of log 2 where folded)
      auto eight = [&](uint32_t (&rs)[8], uint32_t (&rp)[8], uint32_t (&ns)[8], uint32_t (&np)[8], int u) {
        ld_wait8x2(rs, rp);
        if (u < 3) {
          tmem_ld_32x8(t_s + (u + 1) * 8, ns);
          tmem_ld_32x8(t_s + 64 + (u + 1) * 8, np);
        }
        const uint32_t bw[4] = {bias[u].x, bias[u].y, bias[u].z, bias[u].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 s2 = pair(rs[2 * i], rs[2 * i + 1]), d2 = pair(rp[2 * i], rp[2 * i + 1]);
          const int k = u * 8 + 2 * i;
          const float2 sum = make_float2(acc[k], acc[k + 1]);
          float2 t;
          if constexpr (fold.value) {
            const float2 e = __ffma2_rn(s2, scl2, __ffma2_rn(unpack2<T>(bw[i]), l2e2, mk2));
            t = __ffma2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), d2, sum);
          } else {
            const uint32_t at = st_a + (hh * 32 + k) * 4;
            const float2 nm = make_float2(lds32f(at), lds32f(at + 4)), nl = make_float2(lds32f(at + 256), lds32f(at + 260)),
                         nd = make_float2(lds32f(at + 512), lds32f(at + 516));
            const float2 x = __fadd2_rn(__ffma2_rn(s2, sc2, mk2), unpack2<T>(bw[i]));
            const float2 e = __ffma2_rn(__fadd2_rn(x, nm), l2e2, nl);
            t = __fadd2_rn(sum, __fmul2_rn(make_float2(ex2_approx(e.x), ex2_approx(e.y)), __fadd2_rn(d2, nd)));
          }
          acc[k] = t.x;
          acc[k + 1] = t.y;
        }
      };
      uint32_t sA[8], pA[8], sB[8], pB[8];
      tmem_ld_32x8(t_s, sA);
      tmem_ld_32x8(t_s + 64, pA);
      eight(sA, pA, sB, pB, 0);
      eight(sB, pB, sA, pA, 1);
      eight(sA, pA, sB, pB, 2);
      eight(sB, pB, sA, pA, 3);
    };
    int flag = nsteps > 0 ? large[0] : 0;
    for (int j = 0; j < nsteps; ++j) {
      const int stg = j % G::NS, buf = j & 1;
      const bool folded = flag == 0;
      if (j + 1 < nsteps) flag = large[(long long)(j + 1) * a.H];
      ok = mbar_wait(&bar_in[stg], (j / G::NS) & 1, a.err, 43) && ok;   // statistics and mask terms of the row
      ok = mbar_wait(&bar_s[buf], (j >> 1) & 1, a.err, 24) && ok;
      tc_fence_after_sync();
      if (folded) add_row(std::true_type{}, stg, buf);
      else add_row(std::false_type{}, stg, buf);
      fence_proxy_async_smem();   // (TMA writes the row's statistics and mask terms over)
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_free[j & 3]);   // accumulators, statistics and mask terms of the row are consumed
      if (!ok) break;
    }

    const int kj = k0 + r;
    if (kj < a.N && ok) {   // a query at a time: lanes are consecutive keys
      float* at = reinterpret_cast<float*>(a.out0) + (long long)rc * a.B * a.H * a.N * a.N +
                  (((long long)b * a.H + h) * a.N + q0 + hh * 32) * a.N + kj;
      const int valid = a.N - q0 - hh * 32;
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i < valid) at[(long long)i * a.N] = acc[i];
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 256);
  }
}

// What the backward passes read besides the tensors, in one launch.
//   delta[b,s,h,i] = sum_d dO * O (written where the dQ pass reads it); the row constants as factors (see RowFactors), and for flagged
//   rows in the form their packed arithmetic adds (prep[0] = -m, prep[1] = -log l * log2e, prep[2] = -delta); padded to npad entries
//   with zeros.  A block has a (batch, row, head), a warp 32 of its queries at a time, four lanes to a query: a request covers rows of
//   64 bytes whole.
//   The key-mask terms of a (batch, row), by its first head's block: 0 for a kept key, -1e9 for a masked one, -inf beyond N; and in a
//   second plane times log2(e).
//   The first blocks transpose the bias instead: out[b][h][k][q] = bias[b][h][q][k], a 64 x 64 tile each.
// One launch in place of three.  At 301 x 301 residues, 4 heads of 32: 16 us under ncu against 20 + 3 + 9 and the gaps between them; at
// 768 x 768 71 against 87 + 6 + 12 (85 to 97 in a long step at the power limit), where the bytes are 60: what it waits for is the load,
// sum, exchange and store of an item, with 24 warps an SM on it (three blocks; with two 1.3 times as long).  Also clears the status.
struct PrepareArgs {
  const float* stats;
  float *delta, *prep, *mask_terms;
  uint4* aug;
  int* large;
  int* err;
  const uint8_t* mask;
  const uint16_t* bias;
  uint16_t* bias_t;
  int npad, pitch, tiles, transposes;   // tiles of a side of the bias; blocks that transpose
};
template <typename T>
__global__ void __launch_bounds__(256, 3) attn_prepare_kernel(const TriAttnDesc d, const T* o, const T* d_o, const PrepareArgs a) {
  __shared__ uint16_t tile[64][66];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = d.n_res;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.err[0] = a.err[1] = 0;
  if ((int)blockIdx.x < a.transposes) {
    unsigned z = blockIdx.x;
    const int k0 = (int)(z % (unsigned)a.tiles) * 64; z /= (unsigned)a.tiles;
    const int q0 = (int)(z % (unsigned)a.tiles) * 64, bh = (int)(z / (unsigned)a.tiles);
    const uint16_t* src = a.bias + bh / d.H * d.bias_st[0] + bh % d.H * d.bias_st[1];
    uint16_t* dst = a.bias_t + (int64_t)bh * N * a.pitch;
    for (int i = warp; i < 64; i += 8)
#pragma unroll
      for (int e = 0; e < 64; e += 32)
        if (q0 + i < N && k0 + lane + e < N) tile[i][lane + e] = src[(q0 + i) * d.bias_st[2] + k0 + lane + e];
    __syncthreads();
    for (int i = warp; i < 64; i += 8)
#pragma unroll
      for (int e = 0; e < 64; e += 32)
        if (k0 + i < N && q0 + lane + e < N) dst[(int64_t)(k0 + i) * a.pitch + q0 + lane + e] = tile[lane + e][i];
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
  const T* ob = o + b * d.o_st[0] + s * d.o_st[1] + h * d.o_st[3];
  const T* gb = d_o + b * d.do_st[0] + s * d.do_st[1] + h * d.do_st[3];
  const int pieces = d.D / 8;
  int flag = 0;
  for (int n0 = warp * 32; n0 < a.npad; n0 += 256) {
    const int i = n0 + lane;   // this lane's query once the sums are there
    const long long at = (long long)row * a.npad + i, idx = (long long)row * N + i;
    const bool in = i < N;
    const float m = in ? a.stats[idx] : 0.f, ll = in ? a.stats[total + idx] : 0.f;
    float part[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = lane & 3; c < pieces; c += 4) {
      uint4 x[4], y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = n0 + e * 8 + (lane >> 2);
        x[e] = y[e] = make_uint4(0, 0, 0, 0);
        if (n < N) {
          x[e] = reinterpret_cast<const uint4*>(ob + n * d.o_st[2])[c];
          y[e] = reinterpret_cast<const uint4*>(gb + n * d.do_st[2])[c];
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float u[8], w[8];
        unpack8<T>(x[e], u);
        unpack8<T>(y[e], w);
#pragma unroll
        for (int f = 0; f < 8; ++f) part[e] = fmaf(u[f], w[f], part[e]);
      }
    }
    __syncwarp();
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      part[e] += __shfl_xor_sync(0xffffffffu, part[e], 1);
      part[e] += __shfl_xor_sync(0xffffffffu, part[e], 2);
      const float v = __shfl_sync(0xffffffffu, part[e], (lane & 7) * 4);
      if (lane >> 3 == e) acc = v;
    }
    if (in && a.delta != nullptr) a.delta[idx] = acc;
    const float c = in ? -(m + ll) / d.scale : 0.f;
    const bool fits = RowFactors::fits<T>(m, c, acc);
    if (!fits) flag = 1;
    a.aug[at] = fits ? RowFactors::pack<T>(c, -acc) : make_uint4(0, 0, 0, 0);
    a.prep[at] = -m;
    a.prep[plane + at] = -ll * kLog2e;
    a.prep[2 * plane + at] = -acc;
  }
  flag = __syncthreads_or(flag);
  if (threadIdx.x == 0) a.large[row] = flag;
}

// dq = scale * sum over key blocks of the merged pass's partials ([nparts][B][S][N][H][D] contiguous), added in key
// block order in fp32; 8 elements per thread.
// (Rows are counted in 32 bits: 2^31 of them would not fit the device.  With the divisions in 64 bits and a load at a time
// 22.5 us at 301 x 301 residues, 4 heads of 32, 18.9 now; the bytes are 14.)
template <typename T>
__global__ void __launch_bounds__(256) attn_dq_sum_kernel(const T* __restrict__ part, int nparts, long long plane, TriAttnDesc d, T* __restrict__ dq) {
  dependent_trigger();
  const long long c = blockIdx.x * 256LL + threadIdx.x;
  if (c >= plane / 8) return;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  auto add = [&](const uint4& w) {
    float v[8];
    unpack8<T>(w, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += v[e];
  };
  const uint4* src = reinterpret_cast<const uint4*>(part) + c;
  const long long step = plane / 8;
  int p = 0;
  for (; p + 3 <= nparts; p += 3, src += 3 * step) {
    const uint4 w0 = src[0], w1 = src[step], w2 = src[2 * step];
    add(w0); add(w1); add(w2);
  }
  for (; p < nparts; ++p, src += step) add(*src);
  const unsigned dc = d.D / 8;
  unsigned z = (unsigned)(c / dc);
  const unsigned d8 = (unsigned)(c - (long long)z * dc), h = z % (unsigned)d.H; z /= (unsigned)d.H;
  const unsigned q = z % (unsigned)d.n_res; z /= (unsigned)d.n_res;
  const unsigned b = z / (unsigned)d.n_seq, s = z - b * (unsigned)d.n_seq;
  uint4 pk;
  pk.x = pack2<T>(acc[0] * d.scale, acc[1] * d.scale); pk.y = pack2<T>(acc[2] * d.scale, acc[3] * d.scale);
  pk.z = pack2<T>(acc[4] * d.scale, acc[5] * d.scale); pk.w = pack2<T>(acc[6] * d.scale, acc[7] * d.scale);
  T* row = dq + b * d.dq_st[0] + s * d.dq_st[1] + q * d.dq_st[2] + h * d.dq_st[3];
  reinterpret_cast<uint4*>(row)[d8] = pk;
}

__global__ void sum_partials_kernel(const float* partial, int nparts, long long n, float* out) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
  for (int p = 0; p < nparts; ++p) s += partial[p * n + i];
  out[i] = s;
}

// Can a tensor map reach the bias as it is?  Otherwise the tensor-core kernels read a copy with padded rows: rows whose
// length or start is not a multiple of 16 bytes (any N that is not a multiple of eight), broadcast heads or queries.
bool bias_strides_fit_tma(const TriAttnDesc* d) {
  return d->bias_st[0] % 8 == 0 && d->bias_st[1] % 8 == 0 && d->bias_st[2] % 8 == 0 && (d->bias_st[1] != 0 || d->H == 1) &&
         (d->bias_st[2] != 0 || d->n_res == 1);
}
bool bias_fits_tma(const TriAttnDesc* d, const void* bias) { return (reinterpret_cast<uintptr_t>(bias) & 15) == 0 && bias_strides_fit_tma(d); }
int bias_pitch(const TriAttnDesc* d) { return (d->n_res + 7) / 8 * 8; }
int bias_batches(const TriAttnDesc* d) { return d->bias_st[0] != 0 ? d->B : 1; }
size_t bias_copy_bytes(const TriAttnDesc* d) { return align_up((size_t)bias_batches(d) * d->H * d->n_res * bias_pitch(d) * 2); }

// boxes of `rows` queries x 64 keys over the bias itself or its copy (or of keys x queries over the transposed copy)
int bias_map(CUtensorMap* out, const void* bias, const void* copy, const TriAttnDesc* d, int rows) {
  const uint64_t nb = bias_batches(d), pitch = bias_pitch(d);
  const uint64_t dims[4] = {(uint64_t)d->n_res, (uint64_t)d->n_res, (uint64_t)d->H, nb};
  const uint64_t own[3] = {(uint64_t)d->bias_st[2], (uint64_t)d->bias_st[1], (uint64_t)d->bias_st[0]};
  const uint64_t packed[3] = {pitch, pitch * d->n_res, nb > 1 ? pitch * d->n_res * d->H : 0};
  const uint32_t box[4] = {64, (uint32_t)rows, 1, 1};
  return make_tmap(out, copy ? copy : bias, d->dtype, 4, dims, copy ? packed : own, box, 128);
}

// one row of the bias per block row: 16-bit elements to rows of `pitch`
__global__ void pad_bias_kernel(const uint16_t* __restrict__ in, int64_t st_b, int64_t st_h, int64_t st_q, int n, int H, int pitch,
                                long long rows, uint16_t* __restrict__ out) {
  dependent_trigger();
  const long long row = blockIdx.x * (long long)blockDim.y + threadIdx.y;   // (batch, head, query)
  const int q = row % n;
  const long long bh = row / n;
  if (row >= rows) return;
  const uint16_t* src = in + (bh / H) * st_b + (bh % H) * st_h + q * st_q;
  for (int k = threadIdx.x; k < n; k += blockDim.x) out[row * pitch + k] = src[k];
}

int launch_pad_bias(const TriAttnDesc* d, const void* bias, void* copy, cudaStream_t st) {
  const long long rows = (long long)bias_batches(d) * d->H * d->n_res;
  pad_bias_kernel<<<cdiv(rows, 4), dim3(64, 4), 0, st>>>(static_cast<const uint16_t*>(bias), d->bias_st[0], d->bias_st[1], d->bias_st[2],
                                                          d->n_res, d->H, bias_pitch(d), rows, static_cast<uint16_t*>(copy));
  TRI_LAUNCH_OK();
  return 0;
}

template <typename KernelT>
int set_dyn_smem(KernelT kern, int bytes) {
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return 0;
}

struct BwdWs {
  int* err;
  float *delta, *part, *prep, *mask_terms;
  uint4* aug;
  int* large;
  void *bias_t, *dq_part;
  void* bias_c;        // padded copy of the bias, behind the rest
};
int dbias_slots(const TriAttnDesc* d) { return (d->D <= 32 ? 2 : 1) * sm_count(); }   // CTAs of the dbias pass at a time
void carve_bwd(Arena& a, const TriAttnDesc* d, BwdWs* w) {
  const size_t rows = (size_t)d->B * d->n_seq * d->H, npad = ((size_t)d->n_res + 127) / 128 * 128;
  const bool merged = d->D <= 32;
  w->err = a.take<int>(128);
  w->delta = a.take<float>(merged ? 0 : rows * d->n_res);                        // read by the dQ pass
  w->part = a.take<float>(dbias_partial_bytes(d, dbias_slots(d)) / sizeof(float));
  w->bias_t = a.take<char>(bias_copy_bytes(d));                                  // transposed copy of the bias
  w->prep = a.take<float>(3 * rows * npad);                                      // padded per-row constants
  w->mask_terms = a.take<float>(2 * (size_t)d->B * d->n_seq * npad);             // additive key-mask terms
  w->aug = a.take<uint4>(rows * npad);                                           // row constants as factors
  w->large = a.take<int>(rows);                                                  // rows that go without them
  w->dq_part = a.take<uint16_t>(merged ? npad / 128 * rows * d->n_res * d->D : 0);   // merged pass: dQ per 128-key block
  w->bias_c = a.take<char>(0);
}

template <typename T, int HD>
int bwd_launch(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
               const uint8_t* mask, const void* o, const float* stats, const void* d_o, void* dq, void* dk, void* dv,
               float* dbias, const BwdWs& w, cudaStream_t st) {
  const long long rows = (long long)d->B * d->n_seq * d->H * d->n_res;
  const double pairs = (double)rows * d->n_res;
  const double tensor_bytes = 2.0 * d->B * d->n_seq * (double)d->n_res * d->H * d->D;
  const int npad = (d->n_res + 127) / 128 * 128;
  const long long prep_plane = (long long)d->B * d->n_seq * d->H * npad;
  {
    KernelTimer kt("tc_attn_delta", st, 0.0, 2.0 * tensor_bytes);
    PrepareArgs p;
    p.stats = stats; p.delta = HD == 32 ? nullptr : w.delta; p.prep = w.prep; p.mask_terms = w.mask_terms; p.aug = w.aug; p.large = w.large;
    p.err = w.err; p.mask = mask; p.bias = static_cast<const uint16_t*>(bias); p.bias_t = static_cast<uint16_t*>(w.bias_t);
    p.npad = npad; p.pitch = bias_pitch(d); p.tiles = cdiv(d->n_res, 64);
    p.transposes = bias != nullptr ? p.tiles * p.tiles * bias_batches(d) * d->H : 0;
    const long long planes = (long long)d->B * d->n_seq;
    const long long blocks = p.transposes + planes * d->H;
    attn_prepare_kernel<T><<<(unsigned)blocks, 256, 0, st>>>(*d, (const T*)o, (const T*)d_o, p);
    TRI_LAUNCH_OK();
  }
  const int kind = d->dtype == TRI_BF16 ? KIND_BF16 : KIND_F16;
  AttnBwdArgs a;
  a.B = d->B; a.S = d->n_seq; a.N = d->n_res; a.H = d->H; a.D = d->D; a.scale = d->scale;
  a.stats = stats; a.delta = w.delta; a.prep = w.prep; a.prep_plane = prep_plane; a.npad = npad; a.mask_terms = w.mask_terms; a.mask_plane = (long long)d->B * d->n_seq * npad;
  a.aug = w.aug; a.large = w.large; a.mask = mask; a.mask_st[0] = d->mask_st[0]; a.mask_st[1] = d->mask_st[1];
  a.bias_b_mul = d->bias_st[0] != 0 ? 1 : 0; a.err = w.err;
  a.row_chunks = 1;
  const int qblocks = (d->n_res + 127) / 128;
  CUtensorMap tq, tdo, tk, tv, tb;

  // ---- dK / dV -------------------------------------------------------------------------------
  TRI_TRY(qkv_tile_map(&tq, q, d, d->q_st, 64, HD));
  TRI_TRY(qkv_tile_map(&tdo, d_o, d, d->do_st, 64, HD));
  TRI_TRY(qkv_tile_map(&tk, k, d, d->k_st, 128, HD));
  TRI_TRY(qkv_tile_map(&tv, v, d, d->v_st, 128, HD));
  if (bias) {   // the dK/dV pass (thread = key) reads a transposed copy of the bias: [b][h][key][query]
    TRI_TRY(bias_map(&tb, bias, w.bias_t, d, 128));
  } else {
    tb = tq;
  }
  a.out0 = dk; a.out1 = dv;
  for (int i = 0; i < 4; ++i) { a.out0_st[i] = d->dk_st[i]; a.out1_st[i] = d->dv_st[i]; }
  a.idesc_a = make_idesc(kind, 128, 64, false, false);
  a.idesc_b = make_idesc(kind, 128, HD, false, true);
  a.idesc_c = make_idesc(kind, 128, HD, true, true);
  // Head dim 32: dK, dV and dQ come from one pass (dQ as per-key-block partials, summed below); head dim 64 has no
  // TMEM columns to spare for the dQ accumulator and keeps the separate dQ pass.
  constexpr bool kMerge = HD == 32;
  const long long dq_plane = (long long)d->B * d->n_seq * d->n_res * d->H * d->D;
  a.dq_part = w.dq_part; a.dq_part_plane = dq_plane;
  {
    auto kern = bias ? attn_bwd_dkdv_kernel<T, HD, true, kMerge> : attn_bwd_dkdv_kernel<T, HD, false, kMerge>;
    TRI_TRY(set_dyn_smem(kern, GeoC<HD>::SMEM));   // per-device attribute: set on every launch
    KernelTimer kt(kMerge ? "tc_attn_bwd_dkdvdq" : "tc_attn_bwd_dkdv", st, (kMerge ? 10.0 : 8.0) * pairs * d->D,
                   (kMerge ? 7.0 : 6.0) * tensor_bytes);
    launch_dependent(us_of_logits(pairs), kern, (unsigned)((long long)qblocks * d->B * d->n_seq * d->H), 320, GeoC<HD>::SMEM, st, tq, tdo, tk, tv, tb, a);
    TRI_LAUNCH_OK();
  }
  if (kMerge) {
    KernelTimer kt("tc_attn_dq_sum", st, 0.0, (qblocks + 1.0) * tensor_bytes);
    attn_dq_sum_kernel<T><<<cdiv(dq_plane / 8, 256), 256, 0, st>>>(static_cast<const T*>(w.dq_part), qblocks, dq_plane, *d,
                                                               static_cast<T*>(dq));
    TRI_LAUNCH_OK();
  }
  // ---- dQ ------------------------------------------------------------------------------------
  if (!kMerge) {
    CUtensorMap tq, tdo, tk, tv, tb;   // (the dK/dV pass's serve the dbias pass too)
    TRI_TRY(qkv_tile_map(&tq, q, d, d->q_st, 128, HD));
    TRI_TRY(qkv_tile_map(&tdo, d_o, d, d->do_st, 128, HD));
    TRI_TRY(qkv_tile_map(&tk, k, d, d->k_st, 64, HD));
    TRI_TRY(qkv_tile_map(&tv, v, d, d->v_st, 64, HD));
    if (bias) {
      const bool own = bias_fits_tma(d, bias);
      if (!own) TRI_TRY(launch_pad_bias(d, bias, w.bias_c, st));
      TRI_TRY(bias_map(&tb, bias, own ? nullptr : w.bias_c, d, 128));
    } else {
      tb = tq;
    }
    a.out0 = dq; a.out1 = nullptr;
    for (int i = 0; i < 4; ++i) a.out0_st[i] = d->dq_st[i];
    auto kern = bias ? attn_bwd_dq_kernel<T, HD, true> : attn_bwd_dq_kernel<T, HD, false>;
    TRI_TRY(set_dyn_smem(kern, GeoQ<HD>::SMEM));
    KernelTimer kt("tc_attn_bwd_dq", st, 2.0 * pairs * d->D, 5.0 * tensor_bytes);
    launch_dependent(us_of_logits(pairs), kern, (unsigned)((long long)qblocks * d->B * d->n_seq * d->H), 320, GeoQ<HD>::SMEM, st, tq, tdo, tk, tv, tb, a);
    TRI_LAUNCH_OK();
  }
  // ---- dbias ---------------------------------------------------------------------------------
  if (dbias != nullptr) {
    const int chunks = dbias_row_chunks(d, dbias_slots(d));
    const long long combos = (long long)qblocks * cdiv(d->n_res, 64) * d->B * d->H, nb = (long long)d->B * d->H * d->n_res * d->n_res;
    a.row_chunks = chunks;
    a.out0 = chunks > 1 ? w.part : dbias;
    a.idesc_a = make_idesc(kind, 128, 64, false, false);
    auto kern = attn_bwd_dbias_kernel<T, HD>;   // (with the dK/dV pass's maps)
    TRI_TRY(set_dyn_smem(kern, GeoB<HD>::SMEM));
    KernelTimer kt("tc_attn_bwd_dbias", st, 0.0, 4.0 * tensor_bytes);
    launch_dependent(us_of_logits(pairs), kern, (unsigned)(combos * chunks), 320, GeoB<HD>::SMEM, st, tq, tdo, tk, tv, tb, a);
    TRI_LAUNCH_OK();
    if (chunks > 1) TRI_TRY(launch_sum_partials(w.part, chunks, nb, dbias, st));
  }
  return 0;
}

bool forced_simt() {
  const char* e = getenv("TRI_B200_FORCE_SIMT");
  return e != nullptr && e[0] == '1';
}

// A tensor map needs strides that are non-zero multiples of 16 bytes on every axis with more than one entry; a
// broadcast (zero-stride) view therefore goes to the CUDA-core kernels, which take any stride.
bool strides_ok(const TriAttnDesc* d, const int64_t* st) {
  const int extent[4] = {d->B, d->n_seq, d->n_res, d->H};
  for (int i = 0; i < 4; ++i) {
    if (st[i] % 8 != 0) return false;
    if (st[i] == 0 && extent[i] > 1) return false;
  }
  return true;
}

template <typename T, int HD>
int fwd_launch(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
               const uint8_t* mask, void* o, float* stats, int* err, float* mask_terms, void* bias_c, cudaStream_t st) {
  CUtensorMap tq, tk, tv, tb;
  const bool rows = HD == 32 && d->n_seq >= 3 && attn_fwd_rows_fits(d);   // rows that share a bias tile
  AttnArgs a;
  a.B = d->B; a.S = d->n_seq; a.N = d->n_res; a.H = d->H; a.D = d->D; a.scale = d->scale;
  a.o = o; for (int i = 0; i < 4; ++i) a.o_st[i] = d->o_st[i];
  a.stats = stats; a.mask = mask; a.mask_st[0] = d->mask_st[0]; a.mask_st[1] = d->mask_st[1];
  a.bias_b_mul = d->bias_st[0] != 0 ? 1 : 0;
  const int kind = d->dtype == TRI_BF16 ? KIND_BF16 : KIND_F16;
  a.idesc_s = make_idesc(kind, 128, 128, false, false);
  a.idesc_pv = make_idesc(kind, 128, HD, false, true);
  a.status = err;
  const bool own = bias == nullptr || bias_fits_tma(d, bias);   // (else a copy with padded rows is the first kernel)
  if (!own) TRI_TRY(launch_pad_bias(d, bias, bias_c, st));
  if (bias != nullptr) TRI_TRY(bias_map(&tb, bias, own ? nullptr : bias_c, d, 128));
  if (rows) {
    const bool terms = wants_mask_terms(d);
    if (terms) TRI_TRY(launch_mask_terms(d, mask, mask_terms, err, st));
    TRI_TRY(qkv_tile_map(&tq, q, d, d->q_st, 128, 32));
    TRI_TRY(qkv_tile_map(&tk, k, d, d->k_st, 64, 32));
    TRI_TRY(qkv_tile_map(&tv, v, d, d->v_st, 64, 32));
    return attn_fwd_rows(d, tq, tk, tv, bias ? &tb : nullptr, a.bias_b_mul != 0, mask, terms ? mask_terms : nullptr, o, stats, err, own && !terms, st);
  }
  TRI_TRY(qkv_tile_map(&tq, q, d, d->q_st, 128, HD));
  TRI_TRY(qkv_tile_map(&tk, k, d, d->k_st, 128, HD));
  TRI_TRY(qkv_tile_map(&tv, v, d, d->v_st, 128, HD));
  if (bias == nullptr) tb = tq;
  const long long blocks = (long long)((d->n_res + 127) / 128) * d->B * d->n_seq * d->H;
  const double pairs = (double)d->B * d->n_seq * d->H * d->n_res * (double)d->n_res;
  KernelTimer kt("tc_attn_fwd", st, 4.0 * pairs * d->D, 2.0 * 4.0 * d->B * d->n_seq * (double)d->n_res * d->H * d->D);
  auto kern = bias != nullptr ? attn_fwd_tc_kernel<T, HD, true> : attn_fwd_tc_kernel<T, HD, false>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Geo<HD>::SMEM));
  sms_beside_attention() = (int)std::max(0LL, sm_count() - ((blocks - 1) % ((HD == 32 ? 2LL : 1LL) * sm_count()) + 1));   // (32: two CTAs per SM)
  launch_dependent(own ? kLaunchPlainly : us_of_logits(pairs), kern, (unsigned)std::min<long long>({blocks, 2LL * sm_count(), kStatusCtas}), 320, Geo<HD>::SMEM, st, tq, tk, tv, tb, a);
  TRI_LAUNCH_OK();
  return 0;
}

}  // namespace

int& sms_beside_attention() {
  static thread_local int sms = 0;
  return sms;
}

bool wants_mask_terms(const TriAttnDesc* d) {
  return us_of_logits((double)d->B * d->n_seq * d->H * d->n_res * (double)d->n_res) >= kEarlyStartUs;
}
int launch_mask_terms(const TriAttnDesc* d, const uint8_t* mask, float* out, int* err, cudaStream_t st) {
  const int npad = (d->n_res + 127) / 128 * 128;
  mask_terms_kernel<<<cdiv((long long)d->B * d->n_seq * npad, 256), 256, 0, st>>>(mask, d->mask_st[0], d->mask_st[1], d->B, d->n_seq, d->n_res, npad, out, err);
  TRI_LAUNCH_OK();
  return 0;
}

// Row chunks until the CTAs fill the GPU, as few as give the fewest rows in a row: rounds of CTAs times rows of a chunk.  (One
// round more for the last few CTAs costs as much as the rounds before: 301 residues, 60 tiles, 5 chunks 113 us, 4 chunks 84.)
int dbias_row_chunks(const TriAttnDesc* d, int slots) {
  const long long combos = (long long)cdiv(d->n_res, 128) * cdiv(d->n_res, 64) * d->B * d->H;
  int chunks = 1;
  long long best = -1;
  for (int ch = 1; ch <= std::min(8, std::max(1, d->n_seq / 2)); ++ch) {
    const long long steps = (combos * ch + slots - 1) / slots * cdiv(d->n_seq, ch);
    if (best < 0 || steps * 10 < best * 9) { best = steps; chunks = ch; }   // (each chunk costs a partial sum)
  }
  return chunks;
}

size_t dbias_partial_bytes(const TriAttnDesc* d, int slots) {
  const int chunks = dbias_row_chunks(d, slots);
  return chunks > 1 ? align_up((size_t)chunks * d->B * d->H * d->n_res * d->n_res * sizeof(float)) : 0;
}

int launch_sum_partials(const float* partial, int chunks, long long n, float* out, cudaStream_t st) {
  sum_partials_kernel<<<cdiv(n, 256), 256, 0, st>>>(partial, chunks, n, out);
  TRI_LAUNCH_OK();
  return 0;
}

int qkv_tile_map(CUtensorMap* out, const void* p, const TriAttnDesc* d, const int64_t* st, int rows, int width) {
  const uint64_t dims[5] = {(uint64_t)d->D, (uint64_t)d->H, (uint64_t)d->n_res, (uint64_t)d->n_seq, (uint64_t)d->B};
  const uint64_t str[4] = {(uint64_t)st[3], (uint64_t)st[2], (uint64_t)st[1], (uint64_t)st[0]};
  const uint32_t box[5] = {(uint32_t)width, 1, (uint32_t)rows, 1, 1};
  return make_tmap(out, p, d->dtype, 5, dims, str, box, width * 2);
}

// Logits from which on odd lengths (and head dims other than 32 and 64) come here.  Below, calls stay on the CUDA-core kernels,
// which keep P and dS in fp32 (bf16, 203 residues: outputs within 1.7e-3 of fp64, 2.3e-3 here; gradients 1.8e-3 and 3.0e-3).
// The lines lie just above the largest shapes that the tests hold to those kernels (16 rows of 100 residues, 4 heads: 640,000
// logits; 8 rows of 8, 2 heads of 8), not where the times cross.  Forward alone, us on the CUDA cores / here: 53 x 53 residues,
// 4 heads 14 / 18; 16 x 100 16 / 16; 1 x 201, 16 heads 31 / 16.  All kernels of forward and backward: 137 / 67, 132 / 61,
// 156 / 65; 8 x 8, 2 heads of 8 93 / 55.  At 301 x 301 it is 10 ms against 0.45.
constexpr double kMinRagged = 655360.0, kMinPaddedDim = 4096.0;

bool attn_fwd_supported(const TriAttnDesc* d) {
  if (forced_simt()) return false;
  if (d->dtype != TRI_BF16 && d->dtype != TRI_F16) return false;
  if (d->D % 8 != 0 || d->D > 64 || d->n_res > 16384) return false;
  // Head dims below a tile width are padded with zeros by the copies, odd lengths read a copy of the bias with padded rows.
  const double logits = (double)d->B * d->n_seq * d->H * d->n_res * d->n_res;
  if (logits < (d->n_res % 8 != 0 ? kMinRagged : d->D != 32 && d->D != 64 ? kMinPaddedDim : 0.0)) return false;
  if (!strides_ok(d, d->q_st) || !strides_ok(d, d->k_st) || !strides_ok(d, d->v_st) || !strides_ok(d, d->o_st)) return false;
  if ((long long)((d->n_res + 127) / 128) * d->B * d->n_seq * d->H > 2147483647LL) return false;
  return true;
}

bool attn_bwd_supported(const TriAttnDesc* d) {
  return attn_fwd_supported(d) && strides_ok(d, d->do_st) && strides_ok(d, d->dq_st) && strides_ok(d, d->dk_st) &&
         strides_ok(d, d->dv_st) && d->n_seq <= 65535;
}

// everything but the padded copy of the bias, which comes last
static size_t attn_ws_base(const TriAttnDesc* d, int is_bwd) {
  // (the status, the key-mask terms)
  if (!is_bwd) return 8 + kStatusCtas + (wants_mask_terms(d) ? align_up((size_t)d->B * d->n_seq * ((d->n_res + 127) / 128 * 128) * sizeof(float)) : 0);
  Arena a(nullptr, 0);
  BwdWs w;
  carve_bwd(a, d, &w);
  return a.off;
}

// (The descriptor does not say where the bias starts: a copy for that reason alone is not counted here, see attn_bias_has_room.)
size_t attn_ws_bytes(const TriAttnDesc* d, int is_bwd) {
  return attn_ws_base(d, is_bwd) + (bias_strides_fit_tma(d) ? 0 : bias_copy_bytes(d));
}

// a bias that a copy was planned for or that needs none, or a workspace with room for one
bool attn_bias_has_room(const TriAttnDesc* d, const void* bias, size_t ws_size, int is_bwd) {
  return bias == nullptr || bias_fits_tma(d, bias) || !bias_strides_fit_tma(d) || ws_size >= attn_ws_base(d, is_bwd) + bias_copy_bytes(d);
}

int attn_forward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
                 const uint8_t* mask, void* o, float* lse, void* ws, size_t ws_size, cudaStream_t st) {
  if (ws == nullptr || ws_size < attn_ws_bytes(d, 0)) return fail(TRI_ERR_WORKSPACE, "attention forward workspace too small");
  int* err = static_cast<int*>(ws);
  float* mt = reinterpret_cast<float*>(static_cast<char*>(ws) + 8 + kStatusCtas);
  void* bc = static_cast<char*>(ws) + attn_ws_base(d, 0);
  if (d->dtype == TRI_BF16) {
    if (d->D <= 32) return fwd_launch<__nv_bfloat16, 32>(d, q, k, v, bias, mask, o, lse, err, mt, bc, st);
    return fwd_launch<__nv_bfloat16, 64>(d, q, k, v, bias, mask, o, lse, err, mt, bc, st);
  }
  if (d->D <= 32) return fwd_launch<__half, 32>(d, q, k, v, bias, mask, o, lse, err, mt, bc, st);
  return fwd_launch<__half, 64>(d, q, k, v, bias, mask, o, lse, err, mt, bc, st);
}

int attn_backward(const TriAttnDesc* d, const void* q, const void* k, const void* v, const void* bias,
                  const uint8_t* mask, const void* o, const float* lse, const void* d_o, void* dq, void* dk,
                  void* dv, float* dbias, void* ws, size_t ws_size, cudaStream_t st) {
  if (ws == nullptr || ws_size < attn_ws_bytes(d, 1)) return fail(TRI_ERR_WORKSPACE, "attention backward workspace too small");
  Arena a(ws, ws_size);
  BwdWs w;
  carve_bwd(a, d, &w);
  if (d->dtype == TRI_BF16) {
    if (d->D <= 32) return bwd_launch<__nv_bfloat16, 32>(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, w, st);
    return bwd_launch<__nv_bfloat16, 64>(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, w, st);
  }
  if (d->D <= 32) return bwd_launch<__half, 32>(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, w, st);
  return bwd_launch<__half, 64>(d, q, k, v, bias, mask, o, lse, d_o, dq, dk, dv, dbias, w, st);
}

}  // namespace tc
}  // namespace tri

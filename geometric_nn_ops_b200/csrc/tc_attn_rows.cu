// Forward triangle attention, 16-bit types and fp32 with TF32 products, head dim up to 32: three rows of the pair tensor
// (fp32: two) share a pair-bias tile.
//
// The pair bias depends on (head, query, key) only, so rows s .. s+2 of one head and 128-query block read the same
// bias tiles.  A CTA takes such a triple: three groups of four softmax warps, one row each, walk the key axis in steps
// of 64 keys; the bias tile of a step comes to shared memory once for the three of them.  Otherwise a group is on its
// own: its Q, K, V tiles, its 160 TMEM columns and the lane that issues its copies and products.
//
// Per step and thread (one query row, 64 keys), sixteen logits at a time:
//   x = (S scale + mask term) + bias -> P = 2^(x log2e - m log2e), 16 bit -> O += P V.
// The logits are rounded as the backward rounds them, in natural units: beside a bias of -1e8 a row's other terms are lost
// to both, and in units of log 2 the type's lowest value would overflow.
// One sweep without a maximum: P is formed against the reference m of the row (the largest of its first four logits to
// start with).  P, its sum and O are floating point, so a reference that lags the maximum by a factor of up to kTooBig
// loses nothing; the sum of a step shows whether a row has outgrown it, and then O and the sum are rescaled and the step
// is done again.  S stays in TMEM until the check: P is stored over it afterwards.
// m log2e is rounded, so every P of a row carries the factor 2^r, r = m log2e - fl(m log2e), which the statistics take out
// again: 1 within 2^-12 where |m| is below 2^11.  A warp with a row where it is not (masked, or held up, by its bias or its
// mask) does its first step again, and from then on forms P from the differences, 2^((x - m) log2e): one more packed
// instruction per two logits.
//
// S is double buffered and P(c) takes the columns of S(c).  After P(c) the issuing lane sends P V(c) and S(c + 2),
// which run in that order, so S(c + 1) is there before a thread asks for it and one arrival per step (p_ready) is all
// that the softmax warps owe.  With S single buffered each step waited about 600 clocks for the next product, and the
// waiting warps' polling took half of all issue slots.
//
// What bounds it: the instructions of a step (about 330 per warp, three warps to a sub-partition), then the waits a row's four warps,
// which run on four sub-partitions, have for one another.  A quarter of the exponentials as polynomials on the FMA pipe: 714 -> 784 us.
// The bias added by two additions that widen it, in place of two conversions and a packed addition: 714 -> 689.  N = 768, 4
// heads, bf16: 0.69 ms, 62 % of the exponential pipe (which also converts), against 1.05 ms and 41 % for the kernel with two CTAs per SM, two threads per row and a maximum per step (which
// also read 2 bytes of bias per logit from L2; here 0.67).
#include <algorithm>
#include <type_traits>

#include "tc_attn_common.cuh"
#include "tc_attn_rows.cuh"
#include "tc_paths.cuh"

namespace tri {
namespace tc {

namespace {

// fp32: tiles are twice as large, which leaves room for two rows per CTA; operands were rounded to TF32 before, P goes into the
// product as two TF32 terms.  P takes one column per key and so replaces S in place; V is read across its rows, which 32-bit operands can only be
// in the swizzle with 32-byte atoms.
template <typename T> struct RowsCfg {
  static constexpr bool F32 = sizeof(T) == 4;
  static constexpr int kGroups = F32 ? 2 : 3;      // rows per CTA
  static constexpr int kBiasStages = F32 ? 2 : 4;
  static constexpr int kThreads = (4 * kGroups + kGroups + 1) * 32;   // softmax warps, issuing warps, one warp for the bias tiles
  static constexpr int kQ = F32 ? 2 : 3;           // Q buffers (two suffice where a row has two key steps)
  static constexpr int RB = 32 * sizeof(T);        // bytes of a Q, K or V row
  static constexpr int TQ = 128 * RB, TK = 64 * RB, TB = 128 * 64 * sizeof(T);   // bytes: Q tile, K or V tile, bias tile
  static constexpr int OFF_BIAS = 0;
  static constexpr int OFF_Q = OFF_BIAS + kBiasStages * TB;     // [group][kQ]
  static constexpr int OFF_K = OFF_Q + kGroups * kQ * TQ;       // [group][3]
  static constexpr int OFF_V = OFF_K + kGroups * 3 * TK;        // [group][3]
  static constexpr int OFF_M = OFF_V + kGroups * 3 * TK;        // [bias stage][group] x 64 mask terms
  static constexpr int OFF_BAR = OFF_M + kBiasStages * kGroups * 256;
  static constexpr int OFF_ERR = OFF_BAR + 1020;          // this CTA's status
  static constexpr int SMEM = OFF_BAR + 1024 + 1024;
  static constexpr int PC = F32 ? 64 : 32;         // columns of P: a step's 64 keys
  static constexpr int KS = F32 ? 4 : 2;           // products of a step's S: 32 channels, 32 bytes each
  static constexpr int KV = F32 ? 8 : 4;           // ... of its P V: 64 keys
  static constexpr uint32_t HI = F32 ? desc_hi(8 * 128, 2) : desc_hi(8 * 64, 4);        // Q, K: SWIZZLE_128B, SWIZZLE_64B
  static constexpr uint32_t HI_V = F32 ? desc_hi(512, 1) : desc_hi(8 * 64, 4);          // V across its rows
  static constexpr int kind = F32 ? KIND_TF32 : KIND_F16;
  static constexpr int kVecBits = F32 ? 2 : 3, kVec = 1 << kVecBits;   // elements of a 16-byte piece
};
constexpr float kLn2 = 0.6931471805599453f;

struct RowsArgs {
  int B, S, N, H, D;
  float scale;
  void* o;
  int64_t o_st[4];
  float* stats;              // [2][B][S][H][N]: row maximum, log row sum
  const float* mask_terms;   // [B][S][npad] (mask_term), or null: made here
  int npad;
  int bias_b_mul;
  int rows_per_item;         // groups in use (fewer where a triple per CTA would leave SMs idle)
  uint32_t idesc_s, idesc_pv;
  int* status;
  const uint8_t* mask;       // [B][S][N], or null
  int64_t mask_st[2];
};

// barriers of one group
struct GroupBars {
  uint64_t first[2];  // Q, K of the first two S products
  uint64_t in[3];     // [c % 3]: what the issuing lane needs at step c
  uint64_t mma[2];    // [c & 1]: S(c) is in TMEM and P V(c - 2) is done
  uint64_t p_ready[2];   // [c & 1]: the four warps have read S(c) and its mask terms and stored P(c); they may do so for
                         // step c + 1 before the issuing lane has seen step c, hence two
};

// tcgen05.wait::ld that the registers of the load pass through, so that no use of them can move above it
__device__ __forceinline__ void ld_wait16(uint32_t (&v)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]),
                 "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])::"memory");
}

// TERMS: the mask terms were made before
template <typename T, bool HB, bool TERMS>
__global__ void __launch_bounds__(RowsCfg<T>::kThreads, 1)
attn_fwd_rows_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmBias, const RowsArgs a) {
  using M = RowsCfg<T>;
  constexpr int kGroups = M::kGroups, kBiasStages = M::kBiasStages;
  constexpr float kTooBig = std::is_same<T, __half>::value ? 32768.0f : 1.152921504606847e18f;   // fp16 tops out at 2^16; 2^60
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  GroupBars* bars = reinterpret_cast<GroupBars*>(smem + M::OFF_BAR);
  uint64_t* b_full = reinterpret_cast<uint64_t*>(bars + kGroups);   // [kBiasStages]
  uint64_t* b_free = b_full + kBiasStages;                          // [kBiasStages]: the softmax warps of the groups in use
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(b_free + kBiasStages);
  // Without TERMS no kernel has cleared the call's status: see leave_status.  (Formed where it is used: as a variable 41.1 us in place
  // of 40.8 at N = 256.)
  auto err = [&]() { return TERMS ? a.status : reinterpret_cast<int*>(smem + M::OFF_ERR); };

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qblocks = (a.N + 127) / 128, nk = (a.N + 63) / 64;
  const int R = a.rows_per_item, triples = (a.S + R - 1) / R;
  const long long items = (long long)qblocks * a.H * triples * a.B;
  const int my_items = blockIdx.x < items ? (int)((items - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
  struct Item { int q0, h, s0, b; };
  auto item_of = [&](int n) {
    unsigned z = blockIdx.x + (unsigned)n * gridDim.x;
    Item it;
    it.q0 = (int)(z % (unsigned)qblocks) * 128; z /= (unsigned)qblocks;
    it.h = (int)(z % (unsigned)a.H); z /= (unsigned)a.H;
    it.s0 = (int)(z % (unsigned)triples) * R;
    it.b = (int)(z / (unsigned)triples);
    return it;
  };

  if (tid == 0) {
    for (int g = 0; g < kGroups; ++g) {
      mbar_init(&bars[g].first[0], 1); mbar_init(&bars[g].first[1], 1);
      for (int i = 0; i < 3; ++i) mbar_init(&bars[g].in[i], 1);
      mbar_init(&bars[g].mma[0], 1); mbar_init(&bars[g].mma[1], 1); mbar_init(&bars[g].p_ready[0], 4); mbar_init(&bars[g].p_ready[1], 4);
    }
    for (int i = 0; i < kBiasStages; ++i) { mbar_init(&b_full[i], TERMS ? 1 : 1 + 8 * kGroups); mbar_init(&b_free[i], 4 * R); }
    mbar_fence_init();
    if (!TERMS) *err() = 0;
  }
  if (warp == 0) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_trigger();
  if constexpr (M::F32) dependent_wait();   // (else q, k, v are the caller's: only a copied bias comes from before)
  constexpr uint32_t COLS = M::F32 ? 224 : 160, COL_O = 128, COL_LO = 160;   // a group's columns: S / P of even and odd steps at
                                                                             // 0 and 64, O, (fp32) what P's upper bits leave
  bool ok = true;
  // 512 threads of 128 registers: the issuing warps give some of theirs to the softmax warps (12 x 152 + 4 x 56 = 16 x 128), whose step
  // did not fit: 721 -> 714 us at N = 768, 4 heads (with the additions of `add_wide` 730 at 144 and 72, 695 at 152 and 48, 689 so;
  // at 160 and 32 the issuing warps spill: 775).
  if constexpr (!M::F32) {
    static_assert(M::kThreads == 512 && kGroups == 3);
    if (warp >= 4 * kGroups) regs_dec<56>();
    else regs_inc<152>();
  }

  if (warp == 5 * kGroups) {
    // ------------------------------------ bias tiles and mask terms --------------------------------
    if constexpr (TERMS) {
      if (lane == 0) {
        dependent_wait();
        int stg = 0;
        uint32_t ph = 0;
        for (int n = 0; n < my_items && ok; ++n) {
          const Item it = item_of(n);
          for (int j = 0; j < nk; ++j) {
            ok = mbar_wait_relaxed(&b_free[stg], ph ^ 1, err(), 51);
            if (!ok) break;
            const int rows = min(R, a.S - it.s0);
            mbar_expect_tx(&b_full[stg], (HB ? M::TB : 0) + rows * 256);
            for (int g = 0; g < rows; ++g)
              bulk_load(smem + M::OFF_M + (stg * kGroups + g) * 256, a.mask_terms + ((long long)it.b * a.S + it.s0 + g) * a.npad + j * 64, 256, &b_full[stg]);
            if (HB) tma_load_4d(smem + M::OFF_BIAS + stg * M::TB, &tmBias, &b_full[stg], j * 64, it.q0, it.h, it.b * a.bias_b_mul);
            if (HB && M::F32) tma_load_4d(smem + M::OFF_BIAS + stg * M::TB + M::TB / 2, &tmBias, &b_full[stg], j * 64 + 32, it.q0, it.h, it.b * a.bias_b_mul);
            if (++stg == kBiasStages) { stg = 0; ph ^= 1; }
          }
        }
      }
    } else {
      // The terms of short calls are made here, which saves a launch: eight lanes have the 64 keys of a row's step, eight keys each;
      // their mask bytes are fetched a step ahead, as three aligned words of which the funnel shift takes the eight bytes.  The
      // softmax warps of the sub-partition miss the instructions: N = 768 took 761 us so and 729 with terms made before, launch
      // included; N = 256 42.3 and 42.9.  Every lane that writes terms arrives for itself: the lanes then need not meet, and one whose
      // wait runs out may leave alone (meeting at each step, with a vote on the waits: N = 256 40.1 us in place of 39.7, 301 79.1 and
      // 76.0; lane 0 waiting for all 41.2 and 79.8).
      dependent_wait();
      int stg = 0;
      uint32_t ph = 0, w[3] = {};
      const int g = lane >> 3, k_lane = (lane & 7) * 8;
      const bool owner = lane < 8 * kGroups;
      const uint8_t* row = nullptr;
      auto row_of = [&](const Item& it) {
        const bool live = a.mask != nullptr && owner && g < R && it.s0 + g < a.S;
        return live ? a.mask + it.b * a.mask_st[0] + (it.s0 + g) * a.mask_st[1] + k_lane : nullptr;
      };
      auto fetch = [&](int j) {
        w[0] = w[1] = w[2] = 0x01010101u;
        if (row == nullptr) return;
        const uint8_t* at = row + j * 64;
        const int off = (int)(reinterpret_cast<uintptr_t>(at) & 3), left = a.N - j * 64 - k_lane + off;   // bytes from the first word on
        const uint32_t* p = reinterpret_cast<const uint32_t*>(at - off);
        if (left > off) w[0] = p[0];
        if (left > 4) w[1] = p[1];
        if (left > 8 && off > 0) w[2] = p[2];
      };
      Item it = item_of(0);
      if (my_items > 0) { row = row_of(it); fetch(0); }
      for (int n = 0; n < my_items && ok; ++n) {
        const Item after = item_of(n + 1 < my_items ? n + 1 : n);
        for (int j = 0; j < nk; ++j) {
          ok = mbar_wait_relaxed(&b_free[stg], ph ^ 1, err(), 51);
          if (!ok) break;
          if (lane == 0) {
            mbar_expect_tx(&b_full[stg], HB ? M::TB : 0);
            if (HB) tma_load_4d(smem + M::OFF_BIAS + stg * M::TB, &tmBias, &b_full[stg], j * 64, it.q0, it.h, it.b * a.bias_b_mul);
            if (HB && M::F32) tma_load_4d(smem + M::OFF_BIAS + stg * M::TB + M::TB / 2, &tmBias, &b_full[stg], j * 64 + 32, it.q0, it.h, it.b * a.bias_b_mul);
          }
          const uint32_t sh = (uint32_t)(reinterpret_cast<uintptr_t>(row) & 3) * 8;
          const uint32_t lo = __funnelshift_r(w[0], w[1], sh), hi = __funnelshift_r(w[1], w[2], sh);
          float term[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) term[e] = ((e < 4 ? lo : hi) & (0xffu << (8 * (e & 3)))) != 0 ? 0.0f : -kMaskSentinel;
          if (j * 64 + 64 > a.N) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (j * 64 + k_lane + e >= a.N) term[e] = -INFINITY;
          }
          if (owner) {
            float4* to = reinterpret_cast<float4*>(smem + M::OFF_M + (stg * kGroups + g) * 256 + k_lane * 4);
            to[0] = make_float4(term[0], term[1], term[2], term[3]);
            to[1] = make_float4(term[4], term[5], term[6], term[7]);
            mbar_arrive(&b_full[stg]);
          }
          if (j + 1 == nk) row = row_of(after);
          fetch(j + 1 < nk ? j + 1 : 0);
          if (++stg == kBiasStages) { stg = 0; ph ^= 1; }
        }
        it = after;
      }
    }
  } else if (warp >= 4 * kGroups) {
    // ------------------------------------ copies and products of group g --------------------------
    // The whole warp runs this code and one lane issues: every index is warp-uniform and stays in uniform registers.
    const int g = warp - 4 * kGroups;
    if (g < R) {
      GroupBars& gb = bars[g];
      uint8_t* sQ = smem + M::OFF_Q + g * M::kQ * M::TQ;
      uint8_t* sK = smem + M::OFF_K + g * 3 * M::TK;
      uint8_t* sV = smem + M::OFF_V + g * 3 * M::TK;
      const uint32_t t0 = tmem_base + g * COLS;
      const bool leader = elect_one();
      const uint32_t q_lo = desc_lo(smem_u32(sQ), 16), k_lo = desc_lo(smem_u32(sK), 16), v_lo = desc_lo(smem_u32(sV), 64 * M::RB);
      int total = 0;                        // steps of this group: rows beyond S are left out
      for (int n = 0; n < my_items; ++n) total += item_of(n).s0 + g < a.S ? nk : 0;
      // a position in the group's stream: item, key step, ring stage, Q buffer
      struct Cursor { Item it; int n, j, left, stg, q; };
      auto start = [&](Cursor& u) {         // the item at (or after) n that this group has a row in
        while (u.it.s0 + g >= a.S) u.it = item_of(++u.n);
      };
      auto next = [&](Cursor& u) {
        --u.left;
        if (++u.stg == 3) u.stg = 0;
        if (++u.j == nk) {
          u.j = 0;
          if (++u.q == M::kQ) u.q = 0;
          if (u.left > 0) { u.it = item_of(++u.n); start(u); }
        }
      };
      Cursor kc{item_of(0), 0, 0, total, 0, 0};
      if (total > 0) start(kc);
      Cursor vc = kc;
      // What step c needs besides P(c) -- V(c), and K(c + 2) with its Q for S(c + 2) -- arrives on one barrier, in[c % 3].
      auto load = [&](uint64_t* bar, bool k, bool v) {
        if (leader) {
          mbar_expect_tx(bar, (k ? M::TK + (kc.j == 0 ? M::TQ : 0) : 0) + (v ? M::TK : 0));
          if (k && kc.j == 0) tma_load_5d(sQ + kc.q * M::TQ, &tmQ, bar, 0, kc.it.h, kc.it.q0, kc.it.s0 + g, kc.it.b);
          if (k) tma_load_5d(sK + kc.stg * M::TK, &tmK, bar, 0, kc.it.h, kc.j * 64, kc.it.s0 + g, kc.it.b);
          if (v) tma_load_5d(sV + vc.stg * M::TK, &tmV, bar, 0, vc.it.h, vc.j * 64, vc.it.s0 + g, vc.it.b);
        }
        if (k) next(kc);
        if (v) next(vc);
      };
      int sj = 0, sq = 0, sk = 0;           // key step, Q buffer and K stage of the next S product
      auto issue_s = [&](uint32_t t) {
        const uint32_t s_q = q_lo + sq * (M::TQ >> 4), s_k = k_lo + sk * (M::TK >> 4);
        if (leader) {
#pragma unroll
          for (int ks = 0; ks < M::KS; ++ks)
            umma<M::kind>(t, desc_join(s_q + ks * 2, M::HI), desc_join(s_k + ks * 2, M::HI), a.idesc_s, ks > 0);
        }
        if (++sj == nk) { sj = 0; if (++sq == M::kQ) sq = 0; }
        if (++sk == 3) sk = 0;
      };
      for (int c = 0; c < 2 && c < total; ++c) load(&gb.first[c], true, false);
      if (total > 0) load(&gb.in[0], total > 2, true);
      for (int c = 0; c < 2 && c < total; ++c) {
        ok = mbar_wait(&gb.first[c], 0, err(), 52) && ok;
        tc_fence_after_sync();
        issue_s(t0 + c * 64);
        if (leader) umma_commit(&gb.mma[c]);
      }
      int j = 0, stg = 0;                   // key step and ring stage (V and barrier) of step c
      uint32_t ph = 0;
      for (int c = 0; c < total && ok; ++c) {
        const bool more = c + 2 < total;
        const uint32_t v_at = v_lo + stg * (M::TK >> 4), tp = t0 + (c & 1) * 64, first = j > 0 ? 1u : 0u;
        ok = mbar_wait_relaxed(&gb.in[stg], ph, err(), 53) && ok;
        // every warp has stored P(c): it had waited for S(c), which followed P V(c - 2): the K stage of c and the V stage
        // of c - 2 are free
        ok = mbar_wait_relaxed(&gb.p_ready[c & 1], (c >> 1) & 1, err(), 55) && ok;
        tc_fence_after_sync();
        if (leader) {
#pragma unroll
          for (int kk = 0; kk < M::KV; ++kk)
            umma_ts<M::kind>(t0 + COL_O, tp + kk * 8, desc_join(v_at + kk * 64, M::HI_V), a.idesc_pv, kk > 0 ? 1u : first);
          if constexpr (M::F32) {
#pragma unroll
            for (int kk = 0; kk < M::KV; ++kk) umma_ts<M::kind>(t0 + COL_O, t0 + COL_LO + kk * 8, desc_join(v_at + kk * 64, M::HI_V), a.idesc_pv, 1u);
          }
        }
        if (more) issue_s(tp);               // into the columns P V(c) reads: products of one thread run in order
        if (leader) umma_commit(&gb.mma[c & 1]);
        if (++stg == 3) { stg = 0; ph ^= 1; }
        if (c + 1 < total) load(&gb.in[stg], c + 3 < total, true);   // V(c + 1), K(c + 3)
        if (++j == nk) j = 0;
      }
    }
  } else {
    // ------------------------------------ softmax of group g --------------------------------------
    const int g = warp >> 2, r = tid & 127;
    GroupBars& gb = bars[g];
    const uint32_t t_row = tmem_base + g * COLS + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t mask_s = smem_u32(smem + M::OFF_M) + g * 256, bias_row = smem_u32(smem + M::OFF_BIAS) + r * 128 + ((r & 7) << 4);
    const float2 sc2 = splat(a.scale), l2e2 = splat(kLog2e);
    // the exponent r of the factor that P carries against the reference m (see the top), and whether a row goes without
    auto residue = [](float m) { return fmaf(m, kLog2e, -(m * kLog2e)); };
    auto large = [&](float m) { return !(fabsf(residue(m)) <= 0.000244140625f); };
    auto factor = [&](float m) { return large(m) ? 0.0f : residue(m); };
    int c = 0, bstg = 0;
    uint32_t bph = 0;
    bool early_s = false, early_b = false;
    // the row that is finished but for its last P V: statistics, where its results go
    bool pend = false;
    float pm = 0.f, pl = 0.f, pseen = 0.f;
    int po = -1, pstat = 0;   // O row in 16-byte pieces, -1 where the query is beyond N; row of the statistics
    // O and the statistics of the row, once P V of its last step `cl` is done; no later P V can have been issued yet
    auto finish = [&](int cl) {
      if (!mbar_wait(&gb.mma[cl & 1], ((cl >> 1) + 1) & 1, err(), 59)) ok = false;
      tc_fence_after_sync();
      uint32_t o[2][16];
      tmem_ld_32x16(t_row + COL_O, o[0]);
      tmem_ld_32x16(t_row + COL_O + 16, o[1]);
      ld_wait16(o[0]);
      ld_wait16(o[1]);
      if (po >= 0 && ok) {
        const float inv = 1.0f / pl;
#pragma unroll
        for (int h = 0; h < 32 / M::kVec; ++h) {
          if (h * M::kVec < a.D) {
            if constexpr (M::F32) {
              auto f = [&](int i) { return __uint_as_float(o[h >> 2][(h & 3) * 4 + i]) * inv; };
              (reinterpret_cast<float4*>(a.o) + po)[h] = make_float4(f(0), f(1), f(2), f(3));
            } else {
              uint4 pk;
              auto f = [&](int i) { return __uint_as_float(o[h >> 1][(h & 1) * 8 + i]) * inv; };
              pk.x = pack2<T>(f(0), f(1)); pk.y = pack2<T>(f(2), f(3)); pk.z = pack2<T>(f(4), f(5)); pk.w = pack2<T>(f(6), f(7));
              (reinterpret_cast<uint4*>(a.o) + po)[h] = pk;
            }
          }
        }
        // The largest of the steps' sums over 64 keys is 1 to 64 times the largest P, so that m plus log(sum / 64) lies at
        // most 6 ln 2 below the row's maximum.  What m takes on of that (nothing, beside a large m) leaves the logarithm.
        const float top = pm + fmaxf(__log2f(pseen) - 6.0f, 0.f) * kLn2;
        a.stats[pstat] = top;
        a.stats[(long long)a.B * a.S * a.H * a.N + pstat] = (logf(pl) - factor(pm) * kLn2) - (top - pm);
      }
    };
    for (int n = 0; g < R && n < my_items && __all_sync(0xffffffffu, ok); ++n) {
      const Item it = item_of(n);
      if (it.s0 + g >= a.S) {   // no row for this group: let the bias tiles pass
        for (int j = 0; j < nk && ok; ++j) {
          ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&b_full[bstg], bph, err(), 57));
          if (lane == 0) mbar_arrive(&b_free[bstg]);
          if (++bstg == kBiasStages) { bstg = 0; bph ^= 1; }
        }
        early_b = false;
        continue;
      }
      float m = -INFINITY, l = 0.f;   // reference, sum of P
      float seen = 0.f;               // largest sum of a step against this reference
      bool by_diff = false;           // P from differences (the same for the whole warp)
      for (int j = 0; j < nk; ++j, ++c) {
        if (!early_s && !mbar_wait(&gb.mma[c & 1], (c >> 1) & 1, err(), 58)) ok = false;
        if (!early_b && !mbar_wait(&b_full[bstg], bph, err(), 57)) ok = false;
        tc_fence_after_sync();
        const uint32_t mrow = mask_s + bstg * (kGroups * 256), brow = bias_row + bstg * M::TB, t_s = t_row + (c & 1) * 64;
        auto logits = [&](const uint32_t (&cur)[16], int q, float2 (&x)[8]) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float4 mA = lds128f(mrow + (q * 4 + u * 2) * 16), mB = lds128f(mrow + (q * 4 + u * 2 + 1) * 16);
            const float2 mk[4] = {make_float2(mA.x, mA.y), make_float2(mA.z, mA.w), make_float2(mB.x, mB.y), make_float2(mB.z, mB.w)};
            if constexpr (M::F32) {    // (bias: two tiles of 32 keys, 128-byte rows, 16-byte chunks swizzled by the row)
              uint4 b0 = make_uint4(0, 0, 0, 0), b1 = b0;
              if constexpr (HB) {
                const uint32_t at = brow + (q >> 1) * (M::TB / 2), g = (q & 1) * 4 + u * 2;
                b0 = lds128(at ^ (g << 4));
                b1 = lds128(at ^ ((g + 1) << 4));
              }
              const uint32_t bw[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                float2 v = __ffma2_rn(pair(cur[u * 8 + 2 * i], cur[u * 8 + 2 * i + 1]), sc2, mk[i]);
                if constexpr (HB) v = __fadd2_rn(v, pair(bw[2 * i], bw[2 * i + 1]));
                x[u * 4 + i] = v;
              }
              continue;
            }
            uint4 raw = make_uint4(0, 0, 0, 0);
            if constexpr (HB && !M::F32) raw = lds128(brow ^ ((q * 2 + u) << 4));   // (128-byte rows, 16-byte chunks swizzled by the row)
            const uint32_t bw[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float2 v = __ffma2_rn(pair(cur[u * 8 + 2 * i], cur[u * 8 + 2 * i + 1]), sc2, mk[i]);
              if constexpr (HB && !M::F32) v = add_wide<T>(v, bw[i]);
              x[u * 4 + i] = v;
            }
          }
        };
        auto subtract = [](float2 (&x)[8], float m) {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = __fadd2_rn(x[i], splat(-m));
        };
        auto exps = [&](const float2 (&x)[8], float2 nm2, uint32_t* w, float2& sum) {   // P = 2^(x log2e + nm2)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 e = __ffma2_rn(x[i], l2e2, nm2);
            const float2 p = make_float2(ex2_approx(e.x), ex2_approx(e.y));
            sum = __fadd2_rn(sum, p);
            if constexpr (M::F32) {
              w[2 * i] = __float_as_uint(p.x);
              w[2 * i + 1] = __float_as_uint(p.y);
            } else {
              w[i] = pack2<T>(p.x, p.y);
            }
          }
        };
        // fp32: sixteen P as their upper 19 bits, what a product reads of them, and the rest: P V is the sum of two products
        auto store_split = [&](uint32_t t_s, const uint32_t* w, int q) {
          uint32_t hi[16], lo[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            hi[2 * i] = w[2 * i] & 0xffffe000u;
            hi[2 * i + 1] = w[2 * i + 1] & 0xffffe000u;
            const float2 r = __fadd2_rn(pair(w[2 * i], w[2 * i + 1]), pair(hi[2 * i] ^ 0x80000000u, hi[2 * i + 1] ^ 0x80000000u));
            lo[2 * i] = __float_as_uint(r.x);
            lo[2 * i + 1] = __float_as_uint(r.y);
          }
          tmem_st_32x16(t_s + q * 16, hi);
          tmem_st_32x16(t_row + COL_LO + q * 16, lo);
        };
        // P of this thread's 64 keys and their sum
        float2 ps = make_float2(0.f, 0.f);
        uint32_t pw[M::PC], ra[16], rb[16];
        auto chunk = [&](auto diff, uint32_t (&cur)[16], uint32_t (&nxt)[16], int q) {   // sixteen keys; the next sixteen on their way
          ld_wait16(cur);
          if (q < 3) tmem_ld_32x16(t_s + (q + 1) * 16, nxt);
          float2 x[8];
          logits(cur, q, x);
          if constexpr (diff.value) {
            subtract(x, m);
            exps(x, splat(factor(m)), pw + q * (M::PC / 4), ps);
          } else {
            if (q == 0) m = j > 0 ? m : fmaxf(fmaxf(x[0].x, x[0].y), fmaxf(x[1].x, x[1].y));
            exps(x, splat(-(m * kLog2e)), pw + q * (M::PC / 4), ps);
          }
        };
        auto sweep = [&](auto diff) {
          tmem_ld_32x16(t_s, ra);
          chunk(diff, ra, rb, 0);
          chunk(diff, rb, ra, 1);
          chunk(diff, ra, rb, 2);
          chunk(diff, rb, ra, 3);
        };
        if (by_diff) sweep(std::true_type{});
        else sweep(std::false_type{});
        // whether the next step's S and bias tile are there: asked now, needed at the top
        early_s = mbar_test(&gb.mma[(c + 1) & 1], ((c + 1) >> 1) & 1);
        early_b = mbar_test(&b_full[bstg + 1 == kBiasStages ? 0 : bstg + 1], bstg + 1 == kBiasStages ? bph ^ 1 : bph);
        // (fp32: the rest of P has one buffer, and P V of the step before reads it; its commit is the next step's S)
        if (M::F32 && c > 0) {
          if (!early_s) {
            early_s = mbar_wait(&gb.mma[(c + 1) & 1], ((c + 1) >> 1) & 1, err(), 58);
            ok = early_s && ok;
          }
          tc_fence_after_sync();
        }
        float sum = ps.x + ps.y;
        const bool redo = __any_sync(0xffffffffu, !(sum < kTooBig) || (j == 0 && large(m)));
        if (!redo) {
          // over the S values this warp has read: 64 keys as 32 packed columns, or 64
          if constexpr (M::F32) {
#pragma unroll
            for (int q = 0; q < 4; ++q) store_split(t_s, pw + q * 16, q);
          } else {
            tmem_st_32x32(t_s, pw);
          }
        } else {
          // Some row of the warp outgrew its reference, or starts from a large one: take the maximum of the step, scale the sum and O by
          // 2^((m - m_new) log2e) and the quotient of the factors (once P V of the step before is done), and form P again.
          // (Sixteen keys' P end before the next sixteen's S.)
          float top = m;
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            float2 x[8];
            tmem_ld_32x16(t_s + q * 16, ra);
            ld_wait16(ra);
            logits(ra, q, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) top = fmax3(top, x[i].x, x[i].y);
          }
          top = fmaxf(top, -3.402823466e38f);   // (no finite logit yet: P = 2^-inf)
          const float fac = factor(top), alpha = ex2_approx((m - top) * kLog2e + (fac - factor(m)));
          m = top;
          l *= alpha;
          if (j > 0) {
            ok = mbar_wait(&gb.mma[(c - 1) & 1], (((c - 1) >> 1) + 1) & 1, err(), 59) && ok;
            tc_fence_after_sync();
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              tmem_ld_32x16(t_row + COL_O + h * 16, ra);
              ld_wait16(ra);
#pragma unroll
              for (int i = 0; i < 16; ++i) ra[i] = __float_as_uint(__uint_as_float(ra[i]) * alpha);
              tmem_st_32x16(t_row + COL_O + h * 16, ra);
            }
          }
          ps = make_float2(0.f, 0.f);
          seen = 0.f;
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            float2 x[8];
            uint32_t w[M::PC / 4];
            tmem_ld_32x16(t_s + q * 16, ra);
            ld_wait16(ra);
            logits(ra, q, x);
            subtract(x, m);
            exps(x, splat(fac), w, ps);
            if constexpr (M::F32) store_split(t_s, w, q);
            else tmem_st_32x8(t_s + q * 8, w);
          }
          sum = ps.x + ps.y;
        }
        l += sum;
        seen = fmaxf(seen, sum);
        if (redo) by_diff = __any_sync(0xffffffffu, large(m));
        if (j == 0 && pend) finish(c - 1);   // the row before this one
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&gb.p_ready[c & 1]);
          mbar_arrive(&b_free[bstg]);
        }
        if (++bstg == kBiasStages) { bstg = 0; bph ^= 1; }
        if (!ok) break;
      }
      pend = true; pm = m; pl = l; pseen = seen;
      const int qi = it.q0 + r, s = it.s0 + g;
      po = qi < a.N ? (int)((it.b * a.o_st[0] + s * a.o_st[1] + qi * a.o_st[2] + it.h * a.o_st[3]) >> M::kVecBits) : -1;
      pstat = ((it.b * a.S + s) * a.H + it.h) * a.N + qi;
    }
    if (pend && ok) finish(c - 1);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
  if (!TERMS && tid == 0) leave_status(a.status, err());
}

}  // namespace

bool attn_fwd_rows_fits(const TriAttnDesc* d) {
  const int vec = d->dtype == TRI_F32 ? 4 : 8;
  const int64_t last = (d->B - 1) * d->o_st[0] + (d->n_seq - 1) * d->o_st[1] + (d->n_res - 1) * d->o_st[2] + (d->H - 1) * d->o_st[3];
  return (int64_t)d->B * d->n_seq * d->H * d->n_res < (int64_t)1 << 31 && last / vec < ((int64_t)1 << 31) - 8;
}

int attn_fwd_rows(const TriAttnDesc* d, const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap* tbias,
                  bool bias_batched, const uint8_t* mask, const float* mask_terms, void* o, float* stats, int* err, bool first, cudaStream_t st) {
  RowsArgs a;
  a.B = d->B; a.S = d->n_seq; a.N = d->n_res; a.H = d->H; a.D = d->D;
  a.scale = d->scale;
  a.o = o;
  for (int i = 0; i < 4; ++i) a.o_st[i] = d->o_st[i];
  a.stats = stats; a.mask = mask; a.mask_st[0] = d->mask_st[0]; a.mask_st[1] = d->mask_st[1];
  a.mask_terms = mask_terms; a.npad = (d->n_res + 127) / 128 * 128;
  a.bias_b_mul = bias_batched ? 1 : 0;
  a.status = err;
  const int kind = d->dtype == TRI_F32 ? KIND_TF32 : d->dtype == TRI_BF16 ? KIND_BF16 : KIND_F16;
  a.idesc_s = make_idesc(kind, 128, 64, false, false);
  a.idesc_pv = make_idesc(kind, 128, 32, false, true);
  const long long combos = (long long)((d->n_res + 127) / 128) * d->H * d->B;
  int rows = d->dtype == TRI_F32 ? RowsCfg<float>::kGroups : RowsCfg<__half>::kGroups;
  while (rows > 1 && combos * cdiv(d->n_seq, rows) < sm_count()) --rows;   // fewer rows per CTA before an SM stays idle
  a.rows_per_item = rows;
  const long long items = combos * cdiv(d->n_seq, rows);
  const double pairs = (double)d->B * d->n_seq * d->H * d->n_res * (double)d->n_res;
  KernelTimer kt("tc_attn_fwd", st, 4.0 * pairs * d->D, (double)dtype_size(d->dtype) * 4.0 * d->B * d->n_seq * (double)d->n_res * d->H * d->D);
  sms_beside_attention() = (int)(sm_count() - ((items - 1) % sm_count() + 1));
  auto launch = [&](auto elem, auto kern, const CUtensorMap& tb) {
    using M = RowsCfg<decltype(elem)>;
    TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, M::SMEM));
    launch_dependent(first ? kLaunchPlainly : us_of_logits(pairs), kern, (unsigned)std::min<long long>(items, sm_count()), M::kThreads, M::SMEM, st, tq, tk, tv, tb, a);
    TRI_LAUNCH_OK();
    return 0;
  };
  auto start = [&](auto elem) {
    using T = decltype(elem);
    if (mask_terms != nullptr) return tbias ? launch(elem, attn_fwd_rows_kernel<T, true, true>, *tbias) : launch(elem, attn_fwd_rows_kernel<T, false, true>, tq);
    return tbias ? launch(elem, attn_fwd_rows_kernel<T, true, false>, *tbias) : launch(elem, attn_fwd_rows_kernel<T, false, false>, tq);
  };
  if (d->dtype == TRI_F32) return start(float());
  return d->dtype == TRI_BF16 ? start(__nv_bfloat16()) : start(__half());
}

}  // namespace tc
}  // namespace tri

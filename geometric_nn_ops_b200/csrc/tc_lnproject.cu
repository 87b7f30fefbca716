// LayerNorm fused into the attention-input projections (16-bit types, 128 channels): z -> q | k | v and the pair bias.
//
// One persistent CTA per SM, 576 threads:
//   warp 0      TMA: the projection weights once (up to 96 KB and the heads' rows, resident), then 128-pixel z tiles
//   warp 1      tcgen05.mma per tile: one product per block of 128 output columns (M = pixels, K = 128) and one of 16
//               columns for the heads, each into its own TMEM columns, freed block by block
//   warps 2-9   LayerNorm: two lanes per pixel, normalised in place in the swizzled layout the MMA reads
//   warps 10-17 epilogue: thread = pixel, 64 of a block's columns; a block leaves through shared memory by TMA, the heads
//               (head-major, the layout the attention takes its bias in) by the first four warps' stores
//
// What bounds it is DRAM: z is read once and the outputs are written once, 4 tensors with q, k, v against 6 for the
// LayerNorm kernel and the GEMM that it replaces (the normalised z does not leave the SM).  With no q | k | v (the bias of
// attention_pair_bias) it reads z and writes H / 128 of a tensor.
#include <algorithm>

#include "tc_lnproject.cuh"

#include "tc_gemm.cuh"

namespace tri {
namespace tc {

namespace {

constexpr int kThreads = 576;
constexpr int kSub = 16384;                 // one [128 rows x 128 bytes] swizzled sub-tile
constexpr int kTile = 2 * kSub;             // 128 x 128 16-bit values
constexpr int kHeads = 16;                  // columns of the heads' product
constexpr int kHTile = 2 * kHeads * 128;    // their weights: two 64-channel halves
constexpr uint32_t kHCol = 384;             // their TMEM columns
constexpr int kMaxStages = 5;               // z tiles in flight

struct Args {
  long long M;
  int tiles, blocks, heads, stages;
  long long plane;       // pixels per batch entry of the head-major output
  float eps;
  const void* gamma;
  const void* beta;
  void* bias;
  int* status;
};

__device__ __forceinline__ void next_stage(int& b, uint32_t& phase, int stages) {
  if (++b == stages) { b = 0; phase ^= 1; }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
ln_project_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmW,
                  const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmO, const Args g) {
  constexpr int KIND = ElemTraits<T>::kind;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sZ = smem;                       // [stages] z tiles
  uint8_t* sH = sZ + g.stages * kTile;
  uint8_t* sO = sH + kHTile;                // an output block, if there are any
  uint8_t* sW = sO + (g.blocks > 0 ? kTile : 0);
  T* s_gamma = reinterpret_cast<T*>(sW + g.blocks * kTile);
  T* s_beta = s_gamma + 128;
  uint64_t* wfull = reinterpret_cast<uint64_t*>(s_beta + 128);
  uint64_t* zfull = wfull + 1;              // [stages] tile landed
  uint64_t* znorm = zfull + kMaxStages;     // [stages] tile normalised (8 warps)
  uint64_t* zempty = znorm + kMaxStages;    // [stages] the tile's products are done
  uint64_t* tfull = zempty + kMaxStages;    // [4] block complete (3: heads)
  uint64_t* tempty = tfull + 4;             // [4] block read (8 warps; heads: 4)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 4);
  int* const err = reinterpret_cast<int*>(tmem_slot + 1);   // this CTA's (see leave_status)

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(wfull, 1);
    for (int b = 0; b < g.stages; ++b) { mbar_init(&zfull[b], 1); mbar_init(&znorm[b], 8); mbar_init(&zempty[b], 1); }
    for (int b = 0; b < 4; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], b < 3 ? 8 : 4); }
    mbar_fence_init();
    *err = 0;
  }
  if (threadIdx.x < 128) {
    s_gamma[threadIdx.x] = g.gamma ? reinterpret_cast<const T*>(g.gamma)[threadIdx.x] : from_f32<T>(1.f);
    s_beta[threadIdx.x] = g.beta ? reinterpret_cast<const T*>(g.beta)[threadIdx.x] : from_f32<T>(0.f);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(wfull, g.blocks * kTile + kHTile);
      for (int kb = 0; kb < 2; ++kb) {
        tma_load_3d(sH + kb * (kHTile / 2), &tmH, wfull, kb * 64, 0, 0);
        for (int blk = 0; blk < g.blocks; ++blk) tma_load_3d(sW + blk * kTile + kb * kSub, &tmW, wfull, kb * 64, blk * 128, 0);
      }
      int b = 0;
      uint32_t ph = 0;
      for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, next_stage(b, ph, g.stages)) {
        if (!mbar_wait(&zempty[b], ph ^ 1, err, 70)) break;
        mbar_expect_tx(&zfull[b], kTile);
        for (int kb = 0; kb < 2; ++kb) tma_load_3d(sZ + b * kTile + kb * kSub, &tmZ, &zfull[b], kb * 64, tile * 128, 0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc(KIND, 128, 128, false, false), idesc_h = make_idesc(KIND, 128, kHeads, false, false);
      const uint32_t z_base = smem_u32(sZ), w_base = smem_u32(sW), h_base = smem_u32(sH);
      bool ok = mbar_wait(wfull, 0, err, 71);
      int i = 0, b = 0;
      uint32_t ph = 0;
      for (int tile = blockIdx.x; tile < g.tiles && ok; tile += gridDim.x, ++i, next_stage(b, ph, g.stages)) {
        if (!mbar_wait(&znorm[b], ph, err, 72)) break;
        for (int n = 0; n <= g.blocks && ok; ++n) {
          const int blk = n < g.blocks ? n : 3;
          if (!mbar_wait(&tempty[blk], (i & 1) ^ 1, err, 73)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint64_t ad = make_smem_desc(z_base + b * kTile + (ks >> 2) * kSub + (ks & 3) * 32, 16, 1024);
            if (blk < 3) {
              const uint64_t bd = make_smem_desc(w_base + blk * kTile + (ks >> 2) * kSub + (ks & 3) * 32, 16, 1024);
              umma<KIND>(tmem_base + blk * 128, ad, bd, idesc, ks > 0);
            } else {
              const uint64_t bd = make_smem_desc(h_base + (ks >> 2) * (kHTile / 2) + (ks & 3) * 32, 16, 1024);
              umma<KIND>(tmem_base + kHCol, ad, bd, idesc_h, ks > 0);
            }
          }
          umma_commit(&tfull[blk]);
        }
        if (ok) umma_commit(&zempty[b]);
      }
    }
    __syncwarp();
  } else if (warp < 10) {
    // ------------------------------------------------------------------ LayerNorm: two lanes per pixel row, 64 channels each
    // (the odd lane takes its eight pieces from the fifth on, so that a pair of lanes never meets in a bank)
    const int r = (warp - 2) * 16 + (lane >> 1), half = lane & 1;
    const uint32_t sw = (uint32_t)((r & 7) ^ (half << 2)) << 4;
    const T* gam = s_gamma + half * 64;
    const T* bet = s_beta + half * 64;
    const bool shifted = g.beta != nullptr;
    int b = 0;
    uint32_t ph = 0;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, next_stage(b, ph, g.stages)) {
      const bool landed = mbar_wait(&zfull[b], ph, err, 74);
      if (!__all_sync(0xffffffffu, landed)) break;
      const uint32_t rowp = smem_u32(sZ + b * kTile + half * kSub + r * 128);
      auto unpack = [](const uint4& w, float2 (&v)[4]) {
        v[0] = unpack2<T>(w.x); v[1] = unpack2<T>(w.y); v[2] = unpack2<T>(w.z); v[3] = unpack2<T>(w.w);
      };
      // the half row stays in registers: mean, then the squares about it, then the result
      float2 v[8][4], s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        unpack(lds128(rowp + ((c << 4) ^ sw)), v[c]);
        s0 = __fadd2_rn(s0, __fadd2_rn(v[c][0], v[c][1]));
        s1 = __fadd2_rn(s1, __fadd2_rn(v[c][2], v[c][3]));
      }
      float mu = (s0.x + s0.y) + (s1.x + s1.y);
      mu = (mu + __shfl_xor_sync(0xffffffffu, mu, 1)) * (1.0f / 128);
      const float2 nmu = make_float2(-mu, -mu);
      s0 = s1 = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[c][e] = __fadd2_rn(v[c][e], nmu);
          if (e & 1) s1 = __ffma2_rn(v[c][e], v[c][e], s1);
          else s0 = __ffma2_rn(v[c][e], v[c][e], s0);
        }
      float var = (s0.x + s0.y) + (s1.x + s1.y);
      var = (var + __shfl_xor_sync(0xffffffffu, var, 1)) * (1.0f / 128);
      const float rs = 1.0f / sqrtf(var + g.eps);
      const float2 rs2 = make_float2(rs, rs);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int ch = (c ^ (half << 2)) * 8;
        float2 gm[4];
        unpack(*reinterpret_cast<const uint4*>(gam + ch), gm);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[c][e] = __fmul2_rn(__fmul2_rn(v[c][e], rs2), gm[e]);
        if (shifted) {
          float2 bt[4];
          unpack(*reinterpret_cast<const uint4*>(bet + ch), bt);
#pragma unroll
          for (int e = 0; e < 4; ++e) v[c][e] = __fadd2_rn(v[c][e], bt[e]);
        }
        sts128(rowp + ((c << 4) ^ sw), pack2<T>(v[c][0].x, v[c][0].y), pack2<T>(v[c][1].x, v[c][1].y), pack2<T>(v[c][2].x, v[c][2].y),
               pack2<T>(v[c][3].x, v[c][3].y));
      }
      fence_proxy_async_smem();   // the tile is read next by tcgen05.mma
      __syncwarp();
      if (lane == 0) mbar_arrive(&znorm[b]);
    }
  } else {
    // ------------------------------------------------------------------ epilogue: thread = pixel
    const int quarter = warp & 3, part = (warp - 10) >> 2;   // TMEM lane quarter; 64 of a block's columns
    const int row = quarter * 32 + lane;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);
    uint8_t* orow = sO + part * kSub + row * 128;
    T* bias = reinterpret_cast<T*>(g.bias);
    const bool issuer = quarter == 0 && lane == 0;          // ... of this part's 64 columns
    int i = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
      for (int blk = 0; blk < g.blocks; ++blk) {
        ok = mbar_wait(&tfull[blk], i & 1, err, 75) && ok;
        tc_fence_after_sync();
        uint32_t w[32];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[32];
          tmem_ld_32x32(t_row + blk * 128 + part * 64 + h * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) w[h * 16 + e] = pack2<T>(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[blk]);
        if (issuer) bulk_wait_group_read0();                // the previous block has left this half of the staging tile
        named_barrier(1 + part, 128);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          *reinterpret_cast<uint4*>(orow + ((c ^ (row & 7)) << 4)) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
        fence_proxy_async_smem();
        named_barrier(3 + part, 128);
        if (issuer && ok) {
          tma_store_3d(&tmO, sO + part * kSub, blk * 128 + part * 64, tile * 128, 0);
          bulk_commit_group();
        }
      }
      if (part == 0) {
        ok = mbar_wait(&tfull[3], i & 1, err, 76) && ok;
        tc_fence_after_sync();
        uint32_t v[16];
        tmem_ld_32x16(t_row + kHCol, v);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[3]);
        const long long m = (long long)tile * 128 + row;
        if (m < g.M && ok) {
          const long long b = m / g.plane;
          T* dst = bias + b * g.heads * g.plane + (m - b * g.plane);
#pragma unroll
          for (int h = 0; h < kHeads; ++h)
            if (h < g.heads) dst[h * g.plane] = from_f32<T>(__uint_as_float(v[h]));
        }
      }
    }
    if (issuer) bulk_wait_group0();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0) leave_status(g.status, err);
}

template <typename T>
int launch(cudaStream_t st, const LnProject& p) {
  const bool f16 = p.dtype == TRI_F16;
  const uint64_t M = (uint64_t)p.M, n = (uint64_t)std::max(p.n_out, 8);
  const uint64_t zd[3] = {128, M, 1}, zs[2] = {128, 128 * M}, wd[3] = {128, n, 1}, ws[2] = {128, 128 * n};
  const uint64_t hd[3] = {128, (uint64_t)p.heads, 1}, hs[2] = {128, 128 * (uint64_t)p.heads}, od[3] = {n, M, 1}, os[2] = {n, n * M};
  const uint32_t box[3] = {64, 128, 1}, hbox[3] = {64, kHeads, 1};
  CUtensorMap tz, tw, th, to;
  TRI_TRY(make_tmap_3d(&tz, p.z, 2, f16, zd, zs, box, false));
  TRI_TRY(make_tmap_3d(&th, p.w_bias, 2, f16, hd, hs, hbox, false));
  tw = to = tz;
  Args a;
  a.M = p.M; a.tiles = cdiv(p.M, 128); a.blocks = cdiv(p.n_out, 128); a.heads = p.heads; a.plane = p.plane; a.eps = p.eps;
  a.gamma = p.gamma; a.beta = p.beta; a.bias = p.bias; a.status = p.err;
  if (a.blocks > 0) {
    TRI_TRY(make_tmap_3d(&tw, p.w_qkv, 2, f16, wd, ws, box, false));
    TRI_TRY(make_tmap_3d(&to, p.qkv, 2, f16, od, os, box, false));
  }
  // Two z tiles beside 96 KB of weights; five without, to cover the latency of DRAM.
  a.stages = a.blocks > 0 ? 2 : kMaxStages;
  const size_t smem = 1024 + a.stages * kTile + kHTile + (a.blocks > 0 ? (1 + a.blocks) * kTile : 0) + 512 + (2 + 3 * kMaxStages + 8) * 8;
  auto kern = ln_project_kernel<T>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const double unit = 256.0 * p.M;
  KernelTimer kt(a.blocks > 0 ? "tc_ln_project" : "tc_ln_bias", st, 2.0 * p.M * 128 * (p.n_out + p.heads),
                 unit * (1.0 + (p.n_out + p.heads) / 128.0));
  kern<<<std::min(a.tiles, sm_count()), kThreads, smem, st>>>(tz, tw, th, to, a);
  TRI_LAUNCH_OK();
  return 0;
}

}  // namespace

bool ln_project_supported(int dtype, long long M, int n_out, int heads) {
  return (dtype == TRI_BF16 || dtype == TRI_F16) && M > 0 && M < (1LL << 31) - 128 && n_out % 8 == 0 && n_out <= 384 && heads >= 1 &&
         heads <= kHeads;
}

int ln_project(cudaStream_t st, const LnProject& p) {
  if (!ln_project_supported(p.dtype, p.M, p.n_out, p.heads)) return fail(TRI_ERR_ARG, "ln_project: unsupported shape or dtype");
  return p.dtype == TRI_BF16 ? launch<__nv_bfloat16>(st, p) : launch<__half>(st, p);
}

}  // namespace tc
}  // namespace tri

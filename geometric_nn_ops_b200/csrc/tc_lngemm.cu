// LayerNorm fused into the two projection kernels of the triangle multiplicative update (see tc_lngemm.cuh).
//
// ln_gate_in.  One persistent CTA per SM, 832 threads:
//   warp 0       TMA: the concatenated weights once (128 KB, resident), then one 128-pixel x tile per step into one of
//                two 32 KB buffers; stores each tile as z once it is normalised
//   warp 1       tcgen05.mma: per tile and half (a, b) the P and G products, M = the half's 128 channels, N = 128
//                pixels, into the half's 256-column accumulator
//   warps 2-9    LayerNorm: two threads to a pixel row, which is normalised in place (two passes over it in shared memory: one
//                chain of the statistics' sums each, half of the result each); they write the statistics and release the tile
//                to the MMA warp and to the store.
//   warps 10-25  gate epilogue, thread = channel holding consecutive pixels (the order of the channel-major a / b); a set of
//                eight warps for each half, so that one set's waits and stores run beside the other's arithmetic
//
// Against the two-kernel form (LayerNorm kernel, then the gate GEMM reading z once per half) x is read once, z is
// written from shared memory and never read back here, and the weights stay in shared memory.  a and b leave through
// shared memory too, by TMA in whole 128-byte lines; the epilogue threads' own stores carried 32 bytes per request, a
// channel's rows lying a plane apart.  Per launch at 768 x 768 pixels: 0.24 ms for the pair of kernels, 0.197 for this one
// at first, 0.165 with a reciprocal instead of a quotient in the sigmoid, pairwise conversions, the mask read once per
// tile and staged stores, and 0.145 with eight LayerNorm warps (four took 5.3 k cycles a tile, one of them 2 k more for the store of
// z, where a tile takes 8.5 k in all) and the epilogue in two sets (as one, 4.8 k cycles of arithmetic, 1.4 of staging and 1.3 of
// waiting followed one another); floor by bytes 0.092.  What bounds it is likely the path of shared memory and TMEM: counted at 128 bytes a cycle,
// MMA operands, accumulators, the LayerNorm's passes and the tiles' ways in and out take about 6.6 k of the 7.4 k cycles of a tile (an estimate;
// ncu: load / store wavefronts 40 %, XU 54 %, tensor 26 %, DRAM 46 %).  (One reciprocal for two sigmoids changes nothing; rows kept in registers
// between the passes spill at 72 a thread.)
// Every mbarrier wait is bounded; a timeout lands in *err and all roles drain.
#include "tc_lngemm.cuh"

#include "tc_gemm.cuh"

namespace tri {
namespace tc {

namespace {

constexpr int kThreads = 832, kLnWarps = 8, kEpi0 = 2 + kLnWarps;   // warps: TMA, MMA, LayerNorm, 16 for the gate epilogue
constexpr int kSub = 16384;                 // one [128 rows x 128 bytes] swizzled sub-tile
constexpr uint32_t kWBytes = 8 * kSub;      // (Pa, Ga, Pb, Gb) x (k 0..63, k 64..127)
constexpr uint32_t kXBytes = 2 * kSub;      // one pixel tile: two 64-channel halves
constexpr int kXBufs = 2;                 // (a third buffer, which still fits, changed nothing)
constexpr int kMaskRing = 4;              // tile i + 4 lands only after the products of tile i + 2, hence after the epilogue of tile i

struct Args {
  long long M, plane;
  int tiles;
  float eps;
  const void* gamma;
  const void* beta;
  const float* bias;
  const void* mask;
  void* a_cm;
  void* b_cm;
  float* mean;
  float* rstd;
  int n, pitch;         // as in LnGateIn
  int own_pitch;
  int staged;           // a / b leave through shared memory by TMA (planes of whole 64-pixel chunks)
  int* err;
};

template <typename T> __device__ __forceinline__ void unpack8p(const uint4& w, float2 (&v)[4]) {
  v[0] = unpack2<T>(w.x); v[1] = unpack2<T>(w.y); v[2] = unpack2<T>(w.z); v[3] = unpack2<T>(w.w);
}
template <typename T> __device__ __forceinline__ uint4 pack8p(const float2 (&v)[4]) {
  return make_uint4(pack2<T>(v[0].x, v[0].y), pack2<T>(v[1].x, v[1].y), pack2<T>(v[2].x, v[2].y), pack2<T>(v[3].x, v[3].y));
}

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
ln_gate_in_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                  const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmA,
                  const __grid_constant__ CUtensorMap tmB, const Args g) {
  constexpr int KIND = ElemTraits<T>::kind;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sW = smem;
  uint8_t* sX = smem + kWBytes;
  uint8_t* sO = sX + kXBufs * kXBytes;     // two chunks of [128 channels x 64 pixels] of a or b
  T* s_gamma = reinterpret_cast<T*>(sO + kXBytes);
  T* s_beta = s_gamma + 128;
  T* s_mask = s_beta + 128;               // [kMaskRing][128] pixel mask of a tile
  uint64_t* wfull = reinterpret_cast<uint64_t*>(s_mask + kMaskRing * 128);
  uint64_t* xfull = wfull + 1;            // [kXBufs] tile landed (TMA bytes)
  uint64_t* xnorm = xfull + kXBufs;       // [kXBufs] tile normalised (one arrival per LayerNorm warp)
  uint64_t* xempty = xnorm + kXBufs;      // [kXBufs] the tile's products are done (commit)
  uint64_t* tfull = xempty + kXBufs;      // [2] accumulator of half h complete
  uint64_t* tempty = tfull + 2;     // [2] accumulator of half h read by its eight epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(wfull, 1);
    for (int b = 0; b < kXBufs; ++b) { mbar_init(&xfull[b], 1); mbar_init(&xnorm[b], kLnWarps); mbar_init(&xempty[b], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], 8); }
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmZ);
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
  dependent_enter();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer; z leaves from the normalised tiles
    if (elect_one()) {
      mbar_expect_tx(wfull, kWBytes);
      for (int blk = 0; blk < 4; ++blk)
        for (int kb = 0; kb < 2; ++kb) tma_load_3d(sW + (blk * 2 + kb) * kSub, &tmW, wfull, kb * 64, blk * 128, 0);
      // z of the k-th tile, once its rows are normalised; the buffer is free when the store has read it and the products are done
      auto store_z = [&](int k) {
        const int b = k % kXBufs, tile = blockIdx.x + k * gridDim.x;
        if (!mbar_wait(&xnorm[b], (k / kXBufs) & 1, g.err, 15)) return false;
        tma_store_3d(&tmZ, sX + b * kXBytes, 0, tile * 128, 0);
        tma_store_3d(&tmZ, sX + b * kXBytes + kSub, 64, tile * 128, 0);
        bulk_commit_group();
        return true;
      };
      int i = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
        const int b = i % kXBufs;
        if (i >= kXBufs) {
          ok = store_z(i - kXBufs);
          bulk_wait_group_read0();
          if (!ok || !(ok = mbar_wait(&xempty[b], ((i / kXBufs) & 1) ^ 1, g.err, 10))) break;
        }
        mbar_expect_tx(&xfull[b], kXBytes);
        if (!g.own_pitch) {
          for (int kb = 0; kb < 2; ++kb) tma_load_3d(sX + b * kXBytes + kb * kSub, &tmX, &xfull[b], kb * 64, tile * 128, 0);
        } else {   // eight pixels of a row at a time (the pitch is a multiple of eight), zeros where x ends
          int row = tile * 128 / g.pitch, col = tile * 128 - row * g.pitch;
          for (int e = 0; e < 16; ++e) {
            for (int kb = 0; kb < 2; ++kb) tma_load_3d(sX + b * kXBytes + kb * kSub + e * 1024, &tmX, &xfull[b], kb * 64, col, row);
            if ((col += 8) == g.pitch) { col = 0; ++row; }
          }
        }
      }
      for (int k = max(0, i - kXBufs); k < i && ok; ++k) ok = store_z(k);
      bulk_wait_group0();
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = make_idesc(KIND, 128, 128, false, false);
      const uint32_t w_base = smem_u32(sW), x_base = smem_u32(sX);
      bool ok = mbar_wait(wfull, 0, g.err, 11);
      int i = 0;
      for (int tile = blockIdx.x; tile < g.tiles && ok; tile += gridDim.x, ++i) {
        const int b = i % kXBufs;
        if (!mbar_wait(&xnorm[b], (i / kXBufs) & 1, g.err, 12)) break;
        tc_fence_after_sync();
        for (int half = 0; half < 2 && ok; ++half) {
          if (!mbar_wait(&tempty[half], (i & 1) ^ 1, g.err, 13)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int pg = 0; pg < 2; ++pg) {   // P block, G block of this half
            const uint32_t d_addr = tmem_base + half * 256 + pg * 128;
#pragma unroll
            for (int kb = 0; kb < 2; ++kb)
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                const uint64_t ad = make_smem_desc(w_base + ((half * 2 + pg) * 2 + kb) * kSub + ks * 32, 16, 1024);
                const uint64_t bd = make_smem_desc(x_base + b * kXBytes + kb * kSub + ks * 32, 16, 1024);
                umma<KIND>(d_addr, ad, bd, idesc, (kb == 0 && ks == 0) ? 0u : 1u);
              }
          }
          umma_commit(&tfull[half]);
        }
        if (ok) umma_commit(&xempty[b]);
      }
    }
    __syncwarp();
  } else if (warp < kEpi0) {
    // ------------------------------------------------------------------ LayerNorm: two threads to a pixel row of the tile
    const int r = (warp - 2) * 16 + (lane & 15), kb = lane >> 4;
    const uint32_t sw = (uint32_t)(r & 7) << 4;
    const T* mask = reinterpret_cast<const T*>(g.mask);
    int i = 0;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
      const int b = i % kXBufs;
      const bool landed = mbar_wait(&xfull[b], (i / kXBufs) & 1, g.err, 14);
      if (!__all_sync(0xffffffffu, landed)) break;
      uint8_t* rowp = sX + b * kXBytes + r * 128;
      uint8_t* part = rowp + kb * kSub;
      // Statistics in one pass over the row, shifted by its first element K: sums of (x - K) and (x - K)^2.  K is one
      // of the 128 samples, so (mean - K)^2 <= 128 var and the subtraction below loses at most seven bits of fp32.
      // Packed fp32x2 arithmetic: a row's even pairs of channels are one chain of additions and its odd pairs the other, a
      // thread has one of the two.  (So the sums do not depend on how many threads share a row; split by halves of the row they
      // had other last bits, which in 16 bits a stack of blocks carries on.)
      float2 s = make_float2(0.f, 0.f), q = s;
      const float k0 = unpack2<T>(*reinterpret_cast<const uint32_t*>(rowp + sw)).x;
      const float2 nk = make_float2(-k0, -k0);
      const uint8_t* chain = rowp + kb * 4;
#pragma unroll 8
      for (int c = 0; c < 16; ++c) {
        const uint8_t* p = chain + (c >> 3) * kSub + (((c & 7) << 4) ^ sw);
        const float2 d0 = __fadd2_rn(unpack2<T>(*reinterpret_cast<const uint32_t*>(p)), nk);
        const float2 d1 = __fadd2_rn(unpack2<T>(*reinterpret_cast<const uint32_t*>(p + 8)), nk);
        s = __fadd2_rn(s, d0); q = __ffma2_rn(d0, d0, q);
        s = __fadd2_rn(s, d1); q = __ffma2_rn(d1, d1, q);
      }
      float sum = s.x + s.y, sq = q.x + q.y;
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      sq += __shfl_xor_sync(0xffffffffu, sq, 16);
      const float ms = sum * (1.0f / 128);          // mean - K
      const float mu = ms - nk.x;
      const float var = fmaxf(sq * (1.0f / 128) - ms * ms, 0.f);
      const long long m = (long long)tile * 128 + r;
      const float rs = pixel_rstd(var, g.eps, m, g.n, g.pitch);
      const float2 nmu = make_float2(-mu, -mu);
      const float2 rs2 = make_float2(rs, rs);
#pragma unroll 4
      for (int c = 0; c < 8; ++c) {
        uint4* p = reinterpret_cast<uint4*>(part + ((c << 4) ^ sw));
        float2 v[4];
        unpack8p<T>(*p, v);
        float2 gm[4], bt[4], o[4];
        unpack8p<T>(*reinterpret_cast<const uint4*>(s_gamma + kb * 64 + c * 8), gm);
        unpack8p<T>(*reinterpret_cast<const uint4*>(s_beta + kb * 64 + c * 8), bt);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = __ffma2_rn(__fadd2_rn(v[e], nmu), __fmul2_rn(rs2, gm[e]), bt[e]);
        *p = pack8p<T>(o);
      }
      if (m < g.M && kb == 0) {
        g.mean[m] = mu; g.rstd[m] = rs;
        T* keep = s_mask + (i % kMaskRing) * 128 + r;
        if (g.own_pitch) {   // the mask in its own pitch too, zero at the pixels beyond n
          const int py = (int)((uint32_t)m / (uint32_t)g.pitch), px = (int)m - py * g.pitch;
          *keep = py < g.n && px < g.n ? (mask != nullptr ? mask[py * g.n + px] : from_f32<T>(1.f)) : from_f32<T>(0.f);
        } else if (mask != nullptr) {
          *keep = mask[m];
        }
      }
      fence_proxy_async_smem();   // the tile is read next by tcgen05.mma and by the TMA store
      __syncwarp();
      if (lane == 0) mbar_arrive(&xnorm[b]);
    }
  } else {
    // ------------------------------------------------------------------ gate epilogue: thread = channel of the set's half
    const int half = (warp - kEpi0) >> 3, j = (warp - kEpi0) >> 2 & 1, quarter = warp & 3;   // half; 32 pixels of 64; TMEM lane quarter
    const int row = quarter * 32 + lane;
    const bool masked = g.mask != nullptr || g.own_pitch, staged = g.staged != 0;
    const uint32_t plane = (uint32_t)g.plane, M = (uint32_t)g.M;
    // staging: a set's 64-pixel chunk and its issuing thread
    uint8_t* orow = sO + half * kSub + row * 128;
    const bool issuer = j == 0 && quarter == 0 && lane == 0;
    float bp = 0.f, bg = 0.f;
    if (g.bias != nullptr) { bp = g.bias[half * 256 + row]; bg = g.bias[half * 256 + 128 + row]; }
    const float2 bp2 = make_float2(bp, bp), nbg2 = make_float2(-1.4426950408889634f * bg, -1.4426950408889634f * bg);
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * 256;
    int i = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
      const uint32_t n0 = (uint32_t)tile * 128, nb0 = n0 / plane, np0 = n0 - nb0 * plane;   // one division per tile
      ok = mbar_wait(&tfull[half], i & 1, g.err, 16) && ok;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        const uint32_t off = c * 64 + j * 32;
        const uint4* mrow = reinterpret_cast<const uint4*>(s_mask + (i % kMaskRing) * 128 + off);
        Raw8<T> o[4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          float p[16], gt[16];
          ld16x2_f(t_row + off + hf * 16, t_row + 128 + off + hf * 16, p, gt);
          if (c == 1 && hf == 1) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[half]);
          }
#pragma unroll
          for (int uu = 0; uu < 2; ++uu) {
            float2 mk[4];
            if (masked) unpack8p<T>(mrow[hf * 2 + uu], mk);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int e = uu * 8 + 2 * k;
              float2 r = __fmul2_rn(__fadd2_rn(make_float2(p[e], p[e + 1]), bp2), sigmoid2(make_float2(gt[e], gt[e + 1]), nbg2));
              if (masked) r = __fmul2_rn(r, mk[k]);
              putraw8(o[hf * 2 + uu], k, r);
            }
          }
        }
        if (staged) {
          if (issuer) bulk_wait_group_read0();   // the chunk before has left
          named_barrier(1 + half, 256);
#pragma unroll
          for (int u = 0; u < 4; ++u) *reinterpret_cast<uint4*>(orow + (((j * 4 + u) ^ (row & 7)) << 4)) = o[u].w[0];
          fence_proxy_async_smem();
          named_barrier(3 + half, 256);
          const uint32_t px = n0 + c * 64;
          if (issuer && px < M && ok) {          // a chunk of 64 pixels never straddles two batch entries here
            tma_store_3d(half == 0 ? &tmA : &tmB, sO + half * kSub, px % plane, 0, px / plane);
            bulk_commit_group();
          }
        } else if (ok) {
          T* base = reinterpret_cast<T*>(half == 0 ? g.a_cm : g.b_cm) + ((long long)nb0 * 128 + row) * g.plane + np0 + off;
#pragma unroll
          for (int u = 0; u < 4; ++u) {          // 8 pixels: same batch entry, all valid or none
            T* d8 = base + u * 8;
            for (uint32_t pix = np0 + off + u * 8; pix >= plane; pix -= plane) d8 += 127 * g.plane;   // the next batch entry's plane of this channel
            if (n0 + off + u * 8 < M) straw8<T>(d8, o[u]);
          }
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
}

template <typename T>
int launch(cudaStream_t st, const LnGateIn& p) {
  const uint64_t M = (uint64_t)p.M;
  CUtensorMap tmX, tmW, tmZ, tmA, tmB;
  const uint64_t xd[3] = {128, M, 1}, xs[2] = {128, 128 * M};
  const uint64_t wd[3] = {128, 512, 1}, wsd[2] = {128, 128 * 512};
  const uint32_t box[3] = {64, 128, 1};
  const bool f16 = p.dtype == TRI_F16;
  if (p.own_pitch) {
    const uint64_t n = (uint64_t)p.n, nd[3] = {128, n, n}, ns[2] = {128, 128 * n};
    const uint32_t nbox[3] = {64, 8, 1};
    TRI_TRY(make_tmap_3d(&tmX, p.x, 2, f16, nd, ns, nbox, false));
  } else {
    TRI_TRY(make_tmap_3d(&tmX, p.x, 2, f16, xd, xs, box, false));
  }
  TRI_TRY(make_tmap_3d(&tmW, p.wcat, 2, f16, wd, wsd, box, false));
  TRI_TRY(make_tmap_3d(&tmZ, p.z, 2, f16, xd, xs, box, false));
  Args a;
  a.n = p.n; a.pitch = p.pitch; a.own_pitch = p.own_pitch;
  a.staged = p.plane % 64 == 0;
  tmA = tmB = tmX;
  if (a.staged) {
    const uint64_t P = (uint64_t)p.plane, ad[3] = {P, 128, M / P}, as[2] = {P, 128 * P};
    TRI_TRY(make_tmap_3d(&tmA, p.a_cm, 2, f16, ad, as, box, false));
    TRI_TRY(make_tmap_3d(&tmB, p.b_cm, 2, f16, ad, as, box, false));
  }
  a.M = p.M; a.plane = p.plane; a.tiles = (int)((p.M + 127) / 128); a.eps = p.eps;
  a.gamma = p.gamma; a.beta = p.beta; a.bias = p.bias_cat; a.mask = p.mask;
  a.a_cm = p.a_cm; a.b_cm = p.b_cm; a.mean = p.mean; a.rstd = p.rstd; a.err = p.err;
  constexpr size_t smem = 1024 + kWBytes + kXBufs * kXBytes + kXBytes + (2 + kMaskRing) * 128 * sizeof(T) + (1 + 3 * kXBufs + 4) * 8 + 16;
  static_assert(smem <= 232448, "shared memory of one CTA");
  auto kern = ln_gate_in_kernel<T>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = std::min(a.tiles, sm_count());
  const double bytes = 4.0 * p.M * 128 * 2;
  KernelTimer kt("tc_ln_gate_in", st, 2.0 * p.M * 128 * 512, bytes);
  launch_dependent(p.first ? kLaunchPlainly : us_of_bytes(bytes), kern, grid, kThreads, smem, st, tmX, tmW, tmZ, tmA, tmB, a);
  TRI_LAUNCH_OK();
  return 0;
}


// =================================================================================================================
// ln_gate_out: LayerNorm over the channels of channel-major t, fused into the output projection and gate
// =================================================================================================================
// 832 threads as above.  A tile is 128 pixels.  Its t part arrives as the MN-major A operand of the product
// y = u Wo^T: per 64-channel half, two chunks of [64 channel rows x 128 bytes = 64 pixels] (128-byte swizzle), which
// is how the contraction's output lies in memory -- nothing is transposed.  The LayerNorm role normalises every
// pixel's 128 channels in place: a thread sums 4 pixels over 16 of the 128 channels, the eight partial (mean, M2) pairs of a
// pixel are combined through shared memory (Chan's formula), then each thread rewrites 8 pixels (one 16-byte piece of a row) of
// 8 channels and, for training, stores them to the channel-major u the backward pass reads.
// With 128 threads of 16 channels the role took 6.8 k of the 7.1 k cycles of a tile (768 x 768 pixels: 142 us, 118 with 256).
// The z part (K-major) feeds the gate product unchanged.  Output weights and gate weights stay in shared memory.
constexpr uint32_t kOWBytes = 4 * kSub;     // (Wo, Wgo) x (k 0..63, k 64..127)
constexpr uint32_t kOTile = 4 * kSub;       // t: 2 halves x [2 chunks x 8 KB]; z: 2 halves x 16 KB
constexpr int kOBufs = 2;

struct OutArgs {
  long long M;
  int tiles;
  float eps;
  const void* gamma;
  const void* beta;
  const float* bias;
  void* u_cm;
  float* mean;
  float* rstd;
  void* out;
  const void* residual;
  int n, pitch, own_pitch;   // as in LnGateOut
  int* err;
};

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
ln_gate_out_kernel(const __grid_constant__ CUtensorMap tmT, const __grid_constant__ CUtensorMap tmZ,
                   const __grid_constant__ CUtensorMap tmWo, const __grid_constant__ CUtensorMap tmWg, const OutArgs g) {
  constexpr int KIND = ElemTraits<T>::kind;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sW = smem;
  uint8_t* sT = smem + kOWBytes;
  float* s_pm = reinterpret_cast<float*>(sT + kOBufs * kOTile);   // [8][128] partial means
  float* s_pq = s_pm + 8 * 128;                                   // [8][128] partial sums of squared deviations
  float* s_mean = s_pq + 8 * 128;
  float* s_rstd = s_mean + 128;
  float* s_gamma = s_rstd + 128;
  float* s_beta = s_gamma + 128;
  uint64_t* wfull = reinterpret_cast<uint64_t*>(s_beta + 128);
  uint64_t* bfull = wfull + 1;            // [kOBufs] tile landed
  uint64_t* bnorm = bfull + kOBufs;       // [kOBufs] t part normalised (one arrival per LayerNorm warp)
  uint64_t* bempty = bnorm + kOBufs;      // [kOBufs] both products of the tile are done
  uint64_t* tfull = bempty + kOBufs;      // [2] accumulator complete
  uint64_t* tempty = tfull + 2;           // [2] accumulator read by all 16 epilogue warps
  uint64_t* nsync = tempty + 2;           // [2] the two meeting points of the 256 LayerNorm threads
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(nsync + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(wfull, 1);
    for (int b = 0; b < kOBufs; ++b) { mbar_init(&bfull[b], 1); mbar_init(&bnorm[b], kLnWarps); mbar_init(&bempty[b], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], 16); }
    mbar_init(&nsync[0], 256); mbar_init(&nsync[1], 128);
    mbar_fence_init();
    tma_prefetch_desc(&tmT);
    tma_prefetch_desc(&tmZ);
    tma_prefetch_desc(&tmWo);
    tma_prefetch_desc(&tmWg);
  }
  if (threadIdx.x < 128) {
    s_gamma[threadIdx.x] = g.gamma ? to_f32(reinterpret_cast<const T*>(g.gamma)[threadIdx.x]) : 1.f;
    s_beta[threadIdx.x] = g.beta ? to_f32(reinterpret_cast<const T*>(g.beta)[threadIdx.x]) : 0.f;
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // the weights are the caller's and come while the contraction drains
  if (warp == 0 && elect_one()) {
    mbar_expect_tx(wfull, kOWBytes);
    for (int kb = 0; kb < 2; ++kb) {
      tma_load_3d(sW + kb * kSub, &tmWo, wfull, kb * 64, 0, 0);
      tma_load_3d(sW + (2 + kb) * kSub, &tmWg, wfull, kb * 64, 0, 0);
    }
  }
  dependent_enter();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int i = 0;
      for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
        const int b = i % kOBufs;
        if (!mbar_wait(&bempty[b], ((i / kOBufs) & 1) ^ 1, g.err, 20)) break;
        uint8_t* buf = sT + b * kOTile;
        mbar_expect_tx(&bfull[b], kOTile);
        for (int kb = 0; kb < 2; ++kb) {
          for (int c = 0; c < 2; ++c) tma_load_3d(buf + kb * kSub + c * (kSub / 2), &tmT, &bfull[b], tile * 128 + c * 64, kb * 64, 0);
          tma_load_3d(buf + 2 * kSub + kb * kSub, &tmZ, &bfull[b], kb * 64, tile * 128, 0);
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc_y = make_idesc(KIND, 128, 128, true, false);    // A = u tile, pixels contiguous
      const uint32_t idesc_g = make_idesc(KIND, 128, 128, false, false);   // A = z tile, channels contiguous
      const uint32_t w_base = smem_u32(sW), t_base = smem_u32(sT);
      bool ok = mbar_wait(wfull, 0, g.err, 21);
      int i = 0;
      for (int tile = blockIdx.x; tile < g.tiles && ok; tile += gridDim.x, ++i) {
        const int b = i % kOBufs, acc = i & 1;
        if (!mbar_wait(&bnorm[b], (i / kOBufs) & 1, g.err, 22)) break;
        if (!mbar_wait(&tempty[acc], ((i >> 1) & 1) ^ 1, g.err, 23)) break;
        tc_fence_after_sync();
        const uint32_t buf = t_base + b * kOTile, d_addr = tmem_base + acc * 256;
#pragma unroll
        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            // 16 channel rows per MMA; the second 64-pixel chunk of the half lies 8 KB further
            const uint64_t ad = make_smem_desc(buf + kb * kSub + ks * 16 * 128, kSub / 2, 1024);
            const uint64_t bd = make_smem_desc(w_base + kb * kSub + ks * 32, 16, 1024);
            umma<KIND>(d_addr, ad, bd, idesc_y, (kb == 0 && ks == 0) ? 0u : 1u);
          }
#pragma unroll
        for (int kb = 0; kb < 2; ++kb)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t ad = make_smem_desc(buf + (2 + kb) * kSub + ks * 32, 16, 1024);
            const uint64_t bd = make_smem_desc(w_base + (2 + kb) * kSub + ks * 32, 16, 1024);
            umma<KIND>(d_addr + 128, ad, bd, idesc_g, (kb == 0 && ks == 0) ? 0u : 1u);
          }
        umma_commit(&tfull[acc]);
        umma_commit(&bempty[b]);
      }
    }
    __syncwarp();
  } else if (warp < kEpi0) {
    // ------------------------------------------------------------------ LayerNorm over channels
    const int tid = threadIdx.x - 64;
    const int pg = tid & 15, kp = tid >> 4;       // 8-pixel group of the tile; 8-channel part
    const int gg = pg & 7;                        // 16-byte piece within the 128-byte row of its 64-pixel chunk
    const uint32_t part_off = (kp >> 3) * kSub + (pg >> 3) * (kSub / 2) + (kp & 7) * 8 * 128;
    // the statistics: 4-pixel group; 16-channel part (a warp's).  As in ln_gate_in, the sums are those that 128 threads formed.
    const int p4 = tid & 31, k16 = tid >> 5;
    const uint32_t stat_off = (k16 >> 2) * kSub + (p4 >> 4) * (kSub / 2) + (k16 & 3) * 16 * 128 + (p4 & 1) * 8;
    const int g4 = p4 >> 1 & 7;
    T* u_cm = reinterpret_cast<T*>(g.u_cm);
    int i = 0;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
      const int b = i % kOBufs;
      const bool landed = mbar_wait(&bfull[b], (i / kOBufs) & 1, g.err, 24);
      if (!__all_sync(0xffffffffu, landed)) break;
      uint8_t* part = sT + b * kOTile + part_off;   // rows kp*8 .. kp*8+7 of this thread's chunk
      // partial statistics of 4 pixels over 16 channels, shifted by the first channel's values
      const uint8_t* stat = sT + b * kOTile + stat_off;
      float2 nk[2], s[2], q[2];
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const uint2 w = *reinterpret_cast<const uint2*>(stat + r * 128 + ((g4 ^ (r & 7)) << 4));
        const float2 v[2] = {unpack2<T>(w.x), unpack2<T>(w.y)};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (r == 0) {
            nk[e] = make_float2(-v[e].x, -v[e].y);
            s[e] = make_float2(0.f, 0.f);
            q[e] = s[e];
          }
          const float2 d = __fadd2_rn(v[e], nk[e]);
          s[e] = __fadd2_rn(s[e], d);
          q[e] = __ffma2_rn(d, d, q[e]);
        }
      }
      {
        float pm[4], pq[4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float sx = s[e].x * (1.0f / 16), sy = s[e].y * (1.0f / 16);
          pm[2 * e] = sx - nk[e].x;                       // mean of the 16 samples
          pm[2 * e + 1] = sy - nk[e].y;
          pq[2 * e] = fmaxf(q[e].x - s[e].x * sx, 0.f);   // their sum of squared deviations
          pq[2 * e + 1] = fmaxf(q[e].y - s[e].y * sy, 0.f);
        }
        *reinterpret_cast<float4*>(s_pm + k16 * 128 + p4 * 4) = make_float4(pm[0], pm[1], pm[2], pm[3]);
        *reinterpret_cast<float4*>(s_pq + k16 * 128 + p4 * 4) = make_float4(pq[0], pq[1], pq[2], pq[3]);
      }
      mbar_arrive(&nsync[0]);
      const bool met0 = mbar_wait(&nsync[0], i & 1, g.err, 25);
      if (!__all_sync(0xffffffffu, met0)) break;
      if (tid < 128) {
        // thread = pixel: combine the eight partials (equal counts): M2 = sum M2_k + 16 sum (mean_k - mean)^2
        float pm[8], m = 0.f, m2 = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) { pm[k] = s_pm[k * 128 + tid]; m += pm[k]; m2 += s_pq[k * 128 + tid]; }
        m *= (1.0f / 8);
        float dev = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) dev = fmaf(pm[k] - m, pm[k] - m, dev);
        const long long px = (long long)tile * 128 + tid;
        const float rs = pixel_rstd((m2 + 16.f * dev) * (1.0f / 128), g.eps, px, g.n, g.pitch);
        s_mean[tid] = m;
        s_rstd[tid] = rs;
        if (px < g.M) { g.mean[px] = m; g.rstd[px] = rs; }
        mbar_arrive(&nsync[1]);
      }
      const bool met1 = mbar_wait(&nsync[1], i & 1, g.err, 26);
      if (!__all_sync(0xffffffffu, met1)) break;
      {
        const float4 m0 = *reinterpret_cast<const float4*>(s_mean + pg * 8), m1 = *reinterpret_cast<const float4*>(s_mean + pg * 8 + 4);
        const float4 r0 = *reinterpret_cast<const float4*>(s_rstd + pg * 8), r1 = *reinterpret_cast<const float4*>(s_rstd + pg * 8 + 4);
        const float2 nm[4] = {make_float2(-m0.x, -m0.y), make_float2(-m0.z, -m0.w), make_float2(-m1.x, -m1.y), make_float2(-m1.z, -m1.w)};
        const float2 rr[4] = {make_float2(r0.x, r0.y), make_float2(r0.z, r0.w), make_float2(r1.x, r1.y), make_float2(r1.z, r1.w)};
        const long long px0 = (long long)tile * 128 + pg * 8;   // 8 pixels: all inside the tensor or none
        T* udst = (u_cm != nullptr && px0 < g.M) ? u_cm + (long long)(kp * 8) * g.M + px0 : nullptr;
#pragma unroll 4
        for (int r = 0; r < 8; ++r) {
          uint4* p = reinterpret_cast<uint4*>(part + r * 128 + ((gg ^ r) << 4));
          float2 v[4], o[4];
          unpack8p<T>(*p, v);
          const float gm = s_gamma[kp * 8 + r], bt = s_beta[kp * 8 + r];
          const float2 gm2 = make_float2(gm, gm), bt2 = make_float2(bt, bt);
#pragma unroll
          for (int e = 0; e < 4; ++e) o[e] = __ffma2_rn(__fadd2_rn(v[e], nm[e]), __fmul2_rn(rr[e], gm2), bt2);
          const uint4 w = pack8p<T>(o);
          *p = w;
          if (udst != nullptr) *reinterpret_cast<uint4*>(udst + (long long)r * g.M) = w;
        }
      }
      fence_proxy_async_smem();   // the tile is read next by tcgen05.mma
      __syncwarp();
      if (lane == 0) mbar_arrive(&bnorm[b]);
    }
  } else {
    // ------------------------------------------------------------------ gate epilogue: thread = pixel
    const int quarter = warp & 3, j = (warp - kEpi0) >> 2;   // TMEM lane quarter; 32-channel chunk of the output row
    int i = 0;
    for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, ++i) {
      const int acc = i & 1;
      const bool done = mbar_wait(&tfull[acc], (i >> 1) & 1, g.err, 27);
      if (!__all_sync(0xffffffffu, done)) break;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * 256;
      uint32_t w[16];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        float y[16], gt[16];
        ld16x2_f(t_row + j * 32 + hf * 16, t_row + 128 + j * 32 + hf * 16, y, gt);
#pragma unroll
        for (int e = 0; e < 16; e += 2) {
          const int c = j * 32 + hf * 16 + e;
          float2 yv = make_float2(y[e], y[e + 1]), gv = make_float2(gt[e], gt[e + 1]);
          if (g.bias != nullptr) {
            yv = __fadd2_rn(yv, *reinterpret_cast<const float2*>(g.bias + c));
            gv = __fadd2_rn(gv, *reinterpret_cast<const float2*>(g.bias + 128 + c));
          }
          const float2 r = __fmul2_rn(yv, sigmoid2(gv));
          w[hf * 8 + e / 2] = pack2<T>(r.x, r.y);
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      // four lanes exchange their 16-byte pieces, so that a request writes 64 bytes of eight rows and not 16 of 32
      swap_pieces<1>(w, lane);
      swap_pieces<2>(w, lane);
      const long long m0 = (long long)tile * 128 + quarter * 32 + (lane & ~3);
      if (g.own_pitch) {    // out has its own side: the four pixels lie in one row (the pitch is a multiple of eight)
        const int prow = (int)m0 / g.pitch, col = (int)m0 - prow * g.pitch;
        const long long at = (((long long)prow * g.n + col) * 128 + j * 32) / 8 + (lane & 3);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (prow < g.n && col + q < g.n)
            (reinterpret_cast<uint4*>(g.out) + at)[q * 16] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      } else if (m0 < g.M) {   // M is a multiple of four
        const long long at = (m0 * 128 + j * 32) / 8 + (lane & 3);
        uint4 r[4];
        if (g.residual != nullptr) {
#pragma unroll
          for (int q = 0; q < 4; ++q) r[q] = __ldg(reinterpret_cast<const uint4*>(g.residual) + at + q * 16);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            w[4 * q] = add2<T>(w[4 * q], r[q].x); w[4 * q + 1] = add2<T>(w[4 * q + 1], r[q].y);
            w[4 * q + 2] = add2<T>(w[4 * q + 2], r[q].z); w[4 * q + 3] = add2<T>(w[4 * q + 3], r[q].w);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          (reinterpret_cast<uint4*>(g.out) + at)[q * 16] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T>
int launch_out(cudaStream_t st, const LnGateOut& p) {
  const uint64_t M = (uint64_t)p.M;
  CUtensorMap tmT, tmZ, tmWo, tmWg;
  const bool f16 = p.dtype == TRI_F16;
  const uint64_t td[3] = {M, 128, 1}, ts[2] = {M, 128 * M};
  const uint32_t tbox[3] = {64, 64, 1};
  const uint64_t zd[3] = {128, M, 1}, zs[2] = {128, 128 * M};
  const uint64_t wd[3] = {128, 128, 1}, wsd[2] = {128, 128 * 128};
  const uint32_t box[3] = {64, 128, 1};
  TRI_TRY(make_tmap_3d(&tmT, p.t_cm, 2, f16, td, ts, tbox, false));
  TRI_TRY(make_tmap_3d(&tmZ, p.z, 2, f16, zd, zs, box, false));
  TRI_TRY(make_tmap_3d(&tmWo, p.w_out, 2, f16, wd, wsd, box, false));
  TRI_TRY(make_tmap_3d(&tmWg, p.w_gate, 2, f16, wd, wsd, box, false));
  OutArgs a;
  a.M = p.M; a.tiles = (int)((p.M + 127) / 128); a.eps = p.eps; a.gamma = p.gamma; a.beta = p.beta;
  a.bias = p.bias_out; a.u_cm = p.u_cm; a.mean = p.mean; a.rstd = p.rstd; a.out = p.out; a.residual = p.residual; a.n = p.n; a.pitch = p.pitch; a.own_pitch = p.own_pitch; a.err = p.err;
  constexpr size_t smem = 1024 + kOWBytes + kOBufs * kOTile + (2 * 8 * 128 + 4 * 128) * sizeof(float) + (1 + 3 * kOBufs + 6) * 8 + 16;
  static_assert(smem <= 232448, "shared memory of one CTA");
  auto kern = ln_gate_out_kernel<T>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = std::min(a.tiles, sm_count());
  const double bytes = (p.u_cm ? 4.0 : 3.0) * p.M * 128 * 2;
  KernelTimer kt("tc_ln_gate_out", st, 2.0 * p.M * 128 * 256, bytes);
  launch_dependent(p.first ? kLaunchPlainly : us_of_bytes(bytes), kern, grid, kThreads, smem, st, tmT, tmZ, tmWo, tmWg, a);
  TRI_LAUNCH_OK();
  return 0;
}

// =================================================================================================================
// gate_in_bwd: dP = d sig(G) mask, dG = d P sig (1 - sig) mask for d = da, db, with P and G recomputed from z, and the
// gradients of the input weights, dP^T z and dG^T z
// =================================================================================================================
// 608 threads: warp 0 TMA, warp 1 tcgen05.mma for the projections, warps 2-17 the gate epilogue (thread = channel of the
// half, half of the tile's pixels), warp 18 tcgen05.mma for the weights' gradients and the stores.  A tile is 128 bytes of
// pixels: 64 of 16 bits or 32 of fp32.  As in ln_gate_in the weights stay in shared memory, here those of one half: a CTA has
// one half and its neighbour the other, on the same tiles (z comes from L2 the second time).
// dP and dG leave through a staging tile each and a TMA store: whole 128-byte lines.  Written by the threads, a request
// carried 32 bytes (a channel's rows lie a plane apart), 4096 of them per 128 pixels, and the load / store pipe held the
// kernel at 0.29 ms for 768 x 768 pixels.
// The staging tiles are the weight gradients' operands as they lie (channels x pixels, K = pixels), z's tile the other one
// (MN-major; fp32 has that form in the 32-byte-atom swizzle only and loads the tile a second time).  The sums stay in 256 TMEM
// columns for the life of the CTA, so nothing reads dP, dG and z again for them.  (Two halves per CTA, which would read z once,
// need 512 columns for the sums alone.)
// What bounds it is the chain of an item: gradients from DRAM 2000 to 3500 cycles after they are asked for, products,
// sigmoids, products and store, 2700 cycles per item, no unit above half of its rate.  Hence two sets of eight epilogue warps
// on alternate tiles, an issuing warp for each kind of product (with one, the next tile's projections waited for this one's dP
// and dG), and with fp32 the gradients by the threads themselves, an item ahead, which leaves their shared memory to z and a
// third staging tile; for 16 bits that took longer (258 us against 238), and so did a third or fourth gradient tile in place of
// a staging tile (244 to 261).  Launches in us, with the product over pixels that the sums were before: bf16 768 x 768 256 + 140
// -> 230, 384 x 384 63 + 44 -> 62; fp32 with TF32 products 512 x 512 205 + 127 -> 245.
constexpr int kBwdThreads = 608;
constexpr uint32_t kBTile = 16384;        // z tile: kKb blocks of [kPx rows x 128 bytes]; output tile of a half
template <typename T> struct BwdGeo {
  static constexpr bool kZt = sizeof(T) == 4;                  // a second copy of the z tile, MN-major
  static constexpr int kPx = 128 / sizeof(T), kKb = sizeof(T), kBSub = kPx * 128, kE = kPx / 2;   // kE: an epilogue thread's pixels
  static constexpr bool kGradTiles = sizeof(T) == 2;           // the gradients by TMA; fp32: by the threads
  static constexpr int kZ = kZt ? 2 : 4, kG = kGradTiles ? 2 : 0, kO = kZt ? 3 : 4;   // z tiles; gradient tiles; staging tiles
  static constexpr int kAcc = 128 / kPx;                       // accumulators [P | G] in 256 columns
  static constexpr uint32_t kW = 2 * kKb * kSub;               // weights of a half
  static constexpr uint32_t kTiles = kZ + kZt + kG + kO;
  static constexpr size_t smem = 1024 + kW + kTiles * kBTile + 16 * 64 + (2 * (kZ + 1 + kG + kO + kAcc) + 2) * 8 + 16;
};

struct BwdArgs {
  long long M;
  int tiles;
  const float* bias;
  const void* mask;
  const uint8_t *da, *db;
  bool wide;            // da and db start on 32-byte boundaries
  float* partial;       // [CTA pairs][512][128], if SUMS
  int* err;
};

// 16 bytes of a tile row as pairs
template <typename T, int N> __device__ __forceinline__ void unpack_piece(const uint4& w, float2 (&v)[N]) {
  if constexpr (sizeof(T) == 4) {
    v[0] = make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
    v[1] = make_float2(__uint_as_float(w.z), __uint_as_float(w.w));
  } else {
    unpack8p<T>(w, v);
  }
}
template <typename T, int N> __device__ __forceinline__ uint4 pack_piece(const float2 (&v)[N]) {
  if constexpr (sizeof(T) == 4) return make_uint4(__float_as_uint(v[0].x), __float_as_uint(v[0].y), __float_as_uint(v[1].x), __float_as_uint(v[1].y));
  else return pack8p<T>(v);
}

__device__ __forceinline__ void ldg256(const void* p, uint4& lo, uint4& hi) {
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
               : "l"(p));
}

// SUMS: the weights' gradients are asked for.  Without them no second copy of z and no products on the staging tiles, which the stores
// alone give back: TF32, 512 x 512 pixels, 204 us in place of 252 (the call 1225 and 1285), bf16 768 x 768 218 and 229.
template <typename T, bool SUMS>
__global__ void __launch_bounds__(kBwdThreads, 1)
gate_in_bwd_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmZt, const __grid_constant__ CUtensorMap tmW,
                   const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmO, const BwdArgs g) {
  using G = BwdGeo<T>;
  constexpr int KIND = ElemTraits<T>::kind, kKb = G::kKb, kZ = G::kZ, kG = G::kG, kO = G::kO, kAcc = G::kAcc;
  constexpr bool kZt = G::kZt && SUMS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sW = smem;
  uint8_t* sZ = smem + G::kW;              // [kZ] z tiles
  uint8_t* sT = sZ + kZ * kBTile;          // fp32: the z tile as an MN-major operand
  uint8_t* sG = sT + kZt * kBTile;         // [kG] gradient tiles
  uint8_t* sO = sG + kG * kBTile;          // [kO] dP, dG of an item and the next
  uint8_t* sM = sO + kO * kBTile;          // [16 warps] mask of the warp's pixels
  uint64_t* wfull = reinterpret_cast<uint64_t*>(sM + 16 * 64);
  uint64_t* zfull = wfull + 1;             // [kZ]
  uint64_t* zempty = zfull + kZ;           // [kZ] the products that read the tile are done
  uint64_t* ztfull = zempty + kZ;          // the second copy
  uint64_t* ztempty = ztfull + 1;
  uint64_t* gfull = ztempty + 1;           // [kG] gradient tile
  uint64_t* gempty = gfull + kG;           // [kG] ... copied to registers by its set's 8 epilogue warps
  uint64_t* ofull = gempty + kG;           // [kO] staging tile written by its set's 8 epilogue warps
  uint64_t* oempty = ofull + kO;           // [kO] ... read: by the products (commit), if there are any, and by the store
  uint64_t* tfull = oempty + kO;           // [kAcc] accumulator of an item complete
  uint64_t* tempty = tfull + kAcc;         // [kAcc] ... read by its set's 8 epilogue warps
  uint64_t* sums = tempty + kAcc;          // all products are done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sums + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(wfull, 1);
    for (int b = 0; b < kZ; ++b) { mbar_init(&zfull[b], 1); mbar_init(&zempty[b], 1); }
    mbar_init(ztfull, 1);
    mbar_init(ztempty, 1);
    for (int b = 0; b < kG; ++b) { mbar_init(&gfull[b], 1); mbar_init(&gempty[b], 8); }
    for (int b = 0; b < kO; ++b) { mbar_init(&ofull[b], 8); mbar_init(&oempty[b], SUMS ? 2 : 1); }
    for (int b = 0; b < kAcc; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], 8); }
    mbar_init(sums, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();

  const int tile0 = blockIdx.x >> 1, step = gridDim.x >> 1, half = blockIdx.x & 1;
  const int items = tile0 < g.tiles ? (g.tiles - tile0 + step - 1) / step : 0;
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      mbar_expect_tx(wfull, G::kW);
      for (int blk = 0; blk < 2; ++blk)
        for (int kb = 0; kb < kKb; ++kb) tma_load_3d(sW + (blk * kKb + kb) * kSub, &tmW, wfull, kb * G::kPx, (half * 2 + blk) * 128, 0);
      auto load_z = [&](int i) {
        const int b = i % kZ;
        if (!mbar_wait(&zempty[b], ((i / kZ) & 1) ^ 1, g.err, 60)) return false;
        mbar_expect_tx(&zfull[b], kBTile);
        for (int kb = 0; kb < kKb; ++kb) tma_load_3d(sZ + b * kBTile + kb * G::kBSub, &tmZ, &zfull[b], kb * G::kPx, (tile0 + i * step) * G::kPx, 0);
        return true;
      };
      bool ok = true;
      if constexpr (kZt) {
        for (int i = 0; i < items + 1 && ok; ++i) {   // the second copy of an item behind the first copy of the next
          if (i < items) ok = load_z(i);
          if (i == 0 || !ok) continue;
          ok = mbar_wait(ztempty, i & 1, g.err, 67);   // (i - 1: the item)
          if (!ok) break;
          mbar_expect_tx(ztfull, kBTile);
          for (int c = 0; c < 4; ++c) tma_load_3d(sT + c * G::kBSub, &tmZt, ztfull, c * 32, (tile0 + (i - 1) * step) * G::kPx, 0);
        }
      } else {
        for (int i = 0; i < items && ok; ++i) {
          ok = load_z(i);
          if constexpr (G::kGradTiles) {
            ok = ok && mbar_wait(&gempty[i % kG], ((i / kG) & 1) ^ 1, g.err, 61);
            if (!ok) break;
            mbar_expect_tx(&gfull[i % kG], kBTile);
            tma_load_3d(sG + i % kG * kBTile, half == 0 ? &tmA : &tmB, &gfull[i % kG], (tile0 + i * step) * G::kPx, 0, 0);
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer: the projections
    if (elect_one()) {
      const uint32_t idesc = make_idesc(KIND, 128, G::kPx, false, false);
      const uint32_t w_base = smem_u32(sW), z_base = smem_u32(sZ);
      bool ok = mbar_wait(wfull, 0, g.err, 62);
      for (int i = 0; i < items && ok; ++i) {
        const int b = i % kZ, acc = i % kAcc;
        if (!mbar_wait(&zfull[b], (i / kZ) & 1, g.err, 63)) break;
        if (!mbar_wait(&tempty[acc], ((i / kAcc) & 1) ^ 1, g.err, 64)) break;
        tc_fence_after_sync();
#pragma unroll
        for (int pg = 0; pg < 2; ++pg) {   // P block, G block
          const uint32_t d_addr = tmem_base + (acc * 2 + pg) * G::kPx;
#pragma unroll
          for (int kb = 0; kb < kKb; ++kb)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint64_t ad = make_smem_desc(w_base + (pg * kKb + kb) * kSub + ks * 32, 16, 1024);
              const uint64_t bd = make_smem_desc(z_base + b * kBTile + kb * G::kBSub + ks * 32, 16, 1024);
              umma<KIND>(d_addr, ad, bd, idesc, (kb == 0 && ks == 0) ? 0u : 1u);
            }
        }
        if constexpr (kZt || !SUMS) umma_commit(&zempty[b]);   // (before tfull, which is waited for: nothing is on its way at the end)
        umma_commit(&tfull[acc]);
      }
    }
    __syncwarp();
  } else if (warp == 18) {
    // ------------------------------------------------------------------ MMA issuer: the weights' gradients, and the staging tiles' stores
    if (elect_one()) {
      const uint32_t idesc = make_idesc(KIND, 128, 128, false, true);
      const uint32_t z_base = smem_u32(sZ), t_base = smem_u32(sT), o_base = smem_u32(sO);
      bool ok = true;
      for (int i = 0; i < items && ok; ++i) {
        if (kZt) ok = mbar_wait(ztfull, i & 1, g.err, 69);
#pragma unroll
        for (int pg = 0; pg < 2; ++pg) {
          const int n = 2 * i + pg, ob = n % kO;
          ok = ok && mbar_wait(&ofull[ob], (n / kO) & 1, g.err, 68);
          if (!ok) break;
          if constexpr (SUMS) {
            tc_fence_after_sync();
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint64_t ad = make_smem_desc(o_base + ob * kBTile + ks * 32, 16, 1024);
              const uint64_t bd = kZt ? make_smem_desc(t_base + ks * 8 * 128, G::kBSub, 512, 1)
                                      : make_smem_desc(z_base + (i % kZ) * kBTile + ks * 16 * 128, G::kBSub, 1024);
              umma<KIND>(tmem_base + 256 + pg * 128, ad, bd, idesc, (i == 0 && ks == 0) ? 0u : 1u);
            }
            umma_commit(&oempty[ob]);
            if (pg == 1) umma_commit(kZt ? ztempty : &zempty[i % kZ]);
          }
          tma_store_3d(&tmO, sO + ob * kBTile, (tile0 + i * step) * G::kPx, half * 256 + pg * 128, 0);
          bulk_commit_group();
          if (n > 0) {   // the store before this one has left shared memory
            bulk_wait_group_read1();
            mbar_arrive(&oempty[(n - 1) % kO]);
          }
        }
      }
      if constexpr (SUMS) umma_commit(sums);   // (after a wait that ran out too: the products issued before it)
      bulk_wait_group0();
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ gate epilogue: thread = channel of the half
    const int quarter = warp & 3, j = (warp - 2) >> 2, set = j >> 1;   // TMEM lane quarter; part of the 256 columns of sums
    const int row = quarter * 32 + lane, px0 = (j & 1) * G::kE;
    const uint32_t at = row * 128, sw = row & 7, piece0 = (j & 1) * 4;   // this thread's four pieces of a tile row
    const bool masked = g.mask != nullptr;
    float bp = 0.f, bg = 0.f;
    if (g.bias != nullptr) { bp = g.bias[half * 256 + row]; bg = g.bias[half * 256 + 128 + row]; }
    const float2 bp2 = make_float2(bp, bp), nbg2 = make_float2(-1.4426950408889634f * bg, -1.4426950408889634f * bg);
    constexpr int kPair = 16 / sizeof(T) / 2;   // pairs of pixels in a piece
    // one pixel's mask of the set's next item, on its way for an item's time, and with fp32 this thread's 64 bytes of the gradients
    uint4 dn[4];
    T mn = from_f32<T>(1.f);
    auto fetch = [&](int i) {
      const long long px = (long long)(tile0 + i * step) * G::kPx + px0;
      if constexpr (!G::kGradTiles) {
        const uint8_t* src = (half == 0 ? g.da : g.db) + ((long long)row * g.M + px) * sizeof(T);
        if (g.wide) {
          ldg256(src, dn[0], dn[1]);
          ldg256(src + 32, dn[2], dn[3]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u) dn[u] = __ldg(reinterpret_cast<const uint4*>(src) + u);
        }
      }
      if (masked && lane < G::kE) mn = static_cast<const T*>(g.mask)[px + lane];
    };
    if (set < items) fetch(set);
    T* const wmask = reinterpret_cast<T*>(sM + (warp - 2) * 64);
    bool ok = true;
    for (int i = set; i < items; i += 2) {
      const int acc = i % kAcc;
      uint4 d[4];
      if constexpr (G::kGradTiles) {
        ok = mbar_wait(&gfull[i % G::kG], (i / G::kG) & 1, g.err, 65) && ok;
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = lds128(smem_u32(sG + i % G::kG * kBTile) + at + (((piece0 + u) ^ sw) << 4));
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = dn[u];
      }
      if (masked && lane < G::kE) wmask[lane] = mn;
      __syncwarp();
      if (i + 2 < items) fetch(i + 2);
      ok = mbar_wait(&tfull[acc], (i / kAcc) & 1, g.err, 66) && ok;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * 2 * G::kPx + px0;
      uint8_t* const so0 = sO + 2 * i % kO * kBTile + at;
      uint8_t* const so1 = sO + (2 * i + 1) % kO * kBTile + at;
#pragma unroll
      for (int h = 0; h < G::kE / 16; ++h) {       // 16 pixels at a time
        float p[16], gt[16];
        ld16x2_f(t_row + h * 16, t_row + G::kPx + h * 16, p, gt);
        if constexpr (G::kGradTiles) {
          if (h == 0) {
            // TMA writes the gradient buffer after this arrival.  The buffer's loads are of the generic proxy and TMA's writes of the
            // async proxy, which an mbarrier alone does not order: each lane fences its own loads, here, where they have long returned
            // (right behind them the fence cost 11 of 226 us at 768 x 768 pixels).
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&gempty[i % G::kG]);
          }
        }
        if (h == G::kE / 16 - 1) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[acc]);
        }
        constexpr int kPieces = 16 * sizeof(T) / 16;
#pragma unroll
        for (int uu = 0; uu < kPieces; ++uu) {
          const int u = h * kPieces + uu;
          float2 dv[kPair], mk[kPair], dg[kPair];
          unpack_piece<T>(d[u], dv);
          if (masked) {
            unpack_piece<T>(reinterpret_cast<const uint4*>(wmask)[u], mk);
#pragma unroll
            for (int k = 0; k < kPair; ++k) dv[k] = __fmul2_rn(dv[k], mk[k]);
          }
#pragma unroll
          for (int k = 0; k < kPair; ++k) {
            const int e = uu * 2 * kPair + 2 * k;
            const float2 sg = sigmoid2(make_float2(gt[e], gt[e + 1]), nbg2);
            dv[k] = __fmul2_rn(dv[k], sg);
            const float2 oms = __ffma2_rn(sg, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f));
            dg[k] = __fmul2_rn(__fmul2_rn(dv[k], __fadd2_rn(make_float2(p[e], p[e + 1]), bp2)), oms);
          }
          if (u == 0) {   // the tiles' last products and stores have read them
            const int n0 = 2 * i, n1 = 2 * i + 1;
            ok = mbar_wait(&oempty[n0 % kO], ((n0 / kO) & 1) ^ 1, g.err, 70) && ok;
            ok = mbar_wait(&oempty[n1 % kO], ((n1 / kO) & 1) ^ 1, g.err, 72) && ok;
          }
          const uint32_t c = ((piece0 + u) ^ sw) << 4;
          *reinterpret_cast<uint4*>(so0 + c) = pack_piece<T>(dv);
          *reinterpret_cast<uint4*>(so1 + c) = pack_piece<T>(dg);
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&ofull[2 * i % kO]); mbar_arrive(&ofull[(2 * i + 1) % kO]); }
    }
    // the sums: this thread's row of dP and of dG, a quarter of the 256 columns (no product is under way after the wait)
    if (SUMS && items > 0) {
      ok = mbar_wait(sums, 0, g.err, 71) && ok;
      tc_fence_after_sync();
      float* dst = g.partial + ((long long)tile0 * 512 + half * 256 + (j >> 1) * 128 + row) * 128 + (j & 1) * 64;
#pragma unroll 1
      for (int c = 0; c < 64; c += 32) {
        float v[32];
        ld32_f(tmem_base + ((uint32_t)(quarter * 32) << 16) + 256 + j * 64 + c, v);
        store_rows32<float>(dst + c, v, 128, ok, lane);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

template <typename T, bool SUMS>
int launch_bwd(cudaStream_t st, const GateInBwd& p) {
  const uint64_t M = (uint64_t)p.M;
  CUtensorMap tmZ, tmZt, tmW, tmA, tmB, tmO;
  const bool f16 = p.dtype == TRI_F16;
  const uint64_t zd[3] = {128, M, 1}, zs[2] = {128, 128 * M};
  const uint64_t wd[3] = {128, 512, 1}, wsd[2] = {128, 128 * 512};
  const uint64_t gd[3] = {M, 128, 1}, od[3] = {M, 512, 1}, gs[2] = {M, 512 * M};
  using G = BwdGeo<T>;
  constexpr int E = sizeof(T);
  const uint32_t zbox[3] = {G::kPx, G::kPx, 1}, box[3] = {G::kPx, 128, 1};
  TRI_TRY(make_tmap_3d(&tmZ, p.z, E, f16, zd, zs, zbox, false));
  tmZt = tmZ;
  if (G::kZt && SUMS) TRI_TRY(make_tmap_3d(&tmZt, p.z, E, f16, zd, zs, zbox, true));
  TRI_TRY(make_tmap_3d(&tmW, p.wcat, E, f16, wd, wsd, box, false));
  tmA = tmB = tmW;
  if (G::kGradTiles) {
    TRI_TRY(make_tmap_3d(&tmA, p.da_cm, E, f16, gd, gs, box, false));
    TRI_TRY(make_tmap_3d(&tmB, p.db_cm, E, f16, gd, gs, box, false));
  }
  TRI_TRY(make_tmap_3d(&tmO, p.dpg, E, f16, od, gs, box, false));
  BwdArgs a;
  a.M = p.M; a.tiles = (int)(p.M / G::kPx); a.bias = p.bias_cat; a.mask = p.mask; a.da = static_cast<const uint8_t*>(p.da_cm); a.db = static_cast<const uint8_t*>(p.db_cm);
  a.wide = ((reinterpret_cast<uintptr_t>(p.da_cm) | reinterpret_cast<uintptr_t>(p.db_cm)) & 31) == 0;
  a.partial = p.partial; a.err = p.err;
  static_assert(G::smem <= 232448, "shared memory of one CTA");
  auto kern = gate_in_bwd_kernel<T, SUMS>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::smem));
  const double bytes = 7.0 * p.M * 128 * E;
  KernelTimer kt("tc_gate_in_bwd", st, SUMS ? 2.0 * p.M * 128 * 512 : 0.0, bytes);
  launch_dependent(p.first ? kLaunchPlainly : us_of_bytes(bytes), kern, 2 * gate_in_bwd_parts(p.dtype, p.M), kBwdThreads, G::smem, st, tmZ, tmZt, tmW,
                   tmA, tmB, tmO, a);
  TRI_LAUNCH_OK();
  return 0;
}

}  // namespace

int gate_in_bwd_parts(int dtype, long long M) {
  return (int)std::max(1LL, std::min(M / (dtype == TRI_F32 ? 32 : 64), (long long)sm_count() / 2));
}

// one batch entry (its channel planes are M pixels apart), whole tiles (any square of a multiple of eight)
bool gate_in_bwd_supported(int dtype, long long M, long long plane) {
  return (dtype == TRI_BF16 || dtype == TRI_F16 || dtype == TRI_F32) && M > 0 && M == plane && M % 64 == 0 && M < (1LL << 31) - 128;
}

int gate_in_bwd(cudaStream_t st, const GateInBwd& p) {
  if (!gate_in_bwd_supported(p.dtype, p.M, p.M)) return fail(TRI_ERR_ARG, "gate_in_bwd: unsupported shape or dtype");
  auto start = [&](auto elem) { return p.partial != nullptr ? launch_bwd<decltype(elem), true>(st, p) : launch_bwd<decltype(elem), false>(st, p); };
  if (p.dtype == TRI_F32) return start(float());
  return p.dtype == TRI_BF16 ? start(__nv_bfloat16()) : start(__half());
}

bool ln_gate_in_supported(int dtype, long long M, long long plane) {
  return (dtype == TRI_BF16 || dtype == TRI_F16) && M > 0 && plane > 0 && plane % 8 == 0 && M % plane == 0 &&
         M < (1LL << 31) - 128;
}

int ln_gate_in(cudaStream_t st, const LnGateIn& p) {
  if (!ln_gate_in_supported(p.dtype, p.M, p.plane)) return fail(TRI_ERR_ARG, "ln_gate_in: unsupported shape or dtype");
  return p.dtype == TRI_BF16 ? launch<__nv_bfloat16>(st, p) : launch<__half>(st, p);
}

bool ln_gate_out_supported(int dtype, long long M, long long plane) {
  return (dtype == TRI_BF16 || dtype == TRI_F16) && M > 0 && M == plane && M % 8 == 0 && M < (1LL << 31) - 128;
}

int ln_gate_out(cudaStream_t st, const LnGateOut& p) {
  if (!ln_gate_out_supported(p.dtype, p.M, p.M)) return fail(TRI_ERR_ARG, "ln_gate_out: unsupported shape or dtype");
  return p.dtype == TRI_BF16 ? launch_out<__nv_bfloat16>(st, p) : launch_out<__half>(st, p);
}

}  // namespace tc
}  // namespace tri

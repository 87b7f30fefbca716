// Plain batched GEMM, D = A B^T, on pairs of SMs (tcgen05.mma.cta_group::2): 256 x 256 outputs per pair.
//
// A 128 x 256 tile on one SM reads 12 KB of operands from shared memory per 128 cycles of products (16 k of 16 bits) and gets as much
// by TMA: 192 bytes a cycle where shared memory carries 128, which is what the kernel of tc_gemm.cuh runs at (768 x 768 x 768, 128
// planes, bf16: 116 us, 1.0 PFLOP/s).  In a pair each SM has 128 rows of A and half of B: 8 KB and 8 KB for the same products, and two
// thirds of the reads from L2.  The same product takes 95 us alone and 99 to 107 in loops and steps (1.1 to 1.2 PFLOP/s; 69 by the bytes
// or the measured GEMM rate), with TF32 512 x 512 x 512 72 instead of 78 (62 by the bytes), 32 planes of 1024 x 1024 x 1024 in bf16 51
// instead of 61.
//
// A cluster of two CTAs, 320 threads each, persistent.  Warp 0 fetches this CTA's part of a stage; its bytes count on the stage's
// barrier of the first CTA, whose warp 1 issues the products for both and commits to the barriers of both; warps 2-9 are the epilogue:
// this CTA's 128 rows of the accumulator, double buffered (2 x 256 columns).  They free a buffer by arriving at the first CTA's barrier.
// No load is multicast.  Every mbarrier wait is bounded.
#include <algorithm>

#include "tc_gemm.cuh"

namespace tri {
namespace tc {

namespace {

constexpr int kPairStages = 6, kPairThreads = 320, kPairStage = 2 * kStageA;   // bytes: 128 rows of A and of B

struct PairArgs {
  int M, N, kblocks, batches, tiles_m, tiles_n;
  int a_mn, b_mn;
  uint32_t idesc;
  void* out;
  long long ld_out, batch_out;
  int* err;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of the same variable in the pair's first CTA
__device__ __forceinline__ uint32_t in_first(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(0));
  return a;
}
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* m, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"((uint64_t)m), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
template <int KIND>
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (KIND == KIND_TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}
// arrive on `bar` of both CTAs once the products issued so far are done
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

template <typename TIN, typename TOUT>
__global__ void __launch_bounds__(kPairThreads, 1)
tc_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const PairArgs g) {
  constexpr int ES = sizeof(TIN), BKE = 128 / ES, UK = 32 / ES, CE = 128 / ES;   // as in tc_gemm_kernel
  constexpr uint32_t MN_SBO = ES == 4 ? 512 : 1024, MN_LAYOUT = ES == 4 ? 1 : 2;
  constexpr int KIND = ElemTraits<TIN>::kind == KIND_TF32 ? KIND_TF32 : KIND_F16;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStage);   // [stages], of the first CTA: both parts have landed
  uint64_t* empty = full + kPairStages;      // [stages]: the products have read this CTA's part
  uint64_t* tfull = empty + kPairStages;     // [2] accumulator complete
  uint64_t* tempty = tfull + 2;              // [2], of the first CTA: the epilogue warps of both have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 16); }
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();   // both CTAs' barriers are there
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  dependent_enter();

  const int total = g.batches * g.tiles_m * g.tiles_n;
  auto decode = [&](int tile, int& tm, int& tn, int& bz) {
    tn = tile % g.tiles_n; tile /= g.tiles_n;
    tm = tile % g.tiles_m;
    bz = tile / g.tiles_m;
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < total && ok; tile += pairs) {
        int tm, tn, bz;
        decode(tile, tm, tn, bz);
        const int m0 = tm * 256 + rank * 128, n0 = tn * 256 + rank * 128;
        for (int kb = 0; kb < g.kblocks; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1, g.err, 91)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * kPairStage);
          const uint32_t bar = in_first(&full[stage]);
          uint8_t *a = smem + stage * kPairStage, *b = a + kStageA;
          if (!g.a_mn) tma_load_pair(a, &tmA, bar, kb * BKE, m0, bz);
          else for (int c = 0; c < 128 / CE; ++c) tma_load_pair(a + c * (BKE * 128), &tmA, bar, m0 + c * CE, kb * BKE, bz);
          if (!g.b_mn) tma_load_pair(b, &tmB, bar, kb * BKE, n0, bz);
          else for (int c = 0; c < 128 / CE; ++c) tma_load_pair(b + c * (BKE * 128), &tmB, bar, n0 + c * CE, kb * BKE, bz);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer of the pair
    if (rank == 0 && elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      const uint32_t base = smem_u32(smem);
      for (int tile = pair; tile < total && ok; tile += pairs) {
        if (!mbar_wait(&tempty[acc], acc_phase ^ 1, g.err, 92)) break;
        tc_fence_after_sync();
        for (int kb = 0; kb < g.kblocks; ++kb) {
          if (!mbar_wait(&full[stage], phase, g.err, 93)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t a = base + stage * kPairStage, b = a + kStageA;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint64_t ad = g.a_mn ? make_smem_desc(a + ks * UK * 128, BKE * 128, MN_SBO, MN_LAYOUT) : make_smem_desc(a + ks * 32, 16, 1024);
            const uint64_t bd = g.b_mn ? make_smem_desc(b + ks * UK * 128, BKE * 128, MN_SBO, MN_LAYOUT) : make_smem_desc(b + ks * 32, 16, 1024);
            umma_pair<KIND>(tmem_base + acc * 256, ad, bd, g.idesc, kb > 0 || ks > 0 ? 1u : 0u);
          }
          commit_pair(&empty[stage]);
          if (++stage == kPairStages) { stage = 0; phase ^= 1; }
        }
        if (ok) commit_pair(&tfull[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ epilogue: thread = row, two groups of warps with every other 32 columns
    const int quarter = warp & 3, grp = (warp - 2) >> 2, row = quarter * 32 + lane;
    const bool vec_ok = (g.ld_out * sizeof(TOUT)) % 16 == 0 && (g.batch_out * sizeof(TOUT)) % 16 == 0 && (reinterpret_cast<uintptr_t>(g.out) & 15) == 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < total; tile += pairs) {
      int tm, tn, bz;
      decode(tile, tm, tn, bz);
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull[acc], acc_phase, g.err, 94))) break;
      tc_fence_after_sync();
      const int m = tm * 256 + rank * 128 + row;
      const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * 256;
      TOUT* out = reinterpret_cast<TOUT*>(g.out) + bz * g.batch_out + (long long)m * g.ld_out;
#pragma unroll 1
      for (int j = grp; j < 8; j += 2) {
        float v[32];
        ld32_f(t_row + j * 32, v);
        const int n = tn * 256 + j * 32;
        if ((g.M & 3) == 0 && vec_ok && g.N - n >= 32) store_rows32<TOUT>(out + n, v, g.ld_out, m < g.M, lane);
        else if (m < g.M && n < g.N) store_row32<TOUT>(out + n, v, g.N - n, vec_ok);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(in_first(&tempty[acc])) : "memory");
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();   // the other CTA's products and arrivals reach into this one
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

template <typename T>
int start(cudaStream_t st, const CUtensorMap& ta, const CUtensorMap& tb, const PairArgs& a, const GemmPlan& p) {
  constexpr size_t smem = 1024 + kPairStages * kPairStage + (2 * kPairStages + 4) * 8 + 16;
  auto kern = tc_gemm_pair_kernel<T, T>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long total = (long long)a.batches * a.tiles_m * a.tiles_n;
  KernelTimer kt(p.pair_name != nullptr ? p.pair_name : p.name, st, p.flops, p.bytes);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = 2 * (unsigned)std::min<long long>(total, sm_count() / 2);
  cfg.blockDim = kPairThreads; cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = attr;
  cfg.numAttrs = !p.first && us_of_bytes(p.bytes) < kEarlyStartUs ? 2 : 1;   // (see launch_dependent)
  cudaLaunchKernelEx(&cfg, kern, ta, tb, a);
  TRI_LAUNCH_OK();
  return 0;
}

}  // namespace

bool gemm_pair_fits(const GemmPlan& p, int width, int kblocks, int es) {
  if (p.K1 > 0 || p.split_k || p.a_tiles > 0 || p.bias0 != nullptr) return false;
  // A tile's products must outlast the stores of the one before, 256 KB of fp32 or half of that.  128 planes of 512 x 512, us on single
  // SMs and on pairs: 16 bits K = 512 (8 blocks of 128 bytes) 41.3 and 42.9, 576 45.4 and 45.3, 640 49.3 and 47.2, 768 55.5 and 50.0;
  // TF32 K = 256 (8) 50.1 and 55.4, 320 57.2 and 58.0, 384 63.5 and 60.9, 512 78.0 and 71.9.  64 planes of 768 x 768 and 32 of
  // 1024 x 1024 cross there or one block earlier.
  if (kblocks < (es == 4 ? 12 : 9)) return false;
  const auto up = [](long long v, long long u) { return (v + u - 1) / u * u; };
  // The products of a pair's tiles beyond the matrix must not outweigh what it saves (a side of 384, training: 380 us without, 395 with),
  // and there must be two tiles for a pair (256, one and three quarters: 203.5 us without, 206 with).
  return up(p.M, 256) * up(p.N, 256) * 16 <= up(p.M, 128) * up(p.N, width) * 17 && p.batches * up(p.M, 256) * up(p.N, 256) / 65536 >= sm_count();
}

int launch_gemm_pair(cudaStream_t st, int dtype, const CUtensorMap& ta, const CUtensorMap& tb, const GemmPlan& p, int* err) {
  const int bke = dtype == TRI_F32 ? 32 : 64;
  PairArgs a;
  a.M = p.M; a.N = p.N; a.kblocks = (p.K0 + bke - 1) / bke; a.batches = p.batches; a.tiles_m = (p.M + 255) / 256; a.tiles_n = (p.N + 255) / 256;
  a.a_mn = p.a[0].mn_major; a.b_mn = p.b[0].mn_major;
  a.idesc = make_idesc(dtype == TRI_F32 ? KIND_TF32 : dtype == TRI_BF16 ? KIND_BF16 : KIND_F16, 256, 256, a.a_mn, a.b_mn);
  a.out = p.out0; a.ld_out = p.ld_out; a.batch_out = p.batch_out; a.err = err;
  switch (dtype) {
    case TRI_F32: return start<float>(st, ta, tb, a, p);
    case TRI_BF16: return start<__nv_bfloat16>(st, ta, tb, a, p);
    case TRI_F16: return start<__half>(st, ta, tb, a, p);
  }
  return fail(TRI_ERR_ARG, "bad dtype %d", dtype);
}

}  // namespace tc
}  // namespace tri

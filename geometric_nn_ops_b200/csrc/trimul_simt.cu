// Exact-fp32 (CUDA-core) path of the triangle multiplicative update.
//
// This is the path behind fp32 inputs with matmul precision "ieee" (no tensor
// core offers exact fp32 products) and behind every shape the tensor-core path
// does not cover.  All intermediates are fp32 and pixel-major ([B*N*N, channels]);
// only the tensors that cross the ABI (x, mask, weights, out, d_out, dx) are in
// the caller's dtype.  With precision == tf32 the operands of every product are
// rounded to the tf32 grid first, so the two precisions differ bitwise as the
// reference's do (tests/test_trimul.py:185-201 of the reference).
//
// Math follows trimul_torch (geometric_nn_ops_torch/triangle/_reference/trimul.py:57-97).
#include <algorithm>

#include "common.cuh"
#include "trimul_simt.cuh"

namespace tri {
namespace simt {

__device__ __forceinline__ int cdiv_dev(int a, int b) { return (a + b - 1) / b; }

// ============================================================================
// generic strided GEMM   C[m,n] (+)= sum_k A(m,k) * B(n,k)  (+ bias[n])
// ============================================================================
struct GemmP {
  const float* A;
  const float* B;
  float* C;
  const float* bias;
  int M, N, K;
  long long a_m, a_k, b_n, b_k, c_m, c_n;
  int ksplit;
  long long c_split;
  int accumulate;
};

// A tile of 16 T x 16 T outputs, T x T per thread (two runs of T / 2 or one of T, so that operands are read four at a time), K in steps
// of 16 through double-buffered shared memory; the next step's operands are fetched into registers while this one runs.
// T = 8 reads 4 x 16 bytes per 64 FMAs, T = 4 reads 2 per 16; a 4 x 4 tile of scalar reads, eight per 16, was bound by
// them.
template <int T, bool TF32>
__global__ void __launch_bounds__(256, 2) gemm_kernel(GemmP p) {
  constexpr int W = 16 * T, E = T;            // tile width; elements of one operand per thread and step
  __shared__ __align__(16) float As[2][16][W + 4];
  __shared__ __align__(16) float Bs[2][16][W + 4];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * W, n0 = blockIdx.x * W;
  int kper = (p.K + p.ksplit - 1) / p.ksplit;
  kper = (kper + 15) / 16 * 16;
  const int kbeg = blockIdx.z * kper;
  const int kend = min(p.K, kbeg + kper);
  float ra[E], rb[E];
  // an element's row and k: sixteen k of E rows where k is contiguous, else W rows and every (256 / W)-th k
  const bool ak = p.a_k == 1, bk = p.b_k == 1;
  const int a_row = ak ? tid >> 4 : tid % W, a_kk = ak ? tid & 15 : tid / W, b_row = bk ? tid >> 4 : tid % W, b_kk = bk ? tid & 15 : tid / W;
  const int a_dr = ak ? 16 : 0, a_dk = ak ? 0 : 256 / W, b_dr = bk ? 16 : 0, b_dk = bk ? 0 : 256 / W;
  const float* pa = p.A + (long long)(m0 + a_row) * p.a_m + (long long)(kbeg + a_kk) * p.a_k;
  const float* pb = p.B + (long long)(n0 + b_row) * p.b_n + (long long)(kbeg + b_kk) * p.b_k;
  const long long a_e = a_dr * p.a_m + a_dk * p.a_k, b_e = b_dr * p.b_n + b_dk * p.b_k;
  const bool whole = m0 + W <= p.M && n0 + W <= p.N;
  auto fetch = [&](int k0) {
    const float *qa = pa, *qb = pb;
    if (whole && k0 + 16 <= kend) {
#pragma unroll
      for (int e = 0; e < E; ++e, qa += a_e, qb += b_e) { ra[e] = *qa; rb[e] = *qb; }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e, qa += a_e, qb += b_e) {
        ra[e] = m0 + a_row + e * a_dr < p.M && k0 + a_kk + e * a_dk < kend ? *qa : 0.f;
        rb[e] = n0 + b_row + e * b_dr < p.N && k0 + b_kk + e * b_dk < kend ? *qb : 0.f;
      }
    }
    pa += 16 * p.a_k;
    pb += 16 * p.b_k;
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      As[buf][a_kk + e * a_dk][a_row + e * a_dr] = TF32 ? round_tf32(ra[e]) : ra[e];
      Bs[buf][b_kk + e * b_dk][b_row + e * b_dr] = TF32 ? round_tf32(rb[e]) : rb[e];
    }
  };
  float2 acc[T / 2][T] = {};   // rows 2 r, 2 r + 1 packed
  if (kbeg < kend) { fetch(kbeg); put(0); }
  for (int k0 = kbeg, buf = 0; k0 < kend; k0 += 16, buf ^= 1) {
    __syncthreads();
    const bool more = k0 + 16 < kend;
    if (more) fetch(k0 + 16);
#pragma unroll 4
    for (int kk = 0; kk < 16; ++kk) {
      float a[T], b[T];
#pragma unroll
      for (int h = 0; h < T / 4; ++h) {
        const float4 x = *reinterpret_cast<const float4*>(&As[buf][kk][h * 64 + ty * 4]);
        const float4 y = *reinterpret_cast<const float4*>(&Bs[buf][kk][h * 64 + tx * 4]);
        a[h * 4] = x.x; a[h * 4 + 1] = x.y; a[h * 4 + 2] = x.z; a[h * 4 + 3] = x.w;
        b[h * 4] = y.x; b[h * 4 + 1] = y.y; b[h * 4 + 2] = y.z; b[h * 4 + 3] = y.w;
      }
#pragma unroll
      for (int c = 0; c < T; ++c)
#pragma unroll
        for (int r = 0; r < T / 2; ++r) acc[r][c] = __ffma2_rn(make_float2(a[2 * r], a[2 * r + 1]), make_float2(b[c], b[c]), acc[r][c]);
    }
    if (more) put(buf ^ 1);
  }
  float* C = p.C + (long long)blockIdx.z * p.c_split;
#pragma unroll
  for (int r = 0; r < T; ++r) {
    const int m = m0 + (r >> 2) * 64 + ty * 4 + (r & 3);
    if (m >= p.M) continue;
#pragma unroll
    for (int c = 0; c < T; ++c) {
      const int n = n0 + (c >> 2) * 64 + tx * 4 + (c & 3);
      if (n >= p.N) continue;
      float v = r & 1 ? acc[r >> 1][c].y : acc[r >> 1][c].x;
      if (p.bias != nullptr && blockIdx.z == 0) v += p.bias[n];
      const long long o = (long long)m * p.c_m + (long long)n * p.c_n;
      if (p.accumulate) v += C[o];
      C[o] = v;
    }
  }
}

// 128 x 128 tiles where there is one for every SM, else 64 x 64
static int gemm(cudaStream_t st, bool tf32, GemmP p) {
  if (p.M <= 0 || p.N <= 0) return 0;
  KernelTimer kt("simt_gemm", st, 2.0 * p.M * p.N * p.K, 4.0 * ((double)p.M * p.K + (double)p.N * p.K + (double)p.M * p.N));
  const bool wide = (long long)cdiv(p.N, 128) * cdiv(p.M, 128) * p.ksplit >= 148 && p.M > 64 && p.N > 64;
  const int w = wide ? 128 : 64;
  const dim3 grid(cdiv(p.N, w), cdiv(p.M, w), p.ksplit);
  if (wide) {
    if (tf32) gemm_kernel<8, true><<<grid, 256, 0, st>>>(p);
    else gemm_kernel<8, false><<<grid, 256, 0, st>>>(p);
  } else {
    if (tf32) gemm_kernel<4, true><<<grid, 256, 0, st>>>(p);
    else gemm_kernel<4, false><<<grid, 256, 0, st>>>(p);
  }
  TRI_LAUNCH_OK();
  return 0;
}

// out[j] = sum_p partial[p*n + j]
__global__ void reduce_partials_kernel(const float* partial, int nparts, long long n, float* out) {
  long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (j >= n) return;
  float s = 0.f;
  for (int p = 0; p < nparts; ++p) s += partial[(long long)p * n + j];
  out[j] = s;
}

static int reduce_partials(cudaStream_t st, const float* partial, int nparts, long long n, float* out) {
  KernelTimer kt("simt_reduce_partials", st, 0.0, 4.0 * (nparts + 1) * n);
  reduce_partials_kernel<<<cdiv(n, 256), 256, 0, st>>>(partial, nparts, n, out);
  TRI_LAUNCH_OK();
  return 0;
}

// dW[n_out, n_in] = sum_rows D[row, n_out] * Z[row, n_in], split over rows, deterministic.
static int weight_grad(cudaStream_t st, bool tf32, const float* D, int ldd, int n_out, const float* Z,
                       int ldz, int n_in, long long rows, float* partial, int ksplit, float* out) {
  GemmP p{};
  p.A = D; p.a_m = 1; p.a_k = ldd;
  p.B = Z; p.b_n = 1; p.b_k = ldz;
  p.C = partial; p.c_m = n_in; p.c_n = 1;
  p.M = n_out; p.N = n_in; p.K = (int)rows;
  p.ksplit = ksplit; p.c_split = (long long)n_out * n_in;
  TRI_TRY(gemm(st, tf32, p));
  return reduce_partials(st, partial, ksplit, (long long)n_out * n_in, out);
}

// ============================================================================
// per-channel contraction  O[p,q,c] = sum_r X(p,r,c) * Y(q,r,c)
// ============================================================================
struct ContractP {
  const float* X;
  const float* Y;
  float* O;
  int N, Ch;
  long long xs_p, xs_r, ys_q, ys_r, os_p, os_q;  // pixel strides inside one N x N plane
  int ldx, ldy, ldo;                             // channels per pixel in each buffer
  int xoff, yoff, ooff;                          // first channel inside the buffer
  int vec;                                       // channels can be copied four at a time
};

// A CTA has PT x QT output pixels of 32 channels (lane = channel) and steps through the r axis R pixels at a time, double-
// buffered by cp.async; each of its eight warps has TP x TQ of the pixels in registers.  TP + TQ shared loads feed TP * TQ
// FMAs: at 16 x 8 the FMAs bound it (32 TFLOP/s at 384 residues).  One thread per channel reading 8 x 8 pixels from global
// memory took a byte of L2 traffic per FMA and was bound by that (6.6 TFLOP/s; 66 us at 64 residues against 8).
template <int TP, int TQ>
struct ContractTile {
  static constexpr int kWarpsP = TP == 16 ? 2 : 4, kWarpsQ = 8 / kWarpsP, PT = TP * kWarpsP, QT = TQ * kWarpsQ;
  static constexpr int R = TP == 4 ? 16 : 8, kStage = R * (PT + QT) * 32, kSmem = 2 * kStage * 4;
};

template <int TP, int TQ, bool TF32>
__global__ void __launch_bounds__(256) contract_kernel(ContractP p) {
  using L = ContractTile<TP, TQ>;
  constexpr int PT = L::PT, QT = L::QT, R = L::R;
  extern __shared__ __align__(16) float sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cblocks = cdiv_dev(p.Ch, 32), cb = blockIdx.z % cblocks, b = blockIdx.z / cblocks, c0 = cb * 32;
  const int p0 = blockIdx.x * PT, q0 = blockIdx.y * QT;
  const long long plane = (long long)b * p.N * p.N;
  // this thread's copies: four channels of one row of X and one of Y, every 32 / PT (32 / QT) th r
  const int c4 = c0 + (threadIdx.x & 7) * 4, slot = threadIdx.x >> 3, left = p.Ch - c4;
  const int xr = slot / PT, xrow = slot % PT, yr = slot / QT, yrow = slot % QT;
  const float* X = p.X + p.xoff + (plane + min(p0 + xrow, p.N - 1) * p.xs_p + xr * p.xs_r) * p.ldx + c4;
  const float* Y = p.Y + p.yoff + (plane + min(q0 + yrow, p.N - 1) * p.ys_q + yr * p.ys_r) * p.ldy + c4;
  const long long x_step = p.xs_r * p.ldx * (32 / PT), y_step = p.ys_r * p.ldy * (32 / QT);
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  const uint32_t xd = base + ((xr * PT + xrow) * 32 + (threadIdx.x & 7) * 4) * 4, yd = base + (R * PT * 32 + (yr * QT + yrow) * 32 + (threadIdx.x & 7) * 4) * 4;
  auto copy = [&](uint32_t dst, const float* src, bool live, const float* safe) {
    if (p.vec) {
      const bool on = live && left > 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(on ? src : safe), "r"(on ? 16 : 0) : "memory");
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool on = live && e < left;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * e), "l"(on ? src + e : safe), "r"(on ? 4 : 0) : "memory");
      }
    }
  };
  dependent_trigger();
  auto issue = [&](int r0, int buf) {
#pragma unroll
    for (int e = 0; e < R * PT / 32; ++e, X += x_step) copy(xd + buf * L::kStage * 4 + e * 32 * 128, X, r0 + xr + e * (32 / PT) < p.N, p.X);
#pragma unroll
    for (int e = 0; e < R * QT / 32; ++e, Y += y_step) copy(yd + buf * L::kStage * 4 + e * 32 * 128, Y, r0 + yr + e * (32 / QT) < p.N, p.Y);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int wp = warp / L::kWarpsQ * TP, wq = warp % L::kWarpsQ * TQ;
  float2 acc[TP / 2][TQ] = {};   // pixels 2 i, 2 i + 1 packed
  issue(0, 0);
  for (int r0 = 0, buf = 0; r0 < p.N; r0 += R, buf ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (r0 + R < p.N) issue(r0 + R, buf ^ 1);
    const float* xs = sm + buf * L::kStage + wp * 32 + lane;
    const float* ys = sm + buf * L::kStage + R * PT * 32 + wq * 32 + lane;
#pragma unroll 2
    for (int r = 0; r < R; ++r) {
      float xv[TP], yv[TQ];
#pragma unroll
      for (int j = 0; j < TQ; ++j) yv[j] = TF32 ? round_tf32(ys[(r * QT + j) * 32]) : ys[(r * QT + j) * 32];
#pragma unroll
      for (int i = 0; i < TP; ++i) xv[i] = TF32 ? round_tf32(xs[(r * PT + i) * 32]) : xs[(r * PT + i) * 32];
#pragma unroll
      for (int j = 0; j < TQ; ++j)
#pragma unroll
        for (int i = 0; i < TP / 2; ++i) acc[i][j] = __ffma2_rn(make_float2(xv[2 * i], xv[2 * i + 1]), make_float2(yv[j], yv[j]), acc[i][j]);
    }
  }
  if (c0 + lane >= p.Ch) return;
#pragma unroll
  for (int i = 0; i < TP; ++i) {
    if (p0 + wp + i >= p.N) continue;
#pragma unroll
    for (int j = 0; j < TQ; ++j) {
      if (q0 + wq + j >= p.N) continue;
      p.O[(plane + (p0 + wp + i) * p.os_p + (q0 + wq + j) * p.os_q) * p.ldo + p.ooff + c0 + lane] = i & 1 ? acc[i >> 1][j].y : acc[i >> 1][j].x;
    }
  }
}

template <int TP, int TQ>
static int contract_start(cudaStream_t st, bool tf32, int B, const ContractP& p) {
  using L = ContractTile<TP, TQ>;
  const auto kern = tf32 ? contract_kernel<TP, TQ, true> : contract_kernel<TP, TQ, false>;
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmem));
  const dim3 grid(cdiv(p.N, L::PT), cdiv(p.N, L::QT), B * cdiv(p.Ch, 32));
  KernelTimer kt("simt_contract", st, 2.0 * B * p.N * (double)p.N * p.N * p.Ch, 12.0 * B * (double)p.N * p.N * p.Ch);
  kern<<<grid, 256, L::kSmem, st>>>(p);
  TRI_LAUNCH_OK();
  return 0;
}

// The largest tile that still makes a CTA for every SM; of the two smaller ones the larger from 100 CTAs on.  128 channels, fp32,
// us with 16 x 8, 8 x 8 and 4 x 4 pixels a warp: N = 96 (72 CTAs of 8 x 8) 39, 25, 19; N = 104 (112) 42, 26, 29; N = 128 (128) 48,
// 29, 37; N = 192 (144 CTAs of 16 x 8) 69, 64, 93; N = 256 (256) 164, 150, 206.
static int contract(cudaStream_t st, bool tf32, int B, ContractP p) {
  p.vec = p.ldx % 4 == 0 && p.ldy % 4 == 0 && p.xoff % 4 == 0 && p.yoff % 4 == 0 && p.Ch % 4 == 0;
  const long long planes = (long long)B * cdiv(p.Ch, 32);
  if (planes * cdiv(p.N, 32) * cdiv(p.N, 32) >= 148) return contract_start<16, 8>(st, tf32, B, p);
  if (planes * cdiv(p.N, 32) * cdiv(p.N, 16) >= 100) return contract_start<8, 8>(st, tf32, B, p);
  return contract_start<4, 4>(st, tf32, B, p);
}

// ============================================================================
// LayerNorm forward / backward (one warp per row)
// ============================================================================
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename TI>
__global__ void __launch_bounds__(256) ln_fwd_kernel(const TI* x, const float* gamma, const float* beta,
                                                      float eps, long long M, int C, float* z,
                                                      float* mean, float* rstd) {
  const int lane = threadIdx.x & 31;
  long long row = blockIdx.x * 8LL + (threadIdx.x >> 5);
  if (row >= M) return;
  const TI* xr = x + row * C;
  float s = 0.f;
  for (int c = lane; c < C; c += 32) s += to_f32(xr[c]);
  const float mu = warp_sum(s) / C;
  float v = 0.f;
  for (int c = lane; c < C; c += 32) { float d = to_f32(xr[c]) - mu; v += d * d; }
  const float rs = 1.0f / sqrtf(warp_sum(v) / C + eps);
  for (int c = lane; c < C; c += 32) {
    float h = (to_f32(xr[c]) - mu) * rs;
    if (gamma) h *= gamma[c];
    if (beta) h += beta[c];
    z[row * C + c] = h;
  }
  if (lane == 0) { mean[row] = mu; rstd[row] = rs; }
}

// d_in = rstd * (dhat - mean(dhat) - xhat * mean(dhat * xhat)), dhat = d_out * gamma.
// Per-block partial sums of d_out*xhat and d_out go to pg/pb [gridDim.x, C].
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) ln_bwd_kernel(const float* d_out, const TI* x, const float* mean,
                                                      const float* rstd, const float* gamma, long long M,
                                                      int C, TO* d_in, float* pg, float* pb) {
  extern __shared__ float sm[];  // [8][C] dgamma, [8][C] dbeta
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* sg = sm + warp * C;
  float* sb = sm + (8 + warp) * C;
  for (int c = lane; c < C; c += 32) { sg[c] = 0.f; sb[c] = 0.f; }
  for (long long row = blockIdx.x * 8LL + warp; row < M; row += gridDim.x * 8LL) {
    const float mu = mean[row], rs = rstd[row];
    const TI* xr = x + row * C;
    const float* dr = d_out + row * C;
    float s1 = 0.f, s2 = 0.f;
    for (int c = lane; c < C; c += 32) {
      float h = (to_f32(xr[c]) - mu) * rs;
      float d = dr[c];
      float dh = gamma ? d * gamma[c] : d;
      s1 += dh;
      s2 += dh * h;
      sg[c] += d * h;
      sb[c] += d;
    }
    const float m1 = warp_sum(s1) / C, m2 = warp_sum(s2) / C;
    for (int c = lane; c < C; c += 32) {
      float h = (to_f32(xr[c]) - mu) * rs;
      float dh = gamma ? dr[c] * gamma[c] : dr[c];
      d_in[row * C + c] = from_f32<TO>(rs * (dh - m1 - h * m2));
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += 256) {
    float g = 0.f, b = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) { g += sm[w * C + c]; b += sm[(8 + w) * C + c]; }
    pg[(long long)blockIdx.x * C + c] = g;
    pb[(long long)blockIdx.x * C + c] = b;
  }
}

constexpr int kLnBwdBlocks = 296;

template <typename TI, typename TO>
static int ln_bwd(cudaStream_t st, const float* d_out, const TI* x, const float* mean, const float* rstd,
                  const float* gamma, long long M, int C, TO* d_in, float* partial /*2*blocks*C*/,
                  float* dgamma, float* dbeta) {
  int blocks = (int)std::min<long long>(kLnBwdBlocks, (M + 7) / 8);
  size_t smem = 16 * (size_t)C * sizeof(float);
  auto kern = ln_bwd_kernel<TI, TO>;
  if (smem > 48 * 1024) TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  float* pg = partial;
  float* pb = partial + (size_t)blocks * C;
  {
    KernelTimer kt("simt_ln_bwd", st, 0.0, (double)M * C * (4.0 + sizeof(TI) + sizeof(TO)));
    kern<<<blocks, 256, smem, st>>>(d_out, x, mean, rstd, gamma, M, C, d_in, pg, pb);
    TRI_LAUNCH_OK();
  }
  if (dgamma) TRI_TRY(reduce_partials(st, pg, blocks, C, dgamma));
  if (dbeta) TRI_TRY(reduce_partials(st, pb, blocks, C, dbeta));
  return 0;
}

// ============================================================================
// elementwise stages
// ============================================================================
template <typename T>
__global__ void convert_kernel(const T* src, float* dst, long long n) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) dst[i] = to_f32(src[i]);
}

// ab = P * sigmoid(G) * mask  over [M, W]
__global__ void gate_in_kernel(const float* P, const float* G, const float* mask, long long M, int W, float* ab) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= M * W) return;
  float v = P[i] * sigmoidf_acc(G[i]);
  if (mask) v *= mask[i / W];
  ab[i] = v;
}

__global__ void gate_in_bwd_kernel(const float* dab, const float* P, const float* G, const float* mask,
                                   long long M, int W, float* dP, float* dG) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= M * W) return;
  float d = dab[i];
  if (mask) d *= mask[i / W];
  float g = sigmoidf_acc(G[i]);
  dP[i] = d * g;
  dG[i] = d * P[i] * g * (1.0f - g);
}

template <typename T>
__global__ void gate_out_kernel(const float* y, const float* go, long long n, T* out) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = from_f32<T>(y[i] * sigmoidf_acc(go[i]));
}

template <typename T>
__global__ void gate_out_bwd_kernel(const T* d_out, const float* y, const float* go, long long n, float* dy, float* dgo) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float d = to_f32(d_out[i]);
  float g = sigmoidf_acc(go[i]);
  dy[i] = d * g;
  dgo[i] = d * y[i] * g * (1.0f - g);
}

// partial[blockIdx.x][c] = sum over this block's rows of X[row, c]
__global__ void colsum_kernel(const float* X, long long M, int C, float* partial) {
  int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= C) return;
  long long per = (M + gridDim.x - 1) / gridDim.x;
  long long r0 = blockIdx.x * per, r1 = min(M, r0 + per);
  float s = 0.f;
  for (long long r = r0; r < r1; ++r) s += X[r * C + c];
  partial[(long long)blockIdx.x * C + c] = s;
}

constexpr int kColsumBlocks = 256;
static int colsum(cudaStream_t st, const float* X, long long M, int C, float* partial, float* out) {
  dim3 grid(kColsumBlocks, cdiv(C, 128));
  KernelTimer kt("simt_colsum", st, 0.0, 4.0 * M * C);
  colsum_kernel<<<grid, 128, 0, st>>>(X, M, C, partial);
  TRI_LAUNCH_OK();
  return reduce_partials(st, partial, kColsumBlocks, C, out);
}

#define EW_GRID(n) cdiv((n), 256), 256, 0, st

// ============================================================================
// memory plan
// ============================================================================
struct WeightsF32 {
  float *norm_in_w, *norm_in_b, *p_in_w, *p_in_b, *g_in_w, *g_in_b;
  float *norm_out_w, *norm_out_b, *p_out_w, *p_out_b, *g_out_w, *g_out_b, *mask;
};

struct Saved {
  float *z, *P, *G, *ab, *t, *y, *go, *mean_in, *rstd_in, *mean_out, *rstd_out;
};

static size_t carve_saved(Arena& a, const TriMulDesc* d, Saved* s) {
  const size_t M = (size_t)d->B * d->N * d->N;
  s->z = a.take<float>(M * d->C);
  s->P = a.take<float>(M * 2 * d->Ch);
  s->G = a.take<float>(M * 2 * d->Ch);
  s->ab = a.take<float>(M * 2 * d->Ch);
  s->t = a.take<float>(M * d->Ch);
  s->y = a.take<float>(M * d->C);
  s->go = a.take<float>(M * d->C);
  s->mean_in = a.take<float>(M);
  s->rstd_in = a.take<float>(M);
  s->mean_out = a.take<float>(M);
  s->rstd_out = a.take<float>(M);
  return a.off;
}

static void carve_weights(Arena& a, const TriMulDesc* d, WeightsF32* w) {
  const size_t C = d->C, Ch = d->Ch;
  w->norm_in_w = a.take<float>(C); w->norm_in_b = a.take<float>(C);
  w->p_in_w = a.take<float>(2 * Ch * C); w->p_in_b = a.take<float>(2 * Ch);
  w->g_in_w = a.take<float>(2 * Ch * C); w->g_in_b = a.take<float>(2 * Ch);
  w->norm_out_w = a.take<float>(Ch); w->norm_out_b = a.take<float>(Ch);
  w->p_out_w = a.take<float>(C * Ch); w->p_out_b = a.take<float>(C);
  w->g_out_w = a.take<float>(C * C); w->g_out_b = a.take<float>(C);
  w->mask = a.take<float>((size_t)d->B * d->N * d->N);
}

constexpr int kWgradSplit = 128;

size_t saved_bytes(const TriMulDesc* d) {
  Arena a(nullptr, 0);
  Saved s;
  return carve_saved(a, d, &s);
}

size_t ws_bytes(const TriMulDesc* d, int is_bwd) {
  Arena a(nullptr, 0);
  WeightsF32 w;
  carve_weights(a, d, &w);
  Saved s;
  carve_saved(a, d, &s);  // forward without a saved block keeps its intermediates here
  if (is_bwd) {
    const size_t M = (size_t)d->B * d->N * d->N, C = d->C, Ch = d->Ch;
    a.take<float>(M * Ch);      // u
    a.take<float>(M * C);       // dy
    a.take<float>(M * C);       // dgo
    a.take<float>(M * Ch);      // du
    a.take<float>(M * Ch);      // dt
    a.take<float>(M * 2 * Ch);  // dab
    a.take<float>(M * 2 * Ch);  // dP
    a.take<float>(M * 2 * Ch);  // dG
    a.take<float>(M * C);       // dz
    size_t wmax = std::max((size_t)2 * Ch * C, std::max(C * Ch, C * C));
    a.take<float>(std::max((size_t)kWgradSplit * wmax, (size_t)2 * kLnBwdBlocks * std::max(C, Ch)));
  }
  return a.off + 256;
}

template <typename T>
static int convert_weights(cudaStream_t st, const TriMulDesc* d, const TriMulWeights* w, const void* mask, WeightsF32* f) {
  struct Item { const void* src; float** dst; size_t n; };
  const size_t C = d->C, Ch = d->Ch;
  Item items[] = {
      {w->norm_in_w, &f->norm_in_w, C},       {w->norm_in_b, &f->norm_in_b, C},
      {w->p_in_w, &f->p_in_w, 2 * Ch * C},    {w->p_in_b, &f->p_in_b, 2 * Ch},
      {w->g_in_w, &f->g_in_w, 2 * Ch * C},    {w->g_in_b, &f->g_in_b, 2 * Ch},
      {w->norm_out_w, &f->norm_out_w, Ch},    {w->norm_out_b, &f->norm_out_b, Ch},
      {w->p_out_w, &f->p_out_w, C * Ch},      {w->p_out_b, &f->p_out_b, C},
      {w->g_out_w, &f->g_out_w, C * C},       {w->g_out_b, &f->g_out_b, C},
      {mask, &f->mask, (size_t)d->B * d->N * d->N},
  };
  for (auto& it : items) {
    if (it.src == nullptr) { *it.dst = nullptr; continue; }
    convert_kernel<T><<<EW_GRID((long long)it.n)>>>((const T*)it.src, *it.dst, (long long)it.n);
    TRI_LAUNCH_OK();
  }
  return 0;
}

static GemmP linear_p(const float* in, int ld_in, const float* W, const float* bias, float* out, int ld_out,
                      long long rows, int n_out, int n_in) {
  GemmP p{};
  p.A = in; p.a_m = ld_in; p.a_k = 1;
  p.B = W; p.b_n = n_in; p.b_k = 1;
  p.C = out; p.c_m = ld_out; p.c_n = 1;
  p.bias = bias;
  p.M = (int)rows; p.N = n_out; p.K = n_in; p.ksplit = 1;
  return p;
}

// out[rows, n_in] (+)= D[rows, n_out] * W[n_out, n_in]
static GemmP linear_t_p(const float* D, int ldd, const float* W, float* out, long long rows, int n_out, int n_in, int accumulate) {
  GemmP p{};
  p.A = D; p.a_m = ldd; p.a_k = 1;
  p.B = W; p.b_n = 1; p.b_k = n_in;
  p.C = out; p.c_m = n_in; p.c_n = 1;
  p.M = (int)rows; p.N = n_in; p.K = n_out; p.ksplit = 1; p.accumulate = accumulate;
  return p;
}

// ============================================================================
// forward in three kernels: LayerNorm + input projections + gate, contraction, LayerNorms + output projections + gate
// ============================================================================
// A CTA of 256 threads has 64 output channels of two products, whose weights stay in shared memory, and walks over tiles of
// 64 pixels, which it normalises in shared memory: z, the projections and the LayerNormed contraction are written only where
// the backward needs them.  Both operands lie k-major, so that a thread's 8 pixels x 4 + 4 channels take four 16-byte
// shared loads per 64 FMAs (output stage, whose products have their own left operands: three per 32); the two halves of the
// CTA have half of each contraction and exchange half of their sums.  Two CTAs share an SM; one's loads and LayerNorm run
// under the other's products.  The FMAs are packed in pairs: 1.2 clocks per 32 of them against 1.4 for single ones.
//   One stage per kernel -- 9 conversions, 2 LayerNorms, 4 GEMMs of 16 us and two gates -- took 116 us of the 183 us of a
// 64 x 64 x 128 fp32 call; these take 21 and 13 us of 45 (and 0.59 and 0.37 ms at 384 x 384, against 2.1 ms).  The output stage took 19
// of 53 in tiles of 64 pixels, which make 128 CTAs there, launched behind the contraction.  Of the 21 the products are 11 (75 % of
// the FMA rate, 22 k cycles on an SM with two CTAs); weights, LayerNorm and the gate take 1.5 to 2 each.
struct FusedP {
  const void *x, *mask, *norm_in_w, *norm_in_b, *p_w, *p_b, *g_w, *g_b, *norm_out_w, *norm_out_b;
  const float* t;                                   // output stage: the contraction
  float *z, *mean, *rstd, *P, *G, *ab;              // input stage; z, mean, rstd, P, G null unless saved
  void* out;                                        // output stage (y, go: its two products, null unless saved)
  long long M;
  int C, Ch, n_out;                                 // n_out: 2 Ch, or C
  float eps;
};

template <typename T> constexpr bool kCanTf32 = sizeof(T) == 4;
constexpr int kFusedMax = 256;                      // channels of a row: two float4 per lane


template <typename T>
__device__ __forceinline__ float4 load_four(const T* p) {
  if constexpr (sizeof(T) == 4) {
    return *reinterpret_cast<const float4*>(p);
  } else {
    union { uint2 u; T h[4]; } v;
    v.u = *reinterpret_cast<const uint2*>(p);
    return make_float4(to_f32(v.h[0]), to_f32(v.h[1]), to_f32(v.h[2]), to_f32(v.h[3]));
  }
}
template <bool TF32>
__device__ __forceinline__ float4 round_four(float4 v) {
  if constexpr (TF32) return make_float4(round_tf32(v.x), round_tf32(v.y), round_tf32(v.z), round_tf32(v.w));
  return v;
}

// Four rows' values at four consecutive k, transposed into a tile [K][R] of 64 or 32 rows: the 16-byte chunk of four rows is XORed with
// k / 4, which keeps the lanes of a warp (consecutive k / 4) apart.
template <int R>
__device__ __forceinline__ void put_transposed(float* tile, int k, int row0, const float4& v0, const float4& v1, const float4& v2, const float4& v3) {
  float* to = tile + k * R + (((row0 >> 2) ^ (k >> 2 & 7)) << 2);
  *reinterpret_cast<float4*>(to) = make_float4(v0.x, v1.x, v2.x, v3.x);
  *reinterpret_cast<float4*>(to + R) = make_float4(v0.y, v1.y, v2.y, v3.y);
  *reinterpret_cast<float4*>(to + 2 * R) = make_float4(v0.z, v1.z, v2.z, v3.z);
  *reinterpret_cast<float4*>(to + 3 * R) = make_float4(v0.w, v1.w, v2.w, v3.w);
}

// 64 rows of W [n_out, K] and of G [n_out, C] from row n0 into shared memory as [K][64] and [C][64], zero beyond n_out; a warp has eight
// rows of each, four of both at a time
template <typename T, bool TF32>
__device__ __forceinline__ void stage_weights(float* dst_w, float* dst_g, const T* W, const T* G, int n0, int n_out, int K, int C) {
  const int lane = threadIdx.x & 31;
  for (int k = lane * 4; k < max(K, C); k += 128) {
#pragma unroll 1
    for (int r0 = (threadIdx.x >> 5) * 8, end = r0 + 8; r0 < end; r0 += 4) {
      float4 v[2][4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool in = n0 + r0 + r < n_out;
        v[0][r] = in && k < K ? load_four(W + (long long)(n0 + r0 + r) * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[1][r] = in && k < C ? load_four(G + (long long)(n0 + r0 + r) * C + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) { v[0][r] = round_four<TF32>(v[0][r]); v[1][r] = round_four<TF32>(v[1][r]); }
      if (k < K) put_transposed<64>(dst_w, k, r0, v[0][0], v[0][1], v[0][2], v[0][3]);
      if (k < C) put_transposed<64>(dst_g, k, r0, v[1][0], v[1][1], v[1][2], v[1][3]);
    }
  }
}

// N rows of up to 128 J channels, a lane with four channels of every 128; and their LayerNorm's weight and bias
template <int N, int J> struct Rows { float4 v[N][J]; };
template <int J> struct Affine {
  float4 g[J], b[J];
  template <typename T> __device__ __forceinline__ void load(const T* gamma, const T* beta, int K) {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = ((threadIdx.x & 31) + 32 * j) * 4;
      g[j] = gamma && k < K ? load_four(gamma + k) : make_float4(1.f, 1.f, 1.f, 1.f);
      b[j] = beta && k < K ? load_four(beta + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
};
// rows of X [M, K] from row m
template <int N, int J, typename TX>
__device__ __forceinline__ void load_rows(Rows<N, J>& x, const TX* X, long long m, long long M, int K) {
#pragma unroll
  for (int r = 0; r < N; ++r)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int k = ((threadIdx.x & 31) + 32 * j) * 4;
      x.v[r][j] = k < K && m + r < M ? load_four(X + (m + r) * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
// ... LayerNormed into rows r0 .. of a tile [K][R]; z, mean, rstd [M ..]: null, or written
template <int R, bool TF32, int N, int J>
__device__ __forceinline__ void put_normalised(Rows<N, J>& x, const Affine<J>& w, float* dst, int r0, float eps, long long m, long long M, int K, float* z,
                                               float* mean, float* rstd) {
  const int lane = threadIdx.x & 31;
  float s[N], mu[N];
#pragma unroll
  for (int r = 0; r < N; ++r) {
    s[r] = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j) s[r] += (x.v[r][j].x + x.v[r][j].y) + (x.v[r][j].z + x.v[r][j].w);
  }
#pragma unroll
  for (int r = 0; r < N; ++r) {
    mu[r] = warp_sum(s[r]) / K;
    s[r] = 0.f;
#pragma unroll
    for (int j = 0; j < J; ++j)
      if ((lane + 32 * j) * 4 < K) {
        float4& v = x.v[r][j];
        v = make_float4(v.x - mu[r], v.y - mu[r], v.z - mu[r], v.w - mu[r]);
        s[r] += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
      }
  }
#pragma unroll
  for (int r = 0; r < N; ++r) {
    s[r] = 1.0f / sqrtf(warp_sum(s[r]) / K + eps);
    if (mean != nullptr && m + r < M && lane == 0) { mean[m + r] = mu[r]; rstd[m + r] = s[r]; }
  }
#pragma unroll
  for (int j = 0; j < J; ++j) {
    const int k = (lane + 32 * j) * 4;
    if (k >= K) continue;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      float4& v = x.v[r][j];
      v = make_float4(v.x * s[r] * w.g[j].x + w.b[j].x, v.y * s[r] * w.g[j].y + w.b[j].y, v.z * s[r] * w.g[j].z + w.b[j].z, v.w * s[r] * w.g[j].w + w.b[j].w);
      if (z != nullptr && m + r < M) *reinterpret_cast<float4*>(z + (m + r) * K + k) = v;
      v = round_four<TF32>(v);
    }
#pragma unroll
    for (int r = 0; r < N; r += 4) put_transposed<R>(dst, k, r0 + r, x.v[r][j], x.v[r + 1][j], x.v[r + 2][j], x.v[r + 3][j]);
  }
}

// acc[w][i][j] += A^T B[w] over k_begin .. k_end, for pixels 2 i, 2 i + 1 of those in A's chunks of four from ch on (R = 64: two, 32: one)
// and channel j of chunk cn of each of W weight blocks
template <int W, int R>
__device__ __forceinline__ void dot_tile(float2 (&acc)[W][R / 16][4], const float* A, const float* B, int K, int k_begin, int k_end, int ch, int cn) {
#pragma unroll 1
  for (int k4 = k_begin; k4 < k_end; k4 += 4) {
    const int sw = k4 >> 2 & 7;
    const float* a0 = A + k4 * R + ((ch ^ sw) << 2);
    const float* a1 = A + k4 * R + (((ch + 1) ^ sw) << 2);
    const float* b0 = B + k4 * 64 + ((cn ^ sw) << 2);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 a[R / 16];
      const float4 x = *reinterpret_cast<const float4*>(a0 + e * R);
      a[0] = make_float2(x.x, x.y); a[1] = make_float2(x.z, x.w);
      if constexpr (R == 64) {
        const float4 y = *reinterpret_cast<const float4*>(a1 + e * R);
        a[2] = make_float2(y.x, y.y); a[3] = make_float2(y.z, y.w);
      }
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const float4 b = *reinterpret_cast<const float4*>(b0 + (w * K + e) * 64);
        const float2 bb[4] = {make_float2(b.x, b.x), make_float2(b.y, b.y), make_float2(b.z, b.z), make_float2(b.w, b.w)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < R / 16; ++i) acc[w][i][j] = __ffma2_rn(a[i], bb[j], acc[w][i][j]);
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void store_four(T* p, float4 v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    union { uint2 u; T h[4]; } o;
    o.h[0] = from_f32<T>(v.x); o.h[1] = from_f32<T>(v.y); o.h[2] = from_f32<T>(v.z); o.h[3] = from_f32<T>(v.w);
    *reinterpret_cast<uint2*>(p) = o.u;
  }
}

// where the second half of a contraction over K starts
__device__ __forceinline__ int split(int K) { return (K / 4 + 1) / 2 * 4; }

// OUT: the output stage (first product on the LayerNormed contraction), else the input stage (both on z).  R: pixels of a tile; rows of
// up to 128 J channels
template <typename T, bool OUT, bool TF32, int R, int J>
__global__ void __launch_bounds__(256, 2) fused_kernel(const FusedP p) {
  extern __shared__ __align__(16) float sm[];
  const int C = p.C, K0 = OUT ? p.Ch : p.C, n0 = blockIdx.x * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = warp >> 2, t = threadIdx.x & 127;
  const int ty = (warp >> 1 & 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);   // pixels R / 8 ty .., channels 4 tx ..
  constexpr int kChunks = R / 32, kPairs = R / 16;   // of the pixels of a thread
  constexpr int kRows = J == 1 ? R / 8 : 4;          // a warp's rows in registers at a time
  const bool first = blockIdx.x == 0;
  const T* px = static_cast<const T*>(p.x);
  float *sW = sm, *sG = sW + 64 * K0, *sA = sG + 64 * C, *sZ = OUT && R == 32 ? sA + R * K0 : sA;   // (32 pixels: both rows' tiles at once)
  const int n = n0 + 4 * tx, r0 = warp * (R / 8);
  float4 pb = make_float4(0.f, 0.f, 0.f, 0.f), gb = pb;
  stage_weights<T, TF32>(sW, sG, static_cast<const T*>(p.p_w), static_cast<const T*>(p.g_w), n0, p.n_out, K0, C);
  if (n < p.n_out && p.p_b) pb = load_four(static_cast<const T*>(p.p_b) + n);
  if (n < p.n_out && p.g_b) gb = load_four(static_cast<const T*>(p.g_b) + n);
  // LayerNormed rows of the tile from m0 on
  auto put_x = [&](long long m0, float* z, float* mean, float* rstd) {
#pragma unroll 1
    for (int i = 0; i < R / 8; i += kRows) {
      Rows<kRows, J> x;
      Affine<J> w;
      load_rows(x, px, m0 + r0 + i, p.M, C);
      w.load(static_cast<const T*>(p.norm_in_w), static_cast<const T*>(p.norm_in_b), C);
      put_normalised<R, TF32>(x, w, sZ, r0 + i, p.eps, m0 + r0 + i, p.M, C, z, mean, rstd);
    }
  };
  auto put_t = [&](long long m0) {
#pragma unroll 1
    for (int i = 0; i < R / 8; i += kRows) {
      Rows<kRows, J> x;
      Affine<J> w;
      load_rows(x, p.t, m0 + r0 + i, p.M, K0);
      w.load(static_cast<const T*>(p.norm_out_w), static_cast<const T*>(p.norm_out_b), K0);
      put_normalised<R, TF32>(x, w, sA, r0 + i, p.eps, m0 + r0 + i, p.M, K0, nullptr, first ? p.mean : nullptr, p.rstd);
    }
  };
  // t is the kernel's before, all else is the caller's
  if (OUT && R == 32) put_x(blockIdx.y * (long long)R, nullptr, nullptr, nullptr);
  if (OUT && R == 32) dependent_wait();
  for (long long m0 = blockIdx.y * (long long)R; m0 < p.M; m0 += gridDim.y * (long long)R) {
    float2 acc[2][kPairs][4];
    auto clear = [&](int w) {   // (late: the rows on their way need the registers)
#pragma unroll
      for (int x = 0; x < 4 * kPairs; ++x) acc[w][x >> 2][x & 3] = make_float2(0.f, 0.f);
    };
    const bool again = m0 != blockIdx.y * (long long)R;
    if (again) __syncthreads();
    if constexpr (OUT) {
      if (R == 32 && again) put_x(m0, nullptr, nullptr, nullptr);
      put_t(m0);
      __syncthreads();
      clear(0);
      dot_tile<1, R>(reinterpret_cast<float2(&)[1][kPairs][4]>(acc[0]), sA, sW, K0, half ? split(K0) : 0, half ? K0 : split(K0), kChunks * ty, tx);
      if (R == 64) {
        __syncthreads();
        put_x(m0, nullptr, nullptr, nullptr);
        __syncthreads();
      }
      clear(1);
      dot_tile<1, R>(reinterpret_cast<float2(&)[1][kPairs][4]>(acc[1]), sZ, sG, C, half ? split(C) : 0, half ? C : split(C), kChunks * ty, tx);
    } else {
      put_x(m0, first ? p.z : nullptr, first ? p.mean : nullptr, p.rstd);
      __syncthreads();
      clear(0);
      clear(1);
      dot_tile<2, R>(acc, sA, sW, C, half ? split(C) : 0, half ? C : split(C), kChunks * ty, tx);
    }
    // each half keeps half of the pixels: it hands the others' sums over through the row tile
    __syncthreads();
    float2* swap = reinterpret_cast<float2*>(sA);
    constexpr int kHand = 4 * kPairs;   // pairs of both products that change hands
    auto sum = [&](int x, bool upper) -> float2& { return acc[x / (kHand / 2)][(upper ? kPairs / 2 : 0) + x / 4 % (kPairs / 2)][x % 4]; };
#pragma unroll
    for (int x = 0; x < kHand; ++x) swap[(half * kHand + x) * 128 + t] = half ? sum(x, false) : sum(x, true);
    __syncthreads();
#pragma unroll
    for (int x = 0; x < kHand; ++x) {
      const float2 o = swap[((half ^ 1) * kHand + x) * 128 + t], own = half ? sum(x, true) : sum(x, false);
      sum(x, false) = half ? __fadd2_rn(o, own) : __fadd2_rn(own, o);
    }
    if (n >= p.n_out) continue;
#pragma unroll
    for (int i = 0; i < R / 16; ++i) {
      const long long m = m0 + R / 8 * ty + R / 16 * half + i, at = m * p.n_out + n;
      if (m >= p.M) continue;
      float a[4], b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a[j] = i & 1 ? acc[0][i >> 1][j].y : acc[0][i >> 1][j].x;
        b[j] = i & 1 ? acc[1][i >> 1][j].y : acc[1][i >> 1][j].x;
      }
      const float4 v = make_float4(a[0] + pb.x, a[1] + pb.y, a[2] + pb.z, a[3] + pb.w), g = make_float4(b[0] + gb.x, b[1] + gb.y, b[2] + gb.z, b[3] + gb.w);
      if (p.P != nullptr) { store_four(p.P + at, v); store_four(p.G + at, g); }
      const float keep = !OUT && p.mask ? to_f32(static_cast<const T*>(p.mask)[m]) : 1.f;
      const float4 r = make_float4(v.x * sigmoidf_acc(g.x) * keep, v.y * sigmoidf_acc(g.y) * keep, v.z * sigmoidf_acc(g.z) * keep, v.w * sigmoidf_acc(g.w) * keep);
      if constexpr (OUT) store_four(static_cast<T*>(p.out) + at, r);
      else store_four(p.ab + at, r);
    }
  }
}

// Rows of up to 256 channels in whole 16-byte pieces; wider or odd ones go through one stage per kernel.
template <typename T>
static bool fused_fits(const TriMulDesc* d, const void* x, const TriMulWeights* w, void* out) {
  const size_t v = 4 * sizeof(T);
  for (const void* p : {x, static_cast<const void*>(out), w->p_in_b, w->g_in_b, w->p_out_b, w->g_out_b, w->norm_in_w, w->norm_in_b, w->p_in_w, w->g_in_w, w->norm_out_w, w->norm_out_b, w->p_out_w, w->g_out_w})
    if (reinterpret_cast<uintptr_t>(p) % v != 0) return false;
  return d->C % 4 == 0 && d->Ch % 4 == 0 && d->C <= kFusedMax && d->Ch <= kFusedMax;
}

template <typename T, bool OUT, int R, int J>
static int fused_launch(const FusedP& p, bool tf32, cudaStream_t st) {
  const auto kern = tf32 ? fused_kernel<T, OUT, kCanTf32<T>, R, J> : fused_kernel<T, OUT, false, R, J>;
  // the row tile (of 32 pixels: tiles), at least as large as the halves' exchange
  const int rows = OUT && R == 32 ? std::max(128, p.C + p.Ch) : std::max(128, OUT ? std::max(p.C, p.Ch) : p.C);
  const size_t smem = sizeof(float) * (64 * (size_t)(OUT ? p.C + p.Ch : 2 * p.C) + (size_t)R * rows);
  TRI_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const double M = (double)p.M, fma = M * p.n_out * (p.C + (OUT ? p.Ch : p.C));
  KernelTimer kt(OUT ? "simt_fused_out" : "simt_fused_in", st, 2.0 * fma, OUT ? M * (2.0 * p.C * sizeof(T) + 4.0 * p.Ch) : M * (p.C * sizeof(T) + 8.0 * p.Ch));
  const int blocks = cdiv(p.n_out, 64), room = std::max(1, (smem <= 113 * 1024 ? 2 : 1) * sm_count() / blocks);
  // The output stage of a small call starts early: weights and x are staged under the contraction, which leaves the room (64 x 64 pixels:
  // 13 us behind it instead of 21).  With larger ones, early CTAs take their places unevenly (203 x 203: 404 -> 407 us).
  launch_dependent(OUT && R == 32 ? 0.0 : kLaunchPlainly, kern, dim3(blocks, (unsigned)std::min<long long>((p.M + R - 1) / R, room)), 256, smem, st, p);
  TRI_LAUNCH_OK();
  return 0;
}
template <typename T, bool OUT>
static int fused_start(const FusedP& p, bool tf32, cudaStream_t st) {
  const bool narrow = p.C <= 128 && p.Ch <= 128;
  // output stage: tiles of 32 pixels where those of 64 would not make two CTAs for an SM
  if (OUT && (p.M + 63) / 64 * cdiv(p.n_out, 64) <= sm_count()) {
    constexpr int R = OUT ? 32 : 64;
    return narrow ? fused_launch<T, OUT, R, 1>(p, tf32, st) : fused_launch<T, OUT, R, 2>(p, tf32, st);
  }
  return narrow ? fused_launch<T, OUT, 64, 1>(p, tf32, st) : fused_launch<T, OUT, 64, 2>(p, tf32, st);
}

template <typename T>
static int forward_t(const TriMulDesc* d, const void* x, const void* mask, const TriMulWeights* w, void* out,
                     void* saved, void* ws, size_t ws_size, cudaStream_t st) {
  const long long M = (long long)d->B * d->N * d->N;
  const int C = d->C, Ch = d->Ch, N = d->N;
  const bool tf32 = d->dtype == TRI_F32 && d->precision == TRI_PREC_TF32;
  Arena a(ws, ws_size);
  WeightsF32 f;
  carve_weights(a, d, &f);
  Saved s;
  if (saved) { Arena sa(saved, saved_bytes(d)); carve_saved(sa, d, &s); }
  else carve_saved(a, d, &s);
  if (!a.ok()) return fail(TRI_ERR_WORKSPACE, "trimul forward workspace too small: need %zu, got %zu", a.off, ws_size);
  const bool fused = fused_fits<T>(d, x, w, out);
  FusedP fp{};
  if (fused) {
    fp.x = x; fp.mask = mask; fp.norm_in_w = w->norm_in_w; fp.norm_in_b = w->norm_in_b; fp.norm_out_w = w->norm_out_w; fp.norm_out_b = w->norm_out_b;
    fp.p_w = w->p_in_w; fp.p_b = w->p_in_b; fp.g_w = w->g_in_w; fp.g_b = w->g_in_b;
    fp.M = M; fp.C = C; fp.Ch = Ch; fp.n_out = 2 * Ch; fp.eps = d->eps; fp.ab = s.ab;
    if (saved) { fp.z = s.z; fp.mean = s.mean_in; fp.rstd = s.rstd_in; fp.P = s.P; fp.G = s.G; }
    TRI_TRY((fused_start<T, false>(fp, tf32, st)));
  } else {
    TRI_TRY(convert_weights<T>(st, d, w, mask, &f));

    {
      KernelTimer kt("simt_ln_fwd", st, 0.0, (double)M * C * (sizeof(T) + 4.0));
      ln_fwd_kernel<T><<<cdiv(M, 8), 256, 0, st>>>((const T*)x, f.norm_in_w, f.norm_in_b, d->eps, M, C, s.z, s.mean_in, s.rstd_in);
      TRI_LAUNCH_OK();
    }
    TRI_TRY(gemm(st, tf32, linear_p(s.z, C, f.p_in_w, f.p_in_b, s.P, 2 * Ch, M, 2 * Ch, C)));
    TRI_TRY(gemm(st, tf32, linear_p(s.z, C, f.g_in_w, f.g_in_b, s.G, 2 * Ch, M, 2 * Ch, C)));
    {
      KernelTimer kt("simt_gate_in", st, 0.0, 24.0 * M * Ch);
      gate_in_kernel<<<EW_GRID(M * 2 * Ch)>>>(s.P, s.G, f.mask, M, 2 * Ch, s.ab);
      TRI_LAUNCH_OK();
    }
  }
  ContractP cp{};
  cp.X = s.ab; cp.Y = s.ab; cp.O = s.t; cp.N = N; cp.Ch = Ch;
  cp.ldx = cp.ldy = 2 * Ch; cp.ldo = Ch; cp.xoff = 0; cp.yoff = Ch; cp.ooff = 0;
  cp.os_p = N; cp.os_q = 1;
  if (d->direction == TRI_OUTGOING) { cp.xs_p = N; cp.xs_r = 1; cp.ys_q = N; cp.ys_r = 1; }
  else { cp.xs_p = 1; cp.xs_r = N; cp.ys_q = 1; cp.ys_r = N; }
  TRI_TRY(contract(st, tf32, d->B, cp));
  if (fused) {
    fp.p_w = w->p_out_w; fp.p_b = w->p_out_b; fp.g_w = w->g_out_w; fp.g_b = w->g_out_b; fp.n_out = C; fp.t = s.t; fp.out = out;
    if (saved) { fp.mean = s.mean_out; fp.rstd = s.rstd_out; fp.P = s.y; fp.G = s.go; }
    fp.ab = nullptr; fp.z = nullptr;
    return fused_start<T, true>(fp, tf32, st);
  }
  // LayerNormed contraction output: P is dead by now in inference, so it doubles as scratch there;
  // with a saved block P must survive, and the workspace region that would have held it is free.
  float* u_buf = saved ? a.take<float>((size_t)M * Ch) : s.P;
  if (!a.ok()) return fail(TRI_ERR_WORKSPACE, "trimul forward workspace too small: need %zu, got %zu", a.off, ws_size);
  {
    KernelTimer kt("simt_ln_fwd", st, 0.0, 8.0 * M * Ch);
    ln_fwd_kernel<float><<<cdiv(M, 8), 256, 0, st>>>(s.t, f.norm_out_w, f.norm_out_b, d->eps, M, Ch, u_buf, s.mean_out, s.rstd_out);
    TRI_LAUNCH_OK();
  }
  TRI_TRY(gemm(st, tf32, linear_p(u_buf, Ch, f.p_out_w, f.p_out_b, s.y, C, M, C, Ch)));
  TRI_TRY(gemm(st, tf32, linear_p(s.z, C, f.g_out_w, f.g_out_b, s.go, C, M, C, C)));
  {
    KernelTimer kt("simt_gate_out", st, 0.0, (double)M * C * (8.0 + sizeof(T)));
    gate_out_kernel<T><<<EW_GRID(M * C)>>>(s.y, s.go, M * C, (T*)out);
    TRI_LAUNCH_OK();
  }
  return 0;
}

template <typename T>
static int backward_t(const TriMulDesc* d, const void* x, const void* mask, const TriMulWeights* w,
                      const void* saved, const void* d_out, void* dx, const TriMulWeightGrads* g, void* ws,
                      size_t ws_size, cudaStream_t st) {
  const long long M = (long long)d->B * d->N * d->N;
  const int C = d->C, Ch = d->Ch, N = d->N;
  const bool tf32 = d->dtype == TRI_F32 && d->precision == TRI_PREC_TF32;
  Arena a(ws, ws_size);
  WeightsF32 f;
  carve_weights(a, d, &f);
  Saved s;
  { Arena sa(const_cast<void*>(saved), saved_bytes(d)); carve_saved(sa, d, &s); }
  float* u = a.take<float>((size_t)M * Ch);
  float* dy = a.take<float>((size_t)M * C);
  float* dgo = a.take<float>((size_t)M * C);
  float* du = a.take<float>((size_t)M * Ch);
  float* dt = a.take<float>((size_t)M * Ch);
  float* dab = a.take<float>((size_t)M * 2 * Ch);
  float* dP = a.take<float>((size_t)M * 2 * Ch);
  float* dG = a.take<float>((size_t)M * 2 * Ch);
  float* dz = a.take<float>((size_t)M * C);
  size_t wmax = std::max((size_t)2 * Ch * C, std::max((size_t)C * Ch, (size_t)C * C));
  float* partial = a.take<float>(std::max((size_t)kWgradSplit * wmax, (size_t)2 * kLnBwdBlocks * std::max(C, Ch)));
  if (!a.ok()) return fail(TRI_ERR_WORKSPACE, "trimul backward workspace too small: need %zu, got %zu", a.off, ws_size);
  TRI_TRY(convert_weights<T>(st, d, w, mask, &f));

  // output gate and projection
  {
    KernelTimer kt("simt_gate_out_bwd", st, 0.0, (double)M * C * (16.0 + sizeof(T)));
    gate_out_bwd_kernel<T><<<EW_GRID(M * C)>>>((const T*)d_out, s.y, s.go, M * C, dy, dgo);
    TRI_LAUNCH_OK();
  }
  {
    KernelTimer kt("simt_ln_fwd", st, 0.0, 8.0 * M * Ch);
    ln_fwd_kernel<float><<<cdiv(M, 8), 256, 0, st>>>(s.t, f.norm_out_w, f.norm_out_b, d->eps, M, Ch, u, s.mean_out, s.rstd_out);
    TRI_LAUNCH_OK();
  }
  if (g->p_out_w) TRI_TRY(weight_grad(st, tf32, dy, C, C, u, Ch, Ch, M, partial, kWgradSplit, g->p_out_w));
  if (g->p_out_b) TRI_TRY(colsum(st, dy, M, C, partial, g->p_out_b));
  if (g->g_out_w) TRI_TRY(weight_grad(st, tf32, dgo, C, C, s.z, C, C, M, partial, kWgradSplit, g->g_out_w));
  if (g->g_out_b) TRI_TRY(colsum(st, dgo, M, C, partial, g->g_out_b));
  TRI_TRY(gemm(st, tf32, linear_t_p(dy, C, f.p_out_w, du, M, C, Ch, 0)));
  TRI_TRY((ln_bwd<float, float>(st, du, s.t, s.mean_out, s.rstd_out, f.norm_out_w, M, Ch, dt, partial, g->norm_out_w, g->norm_out_b)));

  // contraction backward: da -> dab[:, :Ch], db -> dab[:, Ch:]
  ContractP ca{}, cb{};
  ca.N = cb.N = N; ca.Ch = cb.Ch = Ch;
  ca.O = cb.O = dab; ca.ldo = cb.ldo = 2 * Ch; ca.ooff = 0; cb.ooff = Ch;
  ca.X = dt; ca.ldx = Ch; ca.xoff = 0; ca.Y = s.ab; ca.ldy = 2 * Ch; ca.yoff = Ch;   // dt with b
  if (d->direction == TRI_OUTGOING) {
    // da[i,k] = sum_j dt[i,j] b[j,k]        (p=i, q=k, r=j)
    ca.xs_p = N; ca.xs_r = 1; ca.ys_q = 1; ca.ys_r = N; ca.os_p = N; ca.os_q = 1;
    // db[j,k] = sum_i dt[i,j] a[i,k]        (p=j, q=k, r=i)
    cb.X = dt; cb.ldx = Ch; cb.xoff = 0; cb.Y = s.ab; cb.ldy = 2 * Ch; cb.yoff = 0;
    cb.xs_p = 1; cb.xs_r = N; cb.ys_q = 1; cb.ys_r = N; cb.os_p = N; cb.os_q = 1;
  } else {
    // da[k,i] = sum_j dt[i,j] b[k,j]        (p=i, q=k, r=j), stored at pixel (k,i)
    ca.xs_p = N; ca.xs_r = 1; ca.ys_q = N; ca.ys_r = 1; ca.os_p = 1; ca.os_q = N;
    // db[k,j] = sum_i a[k,i] dt[i,j]        (p=k, q=j, r=i)
    cb.X = s.ab; cb.ldx = 2 * Ch; cb.xoff = 0; cb.Y = dt; cb.ldy = Ch; cb.yoff = 0;
    cb.xs_p = N; cb.xs_r = 1; cb.ys_q = 1; cb.ys_r = N; cb.os_p = N; cb.os_q = 1;
  }
  TRI_TRY(contract(st, tf32, d->B, ca));
  TRI_TRY(contract(st, tf32, d->B, cb));

  // input gate and projections
  {
    KernelTimer kt("simt_gate_in_bwd", st, 0.0, 40.0 * M * Ch);
    gate_in_bwd_kernel<<<EW_GRID(M * 2 * Ch)>>>(dab, s.P, s.G, f.mask, M, 2 * Ch, dP, dG);
    TRI_LAUNCH_OK();
  }
  if (g->p_in_w) TRI_TRY(weight_grad(st, tf32, dP, 2 * Ch, 2 * Ch, s.z, C, C, M, partial, kWgradSplit, g->p_in_w));
  if (g->p_in_b) TRI_TRY(colsum(st, dP, M, 2 * Ch, partial, g->p_in_b));
  if (g->g_in_w) TRI_TRY(weight_grad(st, tf32, dG, 2 * Ch, 2 * Ch, s.z, C, C, M, partial, kWgradSplit, g->g_in_w));
  if (g->g_in_b) TRI_TRY(colsum(st, dG, M, 2 * Ch, partial, g->g_in_b));
  TRI_TRY(gemm(st, tf32, linear_t_p(dP, 2 * Ch, f.p_in_w, dz, M, 2 * Ch, C, 0)));
  TRI_TRY(gemm(st, tf32, linear_t_p(dG, 2 * Ch, f.g_in_w, dz, M, 2 * Ch, C, 1)));
  TRI_TRY(gemm(st, tf32, linear_t_p(dgo, C, f.g_out_w, dz, M, C, C, 1)));
  TRI_TRY((ln_bwd<T, T>(st, dz, (const T*)x, s.mean_in, s.rstd_in, f.norm_in_w, M, C, (T*)dx, partial, g->norm_in_w, g->norm_in_b)));
  return 0;
}

int forward(const TriMulDesc* d, const void* x, const void* mask, const TriMulWeights* w, void* out,
            void* saved, void* ws, size_t ws_size, cudaStream_t st) {
  switch (d->dtype) {
    case TRI_F32: return forward_t<float>(d, x, mask, w, out, saved, ws, ws_size, st);
    case TRI_BF16: return forward_t<__nv_bfloat16>(d, x, mask, w, out, saved, ws, ws_size, st);
    case TRI_F16: return forward_t<__half>(d, x, mask, w, out, saved, ws, ws_size, st);
  }
  return fail(TRI_ERR_ARG, "bad dtype %d", d->dtype);
}

int backward(const TriMulDesc* d, const void* x, const void* mask, const TriMulWeights* w, const void* saved,
             const void* d_out, void* dx, const TriMulWeightGrads* g, void* ws, size_t ws_size, cudaStream_t st) {
  switch (d->dtype) {
    case TRI_F32: return backward_t<float>(d, x, mask, w, saved, d_out, dx, g, ws, ws_size, st);
    case TRI_BF16: return backward_t<__nv_bfloat16>(d, x, mask, w, saved, d_out, dx, g, ws, ws_size, st);
    case TRI_F16: return backward_t<__half>(d, x, mask, w, saved, d_out, dx, g, ws, ws_size, st);
  }
  return fail(TRI_ERR_ARG, "bad dtype %d", d->dtype);
}

}  // namespace simt
}  // namespace tri

// Shared helpers for every translation unit of libtri_b200.so.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "../../include/tri_b200.h"

namespace tri {

// ---- thread-local status ---------------------------------------------------
char* last_error_buf();            // 512 bytes, thread local
void set_path(const char* name);   // "simt" / "tcgen05"
void count_launch(int n = 1);

// Optional per-kernel timing: when enabled (tri_profile_enable), every launch site is bracketed by a
// pair of CUDA events on the launching stream; tri_profile_summary sums them per kernel name.
// `flops` and `bytes` are the ALGORITHMIC work of the launch (not measured traffic).
struct KernelTimer {
  int slot;
  cudaStream_t st;
  KernelTimer(const char* name, cudaStream_t stream, double flops = 0.0, double bytes = 0.0);
  ~KernelTimer();
};

inline int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(last_error_buf(), 512, fmt, ap);
  va_end(ap);
  return code;
}

#define TRI_CUDA_OK(expr)                                                          \
  do {                                                                             \
    cudaError_t e_ = (expr);                                                       \
    if (e_ != cudaSuccess)                                                         \
      return ::tri::fail((int)e_, "%s failed: %s (%s:%d)", #expr,                  \
                         cudaGetErrorString(e_), __FILE__, __LINE__);              \
  } while (0)

#define TRI_LAUNCH_OK()                                                            \
  do {                                                                             \
    ::tri::count_launch();                                                         \
    cudaError_t e_ = cudaGetLastError();                                           \
    if (e_ != cudaSuccess)                                                         \
      return ::tri::fail((int)e_, "kernel launch failed: %s (%s:%d)",              \
                         cudaGetErrorString(e_), __FILE__, __LINE__);              \
  } while (0)

#define TRI_TRY(expr)                                                              \
  do {                                                                             \
    int r_ = (expr);                                                               \
    if (r_ != 0) return r_;                                                        \
  } while (0)

// ---- programmatic dependent launch ---------------------------------------------
// A kernel that `launch_dependent` starts is resident, with its barriers and TMEM set up, before its predecessor has drained.
// It calls `dependent_enter` before it touches what an earlier kernel of the chain writes or reads: the next kernel may come,
// and this one waits until all kernels before it are complete and their results visible.  (Each of them has waited in the same
// way before it ends, so nothing older is in flight either.)
// The first kernel of a call is launched plainly: once it runs, all work before the call is complete, and the later ones may
// read the caller's tensors, which no kernel of the chain writes, without waiting.  (tri_gated_linear_after continues the chain of
// the call before it, and says so.)
// Only the tensor-core kernels are started so.  They fill an SM by their shared memory, whereas CTAs of a small kernel that come
// while others run are packed onto the SMs that have room and keep the little L1 that is left there (with every kernel started
// so: fp32 update at 64 x 64 pixels 53.3 -> 55.3 us, bf16 update with gradients at 768 1806 -> 1835).  As it is, us before and
// after: attention at 64, 256 residues 14.1 -> 13.6, 45.2 -> 42.8, with gradients at 301 469 -> 460; update at 203 61.4 -> 55.1,
// with gradients at 384 497 -> 483.
// And only the short ones: `us` is what the kernel takes at least, by its bytes or its exponentials.  The few us of a ramp do
// not show beside a long kernel, and with every kernel of the pair stack at 1024 residues (86 us and more each, at the power limit
// throughout) started early, its pass took 0.5 to 1 % longer: 23.24-23.34 -> 23.40-23.60 ms.  The kernels that gained take at
// least 1 to 40 us; between that and 70 neither start is measurably better: the update with gradients at 384, 768 and (TF32) 512, whose
// gate kernels lie above the line, takes 450.8, 1711 and 1436 us with it and 450.7, 1710 and 1436 with every kernel started early.
__device__ __forceinline__ void dependent_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependent_enter() {
  dependent_trigger();
  dependent_wait();
}

constexpr double kEarlyStartUs = 60.0, kLaunchPlainly = kEarlyStartUs;
inline double us_of_bytes(double bytes) { return bytes / 6.5e6; }        // the measured copy rate
inline double us_of_logits(double logits) { return logits / 4.6e6; }     // one exponential each, 16 per clock and SM

template <typename... K, typename... A>
inline void launch_dependent(double us, void (*kern)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st; cfg.attrs = &attr; cfg.numAttrs = us < kEarlyStartUs ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, K(args)...);   // (errors: TRI_LAUNCH_OK)
}

// ---- element types -----------------------------------------------------------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

// Round an fp32 value to the tf32 grid (10 explicit mantissa bits, round to nearest).
__device__ __forceinline__ float round_tf32(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

__device__ __forceinline__ float sigmoidf_acc(float v) { return 1.0f / (1.0f + expf(-v)); }

// Multiprocessors of the CURRENT device.  Cached per device: one process may drive several GPUs (one thread each,
// or autograd's backward thread), so neither this nor any launch attribute may be remembered process-wide.
int sm_count();

inline size_t dtype_size(int dtype) { return dtype == TRI_F32 ? 4 : 2; }
inline size_t align_up(size_t v, size_t a = 256) { return (v + a - 1) / a * a; }
inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

// Bump allocator over a caller-provided workspace.
struct Arena {
  char* base;
  size_t cap, off;
  Arena(void* p, size_t bytes) : base((char*)p), cap(bytes), off(0) {}
  template <typename T> T* take(size_t n) {
    size_t bytes = align_up(n * sizeof(T));
    T* r = (T*)(base + off);
    off += bytes;
    return r;
  }
  bool ok() const { return off <= cap; }
};

}  // namespace tri

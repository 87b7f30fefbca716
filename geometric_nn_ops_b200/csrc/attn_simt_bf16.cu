// Triangle attention on bf16: the kernels of attn_simt_kernels.cuh for this type.
#include "attn_simt_kernels.cuh"

namespace tri {
namespace simt {
int forward_bf16(const AttnArgs& a, cudaStream_t st) { return forward_any<__nv_bfloat16, false>(a, st); }
int backward_bf16(const AttnArgs& a, float* part, cudaStream_t st) { return backward_any<__nv_bfloat16, false>(a, part, st); }
}  // namespace simt
}  // namespace tri

// Triangle attention on fp16: the kernels of attn_simt_kernels.cuh for this type.
#include "attn_simt_kernels.cuh"

namespace tri {
namespace simt {
int forward_f16(const AttnArgs& a, cudaStream_t st) { return forward_any<__half, false>(a, st); }
int backward_f16(const AttnArgs& a, float* part, cudaStream_t st) { return backward_any<__half, false>(a, part, st); }
}  // namespace simt
}  // namespace tri

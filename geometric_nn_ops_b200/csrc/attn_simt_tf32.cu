// Triangle attention on fp32 with TF32 products: the kernels of attn_simt_kernels.cuh for this type.
#include "attn_simt_kernels.cuh"

namespace tri {
namespace simt {
int forward_tf32(const AttnArgs& a, cudaStream_t st) { return forward_any<float, true>(a, st); }
int backward_tf32(const AttnArgs& a, float* part, cudaStream_t st) { return backward_any<float, true>(a, part, st); }
}  // namespace simt
}  // namespace tri

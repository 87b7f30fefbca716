// Triangle attention on fp32, exact products: the kernels of attn_simt_kernels.cuh for this type.
#include "attn_simt_kernels.cuh"

namespace tri {
namespace simt {
int forward_f32(const AttnArgs& a, cudaStream_t st) { return forward_any<float, false>(a, st); }
int backward_f32(const AttnArgs& a, float* part, cudaStream_t st) { return backward_any<float, false>(a, part, st); }
}  // namespace simt
}  // namespace tri

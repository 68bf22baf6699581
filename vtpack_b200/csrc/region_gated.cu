// Gated decompress of the training path (region_ops.cuh).
#include "region_ops.cuh"

namespace vtp {
template int region_gated_t<float>(const GatedArgs& a, cudaStream_t st);
template int region_gated_t<bf16>(const GatedArgs& a, cudaStream_t st);
}  // namespace vtp

// Pool of bf16 tokens (region_ops.cuh).
#include "region_ops.cuh"

namespace vtp {
template int region_pool_t<bf16>(const RegionPoolArgs& a, cudaStream_t st);
}  // namespace vtp

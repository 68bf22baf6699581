// Pool of fp32 tokens (region_ops.cuh).
#include "region_ops.cuh"

namespace vtp {
template int region_pool_t<float>(const RegionPoolArgs& a, cudaStream_t st);
}  // namespace vtp

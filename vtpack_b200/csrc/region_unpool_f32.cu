// Unpool of fp32 tokens and the gate (region_ops.cuh).
#include "region_ops.cuh"

namespace vtp {
template int region_unpool_t<float>(const RegionUnpoolArgs& a, cudaStream_t st);
template int region_gate_t<float>(const RegionGateArgs& a, cudaStream_t st);
}  // namespace vtp

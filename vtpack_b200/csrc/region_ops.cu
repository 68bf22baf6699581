// The region movers by element type (kernels: region_ops.cuh).
#include "region_ops.cuh"

namespace vtp {

bool region_ops_supported(const RegionGeom& g, int dtype) {
    const int vn = dtype == VTP_BF16 ? 8 : 4;
    int G, CPL;
    if (g.region != RG || g.C % vn != 0 || g.B <= 0 || g.Hr <= 0 || g.Wr <= 0) return false;
    return pick_layout(g.C / vn, &G, &CPL);
}

extern template int region_pool_t<float>(const RegionPoolArgs&, cudaStream_t);
extern template int region_pool_t<bf16>(const RegionPoolArgs&, cudaStream_t);
extern template int region_unpool_t<float>(const RegionUnpoolArgs&, cudaStream_t);
extern template int region_unpool_t<bf16>(const RegionUnpoolArgs&, cudaStream_t);
extern template int region_gate_t<float>(const RegionGateArgs&, cudaStream_t);
extern template int region_gate_t<bf16>(const RegionGateArgs&, cudaStream_t);
extern template int region_gated_t<float>(const GatedArgs&, cudaStream_t);
extern template int region_gated_t<bf16>(const GatedArgs&, cudaStream_t);

int region_pool(const RegionPoolArgs& a, int dtype, cudaStream_t st) {
    return dtype == VTP_F32 ? region_pool_t<float>(a, st) : region_pool_t<bf16>(a, st);
}
int region_unpool(const RegionUnpoolArgs& a, int dtype, cudaStream_t st) {
    return dtype == VTP_F32 ? region_unpool_t<float>(a, st) : region_unpool_t<bf16>(a, st);
}
int region_gate(const RegionGateArgs& a, int dtype, cudaStream_t st) {
    return dtype == VTP_F32 ? region_gate_t<float>(a, st) : region_gate_t<bf16>(a, st);
}
int region_gated_unpool(const GatedArgs& a, int dtype, cudaStream_t st) {
    return dtype == VTP_F32 ? region_gated_t<float>(a, st) : region_gated_t<bf16>(a, st);
}

}  // namespace vtp

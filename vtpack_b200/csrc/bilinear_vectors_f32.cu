// The vector kernels of the bilinear attention for fp32 rows.
#include "bilinear_vectors.cuh"

namespace vtp {
template void bilinear_vectors<float>(const BvArgs& a, const BvShape& s, bool point, bool grad, cudaStream_t st);
}  // namespace vtp

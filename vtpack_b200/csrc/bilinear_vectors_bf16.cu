// The vector kernels of the bilinear attention for bf16 rows.
#include "bilinear_vectors.cuh"

namespace vtp {
template void bilinear_vectors<bf16>(const BvArgs& a, const BvShape& s, bool point, bool grad, cudaStream_t st);
}  // namespace vtp

// Single-precision instantiation of the cluster tridiagonalisation.
#include "hetrd_kernels.cuh"

namespace bippb200 {
template bool hetrd_cluster<float2, float>(cudaStream_t, int, size_t, size_t, float2*, const int*, int, double*, double*,
                                           float2*, const int*, int, int, int, int);
}  // namespace bippb200

// Double-precision instantiation of the cluster tridiagonalisation.
#include "hetrd_kernels.cuh"

namespace bippb200 {
template bool hetrd_cluster<double2, double>(cudaStream_t, int, size_t, size_t, double2*, const int*, int, double*,
                                             double*, double2*, const int*, int, int, int, int);
}  // namespace bippb200

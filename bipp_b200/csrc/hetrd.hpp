// Batched Householder tridiagonalisation on clusters of CTAs (hetrd_kernels.cuh).
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace bippb200 {

// Tridiagonalise nb matrices of at most nmax rows (leading dimension ld, sizes nred, taken in
// `order`): reflectors in place of A, d, e, tau with stride ld. most: largest cluster size
// (0: by size and batch); grid1: CTAs when the clusters are single CTAs (0: one per matrix). False, with nothing
// launched, when nmax is beyond the kernel or hetrd_blk_kernel is the faster one.
template <typename C, typename R>
bool hetrd_cluster(cudaStream_t st, int smCount, size_t l2Bytes, size_t maxSmem, C* A, const int* nred, int ld, double* d,
                   double* e, C* tau, const int* order, int nb, int nmax, int most, int grid1);

}  // namespace bippb200

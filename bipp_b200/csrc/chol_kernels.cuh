// Cholesky factor and triangular inverse of a batch of real symmetric FP64 matrices (the
// Gram matrices of W = I), tiled 64 x 64 over (tile, matrix) grids (sm_100a).
//
// The reference factors inside LAPACK's ?hegv (src/host/lapack_api.hpp:112-158). One CTA per
// matrix left a small batch on a few SMs and, in a large one, read its operands from shared
// memory at one load per two multiply-adds with 32 serial pivots between block barriers
// (Cholesky + inverse of 512 rows: 4.4 ms for one matrix, 30 ms for 2048). Here every
// launch covers all tiles of all matrices that are ready:
//   chol_diag      pivot block 0: factor and inverse in shared memory, one warp's registers
//                  holding the 32-row sub-block and its column broadcast by shuffles
//   chol_panel k   rows below: P = A X_k^T with X_k = L_kk^-1
//   chol_trail k   A -= P P^T; the CTA of the next pivot block goes on to factor it, so a
//                  panel costs two launches
//   trinv_level    the inverse by doubling: with the diagonal blocks of size B inverted,
//                  the block below the diagonal of each pair is -X22 (L21 X11), two launches
//                  per level and log2(n / 64) levels
// The products run on the FP64 tensor instruction (m8n8k4; 256 multiply-adds per issue, 6
// shared-memory loads per 8 of them). In a batch of 128 matrices of 380-512 rows that pipe is
// 60-65 % busy in the inverse, 29 % in the trailing update, whose tile loads precede each
// product without overlap and one of whose CTAs goes on through a chain of pivots.
// All arithmetic and accumulation is FP64 as before.
#pragma once

#include "common.cuh"
#include "eig_kernels.cuh"

namespace bippb200 {

constexpr int kCtB = 64;                 // tile
constexpr int kCtS = kCtB + 4;           // shared stride: fragment reads of both layouts hit distinct banks
constexpr int kCtThreads = 256;
constexpr size_t kCtSmem = 2 * (size_t)kCtB * kCtS * sizeof(double);

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Tile of a column-major matrix into s[col][row] (stride kCtS); rows r0 .. r0+63 below rEnd
// and columns c0 .. c0+63 below cEnd, zero outside.
__device__ __forceinline__ void ct_load(double* __restrict__ s, const double* __restrict__ M, int ld, int r0, int c0,
                                        int rEnd, int cEnd) {
#pragma unroll 8
  for (int e = threadIdx.x; e < kCtB * kCtB; e += kCtThreads) {
    const int r = e % kCtB, c = e / kCtB;
    s[c * kCtS + r] = (r0 + r < rEnd && c0 + c < cEnd) ? M[(r0 + r) + (long long)(c0 + c) * ld] : 0.0;
  }
}

// acc += A B over k = 0 .. 63 for this warp's 16 x 32 part of the 64 x 64 tile: warp w has
// rows 16 (w % 4), columns 32 (w / 4). As[k][row]; Bs[k][col], or Bs[col][k] with BT.
// Lane (g = lane / 4, t = lane % 4) holds rows g, columns 2t, 2t + 1 of each 8 x 8 fragment.
template <bool BT>
__device__ __forceinline__ void ct_mma(double (&acc)[2][4][2], const double* __restrict__ As,
                                       const double* __restrict__ Bs) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rw = (warp & 3) * 16, cw = (warp >> 2) * 32;
#pragma unroll 4
  for (int k = 0; k < kCtB; k += 4) {
    double a[2], b[4];
#pragma unroll
    for (int i = 0; i < 2; ++i) a[i] = As[(k + t) * kCtS + rw + 8 * i + g];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      b[j] = BT ? Bs[(cw + 8 * j + g) * kCtS + k + t] : Bs[(k + t) * kCtS + cw + 8 * j + g];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
  }
}

// f(row, col, value) for this thread's elements of the 64 x 64 tile
template <typename F>
__device__ __forceinline__ void ct_each(double (&acc)[2][4][2], F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rw = (warp & 3) * 16, cw = (warp >> 2) * 32;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int u = 0; u < 2; ++u) f(rw + 8 * i + g, cw + 8 * j + 2 * t + u, acc[i][j][u]);
}

// Factor the 64 x 64 lower block D in place and form its inverse X (both [col][row], stride
// kCtS; on entry synchronised, X the identity, rows and columns past the matrix an identity
// too): 64 elimination steps on [D | X], each a pivot column scaled by every thread for itself
// and one update of the entries to its right and of X, thread = row tid % 64, columns tid / 64
// + 4 k. Bound by the chain of pivots (root, two barriers, update); for real blocks the
// register form below is twice as fast, and complex ones take this. False when a pivot was not positive.
__device__ __forceinline__ bool ct_eliminate(double2* __restrict__ D, double2* __restrict__ X,
                                             double2* __restrict__ lcol) {
  using E = double2;
  const int r = threadIdx.x % kCtB, g = threadIdx.x / kCtB;
  constexpr int G = kCtThreads / kCtB;
  bool ok = true;
  for (int j = 0; j < kCtB; ++j) {
    double p = e_re(D[j * kCtS + j]);
    if (!(p > 0.0)) {
      ok = false;
      p = 1e-300;
    }
    const double inv = rsqrt(p);
    const E l = r == j ? e_real(e_zero<E>(), p * inv) : e_scale(D[j * kCtS + r], inv);
    if (g == 0 && r >= j) lcol[r] = l;
    // row j of X is final; column j of D is taken, and rewritten below
    const int cx = threadIdx.x;
    if (cx <= j) X[cx * kCtS + j] = e_scale(X[cx * kCtS + j], inv);
    __syncthreads();
    if (r >= j && g == 0) D[j * kCtS + r] = l;
    if (r > j) {
      for (int c = j + 1 + g; c <= r; c += G) {
        E t = D[c * kCtS + r];
        e_sub_mulc(t, l, lcol[c]);
        D[c * kCtS + r] = t;
      }
      for (int c = g; c <= j; c += G) {
        E t = X[c * kCtS + r];
        e_sub_mul(t, l, X[c * kCtS + j]);
        X[c * kCtS + r] = t;
      }
    }
    __syncthreads();
  }
  return ok;
}

// One warp: factor of the 32 x 32 lower block at D (D[col][row], stride kCtS), lane = row;
// invd[j] = 1 / L_jj. False when a pivot was not positive.
__device__ __forceinline__ bool ct_factor32(double* __restrict__ D, double* __restrict__ invd) {
  const int lane = threadIdx.x & 31;
  double a[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) a[c] = D[c * kCtS + lane];
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    double p = __shfl_sync(0xffffffffu, a[j], j);
    if (!(p > 0.0)) {
      ok = false;
      p = 1e-300;
    }
    const double inv = rsqrt(p);
    if (lane == j) invd[j] = inv;
    a[j] = lane == j ? p * inv : a[j] * inv;
#pragma unroll
    for (int c = j + 1; c < 32; ++c) a[c] = fma(-a[j], __shfl_sync(0xffffffffu, a[j], c), a[c]);
  }
#pragma unroll
  for (int c = 0; c < 32; ++c) D[c * kCtS + lane] = lane >= c ? a[c] : 0.0;
  return ok;
}

// One warp: inverse of the factor at D into X (same layout), lane = column
__device__ __forceinline__ void ct_invert32(const double* __restrict__ D, const double* __restrict__ invd,
                                            double* __restrict__ X) {
  const int lane = threadIdx.x & 31;
  double x[32];
#pragma unroll
  for (int r = 0; r < 32; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
  for (int m = 0; m < 32; ++m) {
    x[m] *= invd[m];
#pragma unroll
    for (int r = m + 1; r < 32; ++r) x[r] = fma(-D[m * kCtS + r], x[m], x[r]);
  }
#pragma unroll
  for (int r = 0; r < 32; ++r) X[lane * kCtS + r] = x[r];
}

// 32 x 32 product by the whole CTA, thread = row tid % 32, columns 4 (tid / 32) .. + 3:
// f(row, col, sum_m A(row, m) B(m, col)) with A[m][row]; B[col][m] or, with BT, B[m][col]
template <bool BT, typename F>
__device__ __forceinline__ void ct_gemm32(const double* __restrict__ A, const double* __restrict__ B, F f) {
  const int r = threadIdx.x & 31, c0 = (threadIdx.x >> 5) * 4;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 8
  for (int m = 0; m < 32; ++m) {
    const double a = A[m * kCtS + r];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = fma(a, BT ? B[m * kCtS + c0 + u] : B[(c0 + u) * kCtS + m], s[u]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) f(r, c0 + u, s[u]);
}

// Factor the 64 x 64 lower block D in place and form its inverse X (both [col][row], every
// thread of the CTA; on entry synchronised, rows and columns past the matrix an identity).
__device__ __forceinline__ bool ct_diag(double* __restrict__ D, double* __restrict__ X, double* __restrict__ invd) {
  double *D21 = D + 32, *D22 = D + 32 * kCtS + 32, *X21 = X + 32, *X12 = X + 32 * kCtS, *X22 = X + 32 * kCtS + 32;
  __shared__ int sOk;
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) sOk = 1;
  __syncthreads();
  if (warp == 0) {
    if (!ct_factor32(D, invd) && threadIdx.x == 0) sOk = 0;
    __syncwarp();
    ct_invert32(D, invd, X);
  }
  __syncthreads();
  // L21 = A21 X11^T (kept in registers until every thread has read A21)
  double l[4];
  ct_gemm32<true>(D21, X, [&](int, int c, double v) { l[c & 3] = v; });
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) D21[((threadIdx.x >> 5) * 4 + u) * kCtS + (threadIdx.x & 31)] = l[u];
  __syncthreads();
  ct_gemm32<true>(D21, D21, [&](int r, int c, double v) { D22[c * kCtS + r] -= v; });
  __syncthreads();
  if (warp == 0) {
    if (!ct_factor32(D22, invd) && threadIdx.x == 0) sOk = 0;
    __syncwarp();
    ct_invert32(D22, invd, X22);
  }
  // X21 = -X22 (L21 X11); the inner product passes through the empty upper block
  ct_gemm32<false>(D21, X, [&](int r, int c, double v) { X12[c * kCtS + r] = v; });
  __syncthreads();
  ct_gemm32<false>(X22, X12, [&](int r, int c, double v) { X21[c * kCtS + r] = -v; });
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * 32; e += kCtThreads) {
    X12[(e / 32) * kCtS + e % 32] = 0.0;
    (D + 32 * kCtS)[(e / 32) * kCtS + e % 32] = 0.0;
  }
  __syncthreads();
  return sOk != 0;
}

// Factor the pivot block at k0 held in D, write L, and its inverse to W64 and LinvOut
template <typename E, typename O>
__device__ __forceinline__ void ct_pivot(E* D, E* X, E* lcol /* 64 */, E* __restrict__ Gb, E* __restrict__ Wb,
                                         O* __restrict__ Ob, int n, int k0, int ld, int* __restrict__ status) {
  const int kb = min(kCtB, n - k0);
  const E zero = e_zero<E>();
  for (int e = threadIdx.x; e < kCtB * kCtB; e += kCtThreads) {
    const int r = e % kCtB, c = e / kCtB;
    const E id = e_real(zero, r == c ? 1.0 : 0.0);
    if (r >= kb || c >= kb) D[c * kCtS + r] = id;
    X[c * kCtS + r] = sizeof(E) == 8 ? zero : id;   // the elimination starts from the identity
  }
  __syncthreads();
  bool ok;
  if constexpr (sizeof(E) == 8) ok = ct_diag(D, X, lcol);
  else ok = ct_eliminate(D, X, lcol);
  for (int e = threadIdx.x; e < kCtB * kCtB; e += kCtThreads) {
    const int r = e % kCtB, c = e / kCtB;
    if (r < kb && c < kb) {
      const long long at = (k0 + r) + (long long)(k0 + c) * ld;
      if (r >= c) Gb[at] = D[c * kCtS + r];
      if (Wb) Wb[at] = X[c * kCtS + r];
      store_conv(Ob + at, X[c * kCtS + r]);
    }
  }
  if (threadIdx.x == 0 && !ok) atomicOr(status, (int)kStatusCholeskyNotPD);
}

template <typename O>
__global__ void __launch_bounds__(kCtThreads, 1)
chol_diag_kernel(double* __restrict__ G, double* __restrict__ W64, O* __restrict__ Linv, const int* __restrict__ nred,
                 int ld, int* __restrict__ status) {
  const int b = blockIdx.x, n = nred[b];
  if (n <= 0) return;
  extern __shared__ __align__(16) double ct_smem[];
  __shared__ double lcol[kCtB];
  const long long off = (long long)b * ld * ld;
  ct_load(ct_smem, G + off, ld, 0, 0, n, n);
  ct_pivot<double, O>(ct_smem, ct_smem + kCtB * kCtS, lcol, G + off, W64 + off, Linv + off, n, 0, ld, status + b);
}

// Complex Hermitian matrices of at most 64 rows (beamformed Gram matrices): factor and inverse
// in one launch
constexpr size_t kCtSmemC = 2 * (size_t)kCtB * kCtS * sizeof(double2);
template <typename O>
__global__ void __launch_bounds__(kCtThreads, 1)
chol_small_kernel(double2* __restrict__ G, O* __restrict__ Linv, const int* __restrict__ nred, int ld,
                  int* __restrict__ status) {
  const int b = blockIdx.x, n = nred[b];
  if (n <= 0) return;
  extern __shared__ __align__(16) double2 ct_smem_c[];
  __shared__ double2 lcol[kCtB];
  const long long off = (long long)b * ld * ld;
  for (int e = threadIdx.x; e < kCtB * kCtB; e += kCtThreads) {
    const int r = e % kCtB, c = e / kCtB;
    if (c <= r && r < n) ct_smem_c[c * kCtS + r] = G[off + r + (long long)c * ld];
  }
  ct_pivot<double2, O>(ct_smem_c, ct_smem_c + kCtB * kCtS, lcol, G + off, (double2*)nullptr, Linv + off, n, 0, ld,
                       status + b);
}

// rows below pivot block k0: A <- A X^T, and the zero block of the inverse's upper triangle
template <typename O>
__global__ void __launch_bounds__(kCtThreads, 3)
chol_panel_kernel(double* __restrict__ G, const double* __restrict__ W64, O* __restrict__ Linv,
                  const int* __restrict__ nred, int ld, int k0) {
  const int b = blockIdx.y, n = nred[b], i0 = k0 + kCtB * (1 + blockIdx.x);
  if (i0 >= n) return;
  extern __shared__ __align__(16) double ct_smem[];
  double *As = ct_smem, *Xs = ct_smem + kCtB * kCtS;
  const long long off = (long long)b * ld * ld;
  ct_load(As, G + off, ld, i0, k0, n, n);
  ct_load(Xs, W64 + off, ld, k0, k0, n, n);
  __syncthreads();
  double acc[2][4][2] = {};
  ct_mma<false>(acc, As, Xs);   // sum_m A(r, m) X(c, m), X stored [m][c]
  ct_each(acc, [&](int r, int c, double v) {
    if (i0 + r < n) G[off + (i0 + r) + (long long)(k0 + c) * ld] = v;
  });
  for (int e = threadIdx.x; e < kCtB * kCtB; e += kCtThreads) {
    const int r = e % kCtB, c = e / kCtB;
    if (i0 + c < n) store_conv(Linv + off + (k0 + r) + (long long)(i0 + c) * ld, 0.0);
  }
}

// trailing tiles (ti, tj <= ti) after panel k0; tile (0, 0) is the next pivot block
template <typename O>
__global__ void __launch_bounds__(kCtThreads, 2)
chol_trail_kernel(double* __restrict__ G, double* __restrict__ W64, O* __restrict__ Linv, const int* __restrict__ nred,
                  int ld, int k0, int* __restrict__ status) {
  const int b = blockIdx.y, n = nred[b], t = blockIdx.x;
  int ti = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  while (ti * (ti + 1) / 2 > t) --ti;
  const int tj = t - ti * (ti + 1) / 2;
  const int i0 = k0 + kCtB * (1 + ti), j0 = k0 + kCtB * (1 + tj);
  if (i0 >= n) return;
  extern __shared__ __align__(16) double ct_smem[];
  __shared__ double lcol[kCtB];
  double *Pi = ct_smem, *Pj = ct_smem + kCtB * kCtS;
  const long long off = (long long)b * ld * ld;
  ct_load(Pi, G + off, ld, i0, k0, n, n);
  if (ti != tj) ct_load(Pj, G + off, ld, j0, k0, n, n);
  __syncthreads();
  double acc[2][4][2] = {};
  ct_mma<false>(acc, Pi, ti != tj ? Pj : Pi);
  if (t > 0) {
    ct_each(acc, [&](int r, int c, double v) {
      if (i0 + r < n && j0 + c <= i0 + r) G[off + (i0 + r) + (long long)(j0 + c) * ld] -= v;
    });
    return;
  }
  __syncthreads();
  ct_each(acc, [&](int r, int c, double v) {
    Pi[c * kCtS + r] = (i0 + r < n && c <= r) ? G[off + (i0 + r) + (long long)(i0 + c) * ld] - v : 0.0;
  });
  __syncthreads();
  ct_pivot<double, O>(Pi, Pj, lcol, G + off, W64 + off, Linv + off, n, i0, ld, status + b);
}

// One half of a doubling level of the inverse, diagonal blocks of size B already inverted
// (pairs of them at offsets 2 p B): FIRST forms T = L21 X11, kept transposed in the unused
// upper triangle of W64; then X21 = -X22 T goes to W64 and LinvOut.
template <typename O, bool FIRST>
__global__ void __launch_bounds__(kCtThreads, 3)
trinv_level_kernel(const double* __restrict__ G, double* __restrict__ W64, O* __restrict__ Linv,
                   const int* __restrict__ nred, int ld, int B) {
  const int tiles = B / kCtB;
  const int b = blockIdx.y, n = nred[b];
  const int p = blockIdx.x / (tiles * tiles), ij = blockIdx.x % (tiles * tiles);
  const int c0 = 2 * p * B, r0 = c0 + B;               // first column of the pair, first row below
  const int i = ij / tiles, j = ij % tiles;
  const int ri = r0 + kCtB * i, cj = c0 + kCtB * j;
  if (ri >= n) return;
  extern __shared__ __align__(16) double ct_smem[];
  double *As = ct_smem, *Bs = ct_smem + kCtB * kCtS;
  const long long off = (long long)b * ld * ld;
  double* Wb = W64 + off;
  double acc[2][4][2] = {};
  const int kBeg = FIRST ? j : 0, kEnd = FIRST ? tiles : i + 1;
  for (int k = kBeg; k < kEnd; ++k) {
    __syncthreads();
    if (FIRST) {
      ct_load(As, G + off, ld, ri, c0 + kCtB * k, n, n);            // L21(i, k)
      ct_load(Bs, Wb, ld, c0 + kCtB * k, cj, n, n);                 // X11(k, j): Bs[col][k]
    } else {
      ct_load(As, Wb, ld, ri, r0 + kCtB * k, n, n);                 // X22(i, k)
      ct_load(Bs, Wb, ld, cj, r0 + kCtB * k, n, n);                 // T^T(j, k): Bs[k][col]
    }
    __syncthreads();
    ct_mma<FIRST>(acc, As, Bs);
  }
  ct_each(acc, [&](int r, int c, double v) {
    if (ri + r < n) {
      if (FIRST) {
        Wb[(cj + c) + (long long)(ri + r) * ld] = v;
      } else {
        const long long at = (ri + r) + (long long)(cj + c) * ld;
        Wb[at] = -v;
        store_conv(Linv + off + at, -v);
      }
    }
  });
}

// L (in place of G), and L^-1 to W64 and, rounded to O, to Linv for a batch of nb real
// matrices of at most nmax rows; leading dimension and stride ld, ld^2.
template <typename O>
inline void chol_inverse(cudaStream_t st, double* G, double* W64, O* Linv, const int* nred, int nb, int nmax, int ld,
                         int* status) {
  for (auto k : {(const void*)chol_diag_kernel<O>, (const void*)chol_panel_kernel<O>, (const void*)chol_trail_kernel<O>,
                 (const void*)trinv_level_kernel<O, true>, (const void*)trinv_level_kernel<O, false>})
    B2_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCtSmem));
  count_launch();
  chol_diag_kernel<O><<<nb, kCtThreads, kCtSmem, st>>>(G, W64, Linv, nred, ld, status);
  for (int k0 = 0; k0 + kCtB < nmax; k0 += kCtB) {
    const int below = (nmax - k0 - 1) / kCtB;
    count_launch();
    chol_panel_kernel<O><<<dim3(below, nb), kCtThreads, kCtSmem, st>>>(G, W64, Linv, nred, ld, k0);
    count_launch();
    chol_trail_kernel<O><<<dim3(below * (below + 1) / 2, nb), kCtThreads, kCtSmem, st>>>(G, W64, Linv, nred, ld, k0,
                                                                                       status);
  }
  for (int B = kCtB; B < nmax; B *= 2) {
    const int pairs = (nmax - B + 2 * B - 1) / (2 * B), tiles = B / kCtB;
    const dim3 grid(pairs * tiles * tiles, nb);
    count_launch();
    trinv_level_kernel<O, true><<<grid, kCtThreads, kCtSmem, st>>>(G, W64, Linv, nred, ld, B);
    count_launch();
    trinv_level_kernel<O, false><<<grid, kCtThreads, kCtSmem, st>>>(G, W64, Linv, nred, ld, B);
  }
  B2_CHECK_LAUNCH();
}

}  // namespace bippb200

// Eigenpairs of a batch of real symmetric tridiagonal matrices in FP64: bisection for the
// eigenvalues, twisted factorisations for the eigenvectors, in three launches over
// (matrix, eigenvalue chunk) (sm_100a).
//
// The reference leaves this to LAPACK's ?hegv (src/host/lapack_api.hpp:112-158). Both the
// Sturm counts and the factorisations are n-step recurrences, so the time of a matrix is
// the latency of its serial chain, not arithmetic or bytes. One CTA per matrix with the
// quotient form q_k = (d_k - x) - e_k^2 / q_{k-1} paid a dependent FP64 division per step
// and 53 bisection steps (6.0 ms for one matrix of 550 rows, 13.5 ms for 2048 matrices of
// 380-512 rows). Here
//  - the recurrences run on p_k = (d_k - x) p_{k-1} - e_{k-1}^2 p_{k-2} (q_k = p_k / p_{k-1}),
//    one dependent FMA per step. Each step's rounding is a relative perturbation of d_k - x
//    and e_{k-1}^2, as in the quotient form. The matrix is scaled by a power of two to a norm
//    in [1/2, 1), p is rescaled every 8 steps (4 in the factorisations) and pivots are
//    bounded below (ts_pivot), so that every p is a normal number;
//  - a CTA first counts at 128 points across the whole interval in one sweep, which gives
//    every eigenvalue its starting interval; then M lanes per eigenvalue cut it M + 1 ways
//    per sweep. M (1..32) is chosen so that the lanes of the batch fill the GPU once:
//    more lanes only repeat work when the batch fills it already;
//  - the two factorisations of an eigenvector, from the top and from the bottom, run in two
//    lanes at once, their quotients off the chain.
// One matrix of 550 rows takes 0.46 ms, 64 of 256 0.37, 512 of 380-512 2.4 for all three
// launches; in 128 of 380-512 the search is bound by the latency of its recurrence and the
// integer comparisons around it, the eigenvectors by reading their quotients back with the few
// lanes that the level range leaves (profiled at 41 % and 19 % of the issue slots).
#pragma once

#include "common.cuh"

namespace bippb200 {

constexpr int kTsThreads = 128;

// Pivots q_k = p_k / p_{k-1} below 2^-100 in magnitude (of the scaled matrix) count as
// -2^-100: a perturbation of d_k of that size, far below a rounding of the norm. It bounds
// what a product of pivots can reach between two rescales, so that couplings and differences
// down to the smallest numbers leave no p subnormal.
constexpr double kTsTiny = 7.888609052210118e-31;

// p with its pivot p / prev so bounded
__device__ __forceinline__ double ts_pivot(double p, double prev) {
  const int hp = __double2hiint(p) & 0x7ff00000, hq = __double2hiint(prev) & 0x7ff00000;
  return hp < hq - (100 << 20) ? -kTsTiny * prev : p;
}

// The counts' form, one comparison with a constant: `steps` steps after a rescale p stays at
// or above 2^-100 (steps + 1), by induction over prev
__device__ __forceinline__ double ts_pivot(double p, double prev, int steps) {
  return (__double2hiint(p) & 0x7fffffff) < ((1023 - 100 * (steps + 1)) << 20) ? -kTsTiny * prev : p;
}

// common power-of-two factor that brings the larger of |a|, |b| to [1, 2); b, of which the
// next pivots are multiples, then at least 2^-100 in magnitude, with its sign
__device__ __forceinline__ void ts_rescale(double& a, double& b) {
  const int ha = __double2hiint(a) & 0x7ff00000, hb = __double2hiint(b) & 0x7ff00000;
  const double s = __hiloint2double(0x7fe00000 - max(ha, hb), 0);
  a *= s;
  b *= s;
  const int h = __double2hiint(b);
  if ((h & 0x7fffffff) < (923 << 20)) b = __hiloint2double((h & (int)0x80000000) | (923 << 20), 0);
}

// eigenvalues of the scaled matrix below x; de[k] = (d_k, e_{k-1}^2), de[0].y unused
__device__ __forceinline__ int ts_count(const double2* __restrict__ de, int n, double x) {
  double p0 = 1.0, p1 = ts_pivot(de[0].x - x, 1.0, 0);
  unsigned cnt = (unsigned)__double2hiint(p1) >> 31;
  int k = 1;
  auto step = [&](double2 v, int u) {
    const double p2 = ts_pivot(fma(v.x - x, p1, -v.y * p0), p1, u + 1);
    cnt += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p2;
  };
  for (; k + 8 <= n; k += 8) {
    ts_rescale(p0, p1);
#pragma unroll
    for (int u = 0; u < 8; ++u) step(de[k + u], u);
  }
  ts_rescale(p0, p1);
  for (int u = 0; k < n; ++k, ++u) step(de[k], u);
  return (int)cnt;
}

// Load a matrix scaled by `scale` = 2^-k (norm in [1/2, 1)) and its Gershgorin interval
// [lo, hi] (scaled); red: 32 doubles. Returns with every thread synchronised.
__device__ __forceinline__ void ts_load(const double* __restrict__ d, const double* __restrict__ e, int n,
                                        double2* __restrict__ de, double* red, double& lo, double& hi, double& tnorm,
                                        double& scale) {
  double l = 1e300, h = -1e300;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double ek = k < n - 1 ? fabs(e[k]) : 0.0, em = k > 0 ? fabs(e[k - 1]) : 0.0;
    l = fmin(l, d[k] - (ek + em));
    h = fmax(h, d[k] + (ek + em));
  }
  l = block_min(l, red, 1e300);
  __syncthreads();
  h = block_max(h, red, -1e300);
  const double t = fmax(fabs(l), fabs(h));
  // exponent field of t, kept where both 2^-k and its square products are normal
  const int ex = min(max((__double2hiint(t) >> 20) & 0x7ff, 200), 1800);
  scale = __hiloint2double((2045 - ex) << 20, 0);   // 2^(1022 - ex): t scale in [1/2, 1)
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double em = k > 0 ? e[k - 1] * scale : 0.0;
    de[k] = make_double2(d[k] * scale, em * em);
  }
  tnorm = t * scale;
  const double slack = 4.0 * 2.220446049250313e-16 * tnorm + 1e-290;
  lo = l * scale - slack;
  hi = h * scale + slack;
  __syncthreads();
}

// Eigenvalues: all of them, or (allValues == 0) those in [vecLo, vecHi], whose index range
// two Sturm counts give; the others come out as zero. CTA (c, r): chunk c of
// kTsThreads / M eigenvalues of the matrix of rank r in `order`. range[2b], range[2b+1]:
// the index range. Dynamic shared memory: Nmax double2.
static __global__ void __launch_bounds__(kTsThreads)
tridiag_values_kernel(const double* __restrict__ dIn, const double* __restrict__ eIn, const int* __restrict__ nred,
                      int Nmax, double vecLo, double vecHi, int allValues, int M, double* __restrict__ lamOut,
                      int* __restrict__ range, const int* __restrict__ order) {
  const int b = order ? order[blockIdx.y] : blockIdx.y;
  const int n = nred[b];
  if (n <= 0) {   // every row flagged: an empty range
    if (blockIdx.x == 0 && threadIdx.x < 2) range[2 * b + threadIdx.x] = 0;
    return;
  }
  extern __shared__ __align__(16) double2 ts_smem[];
  double2* de = ts_smem;
  __shared__ double red[32];
  __shared__ int cA[kTsThreads], sRange[2];
  const int tid = threadIdx.x;
  double lo, hi, tnorm, scale;
  ts_load(dIn + (long long)b * Nmax, eIn + (long long)b * Nmax, n, de, red, lo, hi, tnorm, scale);
  if (allValues) {
    if (tid < 2) sRange[tid] = tid ? n : 0;
  } else if (tid < 2) {
    const double x = (tid ? vecHi : vecLo) * scale;
    // bounds beyond the interval keep every eigenvalue on that side
    sRange[tid] = tid ? (x < hi ? ts_count(de, n, x) : n) : (x > lo ? ts_count(de, n, x) : 0);
  }
  __syncthreads();
  const int vLo = sRange[0], vHi = max(sRange[0], sRange[1]);
  double* lam = lamOut + (long long)b * Nmax;
  if (blockIdx.x == 0) {
    for (int i = tid; i < n; i += kTsThreads)
      if (i < vLo || i >= vHi) lam[i] = 0.0;
    if (tid == 0) {
      range[2 * b] = vLo;
      range[2 * b + 1] = vHi;
    }
  }
  const int perCta = kTsThreads / M;
  const int i0 = vLo + blockIdx.x * perCta;
  if (i0 >= vHi) return;
  const double eps = 2.220446049250313e-16;
  if (!allValues) {
    const double a = vecLo * scale, c = vecHi * scale;
    if (a > lo) lo = a - (2.0 * eps * fabs(a) + 1e-290);
    if (c < hi) hi = c + (2.0 * eps * fabs(c) + 1e-290);
  }
  const double w = (hi - lo) / (kTsThreads + 1);
  cA[tid] = ts_count(de, n, lo + w * (tid + 1));
  __syncthreads();
  const int i = i0 + tid / M, j = tid % M;
  const bool act = i < vHi;
  double a = lo, c = hi;
  {
    int l = 0, h = kTsThreads;   // first point with more than i eigenvalues below it
    while (l < h) {
      const int m = (l + h) >> 1;
      if (cA[m] > i) h = m; else l = m + 1;
    }
    if (l > 0) a = lo + w * l;
    if (l < kTsThreads) c = lo + w * (l + 1);
  }
  const double f = 1.0 / (M + 1);
  const unsigned group = (M == 32 ? 0xffffffffu : ((1u << M) - 1u)) << ((tid & 31) / M * M);
  bool done = !act;
  for (int it = 0; it < 64; ++it) {
    // half the width at which halving would end (between eps / 2 and eps of the norm): a cut
    // into many parts can stop anywhere below the bound, and the eigenvectors, which are as
    // exact as the eigenvalue over its gap, were up to 1.7 times further off for it
    done = done || c - a <= fmax(eps * fmax(fabs(a), fabs(c)), 0.5 * eps * tnorm);
    if (!__any_sync(0xffffffffu, !done)) break;
    const double x = a + (c - a) * (f * (j + 1));
    const bool above = done ? false : ts_count(de, n, x) > i;
    const unsigned bal = __ballot_sync(0xffffffffu, above) & group;
    if (!done) {
      const int first = bal ? __ffs(bal) - 1 - (tid & 31) / M * M : M;   // first point above eigenvalue i
      const double an = first > 0 ? a + (c - a) * (f * first) : a;
      const double cn = first < M ? a + (c - a) * (f * (first + 1)) : c;
      done = !(an > a || cn < c);
      a = an;
      c = cn;
    }
  }
  if (act && j == 0) lam[i] = 0.5 * (a + c) / scale;
}

// Eigenvectors of the eigenvalues range[2b] .. range[2b+1]-1 of matrix b (trimmed to
// [vecLo, vecHi] by value), by the twisted factorisation of T - lambda I at the index of
// the smallest |gamma|. CTA (c, r): 64 eigenvectors, lanes of the first half of the CTA
// factorise from the top (quotients L_k = e_k / D+_k), of the second from the bottom
// (U_k = e_k / D-_{k+1}). krange receives the trimmed range (krange may not alias range).
// work: 2 Nmax^2 doubles per matrix, rows of eigenvalue index so that lanes are coalesced.
// Z: row-major Z[k Nmax + i], columns outside the range are not written.
// Dynamic shared memory: Nmax double2.
template <typename R>
__global__ void __launch_bounds__(kTsThreads)
tridiag_vectors_kernel(const double* __restrict__ dIn, const double* __restrict__ eIn, const int* __restrict__ nred,
                       int Nmax, const double* __restrict__ lamIn, double vecLo, double vecHi,
                       const int* __restrict__ range, int* __restrict__ krange, R* __restrict__ Z,
                       double* __restrict__ work, const int* __restrict__ order) {
  const int b = order ? order[blockIdx.y] : blockIdx.y;
  const int n = nred[b];
  if (n <= 0) {
    if (blockIdx.x == 0 && threadIdx.x < 2) krange[2 * b + threadIdx.x] = 0;
    return;
  }
  extern __shared__ __align__(16) double2 ts_smem[];
  double2* de = ts_smem;   // (d_k, e_k), scaled
  __shared__ double red[32], sBest[kTsThreads], sNrm[kTsThreads];
  __shared__ int sArg[kTsThreads], sK[2];
  const int tid = threadIdx.x;
  const double* lam = lamIn + (long long)b * Nmax;
  if (tid == 0) {
    int a = range[2 * b], c = range[2 * b + 1];
    while (a < c && lam[a] < vecLo) ++a;
    while (c > a && lam[c - 1] > vecHi) --c;
    sK[0] = a;
    sK[1] = c;
    if (blockIdx.x == 0) {
      krange[2 * b] = a;
      krange[2 * b + 1] = c;
    }
  }
  __syncthreads();
  constexpr int VPC = kTsThreads / 2;
  const int kHi = sK[1];
  if (sK[0] + (int)blockIdx.x * VPC >= kHi) return;
  double lo, hi, tnorm, scale;
  ts_load(dIn + (long long)b * Nmax, eIn + (long long)b * Nmax, n, de, red, lo, hi, tnorm, scale);
  for (int k = tid; k < n; k += kTsThreads) de[k].y = k < n - 1 ? eIn[(long long)b * Nmax + k] * scale : 0.0;
  __syncthreads();
  const int v = tid % VPC, role = tid / VPC;
  const int iv = sK[0] + blockIdx.x * VPC + v;
  const bool act = iv < kHi;
  const int i = act ? iv : kHi - 1;   // idle lanes repeat the last column without storing
  const double l = lam[i] * scale;
  double* Lp = work + (long long)b * 2 * Nmax * Nmax + i;
  double* Um = Lp + (long long)Nmax * Nmax;
  {
    // role 0: k = 0 .. n-2 from the top; role 1: k = n-2 .. 0 from the bottom
    double p0 = 1.0, p1 = (role ? de[n - 1].x : de[0].x) - l;
    double* out = role ? Um + (long long)max(n - 2, 0) * Nmax : Lp;
    const long long step = role ? -(long long)Nmax : Nmax;
    auto one = [&](int t) {
      const int k = role ? n - 2 - t : t;
      const double ek = de[k].y, dn = de[role ? k : k + 1].x;
      p1 = ts_pivot(p1, p0);
      if (act) *out = ek * p0 / p1;
      out += step;
      const double p2 = fma(dn - l, p1, -(ek * ek) * p0);
      p0 = p1;
      p1 = p2;
    };
    int t = 0;
    for (; t + 4 <= n - 1; t += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) one(t + u);
      p1 = ts_pivot(p1, p0);
      ts_rescale(p0, p1);
    }
    for (; t < n - 1; ++t) one(t);
  }
  __syncthreads();
  // twist index: smallest |gamma_k|, gamma_k = (d_k - l) - L_{k-1} e_{k-1} - U_k e_k; ties
  // go to the larger k
  {
    const int kb = role ? n / 2 : 0, ke = role ? n : n / 2;
    double best = 1e300;
    int arg = kb;
#pragma unroll 4
    for (int k = kb; k < ke; ++k) {
      const double lm = k > 0 ? Lp[(long long)(k - 1) * Nmax] * de[k - 1].y : 0.0;
      const double um = k < n - 1 ? Um[(long long)k * Nmax] * de[k].y : 0.0;
      const double g = fabs((de[k].x - l) - lm - um);
      if (g <= best) {
        best = g;
        arg = k;
      }
    }
    sBest[tid] = best;
    sArg[tid] = arg;
  }
  __syncthreads();
  int r = sArg[v];
  if (n > 1 && sBest[VPC + v] <= sBest[v]) r = sArg[VPC + v];
  if (n == 1) r = 0;
  // z_r = 1; z_k = -L_k z_{k+1} upwards (role 0), z_{k+1} = -U_k z_k downwards (role 1); the
  // values overwrite L and U, 8 quotients loaded ahead of the chain
  {
    double z1 = 1.0, z2 = 0.0, nrm = role ? 1.0 : 0.0;
    double* q = role ? Um : Lp;
    for (int t0 = 0; t0 < n - 1; t0 += 8) {
      double c[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = t0 + u, k = role ? t : n - 2 - t;
        c[u] = t < n - 1 ? q[(long long)k * Nmax] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int t = t0 + u, k = role ? t : n - 2 - t;
        if (t < n - 1 && (role ? k >= r : k < r)) {
          double z;
          if (z1 != 0.0) z = -c[u] * z1;
          else if (de[k].y == 0.0) z = 0.0;
          else z = role ? -((k > 0 ? de[k - 1].y : 0.0) / de[k].y) * z2 : -(de[k + 1].y / de[k].y) * z2;
          nrm = fma(z, z, nrm);
          if (act) q[(long long)k * Nmax] = z;
          z2 = z1;
          z1 = z;
        }
      }
    }
    sNrm[tid] = nrm;
  }
  __syncthreads();
  if (!act) return;
  const double inv = 1.0 / sqrt(sNrm[v] + sNrm[VPC + v]);
  R* Zb = Z + (long long)b * Nmax * Nmax + i;
  const int kb = role ? n / 2 : 0, ke = role ? n : n / 2;
#pragma unroll 8
  for (int k = kb; k < ke; ++k) {
    double z = 1.0;
    if (k < r) z = Lp[(long long)k * Nmax];
    else if (k > r) z = Um[(long long)(k - 1) * Nmax];
    Zb[(long long)k * Nmax] = (R)(z * inv);
  }
}

// fixed pseudo-random number in (-1, 1) for row k of eigenvector i (multiply-and-shift mixing)
__device__ __forceinline__ double ts_random(int i, int k) {
  unsigned h = (unsigned)i * 0x9e3779b1u ^ ((unsigned)k + 1u) * 0x85ebca77u;
  h ^= h >> 15;
  h *= 0x2c1b3c6du;
  h ^= h >> 12;
  h *= 0x297a2d39u;
  h ^= h >> 15;
  return ((double)(int)h + 0.5) * 4.656612873077393e-10;   // 2^-31
}

// One step of inverse iteration: z <- (T - l)^-1 z, normalised, or, at the start, of a vector of
// its own, by Gaussian elimination with partial pivoting (row k of U: u0, u1, u2) and pivots of
// at least `tiny`. One thread; at(a, k): its workspace, a = 0..2 the rows of U, 3 the
// right-hand side and the solution.
template <typename R, typename At>
__device__ __forceinline__ void ts_inverse_step(const double* __restrict__ d, const double* __restrict__ e, int n,
                                                double l, double tiny, bool start, int i, At at, R* __restrict__ z,
                                                long long ldz) {
  auto rhs = [&](int k) { return start ? ts_random(i, k) : (double)z[(long long)k * ldz]; };
  double a = d[0] - l, b = n > 1 ? e[0] : 0.0, r = rhs(0);
  for (int k = 0; k < n - 1; ++k) {
    const double s = e[k], q = d[k + 1] - l, t = k + 2 < n ? e[k + 1] : 0.0, rn = rhs(k + 1);
    if (fabs(a) >= fabs(s)) {
      if (fabs(a) < tiny) a = copysign(tiny, a);
      const double m = s / a;
      at(0, k) = a;
      at(1, k) = b;
      at(2, k) = 0.0;
      at(3, k) = r;
      a = fma(-m, b, q);
      b = t;
      r = fma(-m, r, rn);
    } else {
      const double m = a / s;
      at(0, k) = fabs(s) < tiny ? copysign(tiny, s) : s;
      at(1, k) = q;
      at(2, k) = t;
      at(3, k) = rn;
      a = fma(-m, q, b);
      b = -m * t;
      r = fma(-m, rn, r);
    }
  }
  at(0, n - 1) = fabs(a) < tiny ? copysign(tiny, a) : a;
  at(1, n - 1) = at(2, n - 1) = 0.0;
  at(3, n - 1) = r;
  double x1 = 0.0, x2 = 0.0, big = 0.0, f = 1.0;
  for (int k = n - 1; k >= 0; --k) {
    double x = (at(3, k) * f - at(1, k) * x1 - at(2, k) * x2) / at(0, k);
    if (fabs(x) > 1e150) {   // several vanishing pivots in a row
      x *= 1e-150;
      x1 *= 1e-150;
      f *= 1e-150;
      big *= 1e-150;
      for (int j = k + 1; j < n; ++j) at(3, j) *= 1e-150;
    }
    at(3, k) = x;
    big = fmax(big, fabs(x));
    x2 = x1;
    x1 = x;
  }
  const double scale = big > 0.0 ? 1.0 / big : 1.0;
  double norm2 = 0.0;
  for (int k = 0; k < n; ++k) {
    const double x = at(3, k) * scale;
    norm2 = fma(x, x, norm2);
  }
  const double inv = scale / sqrt(norm2);
  for (int k = 0; k < n; ++k) z[(long long)k * ldz] = (R)(at(3, k) * inv);
}

// Clusters: runs of eigenvalues whose neighbours are closer than 1e-10 of the norm. Twisted
// factorisations at equal eigenvalues give the same vector, so the members are found anew: a
// step of inverse iteration from vectors of their own, one thread each, orthogonalised in
// eigenvalue order (classical Gram-Schmidt, twice), and both once more, since the first
// orthogonalisation of unrelated vectors enlarges what they hold of other eigenvectors. The
// shift lies 8 roundings of the norm beside the eigenvalue: at equal eigenvalues, which come
// out a rounding apart, every direction of their space is then enlarged alike. One CTA per
// matrix, which returns at once when it has no cluster. work: 2 Nmax^2 doubles per matrix. krange null: all n. Dynamic
// shared memory: Nmax doubles.
template <typename R>
__global__ void __launch_bounds__(256)
tridiag_clusters_kernel(const double* __restrict__ dIn, const double* __restrict__ eIn, const int* __restrict__ nred,
                        int Nmax, const double* __restrict__ lamIn, const int* __restrict__ krange, R* __restrict__ Z,
                        double* __restrict__ work, int* __restrict__ status) {
  const int b = blockIdx.x;
  const int n = nred[b];
  if (n <= 0) return;
  extern __shared__ __align__(16) double ts_dots[];
  __shared__ double red[32], part[8][33];
  const double* d = dIn + (long long)b * Nmax;
  const double* e = eIn + (long long)b * Nmax;
  const double* lam = lamIn + (long long)b * Nmax;
  R* Zb = Z + (long long)b * Nmax * Nmax;
  double* wb = work + (long long)b * 2 * Nmax * Nmax;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kLo = krange ? krange[2 * b] : 0, kHi = krange ? krange[2 * b + 1] : n;
  double t = 0.0;
  for (int k = tid; k < n; k += blockDim.x)
    t = fmax(t, fabs(d[k]) + (k < n - 1 ? fabs(e[k]) : 0.0) + (k > 0 ? fabs(e[k - 1]) : 0.0));
  const double tnorm = fmax(block_max(t, red, 0.0), 1e-300), eps = 2.220446049250313e-16;
  const double ctol = 1e-10 * tnorm;
  bool close = false;
  for (int i = kLo + 1 + tid; i < kHi; i += blockDim.x) close = close || lam[i] - lam[i - 1] < ctol;
  if (!__syncthreads_or(close)) return;
  if (tid == 0) atomicOr(status + b, (int)kStatusClusterFix);
  const int P = min((int)blockDim.x, Nmax / 2);   // vectors at a time: four arrays of Nmax each
  for (int j0 = kLo, j1; j0 < kHi; j0 = j1) {
    for (j1 = j0 + 1; j1 < kHi && lam[j1] - lam[j1 - 1] < ctol;) ++j1;
    if (j1 - j0 < 2) continue;
    for (int step = 0; step < 2; ++step) {
      for (int c = j0 + tid; tid < P && c < j1; c += P) {
        auto at = [&](int a, int k) -> double& { return wb[((long long)a * Nmax + k) * P + tid]; };
        ts_inverse_step<R>(d, e, n, lam[c] + 8.0 * eps * tnorm, eps * tnorm, step == 0, c, at, Zb + c, Nmax);
      }
      __syncthreads();
      for (int i = j0; i < j1; ++i) {
        for (int pass = 0; pass < (i > j0 ? 2 : 0); ++pass) {
          // dots[j] = z_{j0+j} . z_i: lanes over 32 vectors, warps over the rows
          for (int jb = j0; jb < i; jb += 32) {
            double s = 0.0;
            if (jb + lane < i) {
#pragma unroll 4
              for (int k = warp; k < n; k += 8)
                s = fma((double)Zb[(long long)k * Nmax + jb + lane], (double)Zb[(long long)k * Nmax + i], s);
            }
            part[warp][lane] = s;
            __syncthreads();
            if (warp == 0) {
#pragma unroll
              for (int w = 1; w < 8; ++w) s += part[w][lane];
              if (jb + lane < i) ts_dots[jb - j0 + lane] = s;
            }
            __syncthreads();
          }
          // z_i -= sum_j dots[j] z_{j0+j}, a warp per row
          for (int k = warp; k < n; k += 8) {
            double s = 0.0;
            for (int j = j0 + lane; j < i; j += 32) s = fma(ts_dots[j - j0], (double)Zb[(long long)k * Nmax + j], s);
            s = warp_sum(s);
            if (lane == 0) Zb[(long long)k * Nmax + i] = (R)((double)Zb[(long long)k * Nmax + i] - s);
          }
          __syncthreads();
          // normalised
          double q = 0.0;
          for (int k = tid; k < n; k += blockDim.x) {
            const double zv = (double)Zb[(long long)k * Nmax + i];
            q = fma(zv, zv, q);
          }
          const double nr = sqrt(block_sum(q, red));
          const double inv = nr > 0 ? 1.0 / nr : 0.0;
          for (int k = tid; k < n; k += blockDim.x)
            Zb[(long long)k * Nmax + i] = (R)((double)Zb[(long long)k * Nmax + i] * inv);
          __syncthreads();
        }
      }
    }
  }
}

}  // namespace bippb200

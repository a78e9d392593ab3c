// Householder tridiagonalisation of a batch of Hermitian matrices, blocked panels, a cluster
// of CTAs per matrix (sm_100a). The reference leaves it to LAPACK's ?hegv
// (src/host/lapack_api.hpp:112-158); reflectors follow ?hetrd/?latrd/?larfg (lower): H_i = I -
// tau v v^H, v(0) = 1 stored below the subdiagonal of column i of A, T in (d, e).
//
// Per column the work is one product y = A v with the trailing lower triangle, per panel of
// NB columns one rank-2 NB update of it. Bytes are the triangle once per column (n^3 / 6
// elements), from L2 while the matrices in flight fit it. A form with 32 x 16 units per warp
// spent 67 instructions per 32 matrix elements and column (16 of them multiply-adds), the rest
// on cross-lane column sums and shared atomics per unit, and kept twice the matrices in flight
// that L2 holds (26 % hits). Here
//  - a warp takes strips of SC columns: lanes hold rows, the SC column sums stay in registers
//    over all the strip's rows and are reduced across lanes once per strip; row sums go to an
//    array of the warp's own, read and written once per SC columns, without atomics. The next
//    32 rows are loaded while the current ones are used;
//  - the rank-2 NB update keeps two rows' V and W in registers against broadcast columns;
//  - a column costs five block barriers: every thread owns its rows through the column update,
//    the reflector, the corrections and w;
//  - 16 warps share a matrix, one matrix per SM, so that 148 triangles of 512 rows fit L2;
//  - with few matrices, or large ones, a cluster of CS CTAs shares one: strips are cut into
//    segments of 128 rows dealt to all warps of the cluster, each CTA sums its own part of y,
//    and one cluster barrier per column lets every CTA read the others' parts from their
//    shared memory. Everything else of a column is repeated by each CTA on its own copies of
//    v, V and W, bit for bit alike, which costs less than distributing it.
// Of the 8.0 ms of 148 matrices of 512 rows the products take 4.0, the updates 2.7 and the
// rest of the columns 1.2, at 2.1 instructions per cycle and SM.
// Measured (FP32, before -> after): 1024 matrices of 380-512 rows 48 -> 40.7 ms, 128 of them
// 10.9 -> 7.3, 64 of 256 3.0 -> 1.56, 37 of 250-333 4.0 -> 2.5, 64 of 768-1024 46.4 -> 28, one of 550
// 11.1 -> 4.1; FP64: one of 512 33.0 -> 4.4.
#pragma once

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "eig_kernels.cuh"
#include "hetrd.hpp"

namespace bippb200 {

constexpr int kHtSeg = 128;   // rows per unit when a cluster shares a matrix
constexpr int kHtAlign = 256;   // of the panel: its widest row (HtPanel::kRow)

// rows in shared memory: whole blocks of 32
__host__ __device__ constexpr int ht_pad(int nmax) { return (nmax + 31) & ~31; }

// bytes of shared memory per matrix row: V/W panel, a row of partial sums per warp, v, and
// (clusters) two buffers of the CTA's part of y
template <typename C, int NB, int T>
constexpr size_t ht_smem(int nmax, bool cluster) {
  return (size_t)ht_pad(nmax) * sizeof(C) * (2 * NB + T / 32 + 1 + (cluster ? 2 : 0));
}

__device__ __forceinline__ uint32_t ht_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void ht_cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// element of another CTA's shared memory
__device__ __forceinline__ float2 ht_remote(const float2* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), m;
  float2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(m) : "memory");
  return v;
}
__device__ __forceinline__ double2 ht_remote(const double2* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), m;
  double2 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(m) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(m) : "memory");
  return v;
}

// V and W of row r, reflector q of the panel: 16-byte pieces of a row, piece p of row r at
// p ^ (r mod 8), so that lanes on consecutive rows read distinct banks. A row's pieces are
// addressed from row(r), whose low bits hold the rotation, by one exclusive or each.
template <typename C, int NB> struct HtPanel;
template <int NB> struct HtPanel<float2, NB> {   // piece q = (V, W)
  static constexpr int kRow = NB * 16;
  static constexpr uint32_t kMask = NB * 16 - 16;
  // the exclusive or must not reach the base's bits, nor leave the row
  static_assert(kRow <= kHtAlign && kHtAlign % kRow == 0, "rows aligned to their own size");
  uint32_t base;   // shared address, aligned to kHtAlign
  __device__ __forceinline__ uint32_t row(int r) const { return base + (uint32_t)r * kRow + (((uint32_t)r << 4) & kMask); }
  static __device__ __forceinline__ void get(uint32_t row, int q, float2& v, float2& w) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(w.x), "=f"(w.y)
                 : "r"(row ^ (uint32_t)(q << 4)));
  }
  static __device__ __forceinline__ void set(uint32_t row, int q, int w, float2 v) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"((row ^ (uint32_t)(q << 4)) + 8 * w), "f"(v.x), "f"(v.y) : "memory");
  }
  static __device__ __forceinline__ float2 one(uint32_t row, int q, int w) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"((row ^ (uint32_t)(q << 4)) + 8 * w));
    return v;
  }
};
template <int NB> struct HtPanel<double2, NB> {   // pieces 2 q = V_q, 2 q + 1 = W_q
  static constexpr int kRow = NB * 32;
  static_assert(kRow <= kHtAlign && kHtAlign % kRow == 0, "rows aligned to their own size");
  uint32_t base;
  __device__ __forceinline__ uint32_t row(int r) const { return base + (uint32_t)r * kRow + (((uint32_t)r << 4) & 112u); }
  static __device__ __forceinline__ double2 one(uint32_t row, int q, int w) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(row ^ (uint32_t)(q * 32 + w * 16)));
    return v;
  }
  static __device__ __forceinline__ void get(uint32_t row, int q, double2& v, double2& w) {
    v = one(row, q, 0);
    w = one(row, q, 1);
  }
  static __device__ __forceinline__ void set(uint32_t row, int q, int w, double2 v) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(row ^ (uint32_t)(q * 32 + w * 16)), "d"(v.x), "d"(v.y) : "memory");
  }
};

// One strip of SC columns from c0, rows [rBeg, rEnd) (multiples of 32): row sums a x_c into
// yw[r], column sums conj(a) x_r into yw[c], for the trailing block of rows and columns
// s0 .. n-1. x is zero outside it, and the column sums of columns outside it are dropped. On
// the diagonal the column sum takes the element and the row sum leaves it out.
template <typename C, typename R, int SC>
__device__ __forceinline__ void ht_strip(const C* __restrict__ A, int ld, int n, int s0, int c0, int rBeg, int rEnd,
                                         const C* __restrict__ x, C* __restrict__ yw) {
  const int lane = threadIdx.x & 31;
  const C zero = mk(R(0), R(0));
  C xc[SC];
#pragma unroll
  for (int u = 0; u < SC; ++u) xc[u] = x[c0 + u];
  C cs[SC];
#pragma unroll
  for (int u = 0; u < SC; ++u) cs[u] = zero;
  const int diag = c0 & ~31;   // row block holding the strip's diagonal
  const int end = min(rEnd, n);
  int r0 = max(rBeg, diag);
  const C* p = A + r0 + lane + (long long)c0 * ld;
  auto get = [&](int u) { return __ldcg(p + (long long)u * ld); };
  // rows past the matrix (last block) read as zero
  auto load = [&](C (&t)[SC], int R0) {
    if (R0 + 32 <= n) {
#pragma unroll
      for (int u = 0; u < SC; ++u) t[u] = get(u);
    } else {
      const bool ok = R0 + lane < n;
#pragma unroll
      for (int u = 0; u < SC; ++u) {
        t[u] = zero;
        if (ok) t[u] = get(u);
      }
    }
    p += 32;
  };
  auto use = [&](const C (&t)[SC], int r) {
    const C xr = x[r];
    C ry = yw[r];
#pragma unroll
    for (int u = 0; u < SC; ++u) {
      cfma_cj(cs[u], t[u], xr);
      cfma(ry, t[u], xc[u]);
    }
    yw[r] = ry;
  };
  C a[SC], b[SC];
  if (r0 == diag) {
    // columns up to r of this row are stored; the diagonal is real, enters the column sum
    // and leaves the row sum
    const int r = r0 + lane, cols = r < n ? r - c0 : -1;   // columns c0 .. c0 + cols
    C dg = zero;
#pragma unroll
    for (int u = 0; u < SC; ++u) {
      a[u] = zero;
      if (u <= cols) a[u] = get(u);
    }
    p += 32;
    if (r0 + 32 < end) load(b, r0 + 32);
#pragma unroll
    for (int u = 0; u < SC; ++u)
      if (u == cols) dg = cscale(xc[u], -a[u].x), a[u].y = R(0);
    use(a, r);
    yw[r] = yw[r] + dg;
    r0 += 32;
  } else {
    load(b, r0);
  }
  // two blocks per turn, the next one loaded while the current one is used
  for (; r0 < end; r0 += 64) {
    if (r0 + 32 < end) load(a, r0 + 32);
    use(b, r0 + lane);
    if (r0 + 32 < end) {
      if (r0 + 64 < end) load(b, r0 + 64);
      use(a, r0 + 32 + lane);
    }
  }
  // column totals: lanes with the same top bits hold column lane / (32 / SC)
  const C t = warp_reduce_scatter<SC>(cs, lane);
  __syncwarp();
  const int c = c0 + lane / (32 / SC);
  if (lane % (32 / SC) == 0 && c >= s0 && c < n) yw[c] = yw[c] + t;
  __syncwarp();
}

// A -= V W^H + W V^H on the lower triangle of rows and columns s0 .. n-1, units of 32 ROWS
// rows x 16 columns dealt to the warps of the cluster
template <typename C, typename R, int NB>
__device__ __forceinline__ void ht_rank2k(C* __restrict__ A, int ld, int n, int s0, const HtPanel<C, NB>& P, int wid,
                                          int nw) {
  constexpr int ROWS = sizeof(C) == 8 ? 2 : 1;
  const int lane = threadIdx.x & 31;
  const int base = s0 & ~31, nI = (n - base + 32 * ROWS - 1) / (32 * ROWS);
  int u = wid;
  for (int I = 0; I < nI; ++I) {
    const int R0 = base + I * 32 * ROWS;
    const int last = min(n, R0 + 32 * ROWS);                 // columns s0 .. last - 1
    const int nJ = (last - s0 + 15) / 16;
    if (u >= nJ) {
      u -= nJ;
      continue;
    }
    C rv[ROWS][NB], rw[ROWS][NB];
    int row[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      row[i] = R0 + 32 * i + lane;
      const int r = min(max(row[i], s0), n - 1);
#pragma unroll
      for (int q = 0; q < NB; ++q) P.get(P.row(r), q, rv[i][q], rw[i][q]);
    }
    auto column = [&](int c, C* p, bool whole) {
      C a[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        a[i] = mk(R(0), R(0));
        if (whole || (row[i] >= c && row[i] < n)) a[i] = __ldcg(p + row[i]);
      }
      const uint32_t pc = P.row(c);
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        C v, w;
        P.get(pc, q, v, w);
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
          a[i].x = fma(-rv[i][q].x, w.x, a[i].x); a[i].x = fma(-rv[i][q].y, w.y, a[i].x);
          a[i].y = fma(-rv[i][q].y, w.x, a[i].y); a[i].y = fma(rv[i][q].x, w.y, a[i].y);
          a[i].x = fma(-rw[i][q].x, v.x, a[i].x); a[i].x = fma(-rw[i][q].y, v.y, a[i].x);
          a[i].y = fma(-rw[i][q].y, v.x, a[i].y); a[i].y = fma(rw[i][q].x, v.y, a[i].y);
        }
      }
#pragma unroll
      for (int i = 0; i < ROWS; ++i)
        if (whole || (row[i] >= c && row[i] < n)) p[row[i]] = a[i];
    };
    for (; u < nJ; u += nw) {
      const int cb = s0 + 16 * u, ce = min(cb + 16, last);
      C* p = A + (long long)cb * ld;
      if (ce == cb + 16 && ce <= R0 && R0 + 32 * ROWS <= n) {
        // no entry on or above the diagonal or past the matrix
#pragma unroll 2
        for (int c = cb; c < cb + 16; ++c, p += ld) column(c, p, true);
      } else {
        for (int c = cb; c < ce; ++c, p += ld) column(c, p, false);
      }
    }
    u -= nJ;
  }
}

// One matrix (n >= 1) on T threads per CTA. RPT: rows per thread (T RPT >= n).
template <typename C, typename R, int NB, int T, int RPT, int CS>
__device__ __forceinline__ void ht_matrix(C* __restrict__ A, int n, int ld, double* __restrict__ d,
                                          double* __restrict__ e, C* __restrict__ taus, unsigned char* smem, int nmax,
                                          uint32_t rank) {
  constexpr int SC = sizeof(C) == 8 ? 8 : 4, kHtThreads = T, kHtWarps = T / 32;
  const C zero = mk(R(0), R(0));
  HtPanel<C, NB> P;
  P.base = (uint32_t)__cvta_generic_to_shared(smem);
  C* yw = reinterpret_cast<C*>(smem) + (size_t)nmax * 2 * NB;   // [warp][nmax]
  C* x = yw + (size_t)nmax * kHtWarps;                          // [nmax] v of the current column
  C* part = x + nmax;                                           // [2][nmax] (clusters)
  __shared__ C tq[2 * NB], sAlpha;
  __shared__ R sNorm[kHtWarps], sDot[2 * kHtWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wid = warp * CS + (int)rank, nw = kHtWarps * CS;    // warp of the cluster
  for (int i = tid; i < kHtWarps * nmax; i += kHtThreads) yw[i] = zero;
  for (int i = tid; i < nmax; i += kHtThreads) x[i] = zero;
  C col[RPT], v[RPT];
  if (n == 1) {
    if (rank == 0 && tid == 0) d[0] = (double)A[0].x;
    return;
  }
  __syncthreads();
  for (int k0 = 0; k0 < n - 1; k0 += NB) {
    const int jn = min(NB, n - 1 - k0);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int r = tid + kHtThreads * i;
      col[i] = (r >= k0 && r < n) ? __ldcg(A + r + (long long)k0 * ld) : zero;
    }
    for (int j = 0; j < jn; ++j) {
      const int c = k0 + j;
      // column c with the panel's earlier reflectors; its norm below the subdiagonal
      R part2 = 0;
      for (int q = 0; q < j; ++q) {
        C vc, wc;
        P.get(P.row(c), q, vc, wc);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + kHtThreads * i;
          if (r >= c && r < n) {
            C vr, wr;
            P.get(P.row(r), q, vr, wr);
            col[i] = col[i] - cmulc(vr, wc) - cmulc(wr, vc);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + kHtThreads * i;
        if (r == c && rank == 0) d[c] = (double)col[i].x;
        if (r == c + 1) sAlpha = col[i];
        if (r > c + 1 && r < n) part2 += cabs2(col[i]);
      }
      part2 = warp_sum(part2);
      if (lane == 0) sNorm[warp] = part2;
      __syncthreads();
      // reflector
      C alpha = sAlpha;
      R xnorm2 = 0, up = R(1), down = R(1);
#pragma unroll
      for (int w = 0; w < kHtWarps; ++w) xnorm2 += sNorm[w];
      if (hh_underflows(alpha, xnorm2)) {   // the same in every thread of the cluster
        up = R(kHhUp), down = R(kHhDown);
        part2 = 0;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + kHtThreads * i;
          if (r > c + 1 && r < n) part2 += cabs2(cscale(col[i], up));
        }
        part2 = warp_sum(part2);
        __syncthreads();
        if (lane == 0) sNorm[warp] = part2;
        __syncthreads();
        xnorm2 = 0;
#pragma unroll
        for (int w = 0; w < kHtWarps; ++w) xnorm2 += sNorm[w];
        alpha = cscale(alpha, up);
        if (hh_underflows(alpha, xnorm2)) alpha = zero, xnorm2 = R(0);
      }
      C tau, sc;
      R beta;
      hh_reflector(alpha, xnorm2, tau, sc, beta);
      beta *= down;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + kHtThreads * i;
        v[i] = zero;
        if (r == c) x[r] = zero;   // leaves the trailing block
        if (r > c && r < n) {
          v[i] = r == c + 1 ? mk(R(1), R(0)) : cmul(cscale(col[i], up), sc);
          x[r] = v[i];
          P.set(P.row(r), j, 0, v[i]);
        }
      }
      __syncthreads();
      // the next column's entries (unchanged within the panel) arrive during the product
      if (j + 1 < jn) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + kHtThreads * i;
          col[i] = (r > c && r < n) ? __ldcg(A + r + (long long)(c + 1) * ld) : zero;
        }
      }
      // tq[q] = W_q^H v, tq[NB + q] = V_q^H v: one warp per product
      for (int t = warp; t < 2 * j; t += kHtWarps) {
        const int q = t >> 1, isV = t & 1;
        C acc = zero;
        for (int r = c + 1 + lane; r < n; r += 32) cfma_cj(acc, P.one(P.row(r), q, 1 - isV), x[r]);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) tq[isV * NB + q] = acc;
      }
      // y = A22 v
      const int s0 = c + 1;
      {
        C* yo = yw + (size_t)warp * nmax;
        const int cb = s0 & ~(SC - 1), nStrips = (n - cb + SC - 1) / SC, rb = s0 & ~31;
        if (CS == 1) {
          // strips shorten to the right: dealt there and back
          for (int t = 0;; ++t) {
            const int k = t * kHtWarps + ((t & 1) ? kHtWarps - 1 - warp : warp);
            if (t * kHtWarps >= nStrips) break;
            if (k < nStrips) ht_strip<C, R, SC>(A, ld, n, s0, cb + SC * k, rb, (n + 31) & ~31, x, yo);
          }
        } else {
          int u = wid;
          for (int g = rb; g < n; g += kHtSeg) {
            const int K = min(nStrips, (g + kHtSeg - 1 - cb) / SC + 1);   // strips that reach rows g ..
            for (; u < K; u += nw) ht_strip<C, R, SC>(A, ld, n, s0, cb + SC * u, g, g + kHtSeg, x, yo);
            u -= K;
          }
        }
      }
      __syncthreads();
      C y[RPT];
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + kHtThreads * i;
        y[i] = zero;
        if (r > c && r < n) {
#pragma unroll
          for (int w = 0; w < kHtWarps; ++w) {
            y[i] = y[i] + yw[w * nmax + r];
            yw[w * nmax + r] = zero;
          }
          if (CS > 1) part[(c & 1) * nmax + r] = y[i];
        }
      }
      if (CS > 1) {
        // a buffer is rewritten two columns later, after another barrier that every reader
        // of this one has passed
        ht_cluster_barrier();
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + kHtThreads * i;
          if (r > c && r < n) {
            C t[CS];
#pragma unroll
            for (int k = 0; k < CS; ++k) t[k] = ht_remote(part + (c & 1) * nmax + r, k);
            y[i] = t[0];
#pragma unroll
            for (int k = 1; k < CS; ++k) y[i] = y[i] + t[k];
          }
        }
      }
      // y -= V (W^H v) + W (V^H v); w = tau y - 1/2 tau ((tau y)^H v) v
      for (int q = 0; q < j; ++q) {
        const C tw = tq[q], tv = tq[NB + q];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
          const int r = tid + kHtThreads * i;
          if (r > c && r < n) {
            C vr, wr;
            P.get(P.row(r), q, vr, wr);
            y[i] = y[i] - cmul(vr, tw) - cmul(wr, tv);
          }
        }
      }
      C dot = zero;
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        y[i] = cmul(tau, y[i]);
        cfma_cj(dot, y[i], v[i]);
      }
      dot.x = warp_sum(dot.x);
      dot.y = warp_sum(dot.y);
      if (lane == 0) {
        sDot[2 * warp] = dot.x;
        sDot[2 * warp + 1] = dot.y;
      }
      __syncthreads();
      dot = zero;
#pragma unroll
      for (int w = 0; w < kHtWarps; ++w) dot = dot + mk(sDot[2 * w], sDot[2 * w + 1]);
      const C alph = cscale(cmul(tau, dot), R(-0.5));
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = tid + kHtThreads * i;
        if (r > c && r < n) {
          P.set(P.row(r), j, 1, y[i] + cmul(alph, v[i]));
          // stored here, not with v above: the other CTAs have read column c by now
          if (rank == 0) A[r + (long long)c * ld] = r == c + 1 ? mk(beta, R(0)) : v[i];
        }
      }
      if (rank == 0 && tid == 0) {
        e[c] = (double)beta;
        taus[c] = tau;
      }
      __syncthreads();
    }
    const int s0 = k0 + jn;
    if (s0 == n - 1) {
      if (rank == 0 && tid == 0) {
        R a = __ldcg(A + (n - 1) + (long long)(n - 1) * ld).x;
        for (int q = 0; q < jn; ++q) {
          C vr, wr;
          P.get(P.row(n - 1), q, vr, wr);
          a -= R(2) * (vr.x * wr.x + vr.y * wr.y);
        }
        d[n - 1] = (double)a;
      }
      break;
    }
    ht_rank2k<C, R, NB>(A, ld, n, s0, P, wid, nw);
    if (CS > 1) ht_cluster_barrier();
    else __syncthreads();
  }
}

// Clusters of CS CTAs, cluster k taking matrices k, k + (number of clusters), .. of the size
// order.
template <typename C, typename R, int NB, int T, int RPT, int CS>
__global__ void __launch_bounds__(T, sizeof(C) == 8 && T == 256 ? 2 : 1)
hetrd_cluster_kernel(C* __restrict__ A, const int* __restrict__ nred, int ld, double* __restrict__ dOut,
                     double* __restrict__ eOut, C* __restrict__ tauOut, const int* __restrict__ order, int nBatch,
                     int nmax) {
  extern __shared__ __align__(kHtAlign) unsigned char ht_smem_raw[];
  const uint32_t rank = CS > 1 ? ht_cluster_rank() : 0;
  for (int w = blockIdx.x / CS; w < nBatch; w += gridDim.x / CS) {
    const int b = order[w], n = nred[b];
    if (n > 0)
      ht_matrix<C, R, NB, T, RPT, CS>(A + (long long)b * ld * ld, n, ld, dOut + (long long)b * ld, eOut + (long long)b * ld,
                                   tauOut + (long long)b * ld, ht_smem_raw, ht_pad(nmax), rank);
    // no CTA leaves, or rewrites its parts of y, while another may still read them
    if (CS > 1) ht_cluster_barrier();
    else __syncthreads();
  }
}

// Matrices of at most 4 NK rows, one CTA of 16 NK threads each, unblocked, the whole matrix in
// registers: thread (row i = tid / 4, part p = tid % 4) holds the elements of columns p + 4 k
// of both triangles. Such a matrix is all latency: with panels in shared memory and the triangle
// in L2 a column took 3.3 us (0.20 ms for 60 rows) for a few hundred multiply-adds. Here a
// column is four barriers and no global load: the rank-2 update hands the next column and its
// norm on, v and w are read as broadcasts.
template <typename C, typename R, int NK>
__global__ void __launch_bounds__(16 * NK)
hetrd_small_kernel(C* __restrict__ A, const int* __restrict__ nred, int ld, double* __restrict__ dOut,
                   double* __restrict__ eOut, C* __restrict__ tauOut, const int* __restrict__ order) {
  constexpr int NMAX = 4 * NK, NW = NK / 2;
  const int b = order[blockIdx.x], n = nred[b];
  if (n <= 0) return;
  __shared__ __align__(16) C vs[NMAX], ws[NMAX], col[NMAX];
  __shared__ R sNorm[NW], sDot[2 * NW];
  C* Ab = A + (long long)b * ld * ld;
  double *d = dOut + (long long)b * ld, *e = eOut + (long long)b * ld;
  C* taus = tauOut + (long long)b * ld;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, i = tid >> 2, p = tid & 3;
  const C zero = mk(R(0), R(0));
  C a[NK];
  R part = 0;
  // element (i, c) of the next column c: the diagonal to d, the rest to col and the norm of
  // the rows below c + 1
  auto hand_on = [&](int c, C x) {
    if (i == c) d[c] = (double)x.x;
    if (i > c) col[i] = x;
    if (i > c + 1) part = cabs2(x);
  };
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    const int j = p + 4 * k;
    a[k] = zero;
    if (i < n && j <= i) a[k] = Ab[i + (long long)j * ld];
    else if (j < n && i < j) a[k] = cconj(Ab[j + (long long)i * ld]);
    if (j == i) a[k].y = R(0);
    if (j == 0) hand_on(0, a[k]);
  }
  for (int c = 0; c + 1 < n; ++c) {
    part = warp_sum(part);
    if (lane == 0) sNorm[warp] = part;
    __syncthreads();
    R xnorm2 = 0, up = R(1), down = R(1);
#pragma unroll
    for (int w = 0; w < NW; ++w) xnorm2 += sNorm[w];
    C alpha = col[c + 1];
    if (hh_underflows(alpha, xnorm2)) {   // the same in every thread
      up = R(kHhUp), down = R(kHhDown);
      part = warp_sum(p == 0 && i > c + 1 && i < n ? cabs2(cscale(col[i], up)) : R(0));
      __syncthreads();
      if (lane == 0) sNorm[warp] = part;
      __syncthreads();
      xnorm2 = 0;
#pragma unroll
      for (int w = 0; w < NW; ++w) xnorm2 += sNorm[w];
      alpha = cscale(alpha, up);
      if (hh_underflows(alpha, xnorm2)) alpha = zero, xnorm2 = R(0);
    }
    C tau, sc;
    R beta;
    hh_reflector(alpha, xnorm2, tau, sc, beta);
    beta *= down;
    const bool in = i > c && i < n;
    const C v = in ? (i == c + 1 ? mk(R(1), R(0)) : cmul(cscale(col[i], up), sc)) : zero;
    if (p == 0) {
      vs[i] = v;
      if (in) Ab[i + (long long)c * ld] = i == c + 1 ? mk(beta, R(0)) : v;
    }
    if (tid == 0) {
      e[c] = (double)beta;
      taus[c] = tau;
    }
    __syncthreads();
    // y = A v over the trailing block (v is zero outside it)
    C y = zero;
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (4 * k + 3 > c) cfma(y, a[k], vs[p + 4 * k]);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      y.x += __shfl_xor_sync(0xffffffffu, y.x, o);
      y.y += __shfl_xor_sync(0xffffffffu, y.y, o);
    }
    // w = tau y - 1/2 tau ((tau y)^H v) v
    y = cmul(tau, y);
    C dot = p == 0 ? cconjmul(y, v) : zero;
    dot.x = warp_sum(dot.x);
    dot.y = warp_sum(dot.y);
    if (lane == 0) {
      sDot[2 * warp] = dot.x;
      sDot[2 * warp + 1] = dot.y;
    }
    __syncthreads();
    dot = zero;
#pragma unroll
    for (int w = 0; w < NW; ++w) dot = dot + mk(sDot[2 * w], sDot[2 * w + 1]);
    const C wv = in ? y + cmul(cscale(cmul(tau, dot), R(-0.5)), v) : zero;
    if (p == 0) ws[i] = wv;
    __syncthreads();
    // A -= v w^H + w v^H
    part = 0;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      if (4 * k + 3 > c) {
        const int j = p + 4 * k;
        const C vj = vs[j], wj = ws[j];
        a[k].x -= v.x * wj.x + v.y * wj.y + wv.x * vj.x + wv.y * vj.y;
        a[k].y -= v.y * wj.x - v.x * wj.y + wv.y * vj.x - wv.x * vj.y;
        if (j == c + 1) hand_on(c + 1, a[k]);
      }
    }
  }
}

template <typename C, typename R, int NB, int T, int RPT, int CS>
inline void ht_launch_cs(cudaStream_t st, int grid, size_t smem, C* A, const int* nred, int ld, double* d, double* e,
                         C* tau, const int* order, int nb, int nmax) {
  auto k = hetrd_cluster_kernel<C, R, NB, T, RPT, CS>;
  B2_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid * CS);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  count_launch();
  B2_CUDA(cudaLaunchKernelEx(&cfg, k, A, nred, ld, d, e, tau, order, nb, nmax));
}

// Cluster sizes 1 to 8 of one kernel shape. CTAs per matrix double while the batch's CTAs fill
// at most 90 % of the SMs (clusters do not pack every SM; 37 matrices of 333 rows: 2.54 ms at
// 2, 2.91 at 4) and a matrix has 64 rows per CTA (below, the repeated work of a column and the
// cluster barrier cost more than the shared product: 60 rows 0.20 ms at 1, 0.24 at 2); and
// while the lower triangles in flight exceed 8/5 of L2 (64 matrices of 1024 rows: 34.0 ms at
// 2, all 64 in flight, 28.1 at 4; 150 of 1000: 109 and 91; 300 of 768 75 at 2, 85 at 4), as
// long as the batch is at most 3/2 matrices per SM: beyond, one CTA each has the highest rate
// (1024 of 768 rows: 218 ms, 227 at 2, 275 at 4), and larger clusters only even out a last
// wave.
template <typename C, typename R, int NB, int T, int RPT>
inline void ht_launch(cudaStream_t st, int smCount, size_t l2Bytes, C* A, const int* nred, int ld, double* d, double* e,
                      C* tau, const int* order, int nb, int nmax, int most, int grid1) {
  int cs = 1;
  while (cs < most && 128 * cs <= nmax) {
    const double inFlight = std::min<double>(nb, (double)smCount / cs) * 0.5 * nmax * nmax * sizeof(C);
    if (10ll * nb * cs * 2 > 9ll * smCount && (2 * nb > 3 * smCount || inFlight <= 1.6 * l2Bytes)) break;
    cs *= 2;
  }
  const size_t smem = ht_smem<C, NB, T>(nmax, cs > 1);
  const int grid = cs == 1 && grid1 > 0 ? std::min(nb, grid1) : nb;
  if (cs == 1) ht_launch_cs<C, R, NB, T, RPT, 1>(st, grid, smem, A, nred, ld, d, e, tau, order, nb, nmax);
  else if (cs == 2) ht_launch_cs<C, R, NB, T, RPT, 2>(st, grid, smem, A, nred, ld, d, e, tau, order, nb, nmax);
  else if (cs == 4) ht_launch_cs<C, R, NB, T, RPT, 4>(st, grid, smem, A, nred, ld, d, e, tau, order, nb, nmax);
  else ht_launch_cs<C, R, NB, T, RPT, 8>(st, grid, smem, A, nred, ld, d, e, tau, order, nb, nmax);
}

// hetrd.hpp; at most 1024 rows, and the panel has to fit shared memory.
// FP32: panels of 8 up to 512 rows, of 4 above (shared memory holds a row of partial sums per
// warp). 512 threads; 256, two CTAs per SM, up to 256 rows when the batch has several matrices
// per SM (1024 of 256 rows: 8.8 ms against 11.3; 64 of them 1.9 against 1.56). FP64: 256 threads (registers), panels of 8 up to
// 512 rows, of 4 while they fit.
template <typename C, typename R>
bool hetrd_cluster(cudaStream_t st, int smCount, size_t l2Bytes, size_t maxSmem, C* A, const int* nred, int ld,
                          double* d, double* e, C* tau, const int* order, int nb, int nmax, int most, int grid1) {
  // in registers up to 96 rows (16 bytes of FP64 complex: 24 elements a thread are 96 registers)
  if (nmax <= 96) {
    count_launch();
    if (nmax <= 64) hetrd_small_kernel<C, R, 16><<<nb, 256, 0, st>>>(A, nred, ld, d, e, tau, order);
    else hetrd_small_kernel<C, R, 24><<<nb, 384, 0, st>>>(A, nred, ld, d, e, tau, order);
    B2_CHECK_LAUNCH();
    return true;
  }
  if constexpr (sizeof(C) == 8) {
    if (nmax > 1024) return false;
    // of many matrices above 896 rows hetrd_blk_kernel, whose panels hold 8 columns at these
    // sizes too, is the faster one (310 of 1000 rows: 175 ms against 200 here, of 800 rows 91
    // against 86; 200 of 1000 115 against 122, 150 of them 112 against 91)
    if (most == 0 && nmax > 896 && 4 * nb > 5 * smCount) return false;
    const auto k = nmax <= 256 && nb > smCount ? ht_launch<C, R, 8, 256, 1>
                   : nmax <= 512               ? ht_launch<C, R, 8, 512, 1>
                                               : ht_launch<C, R, 4, 512, 2>;
    k(st, smCount, l2Bytes, A, nred, ld, d, e, tau, order, nb, nmax, most ? most : 8, grid1);
  } else {
    if (nmax > 1024 || (nmax > 512 && ht_smem<C, 4, 256>(nmax, true) > maxSmem)) return false;
    const auto k = nmax <= 256   ? ht_launch<C, R, 8, 256, 1>
                   : nmax <= 512 ? ht_launch<C, R, 8, 256, 2>
                                 : ht_launch<C, R, 4, 256, 4>;
    k(st, smCount, l2Bytes, A, nred, ld, d, e, tau, order, nb, nmax, most ? most : 8, grid1);
  }
  return true;
}

}  // namespace bippb200

// Batched Bluebild pipeline: per time step S, antenna positions and wavelength go
// through flagging, Gram, generalized eigensolve, energy-level binning, virtual
// visibilities and the NUFFT, with every stage batched over the steps of a call.
//
// Reference flow (per step, serial on the host): bipp::eigh_gram
// (src/eigensolver.cpp:129-225) -> level selection (python/bipp/filter.py,
// src/image_synthesis.cpp:110-122) -> host::virtual_vis (src/host/virtual_vis.cpp:19-73)
// -> NUFFT add/get (src/nufft_synthesis.cpp:134-169). Here the steps of one call share
// one eigensolver launch sequence per chunk of steps and one NUFFT per call ("batched"
// mode) or run one step and one level at a time ("plain" mode, the straightforward GPU
// form used as the comparison point).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <cmath>
#include <memory>
#include <numeric>
#include <vector>

#include "context.hpp"
#include "eig.hpp"
#include "eig_kernels.cuh"
#include "nufft.hpp"
#include "tune.hpp"
#include "vv_tc.cuh"

namespace bippb200 {

// antenna UVW coordinates U[b][i][c] = sum_k xyz[b][i][k] basis[k][c] (FP64), uvw scale,
// and the per-step range of the w coordinate. xyz layout [b][i][3].
__global__ void antenna_uvw_kernel(int nSteps, int nAnt, const double* __restrict__ xyz, const double* __restrict__ wl,
                                   const double* __restrict__ basis, double* __restrict__ U, double* __restrict__ scale,
                                   double* __restrict__ wrange) {
  const int b = blockIdx.x;
  if (b >= nSteps) return;
  __shared__ double bs[9];
  __shared__ double rmin[32], rmax[32];
  if (threadIdx.x < 9) bs[threadIdx.x] = basis[threadIdx.x];
  __syncthreads();
  double lo = 1e300, hi = -1e300;
  for (int i = threadIdx.x; i < nAnt; i += blockDim.x) {
    const double* p = xyz + ((long long)b * nAnt + i) * 3;
    double u[3];
    for (int c = 0; c < 3; ++c) u[c] = p[0] * bs[0 + 3 * c] + p[1] * bs[1 + 3 * c] + p[2] * bs[2 + 3 * c];
    double* o = U + ((long long)b * nAnt + i) * 3;
    o[0] = u[0];
    o[1] = u[1];
    o[2] = u[2];
    lo = fmin(lo, u[2]);
    hi = fmax(hi, u[2]);
  }
  lo = block_min(lo, rmin, 1e300);
  hi = block_max(hi, rmax, -1e300);
  if (threadIdx.x == 0) {
    const double s = 2.0 * 3.14159265358979323846 / wl[b];
    scale[b] = s;
    wrange[b] = (hi - lo) * s;
  }
}

// xyz [b][i][3] -> [b][3][nAnt] for the Gram computation of the eigensolver
__global__ void xyz_transpose_kernel(long long total, int nAnt, const double* __restrict__ in, double* __restrict__ out) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long b = e / (3ll * nAnt);
    const int r = (int)(e % (3ll * nAnt));
    const int c = r / nAnt, i = r % nAnt;
    out[e] = in[(b * nAnt + i) * 3 + c];
  }
}

__device__ __forceinline__ double filter_value(int f, double d) {
  // python/bipp/filter.py:7-26
  switch (f) {
    case 0: return d;
    case 1: return d > 0 ? 1.0 : (d < 0 ? -1.0 : 0.0);
    case 2: { const double s = d > 0 ? 1.0 : (d < 0 ? -1.0 : 0.0); return s * sqrt(s * d); }
    case 3: return d != 0 ? 1.0 / d : 0.0;
    case 4: { const double s = d > 0 ? 1.0 : (d < 0 ? -1.0 : 0.0); const double r = s * sqrt(s * d); return r != 0 ? 1.0 / r : 0.0; }
  }
  return d;
}

// per step: kscale[b][c] = (1/nVis) filter(d_c); per (step, level) the contiguous range of
// eigenvalue indices with lo <= d <= hi (eigenvalues are ascending)
// Per step and level: the eigenvalue index range [kbeg, kend) of the level (eigenvalues
// ascending) inside the computed range krange = [kLo, kHi) of the eigensolver, and the
// column scales filter(d) / nVis.
__global__ void levels_kernel(int nSteps, int Nmax, int nLevels, const double* __restrict__ intervals, int filt,
                              const int* __restrict__ nred, const long long* __restrict__ nvis,
                              const double* __restrict__ lam, const int* __restrict__ krange,
                              float* __restrict__ kscale, int* __restrict__ kbeg, int* __restrict__ kend) {
  const int b = blockIdx.x;
  if (b >= nSteps) return;
  const int n = nred[b];
  const double sc = nvis[b] ? 1.0 / (double)nvis[b] : 0.0;
  const double* d = lam + (long long)b * Nmax;
  for (int c = threadIdx.x; c < Nmax; c += blockDim.x)
    kscale[(long long)b * Nmax + c] = (c < n && d[c] != 0.0) ? (float)(sc * filter_value(filt, d[c])) : 0.0f;
  if (threadIdx.x < nLevels) {
    const int l = threadIdx.x;
    const double lo = intervals[2 * l], hi = intervals[2 * l + 1];
    const int kLo = krange[2 * b], kHi = krange[2 * b + 1];
    int a = kLo;
    while (a < kHi && d[a] < lo) ++a;
    int e = a;
    while (e < kHi && d[e] <= hi) ++e;
    kbeg[b * nLevels + l] = a;
    kend[b * nLevels + l] = e;
  }
}

__global__ void scale_images_kernel(const float* __restrict__ img, long long n, float s, float* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = img[i] * s;
}

}  // namespace bippb200

using namespace bippb200;

struct bipp_pipeline_s {
  bipp_ctx_s* ctx = nullptr;
  size_t nAnt = 0, nLevels = 0, chunk = 256, maxSteps = 0;
  int filter = 0, mode = 0, vvPrecision = 0;
  double tol = 1e-5;
  long long P = 0;
  std::vector<double> intervals;
  NufftCore core;
  EigWork<float> eig;
  DevBuf basis, intervalsD;
  DevBuf S, xyz, xyzT, wl, antUVW, uvwScale, wrange;
  const float2* Sin = nullptr;   // visibilities of the current call (caller's device memory or S)
  DevBuf idx, nred, nvis, status, lam, kscale, kbeg, kend, vv, pairOff;
  DevBuf images;
  long long stepsDone = 0;
  bool timing = false;
  double stageMs[7] = {0, 0, 0, 0, 0, 0, 0};
  double eigMs[kEigTimers] = {0, 0, 0, 0, 0, 0, 0, 0};
  std::vector<double> lastLam;
  std::vector<int> lastNred;
  // staged host inputs (bipp_pipeline_stage): two slots, copied on their own stream so that
  // the next batch's copy runs while the current one is processed
  struct Staged {
    DevBuf S, xyz, wl;
    size_t steps = 0;
    bool full = false;
    cudaEvent_t copied = nullptr;    // the slot's copy is complete
    cudaEvent_t consumed = nullptr;  // its processing no longer reads the slot
  } staged[2];
  int stageNext = 0, stageHead = 0;
  cudaStream_t copyStream = nullptr;
  ~bipp_pipeline_s() {
    for (auto& st : staged) {
      if (st.copied) cudaEventDestroy(st.copied);
      if (st.consumed) cudaEventDestroy(st.consumed);
    }
    if (copyStream) cudaStreamDestroy(copyStream);
  }
};

static void pipeline_alloc(bipp_pipeline_s* p, size_t steps) {
  bipp_ctx_s* ctx = p->ctx;
  const size_t N = p->nAnt, L = p->nLevels;
  if (steps <= p->maxSteps && p->S.bytes()) return;
  p->maxSteps = std::max(steps, p->maxSteps);
  const size_t T = p->maxSteps;
  p->S.alloc(ctx, T * N * N * sizeof(float2));
  p->xyz.alloc(ctx, T * N * 3 * sizeof(double));
  p->xyzT.alloc(ctx, T * N * 3 * sizeof(double));
  p->wl.alloc(ctx, T * sizeof(double));
  p->antUVW.alloc(ctx, T * N * 3 * sizeof(double));
  p->uvwScale.alloc(ctx, T * sizeof(double));
  p->wrange.alloc(ctx, T * sizeof(double));
  p->idx.alloc(ctx, T * N * sizeof(int));
  p->nred.alloc(ctx, T * sizeof(int));
  p->nvis.alloc(ctx, T * sizeof(long long));
  p->status.alloc(ctx, T * sizeof(int));
  p->lam.alloc(ctx, T * N * sizeof(double));
  p->kscale.alloc(ctx, T * N * sizeof(float));
  p->kbeg.alloc(ctx, T * L * sizeof(int));
  p->kend.alloc(ctx, T * L * sizeof(int));
  p->pairOff.alloc(ctx, (T + 1) * sizeof(long long));
}

// eigensolve + levels + VV for steps [s0, s0+nb) of the call, then scatter their points.
static void pipeline_chunk(bipp_pipeline_s* p, int s0, int nb, const std::vector<long long>& pairOffH,
                           int levelsInTransform, int levelOffset, bool scatterOnly, double* ms) {
  bipp_ctx_s* ctx = p->ctx;
  const int N = (int)p->nAnt, L = (int)p->nLevels;
  const long long n2 = (long long)N * N;
  cudaEvent_t e0, e1, e2;
  if (ms) {
    cudaEventCreate(&e0); cudaEventCreate(&e1); cudaEventCreate(&e2);
    cudaEventRecord(e0, ctx->stream);
  }
  float2* X = p->eig.X(true);
  if (!scatterOnly) {
    EigLaunch<float> E{};
    E.nBatch = nb; E.nBeam = N; E.nAnt = N; E.Nmax = N;
    E.S = p->Sin + (long long)s0 * n2; E.sStride = n2; E.lds = N;
    E.xyz = p->xyzT.get<double>(); E.xyzStride = 3ll * N; E.ldxyz = N; E.wl = p->wl.get<double>();
    E.mode = 0; E.eps = std::numeric_limits<float>::epsilon(); E.gram = true; E.identityW = true;
    E.idx = p->idx.get<int>(); E.nred = p->nred.get<int>(); E.nvis = p->nvis.get<long long>();
    E.status = p->status.get<int>(); E.lam = p->lam.get<double>();
    E.doFlag = 0; E.batchOffset = s0;
    E.kernelMs = ms ? p->eigMs : nullptr;
    // only the eigenvectors inside the energy levels enter the virtual visibilities
    E.vecLo = INFINITY;
    E.vecHi = -INFINITY;
    for (size_t l = 0; l < p->intervals.size() / 2; ++l) {
      E.vecLo = std::min(E.vecLo, p->intervals[2 * l]);
      E.vecHi = std::max(E.vecHi, p->intervals[2 * l + 1]);
    }
    E.allValues = 0;
    eig_launch<float>(ctx, E, p->eig);
    if (ms) cudaEventRecord(e1, ctx->stream);
    count_launch();
    levels_kernel<<<nb, 128, 0, ctx->stream>>>(nb, N, L, p->intervalsD.get<double>(), p->filter, p->nred.get<int>() + s0,
                                               p->nvis.get<long long>() + s0, p->lam.get<double>() + (long long)s0 * N,
                                               p->eig.krange.get<int>(), p->kscale.get<float>() + (long long)s0 * N,
                                               p->kbeg.get<int>() + s0 * L,
                                               p->kend.get<int>() + s0 * L);
    B2_CHECK_LAUNCH();
    // VV[b][l] lower triangle = X diag(kscale) X^H over the level's eigenvalue range
    if (p->vvPrecision == 2) {
      GemmArgs<float2> g{};
      g.A = X; g.strideA = n2; g.lda = N; g.opA = 0;
      g.B = X; g.strideB = n2; g.ldb = N; g.opB = 1;
      g.Cm = p->vv.get<float2>(); g.strideC = n2 * L; g.ldc = N; g.strideCLevel = n2;
      g.n = p->nred.get<int>() + s0; g.outMode = 2; g.levels = L;
      g.kscale = p->kscale.get<float>() + (long long)s0 * N; g.strideK = N;
      g.kbeg = p->kbeg.get<int>() + s0 * L; g.kend = p->kend.get<int>() + s0 * L;
      const int tiles = (N + kGemmBM - 1) / kGemmBM;
      count_launch();
      gemm_kernel<float2, float><<<dim3(tiles, tiles, nb * L), kGemmThreads, 0, ctx->stream>>>(g);
    } else {
      VvArgs v{};
      v.X = X; v.strideX = n2; v.ldx = N;
      v.kscale = p->kscale.get<float>() + (long long)s0 * N; v.strideK = N;
      v.kbeg = p->kbeg.get<int>() + s0 * L; v.kend = p->kend.get<int>() + s0 * L;
      v.n = p->nred.get<int>() + s0;
      v.VV = p->vv.get<float2>(); v.strideStep = n2 * L; v.strideLevel = n2; v.ldv = N;
      v.nSteps = nb; v.nLevels = L;
      v.status = p->status.get<int>() + s0;
      if (p->vvPrecision == 3) {
        const int tiles = (N + kVv64Tile - 1) / kVv64Tile;
        v.tilesI = v.tilesJ = tiles;
        count_launch();
        vv_fp64_kernel<<<dim3(tiles, tiles, nb * L), kVv64Threads, 0, ctx->stream>>>(v);
      } else {
        v.tilesI = (N + kVvM - 1) / kVvM;
        v.tilesJ = (N + kVvNC - 1) / kVvNC;
        const long long items = (long long)nb * L * v.tilesI * v.tilesJ;
        const int grid = (int)std::max<long long>(
            1, std::min<long long>(items, (long long)tuned("vv.ctas_per_sm") * ctx->smCount));
        auto k = p->vvPrecision == 0 ? vv_tc_kernel<1> : vv_tc_kernel<2>;
        smem_optin(k, VvShape<1>::Smem);
        count_launch();
        k<<<grid, kVvThreads, VvShape<1>::Smem, ctx->stream>>>(v);
      }
    }
    B2_CHECK_LAUNCH();
  }
  // zero baselines (r == s) of the levels in this transform
  count_launch();
  vv_trace_kernel<<<nb * levelsInTransform, 128, 0, ctx->stream>>>(
      nb, levelsInTransform, p->nred.get<int>() + s0, p->vv.get<float2>() + (long long)levelOffset * n2, n2 * L, n2, N,
      p->core.zero_acc());
  B2_CHECK_LAUNCH();
  if (ms) cudaEventRecord(e2, ctx->stream);
  // scatter points of these steps
  std::vector<long long> rel(nb + 1);
  for (int i = 0; i <= nb; ++i) rel[i] = pairOffH[s0 + i] - pairOffH[s0];
  DevBuf relD(ctx, (nb + 1) * sizeof(long long));
  h2d(ctx, relD.get(), rel.data(), rel.size() * sizeof(long long));
  PipelinePoints pp{};
  pp.nSteps = nb;
  pp.nred = p->nred.get<int>() + s0;
  pp.idx = p->idx.get<int>() + (long long)s0 * N;
  pp.antUVW = p->antUVW.get<double>() + (long long)s0 * N * 3;
  pp.uvwScale = p->uvwScale.get<double>() + s0;
  pp.Nmax = N;
  pp.nAnt = N;
  pp.vv = p->vv.get<float2>() + (long long)levelOffset * n2;
  pp.vvStepStride = n2 * L;
  pp.vvLevelStride = n2;
  pp.levels = levelsInTransform;
  const long long total = rel[nb];
  if (total > 0) {
    const int gb = (int)std::min<long long>((total + 255) / 256, 16384);
    count_launch();
    pipeline_scatter_kernel<<<gb, 256, 0, ctx->stream>>>(p->core.geom(), pp, total, p->core.cursor(), relD.get<long long>(),
                                                         p->core.points(), p->core.point_bytes(), p->core.point_capacity(),
                                                         p->core.sincos64() ? 1 : 0, p->core.value_max());
    B2_CHECK_LAUNCH();
  }
  if (ms) {
    cudaEvent_t e3;
    cudaEventCreate(&e3);
    cudaEventRecord(e3, ctx->stream);
    cudaEventSynchronize(e3);
    float a = 0, b = 0, c = 0;
    if (!scatterOnly) {
      cudaEventElapsedTime(&a, e0, e1);
      cudaEventElapsedTime(&b, e1, e2);
    }
    cudaEventElapsedTime(&c, e2, e3);
    ms[0] += a;
    ms[1] += b;
    ms[2] += c;
    cudaEventDestroy(e0); cudaEventDestroy(e1); cudaEventDestroy(e2); cudaEventDestroy(e3);
  }
}

static void pipeline_count(bipp_pipeline_s* p, int s0, int nb, const std::vector<long long>& pairOffH) {
  bipp_ctx_s* ctx = p->ctx;
  const int N = (int)p->nAnt;
  std::vector<long long> rel(nb + 1);
  for (int i = 0; i <= nb; ++i) rel[i] = pairOffH[s0 + i] - pairOffH[s0];
  DevBuf relD(ctx, (nb + 1) * sizeof(long long));
  h2d(ctx, relD.get(), rel.data(), rel.size() * sizeof(long long));
  PipelinePoints pp{};
  pp.nSteps = nb;
  pp.nred = p->nred.get<int>() + s0;
  pp.idx = p->idx.get<int>() + (long long)s0 * N;
  pp.antUVW = p->antUVW.get<double>() + (long long)s0 * N * 3;
  pp.uvwScale = p->uvwScale.get<double>() + s0;
  pp.Nmax = N;
  pp.nAnt = N;
  const long long total = rel[nb];
  if (total > 0) {
    const int gb = (int)std::min<long long>((total + 255) / 256, 16384);
    count_launch();
    pipeline_count_kernel<<<gb, 256, 0, ctx->stream>>>(p->core.geom(), pp, total, p->core.counts(), relD.get<long long>());
    B2_CHECK_LAUNCH();
  }
  sync(ctx);
}

// Host visibilities to the device: only the lower triangle of each S is read, so it is
// copied as blocks of 64 columns from each block's diagonal row down, one 3-D copy per
// block over all steps (about 56 % of the bytes of the full matrices at 512 antennas).
constexpr int kLowerCopyCols = 64;
static void copy_lower_blocks(cudaStream_t st, float2* dst, const float2* src, int N, int T) {
  for (int c0 = 0; c0 < N; c0 += kLowerCopyCols) {
    const int w = std::min(kLowerCopyCols, N - c0);
    cudaMemcpy3DParms prm = {};
    prm.srcPtr = make_cudaPitchedPtr(const_cast<float2*>(src), (size_t)N * sizeof(float2), N, N);
    prm.dstPtr = make_cudaPitchedPtr(dst, (size_t)N * sizeof(float2), N, N);
    prm.srcPos = make_cudaPos((size_t)c0 * sizeof(float2), (size_t)c0, 0);
    prm.dstPos = prm.srcPos;
    prm.extent = make_cudaExtent((size_t)(N - c0) * sizeof(float2), (size_t)w, (size_t)T);
    prm.kind = cudaMemcpyHostToDevice;
    B2_CUDA(cudaMemcpy3DAsync(&prm, st));
  }
}

// Status words of steps [s0, s0 + nb) after their eigensolve: a failed step ends the call
// before anything is added to the images (the reference throws at the failing step,
// src/host/lapack_api.hpp:133, before its NUFFT update).
static void check_steps(bipp_pipeline_s* p, int s0, int nb) {
  std::vector<int> st(nb);
  d2h(p->ctx, st.data(), p->status.get<int>() + s0, nb * sizeof(int));
  sync(p->ctx);
  for (int b = 0; b < nb; ++b) {
    if (st[b] & kStatusTensorTimeout) throw Error(BIPP_GPU_ERROR, "tensor-core MMA wait timed out");
    if (st[b] & kStatusCholeskyNotPD) throw Error(BIPP_EIGENSOLVER_ERROR, "Gram matrix is not positive definite");
    if (st[b] & kStatusNonFinite) throw Error(BIPP_EIGENSOLVER_ERROR, "non-finite visibility in a kept entry of S");
  }
}

static void pipeline_process(bipp_pipeline_s* p, size_t nSteps, const void* s, const double* xyz, const double* wl,
                             int onDevice) {
  bipp_ctx_s* ctx = p->ctx;
  require(nSteps > 0, "no steps");
  require(s && xyz && wl, "null pointer", BIPP_INVALID_POINTER_ERROR);
  pipeline_alloc(p, nSteps);
  const int N = (int)p->nAnt, L = (int)p->nLevels;
  const long long n2 = (long long)N * N;
  const int T = (int)nSteps;
  cudaEvent_t ev0, ev1;
  if (p->timing) { cudaEventCreate(&ev0); cudaEventCreate(&ev1); cudaEventRecord(ev0, ctx->stream); }
  // inputs
  const cudaMemcpyKind kind = onDevice ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  // device inputs are read in place; host inputs are staged in S
  if (onDevice) {
    p->Sin = static_cast<const float2*>(s);
  } else {
    copy_lower_blocks(ctx->stream, p->S.get<float2>(), static_cast<const float2*>(s), N, T);
    p->Sin = p->S.get<float2>();
  }
  B2_CUDA(cudaMemcpyAsync(p->xyz.get(), xyz, (size_t)T * N * 3 * sizeof(double), kind, ctx->stream));
  B2_CUDA(cudaMemcpyAsync(p->wl.get(), wl, (size_t)T * sizeof(double), kind, ctx->stream));
  count_launch();
  antenna_uvw_kernel<<<T, 256, 0, ctx->stream>>>(T, N, p->xyz.get<double>(), p->wl.get<double>(), p->basis.get<double>(),
                                                 p->antUVW.get<double>(), p->uvwScale.get<double>(),
                                                 p->wrange.get<double>());
  count_launch();
  xyz_transpose_kernel<<<1024, 256, 0, ctx->stream>>>((long long)T * 3 * N, N, p->xyz.get<double>(), p->xyzT.get<double>());
  p->status.zero();
  // flags for every step
  {
    const size_t smem = 2 * (size_t)N * sizeof(int);
    auto k = prep_kernel<float>;
    smem_optin(k, smem);
    count_launch();
    k<<<T, kPrepThreads, smem, ctx->stream>>>(N, p->Sin, n2, N, p->xyzT.get<double>(), 3ll * N, N,
                                              p->wl.get<double>(), 0, std::numeric_limits<float>::epsilon(), 1, N,
                                              p->idx.get<int>(), p->nred.get<int>(), p->nvis.get<long long>(),
                                              nullptr, nullptr, p->status.get<int>(), 0, 0);
    B2_CHECK_LAUNCH();
  }
  std::vector<int> nredH(T);
  std::vector<double> wr(T);
  d2h(ctx, nredH.data(), p->nred.get(), T * sizeof(int));
  d2h(ctx, wr.data(), p->wrange.get(), T * sizeof(double));
  sync(ctx);
  if (p->timing) {
    cudaEventRecord(ev1, ctx->stream);
    cudaEventSynchronize(ev1);
    float a;
    cudaEventElapsedTime(&a, ev0, ev1);
    p->stageMs[2] += a;
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
  }
  std::vector<long long> pairOff(T + 1, 0);
  for (int b = 0; b < T; ++b) pairOff[b + 1] = pairOff[b] + (long long)nredH[b] * (nredH[b] + 1) / 2;
  double Xw = 0;
  for (int b = 0; b < T; ++b) Xw = std::max(Xw, wr[b]);
  const int chunk = (int)p->chunk;
  p->eig.reserve(ctx, std::min(chunk, T), N);
  p->vv.ensure(ctx, (size_t)std::min(chunk, T) * L * n2 * sizeof(float2));
  double* ms = p->timing ? p->stageMs : nullptr;

  if (p->mode == 0) {
    // batched: one NUFFT over all steps of the call, all levels as channels
    p->core.begin(0.0, Xw);  // points are folded to w >= 0 (real image)
    for (int s0 = 0; s0 < T; s0 += chunk) pipeline_count(p, s0, std::min(chunk, T - s0), pairOff);
    p->core.end_count(pairOff[T]);
    for (int s0 = 0; s0 < T; s0 += chunk) pipeline_chunk(p, s0, std::min(chunk, T - s0), pairOff, L, 0, false, ms);
    check_steps(p, 0, T);
    double nm[4] = {0, 0, 0, 0};
    p->core.execute(p->images.get<float>(), p->P, p->timing ? nm : nullptr);
    p->stageMs[3] += nm[0];
    p->stageMs[4] += nm[1];
    p->stageMs[5] += nm[2];
    p->stageMs[6] += nm[3];
  } else {
    // plain: one step at a time, one NUFFT per step and level
    for (int b = 0; b < T; ++b) {
      for (int l = 0; l < L; ++l) {
        p->core.begin(0.0, wr[b]);
        pipeline_count(p, b, 1, pairOff);
        p->core.end_count(pairOff[b + 1] - pairOff[b]);
        pipeline_chunk(p, b, 1, pairOff, 1, l, l > 0, ms);
        if (l == 0) check_steps(p, b, 1);
        double nm[4] = {0, 0, 0, 0};
        p->core.execute(p->images.get<float>() + (long long)l * p->P, p->P, p->timing ? nm : nullptr);
        p->stageMs[3] += nm[0];
        p->stageMs[4] += nm[1];
        p->stageMs[5] += nm[2];
        p->stageMs[6] += nm[3];
      }
    }
  }
  // keep eigenvalues of this call for calibration (host copy on demand)
  p->lastNred = nredH;
  p->stepsDone += T;
  sync(ctx);
}

extern "C" {

BippError bipp_pipeline_create(bipp_ctx_t ctx, const bipp_pipeline_config* cfg, bipp_pipeline_t* out) {
  return guard([&] {
    require(ctx && cfg && out, "null pointer", BIPP_INVALID_POINTER_ERROR);
    require(cfg->nAntenna > 0 && cfg->nAntenna <= 4096, "nAntenna must be in [1, 4096]");
    require(cfg->nLevels >= 1 && cfg->nLevels <= (size_t)kMaxPipelineLevels, "nLevels must be in [1, 8]");
    require(cfg->intervals && cfg->pixelN && cfg->uvwBasis, "null pointer", BIPP_INVALID_POINTER_ERROR);
    require(cfg->gridA >= 2 && cfg->gridB >= 2, "pixel lattice must be at least 2 x 2");
    require(cfg->filter >= 0 && cfg->filter <= 4, "unknown filter");
    for (size_t l = 0; l < cfg->nLevels; ++l)
      require(cfg->intervals[2 * l] <= cfg->intervals[2 * l + 1], "energy-level interval with lo > hi or NaN bounds");
    auto p = std::make_unique<bipp_pipeline_s>();
    p->ctx = ctx;
    p->nAnt = cfg->nAntenna;
    p->nLevels = cfg->nLevels;
    p->chunk = cfg->chunkSteps ? cfg->chunkSteps : 256;
    p->filter = cfg->filter;
    p->mode = cfg->mode;
    require(cfg->vvPrecision >= 0 && cfg->vvPrecision <= 3, "unknown virtual-visibility precision");
    p->vvPrecision = cfg->vvPrecision;
    p->tol = cfg->tolerance > 0 ? cfg->tolerance : 1e-5;
    p->intervals.assign(cfg->intervals, cfg->intervals + 2 * cfg->nLevels);
    Lattice lat;
    lat.ok = true;
    lat.Na = (int)cfg->gridA;
    lat.Nb = (int)cfg->gridB;
    lat.l0 = cfg->lattice[0]; lat.m0 = cfg->lattice[1];
    lat.Al = cfg->lattice[2]; lat.Bl = cfg->lattice[3];
    lat.Am = cfg->lattice[4]; lat.Bm = cfg->lattice[5];
    p->P = (long long)cfg->gridA * cfg->gridB;
    std::vector<double> n(cfg->pixelN, cfg->pixelN + p->P);
    p->core.setup(ctx, lat, n, p->tol, p->mode == 0 ? (int)cfg->nLevels : 1);
    p->basis.alloc(ctx, 9 * sizeof(double));
    h2d(ctx, p->basis.get(), cfg->uvwBasis, 9 * sizeof(double));
    p->intervalsD.alloc(ctx, p->intervals.size() * sizeof(double));
    h2d(ctx, p->intervalsD.get(), p->intervals.data(), p->intervals.size() * sizeof(double));
    p->images.alloc(ctx, (size_t)cfg->nLevels * p->P * sizeof(float));
    p->images.zero();
    if (cfg->maxSteps) pipeline_alloc(p.get(), cfg->maxSteps);
    sync(ctx);
    ctx_retain(ctx);
    *out = p.release();
  });
}

BippError bipp_pipeline_process(bipp_pipeline_t pl, size_t nSteps, const void* s, const double* xyz, const double* wl,
                                int onDevice) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    pipeline_process(pl, nSteps, s, xyz, wl, onDevice);
  });
}

BippError bipp_pipeline_stage(bipp_pipeline_t pl, size_t nSteps, const void* s, const double* xyz, const double* wl) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    require(s && xyz && wl, "null pointer", BIPP_INVALID_POINTER_ERROR);
    require(nSteps > 0, "no steps");
    bipp_ctx_s* ctx = pl->ctx;
    auto& slot = pl->staged[pl->stageNext];
    require(!slot.full, "both staging slots hold unprocessed batches; process one first");
    const int N = (int)pl->nAnt;
    if (!pl->copyStream) B2_CUDA(cudaStreamCreateWithFlags(&pl->copyStream, cudaStreamNonBlocking));
    if (!slot.copied) {
      B2_CUDA(cudaEventCreateWithFlags(&slot.copied, cudaEventDisableTiming));
      B2_CUDA(cudaEventCreateWithFlags(&slot.consumed, cudaEventDisableTiming));
      B2_CUDA(cudaEventRecord(slot.consumed, ctx->stream));
    }
    const size_t sB = nSteps * (size_t)N * N * sizeof(float2), xB = nSteps * (size_t)N * 3 * sizeof(double),
                 wB = nSteps * sizeof(double);
    if (slot.S.bytes() < sB || slot.xyz.bytes() < xB || slot.wl.bytes() < wB) {
      slot.S.ensure(ctx, sB);
      slot.xyz.ensure(ctx, xB);
      slot.wl.ensure(ctx, wB);
      sync(ctx);   // the slot's buffers exist before the copy stream writes them
    }
    // the previous batch of this slot must have been read before it is overwritten
    B2_CUDA(cudaStreamWaitEvent(pl->copyStream, slot.consumed, 0));
    copy_lower_blocks(pl->copyStream, slot.S.get<float2>(), static_cast<const float2*>(s), N, (int)nSteps);
    B2_CUDA(cudaMemcpyAsync(slot.xyz.get(), xyz, nSteps * (size_t)N * 3 * sizeof(double), cudaMemcpyHostToDevice,
                            pl->copyStream));
    B2_CUDA(cudaMemcpyAsync(slot.wl.get(), wl, nSteps * sizeof(double), cudaMemcpyHostToDevice, pl->copyStream));
    B2_CUDA(cudaEventRecord(slot.copied, pl->copyStream));
    slot.steps = nSteps;
    slot.full = true;
    pl->stageNext ^= 1;
  });
}

BippError bipp_pipeline_process_staged(bipp_pipeline_t pl) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    auto& slot = pl->staged[pl->stageHead];
    require(slot.full, "no staged batch (bipp_pipeline_stage)");
    bipp_ctx_s* ctx = pl->ctx;
    B2_CUDA(cudaStreamWaitEvent(ctx->stream, slot.copied, 0));
    slot.full = false;
    pl->stageHead ^= 1;
    struct Release {
      bipp_ctx_s* c;
      cudaEvent_t e;
      ~Release() { cudaEventRecord(e, c->stream); }
    } release{ctx, slot.consumed};
    pipeline_process(pl, slot.steps, slot.S.get(), slot.xyz.get<double>(), slot.wl.get<double>(), 1);
  });
}

BippError bipp_pipeline_images(bipp_pipeline_t pl, float* images, int normalize, int onDevice) {
  return guard([&] {
    require(pl && images, "null pointer", BIPP_INVALID_POINTER_ERROR);
    bipp_ctx_s* ctx = pl->ctx;
    const long long n = (long long)pl->nLevels * pl->P;
    if (normalize && pl->stepsDone > 0) {
      // one pass from the accumulated images to the caller's, or piece by piece through the
      // transform's accumulators, idle here, so that images on the host need no more memory
      // on the device
      const float scale = 1.0f / (float)pl->stepsDone;
      const long long piece = onDevice ? n : std::min(n, pl->core.scratch_floats());
      for (long long i = 0; i < n; i += piece) {
        const long long m = std::min(piece, n - i);
        float* out = onDevice ? images : pl->core.scratch();
        count_launch();
        scale_images_kernel<<<2048, 256, 0, ctx->stream>>>(pl->images.get<float>() + i, m, scale, out);
        B2_CHECK_LAUNCH();
        if (!onDevice) d2h(ctx, images + i, out, m * sizeof(float));
      }
    } else {
      B2_CUDA(cudaMemcpyAsync(images, pl->images.get(), n * sizeof(float),
                              onDevice ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, ctx->stream));
    }
    sync(ctx);
  });
}

BippError bipp_autotune_pipeline(bipp_pipeline_t pl, size_t nSteps, const void* s, const double* xyz,
                                 const double* wl, int onDevice, int repeats, char* report, size_t reportLen) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    require(repeats >= 1 && repeats <= 100, "repeats must be in [1, 100]");
    bipp_ctx_s* ctx = pl->ctx;
    // the caller's images, step count and timers are kept aside and restored afterwards
    const size_t imgBytes = (size_t)pl->nLevels * pl->P * sizeof(float);
    DevBuf saved(ctx, imgBytes);
    B2_CUDA(cudaMemcpyAsync(saved.get(), pl->images.get(), imgBytes, cudaMemcpyDeviceToDevice, ctx->stream));
    const long long stepsDone = pl->stepsDone;
    double stage[7], eigt[kEigTimers];
    std::copy(pl->stageMs, pl->stageMs + 7, stage);
    std::copy(pl->eigMs, pl->eigMs + kEigTimers, eigt);
    const bool timing = pl->timing;
    pl->timing = false;
    std::string rep = "{";
    const char* params[] = {"spread.items_cap", "spread.operands", "spread.stages", "spread.ctas_per_sm", "spread.schedule",
                            "hetrd.threads", "hetrd.ctas_pct", "tridiag.threads", "vv.ctas_per_sm"};
    // Objective of a parameter: the device time of the stage it changes (CUDA events of
    // the pipeline's stage timers): spreading (with the tile clearing) for spread.*, the
    // tridiagonalisation kernel for hetrd.*, the virtual visibilities for vv.*. Every
    // candidate gets one untimed call; the timed calls then go over the candidates
    // forwards and backwards in turn (a drift of the device's speed during the pass hits
    // every candidate alike) and the fastest call of each candidate counts.
    auto objective = [&](const char* name) {
      if (!std::strncmp(name, "spread.", 7)) return pl->stageMs[3] + pl->stageMs[6];
      if (!std::strncmp(name, "hetrd.", 6)) return pl->eigMs[4];
      if (!std::strncmp(name, "tridiag.", 8)) return pl->eigMs[5];
      return pl->stageMs[1];
    };
    // the whole call with a set of values: the faster of two timed calls (CUDA events)
    auto whole_call_ms = [&](const std::vector<int>& vals) {
      for (size_t i = 0; i < vals.size(); ++i) set_tuned(params[i], vals[i]);
      cudaEvent_t a, b;
      B2_CUDA(cudaEventCreate(&a));
      B2_CUDA(cudaEventCreate(&b));
      float best = 0.f;
      for (int r = 0; r < 2; ++r) {
        B2_CUDA(cudaEventRecord(a, ctx->stream));
        pipeline_process(pl, nSteps, s, xyz, wl, onDevice);
        B2_CUDA(cudaEventRecord(b, ctx->stream));
        B2_CUDA(cudaEventSynchronize(b));
        float t = 0.f;
        B2_CUDA(cudaEventElapsedTime(&t, a, b));
        best = r ? std::min(best, t) : t;
      }
      cudaEventDestroy(a);
      cudaEventDestroy(b);
      return (double)best;
    };
    const size_t nParams = sizeof(params) / sizeof(params[0]);
    std::vector<int> startVals(nParams);
    for (size_t i = 0; i < nParams; ++i) startVals[i] = tuned(params[i]);
    auto body = [&] {
      pipeline_process(pl, nSteps, s, xyz, wl, onDevice);   // warm-up (allocations, first-use costs)
      bool first = true;
      for (const char* name : params) {
        if (!std::strcmp(name, "vv.ctas_per_sm") && (pl->vvPrecision == 2 || pl->vvPrecision == 3)) continue;
        const std::vector<int> cands = tuning_candidates(name);
        std::vector<double> best(cands.size(), 0.0);
        for (size_t i = 0; i < cands.size(); ++i) {
          set_tuned(name, cands[i]);
          pipeline_process(pl, nSteps, s, xyz, wl, onDevice);
        }
        pl->timing = true;
        for (int r = 0; r < std::max(2, repeats); ++r) {
          for (size_t j = 0; j < cands.size(); ++j) {
            const size_t i = (r & 1) ? cands.size() - 1 - j : j;
            set_tuned(name, cands[i]);
            std::fill(pl->stageMs, pl->stageMs + 7, 0.0);
            std::fill(pl->eigMs, pl->eigMs + kEigTimers, 0.0);
            pipeline_process(pl, nSteps, s, xyz, wl, onDevice);
            const double t = objective(name);
            best[i] = (r == 0) ? t : std::min(best[i], t);
          }
        }
        pl->timing = false;
        size_t bi = 0;
        for (size_t i = 1; i < cands.size(); ++i)
          if (best[i] < best[bi]) bi = i;
        set_tuned(name, cands[bi]);
        rep += std::string(first ? "" : ", ") + "\"" + name + "\": {";
        first = false;
        for (size_t i = 0; i < cands.size(); ++i) {
          char buf[64];
          std::snprintf(buf, sizeof(buf), "%s\"%d\": %.3f", i ? ", " : "", cands[i], best[i]);
          rep += buf;
        }
        char buf[64];
        std::snprintf(buf, sizeof(buf), ", \"chosen\": %d}", cands[bi]);
        rep += buf;
      }
      // a value can speed up its own stage and slow the call down elsewhere: the tuned set
      // is kept only if the whole call is not slower than with the starting values
      std::vector<int> tunedVals(nParams);
      for (size_t i = 0; i < nParams; ++i) tunedVals[i] = tuned(params[i]);
      pl->timing = false;
      const double t1 = whole_call_ms(tunedVals), s1 = whole_call_ms(startVals);
      const double s2 = whole_call_ms(startVals), t2 = whole_call_ms(tunedVals);
      const double tMs = std::min(t1, t2), sMs = std::min(s1, s2);
      const bool keep = tMs <= sMs;
      if (!keep)
        for (size_t i = 0; i < nParams; ++i) set_tuned(params[i], startVals[i]);
      char buf[160];
      std::snprintf(buf, sizeof(buf), ", \"whole_call_ms\": {\"tuned\": %.3f, \"starting\": %.3f, \"kept\": \"%s\"}",
                    tMs, sMs, keep ? "tuned" : "starting");
      rep += buf;
    };
    // the caller's state comes back on every exit path
    auto restore = [&] {
      cudaMemcpyAsync(pl->images.get(), saved.get(), imgBytes, cudaMemcpyDeviceToDevice, ctx->stream);
      pl->stepsDone = stepsDone;
      std::copy(stage, stage + 7, pl->stageMs);
      std::copy(eigt, eigt + kEigTimers, pl->eigMs);
      pl->timing = timing;
      cudaStreamSynchronize(ctx->stream);
    };
    try {
      body();
    } catch (...) {
      restore();
      throw;
    }
    restore();
    rep += "}";
    if (report && reportLen) {
      const size_t n = std::min(reportLen - 1, rep.size());
      std::memcpy(report, rep.data(), n);
      report[n] = '\0';
    }
  });
}

BippError bipp_pipeline_reset(bipp_pipeline_t pl) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    pl->images.zero();
    pl->stepsDone = 0;
    for (double& x : pl->stageMs) x = 0;
    for (double& x : pl->eigMs) x = 0;
    sync(pl->ctx);
  });
}

BippError bipp_pipeline_last_eigenvalues(bipp_pipeline_t pl, double* d, int* nReduced) {
  return guard([&] {
    require(pl && d && nReduced, "null pointer", BIPP_INVALID_POINTER_ERROR);
    const size_t T = pl->lastNred.size();
    d2h(pl->ctx, d, pl->lam.get(), T * pl->nAnt * sizeof(double));
    sync(pl->ctx);
    for (size_t b = 0; b < T; ++b) {
      nReduced[b] = pl->lastNred[b];
      for (size_t c = pl->lastNred[b]; c < pl->nAnt; ++c) d[b * pl->nAnt + c] = 0.0;
    }
  });
}

BippError bipp_pipeline_stage_times(bipp_pipeline_t pl, int enable, double* ms) {
  return guard([&] {
    require(pl != nullptr, "null pipeline", BIPP_INVALID_HANDLE_ERROR);
    if (enable >= 0) pl->timing = enable != 0;
    if (ms)
      for (int i = 0; i < 7; ++i) ms[i] = pl->stageMs[i];
  });
}

BippError bipp_pipeline_nufft_stats(bipp_pipeline_t pl, long long* stats) {
  return guard([&] {
    require(pl && stats, "null pointer", BIPP_INVALID_POINTER_ERROR);
    const NufftGeom& g = pl->core.geom();
    stats[0] = pl->core.lastPoints;
    stats[1] = pl->core.lastSlabs;
    stats[2] = pl->core.lastGridBytes;
    stats[3] = pl->core.lastItems;
    stats[4] = g.nx;
    stats[5] = g.ny;
    stats[6] = g.nw;
    stats[7] = g.W;
    stats[8] = pl->core.lastSplitTiles;
  });
}

BippError bipp_pipeline_kernel_times(bipp_pipeline_t pl, double* ms) {
  return guard([&] {
    require(pl && ms, "null pointer", BIPP_INVALID_POINTER_ERROR);
    for (int i = 0; i < kEigTimers; ++i) ms[i] = pl->eigMs[i];
  });
}

BippError bipp_pipeline_destroy(bipp_pipeline_t pl) {
  return guard([&] {
    if (!pl) return;
    bipp_ctx_s* ctx = pl->ctx;
    delete pl;
    sync(ctx);
    ctx_release(ctx);
  });
}

}  // extern "C"

// qr.cu — orthonormal basis of the fixed-effects design, and the phenotype's projection, in FP64.
//
// Column-pivoted Householder QR of A = rr∘X (n×c; the reference uses Eigen's ColPivHouseholderQR,
// src/reml.cpp:583-588): at most a few dozen columns, so a column step is one dot product with every
// column on its right, one update of them (which also measures what is left of them, the next
// pivot's norms), and the basis one dot product and one update per step backwards.  One cluster of 16
// blocks takes all steps in one launch: columns stay in L2, a step's numbers go through distributed
// shared memory.  Bound by the FP64 units of its 16 SMs (two lanes a clock each) from some 100,000 rows
// on, by its 3c cluster-wide reductions below.  On the host the factorisation, the forming of A and
// of the FP32 copies were 0.75 ms of an MC-REML fit's 4.52 ms at n = 50,000 with 3 covariates and 0.5 of
// the REML gradient's 5.16 ms with 2, the GPU idle meanwhile; the calls took 3.95 and 4.63 ms with it, and
// slemm_gwa at n = 50,021 with 2 covariates 3.78 (4.00).
#include "qr.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

namespace slemm {

namespace cg = cooperative_groups;

constexpr int kQrBlocks = 16, kQrThreads = 512, kQrWarps = kQrThreads / 32;

struct QrShared {
  double warp[kQrWarps][SLEMM_MAX_COVARIATES];
  double part[2][SLEMM_MAX_COVARIATES];   // the block's sums, read by the others; two turns
  double tot[SLEMM_MAX_COVARIATES];
};

// tot[j] = Σ over the cluster's threads of their v(j), j < cnt, by one order of additions.  A block writes
// part[turn] again two turns later, after a cluster barrier that every block reaches with its reads done.
template <class V>
__device__ __forceinline__ void cluster_sums(QrShared& S, int& turn, int cnt, V v)
{
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = 0; j < cnt; ++j) {
    double x = v(j);
    for (int o = 16; o; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) S.warp[warp][j] = x;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < cnt; j += kQrThreads) {
    double x = 0.0;
    for (int w = 0; w < kQrWarps; ++w) x += S.warp[w][j];
    S.part[turn][j] = x;
  }
  cl.sync();   // and what the threads wrote to A and Q is seen by all of them
  for (int j = threadIdx.x; j < cnt; j += kQrThreads) {
    double x = 0.0;
    for (int b = 0; b < kQrBlocks; ++b) x += cl.map_shared_rank(S.part[turn], b)[j];
    S.tot[j] = x;
  }
  __syncthreads();
  turn ^= 1;
}

// head: [0] a covariate is not finite, [1 …] R·Pᵀ (c×c: columns in X's order), [1 + c² …] the columns' pivot order.
__global__ void __launch_bounds__(kQrThreads, 1)
qr_kernel(const float* __restrict__ X, const float* __restrict__ rr, int64_t n, int c, double* A, double* Q, double* head)
{
  __shared__ QrShared S;
  __shared__ int perm[SLEMM_MAX_COVARIATES];
  __shared__ double tau[SLEMM_MAX_COVARIATES];
  cg::cluster_group cl = cg::this_cluster();
  const int64_t t0 = (int64_t)cl.block_rank() * kQrThreads + threadIdx.x, step = (int64_t)kQrBlocks * kQrThreads;
  const bool first = t0 == 0;
  int turn = 0;
  bool bad = false;
  if ((int)threadIdx.x < c) perm[threadIdx.x] = threadIdx.x;
  cluster_sums(S, turn, c, [&](int j) {
    double s = 0.0;
    for (int64_t i = t0; i < n; i += step) {
      const float x = X[(int64_t)j * n + i];
      bad = bad || !isfinite(x);
      const double a = (double)__fmul_rn(rr[i], x);
      A[(int64_t)j * n + i] = a;
      s = fma(a, a, s);
    }
    return s;
  });
  if (__syncthreads_or(bad) && threadIdx.x == 0) head[0] = 1.0;
  const int kmax = (int)min64(n, c);
  for (int k = 0; k < kmax; ++k) {
    // pivot: the largest remaining column, tot[j] = its rows k … squared (j from k, in pivot order)
    int p = k;
    double best = -1.0;
    for (int j = k; j < c; ++j)
      if (S.tot[j - k] > best) {
        best = S.tot[j - k];
        p = j;
      }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int q = perm[k];
      perm[k] = perm[p];
      perm[p] = q;
    }
    __syncthreads();
    double* a = A + (int64_t)perm[k] * n;
    const double nrm = sqrt(best), ak = a[k];
    if (nrm == 0.0) {   // every remaining column is 0 from row k on
      if (threadIdx.x == 0) tau[k] = 0.0;
      if (first)
        for (int j = k; j < c; ++j) head[1 + (int64_t)perm[j] * c + k] = A[(int64_t)perm[j] * n + k];
      continue;   // and so are the norms of the next step
    }
    const double alpha = ak >= 0.0 ? -nrm : nrm;
    const double r0 = 1.0 / (ak - alpha);
    const double tk = (nrm + fabs(ak)) / nrm;   // 2/(vᵀv) of v = [1, a_i/(a_k − α)]
    if (threadIdx.x == 0) tau[k] = tk;
    if (first) head[1 + (int64_t)perm[k] * c + k] = alpha;
    for (int64_t i = t0; i < n; i += step)
      if (i > k) a[i] *= r0;
    const int rest = c - k - 1;
    if (rest == 0) break;
    cluster_sums(S, turn, rest, [&](int q) {
      const double* b = A + (int64_t)perm[k + 1 + q] * n;
      double s = 0.0;
      for (int64_t i = t0; i < n; i += step)
        if (i > k) s = fma(a[i], b[i], s);
      return s;
    });
    const double* tot = S.tot;
    if (cl.block_rank() == 0)
      for (int q = threadIdx.x; q < rest; q += kQrThreads) {
        const double bk = A[(int64_t)perm[k + 1 + q] * n + k];
        head[1 + (int64_t)perm[k + 1 + q] * c + k] = bk - (bk + tot[q]) * tk;
      }
    cluster_sums(S, turn, rest, [&](int q) {
      double* b = A + (int64_t)perm[k + 1 + q] * n;
      const double f = (b[k] + tot[q]) * tk;
      double s = 0.0;
      for (int64_t i = t0; i < n; i += step)
        if (i > k) {
          const double v = fma(-f, a[i], b[i]);
          b[i] = v;
          s = fma(v, v, s);
        }
      return s;
    });
  }
  __syncthreads();
  if (cl.block_rank() == 0 && (int)threadIdx.x < c) head[1 + (int64_t)c * c + threadIdx.x] = perm[threadIdx.x];
  // Q = H_0 … H_{kmax−1}·I: column j has rows k … only once H_k has been applied
  for (int k = kmax - 1; k >= 0; --k) {
    const double* v = A + (int64_t)perm[k] * n;
    const double tk = tau[k];
    const int rest = kmax - 1 - k;
    if (rest > 0 && tk != 0.0) {
      cluster_sums(S, turn, rest, [&](int q) {
        const double* b = Q + (int64_t)(k + 1 + q) * n;
        double s = 0.0;
        for (int64_t i = t0; i < n; i += step)
          if (i > k) s = fma(v[i], b[i], s);
        return s;
      });
      for (int q = 0; q < rest; ++q) {
        double* b = Q + (int64_t)(k + 1 + q) * n;
        const double f = S.tot[q] * tk;
        for (int64_t i = t0; i < n; i += step)
          if (i >= k) b[i] = i > k ? fma(-f, v[i], b[i]) : -f;
      }
      __syncthreads();   // tot is read
    }
    double* b = Q + (int64_t)k * n;
    for (int64_t i = t0; i < n; i += step) b[i] = i > k ? (tk == 0.0 ? 0.0 : -tk * v[i]) : i == k ? 1.0 - tk : 0.0;
  }
  cl.sync();   // no block leaves while another reads its sums
}

// out = (I − QQᵀ)(rr∘y), column by column of Q, times rr if `scale`.
__global__ void __launch_bounds__(kQrThreads, 1)
qr_project_kernel(const double* __restrict__ Q, const float* __restrict__ rr, const float* __restrict__ y, int64_t n, int c,
                  double* v, float* __restrict__ out, int scale)
{
  __shared__ QrShared S;
  cg::cluster_group cl = cg::this_cluster();
  const int64_t t0 = (int64_t)cl.block_rank() * kQrThreads + threadIdx.x, step = (int64_t)kQrBlocks * kQrThreads;
  int turn = 0;
  for (int64_t i = t0; i < n; i += step) v[i] = (double)__fmul_rn(rr[i], y[i]);
  for (int l = 0; l < c; ++l) {
    const double* q = Q + (int64_t)l * n;
    cluster_sums(S, turn, 1, [&](int) {
      double s = 0.0;
      for (int64_t i = t0; i < n; i += step) s = fma(q[i], v[i], s);
      return s;
    });
    const double s = S.tot[0];
    for (int64_t i = t0; i < n; i += step) v[i] = fma(-s, q[i], v[i]);
    __syncthreads();
  }
  for (int64_t i = t0; i < n; i += step) out[i] = scale ? __fmul_rn(rr[i], (float)v[i]) : (float)v[i];
  cl.sync();
}

__global__ void qr_store_kernel(const double* __restrict__ Q, int64_t n, float* __restrict__ out, int64_t ld, int64_t rows)
{
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < rows) out[(int64_t)blockIdx.y * ld + i] = i < n ? (float)Q[(int64_t)blockIdx.y * n + i] : 0.f;
}

template <class... P, class... A>
static void launch_cluster(void (*kernel)(P...), cudaStream_t st, A... args)
{
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kQrBlocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kQrBlocks);
  cfg.blockDim = dim3(kQrThreads);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  LAUNCH_CHECK();
}

DesignQr::DesignQr(const float* X, int64_t ldx, const float* rr, int64_t n, int c, cudaStream_t st)
    : n_(n), c_(c), st_(st), work_(st), basis_(st), rr_(st), head_(1 + (size_t)c * c + c)
{
  // A | X, and Q | head | v: A and X are only needed by the factorisation
  double* A = (double*)work_.ensure((size_t)n * c * (sizeof(double) + sizeof(float)));
  float* dX = reinterpret_cast<float*>(A + (size_t)n * c);
  Q_ = (double*)basis_.ensure(((size_t)n * (c + 1) + head_.size()) * sizeof(double));
  double* d_head = Q_ + (size_t)n * c;
  v_ = d_head + head_.size();
  d_rr_ = (float*)rr_.ensure((size_t)n * sizeof(float));
  CUDA_TRY(cudaMemcpyAsync(d_rr_, rr, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
  CUDA_TRY(cudaMemcpy2DAsync(dX, (size_t)n * sizeof(float), X, (size_t)ldx * sizeof(float), (size_t)n * sizeof(float), c,
                             cudaMemcpyHostToDevice, st));
  CUDA_TRY(cudaMemsetAsync(d_head, 0, head_.size() * sizeof(double), st));
  launch_cluster(qr_kernel, st, dX, d_rr_, n, c, A, Q_, d_head);
}

void DesignQr::finish()
{
  CUDA_TRY(cudaMemcpyAsync(head_.data(), Q_ + (size_t)n_ * c_, head_.size() * sizeof(double), cudaMemcpyDeviceToHost, st_));
  CUDA_TRY(cudaStreamSynchronize(st_));
  waited_ = true;
  work_.release();
  finite = head_[0] == 0.0;
  const double* R = head_.data() + 1;
  const double* perm = R + (size_t)c_ * c_;
  const int kmax = (int)std::min<int64_t>(n_, c_);
  auto at = [&](int i, int j) { return R[(size_t)perm[j] * c_ + i]; };   // R's own column j
  const double thr = 1.1920928955078125e-07 * kmax * std::fabs(at(0, 0));
  rank = 0;
  for (int k = 0; k < kmax; ++k)
    if (std::fabs(at(k, k)) > thr) ++rank;
  RPt.assign((size_t)rank * c_, 0.0);
  for (int j = 0; j < c_; ++j)
    for (int i = 0; i < rank && i <= j; ++i) RPt[(size_t)perm[j] * rank + i] = at(i, j);
}

void DesignQr::store(float* out, int64_t ld, int64_t rows) const
{
  qr_store_kernel<<<dim3((unsigned)ceil_div(rows, 256), c_), 256, 0, st_>>>(Q_, n_, out, ld, rows);
  LAUNCH_CHECK();
}

void DesignQr::project(const float* d_y, float* out, bool scale) const
{
  launch_cluster(qr_project_kernel, st_, Q_, d_rr_, d_y, n_, c_, v_, out, scale ? 1 : 0);
}

void set_projection_qr(slemm_geno* g, const DesignQr& qr, int c)
{
  g->c = c;
  g->Q.ensure((size_t)g->n_pad * c * sizeof(float));
  qr.store(g->Q.as<float>(), g->n_pad, g->n_pad);
}

}  // namespace slemm

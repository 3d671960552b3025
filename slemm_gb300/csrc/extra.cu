// extra.cu — GEBV prediction (src/pred.cpp:4-141) and the GRAMMAR-Gamma per-variant terms of
// slemm_gamma (bin/slemm_gamma.py:302-325) as exact packed-genotype products.
//
// GEBV: tgv = Σ_j (flip_j ? 2 − x_j : x_j)·α_j = Cnt·α' + 2·Σ_{flip} α_j with α'_j = ±α_j, one
// pass over the individual-major copy (rows = individuals, K = SNPs).
//
// Score terms, with x = allele-1 count = 2 − count (pgenlib's convention) and z = count − gm:
//   x − x̄ = −z, so xy = −zᵀy and xx = ‖(I − QQᵀ)(rr∘z)‖²
//        = Σ rr²z² − Σ_l (Q_lᵀ(rr∘z))²,
//   Σ rr²z² = (S1 + 2·S2) − 2·gm·S1 + gm²·Σrr²   (count² = count + 2·[count = 2])
// where S1 = Σ rr²·count, S2 = Σ rr²·[count = 2], and Q_lᵀ(rr∘z) = Σ rr·Q_l·count − gm·Σ rr·Q_l.
// Two passes over the SNP-major copy (rows = SNPs, K = individuals): the counts against
// [y | rr² | rr·Q_l], and 2·[count = 2] (the high bit of each packed field) against rr².  When
// every rr is 1 (slemm_gamma's is_one_rr case) S1 and S2 are the SNP's integer class counts, and one
// pass against [y | Q_l] does.
//
// Exact products on the tensor cores.  A dense column v is cut into slices of 11 bits,
//   v·2^e = q_0 + 2^−11·q_1 + 2^−22·q_2 + …,   q_p integers, |q_p| ≤ 2^10,
// with e such that max|v|·2^e lies in [2^9, 2^10): six slices hold an FP64 column to 2^−65 of its
// largest value, four hold an FP32 one to 2^−43.  Slices are exact in FP16 and a count is at most
// 2, so a product row's sum over 8,192 K-elements is an integer of at most 2^24: the FP32
// accumulators are exact whatever their order.  K is therefore split every 128 K-tiles at the
// latest, the partials are added as 64-bit integers, and only the last combination of the slices
// rounds (in FP64).  Bound by the narrow tensor-core pass (its decoders).  GB300's FP64 pipe ran the
// same sums by an FMA per genotype and column: at n = 100,000, m = 50,000 the GEBV took 18,988 µs
// and takes 829 µs, the score terms with three covariates and residual weights 112,698 µs and
// 1,221 µs, with the same or a smaller error against 64-bit sums.
#include "internal.h"
#include "decode.cuh"
#include "reduce.cuh"

namespace slemm {

constexpr int kSliceBits = 11;
constexpr int kSlicesF64 = 6;
constexpr int kSlicesF32 = 4;
constexpr int kExactKTiles = 8192 / kTileK;   // K-tiles of one exact FP32 partial sum
constexpr int kXRows = 2048;                  // K-elements of one block of the operand kernels
constexpr int kXThreads = 256;

// e with amax·2^e in [2^9, 2^10) (0 for a zero or non-finite column)
__host__ __device__ inline int slice_exp(double amax)
{
  if (!(amax > 0.0) || !isfinite(amax)) return 0;
  int E;
  frexp(amax, &E);
  return 10 - E;
}

// Slices 0 … S−1 of v·2^e into rows row0 … row0 + S − 1 of the FP16 operand at K-element kidx, times
// the 2^−2s its K position takes (f16sub_pair_of).
template <int S>
__device__ __forceinline__ void store_slices(double v, int e, __half* __restrict__ B, int64_t K_pad, int row0,
                                             int64_t kidx)
{
  double r = ldexp(v, e);
  const float ks = f16sub_kscale(kidx);
#pragma unroll
  for (int p = 0; p < S; ++p) {
    const double q = rint(r);
    B[(int64_t)(row0 + p) * K_pad + kidx] = __float2half_rn(__fmul_rn((float)q, ks));
    r = (r - q) * (double)(1 << kSliceBits);   // exact
  }
}

// Σ_p 2^−11p·(Σ_splits D[s][row0 + p][r]) — the column's product with row r, in units of 2^−e
template <int S>
__device__ __forceinline__ double gather_slices(const float* __restrict__ D, int splits, int kp, int64_t M_pad,
                                                int row0, int64_t r)
{
  long long sum[S] = {};
  for (int s = 0; s < splits; ++s)
#pragma unroll
    for (int p = 0; p < S; ++p) sum[p] += (long long)D[((int64_t)s * kp + row0 + p) * M_pad + r];
  double v = 0.0;
#pragma unroll
  for (int p = S - 1; p >= 0; --p) v = v * (1.0 / (1 << kSliceBits)) + (double)sum[p];
  return v;
}

// GEBV operand: rows 0 … 5 the slices of alpha (0 past m), rows 6 … 15 zero
__global__ void __launch_bounds__(kXThreads)
gebv_operand_kernel(const double* __restrict__ alpha, int64_t m, int64_t m_pad, int e, __half* __restrict__ B)
{
  const int64_t j = (int64_t)blockIdx.x * kXThreads + threadIdx.x;
  if (j >= m_pad) return;
  store_slices<kSlicesF64>(j < m ? alpha[j] : 0.0, e, B, m_pad, 0, j);
#pragma unroll
  for (int q = kSlicesF64; q < 16; ++q) B[(int64_t)q * m_pad + j] = __float2half_rn(0.f);
}

__global__ void __launch_bounds__(kXThreads)
gebv_finish_kernel(const float* __restrict__ D, int splits, int kp, int64_t n_pad, int64_t n, int e, double shift,
                   double* __restrict__ tgv)
{
  const int64_t i = (int64_t)blockIdx.x * kXThreads + threadIdx.x;
  if (i < n) tgv[i] = shift + ldexp(gather_slices<kSlicesF64>(D, splits, kp, n_pad, 0, i), -e);
}

// Score columns: 0 = y, l = 1 … cq: rr·Q_{l−1}, cq + 1 = rr² (FP32 values), i < n; rr == nullptr: all 1
// and no last column.
__device__ __forceinline__ float score_column(const float* __restrict__ y, const float* __restrict__ rr,
                                              const float* __restrict__ Q, int64_t n_pad, int cq, int c, int64_t i)
{
  if (c == 0) return y[i];
  const float r = rr ? rr[i] : 1.f;
  return __fmul_rn(r, c <= cq ? Q[(int64_t)(c - 1) * n_pad + i] : r);
}

// Block partials of each column's sum and largest magnitude (∞ for a non-finite value):
// sums[c][blk], amax[c][blk]; grid (blocks, C).
__global__ void __launch_bounds__(kXThreads)
score_stats_kernel(const float* __restrict__ y, const float* __restrict__ rr, const float* __restrict__ Q, int64_t n,
                   int64_t n_pad, int cq, double* __restrict__ sums, double* __restrict__ amax, int nblk)
{
  __shared__ double sh[32];
  const int c = blockIdx.y;
  const int64_t i0 = (int64_t)blockIdx.x * kXRows, i1 = min64(n, i0 + kXRows);
  DF acc;
  float mx = 0.f;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += kXThreads) {
    const float v = score_column(y, rr, Q, n_pad, cq, c, i);
    df_add(acc, v);
    mx = fmaxf(mx, isfinite(v) ? fabsf(v) : INFINITY);
  }
  const double s = block_sum_d(df_value(acc), sh);
  __syncthreads();
  double w = mx;
  for (int o = 16; o; o >>= 1) w = fmax(w, __shfl_down_sync(0xffffffffu, w, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kXThreads / 32; ++q) w = fmax(w, sh[q]);
    sums[(int64_t)c * nblk + blockIdx.x] = s;
    amax[(int64_t)c * nblk + blockIdx.x] = w;
  }
}

// Operand of the count pass (N1 rows: column c's slices in rows 4c …, the rest zero) and of the
// count-2 pass (16 rows: rr²'s slices, the rest zero).  Blocks y < C write column y of the first,
// y = C the second (rr given), y > C one zero row of the first each.  A non-finite column is stored as zeros
// (its terms come out NaN through its sum in the finish).
__global__ void __launch_bounds__(kXThreads)
score_operand_kernel(const float* __restrict__ y, const float* __restrict__ rr, const float* __restrict__ Q, int64_t n,
                     int64_t n_pad, int cq, int C, const double* __restrict__ amax, int nblk, __half* __restrict__ B1,
                     __half* __restrict__ B2)
{
  __shared__ double sa;
  const int b = blockIdx.y;
  const int64_t i0 = (int64_t)blockIdx.x * kXRows, i1 = min64(n_pad, i0 + kXRows);
  if (b > C) {
    for (int64_t i = i0 + threadIdx.x; i < i1; i += kXThreads)
      B1[(int64_t)(kSlicesF32 * C + b - C - 1) * n_pad + i] = __float2half_rn(0.f);
    return;
  }
  if (b == C && !rr) return;
  const int c = b < C ? b : C - 1;
  if (threadIdx.x < 32) {
    const double v = warp_max_partials(amax + (int64_t)c * nblk, nblk);
    if (threadIdx.x == 0) sa = v;
  }
  __syncthreads();
  const int e = slice_exp(sa);
  const bool fine = isfinite(sa);
  __half* B = b < C ? B1 : B2;
  const int row0 = b < C ? kSlicesF32 * c : 0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += kXThreads) {
    const float v = (i < n && fine) ? score_column(y, rr, Q, n_pad, cq, c, i) : 0.f;
    store_slices<kSlicesF32>((double)v, e, B, n_pad, row0, i);
    if (b == C)
      for (int q = kSlicesF32; q < 16; ++q) B2[(int64_t)q * n_pad + i] = __float2half_rn(0.f);
  }
}

// xy, xx per SNP from the exact sums, MAC filter → NaN.
constexpr int kMaxScoreCols = 16;   // y, rr² and at most 14 projection columns
__global__ void __launch_bounds__(kXThreads)
score_finish_kernel(const float* __restrict__ D1, int splits1, int kp1, const float* __restrict__ D2, int splits2,
                    int kp2, int64_t m_pad, int64_t m, int64_t n, const int32_t* __restrict__ n1,
                    const int32_t* __restrict__ n2, int cq, int C, const double* __restrict__ sums,
                    const double* __restrict__ amax, int nblk, int mac, float* __restrict__ xy, float* __restrict__ xx)
{
  __shared__ double ssum[kMaxScoreCols];
  __shared__ int sexp[kMaxScoreCols];
  for (int c = threadIdx.x >> 5; c < C; c += kXThreads / 32) {
    const double s = warp_sum_partials(sums + (int64_t)c * nblk, nblk);
    const double a = warp_max_partials(amax + (int64_t)c * nblk, nblk);
    if ((threadIdx.x & 31) == 0) {
      ssum[c] = isfinite(a) ? s : NAN;
      sexp[c] = slice_exp(a);
    }
  }
  __syncthreads();
  const int64_t j = (int64_t)blockIdx.x * kXThreads + threadIdx.x;
  if (j >= m) return;
  const double pc = (double)n1[j] + 2.0 * (double)n2[j];
  const double s_a1 = 2.0 * (double)n - pc;   // Σ x with x = 2 − count
  if (s_a1 <= mac || 2.0 * (double)n - s_a1 <= mac) {
    xy[j] = __int_as_float(0x7fc00000);
    xx[j] = __int_as_float(0x7fc00000);
    return;
  }
  const double gm = pc / (double)n;
  auto sum_of = [&](int c) {
    return ldexp(gather_slices<kSlicesF32>(D1, splits1, kp1, m_pad, kSlicesF32 * c, j), -sexp[c]);
  };
  xy[j] = (float)(-(sum_of(0) - gm * ssum[0]));
  double v;
  if (D2 != nullptr) {
    const double S1 = sum_of(C - 1);
    const double S2x2 = ldexp(gather_slices<kSlicesF32>(D2, splits2, kp2, m_pad, 0, j), -sexp[C - 1]);   // 2·S2
    v = (S1 + S2x2) - 2.0 * gm * S1 + gm * gm * ssum[C - 1];
  } else {
    v = (pc + 2.0 * (double)n2[j]) - 2.0 * gm * pc + gm * gm * (double)n;
  }
  for (int c = 1; c <= cq; ++c) {
    const double ql = sum_of(c) - gm * ssum[c];
    v -= ql * ql;
  }
  xx[j] = (float)v;
}

// Split-K count of an exact product over K_tiles K-tiles: at most kExactKTiles of them each.
static int exact_splits(int64_t M_pad, int64_t K_tiles, int N)
{
  return choose_splits(M_pad / gemm_tc_rows_per_cta(N, 0), K_tiles, 1, num_sms(),
                       (int)ceil_div(K_tiles, kExactKTiles));
}

}  // namespace slemm

using namespace slemm;

extern "C" {

int slemm_gpu_gebv(slemm_geno* g, const double* alpha, const uint8_t* flip, double* tgv)
{
  return guarded([&] {
    CHECK_ARG(g && alpha && tgv, "null argument");
    if (g->is_view)
      SLEMM_THROW(SLEMM_ERR_UNSUPPORTED, "slemm_gpu_gebv reads the packed copies directly and is not available on a "
                                         "trait view; create a handle with the keep list instead");
    cudaStream_t st = g->stream;
    std::vector<double> a(g->m);
    double shift = 0.0, amax = 0.0;
    for (int64_t j = 0; j < g->m; ++j) {
      CHECK_ARG(std::isfinite(alpha[j]), "non-finite SNP effect");
      const bool f = flip && flip[j];
      a[j] = f ? -alpha[j] : alpha[j];
      if (f) shift += 2.0 * alpha[j];
      amax = std::max(amax, std::fabs(alpha[j]));
    }
    const int e = slice_exp(amax);
    const int64_t K_tiles = g->m_pad / kTileK;
    const int N = 16, kp = 8;
    const int splits = exact_splits(g->n_pad, K_tiles, N);
    DevBuf d_a(st), d_out(st);
    d_a.ensure(a.size() * sizeof(double));
    d_out.ensure((size_t)g->n * sizeof(double));
    __half* B = (__half*)g->ws_B.ensure((size_t)N * g->m_pad * sizeof(__half));
    float* D = (float*)g->ws_D.ensure((size_t)splits * kp * g->n_pad * sizeof(float));
    CUDA_TRY(cudaMemcpyAsync(d_a.p, a.data(), a.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    gebv_operand_kernel<<<(unsigned)ceil_div(g->m_pad, kXThreads), kXThreads, 0, st>>>(d_a.as<double>(), g->m, g->m_pad,
                                                                                      e, B);
    LAUNCH_CHECK();
    gemm_tc({g->GT.as<uint8_t>(), g->n_pad, g->m_pad, B, N, D, splits, g->err.as<int>(), kp, 1, true}, st);
    gebv_finish_kernel<<<(unsigned)ceil_div(g->n, kXThreads), kXThreads, 0, st>>>(D, splits, kp, g->n_pad, g->n, e, shift,
                                                                                 d_out.as<double>());
    LAUNCH_CHECK();
    CUDA_TRY(cudaMemcpyAsync(tgv, d_out.p, g->n * sizeof(double), cudaMemcpyDeviceToHost, st));
    check_device_error(g);
  });
}

int slemm_gpu_score_terms(slemm_geno* g, const float* y, int mac, float* xy, float* xx)
{
  return guarded([&] {
    CHECK_ARG(g && y && xy && xx, "null argument");
    if (g->is_view)
      SLEMM_THROW(SLEMM_ERR_UNSUPPORTED, "slemm_gpu_score_terms reads the packed copies directly and is not available on a "
                                         "trait view; create a handle with the keep list instead");
    CHECK_ARG(g->weights_set, "set_weights (rr) must be called first");
    const int c = g->c;
    CHECK_ARG(c <= 14, "score terms support up to 14 projection columns");
    cudaStream_t st = g->stream;
    const int64_t n = g->n, n_pad = g->n_pad;
    const float* rr = g->rr_one ? nullptr : g->rr.as<float>();
    const int C = 1 + c + (rr ? 1 : 0);
    const int64_t K_tiles = n_pad / kTileK;
    const int nblk = (int)ceil_div(n_pad, kXRows);
    const int kp1 = (int)round_up(kSlicesF32 * C, 8), kp2 = 8;
    const int N1 = (int)round_up(kp1, 16), N2 = 16;
    const int sp1 = exact_splits(g->m_pad, K_tiles, N1), sp2 = exact_splits(g->m_pad, K_tiles, N2);
    DevBuf dy(st), dstat(st), dcnt(st), dout(st);
    float* yv = (float*)dy.ensure((size_t)n * sizeof(float));
    double* sums = (double*)dstat.ensure((size_t)2 * C * nblk * sizeof(double));
    double* amax = sums + (size_t)C * nblk;
    int64_t* pc = (int64_t*)dcnt.ensure((size_t)g->m * (sizeof(int64_t) + 2 * sizeof(int32_t)));
    int32_t* n1 = reinterpret_cast<int32_t*>(pc + g->m);
    int32_t* n2 = n1 + g->m;
    float* oxy = (float*)dout.ensure((size_t)2 * g->m * sizeof(float));
    float* oxx = oxy + g->m;
    __half* B1 = (__half*)g->ws_B.ensure((size_t)(N1 + N2) * n_pad * sizeof(__half));
    __half* B2 = B1 + (size_t)N1 * n_pad;
    const size_t d1 = (size_t)sp1 * kp1 * g->m_pad, d2 = (size_t)sp2 * kp2 * g->m_pad;
    float* D1 = (float*)g->ws_D.ensure((d1 + d2) * sizeof(float));
    float* D2 = D1 + d1;
    CUDA_TRY(cudaMemcpyAsync(yv, y, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
    row_counts_device(g, pc, n1, n2);
    const float* Q = g->Q.as<float>();
    score_stats_kernel<<<dim3(nblk, C), kXThreads, 0, st>>>(yv, rr, Q, n, n_pad, c, sums, amax, nblk);
    LAUNCH_CHECK();
    score_operand_kernel<<<dim3(nblk, C + 1 + N1 - kSlicesF32 * C), kXThreads, 0, st>>>(yv, rr, Q, n, n_pad, c, C, amax, nblk,
                                                                                      B1, B2);
    LAUNCH_CHECK();
    const uint8_t* G = g->G.as<uint8_t>();
    int* err = g->err.as<int>();
    gemm_tc({G, g->m_pad, n_pad, B1, N1, D1, sp1, err, kp1, 1, true}, st);
    if (rr) gemm_tc({G, g->m_pad, n_pad, B2, N2, D2, sp2, err, kp2, 1, true, 0, true}, st);
    score_finish_kernel<<<(unsigned)ceil_div(g->m, kXThreads), kXThreads, 0, st>>>(
        D1, sp1, kp1, rr ? D2 : nullptr, sp2, kp2, g->m_pad, g->m, n, n1, n2, c, C, sums, amax, nblk, mac, oxy, oxx);
    LAUNCH_CHECK();
    CUDA_TRY(cudaMemcpyAsync(xy, oxy, (size_t)g->m * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(xx, oxx, (size_t)g->m * sizeof(float), cudaMemcpyDeviceToHost, st));
    check_device_error(g);
  });
}

}  // extern "C"

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
// Both products are exact sums (exact.cu).
#include "internal.h"

#include <cstring>
#include <memory>

namespace slemm {

// xy, xx per SNP from the exact sums dots[c][j] (columns y, rr·Q_l, rr²) and twos, MAC filter → NaN.
// twos == nullptr: every rr is 1 and there is no last column.
__global__ void __launch_bounds__(256)
score_finish_kernel(const double* __restrict__ dots, const double* __restrict__ twos, const double* __restrict__ tot,
                    int64_t m, int64_t n, const int32_t* __restrict__ n1, const int32_t* __restrict__ n2, int cq,
                    int mac, float* __restrict__ xy, float* __restrict__ xx)
{
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const double pc = (double)n1[j] + 2.0 * (double)n2[j];
  const double s_a1 = 2.0 * (double)n - pc;   // Σ x with x = 2 − count
  if (s_a1 <= mac || 2.0 * (double)n - s_a1 <= mac) {
    xy[j] = __int_as_float(0x7fc00000);
    xx[j] = __int_as_float(0x7fc00000);
    return;
  }
  const double gm = pc / (double)n;
  xy[j] = (float)(-(dots[j] - gm * tot[0]));
  double v;
  if (twos != nullptr) {
    const double S1 = dots[(int64_t)(cq + 1) * m + j];
    v = (S1 + twos[j]) - 2.0 * gm * S1 + gm * gm * tot[cq + 1];
  } else {
    v = (pc + 2.0 * (double)n2[j]) - 2.0 * gm * pc + gm * gm * (double)n;
  }
  for (int c = 1; c <= cq; ++c) {
    const double ql = dots[(int64_t)c * m + j] - gm * tot[c];
    v -= ql * ql;
  }
  xx[j] = (float)v;
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
    // ±alpha, the shift, and the largest and smallest nonzero magnitude as bits (a zero less 1 is the largest
    // integer); four chains of additions (each with its rounding errors summed beside it, so that the shift is as good
    // as exact) and no branches, since half of the flips are unforeseen (50,000 effects: 146 µs as a plain loop, 67 now)
    const int64_t m = g->m;
    const std::unique_ptr<double[]> a(new double[m]);
    uint64_t most = 0, least = UINT64_MAX;
    double part[4] = {}, rest[4] = {};
    auto add = [](double& sum, double& err, double x) {
      const double t = sum + x, b = t - sum;
      err += (sum - (t - b)) + (x - b);
      sum = t;
    };
    auto take = [&](int64_t j, int q) {
      uint64_t bits;
      std::memcpy(&bits, alpha + j, sizeof(bits));
      const uint64_t f = flip && flip[j] ? 1 : 0, signedbits = bits ^ (f << 63);
      std::memcpy(&a[j], &signedbits, sizeof(bits));
      bits &= ~(1ull << 63);
      most = std::max(most, bits);
      least = std::min(least, bits - 1);
      add(part[q], rest[q], alpha[j] * (double)(2 * f));
    };
    int64_t j = 0;
    for (; j + 4 <= m; j += 4)
      for (int q = 0; q < 4; ++q) take(j + q, q);
    for (; j < m; ++j) take(j, 0);
    CHECK_ARG(most < 0x7FF0000000000000ull, "non-finite SNP effect");
    for (int q = 1; q < 4; ++q) add(part[0], rest[0], part[q]);
    const double shift = std::isfinite(part[0]) ? part[0] + ((rest[0] + rest[1]) + (rest[2] + rest[3])) : part[0];
    double amax, amin = INFINITY;
    std::memcpy(&amax, &most, sizeof(amax));
    if (most > 0) std::memcpy(&amin, &++least, sizeof(amin));
    DevBuf d_a(st), d_out(st);
    d_a.ensure((size_t)m * sizeof(double));
    d_out.ensure((size_t)g->n * sizeof(double));
    CUDA_TRY(cudaMemcpyAsync(d_a.p, a.get(), (size_t)m * sizeof(double), cudaMemcpyHostToDevice, st));
    exact_gebv(g, d_a.as<double>(), amax, amin, shift, d_out.as<double>());
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
    const int64_t n = g->n, m = g->m;
    DevBuf dy(st), ddot(st), dcnt(st), dout(st);
    float* yv = (float*)dy.ensure((size_t)n * sizeof(float));
    const ExactCols cols{yv, g->rr_one ? nullptr : g->rr.as<float>(), g->Q.as<float>(), g->n_pad, c};
    double* dots = (double*)ddot.ensure(((size_t)(cols.count() + 1) * m + cols.count()) * sizeof(double));
    double* twos = cols.rr ? dots + (size_t)cols.count() * m : nullptr;
    double* tot = dots + (size_t)(cols.count() + 1) * m;
    int64_t* pc = (int64_t*)dcnt.ensure((size_t)m * (sizeof(int64_t) + 2 * sizeof(int32_t)));
    int32_t* n1 = reinterpret_cast<int32_t*>(pc + m);
    int32_t* n2 = n1 + m;
    float* oxy = (float*)dout.ensure((size_t)2 * m * sizeof(float));
    float* oxx = oxy + m;
    CUDA_TRY(cudaMemcpyAsync(yv, y, (size_t)n * sizeof(float), cudaMemcpyHostToDevice, st));
    row_counts_device(g, pc, n1, n2);
    for (int guess = exact_dots_guess(g, cols);; guess = 0) {
      exact_dots(g, cols, dots, tot, twos, guess);
      score_finish_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>(dots, twos, tot, m, n, n1, n2, c, mac, oxy, oxx);
      LAUNCH_CHECK();
      CUDA_TRY(cudaMemcpyAsync(xy, oxy, (size_t)m * sizeof(float), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(cudaMemcpyAsync(xx, oxx, (size_t)m * sizeof(float), cudaMemcpyDeviceToHost, st));
      check_device_error(g);
      if (exact_dots_done(g, cols, guess)) break;
    }
  });
}

}  // extern "C"

// gwa.cu — windowed MLMA of slemm_gwa.py (bin/slemm_gwa.py:259-431) on the packed genotypes.
//
// The model SNPs of a chromosome are cut into overlapping blocks of block_size (step
// block_size/2, the last block flush with the end; :322-335); block i serves the tested variants
// from the previous block's bound to model SNP [block_size − block_size/4] of its own (:337-344).
// Per block, with B the block's centred (per-SNP mean), rr-scaled, projected genotypes:
//   H = BBᵀ + model_snp_ct·τ·diag(rvar),  rvar = (2 − mean)·mean/2            (:376-408)
// and per tested variant x (centred, MAC filter on allele-1 counts):
//   xy = xᵀy (before scaling; y is the Py column of .reml.py.txt),
//   xx = ‖x̃‖² − (Bx̃)ᵀH⁻¹(Bx̃) with x̃ = (I − QQᵀ)(rr∘x)                          (:409-428)
// then xx /= τ, β = xy/xx·cf, se = √(snp_var·cf/xx), χ² = (β/se)², p = P(χ²₁ > χ²)  (:430-434).
// Allele-1 counts are 2 − the .bed's allele-2 counts: centring flips the sign of x, which leaves
// xx unchanged and flips xy — computed here with allele-2 counts and xy negated at the end.
//
// GB300 mapping: the model SNPs are gathered into their own packed copy (16-byte rows of the
// tiles), so every block is a contiguous row range.  xᵀy, ‖x̃‖² and Qᵀ(rr∘x) of every variant come from
// one exact pass over the packed matrix, BBᵀ and Bx̃ for all the block's tested variants are projected
// Gram blocks read straight from the packed rows — no dense B or x̃ is ever formed — and the blocks'
// systems are factored together over all SMs with their tested variants' rows riding along, whose
// norms are the quadratic forms (gram.cu).
#include "internal.h"
#include "gram.h"
#include "qr.h"

#include <algorithm>
#include <cmath>

namespace slemm {

// Gs (rows = rows[0 … cnt), tiled like G, rows ≥ cnt zero) from G: one 16-byte tile row each.
__global__ void gather_rows_kernel(const uint4* __restrict__ G, int64_t K_tiles, const int64_t* __restrict__ rows,
                                   int64_t cnt, int64_t total, uint4* __restrict__ Gs)
{
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;   // destination order
  if (q >= total) return;
  const int64_t r = q % 128, t = q / 128, kt = t % K_tiles, mt = t / K_tiles;
  const int64_t jd = mt * 128 + r;
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (jd < cnt) {
    const int64_t js = rows[jd];
    v = G[((js / 128) * K_tiles + kt) * 128 + (js % 128)];
  }
  Gs[q] = v;
}

// The statistics of the tested variants (bin/slemm_gwa.py:413-434), allele-1 orientation.  As a host loop
// over 20,011 variants, with a complementary error function each, this was 0.66 ms of a call's 4.65 ms,
// with the GPU idle; here it is a few µs (the call: 4.65 → 4.00 ms).
__global__ void __launch_bounds__(128)
gwa_final_kernel(const double* __restrict__ xy2, const double* __restrict__ xx2, const double* __restrict__ q,
                 const int64_t* __restrict__ pc, int64_t n, int64_t ntest, int mac, float tau, float cfactor, float snp_var,
                 float* __restrict__ beta, float* __restrict__ se, float* __restrict__ chisq, double* __restrict__ pval)
{
  const int64_t t = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (t >= ntest) return;
  const int64_t s_a1 = 2 * n - pc[t];   // allele-1 count sum
  float b = NAN, e = NAN, c = NAN;
  double p = NAN;
  if (!(s_a1 <= mac || 2 * n - s_a1 <= mac)) {
    const float xx = __fdiv_rn((float)(xx2[t] - q[t]), tau);
    const float xy = (float)-xy2[t];
    b = __fmul_rn(__fdiv_rn(xy, xx), cfactor);
    e = __fsqrt_rn(__fdiv_rn(__fmul_rn(snp_var, cfactor), xx));
    const float z = __fdiv_rn(b, e);
    c = __fmul_rn(z, z);
    p = erfc(sqrt((double)c / 2.0));
  }
  beta[t] = b;
  se[t] = e;
  chisq[t] = c;
  pval[t] = p;
}

}  // namespace slemm

using namespace slemm;

extern "C" int slemm_gpu_gwa_windows(slemm_geno* g, const float* y, const float* R, const float* covar, int64_t ldc,
                                     int c, const int64_t* model_idx, int64_t n_model, int64_t test_begin,
                                     int64_t test_end, int block_size, float tau, int64_t model_snp_ct, float cfactor,
                                     float snp_var, int mac, float* beta, float* se, float* chisq, double* pval)
{
  return guarded([&] {
    CHECK_ARG(g && y && covar && model_idx && beta && se && chisq && pval, "null argument");
    if (g->is_view)
      SLEMM_THROW(SLEMM_ERR_UNSUPPORTED, "slemm_gpu_gwa_windows reads the packed copies directly and is not available on a "
                                         "trait view; create a handle with the keep list instead");
    const int64_t n = g->n, m = g->m;
    CHECK_ARG(c >= 1 && c <= SLEMM_MAX_COVARIATES && ldc >= n, "bad covariate matrix");
    CHECK_ARG(n_model >= 2 && test_begin >= 0 && test_end < m && test_begin <= test_end, "bad SNP ranges");
    for (int64_t k = 0; k < n_model; ++k)
      CHECK_ARG(model_idx[k] >= 0 && model_idx[k] < m && (k == 0 || model_idx[k] > model_idx[k - 1]),
                "model SNP indices must be increasing handle indices");
    // as in the script, the model SNPs and the tested variants are those of one chromosome, so
    // every block's share of the tested range (below) is a non-empty or empty interval
    CHECK_ARG(model_idx[0] >= test_begin && model_idx[n_model - 1] <= test_end,
              "model SNPs must lie inside the tested range (one chromosome)");
    CHECK_ARG(tau > 0.f && std::isfinite(tau), "tau must be positive");
    cudaStream_t st = g->stream;
    // blocks and the tested range each serves (bin/slemm_gwa.py:319-344)
    int bs = block_size;
    if (bs > n_model) bs = (int)(n_model / 2) * 2;
    CHECK_ARG(bs >= 4 && bs <= 5000, "block size out of [4, 5000]");
    const int step = bs / 2, ext = step / 2;
    std::vector<int64_t> start;
    for (int64_t i = 0; i < (n_model - step) / step; ++i) start.push_back(i * step);
    if ((n_model - step) % step != 0) start.push_back(n_model - bs);
    const int nb = (int)start.size();
    std::vector<int64_t> lo(nb), hi(nb);
    lo[0] = test_begin;
    hi[0] = model_idx[start[0] + bs - ext];
    for (int i = 1; i < nb; ++i) {
      lo[i] = hi[i - 1];
      hi[i] = model_idx[start[i] + bs - ext];
    }
    hi[nb - 1] = test_end + 1;
    for (int i = 0; i < nb; ++i)
      CHECK_ARG(test_begin <= lo[i] && lo[i] <= hi[i] && hi[i] <= test_end + 1, "inconsistent block ranges");
    // rr, Q of the covariates (scipy's economic QR in the script; any orthonormal basis gives the
    // same projection)
    std::vector<float> rr(g->n_pad, 0.f);
    bool rr_one = true;
    for (int64_t i = 0; i < n; ++i) {
      const float r = R ? R[i] : 1.0f;
      CHECK_ARG(r > 0.f && std::isfinite(r), "R must be positive");
      rr[i] = 1.0f / std::sqrt(r);
      rr_one = rr_one && rr[i] == 1.0f;
    }
    DesignQr qr(covar, ldc, rr.data(), n, c, st);
    // per-SNP means (allele-2) of the whole handle
    std::vector<float> mean(g->m_pad, 0.f);
    DevBuf d_counts(st);
    int64_t* d_pc = (int64_t*)d_counts.ensure((size_t)m * 16);
    {
      std::vector<int64_t> pc(m);
      row_counts_device(g, d_pc, (int32_t*)(d_pc + m), (int32_t*)(d_pc + m) + m);
      CUDA_TRY(cudaMemcpyAsync(pc.data(), d_pc, m * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(cudaStreamSynchronize(st));
      for (int64_t j = 0; j < m; ++j) mean[j] = (float)pc[j] / (float)n;
    }
    qr.finish();
    CHECK_ARG(qr.rank == c, "covariate matrix is not of full rank");
    // packed copy of the model SNPs, and every variant's statistics
    const int64_t K_tiles = g->n_pad / kTileK;
    const int64_t model_rows = round_up(n_model, kPadRows);
    const int64_t total = model_rows * K_tiles;   // 16-byte tile rows
    DevBuf d_model(st), d_idx(st), d_mean(st), d_y(st), d_Q(st), d_rr(st);
    uint8_t* Gm = (uint8_t*)d_model.ensure((size_t)total * 16);
    int64_t* didx = (int64_t*)d_idx.ensure((size_t)n_model * sizeof(int64_t));
    CUDA_TRY(cudaMemcpyAsync(didx, model_idx, (size_t)n_model * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    gather_rows_kernel<<<(unsigned)ceil_div(total, 256), 256, 0, st>>>(g->G.as<uint4>(), K_tiles, didx, n_model, total,
                                                                       reinterpret_cast<uint4*>(Gm));
    LAUNCH_CHECK();
    float* dQ = (float*)d_Q.ensure((size_t)g->n_pad * c * sizeof(float));
    qr.store(dQ, g->n_pad, g->n_pad);
    float* dmean = (float*)d_mean.ensure(mean.size() * sizeof(float));
    float* dy = (float*)d_y.ensure(n * sizeof(float));
    float* drr = nullptr;
    if (!rr_one) {
      drr = (float*)d_rr.ensure(rr.size() * sizeof(float));
      CUDA_TRY(cudaMemcpyAsync(drr, rr.data(), rr.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    }
    CUDA_TRY(cudaMemcpyAsync(dmean, mean.data(), mean.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(dy, y, n * sizeof(float), cudaMemcpyHostToDevice, st));
    const ExactCols cols{dy, drr, dQ, g->n_pad, c};
    const int batch = 32;   // blocks at a time (bounded memory)
    DevBuf d_status(st), d_out(st);
    const int64_t ntest = test_end - test_begin + 1;
    int* status = (int*)d_status.ensure((1 + (size_t)batch) * sizeof(int));
    double* d_p = (double*)d_out.ensure((size_t)ntest * (sizeof(double) + 3 * sizeof(float)));
    float* d_f = reinterpret_cast<float*>(d_p + ntest);   // beta | se | chisq
    auto attempt = [&](int guess) {   // false: the guess was too small (exact_dots)
      GramStatsBuf all_stats, model_stats;
      gram_stats(g, dmean, cols, guess, all_stats);
      gram_stats_gather(all_stats.s, didx, n_model, c, model_stats, st);
      const GramSide all{g->G.as<uint8_t>(), m, all_stats.s}, model{Gm, n_model, model_stats.s};
      const int64_t rows_max = round_up(bs, kPadRows) + kPadRows;
      DevBuf d_gram(st), d_ridge(st), d_off(st), d_Z(st), d_q(st);
      double* dq = (double*)d_q.ensure((size_t)ntest * sizeof(double));
      CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
      HostKeep keep(st);   // the batches' host tables
      for (int b0 = 0; b0 < nb; b0 += batch) {
        const int bn = std::min(batch, nb - b0);
        const int64_t stride = rows_max * bs;
        float* gram = (float*)d_gram.ensure((size_t)bn * stride * sizeof(float));
        const int64_t tested = hi[b0 + bn - 1] - lo[b0];   // the blocks' tested ranges follow each other
        float* Z = (float*)d_Z.ensure((size_t)std::max<int64_t>(tested, 1) * rows_max * sizeof(float));
        struct Tables {
          std::vector<int64_t> off;   // offA | offZ
          std::vector<int> tb;
          std::vector<float> ridge;
        };
        auto& [off, tb, ridge] = keep.make<Tables>();
        off.resize((size_t)2 * bn);
        tb.resize(bn);
        ridge.resize((size_t)bn * bs);
        std::vector<GramJob> own, tested_by;   // the blocks' own Gram, and with the variants each serves
        int t_max = 0;
        for (int bi = 0; bi < bn; ++bi) {
          const int64_t s0 = start[b0 + bi];
          GramJob job{0, 0, s0, bs, gram + (size_t)bi * stride};
          gram_rows(model, s0, bs, job);
          own.push_back(job);
          for (int t = 0; t < bs; ++t) {
            const float mu = mean[model_idx[s0 + t]];
            ridge[(size_t)bi * bs + t] = (float)model_snp_ct * tau * ((2.0f - mu) * mu / 2.0f);
          }
          off[bi] = s0 - job.r0;
          off[bn + bi] = lo[b0 + bi] - lo[b0];
          tb[bi] = (int)(hi[b0 + bi] - lo[b0 + bi]);
          t_max = std::max(t_max, tb[bi]);
          job.c0 = lo[b0 + bi];
          job.ncols = tb[bi];
          job.out = Z + off[bn + bi] * rows_max;
          tested_by.push_back(job);
        }
        gram_blocks(g, model, model, own, c, drr, rows_max, GramHalf::lower, keep);
        gram_blocks(g, model, all, tested_by, c, drr, rows_max, GramHalf::all, keep);
        float* dr = (float*)d_ridge.ensure(ridge.size() * sizeof(float));
        int64_t* doff = (int64_t*)d_off.ensure(off.size() * sizeof(int64_t));
        CUDA_TRY(cudaMemcpyAsync(dr, ridge.data(), ridge.size() * sizeof(float), cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(doff, off.data(), off.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(status + 1, tb.data(), (size_t)bn * sizeof(int), cudaMemcpyHostToDevice, st));
        spd_row_norms({gram, stride, Z, doff, doff + bn, status + 1, rows_max, bs, bn, t_max}, dr,
                      dq + (lo[b0] - test_begin), status, st);
      }
      gwa_final_kernel<<<(unsigned)ceil_div(ntest, 128), 128, 0, st>>>(
          all_stats.s.xy + test_begin, all_stats.s.xx + test_begin, dq, d_pc + test_begin, n, ntest, mac, tau, cfactor,
          snp_var, d_f, d_f + ntest, d_f + 2 * ntest, d_p);
      LAUNCH_CHECK();
      check_device_error(g);
      keep.waited();
      return exact_dots_done(g, cols, guess);
    };
    if (!attempt(exact_dots_guess(g, cols))) attempt(0);
    int hs = 0;
    CUDA_TRY(cudaMemcpy(&hs, status, sizeof(int), cudaMemcpyDeviceToHost));
    if (hs) SLEMM_THROW(SLEMM_ERR_NUMERIC, "a block's BBᵀ + ridge is not positive definite in FP32");
    CUDA_TRY(cudaMemcpyAsync(beta, d_f, ntest * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(se, d_f + ntest, ntest * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(chisq, d_f + 2 * ntest, ntest * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(pval, d_p, ntest * sizeof(double), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
  });
}

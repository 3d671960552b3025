// lmm.cu — GWAS step 1 quadratic forms (`--lmm` with real markers, src/reml.cpp:919-981): the
// per-marker statistics of the .gstat.txt file that slemm_gamma.py and slemm_gwa.py read.
//
// Marker sample (:919-925): markers with gm·n > 20 and (2 − gm)·n > 20 in file order, shuffled by
// libstdc++'s std::random_shuffle (for i = 1 … N−1: swap(v[i], v[rand() % (i+1)])) driven by the C
// library's rand() in its initial state — glibc's TYPE_3 additive-feedback generator
// (r_i = r_{i−3} + r_{i−31} mod 2^32, output r_i ≫ 1, state from the seed by the Park–Miller
// recurrence 16807·r mod 2^31−1, first 310 outputs discarded), restated here with seed 1.
//
// For the first num_qf markers x (centred counts): xPy = xᵀPy; v = (I − QQᵀ)(rr∘x);
// xPx = vᵀ(H0 + τ1 I)⁻¹v through one projected Lanczos seed on all v and one solve at shift 0;
// xSx = ‖v‖²; xBx = (xSx − zᵀ(ZᵀZ + τ1·diag(1/gw))⁻¹z)/τ1 where Z holds the projected, rr-scaled
// centred counts of the window_size markers around x (clamped at both ends) and z = Zᵀv.
//
// GB300 mapping: z is the row of x in its own window's ZᵀZ (x lies in the window), so each window is
// one projected Gram block read straight from the packed rows (gram.cu).  The windows' systems are
// factored together over all SMs by blocked FP32 panels; the quadratic form is taken as
// 2zᵀx − xᵀMx of the FP32 solution against the kept matrix, which squares the solution's own
// error away, so it is limited by the Gram's accuracy, not by the FP32 factorisation.
#include "internal.h"
#include "reduce.cuh"
#include "dense.cuh"
#include "gram.h"

#include <algorithm>
#include <memory>

namespace slemm {

// ---- C library rand() and std::random_shuffle, restated -----------------------------------------
namespace {
struct LibcRand {
  uint32_t r[34];
  int i = 0;   // ring position
  explicit LibcRand(uint32_t seed)
  {
    std::vector<int64_t> v(344);
    v[0] = seed;
    for (int k = 1; k < 31; ++k) {
      const int64_t hi = v[k - 1] / 127773, lo = v[k - 1] % 127773;
      int64_t w = 16807 * lo - 2836 * hi;   // 16807·r mod (2^31 − 1) without overflow (Schrage)
      if (w < 0) w += 2147483647;
      v[k] = w;
    }
    for (int k = 31; k < 34; ++k) v[k] = v[k - 31];
    std::vector<uint32_t> u(v.begin(), v.begin() + 34);
    for (int k = 34; k < 344; ++k) u.push_back(u[k - 31] + u[k - 3]);
    for (int k = 0; k < 34; ++k) r[k] = u[310 + k];   // the last 34 words of the warm-up
  }
  int next()
  {
    // r holds words k−34 … k−1 (ring); word k = word k−31 + word k−3
    const uint32_t w = r[(i + 34 - 31) % 34] + r[(i + 34 - 3) % 34];
    r[i] = w;
    i = (i + 1) % 34;
    return (int)(w >> 1);
  }
};
}  // namespace

// src/reml.cpp:919-925: the sampled markers (first min(num_qf, count)).
static std::vector<int64_t> lmm_variants(const std::vector<float>& gm, int64_t n, int num_qf)
{
  std::vector<int> v;
  for (int i = 0; i < (int)gm.size(); ++i)
    if (gm[i] * (float)n > 20.0f && (2.0f - gm[i]) * (float)n > 20.0f) v.push_back(i);
  LibcRand rnd(1);
  for (size_t i = 1; i < v.size(); ++i) {
    const size_t j = (size_t)rnd.next() % (i + 1);
    if (i != j) std::swap(v[i], v[j]);
  }
  const int k = std::min<int>(num_qf, (int)v.size());
  return std::vector<int64_t>(v.begin(), v.begin() + k);
}

// out[c] = xx[rows[c]]
__global__ void take_xx_kernel(const double* __restrict__ xx, const int64_t* __restrict__ rows, int k, double* __restrict__ out)
{
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < k) out[c] = xx[rows[c]];
}

}  // namespace slemm

using namespace slemm;

extern "C" int slemm_gpu_lmm_quadforms(slemm_geno* g, const float* Py, float tau1, float tol_L, int num_qf,
                                       int window_size, int64_t* variants, float* xPy, float* xPx, float* xBx,
                                       float* xSx, int* count)
{
  return guarded([&] {
    CHECK_ARG(g && Py && variants && xPy && xPx && xBx && xSx && count, "null argument");
    if (g->is_view)
      SLEMM_THROW(SLEMM_ERR_UNSUPPORTED, "slemm_gpu_lmm_quadforms reads the packed copies directly and is not available on a "
                                         "trait view; create a handle with the keep list instead");
    CHECK_ARG(g->weights_set, "set_weights must be called first");
    CHECK_ARG(num_qf >= 1 && num_qf <= 300, "num_qf_markers out of [1, 300]");
    CHECK_ARG(tau1 > 0.f && std::isfinite(tau1), "tau1 must be positive");
    const int64_t n = g->n, m = g->m;
    CHECK_ARG(window_size >= 2 && window_size % 2 == 0 && window_size <= 5000 && window_size <= m,
              "window_size must be even, in [2, 5000] and <= m");
    cudaStream_t st = g->stream;
    std::vector<float> gm(m), gw(m);
    CUDA_TRY(cudaMemcpyAsync(gm.data(), g->gm.p, m * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaMemcpyAsync(gw.data(), g->w.p, m * sizeof(float), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    const std::vector<int64_t> var = lmm_variants(gm, n, num_qf);
    const int k = (int)var.size();
    *count = k;
    if (k == 0) return;
    std::copy(var.begin(), var.end(), variants);
    const int64_t K_tiles = g->n_pad / kTileK;
    // centred counts of the sampled markers, x'Py, then v = P(rr∘x)
    DevBuf d_rows(st), d_V(st), d_X(st), d_py(st), d_sc(st);
    d_rows.ensure(k * sizeof(int64_t));
    CUDA_TRY(cudaMemcpyAsync(d_rows.p, var.data(), k * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    float* V = (float*)d_V.ensure((size_t)n * k * sizeof(float));
    float* X = (float*)d_X.ensure((size_t)n * k * sizeof(float));
    float* py = (float*)d_py.ensure(n * sizeof(float));
    double* sc = (double*)d_sc.ensure((size_t)4 * k * sizeof(double));
    DevBuf d_qt(st);
    double* qtv = (double*)d_qt.ensure((size_t)g->c * k * sizeof(double));
    CUDA_TRY(cudaMemcpyAsync(py, Py, n * sizeof(float), cudaMemcpyHostToDevice, st));
    centred_rows_kernel<<<dim3((unsigned)ceil_div(n, 256), k), 256, 0, st>>>(
        g->G.as<uint32_t>(), K_tiles, d_rows.as<int64_t>(), 0, g->gm.as<float>(), nullptr, n, V, n);
    LAUNCH_CHECK();
    col_dots(g, V, n, py, 0, n, k, sc);   // every column against Py
    scale_rows_rr_kernel<<<dim3((unsigned)ceil_div(n, 256), k), 256, 0, st>>>(V, n, g->rr.as<float>(), n);
    LAUNCH_CHECK();
    proj_coeffs(g, V, n, k, qtv);
    proj_apply(g, V, n, k, qtv);
    // x'Px through one projected Lanczos seed and a solve at shift 0; x'Sx = ‖v‖²
    slemm_lseed* S = lanczos_seed_device(g, SLEMM_OP_QUADFORM, tau1, V, k, tol_L, 600, false, {}, 5, 0);
    std::unique_ptr<slemm_lseed, void (*)(slemm_lseed*)> hold(S, lseed_free);
    lanczos_solve_device(S, 0.0, 1e-6, X, n, 0);
    col_dots(g, V, n, X, n, n, k, sc + k);
    col_dots(g, V, n, nullptr, 0, n, k, sc + 2 * k);
    // windows: the projected Gram of each marker's window, its own row of it kept as z
    const int ws = window_size;
    DevBuf d_gram(st), d_d(st), d_q(st), d_status(st), d_idx(st);
    const int64_t rows_max = round_up(ws, kPadRows) + kPadRows;
    const int64_t stride = rows_max * (ws + 1);   // ws rows and the room for z
    float* gram = (float*)d_gram.ensure((size_t)k * stride * sizeof(float));
    const float* rr = g->rr_one ? nullptr : g->rr.as<float>();
    const ExactCols cols{nullptr, rr, g->Q.as<float>(), g->n_pad, g->c};
    auto attempt = [&](int guess) {   // false: the guess was too small (exact_dots)
      GramStatsBuf stats;
      gram_stats(g, g->gm.as<float>(), cols, guess, stats);
      take_xx_kernel<<<(unsigned)ceil_div(k, 128), 128, 0, st>>>(stats.s.xx, d_rows.as<int64_t>(), k, sc + 3 * k);
      LAUNCH_CHECK();
      const GramSide side{g->G.as<uint8_t>(), m, stats.s};
      std::vector<int64_t> idx((size_t)3 * k);   // offA | offZ | which
      std::vector<int> one(k, 1);
      std::vector<GramJob> jobs;
      std::vector<float> dd((size_t)k * ws);
      for (int c = 0; c < k; ++c) {
        const int64_t j = var[c];
        int64_t wds;
        if (j < ws / 2) wds = 0;
        else if (j > m - ws / 2) wds = m - ws;
        else wds = j - ws / 2;
        for (int t = 0; t < ws; ++t) dd[(size_t)c * ws + t] = tau1 / gw[wds + t];
        GramJob job{0, 0, wds, ws, gram + (size_t)c * stride};
        gram_rows(side, wds, ws, job);
        jobs.push_back(job);
        idx[c] = wds - job.r0;   // this window's Gram starts at row wds − r0 of its block
        idx[k + c] = (int64_t)c * (ws + 1);
        idx[2 * k + c] = j - wds;
      }
      HostKeep keep(st);
      gram_blocks(g, side, side, jobs, g->c, rr, rows_max, GramHalf::mirrored, keep);
      check_device_error(g);
      keep.waited();
      if (!exact_dots_done(g, cols, guess)) return false;
      // batched systems: q_c = zᵀ(ZᵀZ + D)⁻¹z
      float* dvec = (float*)d_d.ensure((size_t)k * ws * sizeof(float));
      const int nq = spd_quadform_blocks(ws);
      double* q = (double*)d_q.ensure((size_t)k * nq * sizeof(double));
      int* status = (int*)d_status.ensure(((size_t)k + 1) * sizeof(int));
      int64_t* didx = (int64_t*)d_idx.ensure(idx.size() * sizeof(int64_t));
      CUDA_TRY(cudaMemcpyAsync(dvec, dd.data(), dd.size() * sizeof(float), cudaMemcpyHostToDevice, st));
      CUDA_TRY(cudaMemcpyAsync(didx, idx.data(), idx.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st));
      CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
      CUDA_TRY(cudaMemcpyAsync(status + 1, one.data(), (size_t)k * sizeof(int), cudaMemcpyHostToDevice, st));
      spd_quadforms({gram, stride, gram + (size_t)ws * rows_max, didx, didx + k, status + 1, rows_max, ws, k, 1}, dvec,
                    didx + 2 * k, q, status, st);
      std::vector<double> h(4 * k), hq((size_t)k * nq);
      int hs = 0;
      CUDA_TRY(cudaMemcpyAsync(h.data(), sc, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(cudaMemcpyAsync(hq.data(), q, hq.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, st));
      CUDA_TRY(cudaStreamSynchronize(st));
      if (hs) SLEMM_THROW(SLEMM_ERR_NUMERIC, "a window's ZᵀZ + τ1·diag(1/gw) is not positive definite in FP32");
      for (int c = 0; c < k; ++c) {
        double qc = 0.0;
        for (int b = 0; b < nq; ++b) qc += hq[(size_t)c * nq + b];
        xPy[c] = (float)h[c];
        xPx[c] = (float)h[k + c];
        xSx[c] = (float)h[2 * k + c];
        xBx[c] = (float)((h[3 * k + c] - qc) / (double)tau1);   // ‖v‖² as the Gram blocks have it
      }
      return true;
    };
    if (!attempt(exact_dots_guess(g, cols))) attempt(0);
  });
}

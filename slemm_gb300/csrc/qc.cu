// qc.cu — marker quality control on the packed genotypes: minor-allele frequency and the exact
// Hardy–Weinberg test per SNP (src/input.cpp:388-394), and decoded count rows.
//
// MAF (src/weight.cpp:3-15): f = popcount/float(2n) over the kept individuals' 2n bits (a missing
// call counts as one set bit), maf = |[f > 0.5] − f| in FP32.
//
// HWE (src/snphwe.cpp:18 SNPHWE2, called as SNPHWE2(n1, n0, n2, midp) at src/input.cpp:20 with
// n2 = calls with both bits set, n1 = one bit set — hets and missing calls — and n0 = neither):
// the exact test of Wigginton, Cutler & Abecasis (2005).  With N calls and r rare alleles the het
// count h (parity of r) has, under HWE, P(h+2)/P(h) = 4·hom_r·hom_c / ((h+2)(h+1)), hom_r = (r−h)/2,
// hom_c = N − h − hom_r.  p = Σ_{P(h) ≤ P(obs)} P(h) / Σ_h P(h), with a relative tie tolerance of
// 1e-7; the mid-p variant subtracts P(obs)/2.  One thread per SNP works in FP64 relative to the
// mode of the distribution (unimodal, so the terms fall monotonically on both sides), walks each
// side outward and stops where a term is below 1e-18 of min(P(obs), P(mode)) — smaller terms
// cannot move the sums in FP64.  The reference stores the result as FP32 (VectorXf hwep).
//
// The marker QC, whose result is FP32, walks the same terms as double-float pairs (hwe_exact_df): at
// n = 100,000 a SNP has some 1,400 terms of one FP64 division and three more FP64 operations each,
// and GB300's FP64 pipe (two lanes per clock and SM) took 3.1 ms of a 6.3 ms load of 20,011 SNPs, which
// now takes 3.4 ms.  A pair carries about
// 46 bits, far more than the result's 24: 48,000 SNPs of 1,000 to 100,003 calls have the FP64 walk's bits.  It needs fewer than 2^22 calls and P(obs)/P(mode) ≥ 1e-18
// (the terms then stay in FP32's range); anything else takes the FP64 walk.
#include "internal.h"
#include "reduce.cuh"

namespace slemm {

__device__ __forceinline__ double hwe_up(int64_t h, int64_t rare, int64_t n)   // P(h+2)/P(h)
{
  const int64_t hr = (rare - h) / 2, hc = n - h - hr;
  return 4.0 * (double)hr * (double)hc / ((double)(h + 2) * (double)(h + 1));
}

__device__ double hwe_exact_p(int64_t het, int64_t hom1, int64_t hom2, int midp)
{
  const int64_t n = het + hom1 + hom2;
  if (n == 0) return midp ? 0.5 : 1.0;
  const int64_t rare = 2 * min64(hom1, hom2) + het;
  const int64_t hmax = min64(rare, 2 * n - rare);
  const int64_t par = rare & 1;
  int64_t h = (int64_t)((double)rare * (double)(2 * n - rare) / (double)(2 * n - 1));
  if ((h & 1) != par) h += (h + 1 <= hmax) ? 1 : -1;
  h = max64(par, min64(h, hmax));
  while (h + 2 <= hmax && hwe_up(h, rare, n) > 1.0) h += 2;
  while (h >= 2 && hwe_up(h - 2, rare, n) < 1.0) h -= 2;
  const int64_t mode = h;
  double pobs = 1.0;
  if (het > mode)
    for (int64_t k = mode; k < het && pobs > 0.0; k += 2) pobs *= hwe_up(k, rare, n);
  else
    for (int64_t k = mode; k > het && pobs > 0.0; k -= 2) pobs /= hwe_up(k - 2, rare, n);
  const double cut = pobs * (1.0 + 1e-7);
  const double stop = fmin(pobs, 1.0) * 1e-18;
  double tot = 1.0, tail = (1.0 <= cut) ? 1.0 : 0.0;
  double p = 1.0;
  for (int64_t k = mode; k + 2 <= hmax;) {
    p *= hwe_up(k, rare, n);
    k += 2;
    tot += p;
    if (p <= cut) tail += p;
    if (p < stop || p == 0.0) break;
  }
  p = 1.0;
  for (int64_t k = mode; k >= 2;) {
    p /= hwe_up(k - 2, rare, n);
    k -= 2;
    tot += p;
    if (p <= cut) tail += p;
    if (p < stop || p == 0.0) break;
  }
  if (midp) tail -= 0.5 * pobs;
  return fmin(1.0, tail / tot);
}

// a·b and a/b of normalised double-float pairs (a, b > 0), to about 2^−45
__device__ __forceinline__ DF df_norm(float hi, float lo)
{
  DF r;
  r.hi = __fadd_rn(hi, lo);
  r.lo = __fsub_rn(lo, __fsub_rn(r.hi, hi));
  return r;
}
__device__ __forceinline__ DF df_prod(float a, float b)   // exact
{
  DF r;
  r.hi = __fmul_rn(a, b);
  r.lo = __fmaf_rn(a, b, -r.hi);
  return r;
}
__device__ __forceinline__ DF df_mul(const DF& a, const DF& b)
{
  const float p = __fmul_rn(a.hi, b.hi);
  return df_norm(p, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.hi, b.hi, -p))));
}
__device__ __forceinline__ DF df_div(const DF& a, const DF& b)
{
  const float r = __frcp_rn(b.hi), q = __fmul_rn(a.hi, r);
  const float e = __fadd_rn(__fmaf_rn(-q, b.hi, a.hi), __fmaf_rn(-q, b.lo, a.lo));
  return df_norm(q, __fmul_rn(e, r));
}
__device__ __forceinline__ bool df_le(const DF& a, const DF& b) { return a.hi < b.hi || (a.hi == b.hi && a.lo <= b.lo); }

// P(h+2)/P(h) = (2·hom_r)(2·hom_c) / ((h+2)(h+1)); down: its reciprocal.  Fewer than 2^22 calls: exact products.
__device__ __forceinline__ DF hwe_ratio(int h, int rare, int n, bool down)
{
  const int hr = (rare - h) / 2, hc = n - h - hr;
  const DF num = df_prod((float)(2 * hr), (float)(2 * hc)), den = df_prod((float)(h + 2), (float)(h + 1));
  return down ? df_div(den, num) : df_div(num, den);
}

// hwe_exact_p in double-float pairs by two neighbouring lanes, one per side of the mode (lane bit 0; `pair`:
// their mask); both return the same.  False when the case is out of its range.
__device__ bool hwe_exact_df(int64_t het64, int64_t hom1, int64_t hom2, int midp, bool down, unsigned pair, float* out)
{
  const int64_t n64 = het64 + hom1 + hom2;
  if (n64 == 0 || n64 >= (1 << 22)) return false;
  const int n = (int)n64, het = (int)het64, rare = 2 * (int)min64(hom1, hom2) + het;
  const int hmax = min(rare, 2 * n - rare), par = rare & 1;
  int h = (int)((double)rare * (double)(2 * n - rare) / (double)(2 * n - 1));
  if ((h & 1) != par) h += (h + 1 <= hmax) ? 1 : -1;
  h = max(par, min(h, hmax));
  auto up_cmp = [&](int x) {   // sign of P(x+2)/P(x) − 1, in integers
    const int64_t hr = (rare - x) / 2, hc = n - x - hr;
    return 4 * hr * hc - (int64_t)(x + 2) * (x + 1);
  };
  while (h + 2 <= hmax && up_cmp(h) > 0) h += 2;
  while (h >= 2 && up_cmp(h - 2) < 0) h -= 2;
  const int mode = h;
  DF one;
  one.hi = 1.f;
  DF pobs = one;
  constexpr float kLeast = 1e-18f;
  if (het > mode)
    for (int k = mode; k < het && pobs.hi >= kLeast; k += 2) pobs = df_mul(pobs, hwe_ratio(k, rare, n, false));
  else
    for (int k = mode; k > het && pobs.hi >= kLeast; k -= 2) pobs = df_mul(pobs, hwe_ratio(k - 2, rare, n, true));
  if (!(pobs.hi >= kLeast)) return false;
  const DF cut = df_norm(pobs.hi, __fmaf_rn(pobs.hi, 1e-7f, pobs.lo));
  const float stop = fminf(pobs.hi, 1.f) * 1e-18f;
  // this lane's side of the mode, four terms at a time: their ratios do not depend on one another, so only
  // the products are a chain (terms past the end have ratio 0)
  DF tot, tail, p = one;
  auto add = [](DF& s, const DF& v) {
    df_add(s, v.hi);
    s.lo = __fadd_rn(s.lo, v.lo);
  };
  const int terms = down ? mode / 2 : (hmax - mode) / 2;
  for (int t = 0; t < terms; t += 4) {
    DF r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (t + q < terms) r[q] = hwe_ratio(down ? mode - 2 * (t + q) - 2 : mode + 2 * (t + q), rare, n, down);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      p = df_mul(p, r[q]);
      add(tot, p);
      if (df_le(p, cut)) add(tail, p);
    }
    if (p.hi < stop) break;
  }
  // both sides and the mode's own term
  for (DF* s : {&tot, &tail}) {
    DF o;
    o.hi = __shfl_xor_sync(pair, s->hi, 1);
    o.lo = __shfl_xor_sync(pair, s->lo, 1);
    add(*s, o);
  }
  add(tot, one);
  if (df_le(one, cut)) add(tail, one);
  if (midp) {
    df_add(tail, -0.5f * pobs.hi);
    tail.lo = __fmaf_rn(-0.5f, pobs.lo, tail.lo);
  }
  *out = (float)fmin(1.0, df_value(tail) / df_value(tot));
  return true;
}

__global__ void hwe_kernel(const int32_t* __restrict__ het, const int32_t* __restrict__ hom1,
                           const int32_t* __restrict__ hom2, int64_t m, int midp, double* __restrict__ p)
{
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) p[j] = hwe_exact_p(het[j], hom1[j], hom2[j], midp);
}

// From the per-row counts of the G copy: maf (FP32, reference formula) and the HWE p-value; two lanes per
// SNP.
__global__ void marker_qc_kernel(const int64_t* __restrict__ pc, const int32_t* __restrict__ c1,
                                 const int32_t* __restrict__ c2, int64_t m, int64_t n, int midp,
                                 float* __restrict__ maf, float* __restrict__ hwep)
{
  const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 1;
  if (j >= m) return;   // both lanes of a pair
  const int64_t n1 = c1[j], n2 = c2[j], n0 = n - n1 - n2;
  float p;
  const bool fine = hwe_exact_df(n1, n0, n2, midp, threadIdx.x & 1, 3u << (threadIdx.x & 30), &p);
  if (threadIdx.x & 1) return;
  const float f = (float)(int)pc[j] / (float)(2 * n);
  maf[j] = fabsf((f > 0.5f ? 1.0f : 0.0f) - f);
  hwep[j] = fine ? p : (float)hwe_exact_p(n1, n0, n2, midp);
}

// out[c·ld + i] = count of SNP rows[c] for kept individual i (i < n), from the G copy (at packed
// position map[i] for a trait view, else i).
__global__ void genotype_rows_kernel(const uint32_t* __restrict__ G, int64_t K_tiles, const int64_t* __restrict__ rows,
                                     int64_t n, const int32_t* __restrict__ map, float* __restrict__ out, int64_t ld)
{
  const int c = blockIdx.y;
  const int64_t iv = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (iv >= n) return;
  const int64_t i = map ? (int64_t)map[iv] : iv;
  const int64_t j = rows[c];
  const int64_t mt = j / 128, r = j % 128, kt = i / 64, e = i % 64;
  const uint32_t w = G[((mt * K_tiles + kt) * 128 + r) * 4 + e / 16];
  const int q = (int)(e % 16);
  const int sh = (q & 1) ? 16 + (q & ~1) : q;   // even element 2p at bits 2p, odd 2p+1 at 16+2p
  out[(int64_t)c * ld + iv] = (float)((w >> sh) & 3u);
}

}  // namespace slemm

using namespace slemm;

extern "C" {

int slemm_gpu_hwe_exact(const int32_t* het, const int32_t* hom1, const int32_t* hom2, int64_t m, int midp,
                        double* p)
{
  return guarded([&] {
    CHECK_ARG(m >= 0, "m < 0");
    if (m == 0) return;
    CHECK_ARG(het && hom1 && hom2 && p, "null argument");
    for (int64_t j = 0; j < m; ++j)
      CHECK_ARG(het[j] >= 0 && hom1[j] >= 0 && hom2[j] >= 0, "negative genotype count");
    DevBuf d;
    int32_t* dc = (int32_t*)d.ensure((size_t)m * (3 * sizeof(int32_t) + sizeof(double)) + sizeof(double));
    double* dp = reinterpret_cast<double*>(dc + 3 * m + (m & 1));   // 8-byte aligned
    CUDA_TRY(cudaMemcpy(dc, het, m * sizeof(int32_t), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(dc + m, hom1, m * sizeof(int32_t), cudaMemcpyHostToDevice));
    CUDA_TRY(cudaMemcpy(dc + 2 * m, hom2, m * sizeof(int32_t), cudaMemcpyHostToDevice));
    hwe_kernel<<<(unsigned)ceil_div(m, 128), 128>>>(dc, dc + m, dc + 2 * m, m, midp ? 1 : 0, dp);
    LAUNCH_CHECK();
    CUDA_TRY(cudaMemcpy(p, dp, m * sizeof(double), cudaMemcpyDeviceToHost));
  });
}

int slemm_gpu_marker_qc(slemm_geno* g, int midp, float* maf, float* hwep)
{
  return guarded([&] {
    CHECK_ARG(g != nullptr && maf != nullptr && hwep != nullptr, "null argument");
    const int64_t m = g->m;
    DevBuf buf(g->stream);
    uint8_t* b = (uint8_t*)buf.ensure((size_t)m * (sizeof(int64_t) + 2 * sizeof(int32_t) + 2 * sizeof(float)) + 64);
    int64_t* d_pc = reinterpret_cast<int64_t*>(b);
    int32_t* d_c1 = reinterpret_cast<int32_t*>(d_pc + m);
    int32_t* d_c2 = d_c1 + m;
    float* d_maf = reinterpret_cast<float*>(d_c2 + m);
    float* d_hwe = d_maf + m;
    row_counts_device(g, d_pc, d_c1, d_c2);
    marker_qc_kernel<<<(unsigned)ceil_div(2 * m, 128), 128, 0, g->stream>>>(d_pc, d_c1, d_c2, m, g->n, midp ? 1 : 0,
                                                                        d_maf, d_hwe);
    LAUNCH_CHECK();
    CUDA_TRY(cudaMemcpyAsync(maf, d_maf, m * sizeof(float), cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaMemcpyAsync(hwep, d_hwe, m * sizeof(float), cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
  });
}

int slemm_gpu_genotype_rows(slemm_geno* g, const int64_t* rows, int cnt, float* out, int64_t ld, int mem)
{
  return guarded([&] {
    CHECK_ARG(g != nullptr && rows != nullptr && out != nullptr, "null argument");
    CHECK_ARG(cnt >= 1 && cnt <= 65535 && ld >= g->n, "bad count or leading dimension");
    for (int c = 0; c < cnt; ++c) CHECK_ARG(rows[c] >= 0 && rows[c] < g->m, "SNP index out of range");
    DevBuf d_rows(g->stream), d_out(g->stream);
    d_rows.ensure(cnt * sizeof(int64_t));
    CUDA_TRY(cudaMemcpyAsync(d_rows.p, rows, cnt * sizeof(int64_t), cudaMemcpyHostToDevice, g->stream));
    float* dst = out;
    int64_t ldd = ld;
    if (mem == SLEMM_MEM_HOST) {
      dst = (float*)d_out.ensure((size_t)g->n * cnt * sizeof(float));
      ldd = g->n;
    }
    genotype_rows_kernel<<<dim3((unsigned)ceil_div(g->n, 256), cnt), 256, 0, g->stream>>>(
        g->G.as<uint32_t>(), g->n_pad / kTileK, d_rows.as<int64_t>(), g->n,
        g->is_view ? g->ind_map.as<int32_t>() : nullptr, dst, ldd);
    LAUNCH_CHECK();
    if (mem == SLEMM_MEM_HOST)
      CUDA_TRY(cudaMemcpy2DAsync(out, ld * sizeof(float), dst, g->n * sizeof(float), g->n * sizeof(float), cnt,
                                 cudaMemcpyDeviceToHost, g->stream));
    CUDA_TRY(cudaStreamSynchronize(g->stream));
  });
}

}  // extern "C"

// gram.cu — projected Gram blocks of SNP rows, and the batched factorisation of their systems
// (the windows of --lmm and the blocks of slemm_gwa).
//
// With P = I − QQᵀ, z_j = x_j − a_j the centred counts of SNP j and t_j = Qᵀ(rr∘z_j),
//   G_jk = (P(rr∘z_j))ᵀ(P(rr∘z_k)) = Σ_i rr_i²·x_ij·z_ik − a_j·h_k − t_jᵀt_k,   h_k = Σ_i rr_i²·z_ik.
// h and t come from one exact pass over the packed matrix (gram_stats), so a Gram block is one
// packed product of SNP rows with columns that are read straight from the packed rows, and no
// dense FP32 column of n individuals is ever formed.  With residual weights the columns are rr²∘z_k − f_k
// in FP16 hi+lo at each column's own scale, f_k = 0 or their mean h_k/n where that is large, and
//   Σ_i rr_i²·x_ij·z_ik = Σ_i x_ij·(rr_i²·z_ik − f_k) + p_j·f_k,   p_j = Σ_i x_ij;
// with every rr 1 they are the counts themselves, one E4M3 byte each, whose product is an exact integer, and
// f_k = −a_k.  Forming U = rr∘P(rr∘z) as FP32 columns instead (centre, project, scale, measure, split: nine
// passes over n × columns floats) took 38 of the 82 ms of slemm_gwa at n = 50,021 with 20,011 variants and 4,000
// model SNPs, and 31 of the 73 ms of --lmm with 30 windows of 1,000 SNPs at n = 50,000; the two calls now
// take 3.2 and 6.0 ms (7.2 and 9.7 with residual weights).  With 600 variants in 20,000 individuals of weights 1 and
// 1/100, half of them in the light individuals alone, the median error of slemm_gwa's xx is 1.3e-7 (3.5e-6 with
// one scale for all columns, a = gm and t as single floats; 1.2e-6 with the dense columns).
#include "gram.h"
#include "decode.cuh"
#include "reduce.cuh"

#include <cfloat>

namespace slemm {

// ---- per-SNP statistics ------------------------------------------------------------------------
// bound[j] = max_i rr_i²·|x_ij − a_j| (as the bits of a float, to a few units in the last place), zero at first: the
// range of SNP j's column.  One thread per row of a tile and a share of the K-tiles; a count is the subnormal
// x·2^(2s−149) of its masked bits (gemm_simt.cu), so an individual costs a LOP, an FMA, a product and half of a
// three-way maximum.  A single bound 2·max rr² for all columns cost rare variants in individuals of small weight the
// bits that lie between.
constexpr int kBoundTiles = 8;
__global__ void __launch_bounds__(kTileM)
gram_bound_kernel(const uint4* __restrict__ G, int64_t K_tiles, const float* __restrict__ a, const float* __restrict__ rr,
                  int64_t m, int tiles_per_block, unsigned* __restrict__ bound)
{
  __shared__ __align__(16) float r2[kBoundTiles * kTileK];   // rr²·2^49
  const int64_t j = (int64_t)blockIdx.x * kTileM + threadIdx.x;
  const float na = j < m ? __fmul_rn(-a[j], 1.7763568394002505e-15f) : 0.f;   // −a·2^−49
  const int64_t kt0 = (int64_t)blockIdx.y * tiles_per_block, kt1 = min64(K_tiles, kt0 + tiles_per_block);
  float most = 0.f;
  for (int64_t ks = kt0; ks < kt1; ks += kBoundTiles) {
    const int nt = (int)min64(kBoundTiles, kt1 - ks);
    __syncthreads();
    for (int q = threadIdx.x; q < nt * kTileK; q += kTileM) {
      const float r = rr[ks * kTileK + q];
      r2[q] = __fmul_rn(__fmul_rn(r, r), 562949953421312.f);
    }
    __syncthreads();
    for (int u = 0; u < nt; ++u) {
      const uint4 pk = G[((int64_t)blockIdx.x * K_tiles + ks + u) * kTileM + threadIdx.x];
      const uint32_t words[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint32_t top = words[w] >> 24;
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          const float4 r4 = *reinterpret_cast<const float4*>(&r2[u * kTileK + w * 16 + e]);
          const float r[4] = {r4.x, r4.y, r4.z, r4.w};
          float v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float k = __uint_as_float((uint32_t)(127 + 100 - 2 * f32sub_shift(e + q)) << 23);   // (x − a)·2^−49
            v[q] = __fmul_rn(r[q], __fmaf_rn(f32sub_of(words[w], top, e + q), k, na));
          }
          most = fmaxf(fmaxf(most, fabsf(v[0])), fabsf(v[1]));
          most = fmaxf(fmaxf(most, fabsf(v[2])), fabsf(v[3]));
        }
      }
    }
  }
  if (j < m) atomicMax(bound + j, __float_as_uint(most));
}

// sc of every SNP: |rr²·z − f|·2^e below 2^11 (ops.cu, split_exp); an infinite bound stands for 2^128
__global__ void __launch_bounds__(256)
gram_scale_kernel(const unsigned* __restrict__ bound, int64_t m, GramStats s)
{
  const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (j >= m) return;
  const double range = fmin((double)__uint_as_float(bound[j]), 3.4e38) * (1.0 + 1e-6) + fabs((double)s.f[j]);
  int E = 11;
  if (range > 0.0) frexp(range, &E);
  const int e = max(-120, min(120, 11 - E));
  s.sc[j] = make_float2(ldexpf(1.f, e), ldexpf(1.f, -e));
}

__global__ void __launch_bounds__(256)
gram_stats_kernel(const double* __restrict__ dots, const double* __restrict__ twos, const double* __restrict__ tot,
                  int64_t m, int64_t n, const int64_t* __restrict__ pc, const int32_t* __restrict__ n2,
                  const float* __restrict__ gmf, int yb, int cq, GramStats s)
{
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // ‖P(rr∘1)‖² = Σ rr² − Σ_l (Q_lᵀrr)² to FP32's rounding of Q: the projection takes the intercept out
  __shared__ bool intercept;
  const double R = twos != nullptr ? tot[yb + cq] : (double)n;   // the last column is rr²
  if (threadIdx.x < 32) {
    double v = 0.0;
    for (int l = threadIdx.x; l < cq; l += 32) v = fma(tot[yb + l], tot[yb + l], v);
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) intercept = fabs(R - v) <= 0x1p-22 * R;
  }
  __syncthreads();
  if (j >= m) return;
  const double p = (double)pc[j], gm = (double)gmf[j];
  const double S1 = twos != nullptr ? dots[(int64_t)(yb + cq) * m + j] : p;
  const double S2 = twos != nullptr ? twos[j] : 2.0 * (double)n2[j];
  // With the intercept projected out any constant may be taken off a count.  The weighted mean leaves the projection
  // nothing to cancel (with gm it took h²/R of ‖rr∘z‖², more than half where genotypes go with the weights), and as
  // a multiple of 2^−23 it has exact FP32 differences 1 − a and 2 − a.  Else a is gm, and a large mean of rr²∘z (h²/R
  // over a fifth of ‖rr∘z‖²) is taken off the stored columns.
  const double h0 = S1 - gm * R, zz0 = (S1 + S2) - 2.0 * gm * S1 + gm * gm * R;
  const float af = intercept ? (float)(rint(S1 / R * 0x1p23) * 0x1p-23) : gmf[j];
  const double a = (double)af, h = S1 - a * R;
  double xx = (S1 + S2) - 2.0 * a * S1 + a * a * R;
  float x, y;
  for (int l = 0; l < cq; ++l) {
    const double t = dots[(int64_t)(yb + l) * m + j] - a * tot[yb + l];
    split_double(t, x, y);
    s.t[(int64_t)l * s.ld + j] = make_float2(x, y);
    xx -= t * t;
  }
  split_double(h, x, y);
  s.h[j] = make_float2(x, y);
  split_double(p, x, y);
  s.p[j] = make_float2(x, y);
  s.a[j] = af;
  s.f[j] = twos == nullptr ? -af : !intercept && 5.0 * h0 * h0 > R * zz0 ? (float)(h / (double)n) : 0.f;
  s.sc[j] = make_float2(1.f, 1.f);
  s.xy[j] = yb ? dots[j] - gm * tot[0] : 0.0;
  s.xx[j] = xx;
}

void gram_stats(slemm_geno* g, const float* gm, const ExactCols& cols, int guess, GramStatsBuf& out)
{
  cudaStream_t st = g->stream;
  const int64_t m = g->m;
  const float* rr = cols.rr;
  const int C = cols.count(), cq = cols.cq;
  DevBuf d(st), dc(st);
  double* dots = (double*)d.ensure(((size_t)(C + 1) * m + C) * sizeof(double));
  double* twos = rr ? dots + (size_t)C * m : nullptr;
  double* tot = dots + (size_t)(C + 1) * m;
  int64_t* pc = (int64_t*)dc.ensure((size_t)m * (sizeof(int64_t) + 2 * sizeof(int32_t)));
  int32_t* n1 = reinterpret_cast<int32_t*>(pc + m);
  row_counts_device(g, pc, n1, n1 + m);
  if (C > 0) exact_dots(g, cols, dots, tot, twos, guess);
  const GramStats s = out.make(m, cq, st);
  gram_stats_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>(dots, twos, tot, m, g->n, pc, n1 + m, gm, cols.y ? 1 : 0, cq,
                                                                 s);
  LAUNCH_CHECK();
  if (rr == nullptr) return;
  DevBuf db(st);
  unsigned* bound = (unsigned*)db.ensure((size_t)m * sizeof(unsigned));
  CUDA_TRY(cudaMemsetAsync(bound, 0, (size_t)m * sizeof(unsigned), st));
  const int64_t K_tiles = g->n_pad / kTileK, M_tiles = g->m_pad / kTileM;
  // twelve blocks an SM run at once; shares of whole stages
  const int64_t stages = ceil_div(K_tiles, kBoundTiles), shares = std::min(stages, ceil_div(12 * num_sms(), M_tiles));
  const int per = (int)ceil_div(stages, shares) * kBoundTiles;
  gram_bound_kernel<<<dim3((unsigned)M_tiles, (unsigned)ceil_div(K_tiles, per)), kTileM, 0, st>>>(
      g->G.as<uint4>(), K_tiles, s.a, rr, m, per, bound);
  LAUNCH_CHECK();
  gram_scale_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, st>>>(bound, m, s);
  LAUNCH_CHECK();
}

// dst SNP k = src SNP idx[k]
__global__ void gram_stats_gather_kernel(GramStats src, const int64_t* __restrict__ idx, int64_t cnt, int cq, GramStats dst)
{
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const int64_t j = idx[k];
  dst.a[k] = src.a[j];
  dst.h[k] = src.h[j];
  dst.p[k] = src.p[j];
  dst.f[k] = src.f[j];
  dst.sc[k] = src.sc[j];
  dst.xy[k] = src.xy[j];
  dst.xx[k] = src.xx[j];
  for (int l = 0; l < cq; ++l) dst.t[(int64_t)l * dst.ld + k] = src.t[(int64_t)l * src.ld + j];
}

void gram_stats_gather(const GramStats& src, const int64_t* d_idx, int64_t cnt, int cq, GramStatsBuf& out, cudaStream_t st)
{
  const GramStats s = out.make(cnt, cq, st);
  gram_stats_gather_kernel<<<(unsigned)ceil_div(cnt, 256), 256, 0, st>>>(src, d_idx, cnt, cq, s);
  LAUNCH_CHECK();
}

// ---- Gram blocks ----------------------------------------------------------------------------------
// A block's columns go in groups of at most kp; a launch takes groups of several blocks.  The operand of a
// group are the columns SNP c0 … c0 + nc − 1, row c of kp each; rows nc … kp − 1 only reach sums that
// nobody reads and stay as they are.
struct GramGroup {
  int64_t r0, nrows;   // SNP of the product's first row, rows that exist
  int64_t c0, nc;      // SNP of the group's first column, columns
  int64_t b0, bc;      // the block's first column's SNP and columns
  float* out;          // the block's first column
};
//
// Every rr 1: N = kp rows of counts as E4M3 bytes in the decoded order of the matrix's own words
// (decode.cuh), so the product takes one MMA per 32 individuals and its sums are exact integers.  One
// word (16 individuals) per thread; a count x ∈ {0, 1, 2} in a byte is x·0x38 − [x = 2]·0x30 (E4M3 0, 1,
// 2), or x·0x28 − [x = 2]·0x20 times 2^−2, four at a time.  Bound by the bytes it writes.
constexpr int kCountRows = 8;   // rows of one thread: with one, the turnover of blocks bound it (378 µs for 27,000 columns
                                // of slemm_gwa at n = 50,021, 244 now, 5.5 TB/s)
__global__ void __launch_bounds__(256)
gram_counts_kernel(const uint32_t* __restrict__ G, int64_t K_tiles, const GramGroup* __restrict__ groups, int kp,
                   uint8_t* __restrict__ B)
{
  const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x;   // word of the row
  if (q >= K_tiles * 4) return;
  const int grp = blockIdx.z, r0 = blockIdx.y * kCountRows;
  const int64_t nc = groups[grp].nc, c0 = groups[grp].c0;
  uint32_t w[kCountRows];
#pragma unroll
  for (int e = 0; e < kCountRows; ++e) {
    const int64_t j = c0 + r0 + e;
    w[e] = r0 + e < nc ? G[((j / 128 * K_tiles + (q >> 2)) * 128 + j % 128) * 4 + (q & 3)] : 0u;
  }
#pragma unroll
  for (int e = 0; e < kCountRows; ++e) {
    if (r0 + e >= nc) return;
    uint32_t v[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t x = (w[e] >> (2 * p)) & 0x03030303u, two = (x >> 1) & 0x01010101u;
      v[p] = (p & 1) ? x * 0x28u - two * 0x20u : x * 0x38u - two * 0x30u;
    }
    *reinterpret_cast<uint4*>(B + ((int64_t)grp * kp + r0 + e) * K_tiles * kTileK + q * 16) = make_uint4(v[0], v[1], v[2], v[3]);
  }
}

// With residual weights: N = 2·kp rows, FP16 pieces hi and lo of (rr²·z − f)·2^e, each times the 2^−2s of its K
// position (f16sub_pair_of).  A thread writes 8 K-elements (half of a packed word): 16-byte stores, 512
// contiguous bytes per warp.  Bound by the 16-bit operand it writes.
__global__ void __launch_bounds__(256)
gram_operand_kernel(const uint32_t* __restrict__ G, int64_t K_tiles, const GramGroup* __restrict__ groups, int kp,
                    GramStats cs, const float* __restrict__ rr, __half* __restrict__ B)
{
  const int64_t q8 = (int64_t)blockIdx.x * 256 + threadIdx.x;   // K-elements 8·q8 …
  const int64_t K_pad = K_tiles * kTileK;
  if (q8 * 8 >= K_pad) return;
  const int grp = blockIdx.z, r = blockIdx.y;
  if (r >= groups[grp].nc) return;
  __half* dst = B + ((int64_t)grp * 2 * kp + r) * K_pad + q8 * 8;
  uint4 hi, lo;
  {
    const int64_t j = groups[grp].c0 + r, kt = q8 >> 3;
    const int w = (int)(q8 & 7) >> 1, h = (int)(q8 & 1);
    const uint32_t word = G[((j / 128 * K_tiles + kt) * 128 + j % 128) * 4 + w];
    float zv[3], rv[8];
    const float a = cs.a[j], f = cs.f[j], scale = cs.sc[j].x;
#pragma unroll
    for (int x = 0; x < 3; ++x) zv[x] = __fsub_rn((float)x, a);
    const float4 r0 = *reinterpret_cast<const float4*>(rr + q8 * 8);
    const float4 r1 = *reinterpret_cast<const float4*>(rr + q8 * 8 + 4);
    rv[0] = r0.x, rv[1] = r0.y, rv[2] = r0.z, rv[3] = r0.w;
    rv[4] = r1.x, rv[5] = r1.y, rv[6] = r1.z, rv[7] = r1.w;
    uint32_t ph[4], pl[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {   // element pair q = 4h + p of the word
      const int q = 4 * h + p, s = f16sub_shift(q);
      const uint32_t xe = (word >> (2 * q)) & 3u, xo = (word >> (16 + 2 * q)) & 3u;
      const float ks = __uint_as_float((uint32_t)(127 - 2 * s) << 23);
      const float ze = xe == 0 ? zv[0] : xe == 1 ? zv[1] : zv[2], zo = xo == 0 ? zv[0] : xo == 1 ? zv[1] : zv[2];
      const float ve = __fmul_rn(__fmaf_rn(__fmul_rn(rv[2 * p], rv[2 * p]), ze, -f), scale);
      const float vo = __fmul_rn(__fmaf_rn(__fmul_rn(rv[2 * p + 1], rv[2 * p + 1]), zo, -f), scale);
      const float he = rintf(ve), ho = rintf(vo);
      ph[p] = (uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(he, ks))) |
              ((uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(ho, ks))) << 16);
      pl[p] = (uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(__fsub_rn(ve, he), ks))) |
              ((uint32_t)__half_as_ushort(__float2half_rn(__fmul_rn(__fsub_rn(vo, ho), ks))) << 16);
    }
    hi = make_uint4(ph[0], ph[1], ph[2], ph[3]);
    lo = make_uint4(pl[0], pl[1], pl[2], pl[3]);
  }
  *reinterpret_cast<uint4*>(dst) = hi;
  *reinterpret_cast<uint4*>(dst + (int64_t)kp * K_pad) = lo;
}

// 2^−e_c·Σ_splits D − a_row·h_c + p_row·f_c − t_rowᵀt_c of product row i (SNP r) and column cc of group grp
// (SNP c); double-float sums.
__device__ __forceinline__ float gram_entry(const float* __restrict__ D, int splits, int kp, int64_t rows, int64_t i, int grp,
                                            int cc, const GramStats& rs, int64_t r, const GramStats& cs, int64_t c,
                                            int cq)
{
  const float* Dc = D + ((int64_t)grp * splits * kp + cc) * rows + i;
  DF a;
  const float isc = cs.sc[c].y;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) df_add(a, __fmul_rn(Dc[(int64_t)s * kp * rows], isc));
  const float2 h = cs.h[c], p = rs.p[r];
  const float ar = rs.a[r], f = cs.f[c];
  df_fma(a, -ar, h.x);
  df_fma(a, p.x, f);
  a.lo = __fmaf_rn(-ar, h.y, __fmaf_rn(p.y, f, a.lo));
  for (int l = 0; l < cq; ++l) {
    const float2 tr = rs.t[(int64_t)l * rs.ld + r], tc = cs.t[(int64_t)l * cs.ld + c];
    df_fma(a, -tr.x, tc.x);
    a.lo = __fmaf_rn(-tr.x, tc.y, __fmaf_rn(-tr.y, tc.x, a.lo));
  }
  return __fadd_rn(a.hi, a.lo);
}

// out[c·ldo + i] of every product row i and column c of the groups (blockIdx.z).
__global__ void __launch_bounds__(256)
gram_finish_kernel(const float* __restrict__ D, int splits, int kp, int64_t rows, GramStats rs, GramStats cs,
                   const GramGroup* __restrict__ groups, int cq, int64_t ldo)
{
  const GramGroup G = groups[blockIdx.z];
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i >= G.nrows || c >= G.nc) return;
  G.out[(G.c0 - G.b0 + c) * ldo + i] = gram_entry(D, splits, kp, rows, i, blockIdx.z, (int)c, rs, G.r0 + i, cs, G.c0 + c, cq);
}

// The same of blocks of a symmetric product, for the entries with r0 + i ≤ c0 + c; with `mirror` each of them
// also at the other half's place, product row c0 + c − r0 and column r0 + i − b0 (where that is one of the
// block's columns), through shared memory so that both writes are whole lines.
__global__ void __launch_bounds__(256)
gram_finish_sym_kernel(const float* __restrict__ D, int splits, int kp, int64_t rows, GramStats st,
                       const GramGroup* __restrict__ groups, int cq, int64_t ldo, int mirror)
{
  __shared__ float tile[32][33];
  const GramGroup G = groups[blockIdx.z];
  const int64_t i0 = (int64_t)blockIdx.x * 32, ct = (int64_t)blockIdx.y * 32;
  // past the rows, the columns or every column's SNP
  if (i0 >= G.nrows || ct >= G.nc || G.r0 + i0 > G.c0 + min64(ct + 31, G.nc - 1)) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t i = i0 + x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t c = ct + y + 8 * q;
    if (i >= G.nrows || c >= G.nc || G.r0 + i > G.c0 + c) continue;
    const float v = gram_entry(D, splits, kp, rows, i, blockIdx.z, (int)c, st, G.r0 + i, st, G.c0 + c, cq);
    G.out[(G.c0 - G.b0 + c) * ldo + i] = v;
    tile[y + 8 * q][x] = v;
  }
  if (!mirror) return;
  __syncthreads();
  const int64_t c = ct + x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t k = i0 + y + 8 * q, col = G.r0 + k - G.b0;   // product row k becomes column col
    if (k < G.nrows && c < G.nc && G.r0 + k < G.c0 + c && col >= 0 && col < G.bc)
      G.out[col * ldo + G.c0 + c - G.r0] = tile[x][y + 8 * q];
  }
}

// Split-K count of a product of `ctas` CTAs without splits: the least time in K-tiles of a CTA, its waves
// times their K-tiles and what each split costs beside them (ramp, epilogue, and its partial sums written and
// read again by the finishing kernel).  Anything from 24 to 64 is within a percent at n = 7,000 to 50,000; 8,
// the ramp and epilogue alone, took 1 to 3 % more of the calls.
constexpr int64_t kSplitTiles = 32;
// Operand bytes of one launch.  Launches of many blocks' groups fill the GPU's last wave and take few splits,
// which is worth more than an operand that stays in L2: at 48, 96, 192 and 512 MB slemm_gwa (50,021 × 20,011, blocks of
// 1,000) takes 3.81, 3.57, 3.47 and 3.29 ms, with blocks of 100 (46,280 × 16,455) 1.92, 1.57, 1.46 and 1.45 ms
// (3.70 with a launch for each block), --lmm (50,000, 30 windows of 1,000) 6.81, 6.47, 6.32 and 6.13 ms (6.75).
constexpr int64_t kGramOperand = (int64_t)512 << 20;
static int gram_splits(int64_t ctas, int64_t K_tiles, int64_t min_splits)
{
  int64_t best = min_splits, best_cost = INT64_MAX;
  for (int64_t s = min_splits; s == min_splits || (K_tiles / s >= 48 && s <= 64); ++s) {
    const int64_t cost = ceil_div(ctas * s, num_sms()) * (ceil_div(K_tiles, s) + kSplitTiles);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return (int)best;
}

void gram_rows(const GramSide& R, int64_t s0, int64_t cnt, GramJob& job)
{
  const int64_t end = round_up(R.m, kPadRows);
  job.r0 = s0 / kTileM * kTileM;
  job.rows = round_up(s0 + cnt - job.r0, kPadRows);
  job.r0 = std::min(job.r0, end - job.rows);
  if (job.r0 < 0) {
    job.r0 = 0;
    job.rows = end;
  }
}

void gram_blocks(slemm_geno* g, const GramSide& R, const GramSide& C, const std::vector<GramJob>& jobs, int cq, const float* rr,
                 int64_t ldo, GramHalf half, HostKeep& keep)
{
  cudaStream_t st = g->stream;
  const int64_t K_pad = g->n_pad, K_tiles = K_pad / kTileK;
  const bool unit = rr == nullptr, sym = half != GramHalf::all;
  // N ≤ 160 keeps two row tiles, each with its own MMA-issuing thread, in one CTA
  const int most = unit ? 160 : 80;
  auto& groups = keep.make<std::vector<GramGroup>>();
  auto& tiles = keep.make<std::vector<int2>>();   // as GemmArgs::table
  int64_t widest = 0, rows = 0;
  for (const GramJob& j : jobs) {
    if (j.ncols <= 0) continue;
    CHECK_ARG(j.r0 % kTileM == 0 && j.rows % kPadRows == 0 && j.r0 + j.rows <= round_up(R.m, kPadRows), "row range not aligned");
    CHECK_ARG(!sym || (R.G == C.G && j.c0 >= j.r0 && j.c0 + j.ncols <= j.r0 + j.rows), "not a symmetric block");
    const int64_t kc = ceil_div(j.ncols, ceil_div(j.ncols, most));
    for (int64_t f = 0; f < j.ncols; f += kc) {
      const int64_t nc = std::min(kc, j.ncols - f);
      groups.push_back({j.r0, std::min(j.rows, R.m - j.r0), j.c0 + f, nc, j.c0, j.ncols, j.out});
      const int64_t wanted = sym ? std::min(j.rows, j.c0 + f + nc - j.r0) : j.rows;
      tiles.push_back(make_int2((int)(j.r0 / kTileM), (int)ceil_div(wanted, kTileM)));
    }
    widest = std::max(widest, kc);
    rows = std::max(rows, j.rows);
  }
  if (groups.empty()) return;
  const int kp = (int)round_up(widest, unit ? 16 : 8);
  const int N = unit ? kp : 2 * kp;
  const int plan = unit ? 2 : 0;
  const int64_t cta_tiles = gemm_tc_rows_per_cta(N, plan) / kTileM;
  DevBuf d_groups(st), d_tiles(st);
  GramGroup* dg = (GramGroup*)d_groups.ensure(groups.size() * sizeof(GramGroup));
  int2* dt = (int2*)d_tiles.ensure(tiles.size() * sizeof(int2));
  CUDA_TRY(cudaMemcpyAsync(dg, groups.data(), groups.size() * sizeof(GramGroup), cudaMemcpyHostToDevice, st));
  CUDA_TRY(cudaMemcpyAsync(dt, tiles.data(), tiles.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
  // As many groups per launch as kGramOperand of operand and 512 MB of a split's partials hold (at least one)
  const int64_t group_bytes = (int64_t)N * K_pad * (unit ? 1 : 2), total = (int64_t)groups.size();
  int64_t per = std::max<int64_t>(1, std::min({total, kGramOperand / group_bytes, ((int64_t)512 << 20) / ((int64_t)kp * rows * 4),
                                               (int64_t)65535}));
  per = ceil_div(total, ceil_div(total, per));   // launches of about the same size
  for (int64_t g0 = 0; g0 < total; g0 += per) {
    const int ng = (int)std::min(per, total - g0);
    int64_t live = 0;   // CTAs with work
    for (int z = 0; z < ng; ++z) live += ceil_div(tiles[g0 + z].y, cta_tiles);
    // an integer partial sum of 2^22 elements is at most 2^24: exact in FP32
    const int splits = gram_splits(live, K_tiles, ceil_div(K_pad, (int64_t)1 << 22));
    void* B = g->ws_B.ensure((size_t)ng * group_bytes);
    float* D = (float*)g->ws_D.ensure((size_t)ng * splits * kp * rows * sizeof(float));
    const uint32_t* Gc = reinterpret_cast<const uint32_t*>(C.G);
    if (unit)
      gram_counts_kernel<<<dim3((unsigned)ceil_div(K_pad / 16, 256), (unsigned)ceil_div(kp, kCountRows), ng), 256, 0, st>>>(
          Gc, K_tiles, dg + g0, kp, (uint8_t*)B);
    else
      gram_operand_kernel<<<dim3((unsigned)ceil_div(K_pad / 8, 256), kp, ng), 256, 0, st>>>(
          Gc, K_tiles, dg + g0, kp, C.stats, rr, (__half*)B);
    LAUNCH_CHECK();
    GemmArgs a{R.G, rows, K_pad, B, N, D, splits, g->err.as<int>(), kp, unit ? 1 : 2, !unit, plan};
    a.groups = ng;
    a.table = dt + g0;
    gemm_tc(a, st);
    if (sym)
      gram_finish_sym_kernel<<<dim3((unsigned)ceil_div(rows, 32), (unsigned)ceil_div(widest, 32), ng), 256, 0, st>>>(
          D, splits, kp, rows, R.stats, dg + g0, cq, ldo, half == GramHalf::mirrored ? 1 : 0);
    else
      gram_finish_kernel<<<dim3((unsigned)ceil_div(rows, 256), (unsigned)widest, ng), 256, 0, st>>>(
          D, splits, kp, rows, R.stats, C.stats, dg + g0, cq, ldo);
    LAUNCH_CHECK();
  }
}

// ---- batched factorisation ----------------------------------------------------------------------------
// System b is the s×s matrix M_b = A_b + diag(ridge_b) with t_b further rows Z_b below it, all rows
// FP32 and contiguous: row r < s at A + b·strideA + r·ld + offA[b], row s + r at
// Z + (offZ[b] + r)·ld + offA[b].  The right-looking panels of spd_panels turn the rows of A
// (strictly below each diagonal tile) into L's and the rows of Z into L⁻¹Z's columns,
// Z_r ← L⁻¹z_r: one TRSM and one update serve both, so the quadratic forms z_rᵀM⁻¹z_r are row norms
// of the result and a system's work spreads over all its row tiles.  The diagonal tiles' factors go
// to Ld (a panel's CTAs all read the tile, so it stays as it was); the upper triangle of A keeps the
// matrix.  One CTA per system factoring alone (a chain of 1,000 columns on one SM) took 20.4 ms for 7
// systems of 1,000 and its triangular solves another 13.4 ms.
constexpr int kPT = 128;   // panel width and row-tile height of the update

struct SpdRows {
  float* A;
  int64_t strideA;
  float* Z;
  const int64_t* offA;
  const int64_t* offZ;
  const int* t;
  int64_t ld;
  int s;
  // first element (column 0) of row r ≥ 0 of row tile `tile` counted from row c0 of A, or null past the
  // end; A's rows and Z's are tiled separately
  __device__ float* row(int b, int c0, int tile, int r) const
  {
    const int nA = (s - c0 + kPT - 1) / kPT;
    if (tile < nA) {
      const int i = c0 + tile * kPT + r;
      return i < s ? A + (int64_t)b * strideA + (int64_t)i * ld + offA[b] : nullptr;
    }
    const int i = (tile - nA) * kPT + r;
    return i < t[b] ? Z + (offZ[b] + i) * ld + offA[b] : nullptr;
  }
};

// Panel k0: every CTA factors the diagonal tile (tk ≤ 128 columns) and solves its own 256 rows against it
// in the same sweep: the values wait in shared memory, thread (tx, ty) keeps the sums of products of
// its rows' elements tx + 16q in both tiles, and a column, less its sums, is published through shared
// memory, one barrier per column.  Bound by that chain of 128 steps, not by its arithmetic: so the rows
// ride along instead of a launch of their own, and 512 threads on 256 rows (all of the SM's registers)
// halve the CTAs that repeat the diagonal tile and keep the panel in one wave (129 µs for 210 CTAs of 128
// rows and twice the instructions a step, 84 µs now).
constexpr int kPR = 256;   // rows of one CTA
constexpr size_t kPanelSmem = (size_t)(kPT + kPR) * kPT * sizeof(float);
__global__ void __launch_bounds__(512, 1)
spd_panel_kernel(SpdRows S, const float* __restrict__ ridge, int k0, float* __restrict__ Ld, int* __restrict__ status)
{
  extern __shared__ float tiles[];
  __shared__ __align__(16) float scol[2][kPT], srow[2][kPR];
  float* sD = tiles;               // [128][128]
  float* sR = tiles + kPT * kPT;   // [256][128]
  const int b = blockIdx.y, tile = blockIdx.x;
  const int tk = min(kPT, S.s - k0), c0 = k0 + tk;
  const int nA = (S.s - c0 + kPR - 1) / kPR;
  const int ntiles = nA + (S.t[b] + kPR - 1) / kPR;
  if (tile >= ntiles && tile > 0) return;
  // this CTA's rows: nrow of them from row0, S.ld apart
  const float* Ab = S.A + (int64_t)b * S.strideA + S.offA[b];
  const bool inA = tile < nA;
  const int i0 = inA ? c0 + tile * kPR : (tile - nA) * kPR;
  const int nrow = tile < ntiles ? min(kPR, (inA ? S.s : S.t[b]) - i0) : 0;
  float* row0 = (inA ? S.A + (int64_t)b * S.strideA : S.Z + S.offZ[b] * S.ld) + S.offA[b] + (int64_t)i0 * S.ld + k0;
#pragma unroll 16
  for (int e = threadIdx.x; e < kPT * kPT; e += 512) {
    const int i = e / kPT, j = e % kPT;
    float v = (i < tk && j <= i) ? Ab[(int64_t)(k0 + i) * S.ld + k0 + j] : 0.f;
    if (i == j) v = i < tk ? v + ridge[(int64_t)b * S.s + k0 + i] : 1.f;
    sD[e] = v;
  }
#pragma unroll 16
  for (int e = threadIdx.x; e < kPR * kPT; e += 512) {
    const int i = e / kPT, j = e % kPT;
    sR[e] = (i < nrow && j < tk) ? row0[(int64_t)i * S.ld + j] : 0.f;
  }
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // Σ l·l over the columns done so far; afterwards l itself.  Rows 4ty + a of D, rows 4ty + a and
  // 128 + 4ty + a of R: a column's values are read four rows at a time
  float D[4][8] = {}, R[8][8] = {};
  auto rrow = [&](int a) { return 4 * ty + (a & 3) + 128 * (a >> 2); };
  bool bad = false;
#pragma unroll
  for (int jb = 0; jb < 8; ++jb) {
    const bool below = 4 * ty + 3 >= 16 * jb;   // some of this thread's rows of D are not done
    for (int jj = 0; jj < 16; ++jj) {
      const int j = 16 * jb + jj, buf = jj & 1;
      if (tx == jj) {
#pragma unroll
        for (int a = 0; a < 4; ++a) scol[buf][4 * ty + a] = sD[(4 * ty + a) * kPT + j] - D[a][jb];
#pragma unroll
        for (int a = 0; a < 8; ++a) srow[buf][rrow(a)] = sR[rrow(a) * kPT + j] - R[a][jb];
      }
      __syncthreads();
      const float d = scol[buf][j];
      bad = bad || !(d > 0.f);
      // 1/√d to half a unit in the last place, by one Newton step with the residual 1 − d·inv² in two pieces (0 for an
      // infinite pivot, whose row the ridge takes out): the pivot's chain is in every step's way, and a square root and
      // a division (IEEE) are some 40 instructions of it
      float inv = rsqrtf(d);
      const float hi = d * inv, rest = fmaf(-fmaf(d, inv, -hi), inv, fmaf(-hi, inv, 1.f));
      inv = d <= FLT_MAX ? fmaf(inv * 0.5f, rest, inv) : inv;
      const float inv2 = inv * inv;   // l_i·l_k = v_i·(v_k·inv²) of the published values
      float lk[8];
#pragma unroll
      for (int q = jb; q < 8; ++q) lk[q] = scol[buf][tx + 16 * q] * inv2;
      const bool own = tx == jj;
      lk[jb] = tx > jj ? lk[jb] : 0.f;   // column tx + 16·jb lies right of j
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v4 = *reinterpret_cast<const float4*>(&srow[buf][128 * h + 4 * ty]);
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
          for (int q = jb; q < 8; ++q) R[4 * h + a][q] = fmaf(v[a], lk[q], R[4 * h + a][q]);
          R[4 * h + a][jb] = own ? v[a] * inv : R[4 * h + a][jb];
        }
      }
      if (below) {
        const float4 v4 = *reinterpret_cast<const float4*>(&scol[buf][4 * ty]);
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
          for (int q = jb; q < 8; ++q) D[a][q] = fmaf(v[a], lk[q], D[a][q]);
          D[a][jb] = own ? v[a] * inv : D[a][jb];   // v = d on the diagonal: d/√d
        }
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 8; ++a) {
    if (rrow(a) >= nrow) continue;
    float* r = row0 + (int64_t)rrow(a) * S.ld;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (tx + 16 * q < tk) r[tx + 16 * q] = R[a][q];
  }
  if (tile == 0) {
    if (bad && threadIdx.x == 0) atomicOr(status, 1);
    float* L = Ld + ((int64_t)b * ((S.s + kPT - 1) / kPT) + k0 / kPT) * kPT * kPT;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 8; ++q) L[(4 * ty + a) * kPT + tx + 16 * q] = (tx + 16 * q <= 4 * ty + a) ? D[a][q] : 0.f;
  }
}

// Trailing update after panel k0: C[I, J] −= P_I·P_Jᵀ over the panel's tk columns, for A's row tiles
// (J ≤ I, the lower triangle alone) and Z's (every J).  128×128 per CTA, 8×8 per thread (rows 4ty … and
// 64 + 4ty …, columns alike), the panels through shared memory 16 columns at a time, the next 16 loaded
// into registers meanwhile.  Operands are read four at a time: single words cost as many shared-memory
// cycles as the 64 FMAs they feed.  Bound by FP32 FMA issue.
constexpr int kUD = 16;          // panel columns of one stage
constexpr int kUS = kPT + 4;     // row stride of a staged column
__global__ void __launch_bounds__(256, 2)
spd_update_kernel(SpdRows S, int k0)
{
  __shared__ __align__(16) float Pa[kUD][kUS], Pb[kUD][kUS];
  const int b = blockIdx.y;
  const int tk = min(kPT, S.s - k0), c0 = k0 + tk;
  const int nA = (S.s - c0 + kPT - 1) / kPT;
  const int nZ = (S.t[b] + kPT - 1) / kPT;
  const int tri = nA * (nA + 1) / 2;
  const int q = blockIdx.x;
  int ti, tj;
  if (q < tri) {
    ti = (int)((sqrtf(8.f * (float)q + 1.f) - 1.f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= q) ++ti;
    while (ti * (ti + 1) / 2 > q) --ti;
    tj = q - ti * (ti + 1) / 2;
  } else {
    if (q - tri >= nA * nZ) return;
    ti = nA + (q - tri) / nA;
    tj = (q - tri) % nA;
  }
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // loads: panel column lu of rows lr, lr + 16, …
  const int lu = threadIdx.x & 15, lr = threadIdx.x >> 4;
  const float *base_a = S.row(b, c0, ti, 0), *base_b = S.row(b, c0, tj, 0);   // a tile has a first row
  const int rows_a = ti < nA ? min(kPT, S.s - c0 - ti * kPT) : min(kPT, S.t[b] - (ti - nA) * kPT);
  const int rows_b = min(kPT, S.s - c0 - tj * kPT);
  float na[8], nb[8];
  auto fetch = [&](int u0) {
    const bool cu = u0 + lu < tk;
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      const int r = lr + 16 * v;
      na[v] = (cu && r < rows_a) ? base_a[(int64_t)r * S.ld + k0 + u0 + lu] : 0.f;
      nb[v] = (cu && r < rows_b) ? base_b[(int64_t)r * S.ld + k0 + u0 + lu] : 0.f;
    }
  };
  float acc[8][8] = {};
  fetch(0);
  for (int u0 = 0; u0 < tk; u0 += kUD) {
    __syncthreads();
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      Pa[lu][lr + 16 * v] = na[v];
      Pb[lu][lr + 16 * v] = nb[v];
    }
    __syncthreads();
    if (u0 + kUD < tk) fetch(u0 + kUD);
#pragma unroll
    for (int u = 0; u < kUD; ++u) {
      float x[8], y[8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 fx = *reinterpret_cast<const float4*>(&Pa[u][64 * h + 4 * ty]);
        const float4 fy = *reinterpret_cast<const float4*>(&Pb[u][64 * h + 4 * tx]);
        x[4 * h] = fx.x, x[4 * h + 1] = fx.y, x[4 * h + 2] = fx.z, x[4 * h + 3] = fx.w;
        y[4 * h] = fy.x, y[4 * h + 1] = fy.y, y[4 * h + 2] = fy.z, y[4 * h + 3] = fy.w;
      }
#pragma unroll
      for (int v = 0; v < 8; ++v)
#pragma unroll
        for (int w = 0; w < 8; ++w) acc[v][w] = fmaf(x[v], y[w], acc[v][w]);
    }
  }
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int i = 64 * (v >> 2) + 4 * ty + (v & 3);
    if (i >= rows_a) continue;
    float* row = const_cast<float*>(base_a) + (int64_t)i * S.ld + c0 + tj * kPT;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int j = 64 * (w >> 2) + 4 * tx + (w & 3);   // column c0 + tj·128 + j
      if (j < rows_b && (ti != tj || j <= i)) row[j] -= acc[v][w];
    }
  }
}

// q[offZ[b] + r] = Σ_j Z_r[j]² (FP64 sum of the FP32 values), one warp per row of Z; grid (rows, systems)
__global__ void __launch_bounds__(256)
spd_norms_kernel(SpdRows S, double* __restrict__ q)
{
  const int b = blockIdx.y, r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= S.t[b]) return;
  const float* z = S.Z + (S.offZ[b] + r) * S.ld + S.offA[b];
  DF a;
  for (int j = lane; j < S.s; j += 32) df_fma(a, z[j], z[j]);
  double v = df_value(a);
  for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) q[S.offZ[b] + r] = v;
}

// x ← L⁻ᵀy for the first row y of each system's Z (x[b·s …]): panels from the last, one CTA each.
constexpr int kBackThreads = 512;
__global__ void __launch_bounds__(kBackThreads)
spd_back_kernel(SpdRows S, const float* __restrict__ Ld, float* __restrict__ x)
{
  extern __shared__ float sm[];
  float* xs = sm;                     // s
  float* L = sm + ((S.s + 31) & ~31);  // 128×129
  float* red = L + kPT * (kPT + 1);   // 4×128
  const int b = blockIdx.x, tid = threadIdx.x, s = S.s;
  const int np = (s + kPT - 1) / kPT;
  const float* y = S.Z + S.offZ[b] * S.ld + S.offA[b];
  for (int j = tid; j < s; j += kBackThreads) xs[j] = y[j];
  __syncthreads();
  for (int p = np - 1; p >= 0; --p) {
    const int k0 = p * kPT, tk = min(kPT, s - k0), c0 = k0 + tk;
    const float* Lp = Ld + ((int64_t)b * np + p) * kPT * kPT;
    for (int e = tid; e < kPT * kPT; e += kBackThreads) L[(e / kPT) * (kPT + 1) + e % kPT] = Lp[e];
    const int j = tid & (kPT - 1), grp = tid / kPT;
    float a = 0.f;
    if (j < tk) {
      const float* col = S.A + (int64_t)b * S.strideA + S.offA[b] + k0 + j;
#pragma unroll 8
      for (int i = c0 + grp; i < s; i += kBackThreads / kPT) a = fmaf(col[(int64_t)i * S.ld], xs[i], a);
    }
    red[grp * kPT + j] = a;
    __syncthreads();
    if (tid < 32) {   // L_kkᵀ x_k = rhs: lane holds elements lane + 32q
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = tid + 32 * q;
        v[q] = i < tk ? xs[k0 + i] - (red[i] + red[kPT + i] + red[2 * kPT + i] + red[3 * kPT + i]) : 0.f;
      }
#pragma unroll
      for (int q = 3; q >= 0; --q)
        for (int l = 31; l >= 0; --l) {
          const int jj = 32 * q + l;
          if (jj >= tk) continue;
          const float xj = __shfl_sync(0xffffffffu, v[q], l) / L[jj * (kPT + 1) + jj];
          if (tid == l) v[q] = xj;
#pragma unroll
          for (int w = 0; w <= q; ++w) {
            const int i = tid + 32 * w;
            if (i < jj) v[w] = fmaf(-L[jj * (kPT + 1) + i], xj, v[w]);
          }
        }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (tid + 32 * q < tk) xs[k0 + tid + 32 * q] = v[q];
    }
    __syncthreads();
  }
  for (int j = tid; j < s; j += kBackThreads) x[(int64_t)b * s + j] = xs[j];
}

// part[b·nblk + blk] = Σ_{i in block} x_i·(2z_i − (M x)_i) with M = A + diag(ridge): A's upper triangle
// (kept by the factorisation) and its diagonal diag0, double-float products, FP64 per row.
__global__ void __launch_bounds__(256)
spd_quad_kernel(SpdRows S, const float* __restrict__ ridge, const float* __restrict__ diag0,
                const float* __restrict__ z, const float* __restrict__ x, double* __restrict__ part)
{
  __shared__ double sh[32];
  const int b = blockIdx.y, s = S.s, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* xb = x + (int64_t)b * s;
  double tot = 0.0;
  for (int i = blockIdx.x * 64 + warp; i < min(s, (int)(blockIdx.x + 1) * 64); i += 8) {
    const float* row = S.A + (int64_t)b * S.strideA + (int64_t)i * S.ld + S.offA[b];
    DF a;
    for (int j = i + 1 + lane; j < s; j += 32) df_fma(a, row[j], xb[j]);
    double v = 2.0 * df_value(a);
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) {
      const double xi = (double)xb[i];
      v += ((double)diag0[(int64_t)b * s + i] + (double)ridge[(int64_t)b * s + i]) * xi;
      tot += xi * (2.0 * (double)z[(int64_t)b * s + i] - v);
    }
  }
  const double r = block_sum_d(tot, sh);
  if (threadIdx.x == 0) part[(int64_t)b * gridDim.x + blockIdx.x] = r;
}

// diag0 = A's diagonal, z = A's row `which` (its own entries left of the diagonal by symmetry are the
// same memory: the block is full), zrow = Z's first row ← z
__global__ void __launch_bounds__(256)
spd_take_kernel(SpdRows S, const int64_t* __restrict__ which, float* __restrict__ diag0, float* __restrict__ z)
{
  const int b = blockIdx.y, j = blockIdx.x * 256 + threadIdx.x;
  if (j >= S.s) return;
  const float* A = S.A + (int64_t)b * S.strideA + S.offA[b];
  const float v = A[which[b] * S.ld + j];
  diag0[(int64_t)b * S.s + j] = A[(int64_t)j * S.ld + j];
  z[(int64_t)b * S.s + j] = v;
  S.Z[S.offZ[b] * S.ld + S.offA[b] + j] = v;
}

static SpdRows rows_of(const SpdBatch& B)
{
  return SpdRows{B.A, B.strideA, B.Z, B.offA, B.offZ, B.t, B.ld, B.s};
}

// Factors the systems and solves their Z rows (see above); status gets 1 on a pivot that is not positive.
static void spd_panels(const SpdBatch& B, const float* ridge, float* Ld, int* status, cudaStream_t st)
{
  const SpdRows S = rows_of(B);
  const int nZ = (B.t_max + kPT - 1) / kPT;
  CUDA_TRY(cudaFuncSetAttribute(spd_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem));
  for (int k0 = 0; k0 < B.s; k0 += kPT) {
    const int c0 = std::min(k0 + kPT, B.s);
    const int nA = (B.s - c0 + kPT - 1) / kPT;
    const int pr = (B.s - c0 + kPR - 1) / kPR + (B.t_max + kPR - 1) / kPR;
    spd_panel_kernel<<<dim3(std::max(1, pr), B.nb), 512, kPanelSmem, st>>>(S, ridge, k0, Ld, status);
    LAUNCH_CHECK();
    const int tiles = nA * (nA + 1) / 2 + nA * nZ;
    if (tiles == 0) continue;
    spd_update_kernel<<<dim3(tiles, B.nb), 256, 0, st>>>(S, k0);
    LAUNCH_CHECK();
  }
}

static size_t ld_bytes(const SpdBatch& B) { return (size_t)B.nb * ceil_div(B.s, kPT) * kPT * kPT * sizeof(float); }

void spd_row_norms(const SpdBatch& B, const float* ridge, double* q, int* status, cudaStream_t st)
{
  DevBuf d(st);
  float* Ld = (float*)d.ensure(ld_bytes(B));
  spd_panels(B, ridge, Ld, status, st);
  if (B.t_max > 0) {
    spd_norms_kernel<<<dim3((unsigned)ceil_div(B.t_max, 8), B.nb), 256, 0, st>>>(rows_of(B), q);
    LAUNCH_CHECK();
  }
}

int spd_quadform_blocks(int s) { return (int)ceil_div(s, 64); }

void spd_quadforms(const SpdBatch& B, const float* ridge, const int64_t* which, double* part, int* status, cudaStream_t st)
{
  DevBuf d(st), dv(st);
  float* Ld = (float*)d.ensure(ld_bytes(B));
  float* diag0 = (float*)dv.ensure((size_t)3 * B.nb * B.s * sizeof(float));
  float* z = diag0 + (size_t)B.nb * B.s;
  float* x = z + (size_t)B.nb * B.s;
  const SpdRows S = rows_of(B);
  spd_take_kernel<<<dim3((unsigned)ceil_div(B.s, 256), B.nb), 256, 0, st>>>(S, which, diag0, z);
  LAUNCH_CHECK();
  spd_panels(B, ridge, Ld, status, st);
  const size_t smem = (size_t)(((B.s + 31) & ~31) + kPT * (kPT + 1) + 4 * kPT) * sizeof(float);
  CUDA_TRY(cudaFuncSetAttribute(spd_back_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  spd_back_kernel<<<B.nb, kBackThreads, smem, st>>>(S, Ld, x);
  LAUNCH_CHECK();
  spd_quad_kernel<<<dim3(spd_quadform_blocks(B.s), B.nb), 256, 0, st>>>(S, ridge, diag0, z, x, part);
  LAUNCH_CHECK();
}

}  // namespace slemm

// columns.cuh — the row-wise passes of an operator application, one thread-block cluster per column.
//
// Between two packed products every column needs a few column-wide numbers (QᵀV, the mean and the
// range that set its scale, the largest value, the recurrence's dot products), each of which the
// next element-wise pass reads.  As separate kernels that is a launch, a preamble that re-reduces the
// previous kernel's block partials and a pass over the column for each number: 13 kernels of 4–16 µs
// per Lanczos step at n = 50,000 with 7 columns, where the two products take 134 of 254 µs.  Here a
// cluster of up to 16 blocks owns a column: the numbers go through distributed shared memory (one cluster
// barrier each), a thread keeps its first 8 rows in registers from pass to pass, and the others are
// re-read from L2, where a column (2 MB at n = 500,000) stays.  So an operator takes three of these
// kernels and a Lanczos step no more.  Bound by the latency of their four to six cluster-wide reductions
// for short columns, by L2 and HBM for long ones.  One projected operator at n = 2,000, m = 10,000 with 31
// columns takes 62 µs (102 with ten kernels); the REML gradient at n = 50,000, m = 25,000 with 30
// probes went from 6.0 to 5.6 ms with them and takes 4.4 now, an MC-REML fit at n = 50,000, m = 20,000 from 7.8 to
// 7.3 and takes 3.7; at n = 500,000 with 66 columns, where the products are 95 %, nothing changes.  Clusters of 16
// where 8 columns or fewer leave half of the GPU idle with 8: 1.5 % of that gradient and of the fit.
//
// A thread works on half of a packed word, elements 4h … 4h + 3 and 8 + 4h … 11 + 4h: two 4-wide loads,
// and its digits are 8 contiguous bytes of each operand row (four neighbours' would be single bytes).
// Whole words (16 rows) took twice the registers, one block per SM, and were slower than the separate
// kernels from 31 columns on (76 and 98 µs for the operand and the step at n = 50,000).  All sums are
// double-float per thread and FP64 above, in a fixed order (warps, then blocks by rank), so results are
// bit-reproducible for the same block of columns.  A column's bits depend on how many stand beside it: their number
// sets the cluster and block sizes here, and up to 32 the products' number format (ops.cu).
//
// The operand's padding rows (from k to kp in each piece, and up to N) are left as they are: they only
// reach product columns that nobody reads (66 columns at n = 100,000, m = 50,000: 1,554 → 1,534 µs).
//
// Included by ops.cu (its operand helpers).  Every kernel waits for the one before it
// (griddepcontrol.wait) and lets the next one be set up meanwhile.
#pragma once

#include <cooperative_groups.h>

namespace slemm {

constexpr int kColThreads = 512;   // most threads of a block (two blocks per SM: 64 registers each)
constexpr int kColCluster = 16;    // most blocks of a column; more than 8, the portable size, only where
constexpr int kColFew = 8;         // there are at most this many columns
constexpr int kColRows = 8;        // rows of one thread and sweep

struct ColPlan {
  int cluster, threads;
};
// Blocks and threads for `columns` columns of `units` half-words: as many blocks per column as have 64
// units each, but no more blocks in all than run at once (two per SM less what clusters leave over);
// then as many threads as give each one unit, at most 512.
static ColPlan col_plan(int64_t units, int columns)
{
  int cs = 1;
  while (cs < (columns <= kColFew ? kColCluster : 8) && units >= (int64_t)cs * 2 * 64 && (int64_t)columns * cs * 2 <= 2 * num_sms() * 7 / 8) cs *= 2;
  return {cs, (int)std::min<int64_t>(kColThreads, round_up(ceil_div(units, cs), 32))};
}

template <class... P, class... A>
static void launch_columns(void (*kernel)(P...), int64_t units, int columns, cudaStream_t st, A... args)
{
  const ColPlan p = col_plan(units, columns);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.cluster, (unsigned)columns);
  cfg.blockDim = dim3((unsigned)p.threads);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  if (p.cluster > 8) CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
  LAUNCH_CHECK();
}

// First row of unit w: its rows are first … first + 3 and first + 8 … first + 11.
__device__ __forceinline__ int64_t unit_row(int64_t w) { return (w >> 1) * 16 + (w & 1) * 4; }
__device__ __forceinline__ int unit_off(int u) { return (u & 3) + (u >> 2) * 8; }

// The unit's 8 values of a column, 0 from row n on; VEC: 16-byte loads (n % 4 == 0, aligned columns)
template <bool VEC>
__device__ __forceinline__ void load8(const float* __restrict__ col, int64_t w, int64_t n, float (&x)[8])
{
  const int64_t i = unit_row(w);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if constexpr (VEC) {
      float t[4] = {};
      if (i + 8 * h < n) ldv<4>(col + i + 8 * h, t);
      x[4 * h] = t[0], x[4 * h + 1] = t[1], x[4 * h + 2] = t[2], x[4 * h + 3] = t[3];
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) x[4 * h + q] = i + 8 * h + q < n ? col[i + 8 * h + q] : 0.f;
    }
  }
}
template <bool VEC>
__device__ __forceinline__ void store8(float* col, int64_t w, int64_t n, const float (&x)[8])
{
  const int64_t i = unit_row(w);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if constexpr (VEC) {
      const float t[4] = {x[4 * h], x[4 * h + 1], x[4 * h + 2], x[4 * h + 3]};
      if (i + 8 * h < n) stv<4>(col + i + 8 * h, t);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + 8 * h + q < n) col[i + 8 * h + q] = x[4 * h + q];
    }
  }
}

// proj_dot of the unit's rows (Q is zero-padded to a multiple of 256 rows): 16-byte loads, the same
// arithmetic for each row.
__device__ __forceinline__ void proj_dot8(const float* __restrict__ Q, int64_t ldq, int cq, int64_t w, const float2* qt,
                                          float (&out)[8])
{
  const int64_t i = unit_row(w);
  DF a[8];
  for (int l = 0; l < cq; ++l) {
    const float2 t = qt[l];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float q[4];
      ldv<4>(Q + (int64_t)l * ldq + i + 8 * h, q);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        df_fma(a[4 * h + e], q[e], t.x);
        a[4 * h + e].lo = __fmaf_rn(q[e], t.y, a[4 * h + e].lo);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) out[u] = __fadd_rn(a[u].hi, a[u].lo);
}

// Shared state of a column's reductions: block results of two successive reductions (a block may
// write the next one's while others still read this one's), the totals, and the scalars one thread
// derives from them (an FP64 instruction of a whole block costs 256 cycles of the SM's two FP64 lanes:
// a square root and a division in every thread took longer than the rest of the kernel).
struct ColShared {
  double warp[kColThreads / 32][4];
  double block[2][SLEMM_MAX_COVARIATES];
  double total[4];
  float f[4];
};

// Σ over the warp of one double-float pair per lane, in lane 0.
__device__ __forceinline__ void warp_df_sum(DF& a)
{
  for (int o = 16; o; o >>= 1) {
    const float h = __shfl_down_sync(0xffffffffu, a.hi, o), l = __shfl_down_sync(0xffffffffu, a.lo, o);
    df_add(a, h);
    a.lo = __fadd_rn(a.lo, l);
  }
}
__device__ __forceinline__ float warp_max_f(float v)
{
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

// Σ (or maximum) of one double per lane over the warp, the same in every lane: a fixed butterfly.
__device__ __forceinline__ double warp_all(double v, bool mx)
{
  for (int o = 16; o; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, v, o);
    v = mx ? fmax(v, t) : v + t;
  }
  return v;
}

// Combines S.warp[·][q], q < NV, over the column's warps (sum, or maximum where bit q of MAX is set) into
// S.total; then thread 0 of every block runs done(S.total), which leaves what all threads need in S.f.
// One warp does it, a lane per warp and then per block: walking them one after another took 2 µs.
template <int NV, unsigned MAX, class F>
__device__ __forceinline__ void col_combine(ColShared& S, int& turn, F&& done)
{
  namespace cg = cooperative_groups;
  const int nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  cg::cluster_group cl = cg::this_cluster();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const bool mx = (MAX >> q) & 1u;
      const double r = warp_all(lane < nw ? S.warp[lane][q] : (mx ? -INFINITY : 0.0), mx);
      if (lane == 0) S.block[turn][q] = r;
    }
  }
  cl.sync();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      const bool mx = (MAX >> q) & 1u;
      const bool has = lane < (int)cl.num_blocks();
      const double r = warp_all(has ? *cl.map_shared_rank(&S.block[turn][q], has ? lane : 0) : (mx ? -INFINITY : 0.0), mx);
      if (lane == 0) S.total[q] = r;
    }
    if (lane == 0) done(S.total);
  }
  __syncthreads();
  turn ^= 1;
}

// The same for one double-float sum per thread.
template <class F>
__device__ __forceinline__ void col_sum(DF a, ColShared& S, int& turn, F&& done)
{
  warp_df_sum(a);
  if ((threadIdx.x & 31) == 0) S.warp[threadIdx.x >> 5][0] = df_value(a);
  col_combine<1, 0u>(S, turn, done);
}

// qt[l] = Σ_rows Q[r, l]·x[r] over the column for l < cq, as hi+lo pairs.  `rows(w, x)` gives unit w's 8
// values; rows of Q: the unit's own, or inv[…] of them (−1: none) for a trait view.
template <class Rows>
__device__ __forceinline__ void col_project(const float* __restrict__ Q, int64_t ldq, int cq, int64_t units, int64_t w0,
                                            int64_t step, const int32_t* __restrict__ inv, Rows&& rows, float2* qt,
                                            ColShared& S, int& turn)
{
  namespace cg = cooperative_groups;
  constexpr int L = 4;   // covariates per pass over the column
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int l0 = 0; l0 < cq; l0 += L) {
    const int nl = min(L, cq - l0);
    DF a[L];
    for (int64_t w = w0; w < units; w += step) {
      float x[8];
      rows(w, x);
      const int64_t i = unit_row(w);
#pragma unroll
      for (int l = 0; l < L; ++l) {
        if (l < nl) {
          const float* ql = Q + (int64_t)(l0 + l) * ldq;
          float q[8];
          if (inv == nullptr) {
            load8<true>(ql, w, INT64_MAX, q);   // Q is zero-padded to a multiple of 256 rows
          } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int64_t r = inv[i + unit_off(u)];
              q[u] = r >= 0 ? ql[r] : 0.f;
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) df_fma(a[l], q[u], x[u]);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < L; ++l) {
      if (l < nl) {
        warp_df_sum(a[l]);
        if (lane == 0) S.warp[warp][l] = df_value(a[l]);
      }
    }
    __syncthreads();
    if (threadIdx.x < 32) {
#pragma unroll
      for (int l = 0; l < L; ++l) {
        if (l < nl) {
          const double r = warp_all(lane < nw ? S.warp[lane][l] : 0.0, false);
          if (lane == 0) S.block[turn][l0 + l] = r;
        }
      }
    }
    __syncthreads();
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  for (int l = warp; l < cq; l += nw) {
    const bool has = lane < (int)cl.num_blocks();
    const double r = warp_all(has ? *cl.map_shared_rank(&S.block[turn][l], has ? lane : 0) : 0.0, false);
    if (lane == 0) split_double(r, qt[l].x, qt[l].y);
  }
  __syncthreads();
  turn ^= 1;
}

__device__ __forceinline__ void pdl_wait_and_go()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void col_leave() { cooperative_groups::this_cluster().sync(); }   // peers may still read

// What the products will see of a column, summed in the units of x (weighted by wt when kWeighted): the
// values less the digits' remainders, which are 2^−24 of them and need FP32 only.
struct Stored {
  DF sum;
  float rest = 0.f;
  // the sum, its remainders in units of rest_scale
  __device__ __forceinline__ DF total(float rest_scale) const
  {
    DF a = sum;
    df_add(a, -__fmul_rn(rest, rest_scale));
    return a;
  }
};

// The operand of one unit of x·scale: digits (every step exact), or FP16 pieces (4-wide stores).
template <bool DIGITS, bool kWeighted>
__device__ __forceinline__ void store_unit(const float (&x)[8], int np, void* B, int64_t K_pad, int kp, int c, int64_t w,
                                           Stored& acc, const float (&wt)[8], float scale, float inv_scale)
{
  if constexpr (DIGITS) {
    uint8_t* dst = static_cast<uint8_t*>(B) + piece_row(0, kp, c) * K_pad + w * 8;
    float r[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) r[u] = __fmul_rn(x[u], scale);
#pragma unroll 1
    for (int p = 0; p < np; ++p) {
      float d[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        d[u] = rintf(r[u]);
        r[u] = __fmul_rn(__fsub_rn(r[u], d[u]), 32.f);
      }
      *reinterpret_cast<uint2*>(dst) = e4m3_half(d);
      dst += (int64_t)kp * K_pad;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (kWeighted) {
        df_fma(acc.sum, wt[u], x[u]);
        acc.rest = __fmaf_rn(wt[u], r[u], acc.rest);
      } else {
        df_add(acc.sum, x[u]);
        acc.rest = __fadd_rn(acc.rest, r[u]);
      }
    }
  } else {
    const int64_t i = unit_row(w);
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      const float t[4] = {x[h], x[h + 1], x[h + 2], x[h + 3]}, g[4] = {wt[h], wt[h + 1], wt[h + 2], wt[h + 3]};
      store_operand<4, kWeighted, true>(t, np, B, K_pad, kp, c, i + 2 * h, acc.sum, g, scale, inv_scale);
    }
  }
}
// Units of x per unit of a remainder after kDigits digits: 32^−5·2^−e
__device__ __forceinline__ float rest_scale(float inv_scale) { return __fmul_rn(inv_scale, 2.98023223876953125e-8f); }

// Direction-1 operand (K = individuals) of column c: x = in − Q(Qᵀin) for c < nq, times rr, less its mean,
// scaled to its range and split; rows that hold no individual are 0.  sums[c] = {the mean, 2^−e, and the sum
// of what is stored as a hi+lo pair}.
template <bool DIGITS, bool VEC>
__global__ void __launch_bounds__(kColThreads, 2)
col_operand_kernel(const float* __restrict__ in, int64_t ld, int64_t n, int64_t n_pad, int kp,
                   const float* __restrict__ Q, int64_t ldq, int cq, int nq, const float* __restrict__ rr, int np,
                   void* B, float4* __restrict__ sums, const int32_t* __restrict__ inv)
{
  __shared__ ColShared S;
  __shared__ float2 qt[SLEMM_MAX_COVARIATES];
  pdl_wait_and_go();
  const int c = blockIdx.y;
  const int64_t units = n_pad / kColRows, w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int turn = 0;
  const float* col = in + (int64_t)c * ld;
  auto raw = [&](int64_t w, float (&x)[8]) {
    if (inv != nullptr) {   // trait view: packed position i holds view row inv[i], or no individual of it
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int64_t r = inv[unit_row(w) + unit_off(u)];
        x[u] = r >= 0 ? col[r] : 0.f;
      }
    } else {
      load8<VEC>(col, w, n, x);
    }
  };
  // bit u: the unit's row u is an individual
  auto valid = [&](int64_t w) {
    const int64_t i = unit_row(w);
    unsigned m = 0xFFu;
    if (inv != nullptr) {
      m = 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) m |= (unsigned)(inv[i + unit_off(u)] >= 0) << u;
    } else if (i + 12 > n) {
      m = 0u;
#pragma unroll
      for (int u = 0; u < 8; ++u) m |= (unsigned)(i + unit_off(u) < n) << u;
    }
    return m;
  };
  const bool proj = cq > 0 && c < nq;
  if (proj) col_project(Q, ldq, cq, units, w0, step, inv, raw, qt, S, turn);
  auto value = [&](int64_t w, float (&x)[8]) {   // in − projection, times rr
    raw(w, x);
    if (inv != nullptr) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int64_t r = inv[unit_row(w) + unit_off(u)];
        if (r < 0) continue;
        if (proj) x[u] = __fsub_rn(x[u], proj_dot(Q, ldq, cq, r, qt));
        if (rr) x[u] = __fmul_rn(x[u], rr[r]);
      }
      return;
    }
    float t[8];
    if (proj) {
      proj_dot8(Q, ldq, cq, w, qt, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fsub_rn(x[u], t[u]);
    }
    if (rr) {
      load8<true>(rr, w, INT64_MAX, t);   // rr is zero-padded to n_pad
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fmul_rn(x[u], t[u]);
    }
  };
  float x0[8];
  DF sum;
  float hi = -INFINITY, nlo = -INFINITY;
  for (int64_t w = w0; w < units; w += step) {
    float x[8];
    value(w, x);
    const unsigned ok = valid(w);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (w == w0) x0[u] = x[u];
      df_add(sum, x[u]);   // 0 where there is no individual
      hi = fmaxf(hi, (ok >> u) & 1u ? x[u] : -INFINITY);
      nlo = fmaxf(nlo, (ok >> u) & 1u ? -x[u] : -INFINITY);
    }
  }
  warp_df_sum(sum);
  hi = warp_max_f(hi);
  nlo = warp_max_f(nlo);
  if ((threadIdx.x & 31) == 0) {
    double* v = S.warp[threadIdx.x >> 5];
    v[0] = df_value(sum), v[1] = (double)hi, v[2] = (double)nlo;
  }
  col_combine<3, 6u>(S, turn, [&](const double* v) {
    const float mu_ = (float)(v[0] * (1.0 / (double)n));
    const int e = split_exp(fmax(v[1] - (double)mu_, v[2] + (double)mu_), DIGITS ? kDigitTop : kF16Top);
    S.f[0] = mu_, S.f[1] = ldexpf(1.f, e), S.f[2] = ldexpf(1.f, -e);
  });
  const float mu = S.f[0], sc = S.f[1], isc = S.f[2];
  Stored acc;
  const float none[8] = {};
  for (int64_t w = w0; w < units; w += step) {
    float x[8];
    if (w == w0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = x0[u];
    } else {
      value(w, x);
    }
    const unsigned ok = valid(w);
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = (ok >> u) & 1u ? __fsub_rn(x[u], mu) : 0.f;
    store_unit<DIGITS, false>(x, np, B, n_pad, kp, c, w, acc, none, sc, isc);
  }
  col_sum(acc.total(rest_scale(isc)), S, turn, [&](const double* v) {
    float h, l;
    split_double(v[0], h, l);
    if (blockIdx.x == 0) sums[c] = make_float4(mu, isc, h, l);
  });
  col_leave();
}

// Direction-2 operand (K = SNPs) of column c: from the first product (FROM_D: raw·2^−e1 − gm_j·colsum_c
// + μ_c·gcorr_j, times w_j, as finalize_snp_kernel), else `in`; scaled to its largest value and split.
// tsums[c] = {–, 2^−e2, Σ_j gm_j·stored as a hi+lo pair}.  V2[c][j] keeps the values of a thread's
// units past its first (FROM_D).
template <bool DIGITS, bool FROM_D, bool VEC>
__global__ void __launch_bounds__(kColThreads, 2)
col_snp_kernel(const float* __restrict__ D, int splits, int kp1, const float* __restrict__ w_,
               const float4* __restrict__ sums, const float* __restrict__ gcorr, float* __restrict__ V2, const float* __restrict__ in, int64_t ld,
               int64_t m, int64_t m_pad, int kp, const float* __restrict__ gm, int np, void* B,
               float4* __restrict__ tsums)
{
  __shared__ ColShared S;
  pdl_wait_and_go();
  const int c = blockIdx.y;
  const int64_t units = m_pad / kColRows, w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int turn = 0;
  const float4 s1 = FROM_D ? sums[c] : make_float4(0.f, 1.f, 0.f, 0.f);
  const float mu = s1.x, isc1 = s1.y, ch = s1.z, cl = s1.w;
  auto value = [&](int64_t w, float (&x)[8]) {
    if constexpr (FROM_D) {   // D, gm, gcorr and w are zero-padded to m_pad rows
      const int64_t j = unit_row(w);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float t[4], g[4], e[4], ws[4];
        gather_D<4>(D, splits, kp1, m_pad, c, j + 8 * h, isc1, t);
        ldv<4>(gm + j + 8 * h, g);
        ldv<4>(gcorr + j + 8 * h, e);
        if (w_) ldv<4>(w_ + j + 8 * h, ws);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v = __fmaf_rn(-g[q], cl, __fmaf_rn(-g[q], ch, t[q]));
          v = __fmaf_rn(mu, e[q], v);
          if (w_) v = __fmul_rn(v, ws[q]);
          x[4 * h + q] = j + 8 * h + q < m ? v : 0.f;
        }
      }
    } else {
      load8<VEC>(in + (int64_t)c * ld, w, m, x);
    }
  };
  float x0[8];
  float amax = 0.f;
  for (int64_t w = w0; w < units; w += step) {
    float x[8];
    value(w, x);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (w == w0) x0[u] = x[u];
      amax = fmaxf(amax, fabsf(x[u]));
    }
    if (FROM_D && w != w0) store8<true>(V2 + (int64_t)c * m_pad, w, m_pad, x);
  }
  amax = warp_max_f(amax);
  if ((threadIdx.x & 31) == 0) S.warp[threadIdx.x >> 5][0] = (double)amax;
  col_combine<1, 1u>(S, turn, [&](const double* v) {
    const int e = split_exp(v[0], DIGITS ? kDigitTop : kF16Top);
    S.f[0] = ldexpf(1.f, e), S.f[1] = ldexpf(1.f, -e);
  });
  const float sc = S.f[0], isc = S.f[1];
  Stored acc;
  for (int64_t w = w0; w < units; w += step) {
    float x[8], g[8];
    if (w == w0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = x0[u];
    } else if constexpr (FROM_D) {
      load8<true>(V2 + (int64_t)c * m_pad, w, m_pad, x);
    } else {
      value(w, x);
    }
    load8<true>(gm, w, INT64_MAX, g);   // gm is zero-padded to m_pad
    store_unit<DIGITS, true>(x, np, B, m_pad, kp, c, w, acc, g, sc, isc);
  }
  col_sum(acc.total(rest_scale(isc)), S, turn, [&](const double* v) {
    float h, l;
    split_double(v[0], h, l);
    if (blockIdx.x == 0) tsums[c] = make_float4(0.f, isc, h, l);
  });
  col_leave();
}

// Results of the second product for column c (rows = individuals): T = raw·2^−e2 − t_c, times rr; the first
// nq columns are projected, T − Q(QᵀT); plus tau0·Vin when Vin is given.
//
// LZ: and the rest of the Lanczos step on it (lanczos.cu): x −= β·U_prev (β the last step's ‖x‖ as a hi+lo
// pair, U_prev given), δ = Vinᵀx, x −= δ·Vin, β = ‖x‖, U_next = x/β and ‖U_next‖² of the stored
// values.  `out` then holds only a thread's units past its first; scal[c], scal[stride + c],
// scal[2·stride + c] get δ, β², ‖U_next‖² (host-mapped), and column 0 the kernels' error word in scal_err.
struct LzColumn {
  const float* Uprev;
  float* Unext;
  float2* beta;
  double* scal;
  int stride;
  double* scal_err;
  const int* err;
};
template <bool VEC, bool LZ>
__global__ void __launch_bounds__(kColThreads, 2)
col_out_kernel(const float* __restrict__ D, int splits, int kp2, int64_t n_pad, int64_t n,
               const float4* __restrict__ tsums, const float* __restrict__ rr, const float* __restrict__ Vin, int64_t ld_v, float tau0, int nq,
               const float* __restrict__ Q, int64_t ldq, int cq, float* out, int64_t ldo,
               const int32_t* __restrict__ map, LzColumn lz)
{
  __shared__ ColShared S;
  __shared__ float2 qt[SLEMM_MAX_COVARIATES];
  pdl_wait_and_go();
  const int c = blockIdx.y;
  const int64_t units = (n + 15) / 16 * 2, w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  int turn = 0;
  const float4 s2 = tsums[c];
  const float isc = s2.y, th = s2.z, tl = s2.w;
  float* col = out + (int64_t)c * ldo;
  const float* vcol = Vin ? Vin + (int64_t)c * ld_v : nullptr;
  float x0[8];
  // a thread's first unit stays in x0, its others in out; rows past n are 0
  auto get = [&](int64_t w, float (&x)[8]) {
    if (w == w0) {
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = x0[u];
    } else {
      load8<VEC>(col, w, n, x);
    }
  };
  auto put = [&](int64_t w, const float (&x)[8], bool last) {
    if (w == w0)
#pragma unroll
      for (int u = 0; u < 8; ++u) x0[u] = x[u];
    if (w != w0 || (last && !LZ)) store8<VEC>(col, w, n, x);
  };
  const bool proj = c < nq;   // T − Q(QᵀT) + tau0·Vin; else T + tau0·Vin at once
  for (int64_t w = w0; w < units; w += step) {
    float x[8], t[8];
    const int64_t i = unit_row(w);
    if (map != nullptr) {   // trait view: view row i is packed row map[i]
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = 0.f;
        if (i + unit_off(u) < n) {
          float d[1];
          gather_D<1>(D, splits, kp2, n_pad, c, map[i + unit_off(u)], isc, d);
          x[u] = d[0];
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h) {   // D has n_pad rows, n_pad a multiple of 256
        float d[4];
        gather_D<4>(D, splits, kp2, n_pad, c, i + 8 * h, isc, d);
#pragma unroll
        for (int q = 0; q < 4; ++q) x[4 * h + q] = d[q];
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = __fsub_rn(__fsub_rn(x[u], th), tl);
    if (rr) {
      load8<true>(rr, w, INT64_MAX, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fmul_rn(x[u], t[u]);
    }
    if (vcol && !proj) {
      load8<VEC>(vcol, w, n, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fmaf_rn(tau0, t[u], x[u]);
    }
    if (i + 12 > n)
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = i + unit_off(u) < n ? x[u] : 0.f;
    put(w, x, !proj);
  }
  if (proj) {
    if (cq > 0) col_project(Q, ldq, cq, units, w0, step, nullptr, get, qt, S, turn);
    for (int64_t w = w0; w < units; w += step) {
      float x[8], t[8];
      get(w, x);
      if (cq > 0) {
        proj_dot8(Q, ldq, cq, w, qt, t);   // 0 past n: Q's rows are
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = __fsub_rn(x[u], t[u]);
      }
      load8<VEC>(vcol, w, n, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fmaf_rn(tau0, t[u], x[u]);
      put(w, x, true);
    }
  }
  if constexpr (LZ) {
    const float* pcol = lz.Uprev ? lz.Uprev + (int64_t)c * n : nullptr;
    const float bh = pcol ? lz.beta[c].x : 0.f, bl = pcol ? lz.beta[c].y : 0.f;
    DF acc;
    for (int64_t w = w0; w < units; w += step) {
      float x[8], t[8];
      get(w, x);
      if (pcol) {
        load8<VEC>(pcol, w, n, t);
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = __fmaf_rn(-bl, t[u], __fmaf_rn(-bh, t[u], x[u]));
        put(w, x, false);
      }
      load8<VEC>(vcol, w, n, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) df_fma(acc, t[u], x[u]);
    }
    const bool first = blockIdx.x == 0;
    col_sum(acc, S, turn, [&](const double* v) {
      split_double(v[0], S.f[0], S.f[1]);
      if (first) lz.scal[c] = v[0];
    });
    const float dh = S.f[0], dl = S.f[1];
    acc = DF();
    for (int64_t w = w0; w < units; w += step) {
      float x[8], t[8];
      get(w, x);
      load8<VEC>(vcol, w, n, t);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = __fmaf_rn(-dl, t[u], __fmaf_rn(-dh, t[u], x[u]));
        df_fma(acc, x[u], x[u]);
      }
      put(w, x, false);
    }
    col_sum(acc, S, turn, [&](const double* v) {
      const double r = sqrt(v[0]);
      split_double(1.0 / r, S.f[2], S.f[3]);
      if (first) {
        float2 bt;
        split_double(r, bt.x, bt.y);
        lz.beta[c] = bt;   // every block has read the last step's before this sum
        lz.scal[lz.stride + c] = v[0];
      }
    });
    const float ih = S.f[2], il = S.f[3];
    acc = DF();
    for (int64_t w = w0; w < units; w += step) {
      float x[8];
      get(w, x);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        x[u] = __fmaf_rn(x[u], ih, __fmul_rn(x[u], il));
        df_fma(acc, x[u], x[u]);   // 0 past n
      }
      store8<VEC>(lz.Unext + (int64_t)c * n, w, n, x);
    }
    col_sum(acc, S, turn, [&](const double* v) {
      if (!first) return;
      lz.scal[2 * lz.stride + c] = v[0];
      if (c == 0) lz.scal_err[0] = (double)*lz.err;
    });
  }
  col_leave();
}

// MC-REML's first-order terms of one shift, column c: e = P(A_c + st·A_{q+c}) for c ≥ 1 (P·A_0 for c = 0), its
// norm norms[c] = ‖e‖², out_c = rr∘e.  Combination, projection (three kernels), norm (two) and scaling as
// kernels of their own were 35 µs and seven launches of each evaluation of the criterion, the SNP effects'
// (below) another three: an MC-REML fit at n = 50,000, m = 20,000 with five of them took 3.95 ms (3.74 now).
template <bool VEC>
__global__ void __launch_bounds__(kColThreads, 2)
col_first_kernel(const float* __restrict__ A, int64_t n, int64_t units, int q, float st, const float* __restrict__ Q, int64_t ldq,
                 int cq, const float* __restrict__ rr, float* __restrict__ out, double* __restrict__ norms)
{
  __shared__ ColShared S;
  __shared__ float2 qt[SLEMM_MAX_COVARIATES];
  pdl_wait_and_go();
  const int c = blockIdx.y;
  const int64_t w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  int turn = 0;
  const float *a = A + (int64_t)c * n, *b = A + (int64_t)(q + c) * n;
  auto rows = [&](int64_t w, float (&x)[8]) {
    load8<VEC>(a, w, n, x);
    if (c > 0) {
      float y[8];
      load8<VEC>(b, w, n, y);
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = __fmaf_rn(st, y[u], x[u]);
    }
  };
  if (cq > 0) col_project(Q, ldq, cq, units, w0, step, nullptr, rows, qt, S, turn);
  DF sum;
  for (int64_t w = w0; w < units; w += step) {
    float x[8], p[8], r[8];
    rows(w, x);
    proj_dot8(Q, ldq, cq, w, qt, p);
    load8<VEC>(rr, w, n, r);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x[u] = __fsub_rn(x[u], p[u]);
      df_fma(sum, x[u], x[u]);
      x[u] = __fmul_rn(x[u], r[u]);
    }
    store8<VEC>(out + (int64_t)c * n, w, n, x);
  }
  col_sum(sum, S, turn, [&](const double* t) {
    if (blockIdx.x == 0) norms[c] = t[0];
  });
  col_leave();
}

// X_c ← √w∘X_c and norms[c] = ‖X_c‖² (the same terms of the SNP effects).
template <bool VEC>
__global__ void __launch_bounds__(kColThreads, 2)
col_weigh_kernel(float* X, int64_t m, int64_t units, const float* __restrict__ w_, double* __restrict__ norms)
{
  __shared__ ColShared S;
  pdl_wait_and_go();
  const int c = blockIdx.y;
  const int64_t w0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  int turn = 0;
  DF sum;
  for (int64_t w = w0; w < units; w += step) {
    float x[8], f[8];
    load8<VEC>(X + (int64_t)c * m, w, m, x);
    load8<VEC>(w_, w, m, f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x[u] = __fmul_rn(x[u], __fsqrt_rn(f[u]));
      df_fma(sum, x[u], x[u]);
    }
    store8<VEC>(X + (int64_t)c * m, w, m, x);
  }
  col_sum(sum, S, turn, [&](const double* t) {
    if (blockIdx.x == 0) norms[c] = t[0];
  });
  col_leave();
}

}  // namespace slemm

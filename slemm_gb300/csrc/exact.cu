// exact.cu — products of the packed counts with FP32 or FP64 columns whose sums are exact.
//
// A dense column v is cut into base-32 digits,
//   v·2^e = d_0 + 2^−5·d_1 + 2^−10·d_2 + …,   d_p integers, |d_p| ≤ 16,
// with e such that max|v|·2^e lies in [2^3, 2^4), and as many digits as reach the last bit of the smallest nonzero
// value: for an FP64 column 11 where all values are of one size, 15 for a million between the largest and the smallest,
// up to 420 (in passes of 160); for an FP32 column five to 56, found on the device.  Digits are exact in E4M3 and a count is at
// most 2, so a product row's sum over 2^19 K-elements is an integer of at most 2^24: the tensor cores' FP32
// accumulators are exact whatever their order.  K is therefore split every 8,192 K-tiles at
// the latest, the partials are added as 64-bit integers, and only the last combination of the digits
// rounds (in FP64).  Bound by the narrow tensor-core pass.  GB300's FP64 pipe ran the same sums by an
// FMA per genotype and column: at n = 100,000, m = 50,000 the GEBV took 18,988 µs and takes 435 µs, the
// score terms with three covariates and residual weights 112,698 µs and 691 µs, with the same or a
// smaller error against 64-bit sums.
#include "internal.h"
#include "decode.cuh"
#include "reduce.cuh"

namespace slemm {

constexpr int kDigitBits = 5;
constexpr int kDigitRows = 160;   // digits of one pass
constexpr int kDigitCols = 32;    // most columns of one pass (an FP32 value has five digits at least)
constexpr int kXRows = 2048;                  // K-elements of one block of the operand kernels
constexpr int kXThreads = 256;

// e with amax·2^e in [2^3, 2^4) (0 for a zero or non-finite column)
__host__ __device__ inline int digit_exp(double amax)
{
  if (!(amax > 0.0) || !isfinite(amax)) return 0;
  int E;
  frexp(amax, &E);
  return 4 - E;
}

// Digits of a column at exponent e that reach the last of the `bits` bits of its smallest nonzero magnitude (at
// 2^least the lowest bit of the type).
__host__ __device__ inline int digit_count(int e, double amin, int bits, int least)
{
  if (!(amin > 0.0) || !isfinite(amin)) return 1;
  int E;
  frexp(amin, &E);
  const int low = -((E - bits > least ? E - bits : least) + e);   // the bit is 2^−low of a unit
  return 1 + (low > 0 ? (low + kDigitBits - 1) / kDigitBits : 0);
}

// v·2^e = I·2^−5K with integers I and K ≥ 0 (|v·2^e| ≤ 2^4).
__device__ __forceinline__ void digit_int(double v, int e, long long& I, int& K)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int ex = (int)(b >> 52) & 0x7FF;
  const long long M = (long long)((b & 0xFFFFFFFFFFFFFull) | (ex ? 0x10000000000000ull : 0ull));
  const int L = 1075 - max(ex, 1) - e;   // |v·2^e| = M·2^−L
  K = L > 0 ? (L + kDigitBits - 1) / kDigitBits : 0;
  I = M << (K * kDigitBits - L);
  I = (long long)b < 0 ? -I : I;
}
__device__ __forceinline__ void digit_int(float v, int e, int& I, int& K)
{
  const unsigned b = __float_as_uint(v);
  const int ex = (int)(b >> 23) & 0xFF;
  const int M = (int)((b & 0x7FFFFFu) | (ex ? 0x800000u : 0u));
  const int L = 150 - max(ex, 1) - e;
  K = L > 0 ? (L + kDigitBits - 1) / kDigitBits : 0;
  I = M << (K * kDigitBits - L);
  I = (int)b < 0 ? -I : I;
}

// Digits p0 … p0 + cnt − 1, of `digits` that hold every bit, of the 16 values v[·]·2^e of K-elements kidx …
// kidx + 15 (one packed word) into rows row0 … row0 + cnt − 1 of the operand.  From the last digit up: the low five
// bits of I as −16 … 15 in each step, and what is left as the first; in integers, since GB300's FP64 pipe has two
// lanes (50,000 effects: 7 µs; the same digits by FP64 rounding and differences took 45 µs more).
template <class T, class Int>
__device__ __forceinline__ void store_digits(const T (&v)[16], int e, uint8_t* __restrict__ B, int64_t K_pad,
                                             int row0, int digits, int p0, int cnt, int64_t kidx)
{
  Int I[16];
  int K[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) digit_int(v[u], e, I[u], K[u]);
#pragma unroll 1
  for (int p = digits - 1; p >= p0; --p) {
    float d[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      int q = p > 0 ? (((int)I[u] + 16) & 31) - 16 : (int)I[u];
      if (p > K[u]) q = 0;
      d[u] = (float)q;
      I[u] = p > K[u] ? I[u] : (I[u] - q) >> kDigitBits;
    }
    if (p < p0 + cnt) *reinterpret_cast<uint4*>(B + (int64_t)(row0 + p - p0) * K_pad + kidx) = e4m3_word(d);
  }
}

// 2^−5cnt·v + Σ_p 2^−5p·(Σ_splits D[s][row0 + p][r]), p < cnt — the column's product with row r, in units of 2^−e,
// with v what the digits after these gave.  Six digits at a time are one integer (a digit's sum is below 2^31 up to
// 2^26 K-elements), so that they take one conversion and one FMA of the FP64 pipe instead of six.
__device__ __forceinline__ double gather_digits(const float* __restrict__ D, int splits, int kp, int64_t M_pad,
                                                int row0, int cnt, int64_t r, double v)
{
  constexpr int G = 6;
  const float* Dr = D + (int64_t)row0 * M_pad + r;
  v *= (double)(1 << kDigitBits * ((cnt + G - 1) / G * G - cnt));   // to the unit of the last group
  for (int p = (cnt - 1) / G * G; p >= 0; p -= G) {
    long long sum[G] = {};
#pragma unroll 4
    for (int s = 0; s < splits; ++s)
#pragma unroll
      for (int q = 0; q < G; ++q)
        if (p + q < cnt) sum[q] += (long long)__float2int_rn(Dr[((int64_t)s * kp + p + q) * M_pad]);
    long long I = sum[0];
#pragma unroll
    for (int q = 1; q < G; ++q) I = I * (1 << kDigitBits) + sum[q];
    // v counts 2^−5 of the group's last digit
    v = fma(v, 1.0 / (1 << kDigitBits), (double)I);
    if (p > 0) v *= 1.0 / (1 << kDigitBits * (G - 1));
  }
  return v * (1.0 / (1 << kDigitBits * (G - 1)));
}

// GEBV operand: digits p0 … p0 + cnt − 1 of alpha (0 past m); 16 K-elements per thread
// (32 threads a block, so that the blocks spread over all SMs)
__global__ void __launch_bounds__(32)
gebv_operand_kernel(const double* __restrict__ alpha, int64_t m, int64_t m_pad, int e, int digits, int p0, int cnt,
                    uint8_t* __restrict__ B)
{
  const int64_t j = ((int64_t)blockIdx.x * 32 + threadIdx.x) * 16;
  if (j >= m_pad) return;
  double v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) v[u] = j + u < m ? alpha[j + u] : 0.0;
  store_digits<double, long long>(v, e, B, m_pad, 0, digits, p0, cnt, j);
}

// tgv = the digits' sums and, if `more`, the later digits' in tgv before; the first pass's result is shift + 2^−e·it.
__global__ void __launch_bounds__(kXThreads)
gebv_finish_kernel(const float* __restrict__ D, int splits, int kp, int64_t n_pad, int64_t n, int cnt, int more, int first,
                   int e, double shift, double* __restrict__ tgv)
{
  const int64_t i = (int64_t)blockIdx.x * kXThreads + threadIdx.x;
  if (i >= n) return;
  const double v = gather_digits(D, splits, kp, n_pad, 0, cnt, i, more ? tgv[i] : 0.0);
  tgv[i] = first ? shift + ldexp(v, -e) : v;
}

// The columns of exact_dots (FP32 values), i < n.
__device__ __forceinline__ float dot_column(const ExactCols& a, int c, int64_t i)
{
  if (a.y) {
    if (c == 0) return a.y[i];
    --c;
  }
  const float r = a.rr ? a.rr[i] : 1.f;
  return __fmul_rn(r, c < a.cq ? a.Q[(int64_t)c * a.ldq + i] : r);
}

// Block partials of each column's sum and largest magnitude (∞ for a non-finite value), and of its smallest
// nonzero magnitude negated (−∞: none): sums[c][blk], amax[c][blk], namin[c][blk]; grid (blocks, C).
__global__ void __launch_bounds__(kXThreads)
dots_stats_kernel(ExactCols a, int64_t n, double* __restrict__ sums, double* __restrict__ amax, double* __restrict__ namin,
                  int nblk)
{
  __shared__ double sh[32];
  __shared__ float ext[2][kXThreads / 32];
  const int c = blockIdx.y;
  const int64_t i0 = (int64_t)blockIdx.x * kXRows + threadIdx.x;
  double acc = 0.0;
  float mx = 0.f, nmn = -INFINITY, v[kXRows / kXThreads];
#pragma unroll
  for (int u = 0; u < kXRows / kXThreads; ++u) v[u] = i0 + u * kXThreads < n ? dot_column(a, c, i0 + u * kXThreads) : 0.f;
#pragma unroll
  for (int u = 0; u < kXRows / kXThreads; ++u) {
    const float mag = isfinite(v[u]) ? fabsf(v[u]) : INFINITY;
    acc += (double)v[u];
    mx = fmaxf(mx, mag);
    nmn = fmaxf(nmn, mag > 0.f ? -mag : -INFINITY);
  }
  const double s = block_sum_d(acc, sh);
  for (int o = 16; o; o >>= 1) {
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    nmn = fmaxf(nmn, __shfl_down_sync(0xffffffffu, nmn, o));
  }
  if ((threadIdx.x & 31) == 0) ext[0][threadIdx.x >> 5] = mx, ext[1][threadIdx.x >> 5] = nmn;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < kXThreads / 32; ++q) mx = fmaxf(mx, ext[0][q]), nmn = fmaxf(nmn, ext[1][q]);
    sums[(int64_t)c * nblk + blockIdx.x] = s;
    amax[(int64_t)c * nblk + blockIdx.x] = mx;
    namin[(int64_t)c * nblk + blockIdx.x] = nmn;
  }
}

// Column c's total (NaN when it holds a non-finite value), digit exponent and number of digits (host-mapped), one
// warp each.
__global__ void dots_scale_kernel(const double* __restrict__ sums, const double* __restrict__ amax,
                                  const double* __restrict__ namin, int nblk, int C, double* __restrict__ tot,
                                  int* __restrict__ exps, double* __restrict__ digits)
{
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= C) return;
  double s = 0.0, a = 0.0, mn = -INFINITY;
  for (int b = threadIdx.x & 31; b < nblk; b += 32) {
    s += sums[(int64_t)c * nblk + b];
    a = fmax(a, amax[(int64_t)c * nblk + b]);
    mn = fmax(mn, namin[(int64_t)c * nblk + b]);
  }
  for (int o = 16; o; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
    mn = fmax(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  mn = -mn;
  if ((threadIdx.x & 31) == 0) {
    tot[c] = isfinite(a) ? s : NAN;
    exps[c] = digit_exp(a);
    digits[c] = isfinite(a) ? digit_count(digit_exp(a), mn, 24, -149) : 1;
  }
}

// The columns c0 … c0 + count − 1 of one pass: column c0 + b has the operand rows off[b] … off[b + 1] − 1, its digits.
struct DotsPass {
  int c0, count;
  int off[kDigitCols + 1];
};

// Their operand.  A non-finite column is stored as zeros (its products come out NaN through its total).
constexpr int kOpThreads = 64;   // small blocks: a short column's few threads spread over the SMs
__global__ void __launch_bounds__(kOpThreads)
dots_operand_kernel(ExactCols a, int64_t n, int64_t n_pad, const __grid_constant__ DotsPass P, const double* __restrict__ tot,
                    const int* __restrict__ exps, uint8_t* __restrict__ B)
{
  const int b = blockIdx.y, c = P.c0 + b;
  const int64_t i = ((int64_t)blockIdx.x * kOpThreads + threadIdx.x) * 16;
  if (i >= n_pad) return;
  const bool fine = !isnan(tot[c]);
  float v[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) v[u] = (i + u < n && fine) ? dot_column(a, c, i + u) : 0.f;
  const int digits = P.off[b + 1] - P.off[b];
  store_digits<float, int>(v, exps[c], B, n_pad, P.off[b], digits, 0, digits, i);
}

// out[b][j] of the pass; grid (rows, columns)
__global__ void __launch_bounds__(kXThreads)
dots_gather_kernel(const float* __restrict__ D, int splits, int kp, int64_t m_pad, int64_t m, const __grid_constant__ DotsPass P,
                   const double* __restrict__ tot, const int* __restrict__ exps, double* __restrict__ out)
{
  const int64_t j = (int64_t)blockIdx.x * kXThreads + threadIdx.x;
  if (j >= m) return;
  const int b = blockIdx.y, c = P.c0 + b;
  const double v = gather_digits(D, splits, kp, m_pad, P.off[b], P.off[b + 1] - P.off[b], j, 0.0);
  out[(int64_t)b * m + j] = isnan(tot[c]) ? NAN : ldexp(v, -exps[c]);
}

// Split-K count of an exact product over K_tiles K-tiles: at most kDigitKTiles of them each.
static int exact_splits(int64_t M_pad, int64_t K_tiles, int N)
{
  return choose_splits(M_pad / gemm_tc_rows_per_cta(N, 2), K_tiles, 1, num_sms(),
                       (int)ceil_div(K_tiles, kDigitKTiles));
}

void exact_gebv(slemm_geno* g, const double* d_alpha, double amax, double amin, double shift, double* d_tgv)
{
  cudaStream_t st = g->stream;
  const int e = digit_exp(amax), digits = digit_count(e, amin, 53, -1074);
  for (int p0 = (digits - 1) / kDigitRows * kDigitRows; p0 >= 0; p0 -= kDigitRows) {   // the last digits first
    const int cnt = std::min(kDigitRows, digits - p0);
    const int kp = (int)round_up(cnt, 8), N = (int)round_up(kp, 16);
    const int splits = exact_splits(g->n_pad, g->m_pad / kTileK, N);
    uint8_t* B = (uint8_t*)g->ws_B.ensure((size_t)N * g->m_pad);
    float* D = (float*)g->ws_D.ensure((size_t)splits * kp * g->n_pad * sizeof(float));
    gebv_operand_kernel<<<(unsigned)ceil_div(g->m_pad, 16 * 32), 32, 0, st>>>(d_alpha, g->m, g->m_pad, e, digits, p0, cnt,
                                                                                B);
    LAUNCH_CHECK();
    gemm_tc({g->GT.as<uint8_t>(), g->n_pad, g->m_pad, B, N, D, splits, g->err.as<int>(), kp, 1, false, 2}, st);
    gebv_finish_kernel<<<(unsigned)ceil_div(g->n, kXThreads), kXThreads, 0, st>>>(
        D, splits, kp, g->n_pad, g->n, cnt, p0 + cnt < digits, p0 == 0, e, shift, d_tgv);
    LAUNCH_CHECK();
  }
}

int exact_dots_guess(const slemm_geno* g, const ExactCols& a)
{
  constexpr int kGuess = 12;
  return kGuess * a.count() <= 96 && g->n_pad * g->m_pad <= (int64_t)1 << 31 ? kGuess : 0;
}

bool exact_dots_done(const slemm_geno* g, const ExactCols& a, int guess)
{
  for (int c = 0; c < a.count(); ++c)
    if (guess > 0 && g->scal.h[c] > (double)guess) return false;
  return true;
}

void exact_dots(slemm_geno* g, const ExactCols& a, double* dots, double* tot, double* twos, int guess)
{
  cudaStream_t st = g->stream;
  const int C = a.count();
  const int64_t n_pad = g->n_pad, m_pad = g->m_pad, K_tiles = n_pad / kTileK;
  const int nblk = (int)ceil_div(n_pad, kXRows);
  DevBuf dst(st);
  double* sums = (double*)dst.ensure((size_t)3 * C * nblk * sizeof(double) + C * sizeof(int));
  double *amax = sums + (size_t)C * nblk, *namin = amax + (size_t)C * nblk;
  int* exps = reinterpret_cast<int*>(namin + (size_t)C * nblk);
  const unsigned rows = (unsigned)ceil_div(g->m, kXThreads), oblk = (unsigned)ceil_div(n_pad, 16 * kOpThreads);
  dots_stats_kernel<<<dim3(nblk, C), kXThreads, 0, st>>>(a, g->n, sums, amax, namin, nblk);
  LAUNCH_CHECK();
  dots_scale_kernel<<<(unsigned)ceil_div(C * 32, 128), 128, 0, st>>>(sums, amax, namin, nblk, C, tot, exps,
                                                                     g->scal.ensure(C));
  LAUNCH_CHECK();
  if (guess == 0) CUDA_TRY(cudaStreamSynchronize(st));   // the columns' numbers of digits
  auto run = [&](const DotsPass& P, double* out, bool high) {
    const int kp = (int)round_up(P.off[P.count], 8), N = (int)round_up(kp, 16);
    const int splits = exact_splits(m_pad, K_tiles, N);
    uint8_t* B = (uint8_t*)g->ws_B.ensure((size_t)N * n_pad);
    float* D = (float*)g->ws_D.ensure((size_t)splits * kp * m_pad * sizeof(float));
    dots_operand_kernel<<<dim3(oblk, P.count), kOpThreads, 0, st>>>(a, g->n, n_pad, P, tot, exps, B);
    LAUNCH_CHECK();
    gemm_tc({g->G.as<uint8_t>(), m_pad, n_pad, B, N, D, splits, g->err.as<int>(), kp, 1, false, 2, high}, st);
    dots_gather_kernel<<<dim3(rows, P.count), kXThreads, 0, st>>>(D, splits, kp, m_pad, g->m, P, tot, exps, out);
    LAUNCH_CHECK();
  };
  std::vector<double> digits(C, (double)guess);
  if (guess == 0) digits.assign(g->scal.h, g->scal.h + C);
  for (int c = 0; c < C;) {   // as many columns per pass as fit
    DotsPass P{c, 0, {0}};
    while (c < C && P.count < kDigitCols && P.off[P.count] + (int)digits[c] <= kDigitRows) {
      P.off[P.count + 1] = P.off[P.count] + (int)digits[c];
      ++P.count;
      ++c;
    }
    run(P, dots + (size_t)P.c0 * g->m, false);
  }
  if (twos != nullptr)   // 2·Σ rr²·[count = 2]: the last column (rr²) against the high bits
    run({C - 1, 1, {0, (int)digits[C - 1]}}, twos, true);
}

}  // namespace slemm

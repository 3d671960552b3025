// gemm_simt.cu — FP32 CUDA-core packed product (the plain FP32 path).
//
// D[s][c][r] = Σ_{K in split s} count[r,K] · B[c][K] for a 128-row tile per CTA: thread t owns
// row t, reads its 16 packed bytes of each tile (the CTA's 128 threads read one contiguous
// 2048-byte tile), decodes exact counts to FP32 and multiplies and adds in FP32 like the
// reference's SGEMM (src/reml.cpp:36, 144, 182, 220), one K-tile at a time, folding each tile's
// sum into a double-float accumulator.  B columns are staged in shared memory for kStageTiles
// tiles at a time and read as broadcasts.
//
// Bound by the SMs' issue slots: with one column, a pair of counts took a LOP3 and an HFMA2 (BF16 pair),
// two unpacking instructions and two FMAs, 3.5 instructions a count with the broadcast loads.  A masked
// 2-bit field is already an FP32 number: at bits 2s, 2s + 1 of a word (s ≤ 11) it reads as x·2^(2s−149),
// a subnormal (bit 23 is the exponent's lowest, and 2^−126 = 2·2^(22−149)), which FMAs take at full
// rate.  So a count costs one LOP and one FMA, and one shift serves the last four fields of a word.  The
// staged B carries 2^(100−2s) for its position, so that products are x·b·2^−49.  That gives the same bits
// as x·b where every nonzero |b| of the stage lies in [2^−76, 2^28): the staged value is finite, products are
// normal, and a sum that cancels below 2^−126 is a multiple of 2^−148 like its terms, so nothing rounds there
// that would not have.  A stage with any other value (subnormal, non-finite or just far from 1) takes the
// counts as BF16 pairs instead, at the old cost.  One column at n = 100,000, m = 20,000, H0_ldet_mv: 652 → 433 µs.
#include "common.h"
#include "decode.cuh"
#include "reduce.cuh"

namespace slemm {

constexpr int kStageTiles = 8;                 // 512 K elements per shared-memory stage
constexpr int kStageK = kStageTiles * kTileK;

template <int KC>
__global__ void __launch_bounds__(128)
gemm_simt_kernel(const uint4* __restrict__ A, int64_t M_pad, int64_t K_tiles,
                 const float* __restrict__ B, int64_t K_pad, int c0, int k_total,
                 float* __restrict__ D, int N, int tiles_per_split)
{
  __shared__ __align__(16) float sB[kStageK * KC];   // [element][column]
  const int t = threadIdx.x;
  const int64_t mt = blockIdx.x;
  const int s = blockIdx.y;
  const int64_t kt0 = (int64_t)s * tiles_per_split;
  const int64_t kt1 = min64(K_tiles, kt0 + tiles_per_split);
  // Each K-tile's 64 products are summed in FP32 and folded into a double-float sum per column:
  // one FP32 chain over a whole split (10^5 elements at 500,000 individuals) loses ~1e-5 of the
  // result to rounding, 64-element chains ~3e-7.
  DF acc[KC];

  for (int64_t ks = kt0; ks < kt1; ks += kStageTiles) {
    const int ntile = (int)min64(kStageTiles, kt1 - ks);
    uint4 pk[kStageTiles];
#pragma unroll
    for (int u = 0; u < kStageTiles; ++u)
      pk[u] = u < ntile ? A[((mt * K_tiles + ks + u) * 128 + t)] : make_uint4(0u, 0u, 0u, 0u);
    // stage B[c0 .. c0+KC)[ks*64 .. +ntile*64), element t + 128i of each column
    float raw[KC][kStageK / 128];
    bool near = true;   // 0 or in [2^−76, 2^28)
#pragma unroll
    for (int c = 0; c < KC; ++c)
#pragma unroll
      for (int i = 0; i < kStageK / 128; ++i) {
        const int kk = t + 128 * i, col = c0 + c;
        raw[c][i] = (col < k_total && kk < ntile * kTileK) ? B[(int64_t)col * K_pad + ks * kTileK + kk] : 0.f;
        const uint32_t mag = __float_as_uint(raw[c][i]) & 0x7FFFFFFFu;
        near = near && (mag == 0u || mag - ((127u - 76u) << 23) < (104u << 23));
      }
    near = __syncthreads_and(near);   // and every thread is done with the last stage
    const float kscale = near ? __uint_as_float((uint32_t)(127 + 100 - 2 * f32sub_shift(t & 15)) << 23) : 1.f;   // 128 ≡ 0 mod 16
#pragma unroll
    for (int c = 0; c < KC; ++c)
#pragma unroll
      for (int i = 0; i < kStageK / 128; ++i)
        sB[(t + 128 * i) * KC + c] = __fmul_rn(raw[c][i], kscale);
    __syncthreads();
    if (!near) {
      for (int u = 0; u < ntile; ++u) {
        const uint4 p4 = A[(mt * K_tiles + ks + u) * 128 + t];
        const uint32_t words[4] = {p4.x, p4.y, p4.z, p4.w};
        float part[KC];
#pragma unroll
        for (int c = 0; c < KC; ++c) part[c] = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w)
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t pair = bf16pair_of(words[w], q);   // FP32 in either half
            const float* b = &sB[(u * kTileK + w * 16 + 2 * q) * KC];
#pragma unroll
            for (int c = 0; c < KC; ++c)
              part[c] = fmaf(__uint_as_float(pair << 16), b[c], fmaf(__uint_as_float(pair & 0xFFFF0000u), b[KC + c], part[c]));
          }
#pragma unroll
        for (int c = 0; c < KC; ++c) df_add(acc[c], part[c]);
      }
      continue;
    }
#pragma unroll
    for (int u = 0; u < kStageTiles; ++u) {
      if (u >= ntile) break;
      const uint32_t words[4] = {pk[u].x, pk[u].y, pk[u].z, pk[u].w};
      float part[KC];
#pragma unroll
      for (int c = 0; c < KC; ++c) part[c] = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint32_t top = words[w] >> 24;
#pragma unroll
        for (int q = 0; q < 8; q += 2) {   // elements 2q … 2q + 3
          const float4* bp = reinterpret_cast<const float4*>(&sB[(u * kTileK + w * 16 + 2 * q) * KC]);
          float bb[4 * KC];
#pragma unroll
          for (int i = 0; i < KC; ++i) {
            const float4 v = bp[i];
            bb[4 * i] = v.x, bb[4 * i + 1] = v.y, bb[4 * i + 2] = v.z, bb[4 * i + 3] = v.w;
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int qq = q + h;
            const float xe = f32sub_of(words[w], top, 2 * qq), xo = f32sub_of(words[w], top, 2 * qq + 1);
#pragma unroll
            for (int c = 0; c < KC; ++c)
              part[c] = fmaf(xe, bb[2 * h * KC + c], fmaf(xo, bb[(2 * h + 1) * KC + c], part[c]));
          }
        }
      }
#pragma unroll
      for (int c = 0; c < KC; ++c) df_add(acc[c], __fmul_rn(part[c], 562949953421312.f));   // 2^49
    }
  }
#pragma unroll
  for (int c = 0; c < KC; ++c) {
    const int col = c0 + c;
    if (col < k_total) D[((int64_t)s * N + col) * M_pad + mt * 128 + t] = __fadd_rn(acc[c].hi, acc[c].lo);
  }
}

void gemm_simt(const GemmArgs& a, cudaStream_t st)
{
  const int64_t M_tiles = a.M_pad / kTileM, K_tiles = a.K_pad / kTileK;
  const int tps = (int)ceil_div(K_tiles, a.splits);
  dim3 grid((unsigned)M_tiles, (unsigned)a.splits);
  const float* B = static_cast<const float*>(a.B);
  int c0 = 0;
  while (c0 < a.N) {
    const int rem = a.N - c0;
    if (rem >= 8) {
      gemm_simt_kernel<8><<<grid, 128, 0, st>>>((const uint4*)a.A, a.M_pad, K_tiles, B, a.K_pad, c0,
                                                a.N, a.D, a.N, tps);
      c0 += 8;
    } else if (rem >= 4) {
      gemm_simt_kernel<4><<<grid, 128, 0, st>>>((const uint4*)a.A, a.M_pad, K_tiles, B, a.K_pad, c0,
                                                a.N, a.D, a.N, tps);
      c0 += 4;
    } else if (rem >= 2) {
      gemm_simt_kernel<2><<<grid, 128, 0, st>>>((const uint4*)a.A, a.M_pad, K_tiles, B, a.K_pad, c0,
                                                a.N, a.D, a.N, tps);
      c0 += 2;
    } else {
      gemm_simt_kernel<1><<<grid, 128, 0, st>>>((const uint4*)a.A, a.M_pad, K_tiles, B, a.K_pad, c0,
                                                a.N, a.D, a.N, tps);
      c0 += 1;
    }
    LAUNCH_CHECK();
  }
}

}  // namespace slemm

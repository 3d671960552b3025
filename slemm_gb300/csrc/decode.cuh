// decode.cuh — 2-bit packed counts → BF16 / FP16 / FP32 (device helpers shared by the kernels).
//
// A 32-bit word holds 16 counts x ∈ {0,1,2} as 2-bit binary fields (layout in geno.cu): the even
// elements 2q in bits 2q..2q+1 of the low half-word, the odd elements 2q+1 in bits 16+2q.. of the
// high half-word.  For the element pair q (elements 2q, 2q+1) and k = 2·(q mod 4), taking
// src = word (q < 4) or word ≫ 8 (q ≥ 4):
//   (src & (0x00030003 ≪ k)) | 0x43004300
// is a BF16 pair whose halves are exactly 128 + x·2^k (0x4300 is 128; the count lands in the
// mantissa, or for k = 6 and x = 2 carries into the exponent, which is still 256 = 128 + 2·64).
// One BF16 FMA, v·2^−k − 128·2^−k, then gives x exactly.  So a pair costs one AND-OR on the
// integer pipe and one HFMA2 on the FMA pipe (plus one shift per 8 pairs).
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

namespace slemm {

__device__ __forceinline__ uint32_t bf16pair_of(uint32_t word, int q)
{
  const uint32_t src = (q < 4) ? word : (word >> 8);
  const int k = 2 * (q & 3);
  const uint32_t bits = (src & (0x00030003u << k)) | 0x43004300u;
  const float sc = 1.0f / (float)(1 << k);
  const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&bits);
  const __nv_bfloat162 r = __hfma2(v, __float2bfloat162_rn(sc), __float2bfloat162_rn(-128.0f * sc));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// The pair as FP16 subnormals, by masking alone: an FP16 whose exponent field is zero is
// mantissa·2^−24, so a count x whose 2-bit field sits at bits 2s, 2s+1 of a half-word (s ≤ 4,
// inside the 10-bit mantissa) reads as x·2^(2s−24).  Pairs q = 0 … 4 are masked in place
// (s = q); pairs 5 … 7 from the word shifted right by 10 (s = q − 5).  The product's other
// operand carries the factor 2^−2s of its K position (f16sub_kscale) and the accumulator is
// multiplied by 2^24, so count·operand is the same product, exactly: one LOP per pair and one
// shift per word.
__device__ __forceinline__ int f16sub_shift(int q) { return q < 5 ? q : q - 5; }
__device__ __forceinline__ uint32_t f16sub_pair_of(uint32_t word, int q)
{
  const uint32_t src = (q < 5) ? word : (word >> 10);
  return src & (0x00030003u << (2 * f16sub_shift(q)));
}
// 2^−2s for the element at K index kidx (K-tiles start at multiples of 64; element j of a
// 16-element word is K index ≡ j mod 16, pair q = j / 2).
__device__ __forceinline__ float f16sub_kscale(int64_t kidx)
{
  const int s = f16sub_shift((int)((kidx & 15) >> 1));
  return __uint_as_float((uint32_t)(127 - 2 * s) << 23);
}
__device__ __forceinline__ float f16sub_kunscale(int64_t kidx)
{
  const int s = f16sub_shift((int)((kidx & 15) >> 1));
  return __uint_as_float((uint32_t)(127 + 2 * s) << 23);
}
constexpr float kF16SubUnscale = 16777216.0f;   // 2^24

template <bool F16>
__device__ __forceinline__ uint32_t pair_of(uint32_t word, int q)
{
  if constexpr (F16) return f16sub_pair_of(word, q);
  else return bf16pair_of(word, q);
}

// Half the bit position s of element j (0 … 15) of a word read as an FP32 subnormal (x·2^(2s−149), gemm_simt.cu): even elements 2q at bits 2q, odd ones at 16 + 2q, the odd ones
// from q = 4 on read from the word shifted right by 24.
__host__ __device__ constexpr int f32sub_shift(int j)
{
  const int q = j >> 1;
  return (j & 1) == 0 ? q : (q < 4 ? 8 + q : q - 4);
}

// Those bits: top is the word shifted right by 24.
__device__ __forceinline__ float f32sub_of(uint32_t word, uint32_t top, int j)
{
  const int q = j >> 1;
  return __uint_as_float((j & 1) == 0 ? word & (3u << (2 * q)) : q < 4 ? word & (3u << (16 + 2 * q)) : top & (3u << (2 * q - 8)));
}

// Four counts of a word as E4M3 bytes, by masking alone: a byte whose low two bits hold x is the
// subnormal x·2^−9, and one whose bits 2, 3 hold x (mantissa and exponent zero elsewhere) reads as
// x·2^−7 — x = 1 is the subnormal 4·2^−9, x = 2 the exponent field 1, 2^−6.  Group p = 0 … 3 of a
// word is the mask 0x03 (p even) or 0x0C (p odd) on every byte of the word (p < 2) or of the
// word shifted right by 4: four LOPs and one shift for 16 counts.  Byte b of group p is element
// {2p, 8+2p, 2p+1, 9+2p}[b] of the word, the order the dense operand's K positions 4p + b follow, and
// the operand carries 2^−2 at odd p; the accumulator is multiplied by 2^9.  TWOS: 2·[x = 2] instead of x.
template <bool TWOS>
__device__ __forceinline__ uint32_t f8_quad_of(uint32_t word, int p)
{
  const uint32_t src = (p < 2) ? word : (word >> 4);
  return src & ((p & 1) ? (TWOS ? 0x08080808u : 0x0C0C0C0Cu) : (TWOS ? 0x02020202u : 0x03030303u));
}
constexpr float kF8Unscale = 512.0f;   // 2^9

// Four integers |d| ≤ 16 as E4M3 bytes (4 significant bits: exact), times 1 or 2^−2.
__device__ __forceinline__ uint32_t e4m3x4(float d0, float d1, float d2, float d3, float s)
{
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(d0 * s, d1 * s), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(d2 * s, d3 * s), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}
// The 16 K positions of one word's elements d[0 … 15] in the decoded order.
__device__ __forceinline__ uint4 e4m3_word(const float (&d)[16])
{
  return make_uint4(e4m3x4(d[0], d[8], d[1], d[9], 1.f), e4m3x4(d[2], d[10], d[3], d[11], 0.25f),
                    e4m3x4(d[4], d[12], d[5], d[13], 1.f), e4m3x4(d[6], d[14], d[7], d[15], 0.25f));
}

// The 8 K positions 8h … 8h + 7 of a word: digits of its elements 4h … 4h + 3 (d[0 … 3]) and
// 8 + 4h … 11 + 4h (d[4 … 7]).
__device__ __forceinline__ uint2 e4m3_half(const float (&d)[8])
{
  return make_uint2(e4m3x4(d[0], d[4], d[1], d[5], 1.f), e4m3x4(d[2], d[6], d[3], d[7], 0.25f));
}

}  // namespace slemm

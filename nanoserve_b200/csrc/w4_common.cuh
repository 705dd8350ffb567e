// Device helpers shared by the W4A16 kernels: the packed-int4 format and its unpack.
//
// Format (fixed by the operator boundary; reference kernels/quant/w4a16.cuh:5-9):
//   Wq [N, K/8] uint32, word j of row n packs k = 8j..8j+7, value 8j+i in bits 4i..4i+3
//   S  [N, K/G] bf16,   w[n,k] = (q - 8) * S[n, k/G]
#pragma once
#include <cstdint>
#include <cuda_bf16.h>

namespace b2 {

// bf16 bit patterns used by the unpack: 0x4300 = 128.0 (exponent 2^7, so the 7 mantissa bits count
// in units of 1), 0x4308 = 136.0 = 128 + the zero-point 8.
constexpr uint32_t kMagic128x2 = 0x43004300u;
constexpr uint32_t kMagic136x2 = 0x43084308u;
constexpr uint32_t kNibblePairMask = 0x000F000Fu;

// One packed word -> four bf16x2 registers holding 128 + q, with the pairing the bit layout gives for
// free: r[p] = { 128 + q[p] (low half), 128 + q[p + 4] (high half) }, p = 0..3.  Three shifts and four
// three-input logic ops per eight weights; the integers 128..143 are exact in bf16.
__device__ __forceinline__ void unpack_w4_biased(uint32_t w, uint32_t (&r)[4]) {
  r[0] = (w & kNibblePairMask) | kMagic128x2;
  r[1] = ((w >> 4) & kNibblePairMask) | kMagic128x2;
  r[2] = ((w >> 8) & kNibblePairMask) | kMagic128x2;
  r[3] = ((w >> 12) & kNibblePairMask) | kMagic128x2;
}

// bf16x2 subtract of 136: (128 + q) - 136 = q - 8, exact.
__device__ __forceinline__ uint32_t sub136_bf16x2(uint32_t v) {
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&v);
  const uint32_t c = kMagic136x2;
  a = __hsub2(a, *reinterpret_cast<const __nv_bfloat162*>(&c));
  return *reinterpret_cast<uint32_t*>(&a);
}
// bf16x2 multiply (round-to-nearest-even per half).
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t v, uint32_t s2) {
  __nv_bfloat162 a = *reinterpret_cast<__nv_bfloat162*>(&v);
  a = __hmul2(a, *reinterpret_cast<const __nv_bfloat162*>(&s2));
  return *reinterpret_cast<uint32_t*>(&a);
}
__device__ __forceinline__ uint32_t bf16_dup(__nv_bfloat16 s) {
  const uint32_t b = __bfloat16_as_ushort(s);
  return b | (b << 16);
}

// One packed word -> four bf16 pairs of (q - 8) * s in their natural order {w0,w1} {w2,w3} {w4,w5} {w6,w7}, each rounded once.
// A byte b in the low half of a bf16 is the number b * 2^-133 (up to 127 a subnormal, above it a normal, on one line), so
// the even nibbles of the word, as 8 q, are q * 2^-130, the odd ones, left where they are as 16 q, q * 2^-129; the byte above
// is zero, the sign of an even nibble's byte.  The rest is one fused multiply-add per pair: q * s - 8 s, whose addend is exact
// (8 is a power of two, the 136 of a biased nibble is not), is rounded once, as the product (q - 8) * s is.  Eleven
// instructions per eight weights, six of them on the ALU pipe that bounds the conversion (two cycles each); unpacked to 128 + q,
// 136 subtracted and multiplied it took 17 and nine.  (Even nibbles as q, a shift less, leave s * 2^133 finite only below 1/32; weights
// carried at 2^-8 of their size to make up for that lost bits below 2^-118.)
// The multiplier s * 2^130 is finite for scales below a quarter.  Other scales, infinities and nans among them: dequant_word_any.
struct DequantScale {
  uint32_t mul, add;
};
__device__ __forceinline__ DequantScale dequant_scale(uint32_t s2) {
  return {mul_bf16x2(mul_bf16x2(s2, 0x7E807F00u), 0x41004100u), mul_bf16x2(s2, 0xC100C100u)};  // s * {2^127, 2^126} * 8, -s * 8
}
__device__ __forceinline__ bool dequant_scale_plain(uint32_t s2) { return (s2 & 0x7FFFu) < 0x3E80u; }
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
template <int I>
__device__ __forceinline__ uint32_t nibble_pair(uint32_t even, uint32_t odd) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(even), "r"(odd), "n"(I | (8 | I) << 4 | (4 + I) << 8 | (8 | I) << 12));
  return d;
}
__device__ __forceinline__ void dequant_word(uint32_t w, const DequantScale& sc, uint32_t* o) {
  const uint32_t even = (w << 3) & 0x78787878u, odd = w & 0xF0F0F0F0u;
  o[0] = fma_bf16x2(nibble_pair<0>(even, odd), sc.mul, sc.add);
  o[1] = fma_bf16x2(nibble_pair<1>(even, odd), sc.mul, sc.add);
  o[2] = fma_bf16x2(nibble_pair<2>(even, odd), sc.mul, sc.add);
  o[3] = fma_bf16x2(nibble_pair<3>(even, odd), sc.mul, sc.add);
}
// Any scale: (q - 8) / 8 and q - 8 exactly, then the product.
__device__ __forceinline__ void dequant_word_any(uint32_t w, uint32_t s2, uint32_t* o) {
  const DequantScale eighth = {0x7E807F00u, 0xBF80BF80u};  // {2^127, 2^126}, -1
  dequant_word(w, eighth, o);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = mul_bf16x2(mul_bf16x2(o[i], 0x41004100u), s2);
}

// 16-byte shared-memory accesses by 32-bit shared address.
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

}  // namespace b2

// Arithmetic that the kernels of the packed linears share: packed words to 16-bit weights, pairs of 16-bit numbers, silu(gate) * up,
// and the order of columns in tensor memory.
#pragma once
#include "common.cuh"
#include "tma_utils.cuh"
#include "umma_utils.cuh"

namespace nqb200 {

template <bool BF16> __device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF16) asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF16> __device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  uint32_t r;
  if (BF16) asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  else asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
template <bool BF16> __device__ __forceinline__ uint32_t round2(float lo, float hi) {
  uint32_t r;
  if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t fma2_f16(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}
// (a & mask) | bits, with mask and bits in registers: one instruction.  (Written with both as constants 777 tokens of 12288 -> 4096 took 101.9
// us instead of 100.5, and 4096 of 5120 -> 25600 829 instead of 825.)
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
  return r;
}

// silu(g) * u of two 16-bit pairs with the roundings of the separate steps (g / (1 + exp(-g)) in float, rounded; the product,
// rounded).  The quotient is a reciprocal estimate with one correction by its remainder (Markstein's): the same 16 bits as the
// divide for every g, at half its instructions.  The product of two 16-bit values needs no float: one rounding either way.
__device__ __forceinline__ uint64_t pack_f2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul_f2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
template <bool BF16> __device__ __forceinline__ uint32_t silu_mul2(uint32_t gw, uint32_t uw) {
  const float g0 = raw16_to_float<BF16>((uint16_t)gw), g1 = raw16_to_float<BF16>((uint16_t)(gw >> 16));
  const float d0 = 1.f + expf(-g0), d1 = 1.f + expf(-g1);
  float r0, r1, q0, q1, p0, p1;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r0) : "f"(d0));
  asm("rcp.approx.f32 %0, %1;" : "=f"(r1) : "f"(d1));
  const uint64_t g = pack_f2(g0, g1), r = pack_f2(r0, r1), q = mul_f2(g, r);
  const uint64_t p = fma_f2(fma_f2(q, pack_f2(-d0, -d1), g), r, q);
  asm("mov.b64 {%0, %1}, %2;" : "=f"(q0), "=f"(q1) : "l"(q));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(p0), "=f"(p1) : "l"(p));
  // an infinite gate or divisor has no remainder, and that of -0 would take its sign
  const float s0 = p0 == p0 && q0 != 0.f ? p0 : q0, s1 = p1 == p1 && q1 != 0.f ? p1 : q1;
  return mul2<BF16>(round2<BF16>(s0, s1), uw);
}

// The column of an A block's 128 that lane `l` of tensor memory holds (the order the dequantisers' stores give).
__device__ __forceinline__ int column_of_lane(int l) {
  const int q = l >> 5, ph = (l >> 4) & 1, r = (l >> 3) & 1, g = l & 7;
  return 32 * q + 8 * (g >> 1) + 4 * ph + 2 * r + (g & 1);
}

}  // namespace nqb200

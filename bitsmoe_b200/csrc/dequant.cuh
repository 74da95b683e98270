// Arena words -> fp16 weights, and the activation, shared by the kernels that multiply (q * scale) operands.
#pragma once

#include "fast_layout.cuh"

namespace bm {

// One arena word (a 16x16 block's codes owned by lane (g, t), see fast_layout.cuh) -> four fp16 pairs
// (q * scale): r[0] = row g, k (2t, 2t+1); r[1] = row g+8, same k; r[2] = row g, k (2t+8, 2t+9); r[3] = row g+8.
// The code sits in the mantissa of 1024 (fields at bit 0) or of 64 (fields at bit 4); subtracting
// 1024 + offset or 64 + offset is exact, the multiplication by the scale rounds once, as fp16(q * scale) does.
// The exponents 1024 and 64 as fp16 pairs, held in registers as opaque values, so that (w & mask) | k needs one immediate
// operand only (8192 tokens 185 -> 179 us against constants).
struct DqMagic {
  uint32_t lo, hi;
  __device__ __forceinline__ DqMagic() {
    asm volatile("mov.b32 %0, 0x64006400;" : "=r"(lo));
    asm volatile("mov.b32 %0, 0x54005400;" : "=r"(hi));
  }
};
template <uint32_t MASK>
__device__ __forceinline__ uint32_t and_or(uint32_t w, uint32_t k) {
  uint32_t v;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(v) : "r"(w), "n"(MASK), "r"(k));
  return v;
}
template <bool DENSE>
__device__ __forceinline__ void dequant_block(const DqMagic& k, uint32_t w, __half2 s0, __half2 s1, __half2 s2, __half2 s3, uint32_t (&r)[4]) {
  constexpr uint32_t mlo = DENSE ? 0x00030003u : 0x000F000Fu, mhi = DENSE ? 0x00300030u : 0x00F000F0u;
  constexpr uint32_t off = DENSE ? FAST_DENSE_OFFSET : FAST_NIB_OFFSET;
  constexpr uint32_t blo_bits = 0x64006400u + off * 0x00010001u;          // fp16x2 of 1024 + offset
  constexpr uint32_t bhi_bits = 0x54005400u + off * 0x00100010u;          // fp16x2 of 64 + offset
  const uint32_t blo_u = blo_bits, bhi_u = bhi_bits;
  const __half2 blo = *reinterpret_cast<const __half2*>(&blo_u), bhi = *reinterpret_cast<const __half2*>(&bhi_u);
  const uint32_t sh = w >> (DENSE ? 2 : 8);
  uint32_t v[4] = {and_or<mlo>(w, k.lo), and_or<mhi>(w, k.hi), and_or<mlo>(sh, k.lo), and_or<mhi>(sh, k.hi)};
  const __half2 o0 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&v[0]), blo), s0);
  const __half2 o1 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&v[1]), bhi), s1);
  const __half2 o2 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&v[2]), blo), s2);
  const __half2 o3 = __hmul2(__hsub2(*reinterpret_cast<__half2*>(&v[3]), bhi), s3);
  r[0] = *reinterpret_cast<const uint32_t*>(&o0);
  r[1] = *reinterpret_cast<const uint32_t*>(&o1);
  r[2] = *reinterpret_cast<const uint32_t*>(&o2);
  r[3] = *reinterpret_cast<const uint32_t*>(&o3);
}

// silu(g) * u = g * u / (1 + e^-g), with e^-g as 2^(-g log2 e); where that power is subnormal and flushed to zero it could not
// have changed the sum 1 + e^-g
__device__ __forceinline__ float silu_mul(float g, float u) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-1.4426950408889634f * g));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return g * u * r;
}

}  // namespace bm

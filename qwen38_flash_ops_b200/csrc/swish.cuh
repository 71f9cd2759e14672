// swish_mul in the BF16 arithmetic of SharedExpertDown, two values per word.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace qfg {
namespace {

// sigmoid(a) before its rounding, for a BF16 a: exp(-|a|) as 2^y with y = -|a| h exact (h: the upper 16 bits of log2 e,
// against the eight of a) and the rest of the exponent to first order, then a reciprocal; next to zero, where a / 4 can
// lie on a rounding boundary to within less than an ulp, the Taylor polynomial.  Fifteen instructions where expf and an
// IEEE division take over forty; after rounding the same for each of the 65536 inputs.
__device__ __forceinline__ float SigmoidOfBf16(float a) {
  const float x = fminf(fabsf(a), 256.f);  // 2^-369 is zero
  constexpr float h = 47274.f / 32768.f, rest = 4.888495e-06f;  // log2 e = h + 7.052608e-6; that times ln 2
  float e, r;
  asm("ex2.approx.f32 %0, %1;" : "=f"(e) : "f"(x * -h));
  e = fmaf(e, x * -rest, e);
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.0f + e));
  const float far = (a > 0.0f ? 1.0f : e) * r, near = fmaf(a, fmaf(a * a, -1.f / 48.f, 0.25f), 0.5f);
  return x < 0.03125f ? near : far;
}
__device__ __forceinline__ uint32_t PackBf16(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&b);
}
__device__ __forceinline__ uint32_t MulBf16x2(uint32_t a, uint32_t b) {  // one rounding, like the FP32 product rounded
  uint32_t r;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ float Lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float Hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t SwishMul2(uint32_t g2, uint32_t u2) {  // two BF16 per word
  return MulBf16x2(MulBf16x2(g2, PackBf16(SigmoidOfBf16(Lo(g2)), SigmoidOfBf16(Hi(g2)))), u2);
}

}  // namespace
}  // namespace qfg

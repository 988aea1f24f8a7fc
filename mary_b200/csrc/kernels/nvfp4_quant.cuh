// NVFP4 activation quantiser pieces shared by the kernels that quantise in flight (dispatch, GLU epilogue).
// Rules (src/models/inkling/fp4quant.rs:10-54): per 16 elements amax -> sf = min(amax / 6, 448) -> E4M3 round-to-nearest-even;
// codes by the thresholds .25 .75 1.25 1.75 2.5 3.5 5 on |x / sf| with >= (ties away from zero), the sign bit kept for values
// that round to zero, a zero block -> scale byte 0 and codes 0.
#pragma once
#include <cuda_fp8.h>

#include "common.cuh"

namespace mary {

// Codes by the conversion instruction.  It rounds ties to even, the rule rounds them away from zero, so the quotient is first raised by 2^-12 of itself:
// a value is bf16 (8 significant bits) and a threshold times a scale has at most 7, so a quotient that is not ON a threshold is at least 2^-8 of it
// away, which neither the raise nor the rounding of the reciprocal and the product (2^-23) can cross.  Against a division and seven comparisons per
// value this is one product and half a conversion.
__device__ __forceinline__ float nvfp4_inverse(float scale) { return __frcp_rn(scale) * (1.0f + 1.0f / 4096.0f); }      // scale > 0
__device__ __forceinline__ float nvfp4_quotient(float v, float inverse) {
  const float y = v * inverse;
  return y == y ? y : copysignf(0.f, v);                   // not a number: code 0 with its sign
}
// low byte: the code of y0 in bits 0-3, of y1 in bits 4-7
__device__ __forceinline__ uint32_t nvfp4_pair(float y0, float y1) {
  uint32_t r;
  asm("{\n\t.reg .b8 c;\n\tcvt.rn.satfinite.e2m1x2.f32 c, %2, %1;\n\tmov.b32 %0, {c, 0, 0, 0};\n\t}" : "=r"(r) : "f"(y0), "f"(y1));
  return r;
}
__device__ __forceinline__ uint32_t nvfp4_pack8(const float* v, float inverse) {
  float y[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) y[j] = nvfp4_quotient(v[j], inverse);
  uint32_t r;
  asm("{\n\t.reg .b8 c0, c1, c2, c3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 c0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 c1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 c2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 c3, %8, %7;\n\t"
      "mov.b32 %0, {c0, c1, c2, c3};\n\t}"
      : "=r"(r) : "f"(y[0]), "f"(y[1]), "f"(y[2]), "f"(y[3]), "f"(y[4]), "f"(y[5]), "f"(y[6]), "f"(y[7]));
  return r;
}
// Scale byte of a block with absolute maximum `amax`, and its decoded value.
__device__ __forceinline__ uint8_t nvfp4_scale_byte(float amax, float* decoded) {
  const float sfv = fminf(__fdiv_rn(amax, 6.0f), 448.0f);
  const __nv_fp8_storage_t sb = __nv_cvt_float_to_fp8(sfv, __NV_SATFINITE, __NV_E4M3);
  *decoded = __half2float(__half(__nv_cvt_fp8_to_halfraw(sb, __NV_E4M3)));
  return (uint8_t)sb;
}

// 16 values (two 16-byte vectors of bf16) -> 8 code bytes and the scale byte of their block
__device__ __forceinline__ uint2 nvfp4_block16(const uint4& v0, const uint4& v1, uint8_t* scale) {
  float f[16];
  const __nv_bfloat162* p0 = (const __nv_bfloat162*)&v0;
  const __nv_bfloat162* p1 = (const __nv_bfloat162*)&v1;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = __bfloat1622float2(p0[j]), c = __bfloat1622float2(p1[j]);
    f[2 * j] = a.x; f[2 * j + 1] = a.y; f[8 + 2 * j] = c.x; f[8 + 2 * j + 1] = c.y;
  }
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
  float s;
  *scale = nvfp4_scale_byte(amax, &s);
  if (!(s > 0.f)) return make_uint2(0, 0);
  const float inverse = nvfp4_inverse(s);
  return make_uint2(nvfp4_pack8(f, inverse), nvfp4_pack8(f + 8, inverse));
}

}  // namespace mary

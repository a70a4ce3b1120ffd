// The per-16 fp4 quantizer of activations for one block that is in registers as bf16, shared by the stand-alone quantizers
// and by the GEMM epilogue that emits the next GEMM's operand directly. Internal linkage: each user includes it once.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include <cstdint>

#include "ptx.cuh"

namespace sfq {
namespace {

__device__ __forceinline__ uint32_t habs2(uint32_t a) {
  uint32_t d;
  asm("abs.bf16x2 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ uint32_t hmax2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// The scale byte of a block from its largest magnitude, bf16 in the low half of `m`: e4m3_rn_sat(amax / 6).
__device__ __forceinline__ uint8_t fp4_scale_byte(uint32_t m) {
  return uint8_t(__nv_cvt_float_to_fp8(__uint_as_float(m << 16) * (1.0f / 6.0f), __NV_SATFINITE, __NV_E4M3));
}

// Eight values -> four bytes of e2m1 pairs. HIGH_EVEN: the even element in the high nibble (GEMM feed), else in the low one.
template <bool HIGH_EVEN> __device__ __forceinline__ uint32_t e2m1_word(const float (&v)[8]) {
  uint32_t w;
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b0, %1, %2;\n\tcvt.rn.satfinite.e2m1x2.f32 b1, %3, %4;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 b2, %5, %6;\n\tcvt.rn.satfinite.e2m1x2.f32 b3, %7, %8;\n\t"
      "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
      : "=r"(w)
      : "f"(v[HIGH_EVEN ? 0 : 1]), "f"(v[HIGH_EVEN ? 1 : 0]), "f"(v[HIGH_EVEN ? 2 : 3]), "f"(v[HIGH_EVEN ? 3 : 2]),
        "f"(v[HIGH_EVEN ? 4 : 5]), "f"(v[HIGH_EVEN ? 5 : 4]), "f"(v[HIGH_EVEN ? 6 : 7]), "f"(v[HIGH_EVEN ? 7 : 6]));
  return w;
}

// s8 = fp4_scale_byte, inv = 1 / decode(s8) (0 for an all-zero block), code = e2m1_rn_sat(x * inv)
// (quantize_act_kernel, src/cuda/nvfp4_gemm.cu:107-158). A block of NaNs alone has a NaN scale here; the norm in front of the
// quantizer, which makes whole rows NaN, lets the maximum start at 0 like the reference.
template <bool FEED>
__device__ __forceinline__ void quantize_block16(const uint4 r0, const uint4 r1, uint2& codes, uint8_t& s8) {
  const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};  // element 2i in the low half of word i
  uint32_t m = hmax2(hmax2(hmax2(habs2(w[0]), habs2(w[1])), hmax2(habs2(w[2]), habs2(w[3]))),
                     hmax2(hmax2(habs2(w[4]), habs2(w[5])), hmax2(habs2(w[6]), habs2(w[7]))));
  m = hmax2(m, m >> 16);
  s8 = fp4_scale_byte(m);
  const float decoded = __half2float(__half(__nv_cvt_fp8_to_halfraw(s8, __NV_E4M3)));
  const float inv = decoded > 0.0f ? __frcp_rn(decoded) : 0.0f;  // the correctly rounded reciprocal, as 1.0f / decoded
  const ptx::f32x2 inv2 = ptx::pack2(inv, inv);
  uint32_t out[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float q[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t u = w[4 * h + i];
      ptx::unpack2(ptx::mul2(ptx::pack2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u)), inv2), q[2 * i], q[2 * i + 1]);
    }
    out[h] = e2m1_word<FEED>(q);
  }
  codes = make_uint2(out[0], out[1]);
}

}  // namespace
}  // namespace sfq

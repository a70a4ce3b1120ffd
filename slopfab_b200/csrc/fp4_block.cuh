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

// s8 = e4m3_rn_sat(amax / 6), inv = 1 / decode(s8) (0 for an all-zero block), code = e2m1_rn_sat(x * inv)
// (quantize_act_kernel, src/cuda/nvfp4_gemm.cu:107-158).
template <bool FEED>
__device__ __forceinline__ void quantize_block16(const uint4 r0, const uint4 r1, uint2& codes, uint8_t& s8) {
  const uint32_t w[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};  // element 2i in the low half of word i
  uint32_t m = hmax2(hmax2(hmax2(habs2(w[0]), habs2(w[1])), hmax2(habs2(w[2]), habs2(w[3]))),
                     hmax2(hmax2(habs2(w[4]), habs2(w[5])), hmax2(habs2(w[6]), habs2(w[7]))));
  m = hmax2(m, m >> 16);
  const float amax = __uint_as_float(m << 16);
  s8 = uint8_t(__nv_cvt_float_to_fp8(amax * (1.0f / 6.0f), __NV_SATFINITE, __NV_E4M3));
  const float decoded = __half2float(__half(__nv_cvt_fp8_to_halfraw(s8, __NV_E4M3)));
  const float inv = decoded > 0.0f ? __frcp_rn(decoded) : 0.0f;  // the correctly rounded reciprocal, as 1.0f / decoded
  const ptx::f32x2 inv2 = ptx::pack2(inv, inv);
  uint32_t out[2] = {0, 0};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float even, odd;
    ptx::unpack2(ptx::mul2(ptx::pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xFFFF0000u)), inv2), even, odd);
    // The conversion puts its first component in the low nibble. The reference layout wants the even element there; the
    // GEMM feed wants it in the high nibble, like the weight files.
    const __nv_fp4x2_storage_t b = FEED ? __nv_cvt_float2_to_fp4x2(make_float2(odd, even), __NV_E2M1, cudaRoundNearest)
                                        : __nv_cvt_float2_to_fp4x2(make_float2(even, odd), __NV_E2M1, cudaRoundNearest);
    out[i >> 2] |= uint32_t(b) << (8 * (i & 3));
  }
  codes = make_uint2(out[0], out[1]);
}

}  // namespace
}  // namespace sfq

// Fused activation front end of the quantized Linear, one pass over HBM:
//
//   [RMSNorm | RMSNorm + adaLN modulate]  ->  [ConvRot-256 -> per-token int8]  |  [per-16-block fp4]
//
// Replaces, with identical bits, the separate launches of the reference:
// rmsnorm_modulate_bf16_kernel (src/cuda/nn_kernels.cu:153-198), convrot_kernel
// (src/cuda/linear_weights.cu:422-471), quantize_bf16 (src/cuda/w4a8.cu:193-216)
// and quantize_act_kernel (src/cuda/nvfp4_gemm.cu:107-158). The activation is read
// once (2 bytes/element, 128-bit loads) and only the quantized form is written.
//
// Work split of the int8 form: one CTA per token row, one thread per 16 consecutive
// elements (16 threads = one 256-wide rotation group, always inside one
// warp); the norm without a rotation behind it has a kernel of its own. The rotation runs two radix-4 stages in registers, transposes the group
// through a padded, conflict-free shared-memory tile, and runs the other two.
//
// Bit-exactness notes. The sum of squares is accumulated in the order of the
// reference's 256-thread block kernel (thread v owns packs v, v+256, ... with a
// fused multiply-add chain, then the shfl_down tree); 1/sqrt is the reference's
// integer Newton iteration; the butterfly adds associate left to right; bf16
// roundings sit where the reference stores bf16 between its kernels.
#include "kernels.cuh"
#include "runtime.h"

#include <cuda_fp4.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "codec.cuh"
#include "fp4_block.cuh"
#include "ptx.cuh"

namespace sfq {
namespace {

enum Mode { kModeInt8 = 0, kModeRotOnly = 1 };
enum NormMode { kNormOnly = 0, kNormFp4Ref = 1, kNormFp4Feed = 2 };

struct FusedArgs {
  const __nv_bfloat16* x;
  const __nv_bfloat16* norm_w;
  const float* mod_scale;
  const float* mod_shift;
  const int32_t* mod_index;
  float eps;
  int rows, dim;
  int apply_convrot;
  int8_t* q;
  float* row_scale;
  uint8_t* packed;
  uint8_t* scales;
  __nv_bfloat16* bf16_out;  // normed activation (optional) or the rotated one (rot-only mode)
};

// ---- integer-exact norm reciprocal (include/slopfab/cuda/deterministic_math.cuh:26-197) ----
// RNE(v / 2^S) of a product whose result fits 32 bits: half minus one, plus one more when the kept part is odd.
template <int S> __device__ __forceinline__ uint32_t shift_rne32(uint64_t v) {
  return uint32_t((v + ((uint64_t(1) << (S - 1)) - 1) + (uint32_t(v >> S) & 1u)) >> S);
}
// 1/sqrt(v) for a positive normal v: Newton in unsigned Q30 with round-half-even shifts, six
// steps from a seed chosen by the exponent's parity, then rounded to 24 bits. Every operand fits 32 bits (checked on the
// host for all 2^24 significand / parity pairs), so a step is three 32 x 32 -> 64 multiplications: the steps are a serial
// chain that the threads of a row wait for.
__device__ __forceinline__ float rsqrt_q30(float value) {
  const uint32_t mag = __float_as_uint(value) & 0x7FFFFFFFu;
  if (mag == 0u) return __uint_as_float(0x7F800000u);
  if ((__float_as_uint(value) & 0x80000000u) || mag > 0x7F800000u) return __uint_as_float(0x7FC00000u);
  if (mag == 0x7F800000u) return 0.0f;
  uint32_t sig = mag & 0x007FFFFFu;
  int expo;
  if (mag < 0x00800000u) {
    const int t = 31 - __clz(sig);
    expo = t - 149;
    sig <<= unsigned(23 - t);
  } else {
    expo = int(mag >> 23) - 127;
    sig |= 0x00800000u;
  }
  const int odd = expo & 1;
  const uint32_t m = sig << (7 + odd);
  const int out_scale = -(expo - odd) / 2;
  uint32_t y = odd ? 637534208u : 872415232u;
#pragma unroll
  for (int it = 0; it < 6; ++it) {
    const uint32_t y2 = shift_rne32<30>(uint64_t(y) * y);
    const uint32_t my2 = shift_rne32<30>(uint64_t(m) * y2);
    y = shift_rne32<31>(uint64_t(y) * (3u * (1u << 30) - my2));
  }
  int t = 31 - __clz(y);  // 28 .. 30
  const uint32_t drop = uint32_t(t - 23), half = 1u << (drop - 1), rem = y & ((1u << drop) - 1);
  uint32_t r = y >> drop;
  r += rem > half || (rem == half && (r & 1u)) ? 1u : 0u;
  if (r == (1u << 24)) {
    r >>= 1;
    ++t;
  }
  return __uint_as_float((uint32_t(t - 30 + out_scale + 127) << 23) | (r & 0x007FFFFFu));
}
// rsqrt(RNE(sum / dim) + eps); IEEE division and addition are the reference's integer forms.
__device__ float norm_rsqrt(float sum, int dim, float eps) {
  const float mean = sum == 0.0f ? 0.0f : __fdiv_rn(sum, float(dim));
  return rsqrt_q30(__fadd_rn(mean, eps));
}

// One radix-4 stage of the regular Hadamard on (a,b,c,d) -> rows of h4, each a left-to-right
// sum as in convrot_kernel (src/cuda/linear_weights.cu:458-461). a-b is exactly -(b-a), so the
// four outputs cost ten additions instead of twelve.
__device__ __forceinline__ void h4(float& a, float& b, float& c, float& d) {
  const float s = __fadd_rn(a, b);
  const float u = __fsub_rn(a, b);
  const float r0 = __fsub_rn(__fadd_rn(s, c), d);
  const float r1 = __fadd_rn(__fsub_rn(s, c), d);
  const float r2 = __fadd_rn(__fadd_rn(u, c), d);
  const float r3 = __fadd_rn(__fadd_rn(-u, c), d);
  a = r0, b = r1, c = r2, d = r3;
}
// Two stages (strides 1 and 4) over 16 values held by one thread.
__device__ __forceinline__ void two_stages(float (&v)[16]) {
#pragma unroll
  for (int b = 0; b < 4; ++b) h4(v[4 * b], v[4 * b + 1], v[4 * b + 2], v[4 * b + 3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) h4(v[i], v[i + 4], v[i + 8], v[i + 12]);
}

__device__ __forceinline__ float round_bf16(float f) { return __bfloat162float(__float2bfloat16(f)); }

// One token row. `r0`, `r1` are this thread's 16 bf16 elements, already loaded (zero for an inactive thread).
// A thread may return early only where no block-wide barrier follows in this function.
template <int MODE>
__device__ __forceinline__ void process_row(const FusedArgs& a, const int row, uint4 r0, uint4 r1, uint8_t* smem) {
  // [tile: 17 floats per thread][partials: 256 + 8 + 8 floats][raw row: dim bf16 when the norm is on]
  float* tile = reinterpret_cast<float*>(smem);
  float* partial = tile + size_t(blockDim.x) * 17;
  float* warp_tot = partial + 256;
  float* bcast = warp_tot + 8;
  uint4* raw = reinterpret_cast<uint4*>(bcast + 8);

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int chunks = a.dim >> 4;
  const bool active = tid < chunks;

  float v[16];
  {
    const __nv_bfloat162* h0 = reinterpret_cast<const __nv_bfloat162*>(&r0);
    const __nv_bfloat162* h1 = reinterpret_cast<const __nv_bfloat162*>(&r1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f0 = __bfloat1622float2(h0[i]), f1 = __bfloat1622float2(h1[i]);
      v[2 * i] = f0.x, v[2 * i + 1] = f0.y, v[8 + 2 * i] = f1.x, v[8 + 2 * i + 1] = f1.y;
    }
    if (a.norm_w != nullptr && active) {
      raw[tid * 2] = r0;
      raw[tid * 2 + 1] = r1;
    }
  }

  // ---------------------------------------------------------------- RMSNorm [+ modulate]
  if (a.norm_w != nullptr) {
    __syncthreads();
    const int packs = a.dim >> 3;
    for (int vt = tid; vt < 256; vt += blockDim.x) {  // virtual thread vt of the 256-thread block kernel
      float s = 0.0f;
      for (int p = vt; p < packs; p += 256) {
        const uint4 pk = raw[p];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&pk);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 f = __bfloat1622float2(h[i]);
          s = __fmaf_rn(f.x, f.x, s);
          s = __fmaf_rn(f.y, f.y, s);
        }
      }
      partial[vt] = s;
    }
    __syncthreads();
    if (tid < 32) {
      for (int w = 0; w < 8; ++w) {  // shfl_down tree of each virtual warp
        float s = partial[w * 32 + lane];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xFFFFFFFFu, s, off));
        if (lane == 0) warp_tot[w] = s;
      }
      __syncwarp();
      float s = lane < 8 ? warp_tot[lane] : 0.0f;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xFFFFFFFFu, s, off));
      if (lane == 0) bcast[0] = norm_rsqrt(s, a.dim, a.eps);
    }
    __syncthreads();
    const float inv = bcast[0];
    if (active) {
      const uint4* wp = reinterpret_cast<const uint4*>(a.norm_w) + tid * 2;
      const uint4 w0 = wp[0], w1 = wp[1];
      const __nv_bfloat162* wh0 = reinterpret_cast<const __nv_bfloat162*>(&w0);
      const __nv_bfloat162* wh1 = reinterpret_cast<const __nv_bfloat162*>(&w1);
      float w[16];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f0 = __bfloat1622float2(wh0[i]), f1 = __bfloat1622float2(wh1[i]);
        w[2 * i] = f0.x, w[2 * i + 1] = f0.y, w[8 + 2 * i] = f1.x, w[8 + 2 * i + 1] = f1.y;
      }
      if (a.mod_scale != nullptr) {
        const size_t mod = size_t(a.mod_index[row]) * a.dim + size_t(tid) * 16;
        const float4* sc = reinterpret_cast<const float4*>(a.mod_scale + mod);
        const float4* sh = reinterpret_cast<const float4*>(a.mod_shift + mod);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 s4 = sc[j], h4v = sh[j];
          const float ss[4] = {s4.x, s4.y, s4.z, s4.w}, hh[4] = {h4v.x, h4v.y, h4v.z, h4v.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float n = __fmul_rn(__fmul_rn(v[4 * j + i], inv), w[4 * j + i]);
            v[4 * j + i] = round_bf16(__fmaf_rn(n, __fadd_rn(1.0f, ss[i]), hh[i]));
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = round_bf16(__fmul_rn(__fmul_rn(v[i], inv), w[i]));
      }
    }
    if (a.bf16_out != nullptr && MODE != kModeRotOnly && active) {
      uint4 o[2];
      __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
      for (int i = 0; i < 8; ++i) op[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      uint4* dst = reinterpret_cast<uint4*>(a.bf16_out + size_t(row) * a.dim) + tid * 2;
      dst[0] = o[0];
      dst[1] = o[1];
    }
  }
  {
    // ------------------------------------------------------------ ConvRot-256
    if (a.apply_convrot) {
      // Element i = 16*T + e of the group sits at word 17*T + e of the group's tile: a thread's own 16
      // words are consecutive, and the 16 threads' words for a fixed e fall in 16 distinct banks.
      float* grp = tile + (tid >> 4) * 272;
      const int T = tid & 15;
      two_stages(v);  // strides 1 and 4
#pragma unroll
      for (int e = 0; e < 16; ++e) grp[17 * T + e] = v[e];
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 16; ++t) v[t] = grp[17 * t + T];  // now v[t] = element 16*t + T
      two_stages(v);  // strides 16 and 64
      __syncwarp();
#pragma unroll
      for (int t = 0; t < 16; ++t) grp[17 * t + T] = round_bf16(v[t] * 0.0625f);  // 1/16, then the bf16 store
      __syncwarp();
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] = grp[17 * T + e];
    }
    if constexpr (MODE == kModeRotOnly) {
      if (active) {
        uint4 o[2];
        __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(o);
#pragma unroll
        for (int i = 0; i < 8; ++i) op[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        uint4* dst = reinterpret_cast<uint4*>(a.bf16_out + size_t(row) * a.dim) + tid * 2;
        dst[0] = o[0];
        dst[1] = o[1];
      }
      return;
    }
    // ------------------------------------------------------------ per-token int8 (src/cuda/w4a8.cu:193-216)
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    __syncthreads();  // `partial` may still be read by slow warps of the norm phase
    if (lane == 0) partial[tid >> 5] = amax;
    __syncthreads();
    if (tid < 32) {
      float m = tid < int(blockDim.x >> 5) ? partial[tid] : 0.0f;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
      if (tid == 0) {
        const float scale = fmaxf(__fdiv_rn(m, 127.0f), 1e-30f);
        bcast[1] = scale;
        a.row_scale[row] = scale;
      }
    }
    __syncthreads();
    const float divisor = round_bf16(bcast[1]);
    // x / divisor, correctly rounded, without a division per element: with r = RN(1/d) exactly rounded,
    // q0 = RN(x r), e = x - d q0 (exact in one fused multiply-add) and q = RN(q0 + e r) is the IEEE quotient.
    const float rcp = __frcp_rn(divisor);
    if (active) {
      uint32_t o[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        int q[4];
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          const float x0 = v[4 * w + j], x1 = v[4 * w + j + 1];
          const float a0 = __fmul_rn(x0, rcp), a1 = __fmul_rn(x1, rcp);
          const float q0 = __fmaf_rn(__fmaf_rn(-a0, divisor, x0), rcp, a0);
          const float q1 = __fmaf_rn(__fmaf_rn(-a1, divisor, x1), rcp, a1);
          const float2 f = __bfloat1622float2(__floats2bfloat162_rn(q0, q1));  // the quotient is rounded to bf16 first
          q[j] = __float2int_rn(f.x);
          q[j + 1] = __float2int_rn(f.y);
        }
        // saturating pack to int8 = clamp to [-128, 127]
        uint32_t hi, all;
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(q[3]), "r"(q[2]), "r"(0));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(all) : "r"(q[1]), "r"(q[0]), "r"(hi));
        o[w] = all;
      }
      reinterpret_cast<uint4*>(a.q + size_t(row) * a.dim)[tid] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// The kernel: a CTA walks rows blockIdx.x, blockIdx.x + gridDim.x, ... and loads the NEXT row's 32 bytes per
// thread before working on the current one, so every resident warp always has a load in flight (one row per
// CTA without prefetch keeps too few bytes in flight to cover HBM latency).
// BESIDE: the kernel in front neither writes x nor reads the output: wait for it at the end instead of at the start (see kernels.cuh).
template <int MODE, bool BESIDE>
__global__ void __launch_bounds__(1024, 1) fused_act_kernel(const FusedArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  ptx::grid_dependency_release();
  if constexpr (!BESIDE) ptx::grid_dependency_wait();
  const int chunks = a.dim >> 4;
  const bool active = int(threadIdx.x) < chunks;
  auto load = [&](int row, uint4& r0, uint4& r1) {
    r0 = make_uint4(0, 0, 0, 0);
    r1 = r0;
    if (active && row < a.rows) {
      const uint4* src = reinterpret_cast<const uint4*>(a.x + size_t(row) * a.dim) + threadIdx.x * 2;
      r0 = src[0];
      r1 = src[1];
    }
  };
  uint4 r0, r1, n0, n1;
  int row = blockIdx.x;
  load(row, r0, r1);
  for (; row < a.rows; row += gridDim.x) {
    load(row + gridDim.x, n0, n1);
    process_row<MODE>(a, row, r0, r1, smem);
    __syncthreads();  // shared memory is reused by the next row
    r0 = n0;
    r1 = n1;
  }
  if constexpr (BESIDE) ptx::grid_dependency_wait();
}

// ---- RMSNorm [+ modulate], alone or in front of the per-16-block fp4 quantizer ---------------------------------------
// In the reference's 256-thread block thread v accumulates the squares of the 8-element packs v, v + 256, ... in that order.
// Here thread t of 128 owns packs t, t + 128, ..., i.e. the virtual threads t and t + 128, and keeps them in registers: the
// row never goes through shared memory, and a 16-element fp4 block is the packs of two neighbouring threads (one shuffle for
// its maximum). Bound by instruction issue (3600 warp instructions per 5120-wide row) and by the row's serial part - tree,
// integer reciprocal, barrier -, not by HBM (2.56 bytes per element). Hence 128 threads, not 256 (the reciprocal is computed
// by every warp, and 640 packs at dim = 5120 divide evenly), and two rows per CTA: their loads are in flight together, their
// trees run side by side, their reciprocals are computed in different lanes behind ONE barrier, and the modulation tables
// (8 bytes per element, from L1 / L2) are read once for rows of the same index. A CTA leaves after its rows; the next one's
// loads run under the arithmetic of the others on the SM. Measured with modulation, 5120 wide, fp4 out: 75600 rows 375 us
// (2.64 TB/s), 4747 rows 30 us; the one-row kernel with the row in shared memory took 1018 and 58 us. Not faster: 256 threads
// (555 us), CTAs that stay with the next rows prefetched and the tables in shared memory (469 us, fewer warps per SM), the
// reciprocal in warp 0 alone behind a second barrier (407 us).
// FEW rows leave nothing else on the SM to hide a CTA's latencies, and 128 threads meet the weight and the tables of a wide row in up
// to 16 dependent steps. There a CTA has 256 threads and one row, and everything the row needs is on its way before the tree. As
// long as all CTAs are resident at once: two per SM up to 8192 wide (four packs per thread), one beyond. Modulated, fp4 out, inputs
// from HBM, FEW against 128 threads: 64 rows of 3072 8.2 / 12.3 us, 5120 10.2 / 14.3, 16384 14.3 / 22.5; 296 rows of 5120 10.2 / 14.3, of
// 13824 22.5 / 20.5; 444 of 5120 14.3 / 14.3; 888 of 5120 18.4 / 14.3.
template <bool FEW> constexpr int kNormThreads = FEW ? 256 : 128;
// Rows a CTA takes at a time: two while a thread's share of a row is at most six packs (dim <= 6144), one beyond that.
template <int MAXP, bool FEW> constexpr int kNormRows = MAXP <= 6 && !FEW ? 2 : 1;

// 1 / decode(s8) correctly rounded for the positive e4m3 scales, 0 for scale 0 (and for the NaN code, which is never produced).
struct E4m3Reciprocals {
  float v[128];
  constexpr E4m3Reciprocals() : v() {
    for (int i = 1; i < 127; ++i) {
      const int e = i >> 3, m = i & 7;
      float d = e == 0 ? float(m) : float(8 + m);  // decode = d * 2^(max(e, 1) - 10), exact at every step
      for (int k = (e == 0 ? 1 : e); k < 10; ++k) d *= 0.5f;
      for (int k = 10; k < e; ++k) d *= 2.0f;
      v[i] = 1.0f / d;
    }
  }
};
__device__ const E4m3Reciprocals kE4m3Reciprocal;

template <int MODE, int MAXP, bool FEW>
__global__ void __launch_bounds__(kNormThreads<FEW>, FEW ? (MAXP <= 4 ? 2 : 1) : (MAXP <= 2 ? 8 : 4)) norm_rows_kernel(const FusedArgs a, int total_rows) {
  constexpr int T = kNormThreads<FEW>, R = kNormRows<MAXP, FEW>;
  constexpr int V = 256 / T;  // virtual threads per thread
  ptx::grid_dependency_release();
  ptx::grid_dependency_wait();
  __shared__ float warp_tot[R][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int packs = a.dim >> 3, chunks = a.dim >> 4;
  const int row0 = blockIdx.x * R;
  if (MODE == kNormFp4Feed && row0 >= a.rows) {  // padding rows of the last 128-row scale tile: zero scales
    for (int r = 0; r < R && row0 + r < total_rows; ++r)
      for (int c = tid; c < chunks; c += T) a.scales[nvfp4_scale_offset(row0 + r, c, chunks)] = 0;
    return;
  }
  uint4 raw[R][MAXP];
#pragma unroll
  for (int j = 0; j < MAXP; ++j)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int p = tid + j * T;
      raw[r][j] = make_uint4(0, 0, 0, 0);
      if (p < packs && row0 + r < a.rows) raw[r][j] = reinterpret_cast<const uint4*>(a.x + size_t(row0 + r) * a.dim)[p];
    }
  int index[R] = {};
  if (a.mod_scale != nullptr) {
#pragma unroll
    for (int r = 0; r < R; ++r) index[r] = a.mod_index[min(row0 + r, a.rows - 1)];
  }
  // the weight and the tables of pack j; FEW fetches all of them here, ahead of the row's tree
  constexpr int A = FEW ? MAXP : 1;
  uint4 wr[A];
  ptx::f32x2 sc[A][4], sh[A][4];
  auto load_weight = [&](int j) { return tid + j * T < packs ? reinterpret_cast<const uint4*>(a.norm_w)[tid + j * T] : make_uint4(0, 0, 0, 0); };
  auto load_tables = [&](int j, int row_index, ptx::f32x2 (&s)[4], ptx::f32x2 (&h)[4]) {
    const size_t at = size_t(row_index) * a.dim + size_t(tid + j * T < packs ? tid + j * T : 0) * 8;
    const float4* sp = reinterpret_cast<const float4*>(a.mod_scale + at);
    const float4* hp = reinterpret_cast<const float4*>(a.mod_shift + at);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float4 s4 = sp[i], h4v = hp[i];
      s[2 * i] = ptx::pack2(s4.x, s4.y), s[2 * i + 1] = ptx::pack2(s4.z, s4.w);
      h[2 * i] = ptx::pack2(h4v.x, h4v.y), h[2 * i + 1] = ptx::pack2(h4v.z, h4v.w);
    }
  };
  if constexpr (FEW) {
#pragma unroll
    for (int j = 0; j < MAXP; ++j) {
      wr[j] = load_weight(j);
      if (a.mod_scale != nullptr) load_tables(j, index[0], sc[j], sh[j]);
    }
  }
  // sum of squares: the chains of virtual threads t and, of 128, t + 128 (odd packs), the shfl_down tree of their virtual
  // warps, then the tree over the eight warps' totals
  float sum[R][V];
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int k = 0; k < V; ++k) sum[r][k] = 0.0f;
#pragma unroll
    for (int j = 0; j < MAXP; ++j) {  // absent packs are zeros: fma(0, 0, s) = s
      const uint32_t u[4] = {raw[r][j].x, raw[r][j].y, raw[r][j].z, raw[r][j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float lo = __uint_as_float(u[i] << 16), hi = __uint_as_float(u[i] & 0xFFFF0000u);
        sum[r][j % V] = __fmaf_rn(lo, lo, sum[r][j % V]);
        sum[r][j % V] = __fmaf_rn(hi, hi, sum[r][j % V]);
      }
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < V; ++k) sum[r][k] = __fadd_rn(sum[r][k], __shfl_down_sync(0xFFFFFFFFu, sum[r][k], off));
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int k = 0; k < V; ++k) warp_tot[r][warp + k * (T / 32)] = sum[r][k];
  }
  __syncthreads();
  // Every warp folds the totals itself: lanes 8 r .. 8 r + 7 hold row r (the reference's steps 16 and 8 add zeros).
  float tot = warp_tot[(lane >> 3) % R][lane & 7];
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) tot = __fadd_rn(tot, __shfl_down_sync(0xFFFFFFFFu, tot, off));
  const float inv_mine = norm_rsqrt(tot, a.dim, a.eps);
  float inv[R];
#pragma unroll
  for (int r = 0; r < R; ++r) inv[r] = __shfl_sync(0xFFFFFFFFu, inv_mine, 8 * r);

#pragma unroll
  for (int j = 0; j < MAXP; ++j) {
    const int p = tid + j * T;
    const bool active = p < packs;
    if (!__any_sync(0xFFFFFFFFu, active)) break;
    constexpr bool kFetched = FEW;
    const int at = kFetched ? j : 0;
    if constexpr (!kFetched) wr[0] = load_weight(j);
    const uint32_t wu[4] = {wr[at].x, wr[at].y, wr[at].z, wr[at].w};
    const ptx::f32x2 one = ptx::pack2(1.0f, 1.0f);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = row0 + r;
      if (a.mod_scale != nullptr && (r == 0 || index[r] != index[r - 1])) {
        if constexpr (!kFetched) load_tables(j, index[r], sc[0], sh[0]);
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[at][i] = ptx::add2(one, sc[at][i]);
      }
      const uint32_t u[4] = {raw[r][j].x, raw[r][j].y, raw[r][j].z, raw[r][j].w};
      const ptx::f32x2 inv2 = ptx::pack2(inv[r], inv[r]);
      uint32_t n[4];  // the normed row rounded to bf16, as the reference stores it
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ptx::f32x2 x2 = ptx::pack2(__uint_as_float(u[i] << 16), __uint_as_float(u[i] & 0xFFFF0000u));
        ptx::f32x2 v = ptx::mul2(ptx::mul2(x2, inv2), ptx::pack2(__uint_as_float(wu[i] << 16), __uint_as_float(wu[i] & 0xFFFF0000u)));
        if (a.mod_scale != nullptr) v = ptx::fma2(v, sc[at][i], sh[at][i]);
        float lo, hi;
        ptx::unpack2(v, lo, hi);
        const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
        n[i] = *reinterpret_cast<const uint32_t*>(&b);
      }
      const bool write = active && row < a.rows;
      if (a.bf16_out != nullptr && write) reinterpret_cast<uint4*>(a.bf16_out + size_t(row) * a.dim)[p] = make_uint4(n[0], n[1], n[2], n[3]);
      if constexpr (MODE != kNormOnly) {
        // per-16 fp4 (src/cuda/nvfp4_gemm.cu:107-158): this thread's eight elements and its neighbour's share a scale
        uint32_t m = hmax2(hmax2(habs2(n[0]), habs2(n[1])), hmax2(habs2(n[2]), habs2(n[3])));
        m = hmax2(m, __shfl_xor_sync(0xFFFFFFFFu, m, 1));
        m = hmax2(hmax2(m, m >> 16), 0u);  // the reference's maximum starts at 0, which a block of NaNs alone leaves: scale 0
        uint32_t s8 = row < a.rows ? uint32_t(fp4_scale_byte(m)) : 0u;
        const float rcp = __ldg(kE4m3Reciprocal.v + s8);
        const ptx::f32x2 rcp2 = ptx::pack2(rcp, rcp);
        float q[8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          ptx::unpack2(ptx::mul2(ptx::pack2(__uint_as_float(n[i] << 16), __uint_as_float(n[i] & 0xFFFF0000u)), rcp2), q[2 * i], q[2 * i + 1]);
        if (write) reinterpret_cast<uint32_t*>(a.packed + size_t(row) * (a.dim >> 1))[p] = e2m1_word<MODE == kNormFp4Feed>(q);
        if constexpr (MODE == kNormFp4Ref) {
          if (write && (lane & 1) == 0) a.scales[size_t(row) * chunks + (p >> 1)] = uint8_t(s8);
        } else {
          // four neighbouring blocks are the four bytes of one word of the tiled layout (dim % 64 == 0: whole words);
          // the second row of the last pair may be a padding row, whose scales are zero
          s8 <<= 8 * ((lane >> 1) & 3);
          s8 |= __shfl_xor_sync(0xFFFFFFFFu, s8, 2);
          s8 |= __shfl_xor_sync(0xFFFFFFFFu, s8, 4);
          if (active && (lane & 7) == 0 && row < total_rows) {
            // T / 2 blocks further on are T / 8 tiles of 512 bytes
            uint8_t* dst = a.scales + nvfp4_scale_offset(row, tid >> 1, chunks) + size_t(j) * (T / 8 * 512);
            if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0)
              *reinterpret_cast<uint32_t*>(dst) = s8;
            else  // an array that starts off a word boundary
              for (int i = 0; i < 4; ++i) dst[i] = uint8_t(s8 >> (8 * i));
          }
        }
      }
    }
  }
}

// Generic rotation for the other power-of-four groups (4, 16, 64): not on the hot path (the INT8
// weight-only format of the text encoder); one block of 64 threads per 256 columns.
__global__ void __launch_bounds__(64)
convrot_small_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, int dim, int stages,
                     float norm) {
  __shared__ float v[256 + 64];
  const int row = blockIdx.x, c0 = blockIdx.y * 256, t = threadIdx.x;
  const int n = min(256, dim - c0);
  const size_t base = size_t(row) * dim + c0;
  for (int i = t; i < n; i += 64) v[i + (i >> 2)] = __bfloat162float(in[base + i]);
  __syncthreads();
  int stride = 1;
  for (int s = 0; s < stages; ++s) {
    const int i = (t / stride) * 4 * stride + (t % stride);
    const bool live = i + 3 * stride < n;
    const int j0 = i, j1 = i + stride, j2 = i + 2 * stride, j3 = i + 3 * stride;
    float a = 0, b = 0, c = 0, d = 0;
    if (live) a = v[j0 + (j0 >> 2)], b = v[j1 + (j1 >> 2)], c = v[j2 + (j2 >> 2)], d = v[j3 + (j3 >> 2)];
    __syncthreads();
    if (live) {
      h4(a, b, c, d);
      v[j0 + (j0 >> 2)] = a, v[j1 + (j1 >> 2)] = b, v[j2 + (j2 >> 2)] = c, v[j3 + (j3 >> 2)] = d;
    }
    __syncthreads();
    stride *= 4;
  }
  for (int i = t; i < n; i += 64) out[base + i] = __float2bfloat16(v[i + (i >> 2)] * norm);
}

inline void check_launch(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

void check_row_args(const FusedArgs& a, const char* what) {
  if (a.dim % 16 != 0 || a.dim > 16384)
    throw std::invalid_argument(std::string(what) + ": dim must be a multiple of 16 and at most 16384");
  if (reinterpret_cast<uintptr_t>(a.x) % 16 != 0)
    throw std::invalid_argument(std::string(what) + ": activation pointer must be 16-byte aligned");
  if (a.norm_w != nullptr && a.mod_scale != nullptr && (a.mod_shift == nullptr || a.mod_index == nullptr))
    throw std::invalid_argument(std::string(what) + ": modulation needs scale, shift and the row index");
}

template <int MODE, bool BESIDE = false> void launch_fused(const FusedArgs& a, cudaStream_t stream, const char* what) {
  check_row_args(a, what);
  const int threads = ((a.dim / 16 + 31) / 32) * 32;
  const size_t smem = size_t(threads) * 17 * 4 + (256 + 16) * 4 + (a.norm_w ? size_t(a.dim) * 2 : 0);
  reserve_dynamic_smem(reinterpret_cast<const void*>(&fused_act_kernel<MODE, BESIDE>), smem, what);
  // As many CTAs as stay resident at once; each walks rows with a stride of the grid size.
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_act_kernel<MODE, BESIDE>, threads, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  const int grid = std::min(a.rows, per_sm * device_sm_count());
  check_launch(launch_overlapped(size_t(a.rows) * a.dim * 4, fused_act_kernel<MODE, BESIDE>, dim3(grid), dim3(threads), smem, stream, a), what);
}

template <int MODE, int MAXP, bool FEW> cudaError_t launch_norm_as(const FusedArgs& a, int total_rows, cudaStream_t stream) {
  constexpr int R = kNormRows<MAXP, FEW>;
  return launch_overlapped(size_t(a.rows) * a.dim * 3, norm_rows_kernel<MODE, MAXP, FEW>, dim3((total_rows + R - 1) / R), dim3(kNormThreads<FEW>), 0,
                           stream, a, total_rows);
}

// A thread's packs per row decide the registers of the kernel.
template <int MODE> void launch_norm(const FusedArgs& a, int total_rows, cudaStream_t stream, const char* what) {
  check_row_args(a, what);
  const auto packs = [&](int threads) { return (a.dim / 8 + threads - 1) / threads; };
  const bool few = a.rows <= device_sm_count() * (packs(kNormThreads<true>) <= 4 ? 2 : 1);
  const int per_thread = packs(few ? kNormThreads<true> : kNormThreads<false>);
  cudaError_t e = cudaSuccess;
  if (few)
    e = per_thread <= 1   ? launch_norm_as<MODE, 1, true>(a, total_rows, stream)
        : per_thread <= 3 ? launch_norm_as<MODE, 3, true>(a, total_rows, stream)
        : per_thread <= 4 ? launch_norm_as<MODE, 4, true>(a, total_rows, stream)
                          : launch_norm_as<MODE, 8, true>(a, total_rows, stream);
  else
    e = per_thread <= 2   ? launch_norm_as<MODE, 2, false>(a, total_rows, stream)
        : per_thread <= 5 ? launch_norm_as<MODE, 5, false>(a, total_rows, stream)
        : per_thread <= 6 ? launch_norm_as<MODE, 6, false>(a, total_rows, stream)
                          : launch_norm_as<MODE, 16, false>(a, total_rows, stream);
  check_launch(e, what);
}

FusedArgs base_args(const __nv_bfloat16* x, const NormArgs& n, int rows, int dim) {
  FusedArgs a{};
  a.x = x;
  a.norm_w = n.weight;
  a.mod_scale = n.weight ? n.scale : nullptr;
  a.mod_shift = n.weight ? n.shift : nullptr;
  a.mod_index = n.weight ? n.index : nullptr;
  a.eps = n.eps;
  a.rows = rows;
  a.dim = dim;
  return a;
}

}  // namespace

void rmsnorm(const __nv_bfloat16* x, const NormArgs& norm, __nv_bfloat16* out, int rows, int dim, cudaStream_t stream) {
  if (rows <= 0 || dim <= 0) throw std::invalid_argument("rmsnorm: rows and dim must be positive");
  if (!x || !out || !norm.weight) throw std::invalid_argument("rmsnorm: null buffer");
  FusedArgs a = base_args(x, norm, rows, dim);
  a.bf16_out = out;
  launch_norm<kNormOnly>(a, rows, stream, "rmsnorm");
}

void convrot(const __nv_bfloat16* x, __nv_bfloat16* out, int rows, int dim, int group, cudaStream_t stream, bool beside) {
  if (rows <= 0 || dim <= 0) return;
  if (!x || !out) throw std::invalid_argument("convrot: null buffer");
  int stages = 0, n = 1;
  while (n < group) n *= 4, ++stages;
  if (n != group) throw std::runtime_error("convrot: group size must be a power of four, got " + std::to_string(group));
  if (dim % group != 0) throw std::runtime_error("convrot: dim must be a multiple of the group size");
  if (group == 256 && dim <= 16384) {
    FusedArgs a = base_args(x, NormArgs{}, rows, dim);
    a.apply_convrot = 1;
    a.bf16_out = out;
    if (beside)
      launch_fused<kModeRotOnly, true>(a, stream, "convrot");
    else
      launch_fused<kModeRotOnly>(a, stream, "convrot");
    return;
  }
  if (group > 256) throw std::runtime_error("convrot: groups above 256 are not supported");
  convrot_small_kernel<<<dim3(rows, (dim + 255) / 256), 64, 0, stream>>>(x, out, dim, stages, 1.0f / float(1 << stages));
  check_launch(cudaGetLastError(), "convrot");
}

void quantize_int8_token(const __nv_bfloat16* x, const NormArgs& norm, int8_t* q, float* row_scale,
                         __nv_bfloat16* normed_out, int rows, int dim, bool apply_convrot, cudaStream_t stream, bool overlap) {
  if (rows <= 0 || dim <= 0) throw std::invalid_argument("W4A8 activation shape");
  if (!x || !q || !row_scale) throw std::invalid_argument("quantize_int8_token: null buffer");
  if (apply_convrot && dim % 256 != 0) throw std::invalid_argument("W4A8 activation requires K divisible by 256");
  if (reinterpret_cast<uintptr_t>(q) % 16 != 0) throw std::invalid_argument("quantize_int8_token: output must be 16-byte aligned");
  // The Linear's own case (rotation on, nothing fused in front, K <= 6144) has a two-rows-per-step kernel.
  if (apply_convrot && norm.weight == nullptr && quantize_int8_rot_pairs(x, q, row_scale, rows, dim, stream, overlap)) return;
  FusedArgs a = base_args(x, norm, rows, dim);
  a.q = q;
  a.row_scale = row_scale;
  a.apply_convrot = apply_convrot ? 1 : 0;
  a.bf16_out = norm.weight ? normed_out : nullptr;
  launch_fused<kModeInt8>(a, stream, "quantize_int8_token");
}

size_t nvfp4_act_scale_bytes(int rows, int dim) {
  if (rows <= 0 || dim <= 0) return 0;
  return size_t((rows + 127) / 128) * 128 * size_t(dim / 16);
}

// ---- per-16-block fp4 quantizer without a norm in front (the Linear's own case) --------------------------------------
// The arithmetic of fp4_block.cuh (quantize_act_kernel, src/cuda/nvfp4_gemm.cu:107-158): per 16
// elements s8 = e4m3_rn_sat(amax / 6), inv = 1 / decode(s8) (0 for an all-zero block), code = e2m1_rn_sat(x * inv). A
// block's scale depends on that block alone, so there is nothing to exchange between threads: the activation is walked as
// a flat array of 16-element blocks, two per thread in flight, with no barrier and no shared memory, the maximum on
// bf16x2 words and the products on packed fp32 pairs. FEED: high nibble = even element, scales in the 128x4-tiled layout
// with the rows padded to a multiple of 128 (the pad rows' scales are written as zero).
namespace {
template <bool FEED>
__global__ void __launch_bounds__(256) quantize_nvfp4_flat_kernel(const __nv_bfloat16* x, uint8_t* __restrict__ packed,
                                                                  uint8_t* __restrict__ scales, int rows, int padded_rows, int chunks) {
  ptx::grid_dependency_release();
  ptx::grid_dependency_wait();
  // item g = (row, chunk): advance by the grid's stride without a division per item
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
  int row = int(first / uint32_t(chunks)), c = int(first % uint32_t(chunks));
  const int drow = int(stride / uint32_t(chunks)), dc = int(stride % uint32_t(chunks));
  auto load = [&](int r, int cc, uint4& a, uint4& b) {
    a = make_uint4(0, 0, 0, 0);
    b = a;
    if (r < rows) {
      const uint4* src = reinterpret_cast<const uint4*>(x) + (size_t(r) * chunks + cc) * 2;
      a = src[0];
      b = src[1];
    }
  };
  auto emit = [&](int r, int cc, const uint4& a, const uint4& b) {
    if (r >= padded_rows) return;
    uint2 codes;
    uint8_t s8 = 0;
    if (r < rows) {
      quantize_block16<FEED>(a, b, codes, s8);
      reinterpret_cast<uint2*>(packed)[size_t(r) * chunks + cc] = codes;
    }
    scales[FEED ? nvfp4_scale_offset(r, cc, chunks) : size_t(r) * chunks + cc] = s8;
  };
  while (row < padded_rows) {
    int row2 = row + drow, c2 = c + dc;
    if (c2 >= chunks) c2 -= chunks, ++row2;
    uint4 a0, b0, a1, b1;
    load(row, c, a0, b0);
    load(row2, c2, a1, b1);
    emit(row, c, a0, b0);
    emit(row2, c2, a1, b1);
    row = row2 + drow, c = c2 + dc;
    if (c >= chunks) c -= chunks, ++row;
  }
}

template <bool FEED>
void launch_nvfp4_flat(const __nv_bfloat16* x, uint8_t* packed, uint8_t* scales, int rows, int dim, cudaStream_t stream) {
  const int chunks = dim / 16;
  const int padded = FEED ? (rows + 127) / 128 * 128 : rows;
  const size_t items = size_t(padded) * chunks;
  if (items >= (size_t(1) << 31)) throw std::invalid_argument("quantize_nvfp4_block: too many 16-element blocks for one launch");
  const int ctas = int(std::min<size_t>((items + 511) / 512, size_t(device_sm_count()) * 8));  // two items per thread and trip
  check_launch(launch_overlapped(items * 41, quantize_nvfp4_flat_kernel<FEED>, dim3(ctas), dim3(256), 0, stream, x, packed, scales, rows, padded, chunks),
               "quantize_nvfp4_block");
}
}  // namespace

void quantize_nvfp4_block(const __nv_bfloat16* x, const NormArgs& norm, uint8_t* packed, uint8_t* scales,
                          __nv_bfloat16* normed_out, int rows, int dim, int layout, cudaStream_t stream) {
  if (rows <= 0 || dim <= 0) return;
  if (!x || !packed || !scales) throw std::invalid_argument("quantize_nvfp4_block: null buffer");
  if (dim % 16 != 0)
    throw std::runtime_error("nvfp4: activation dim must be a multiple of 16, got " + std::to_string(dim));
  if (reinterpret_cast<uintptr_t>(packed) % 8 != 0) throw std::invalid_argument("quantize_nvfp4_block: output must be 8-byte aligned");
  if (layout != SFQ_NVFP4_ACT_REFERENCE && layout != SFQ_NVFP4_ACT_GEMM_FEED) throw std::invalid_argument("quantize_nvfp4_block: unknown layout");
  if (layout == SFQ_NVFP4_ACT_GEMM_FEED && dim % 64 != 0)
    throw std::invalid_argument("quantize_nvfp4_block: the tiled scale layout needs dim % 64 == 0");
  if (norm.weight == nullptr) {  // no norm in front: the barrier-free kernel
    if (reinterpret_cast<uintptr_t>(x) % 16 != 0) throw std::invalid_argument("quantize_nvfp4_block: activation pointer must be 16-byte aligned");
    if (layout == SFQ_NVFP4_ACT_REFERENCE)
      launch_nvfp4_flat<false>(x, packed, scales, rows, dim, stream);
    else
      launch_nvfp4_flat<true>(x, packed, scales, rows, dim, stream);
    return;
  }
  FusedArgs a = base_args(x, norm, rows, dim);
  a.packed = packed;
  a.scales = scales;
  a.bf16_out = norm.weight ? normed_out : nullptr;
  if (layout == SFQ_NVFP4_ACT_REFERENCE)
    launch_norm<kNormFp4Ref>(a, rows, stream, "quantize_nvfp4_block");
  else
    launch_norm<kNormFp4Feed>(a, (rows + 127) / 128 * 128, stream, "quantize_nvfp4_block");
}

// ---- head-wise q/k RMSNorm and MM-RoPE, the two steps between the fused projection and attention ----
// launch_head_rmsnorm (src/cuda/nn_kernels.cu:296-305 -> rmsnorm_warp_kernel, :100-136) followed by launch_rope_h3
// (src/cuda/nn_position.cu:15-68,111-123), in place, head_dim 128, on a row pitch so that the q and k thirds of the fused
// projection are processed where they lie. Bit-exact: 16 lanes hold 8 channels each; the sum of squares is the reference's
// per-lane chain and xor butterfly (whose first step adds the zeros of its idle upper lanes); the normalised value is
// rounded to bf16 before the rotation (the reference stores it between its two kernels); the rotation pairs channel j with
// j + 48 over the first 96 channels with the reference's subnormal canonicalisation.
//
// What bounds it: HBM (read and write 256 bytes per head) once the instruction count is down, so a warp takes EIGHT heads of
// one row, four per half warp: four 16-byte loads per lane in flight, the row's cos / sin read once for all of them, and the
// serial part of the norm - the integer Newton reciprocal - run once for the eight heads side by side in different lanes.
// The canonicalisation costs one running minimum: a lane whose channels, table entries, products and results are all normal numbers
// has nothing to canonicalise; one that saw a smaller magnitude (a zero counts) recomputes its eight channels step by step.
// Measured, q and k of 4747 rows x 40 heads: 61 us (3.2 TB/s); one warp per head with the reciprocal in one lane and the
// canonicalisation in every channel: 436 us.
namespace {
constexpr int kHeadsPerWarp = 8;

__device__ __forceinline__ float rope_bf16_value(unsigned short bits) {
  return (bits & 0x7fffu) < 0x0080u ? __uint_as_float(unsigned(bits & 0x8000u) << 16) : __uint_as_float(unsigned(bits) << 16);
}
__device__ __forceinline__ float rope_float_value(float value) {
  const unsigned bits = __float_as_uint(value);
  return (bits & 0x7fffffffu) < 0x00800000u ? __uint_as_float(bits & 0x80000000u) : value;
}
__device__ __forceinline__ unsigned short rope_bf16_result(float value) {
  const unsigned short bits = __bfloat16_as_ushort(__float2bfloat16(value));
  return (bits & 0x7fffu) < 0x0080u ? (unsigned short)(bits & 0x8000u) : bits;
}
__device__ __forceinline__ float rope_fma_product(float a, float b, float base) {
  const float product = __fmul_rn(a, b);
  const unsigned magnitude = __float_as_uint(product) & 0x7fffffffu;
  if (magnitude < 0x00800000u && (__float_as_uint(a) & 0x7fffffffu) != 0u && (__float_as_uint(b) & 0x7fffffffu) != 0u) return base;
  return fmaf(a, b, base);
}
// One channel with every canonicalisation spelled out. `low`: channels 0-47 of the head, `other` is the partner's value.
__device__ __forceinline__ unsigned short rope_channel(bool low, unsigned short own, unsigned short other, float cos_v, float sin_v) {
  const float c = rope_float_value(cos_v), s = rope_float_value(sin_v), x = rope_bf16_value(own), o = rope_bf16_value(other);
  const float base = rope_float_value(__fmul_rn(x, c));
  return rope_bf16_result(low ? __fsub_rn(base, rope_float_value(__fmul_rn(o, s))) : rope_fma_product(o, s, base));
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <bool NORM, bool ROPE>
__global__ void __launch_bounds__(256) head_norm_rope_kernel(__nv_bfloat16* __restrict__ x, int ld, const __nv_bfloat16* w,
                                                             const float* cos_tab, const float* sin_tab,
                                                             int tables_vec, int rows, int heads, float eps) {
  constexpr int kPer = kHeadsPerWarp / 2;  // heads per half warp
  ptx::grid_dependency_release();
  ptx::grid_dependency_wait();
  const int lane = threadIdx.x & 31, l = lane & 15, half = lane >> 4;
  const int groups = (heads + kHeadsPerWarp - 1) / kHeadsPerWarp;
  const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // (row, group of heads)
  if (unit >= (long long)rows * groups) return;
  const int row = int(unit / groups), head0 = int(unit % groups) * kHeadsPerWarp + half;
  __nv_bfloat16* v = x + size_t(row) * ld + size_t(head0) * 128 + l * 8;
  uint32_t h[kPer][4];
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (head0 + 2 * i < heads) raw = *reinterpret_cast<const uint4*>(v + i * 256);
    h[i][0] = raw.x, h[i][1] = raw.y, h[i][2] = raw.z, h[i][3] = raw.w;
  }
  // lanes 0-5 hold channels 8 l .. (the low halves), lanes 6-11 their partners j + 48, lanes 12-15 pass through
  const bool low = l < 6, rotates = l < 12;
  float c[8], s[8];
  if constexpr (ROPE) {
    const size_t at = size_t(row) * 96 + (low ? l : (rotates ? l - 6 : 0)) * 8;
    if (tables_vec) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float4 c4 = reinterpret_cast<const float4*>(cos_tab + at)[i], s4 = reinterpret_cast<const float4*>(sin_tab + at)[i];
        c[4 * i] = c4.x, c[4 * i + 1] = c4.y, c[4 * i + 2] = c4.z, c[4 * i + 3] = c4.w;
        s[4 * i] = s4.x, s[4 * i + 1] = s4.y, s[4 * i + 2] = s4.z, s[4 * i + 3] = s4.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) c[i] = cos_tab[at + i], s[i] = sin_tab[at + i];
    }
  }
  if constexpr (NORM) {
    float sum[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      sum[i] = 0.0f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        sum[i] = fmaf(bf16_lo(h[i][k]), bf16_lo(h[i][k]), sum[i]);
        sum[i] = fmaf(bf16_hi(h[i][k]), bf16_hi(h[i][k]), sum[i]);
      }
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1)
#pragma unroll
      for (int i = 0; i < kPer; ++i) sum[i] = __fadd_rn(sum[i], __shfl_xor_sync(0xFFFFFFFFu, sum[i], off));
    // lane l of a half takes the reciprocal of head l % 4 of that half
    static_assert(kPer == 4, "the selection below");
    const float even = (l & 2) ? sum[2] : sum[0], odd = (l & 2) ? sum[3] : sum[1];
    const float mine = (l & 1) ? odd : even;
    // mean = RNE(sum / 128), the same as the product with the power of two
    const float inv_mine = rsqrt_q30(__fadd_rn(__fmul_rn(mine, 1.0f / 128.0f), eps));
    const uint4 wr = *reinterpret_cast<const uint4*>(w + l * 8);
    const uint32_t wu[4] = {wr.x, wr.y, wr.z, wr.w};
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const float inv = __shfl_sync(0xFFFFFFFFu, inv_mine, (lane & 16) | i);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        h[i][k] = bf16_pair(__fmul_rn(__fmul_rn(bf16_lo(h[i][k]), inv), bf16_lo(wu[k])), __fmul_rn(__fmul_rn(bf16_hi(h[i][k]), inv), bf16_hi(wu[k])));
    }
  }
  if constexpr (ROPE) {
    const int partner = low ? lane + 6 : (rotates ? lane - 6 : lane);
    constexpr float kMinNormal = 1.17549435e-38f;
    float least_entry = kMinNormal;  // a subnormal table entry can give normal products
#pragma unroll
    for (int i = 0; i < 8; ++i) least_entry = fminf(least_entry, fminf(fabsf(c[i]), fabsf(s[i])));
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      uint32_t o[4], r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] = __shfl_sync(0xFFFFFFFFu, h[i][k], partner);
      float least = least_entry;  // of every magnitude that the reference would canonicalise
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float out[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float xv = e ? bf16_hi(h[i][k]) : bf16_lo(h[i][k]), ov = e ? bf16_hi(o[k]) : bf16_lo(o[k]);
          const float base = __fmul_rn(xv, c[2 * k + e]), p = __fmul_rn(ov, s[2 * k + e]);
          out[e] = low ? __fsub_rn(base, p) : fmaf(ov, s[2 * k + e], base);
          least = fminf(fminf(least, fabsf(base)), fabsf(p));
          least = fminf(fminf(least, fabsf(xv)), fminf(fabsf(ov), fabsf(out[e])));
        }
        r[k] = bf16_pair(out[0], out[1]);
      }
      if (rotates && head0 + 2 * i < heads) {  // a head that does not exist is zeros: not a reason for the step-by-step path
        if (least < kMinNormal) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned short a = rope_channel(low, (unsigned short)(h[i][k] & 0xFFFFu), (unsigned short)(o[k] & 0xFFFFu), c[2 * k], s[2 * k]);
            const unsigned short b = rope_channel(low, (unsigned short)(h[i][k] >> 16), (unsigned short)(o[k] >> 16), c[2 * k + 1], s[2 * k + 1]);
            r[k] = unsigned(a) | (unsigned(b) << 16);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) h[i][k] = r[k];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kPer; ++i)
    if (head0 + 2 * i < heads) *reinterpret_cast<uint4*>(v + i * 256) = make_uint4(h[i][0], h[i][1], h[i][2], h[i][3]);
}
}  // namespace

void head_norm_rope(__nv_bfloat16* x, int ld, const __nv_bfloat16* norm_weight, const float* cos_tab, const float* sin_tab, int rows,
                    int heads, int head_dim, float eps, cudaStream_t stream) {
  if (rows <= 0 || heads <= 0) throw std::runtime_error("head_norm_rope: rows and heads must be positive");
  if (head_dim != 128) throw std::runtime_error("head_norm_rope: built for head_dim 128 (96 rotary channels + 32 passed through)");
  if (x == nullptr || (norm_weight == nullptr && cos_tab == nullptr)) throw std::invalid_argument("head_norm_rope: nothing to do");
  if ((cos_tab == nullptr) != (sin_tab == nullptr)) throw std::invalid_argument("head_norm_rope: cos and sin come together");
  if (ld < heads * 128 || ld % 8 != 0 || reinterpret_cast<uintptr_t>(x) % 16 != 0 ||
      (norm_weight != nullptr && reinterpret_cast<uintptr_t>(norm_weight) % 16 != 0))
    throw std::invalid_argument("head_norm_rope: the row pitch must cover heads * 128 and keep 16-byte alignment");
  const long long units = (long long)rows * ((heads + kHeadsPerWarp - 1) / kHeadsPerWarp);
  const int tables_vec = ((reinterpret_cast<uintptr_t>(cos_tab) | reinterpret_cast<uintptr_t>(sin_tab)) & 15) == 0;
  const unsigned grid = unsigned((units + 7) / 8);
  const size_t bytes = size_t(rows) * heads * 512;
  cudaError_t e = cudaSuccess;
  if (norm_weight != nullptr && cos_tab != nullptr)
    e = launch_overlapped(bytes, head_norm_rope_kernel<true, true>, dim3(grid), dim3(256), 0, stream, x, ld, norm_weight, cos_tab, sin_tab, tables_vec, rows, heads, eps);
  else if (norm_weight != nullptr)
    e = launch_overlapped(bytes, head_norm_rope_kernel<true, false>, dim3(grid), dim3(256), 0, stream, x, ld, norm_weight, cos_tab, sin_tab, tables_vec, rows, heads, eps);
  else
    e = launch_overlapped(bytes, head_norm_rope_kernel<false, true>, dim3(grid), dim3(256), 0, stream, x, ld, norm_weight, cos_tab, sin_tab, tables_vec, rows, heads, eps);
  check_launch(e, "head_norm_rope");
}

}  // namespace sfq

// The LoRA side branch in one launch: y = bf16(y + bf16(hidden B^T)), hidden = bf16(x A^T), hidden never leaving the SM.
//
// Bound by memory: x is read once, y read and written once (126 MB at 4096 x 5120 -> 5120, 19 us at the measured copy
// rate), and the two products are small (2.7 GFLOP at rank 32). As two tcgen05 GEMMs the first one has rank <= 128 output
// columns, i.e. one 256-row tile per CTA pair and 16 pairs for 4096 rows, each walking all of K alone; here a CTA owns
// ROWS = 32 rows, so 4096 rows fill 128 SMs, and its warps split K. mma.sync rather than tcgen05: its 16-row
// granularity is what gives that many CTAs, its operands come straight from global memory into registers, and its rate is
// not the bound.
//
// Phase 1: warp w takes every WARPS-th 32-wide slice of K. An MMA may see K in any order as long as both operands use the
// same one, so lane (g = lane / 4, q = lane % 4) holds elements [8 q, 8 q + 8) of the slice -- one 16-byte load per row of x
// and per row of A -- and two m16n8k16 steps consume them. The warps' partial sums meet in shared memory and leave as bf16.
// Phase 2: a warp takes 32 output features at a time; column 2 q + i of its n8 tile j stands for feature 8 q + 2 j + i, so a
// lane ends up with eight consecutive features of a row: y moves in 16-byte accesses, and the next group's y is fetched
// under the current one's products. When the row tiles alone leave SMs idle, blockIdx.y splits the features and each such
// CTA computes its hidden rows again from L2. 4096 x 5120 -> 5120, rank 32: 32.8 us (as two GEMMs 114.8 us).
#include <cuda_bf16.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "kernels.cuh"
#include "runtime.h"

namespace sfq {
namespace {

constexpr int kLoraRows = 32;

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 zero4() { return make_uint4(0, 0, 0, 0); }

// Two m16n8k16 steps over one 32-wide slice: `lo` / `hi` = this lane's eight elements of rows g / g + 8, `b` of column g.
__device__ __forceinline__ void mma_slice(float (&d)[4], const uint4& lo, const uint4& hi, const uint4& b) {
  const uint32_t a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
  mma_16816(d, a0, b.x, b.y);
  mma_16816(d, a1, b.z, b.w);
}

// NT: rank in tiles of 8, a multiple of 4 (32, 64, 96 or 128 ranks); ranks past `rank` are zeros.
template <int NT, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
lora_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ fa, const __nv_bfloat16* __restrict__ fb,
            __nv_bfloat16* __restrict__ y, int rows, int in, int out, int rank) {
  constexpr int RANK = NT * 8;
  constexpr int kPitch = RANK + 4;  // fp32 words per row of a warp's partial sums: lanes of a quad land in different banks
  extern __shared__ float part[];   // [WARPS][32][kPitch]; afterwards the bf16 hidden rows, [32][RANK + 8]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, q = lane & 3;
  const int row0 = blockIdx.x * kLoraRows;

  // ---- phase 1: partial hidden[32][RANK] of this warp's K slices
  float acc[2][NT][4];
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
  const __nv_bfloat16* xr[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) xr[r] = x + size_t(min(row0 + g + 8 * r, rows - 1)) * in;  // rows past the end: read, not stored
  constexpr int kStep = WARPS * 32;
  constexpr int U = NT <= 4 ? 4 : 2;  // slices in flight together
  for (int k0 = warp * 32; k0 < in; k0 += U * kStep) {
    uint4 xv[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * kStep + q * 8;
#pragma unroll
      for (int r = 0; r < 4; ++r) xv[u][r] = k < in ? __ldg(reinterpret_cast<const uint4*>(xr[r] + k)) : zero4();
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * kStep + q * 8;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int a_row = n * 8 + g;
        const uint4 b = (k < in && a_row < rank) ? __ldg(reinterpret_cast<const uint4*>(fa + size_t(a_row) * in + k)) : zero4();
#pragma unroll
        for (int m = 0; m < 2; ++m) mma_slice(acc[m][n], xv[u][2 * m], xv[u][2 * m + 1], b);
      }
    }
  }
  float* mine = part + size_t(warp) * kLoraRows * kPitch;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      *reinterpret_cast<float2*>(mine + (m * 16 + g) * kPitch + n * 8 + q * 2) = make_float2(acc[m][n][0], acc[m][n][1]);
      *reinterpret_cast<float2*>(mine + (m * 16 + g + 8) * kPitch + n * 8 + q * 2) = make_float2(acc[m][n][2], acc[m][n][3]);
    }
  __syncthreads();
  constexpr int kPairs = kLoraRows * RANK / 2 / (WARPS * 32);  // hidden pairs per thread
  static_assert(kPairs * WARPS * 64 == kLoraRows * RANK, "the hidden tile divides evenly over the threads");
  float2 h[kPairs];
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const int e = (i * WARPS * 32 + int(threadIdx.x)) * 2;
    const float* p = part + (e / RANK) * kPitch + e % RANK;
    float2 s = *reinterpret_cast<const float2*>(p);
#pragma unroll
    for (int w = 1; w < WARPS; ++w) {
      const float2 v = *reinterpret_cast<const float2*>(p + size_t(w) * kLoraRows * kPitch);
      s.x += v.x, s.y += v.y;
    }
    h[i] = e % RANK < rank ? s : make_float2(0.0f, 0.0f);  // ranks that do not exist stay zero whatever x holds (inf * 0)
  }
  __syncthreads();
  constexpr int kHPitch = RANK + 8;  // bf16 per hidden row: 16-byte units of neighbouring rows land in different banks
  __nv_bfloat16* hidden = reinterpret_cast<__nv_bfloat16*>(part);
#pragma unroll
  for (int i = 0; i < kPairs; ++i) {
    const int e = (i * WARPS * 32 + int(threadIdx.x)) * 2;
    *reinterpret_cast<__nv_bfloat162*>(hidden + (e / RANK) * kHPitch + e % RANK) = __floats2bfloat162_rn(h[i].x, h[i].y);
  }
  __syncthreads();

  // ---- phase 2: 32 features at a time
  constexpr int KS = NT / 4;  // 32-wide slices of the rank
  uint4 hv[KS][4];
#pragma unroll
  for (int s = 0; s < KS; ++s)
#pragma unroll
    for (int r = 0; r < 4; ++r) hv[s][r] = *reinterpret_cast<const uint4*>(hidden + (g + 8 * r) * kHPitch + s * 32 + q * 8);
  const int groups = (out + 31) / 32;
  const int stride = WARPS * int(gridDim.y);
  auto load_y = [&](int grp, uint4 (&v)[4]) {
    const int f = grp * 32 + q * 8;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = row0 + g + 8 * r;
      v[r] = (grp < groups && f < out && row < rows) ? *reinterpret_cast<const uint4*>(y + size_t(row) * out + f) : zero4();
    }
  };
  int grp = int(blockIdx.y) * WARPS + warp;
  uint4 next[4];
  load_y(grp, next);
  for (; grp < groups; grp += stride) {
    uint4 cur[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) cur[r] = next[r];
    uint4 bv[4][KS];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int feature = min(grp * 32 + 8 * (g >> 1) + 2 * j + (g & 1), out - 1);
#pragma unroll
      for (int s = 0; s < KS; ++s)
        bv[j][s] = s * 32 + q * 8 < rank ? __ldg(reinterpret_cast<const uint4*>(fb + size_t(feature) * rank + s * 32 + q * 8)) : zero4();
    }
    load_y(grp + stride, next);
    float d[2][4][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        d[m][j][0] = d[m][j][1] = d[m][j][2] = d[m][j][3] = 0.0f;
#pragma unroll
        for (int s = 0; s < KS; ++s) mma_slice(d[m][j], hv[s][2 * m], hv[s][2 * m + 1], bv[j][s]);
      }
    const int f = grp * 32 + q * 8;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = row0 + g + 8 * r;
      const __nv_bfloat162* yp = reinterpret_cast<const __nv_bfloat162*>(&cur[r]);
      uint4 o;
      __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float* dv = &d[r >> 1][j][(r & 1) * 2];
        const float2 b = __bfloat1622float2(__floats2bfloat162_rn(dv[0], dv[1])), c = __bfloat1622float2(yp[j]);
        op[j] = __floats2bfloat162_rn(b.x + c.x, b.y + c.y);
      }
      if (f < out && row < rows) *reinterpret_cast<uint4*>(y + size_t(row) * out + f) = o;
    }
  }
}

template <int NT, int WARPS>
void launch(const __nv_bfloat16* x, const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* y, int rows, int in, int out, int rank,
            cudaStream_t stream) {
  constexpr int kSmem = WARPS * kLoraRows * (NT * 8 + 4) * 4;
  reserve_dynamic_smem(reinterpret_cast<const void*>(&lora_kernel<NT, WARPS>), kSmem, "sfq lora");
  const int row_tiles = (rows + kLoraRows - 1) / kLoraRows;
  // features split over CTAs while row tiles alone leave SMs idle, at most eight ways (each repeats phase 1 from L2)
  const int most = std::max(1, std::min(8, (out + 32 * WARPS - 1) / (32 * WARPS)));
  const int splits = std::max(1, std::min(most, device_sm_count() / row_tiles));
  lora_kernel<NT, WARPS><<<dim3(row_tiles, splits), WARPS * 32, kSmem, stream>>>(x, a, b, y, rows, in, out, rank);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("sfq lora: launch failed: ") + cudaGetErrorString(e));
}

}  // namespace

bool lora_fused(const __nv_bfloat16* x, const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* y, int rows, int in, int out, int rank,
                cudaStream_t stream) {
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (rank <= 0 || rank > 128 || rank % 8 != 0 || in % 8 != 0 || out % 8 != 0 || !aligned(x) || !aligned(a) || !aligned(b) || !aligned(y)) return false;
  // A CTA fetches y ahead of its stores, and the CTAs that share a row tile each read all of its x rows while the others store: x and
  // y have to be apart. An update in place goes through the two GEMMs, where a slice's hidden rows are complete before its y is touched.
  const __nv_bfloat16 *x_end = x + size_t(rows) * in, *y_end = y + size_t(rows) * out;
  if (x < y_end && y < x_end) return false;
  // Above rank 64 every CTA reads all of A (in x rank) from L2 for its 32 rows, with registers for no more than two slices in flight,
  // so what decides is in x rank, and whether the two GEMMs need more than one slice. This kernel against two GEMMs, inputs from HBM:
  // one slice (2048 rows) 2560 -> 5120 rank 72 48.1 / 58.2 us, rank 128 60.4 / 56.3; 5120 -> 5120 rank 72 70.7 / 66.6; 512 rows 13824 -> 5120
  // rank 128 199 / 79. More (4096 rows) 13824 -> 5120 rank 72 169 / 190; rank 128 5120 -> 5120 113 / 126, 7680 -> 5120 146 / 139, and with few
  // outputs 5120 -> 1024 85 / 75 (20000 rows 286 / 337). Ranks up to 64: never slower (closest: rank 64, 2048 rows 13824 -> 512, 75.8 / 74.8).
  const size_t factor = size_t(in) * rank;
  const bool one_launch = rank <= 64 || (rows <= 2048 ? factor <= 200000
                                                      : rank <= 80 || (factor <= 660000 && (in <= out || in <= 2560 || rows > 8192)));
  if (!one_launch) return false;
  if (rank <= 32)
    launch<4, 16>(x, a, b, y, rows, in, out, rank, stream);
  else if (rank <= 64)
    launch<8, 8>(x, a, b, y, rows, in, out, rank, stream);
  else
    launch<16, 8>(x, a, b, y, rows, in, out, rank, stream);
  return true;
}

}  // namespace sfq

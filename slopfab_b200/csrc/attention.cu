// Full (unmasked, non-causal) self-attention with head_dim 128 on tcgen05: out = softmax(q k^T * scale) v per head.
//
// The reference's interface is attention_forward / attention_forward_query_chunk
// (include/slopfab/cuda/attention.cuh:176-196): q, k, v are [seq, heads * 128] row-major bf16, exactly the thirds of the
// fused QKV projection; queries may be a compact chunk of the sequence; no mask exists anywhere in the model.
//
// One CTA owns TWO tiles of 128 queries of one head and walks the keys in steps of 64 with an online softmax. The scores of a
// query tile lie in two halves of 64 columns that take turns, so a step's scores are computed while the softmax warps work on the
// step before and a query tile's chain (scores -> softmax -> product -> next scores) has two steps in it at a time.
//   warp 0      TMA producer: both Q tiles once, then a two-stage ring of K and V tiles [128 keys x 128 d]. The second product
//               reads V as it lies, as an N-major operand (its N is d, its K the keys), or - VT, where its rows are not aligned -
//               V transposed once per call by transpose_v_kernel, [128 d x 128 keys], K-major like the other operands
//   warp 1      one lane issues, per step h and query tile t: O_t += P_t(h) V(h) (four MMAs 128x128x16), S_t(h + 2) = Q_t K(h + 2)^T
//               (eight MMAs 128x64x16) over the columns P_t(h) was read from, and a commit. S and O of both query tiles live in
//               TMEM (4 x 128 columns); P is read by the second product straight from TMEM, where it overwrites the first
//               32 columns of the 64 scores it was computed from
//   warps 4-7   softmax of query tile 0, warps 8-11 of query tile 1 (warps 2-3 only hand their registers over), one query row per
//               thread with all 64 keys of the step: S from TMEM, P = exp2(s - m) as bf16 pairs back into TMEM, the running sum,
//               and - only when the probabilities of the key tile so far sum to more than 2^15, i.e. the row has outgrown the reference
//               m the accumulator was last scaled to - the maximum of m and this step's scores as the new reference, a rescale of O
//               in TMEM and the step's probabilities again, none of them above 1. A stale reference, or one that is not the
//               maximum of all keys so far, changes nothing in exact arithmetic (numerator and denominator
//               carry the same factor); the limit keeps every p far inside the range of bf16 and fp32, and no maximum over
//               the scores is computed on the common path.
// 40 heads, 2048 / 4747 / 18900 tokens in bursts: 0.096 / 0.406 / 5.48 ms (75600: 96.6 ms); steps of 128 keys, whose next scores wait for the
// product that still reads P from their columns, 0.107 / 0.448 / 5.72 ms. What bounds it (timing-only ablations at 18900 tokens, of a
// build that took 5.3 to 5.5 ms whole): the tensor side alone takes 4.6 ms, most of it shared memory (a 128x64x16 MMA reads 6 KB in the
// 32 cycles its arithmetic takes and runs in 48), the softmax side alone 4.2.
// A row whose scores keep growing pays for its moves: 4747 tokens whose scores rise by 26 (104) log2 units along the keys, where a warp
// moves in 16 % (60 %) of its steps, 0.490 (0.671) ms; the steps of 128 keys 0.578 (0.653).
// Every wait is bounded; a wait that runs out stores a code in the status word and the CTA leaves.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <stdexcept>
#include <string>

#include "gemm_common.cuh"
#include "kernels.cuh"
#include "ptx.cuh"
#include "runtime.h"

namespace sfq {
namespace {

using namespace ptx;

constexpr int kTile = 128;             // queries per query tile (two per CTA), keys per stage of K and V, head_dim
constexpr int kSlab = kTile * 128;     // 128 rows x 128 bytes: 64 bf16 columns of a tile
constexpr int kTileBytes = 2 * kSlab;  // [128 x 128] bf16
constexpr int kStep = 64;              // keys per softmax step: half a key tile, half of a query tile's score columns
constexpr int kAttnThreads = 384;  // warpgroup 0: producer, MMA issuer, two idle warps; warpgroups 1 and 2: the softmax of query tiles 0 and 1
constexpr int kAttnRegsLean = 64, kAttnRegsSoftmax = 216;  // after setmaxnreg: 128 x 64 + 256 x 216 < 384 x 168, what the launch allocates
constexpr int kTailWaves = 16;
constexpr float kTileSumLimit = 32768.0f;  // a row's probabilities of a key tile may sum to this before its reference moves

struct AttnShared {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2][2], p_full[2][2];
  uint32_t tmem_base;
  volatile int abort;
};
constexpr int kAttnSmem = 1024 /* alignment slack */ + 6 * kTileBytes /* Q x2, K x2, V x2 */ + 1024;

struct AttnArgs {
  __nv_bfloat16* out;
  int ld_out;
  int seq_q, seq_kv;
  int q_blocks;  // blocks of 256 queries per head
  int whole;     // the first `whole` CTAs take a (block, head) each; behind them a unit is two CTAs, one per query tile
  int group;         // query heads per key/value head
  float scale_log2;  // scale * log2(e)
  int* status;
};

// `nap` > 0: sleep that many nanoseconds between polls. The softmax warps and the producer wait for long stretches by
// design; polling flat out they would take issue slots from the one warp that feeds the tensor pipe.
template <int nap = 0>
__device__ __forceinline__ bool attn_wait(uint32_t bar, uint32_t parity, AttnShared* sh, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock_now();
  for (;;) {
    for (int i = 0; i < 64; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
      if (nap > 0) __nanosleep(nap);
    }
    if (sh->abort) return false;
    if (clock_now() - start > kWaitCycles) {
      atomicCAS(status, 0, code);
      sh->abort = 1;
      return false;
    }
  }
}

// Minima and maxima that a NaN goes through (fminf and fmaxf drop it), one instruction each.
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float min_nan(float a, float b) {
  float d;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 2^x for a pair of arguments on the FMA pipe instead of the special-function unit, which would need 2048 cycles for the 32768
// exponentials of two query tiles and a key tile (16 per clock), where their products take about 2500. A quarter of the pairs
// taken here / none, 40 heads in bursts: 2048 tokens 0.0956 / 0.0975 ms, 4747 0.406 / 0.412, 18900 5.48 / 5.52, 75600 level.
// x = n + f with n = round(x), f in [-1/2, 1/2]: a cubic for 2^f (relative error 7.5e-5, a sixtieth of the bf16 rounding
// the result goes through) and n added into the exponent field. Arguments are clamped at -125 below, where the result
// (~2e-38) is as good as the zero the hardware instruction returns, and at 126 above: a row that has outgrown its
// reference by that much must still produce a huge value, which the caller's sum test then catches. So does a NaN, whose
// exponent field the addition leaves at 0x7f7fffff, the largest finite number: the caller looks for NaN where it moves the reference.
__device__ __forceinline__ f32x2 exp2_pair_fma(f32x2 x) {
  float x0, x1;
  unpack2(x, x0, x1);
  const f32x2 xc = pack2(min_nan(max_nan(x0, -125.0f), 126.0f), min_nan(max_nan(x1, -125.0f), 126.0f));
  const f32x2 magic = pack2(12582912.0f, 12582912.0f);  // 1.5 * 2^23: the sum's low mantissa bits hold round(x)
  const f32x2 t = add2(xc, magic);
  const f32x2 f = sub2(xc, sub2(t, magic));
  f32x2 p = fma2(pack2(0.0551716648f, 0.0551716648f), f, pack2(0.2426111251f, 0.2426111251f));
  p = fma2(p, f, pack2(0.6932609677f, 0.6932609677f));
  p = fma2(p, f, pack2(0.9999280572f, 0.9999280572f));
  float p0, p1, t0, t1;
  unpack2(p, p0, p1);
  unpack2(t, t0, t1);
  return pack2(__int_as_float(__float_as_int(p0) + (__float_as_int(t0) << 23)), __int_as_float(__float_as_int(p1) + (__float_as_int(t1) << 23)));
}
constexpr int kFmaPairsOfFour = 1;  // of every four pairs of probabilities, how many take the FMA-pipe exponential

// TAIL: the units of the last wave run as CTAs of one query tile each (see attention_forward). Without it every CTA has two
// tiles at compile time and the grid is (blocks of 256 queries, heads).
template <bool VT, bool TAIL>
__global__ void __launch_bounds__(kAttnThreads, 1)
    attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                     const __grid_constant__ CUtensorMap map_v, const AttnArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;                    // two query tiles
  uint8_t* k_s = smem + 2 * kTileBytes;   // two stages
  uint8_t* v_s = smem + 4 * kTileBytes;   // two stages
  AttnShared* sh = reinterpret_cast<AttnShared*>(smem + 6 * kTileBytes);

  const int warp = int(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int tail_cta = TAIL ? int(blockIdx.x) - g.whole : -1;
  const int unit = tail_cta < 0 ? int(blockIdx.x) : g.whole + (tail_cta >> 1);
  const int q0 = (TAIL ? unit % g.q_blocks : unit) * (2 * kTile) + (tail_cta < 0 ? 0 : (tail_cta & 1) * kTile);
  const int head = TAIL ? unit / g.q_blocks : int(blockIdx.y);
  if (TAIL && q0 >= g.seq_q) return;  // the second half of a split block may have no queries
  const bool two = !TAIL || (tail_cta < 0 && q0 + kTile < g.seq_q);  // otherwise query tile 0 alone
  const int kv_head = head / g.group;
  const int tiles = (g.seq_kv + kTile - 1) / kTile, steps = (g.seq_kv + kStep - 1) / kStep;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sh->q_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sh->k_full[i]), 1);
      mbar_init(smem_u32(&sh->k_empty[i]), 1);
      mbar_init(smem_u32(&sh->v_full[i]), 1);
      mbar_init(smem_u32(&sh->v_empty[i]), 1);
      for (int half = 0; half < 2; ++half) {  // per query tile i and half of its score columns
        mbar_init(smem_u32(&sh->s_full[i][half]), 1);  // the product that read the half has completed, and the next scores are in it
        mbar_init(smem_u32(&sh->p_full[i][half]), 4);  // the four softmax warps have written P over it (and rescaled O)
      }
    }
    sh->abort = 0;
    fence_barrier_init();
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  grid_dependency_release();
  grid_dependency_wait();  // q, k and the transposed v
  const uint32_t tmem = warp_uniform(sh->tmem_base);  // columns: S/P of tile 0 [0,128), of tile 1 [128,256), O of tile 0 [256,384), of tile 1 [384,512)

  // Each role's code sits directly under its warpgroup's setmaxnreg, so the compiler budgets it accordingly.
  if (warp < 4) {
    reg_dec<kAttnRegsLean>();
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      mbar_arrive_expect_tx(smem_u32(&sh->q_full), (two ? 2 : 1) * kTileBytes);
      for (int t = 0; t < (two ? 2 : 1); ++t) {
        tma_load_2d(smem_u32(q_s + t * kTileBytes), &map_q, head * 256, q0 + t * kTile, smem_u32(&sh->q_full));
        tma_load_2d(smem_u32(q_s + t * kTileBytes + kSlab), &map_q, head * 256 + 128, q0 + t * kTile, smem_u32(&sh->q_full));
      }
      for (int j = 0; j < tiles; ++j) {
        const int st = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        if (!attn_wait<200>(smem_u32(&sh->k_empty[st]), ph, sh, g.status, 11)) break;
        mbar_arrive_expect_tx(smem_u32(&sh->k_full[st]), kTileBytes);
        tma_load_2d(smem_u32(k_s + st * kTileBytes), &map_k, kv_head * 256, j * kTile, smem_u32(&sh->k_full[st]));
        tma_load_2d(smem_u32(k_s + st * kTileBytes + kSlab), &map_k, kv_head * 256 + 128, j * kTile, smem_u32(&sh->k_full[st]));
        if (!attn_wait<200>(smem_u32(&sh->v_empty[st]), ph, sh, g.status, 12)) break;
        mbar_arrive_expect_tx(smem_u32(&sh->v_full[st]), kTileBytes);
        if (VT) {  // rows are (kv_head, d), columns are keys; 64 keys = 128 bytes per slab
          tma_load_2d(smem_u32(v_s + st * kTileBytes), &map_v, j * 256, kv_head * kTile, smem_u32(&sh->v_full[st]));
          tma_load_2d(smem_u32(v_s + st * kTileBytes + kSlab), &map_v, j * 256 + 128, kv_head * kTile, smem_u32(&sh->v_full[st]));
        } else {
          tma_load_2d(smem_u32(v_s + st * kTileBytes), &map_v, kv_head * 256, j * kTile, smem_u32(&sh->v_full[st]));
          tma_load_2d(smem_u32(v_s + st * kTileBytes + kSlab), &map_v, kv_head * 256 + 128, j * kTile, smem_u32(&sh->v_full[st]));
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (one lane)
    // S_t(h + 2) overwrites the columns that P_t(h) V(h) reads its A operand from, with nothing between the two but the order of
    // issue. That the tensor pipe executes MMAs of one thread in order is documented for MMAs of one accumulator and shape; these two
    // differ in both, so here it is relied on beyond that, as the form in steps of 128 keys relied on it for the accumulators (a
    // wait for the product's completion in its place would put the round trip back into the chain). The commit behind both, on
    // the half's s_full, also says that O_t holds the sum up to step h. It is sent without scores, too, at the end of the keys.
    constexpr uint32_t idesc_s = idesc_bf16(kTile, kStep);
    constexpr uint32_t idesc_pv = VT ? idesc_bf16(kTile, kTile) : idesc_bf16(kTile, kTile) | kIdescBMajorN;
    // B of the second product = V [keys x d], N-major (16 keys are two groups of eight 128-byte rows), or V^T [d x keys] (four
    // MMAs per slab of 64 keys, 32 bytes of each row apiece)
    constexpr uint64_t kKeys16 = VT ? 2 : 16 * 128 >> 4;                   // 16 keys on
    constexpr uint64_t kKeys64 = VT ? uint64_t(kSlab >> 4) : 4 * kKeys16;  // 64 keys on
    if (elect_one()) {
      auto wait = [&](uint64_t* bar, uint32_t parity, int code) {  // one non-suspending probe; only a real wait takes the polling loop
        return mbar_test_wait(smem_u32(bar), parity) || attn_wait(smem_u32(bar), parity, sh, g.status, code);
      };
      auto issue_s = [&](int t, int half, uint64_t k_desc) {  // scores of query tile t and 64 keys into that half of its columns
        const uint64_t a = smem_desc_sw128(smem_u32(q_s + t * kTileBytes)), b = k_desc + half * (kStep * 128 >> 4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint64_t adv = uint64_t((i >> 2) * (kSlab >> 4) + (i & 3) * 2);
          mma_f16(tmem + t * kTile + half * kStep, a + adv, b + adv, idesc_s, i ? 1u : 0u);
        }
      };
      bool ok = wait(&sh->q_full, 0, 13) && wait(&sh->k_full[0], 0, 14);
      if (ok) {
        tc_fence_after_sync();
        for (int half = 0; half < (steps > 1 ? 2 : 1); ++half)
          for (int t = 0; t < (two ? 2 : 1); ++t) {
            issue_s(t, half, smem_desc_sw128(smem_u32(k_s)));
            tc_commit(smem_u32(&sh->s_full[t][half]));
          }
        tc_commit(smem_u32(&sh->k_empty[0]));
      }
      for (int j = 0; j < tiles && ok; ++j) {
        const int st = j & 1;
        const uint64_t k_desc = smem_desc_sw128(smem_u32(k_s + (st ^ 1) * kTileBytes));
        const uint64_t v_desc = VT ? smem_desc_sw128(smem_u32(v_s + st * kTileBytes)) : smem_desc_sw128_mn(smem_u32(v_s + st * kTileBytes), kSlab);
        if (!(ok = wait(&sh->v_full[st], (j >> 1) & 1, 16))) break;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int h = 2 * j + half;
          if (h >= steps || !ok) break;
          const bool more = h + 2 < steps;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (t == 1 && !two) break;
            if (!(ok = wait(&sh->p_full[t][half], j & 1, 17))) break;
            tc_fence_after_sync();
            // A = P_t in tensor memory [queries x keys], 16 keys (eight 32-bit columns of bf16 pairs) per MMA
            const uint32_t d = tmem + 2 * kTile + t * kTile, a = tmem + t * kTile + half * kStep;
#pragma unroll
            for (int i = 0; i < 4; ++i) mma_f16_ts(d, a + 8 * i, v_desc + half * kKeys64 + i * kKeys16, idesc_pv, (i || h) ? 1u : 0u);
            if (more) {
              if (half == 0 && t == 0) {  // the first reader of the next K tile waits for it
                if (!(ok = wait(&sh->k_full[st ^ 1], ((j + 1) >> 1) & 1, 14))) break;
                tc_fence_after_sync();
              }
              issue_s(t, half, k_desc);
            }
            tc_commit(smem_u32(&sh->s_full[t][half]));
          }
          if (half == 1 || h + 1 == steps) tc_commit(smem_u32(&sh->v_empty[st]));
          if (more && (half == 1 || h + 3 == steps)) tc_commit(smem_u32(&sh->k_empty[st ^ 1]));
        }
      }
    }
    __syncwarp();
  }
  } else {
    reg_inc<kAttnRegsSoftmax>();
    // ------------------------------------------------------------ softmax, rescale, output
    // Warps 4-7 serve query tile 0, warps 8-11 query tile 1; within a tile a warp owns the 32 rows of the TMEM quadrant
    // it may access (warp index % 4) and a thread one query row with all 64 keys of the step, so nothing is exchanged
    // between threads.
    const int t = (warp - 4) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const uint32_t tmem_s = tmem + lane_base + t * kTile;
    const uint32_t tmem_o = tmem + lane_base + 2 * kTile + t * kTile;
    // The maximum the accumulator and the running sum are expressed against (log2 units). It stays at the lowest number while all of
    // a row's scores are -inf: against -inf itself they would be NaN.
    float m_used = -FLT_MAX;
    float l = 0.0f;
    bool ok = true;
    uint32_t r[2][32];  // the step's scores
    const f32x2 scale2 = pack2(g.scale_log2, g.scale_log2);
    // p = 2^(s * scale - m) for the 32 keys of chunk c as bf16 pairs, written over columns [16 c, 16 c + 16) of the step's
    // scores (chunk 0's, which are in registers by then); returns their sum.
    auto emit_chunk = [&](uint32_t cols, int c, float m, f32x2 sum2) {
      const f32x2 negm2 = pack2(-m, -m);
      uint32_t pk[16];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const f32x2 x = fma2(pack2(__uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1])), scale2, negm2);
        f32x2 p;
        if (((i >> 1) & 3) < kFmaPairsOfFour) {
          p = exp2_pair_fma(x);
        } else {
          float x0, x1;
          unpack2(x, x0, x1);
          p = pack2(fast_exp2(x0), fast_exp2(x1));
        }
        sum2 = add2(sum2, p);
        float p0, p1;
        unpack2(p, p0, p1);
        const __nv_bfloat162 pb = __floats2bfloat162_rn(p0, p1);  // key 2i in the low half: the lower K index
        pk[i >> 1] = *reinterpret_cast<const uint32_t*>(&pb);
      }
      tmem_st_32x16(cols + c * 16, pk);
      return sum2;
    };
    auto load_step = [&](int h) {
      const uint32_t cols = tmem_s + (h & 1) * kStep;
      tmem_ld_32x32(cols, r[0]);
      tmem_ld_32x32(cols + 32, r[1]);
      tmem_ld_wait();
      const int valid = g.seq_kv - h * kStep;  // keys of this step that exist; the last step may have fewer than 64
      if (valid < kStep)
#pragma unroll
        for (int i = 0; i < kStep; ++i)
          if (i >= valid) r[i >> 5][i & 31] = __float_as_uint(-INFINITY);
    };
    auto chunk_max = [&](int c) {
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four short chains instead of one of 32 steps
#pragma unroll
      for (int i = 0; i < 32; i += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k) m4[k] = max3(m4[k], __uint_as_float(r[c][i + 2 * k]), __uint_as_float(r[c][i + 2 * k + 1]));
      return max_nan(max_nan(m4[0], m4[1]), max_nan(m4[2], m4[3]));
    };
    // The reference maximum becomes m_new in the rows that outgrew it; O and the running sum follow (the TMEM accesses are
    // warp-wide; rows within their limit use a factor of 1). O_t has to be at rest.
    auto move_reference = [&](float m_new, bool rescale) {
      if (rescale) {
        const float f = m_new == m_used ? 1.0f : fast_exp2(m_used - m_new);
        l *= f;
        uint32_t o[32];
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          tmem_ld_32x32(tmem_o + c * 32, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
          tmem_st_32x32(tmem_o + c * 32, o);
        }
      }
      m_used = m_new;
    };
    auto total = [&](f32x2 sum2) {
      float a, b;
      unpack2(sum2, a, b);
      return a + b;
    };
    auto wait_half = [&](int h, int code) {  // the scores of step h are in its half; the product of step h - 2 has completed
      ok = __all_sync(0xffffffffu, attn_wait<40>(smem_u32(&sh->s_full[t][h & 1]), (h >> 1) & 1, sh, g.status, code));
      tc_fence_after_sync();
      return ok;
    };
    const int my_steps = t == 0 || two ? steps : 0;
    // The first reference is the maximum over the first 128 keys.
    for (int h = 0; h < min(my_steps, 2); ++h) {
      if (!wait_half(h, 18)) break;
      load_step(h);
      m_used = max_nan(m_used, max_nan(chunk_max(0), chunk_max(1)) * g.scale_log2);  // scale > 0: the maximum commutes with it
    }
    f32x2 sum2 = pack2(0.0f, 0.0f);  // of the 128-key tile so far: one chain over its keys, so that the bits of rows that keep their first reference do not depend on the steps
    // One body for both halves: two bodies no longer fit the instruction cache (2048 / 4747 / 18900 tokens 0.0988 / 0.417 / 5.58 ms,
    // 0.0956 / 0.406 / 5.48 as it is).
#pragma unroll 1
    for (int h = 0; h < my_steps && ok; ++h) {
      const int half = h & 1;
      const uint32_t cols = tmem_s + half * kStep;
      if (!wait_half(h, 18)) break;
      load_step(h);
      // The probabilities are computed against the reference maximum the accumulator was last scaled to. No maximum is taken on
      // this path: that the reference is still good enough is read off the sum of the probabilities.
      f32x2 start = half ? sum2 : pack2(0.0f, 0.0f);
      sum2 = emit_chunk(cols, 0, m_used, start);
      sum2 = emit_chunk(cols, 1, m_used, sum2);
      const bool over = !(total(sum2) <= kTileSumLimit);  // a row that outgrew its reference; inf or NaN
      if (__any_sync(0xffffffffu, over)) {
        // Rare. The reference becomes the maximum of itself and this step's scores (itself, where only the sum carried over from the
        // tile's first half is above the limit: the sum then starts anew). O_t is at rest once the product of the step before has completed, which that
        // step's half says the next time it is handed over. The probabilities are computed again -- every score is still in
        // registers -- over the ones just written; rows within their limit keep reference and sum, so that they do not
        // depend on their neighbours.
        if (h > 0 && !wait_half(h + 1, 21)) break;
        float m_new = m_used;
        if (over) {
          m_new = max_nan(m_used, max_nan(chunk_max(0), chunk_max(1)) * g.scale_log2);
          m_new = fmaf(m_new, 0.0f, m_new);  // a score of +inf or NaN makes its row NaN: the reference becomes it, and with it all that follows
          l += total(start);
          start = pack2(0.0f, 0.0f);
        }
        move_reference(m_new, h > 0);
        sum2 = emit_chunk(cols, 0, m_used, start);
        sum2 = emit_chunk(cols, 1, m_used, sum2);
      }
      if (half == 1 || h + 1 == my_steps) l += total(sum2);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sh->p_full[t][half]));
    }
    if (ok && my_steps > 0 &&  // the last step's product has completed
        (ok = __all_sync(0xffffffffu, attn_wait(smem_u32(&sh->s_full[t][(my_steps - 1) & 1]), ((my_steps + 1) >> 1) & 1, sh, g.status, 20)))) {
      tc_fence_after_sync();
      const float inv = m_used > -FLT_MAX ? 1.0f / l : NAN;  // NaN: no score of the row is finite, or one of them is NaN or +inf
      const int qrow = q0 + t * kTile + row;
      const bool row_ok = qrow < g.seq_q;
      __nv_bfloat16* dst = g.out + size_t(row_ok ? qrow : 0) * g.ld_out + head * kTile;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t o[32];
        tmem_ld_32x32(tmem_o + c * 32, o);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(o[q * 8 + 2 * h]) * inv, __uint_as_float(o[q * 8 + 2 * h + 1]) * inv);
              w[h] = *reinterpret_cast<const uint32_t*>(&v);
            }
            *reinterpret_cast<uint4*>(dst + c * 32 + q * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      }
      tc_fence_before_sync();
    }
  }
  if (sh->abort) {
    // Leaving early: loads may still be in flight into this CTA's shared memory; give them far more time than a
    // load takes before the memory is released.
    const long long start = clock_now();
    while (clock_now() - start < 4000000ll) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

// V [seq, width] (row pitch ld_v) -> V^T [width, ld_t] with the columns [seq, ld_t) zeroed.
__global__ void __launch_bounds__(256) transpose_v_kernel(const __nv_bfloat16* v, int ld_v, __nv_bfloat16* __restrict__ vt, int ld_t,
                                                          int seq, int width) {
  __shared__ __nv_bfloat16 tile[64][66];
  grid_dependency_release();
  grid_dependency_wait();
  const int s0 = blockIdx.x * 64, w0 = blockIdx.y * 64;
  for (int i = threadIdx.x; i < 64 * 64; i += 256) {
    const int rs = i >> 6, cw = i & 63;
    tile[rs][cw] = (s0 + rs < seq && w0 + cw < width) ? v[size_t(s0 + rs) * ld_v + w0 + cw] : __float2bfloat16(0.0f);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 64 * 64; i += 256) {
    const int rw = i >> 6, cs = i & 63;
    if (w0 + rw < width && s0 + cs < ld_t) vt[size_t(w0 + rw) * ld_t + s0 + cs] = tile[cs][rw];
  }
}

// [rows, cols] bf16 with a row pitch, boxes of {64 columns, 128 rows}, 128-byte swizzle, zero fill outside.
CUtensorMap make_attn_map(const void* base, size_t rows, size_t cols, size_t pitch_elems) {
  if (reinterpret_cast<uintptr_t>(base) % 16 != 0 || (pitch_elems * 2) % 16 != 0)
    throw std::invalid_argument("sfq attention: operand base and row pitch must be 16-byte aligned for TMA");
  CUtensorMap m;
  const cuuint64_t dims[2] = {cols * 2, rows};
  const cuuint64_t strides[1] = {pitch_elems * 2};
  const cuuint32_t box[2] = {128, cuuint32_t(kTile)};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem,
                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw std::runtime_error("sfq attention: cuTensorMapEncodeTiled failed (" + std::to_string(int(r)) + ")");
  return m;
}

size_t align256(size_t n) { return (n + 255) / 256 * 256; }
int padded_keys(int seq_kv) { return (seq_kv + 63) / 64 * 64; }

}  // namespace

size_t attention_workspace_bytes(int seq_kv, int kv_heads, int head_dim) {
  if (seq_kv <= 0 || kv_heads <= 0 || head_dim != kTile) throw std::invalid_argument("sfq attention: head_dim must be 128 and the extents positive");
  return align256(size_t(kv_heads) * kTile * padded_keys(seq_kv) * sizeof(__nv_bfloat16));
}

void attention_forward(const __nv_bfloat16* q, int ld_q, const __nv_bfloat16* k, const __nv_bfloat16* v, int ld_kv, __nv_bfloat16* out, int ld_out,
                       int seq_q, int seq_kv, int heads, int kv_heads, int head_dim, float scale, void* workspace, size_t workspace_bytes,
                       cudaStream_t stream) {
  if (seq_q <= 0) return;
  if (head_dim != kTile) throw std::invalid_argument("sfq attention: only head_dim 128 is built");
  if (seq_kv <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0) throw std::invalid_argument("sfq attention: bad extents");
  if (!q || !k || !v || !out || !workspace) throw std::invalid_argument("sfq attention: null operand");
  if (ld_q < heads * kTile || ld_kv < kv_heads * kTile || ld_out < heads * kTile || ld_out % 8 != 0 || reinterpret_cast<uintptr_t>(out) % 16 != 0)
    throw std::invalid_argument("sfq attention: row pitches must cover heads * 128 columns and keep 16-byte alignment");
  if (workspace_bytes < attention_workspace_bytes(seq_kv, kv_heads, head_dim)) throw std::invalid_argument("sfq attention: workspace too small");
  if (out == q || out == k || out == v) throw std::invalid_argument("sfq attention: out may not alias q, k or v");
  if ((seq_q + kTile - 1) / kTile > 0x7FFFFFFF / 2 || heads > 65535 || (long long)((seq_q + 2 * kTile - 1) / (2 * kTile)) * heads > 0x3FFFFFFF) throw std::invalid_argument("sfq attention: too many query tiles or heads");
  for (auto kernel : {attention_kernel<false, false>, attention_kernel<false, true>, attention_kernel<true, false>, attention_kernel<true, true>})
    reserve_dynamic_smem(reinterpret_cast<const void*>(kernel), kAttnSmem, "sfq attention");

  // V is read as it lies, except one whose rows do not start on 16 bytes, which TMA cannot read: that one is transposed first.
  // 40 heads in loops of 0.25 s, as it lies against transposed (pass included): 2048 tokens 0.099 / 0.124 ms, 4747 0.465 / 0.518,
  // 18900 6.35 / 6.53.
  const bool transposed = reinterpret_cast<uintptr_t>(v) % 16 != 0;
  cudaError_t e = cudaSuccess;
  const int width = kv_heads * kTile, ld_t = padded_keys(seq_kv);
  const size_t kv_bytes = size_t(seq_kv) * width * 4;
  __nv_bfloat16* vt = static_cast<__nv_bfloat16*>(workspace);
  if (transposed) {
    e = launch_overlapped(kv_bytes, transpose_v_kernel, dim3((ld_t + 63) / 64, (width + 63) / 64), dim3(256), 0, stream, v, ld_kv, vt, ld_t, seq_kv, width);
    if (e != cudaSuccess) throw std::runtime_error(std::string("sfq attention: launch failed: ") + cudaGetErrorString(e));
  }

  const CUtensorMap mq = make_attn_map(q, size_t(seq_q), size_t(heads) * kTile, size_t(ld_q));
  const CUtensorMap mk = make_attn_map(k, size_t(seq_kv), size_t(width), size_t(ld_kv));
  const CUtensorMap mv = transposed ? make_attn_map(vt, size_t(width), size_t(ld_t), size_t(ld_t)) : make_attn_map(v, size_t(seq_kv), size_t(width), size_t(ld_kv));
  AttnArgs a;
  a.out = out, a.ld_out = ld_out, a.seq_q = seq_q, a.seq_kv = seq_kv, a.group = heads / kv_heads;
  a.scale_log2 = (scale > 0.0f ? scale : 1.0f / sqrtf(float(head_dim))) * 1.4426950408889634f;
  a.status = device_status_word();
  // Units (256 queries of a head) run one per SM, all equally long, so a last wave that is nearly empty costs as much as a full
  // one: 4747 tokens x 40 heads are 760 units = 5.14 waves of 148. When the last wave's units fit the SMs twice over, they run
  // as two CTAs of one query tile each, which take 0.75 of the time (74 units against 1000 / 4747 / 18900 keys 0.0161 / 0.0542 / 0.191 ms as
  // single tiles, 0.0213 / 0.0729 / 0.252 whole). 40 heads with the split / without: 2048 tokens 0.0954 / 0.1043 ms, 4747 0.407 / 0.424, 7500
  // 0.934 / 0.978. A row's arithmetic is the same either way. Past kTailWaves waves little is left to gain: 16200 tokens
  // (17.3 waves) 4.08 / 4.13 ms, 19200 (20.3) 5.63 / 5.68, 36000 (38.1) level within the noise of 1 %.
  a.q_blocks = (seq_q + 2 * kTile - 1) / (2 * kTile);
  const int units = a.q_blocks * heads, sms = device_sm_count(), rest = units % sms;
  const int split = 2 * rest <= sms && units < kTailWaves * sms && seq_q > kTile ? rest : 0;
  a.whole = units - split;
  if (split > 0)
    e = launch_overlapped(kv_bytes, transposed ? attention_kernel<true, true> : attention_kernel<false, true>, dim3(units + split), dim3(kAttnThreads), kAttnSmem,
                          stream, mq, mk, mv, a);
  else
    e = launch_overlapped(kv_bytes, transposed ? attention_kernel<true, false> : attention_kernel<false, false>, dim3(a.q_blocks, heads), dim3(kAttnThreads),
                          kAttnSmem, stream, mq, mk, mv, a);
  if (e != cudaSuccess) throw std::runtime_error(std::string("sfq attention: launch failed: ") + cudaGetErrorString(e));
}

}  // namespace sfq

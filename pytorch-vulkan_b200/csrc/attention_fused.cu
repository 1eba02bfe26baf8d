// Fused scaled dot-product attention on tcgen05, forward and backward, for calls without mask and dropout and heads of up to
// 64 dimensions: the scores never reach memory.  FP32 by the split-precision scheme of tc_common.cuh.
//
// What bounds it and what follows from that.  The composed form (attention.cu) writes, rewrites and reads the [tokens,
// tokens] matrix: 139 us forward and 258 us backward for 16 heads of 1024 tokens x 64, of which 60 us are products.  Here a CTA owns 128
// rows of one result and walks the other side's tokens in blocks of 64 columns:
//   S = own1 * col1^T                    (both operands in shared memory)
//   [dP = own2 * col2^T]
//   T = f(S, dP) element by element      (tensor memory -> registers -> tensor memory, TF32 + BF16 parts over S and dP)
//   acc += T * colB                      (T is the A operand in tensor memory)
//        own rows   S           dP            T                       acc    colB
//   FWD  queries    Q K^T                     P (running maximum)     O      V
//   DQ   queries    Q K^T       dO V^T        P (dP - delta)          dQ     K
//   DV   keys       K Q^T                     P^T                     dV     dO
//   DK   keys       K Q^T       V dO^T        (P (dP - delta))^T      dK     Q
// so each gradient has one writer and needs no atomics (eight products instead of five).  The own rows are staged once, in tensor
// memory where an operand costs no shared-memory bandwidth (the BF16 part of own2 does not fit there).  Two streams take alternate
// blocks, so that the element-wise work of one runs under the products of the other; a stream is eight warps, a thread half a row
// (32 columns: 64 left 168 registers a thread and 8 warps, which could not hide the latency of their own chain).  In the forward
// pass each stream keeps its own maximum, sum and accumulator, merged at the end, and rescales its accumulator only when the maximum
// has grown by more than 8 (a factor 256 of head room in FP32; the method of FlashAttention-4).  The column operands are split once per call into ready-made
// shared-memory images by stage_kernel, which also prepares log-sum-exp and delta; one thread fetches them with bulk copies.
//
// Measured, 16 heads of 1024 tokens x 64: forward 139 us composed -> 39 with four warps a stream -> 31; backward 258 -> 151 (three
// launches, four warps a stream) -> 100.  What is left is the element-wise work (about 14 instructions a score) beside 60 %
// of it in products, and 10 us of staging.  The log-sum-exp and the maxima are in base 2: the scale is folded into the operands.
//
// Replaces attention_forward / attention_backward of the reference (csrc/ops/attention.cpp:16-34, sdpa_training.comp) for
// these calls.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <initializer_list>
#include <mutex>

#include "attention_fused.cuh"
#include "common.cuh"
#include "dweight_stage.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace fa {
using namespace tc;

constexpr int M = 128, BC = 64;               // rows of a CTA, columns of a block
constexpr int STREAM_WARPS = 8, STREAMS = 2, LOAD_WARP = 16, MMA_WARP = 17, THREADS = 576;
constexpr int STAGES = 2;
constexpr uint32_t IMG_CHUNK = BC * 256u;     // one block x 32 dimensions of an image: 16 KB in either orientation
constexpr float LOG2E = 1.4426950408889634f;
enum { FWD = 0, DQ = 1, DV = 2, DK = 3 };

struct Args {
  const float *own1, *own2;                   // raw rows [batch][rows][d]
  const unsigned char *col1, *col2, *colb;    // images [batch][blocks][chunks] of the other side
  const float *lse2, *delta;                  // [batch][padded queries]: log-sum-exp in base 2 (+inf: no key), rowsum(dO O)
  float* out;                                 // [batch][rows][d]
  float* lse;                                 // FWD: [batch][rows]
  int rows, cols, d, blocks, q_pad;
  int causal;
  float scale, scale2;                        // score scale; the same times log2(e)
  int* status;
};

struct Ctrl {
  unsigned long long c_full[STAGES], c_empty[STAGES], b_full[STAGES], b_empty[STAGES], s_full[STREAMS], t_full[STREAMS], t_done[STREAMS], last;
  unsigned long long max_full[STREAMS][4];    // FWD: the two warps of 32 rows have left their maxima
  uint32_t tmem_base;
  int abort_flag;
  float m[STREAMS][M], l[STREAMS][2][M];      // FWD only, as is everything from here on (last: the other kernels do not allocate it)
  float block_max[2][STREAMS][2][M];
};

__device__ __forceinline__ float exp2_ftz(float x) {          // 2^x; results below 2^-126 are zero
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 32 dimensions of a row, scaled -> A operand in tensor memory: 32 columns of TF32 values and, at `t16`, 16 of bf16 pairs of the
// high parts and 16 of the low parts (t16 = 0: [bf16(hi) x32 | bf16(lo) x32] rows in shared memory instead)
__device__ __forceinline__ void stage_own(uint32_t t, uint32_t t16, uint32_t smem16, const float* src, int row, bool inside, int c0, int d, float scale) {
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = 0.f;
  if (inside) {
    if (c0 + 32 <= d && (d & 3) == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(src + c0) + i);
        v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = c0 + i < d ? __ldg(src + c0 + i) : 0.f;
    }
  }
  uint32_t hi[32], w[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float h0, l0, h1, l1;
    split_tf32(v[2 * i] * scale, h0, l0);
    split_tf32(v[2 * i + 1] * scale, h1, l1);
    hi[2 * i] = __float_as_uint(h0); hi[2 * i + 1] = __float_as_uint(h1);
    w[i] = pack_bf16x2(h0, h1); w[16 + i] = pack_bf16x2(l0, l1);
  }
  tmem_st32(t, hi);
  if (t16) {
    tmem_st32(t16, w);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) sts_b32x4(smem16 + sw128_offset_bf16(row, 8 * i), w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
  tmem_wait_st();
}

// 32 values of a row -> T in tensor memory: 32 columns of TF32 values at t, 16 of bf16 pairs of the high and 16 of the low parts at t16
__device__ __forceinline__ void store_t(uint32_t t, uint32_t t16, const float (&v)[32]) {
  uint32_t hi[32], w[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float h0, l0, h1, l1;
    split_tf32_fast(v[2 * i], h0, l0);
    split_tf32_fast(v[2 * i + 1], h1, l1);
    hi[2 * i] = __float_as_uint(h0); hi[2 * i + 1] = __float_as_uint(h1);
    w[i] = pack_bf16x2(h0, h1); w[16 + i] = pack_bf16x2(l0, l1);
  }
  tmem_st32(t, hi);
  tmem_st32(t16, w);
  tmem_wait_st();
}

template <int MODE, int DP>
constexpr int smem_bytes() {
  constexpr int CH = DP / 32, PAIR = MODE == DQ || MODE == DK;
  return PAIR * M * 128 * CH + STAGES * (PAIR + 2) * (int)IMG_CHUNK * CH + (MODE == FWD ? (int)sizeof(Ctrl) : (int)offsetof(Ctrl, m)) + 1024 + 64;
}

template <int MODE, int DP>
__device__ __forceinline__ void attention_tile(const Args& a) {
  constexpr bool PAIR = MODE == DQ || MODE == DK;               // needs dP
  constexpr bool OWN_Q = MODE == FWD || MODE == DQ;             // rows are queries
  constexpr int CH = DP / 32;
  constexpr uint32_t COL_BYTES = IMG_CHUNK * CH, C_STAGE = (PAIR ? 2u : 1u) * COL_BYTES;
  // tensor memory: per stream 128 columns [S | dP], overwritten by T; accumulators; own rows
  constexpr uint32_t ACC = 256, OWN2 = 320, OWN1 = 384;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), own2s = (raw + 1023u) & ~1023u, cols = own2s + (PAIR ? M * 128u * CH : 0u);
  const uint32_t colb = cols + STAGES * C_STAGE;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (colb - raw) + STAGES * COL_BYTES);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * M;
  const long long batch = blockIdx.y;
  if (row0 >= a.rows) return;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctrl->c_full[s]), 1);
      mbar_init(smem_u32(&ctrl->c_empty[s]), 1);
      mbar_init(smem_u32(&ctrl->b_full[s]), 1);
      mbar_init(smem_u32(&ctrl->b_empty[s]), 1);
      mbar_init(smem_u32(&ctrl->s_full[s]), 1);
      mbar_init(smem_u32(&ctrl->t_full[s]), STREAM_WARPS);
      mbar_init(smem_u32(&ctrl->t_done[s]), 1);
      for (int q = 0; q < 4; ++q) mbar_init(smem_u32(&ctrl->max_full[s][q]), 2);
    }
    mbar_init(smem_u32(&ctrl->last), 1);
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  const int quad_row = (warp & 3) * 32 + lane;                  // a warp reaches the 32 lanes of its quarter
  const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
  if (warp < 16) {                                              // one 32-dimension piece of the own rows for each four warps
    const int piece = warp >> 2, c = piece % CH;
    const bool inside = row0 + quad_row < a.rows;
    const long long at = (batch * a.rows + row0 + quad_row) * a.d;
    const uint32_t t1 = tmem + lane_base + OWN1 + (uint32_t)c * 64u;
    if (piece < CH) stage_own(t1, t1 + 32u, 0, a.own1 + at, quad_row, inside, c * 32, a.d, OWN_Q ? a.scale2 : 1.f);
    else if (PAIR && piece < 2 * CH)
      stage_own(tmem + lane_base + OWN2 + (uint32_t)c * 32u, 0, own2s + (uint32_t)c * (M * 128u), a.own2 + at, quad_row, inside, c * 32, a.d, 1.f);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // blocks this tile needs: causal hides keys beyond the query
  const int b_begin = a.causal && !OWN_Q ? row0 / BC : 0;
  const int b_end = a.causal && OWN_Q ? min(a.blocks, (row0 + M - 1) / BC + 1) : a.blocks;
  const int nb = max(0, b_end - b_begin);

  if (warp == MMA_WARP) {
    const bool leader = elect_one();
    constexpr uint32_t id_s = make_idesc_tf32(M, BC), id_s16 = make_idesc_bf16(M, BC);
    constexpr uint32_t id_t = make_idesc_tf32(M, DP) | (1u << 16), id_t16 = make_idesc_bf16(M, DP) | (1u << 16);
    const uint64_t a2 = make_kmajor_sw128_desc(own2s), b1 = make_kmajor_sw128_desc(cols);
    const uint64_t bt = tcdw::make_mn_desc(colb, IMG_CHUNK), bt16 = tcdw::make_mn_desc16(colb + BC * 128u, IMG_CHUNK);
    bool alive = true;
    for (int i = 0; i <= nb && alive; ++i) {
      if (i < nb) {                                             // S (and dP) of block i
        const uint32_t st = (uint32_t)i & 1u, parity = (uint32_t)(i >> 1) & 1u;
        if (i >= 2 && !warp_wait(smem_u32(&ctrl->t_done[st]), parity ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
        if (!warp_wait(smem_u32(&ctrl->c_full[st]), parity, abort_flag, a.status, STATUS_TIMEOUT_FULL)) break;
        tc_fence_after();
        if (leader) {
          const uint32_t d = tmem + st * 128u;
#pragma unroll
          for (int c = 0; c < CH; ++c) {
            const uint32_t ta = tmem + OWN1 + c * 64;
            const uint64_t bh = b1 + st * (C_STAGE >> 4) + c * (IMG_CHUNK / 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_tf32_ts(d, ta + 8 * k, bh + 2 * k, id_s, (uint32_t)((c | k) != 0));
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_bf16_ts(d, ta + 32 + 8 * k, bh + BC * 128 / 16 + 2 * k, id_s16, 1);
          }
          if (PAIR) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
              const uint64_t bh = b1 + st * (C_STAGE >> 4) + (COL_BYTES >> 4) + c * (IMG_CHUNK / 16);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_tf32_ts(d + 64, tmem + OWN2 + c * 32 + 8 * k, bh + 2 * k, id_s, (uint32_t)((c | k) != 0));
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_bf16(d + 64, a2 + c * (M * 128 / 16) + 2 * k, bh + BC * 128 / 16 + 2 * k, id_s16, 1);
            }
          }
          umma_commit(smem_u32(&ctrl->s_full[st]));
          umma_commit(smem_u32(&ctrl->c_empty[st]));
        }
      }
      if (i > 0) {                                              // T * colB of block i - 1
        const int j = i - 1;
        const uint32_t st = (uint32_t)j & 1u, parity = (uint32_t)(j >> 1) & 1u;
        if (!warp_wait(smem_u32(&ctrl->b_full[st]), parity, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        if (!warp_wait(smem_u32(&ctrl->t_full[st]), parity, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        tc_fence_after();
        if (leader) {
          const uint32_t t = tmem + st * 128u, d = tmem + ACC + (MODE == FWD ? st * (uint32_t)DP : 0u);
          const uint32_t first = MODE == FWD ? (uint32_t)(j >= 2) : (uint32_t)(j > 0);
          const uint64_t bh = bt + st * (COL_BYTES >> 4), b_h16 = bt16 + st * (COL_BYTES >> 4), b_l16 = b_h16 + (BC * 64 >> 4);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_tf32_ts(d, t + 8 * k, bh + 64 * k, id_t, k == 0 ? first : 1u);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, t + 64 + 32 * (k >> 1) + 8 * (k & 1), b_l16 + 64 * k, id_t16, 1);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, t + 80 + 32 * (k >> 1) + 8 * (k & 1), b_h16 + 64 * k, id_t16, 1);
          umma_commit(smem_u32(&ctrl->t_done[st]));
          umma_commit(smem_u32(&ctrl->b_empty[st]));
        }
      }
    }
    if (leader) umma_commit(smem_u32(&ctrl->last));
  } else if (warp == LOAD_WARP) {
    if (lane == 0) {
      asm volatile("griddepcontrol.wait;" ::: "memory");        // the images come from the kernel ahead
      const long long first = batch * a.blocks + b_begin;
      int issued_c = 0, issued_b = 0;
      bool alive = true;
      for (int i = 0; i < nb && alive; ++i) {
        const uint32_t slot = (uint32_t)i & 1u, parity = (uint32_t)(i >> 1) & 1u;
        if (!(alive = mbar_wait(smem_u32(&ctrl->c_empty[slot]), parity ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY))) break;
        mbar_expect_tx(smem_u32(&ctrl->c_full[slot]), C_STAGE);
        bulk_g2s(cols + slot * C_STAGE, a.col1 + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->c_full[slot]));
        if (PAIR) bulk_g2s(cols + slot * C_STAGE + COL_BYTES, a.col2 + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->c_full[slot]));
        ++issued_c;
        if (!(alive = mbar_wait(smem_u32(&ctrl->b_empty[slot]), parity ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY))) break;
        mbar_expect_tx(smem_u32(&ctrl->b_full[slot]), COL_BYTES);
        bulk_g2s(colb + slot * COL_BYTES, a.colb + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->b_full[slot]));
        ++issued_b;
      }
      // after an abort nobody consumes the stages: wait (bounded) for the copies still in flight
      if (!alive)
        for (int k = 0; k < 2; ++k) {
          const int n = k ? issued_b : issued_c;
          for (int j = max(0, n - STAGES); j < n; ++j)
            mbar_wait(smem_u32(k ? &ctrl->b_full[j % STAGES] : &ctrl->c_full[j % STAGES]), (uint32_t)(j / STAGES) & 1u, nullptr, a.status, STATUS_TIMEOUT_FULL);
        }
    }
  } else {
    // ------------------------------ element-wise streams ------------------------------
    const int stream = warp >> 3, half = warp >> 2 & 1, row = quad_row, own = row0 + row;
    const uint32_t t = tmem + (uint32_t)stream * 128u + (uint32_t)half * 32u + lane_base;
    float m = -INFINITY, l = 0.f, lse2 = INFINITY, delta = 0.f;
    if (MODE != FWD) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (MODE == DQ && own < a.rows) { lse2 = a.lse2[batch * a.q_pad + own]; delta = a.delta[batch * a.q_pad + own]; }
    int done = 0;                                               // blocks of this stream whose product has been waited for
    for (int i = stream, n = 0; i < nb; i += 2, ++n) {
      const int c0 = (b_begin + i) * BC + half * 32;            // first column of this warp
      if (!warp_wait(smem_u32(&ctrl->s_full[stream]), (uint32_t)n & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
      float v[32];
      tmem_ld32(t, v);
      // columns that exist and are visible to this row: [lo, hi)
      int lo = 0, hi = a.cols - c0;
      if (a.causal) {
        if (OWN_Q) hi = min(hi, own - c0 + 1);
        else lo = own - c0;
      }
      const bool all = __all_sync(0xffffffffu, lo <= 0 && hi >= 32);
      if (MODE == FWD) {
        if (!all) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = j < hi ? v[j] : -INFINITY;
        }
        float x0 = v[0], x1 = v[1];
#pragma unroll
        for (int j = 2; j < 32; j += 2) { x0 = fmaxf(x0, v[j]); x1 = fmaxf(x1, v[j + 1]); }
        // the maximum of the other 32 columns of the block
        float(&shared_max)[2][M] = ctrl->block_max[n & 1][stream];
        const uint32_t bar = smem_u32(&ctrl->max_full[stream][warp & 3]);
        x0 = fmaxf(x0, x1);
        shared_max[half][row] = x0;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
        if (!warp_wait(bar, (uint32_t)n & 1u, abort_flag, a.status, STATUS_TIMEOUT_FULL)) break;
        const float bm = fmaxf(x0, *(volatile float*)&shared_max[half ^ 1][row]);
        // the maximum moves, and the accumulator is rescaled, only when it has to
        if (__any_sync(0xffffffffu, bm > m + 8.f)) {
          const float m_new = fmaxf(m, bm), alpha = m == -INFINITY ? 0.f : exp2_ftz(m - m_new);
          if (n > 0) {
            if (done < n) {
              if (!warp_wait(smem_u32(&ctrl->t_done[stream]), (uint32_t)(n - 1) & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
              tc_fence_after();
              done = n;
            }
            if (half * 32 < DP) {                               // 32 columns of the accumulator each
              const uint32_t o = tmem + ACC + (uint32_t)(stream * DP + half * 32) + lane_base;
#pragma unroll
              for (int c = 0; c < 32; c += 16) {
                float x[16];
                uint32_t y[16];
                tmem_ld16(o + (uint32_t)c, x);
#pragma unroll
                for (int j = 0; j < 16; ++j) y[j] = __float_as_uint(x[j] * alpha);
                tmem_st16(o + (uint32_t)c, y);
              }
              tmem_wait_st();
            }
          }
          m = m_new;
          l *= alpha;
        }
        const float mm = m == -INFINITY ? 0.f : m;
        float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          v[j] = exp2_ftz(v[j] - mm);
          v[j + 1] = exp2_ftz(v[j + 1] - mm);
          sum0 += v[j]; sum1 += v[j + 1];
        }
        l += sum0 + sum1;
      } else {
        const float4* lse4 = reinterpret_cast<const float4*>(a.lse2 + batch * a.q_pad + c0);
        const float4* del4 = reinterpret_cast<const float4*>(a.delta + batch * a.q_pad + c0);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          float ls[4] = {lse2, lse2, lse2, lse2};
          if (!OWN_Q) {                                         // per column: the same address for the whole warp
            const float4 f = __ldg(lse4 + j / 4);
            ls[0] = f.x; ls[1] = f.y; ls[2] = f.z; ls[3] = f.w;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) v[j + k] = exp2_ftz(v[j + k] - ls[k]);      // 0 where the query has no key (ls = +inf)
        }
        if (!all) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = j >= lo && j < hi ? v[j] : 0.f;
        }
        if (PAIR) {                                             // the score scale follows with the result
          float dp[32];
          tmem_ld32(t + 64, dp);
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            float de[4] = {delta, delta, delta, delta};
            if (!OWN_Q) {
              const float4 e = __ldg(del4 + j / 4);
              de[0] = e.x; de[1] = e.y; de[2] = e.z; de[3] = e.w;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) v[j + k] *= dp[j + k] - de[k];
          }
        }
      }
      store_t(t, t + 64u, v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->t_full[stream]));
    }
    // ------------------------------ results ------------------------------
    if (MODE == FWD) {
      if (half == 0) ctrl->m[stream][row] = m;
      ctrl->l[stream][half][row] = l;
    }
    const bool complete = warp_wait(smem_u32(&ctrl->last), 0, abort_flag, a.status, STATUS_TIMEOUT_ACCUM);
    asm volatile("bar.sync 1, 512;" ::: "memory");              // every stream warp, also after an abort
    const int c = (warp >> 2) * 16;                             // 16 columns for each four warps
    if (complete && c < DP) {
      tc_fence_after();
      float w0 = PAIR ? a.scale : 1.f, w1 = 0.f;
      if (MODE == FWD) {
        const float m0 = ctrl->m[0][row], m1 = ctrl->m[1][row], mx = fmaxf(m0, m1);
        const float a0 = m0 == -INFINITY ? 0.f : exp2_ftz(m0 - mx), a1 = m1 == -INFINITY ? 0.f : exp2_ftz(m1 - mx);
        const float sum = (ctrl->l[0][0][row] + ctrl->l[0][1][row]) * a0 + (ctrl->l[1][0][row] + ctrl->l[1][1][row]) * a1;
        const bool dead = !(sum > 0.f);
        w0 = dead ? 0.f : a0 / sum;
        w1 = dead ? 0.f : a1 / sum;
        if (c == 0 && own < a.rows) a.lse[batch * a.rows + own] = dead ? -INFINITY : mx * 0.6931471805599453f + logf(sum);
      }
      float x[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = 0.f;
      if (nb > 0) {
        tmem_ld16(tmem + ACC + (uint32_t)c + lane_base, x);
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = w0 == 0.f ? 0.f : x[j] * w0;
        if (MODE == FWD && nb > 1) {
          float y[16];
          tmem_ld16(tmem + ACC + (uint32_t)(DP + c) + lane_base, y);
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = w1 == 0.f ? x[j] : fmaf(y[j], w1, x[j]);
        }
      }
      if (own < a.rows) {
        float* dst = a.out + (batch * a.rows + own) * a.d + c;
        if (c + 16 <= a.d && (a.d & 3) == 0) {
#pragma unroll
          for (int j = 0; j < 4; ++j) reinterpret_cast<float4*>(dst)[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c + j < a.d) dst[j] = x[j];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int DP>
__global__ void __launch_bounds__(THREADS, 1) attention_forward_kernel(const Args a) { attention_tile<FWD, DP>(a); }

struct BackwardArgs { Args dk, dq, dv; };
// The three gradients in one launch, the two with more work first: the CTAs of one fill the last wave of the other.
template <int DP>
__global__ void __launch_bounds__(THREADS, 1) attention_backward_kernel(const __grid_constant__ BackwardArgs a) {
  if (blockIdx.z == 0) attention_tile<DK, DP>(a.dk);
  else if (blockIdx.z == 1) attention_tile<DQ, DP>(a.dq);
  else attention_tile<DV, DP>(a.dv);
}

// ---- column images, log-sum-exp and delta ------------------------------------------------------------------------------
struct StageTask {
  const float* src;            // [batch][tokens][d]
  unsigned char *kmajor, *mn;  // images to write (null: not wanted), [batch][blocks][chunks]
  int tokens, blocks;
  float scale;                 // of the K-major image
};
struct StageArgs {
  StageTask task[4];
  const float *grad, *out, *lse;   // backward: delta = rowsum(grad * out) and lse in base 2, per query of task 0's blocks
  float *lse2, *delta;
  int tasks, d, q_pad;
};
// One CTA per (block of 64 tokens, batch, task); four values per thread and step.
template <int DP>
__global__ void __launch_bounds__(256) stage_kernel(const StageArgs a) {
  wait_previous();
  asm volatile("griddepcontrol.launch_dependents;");
  const StageTask& t = a.task[blockIdx.z];
  const int blk = blockIdx.x;
  if (blk >= t.blocks) return;
  const long long batch = blockIdx.y, image = (batch * t.blocks + blk) * (long long)(IMG_CHUNK * (DP / 32));
  for (int i = threadIdx.x; i < BC * (DP / 4); i += 256) {
    const int r = i / (DP / 4), c = i % (DP / 4) * 4, token = blk * BC + r;
    float v[4] = {0.f, 0.f, 0.f, 0.f}, h[4], l[4];
    if (token < t.tokens) {
      const float* p = t.src + (batch * t.tokens + token) * a.d + c;
      if (c + 3 < a.d && (a.d & 3) == 0) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < a.d) v[j] = __ldg(p + j);
      }
    }
    const int k = c & 31;
    const long long chunk = image + (long long)(c >> 5) * IMG_CHUNK;
    if (t.kmajor) {            // second plane [bf16(lo) | bf16(hi)], pairing with the rows' [hi | lo]
      unsigned char* p = t.kmajor + chunk;
#pragma unroll
      for (int j = 0; j < 4; ++j) split_tf32(v[j] * t.scale, h[j], l[j]);
      *reinterpret_cast<float4*>(p + sw128_offset(r, k)) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint2*>(p + BC * 128 + sw128_offset_bf16(r, k)) = make_uint2(pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
      *reinterpret_cast<uint2*>(p + BC * 128 + sw128_offset_bf16(r, 32 + k)) = make_uint2(pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
    }
    if (t.mn) {                // token-major planes: TF32, bf16(hi), bf16(lo)
      unsigned char* p = t.mn + chunk;
#pragma unroll
      for (int j = 0; j < 4; ++j) split_tf32(v[j], h[j], l[j]);
      *reinterpret_cast<float4*>(p + tcdw::sw32b_offset(r, k)) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint2*>(p + BC * 128 + tcdw::sw64_offset(r, k)) = make_uint2(pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
      *reinterpret_cast<uint2*>(p + BC * 192 + tcdw::sw64_offset(r, k)) = make_uint2(pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
    }
  }
  if (a.lse2 && blockIdx.z == 0) {
    const int r = threadIdx.x >> 2, part = threadIdx.x & 3, token = blk * BC + r;
    float sum = 0.f;
    if (token < t.tokens) {
      const float *g = a.grad + (batch * t.tokens + token) * a.d, *o = a.out + (batch * t.tokens + token) * a.d;
      for (int c = part; c < a.d; c += 4) sum = fmaf(__ldg(g + c), __ldg(o + c), sum);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (part == 0) {
      const float ls = token < t.tokens ? __ldg(a.lse + batch * t.tokens + token) : -INFINITY;
      a.lse2[batch * a.q_pad + token] = ls > -INFINITY ? ls * LOG2E : INFINITY;
      a.delta[batch * a.q_pad + token] = sum;
    }
  }
}

static size_t image_bytes(int64_t batch, int64_t tokens, int64_t d) {
  return (size_t)batch * (size_t)((tokens + BC - 1) / BC) * IMG_CHUNK * (size_t)((d + 31) / 32);
}

bool supported(int64_t batch, int64_t tq, int64_t tk, int64_t d, int64_t dv) {
  // two heads' worth of dimensions and more do not fit shared memory beside two operand tiles; tiny problems are left to the composed form
  return d == dv && d >= 16 && d <= 64 && batch <= 65535 && tq >= 32 && tk >= 32 && tq < (1 << 24) && tk < (1 << 24);
}
bool aligned(std::initializer_list<const void*> pointers) {   // rows are read and written in 16-byte pieces
  for (const void* p : pointers)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}
size_t workspace(int64_t batch, int64_t tq, int64_t tk, int64_t d, bool backward) {
  if (!backward) return 2 * image_bytes(batch, tk, d);
  const size_t q_pad = (size_t)((tq + BC - 1) / BC * BC);
  return 4 * image_bytes(batch, tq, d) + 3 * image_bytes(batch, tk, d) + 2 * (size_t)batch * q_pad * sizeof(float);
}

template <typename Kernel, typename A>
static int launch(Kernel kernel, std::once_flag& once, cudaError_t& opt_in, dim3 grid, int smem, const A& args, cudaStream_t st) {
  std::call_once(once, [&] { opt_in = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  B200_CUDA(opt_in);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = (size_t)smem; cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;   // the own rows are staged while the images are made
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, args));
  count_launch();
  return launch_check("attention kernel");
}

template <int DP>
static int forward_dp(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* q, const float* k, const float* v, int causal, float scale,
                      float* out, float* lse, unsigned char* ws, cudaStream_t st) {
  const int kb = (int)((tk + BC - 1) / BC);
  StageArgs s{};
  s.d = (int)d; s.tasks = 2;
  s.task[0] = StageTask{k, ws, nullptr, (int)tk, kb, 1.f};
  s.task[1] = StageTask{v, nullptr, ws + image_bytes(batch, tk, d), (int)tk, kb, 1.f};
  launch_next(stage_kernel<DP>, dim3((unsigned)kb, (unsigned)batch, 2), 256, 0, st, s);
  count_launch();
  if (int rc = launch_check("stage_kernel")) return rc;
  Args a{};
  a.own1 = q; a.col1 = s.task[0].kmajor; a.colb = s.task[1].mn; a.out = out; a.lse = lse;
  a.rows = (int)tq; a.cols = (int)tk; a.d = (int)d; a.blocks = kb;
  a.causal = causal; a.scale = scale; a.scale2 = scale * LOG2E;
  a.status = device_status_word();
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  return launch(attention_forward_kernel<DP>, once, opt_in, dim3((unsigned)((tq + M - 1) / M), (unsigned)batch), smem_bytes<FWD, DP>(), a, st);
}

template <int DP>
static int backward_dp(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* grad, const float* q, const float* k, const float* v,
                       const float* out, const float* lse, int causal, float scale, float* dq, float* dk, float* dv, unsigned char* ws,
                       cudaStream_t st) {
  const int kb = (int)((tk + BC - 1) / BC), qb = (int)((tq + BC - 1) / BC);
  const size_t iq = image_bytes(batch, tq, d), ik = image_bytes(batch, tk, d);
  unsigned char *g_k = ws, *g_mn = g_k + iq, *q_k = g_mn + iq, *q_mn = q_k + iq, *k_k = q_mn + iq, *k_mn = k_k + ik, *v_k = k_mn + ik;
  StageArgs s{};
  s.d = (int)d; s.tasks = 4; s.q_pad = qb * BC;
  s.lse2 = reinterpret_cast<float*>(v_k + ik);
  s.delta = s.lse2 + batch * s.q_pad;
  s.grad = grad; s.out = out; s.lse = lse;
  s.task[0] = StageTask{grad, g_k, g_mn, (int)tq, qb, 1.f};
  s.task[1] = StageTask{q, q_k, q_mn, (int)tq, qb, scale * LOG2E};
  s.task[2] = StageTask{k, k_k, k_mn, (int)tk, kb, 1.f};
  s.task[3] = StageTask{v, v_k, nullptr, (int)tk, kb, 1.f};
  launch_next(stage_kernel<DP>, dim3((unsigned)std::max(kb, qb), (unsigned)batch, 4), 256, 0, st, s);
  count_launch();
  if (int rc = launch_check("stage_kernel")) return rc;
  Args a{};
  a.d = (int)d; a.q_pad = s.q_pad; a.lse2 = s.lse2; a.delta = s.delta;
  a.causal = causal; a.scale = scale; a.scale2 = scale * LOG2E;
  a.status = device_status_word();
  BackwardArgs b{a, a, a};
  b.dk.own1 = k; b.dk.own2 = v; b.dk.col1 = q_k; b.dk.col2 = g_k; b.dk.colb = q_mn; b.dk.out = dk;     // dS^T Q
  b.dk.rows = (int)tk; b.dk.cols = (int)tq; b.dk.blocks = qb;
  b.dq.own1 = q; b.dq.own2 = grad; b.dq.col1 = k_k; b.dq.col2 = v_k; b.dq.colb = k_mn; b.dq.out = dq;  // dS K
  b.dq.rows = (int)tq; b.dq.cols = (int)tk; b.dq.blocks = kb;
  b.dv.own1 = k; b.dv.col1 = q_k; b.dv.colb = g_mn; b.dv.out = dv;                                     // P^T dO
  b.dv.rows = (int)tk; b.dv.cols = (int)tq; b.dv.blocks = qb;
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  const dim3 grid((unsigned)((std::max(tq, tk) + M - 1) / M), (unsigned)batch, 3);
  return launch(attention_backward_kernel<DP>, once, opt_in, grid, smem_bytes<DK, DP>(), b, st);
}

int forward(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* q, const float* k, const float* v, int causal, float scale, float* out,
            float* lse, void* ws, cudaStream_t st) {
  return d <= 32 ? forward_dp<32>(batch, tq, tk, d, q, k, v, causal, scale, out, lse, (unsigned char*)ws, st)
                 : forward_dp<64>(batch, tq, tk, d, q, k, v, causal, scale, out, lse, (unsigned char*)ws, st);
}
int backward(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* grad, const float* q, const float* k, const float* v, const float* out,
             const float* lse, int causal, float scale, float* dq, float* dk, float* dv, void* ws, cudaStream_t st) {
  return d <= 32 ? backward_dp<32>(batch, tq, tk, d, grad, q, k, v, out, lse, causal, scale, dq, dk, dv, (unsigned char*)ws, st)
                 : backward_dp<64>(batch, tq, tk, d, grad, q, k, v, out, lse, causal, scale, dq, dk, dv, (unsigned char*)ws, st);
}

}  // namespace fa
}  // namespace b200

// Fused scaled dot-product attention on tcgen05, forward and backward, for calls without mask and dropout and heads of up to
// 64 dimensions: the scores never reach memory.  FP32 by the split-precision scheme of tc_common.cuh.
//
// What bounds it and what follows from that.  The composed form (attention.cu) writes, rewrites and reads the [tokens,
// tokens] matrix: 144 us forward and 265 us backward for 16 heads of 1024 tokens x 64, of which 60 us are products.  Here a CTA owns 128
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
// so each gradient has one writer and needs no atomics (eight products instead of five).  Two streams of four warps (a thread
// = a row) take alternate blocks, so that the element-wise work of one runs under the products of the other; in the forward
// pass each stream keeps its own maximum, sum and accumulator, merged at the end, and rescales its accumulator only when the maximum
// has grown by more than 8 (a factor 256 of head room in FP32).  The column operands are split once per call into ready-made
// shared-memory images by stage_kernel, which also prepares log-sum-exp and delta; one thread fetches them with bulk copies.
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
constexpr int STREAM_WARPS = 4, LOAD_WARP = 8, MMA_WARP = 9, THREADS = 320;
constexpr uint32_t IMG_CHUNK = BC * 256u;     // one block x 32 dimensions of an image: 16 KB in either orientation
constexpr int SMEM_MAX = 232448;
constexpr float LOG2E = 1.4426950408889634f;
enum { FWD = 0, DQ = 1, DV = 2, DK = 3 };

struct Args {
  const float *own1, *own2;                   // raw rows [batch][rows][d]
  const unsigned char *col1, *col2, *colb;    // images [batch][blocks][chunks] of the other side
  const float *lse2, *delta;                  // [batch][padded queries]: log-sum-exp in base 2 (+inf: no key), rowsum(dO O)
  float* out;                                 // [batch][rows][d]
  float* lse;                                 // FWD: [batch][rows]
  int rows, cols, d, blocks, q_pad;
  int causal, stages;
  float scale, scale2;                        // score scale; the same times log2(e)
  int* status;
};

struct Ctrl {
  unsigned long long c_full[2], c_empty[2], b_full[2], b_empty[2], s_full[2], t_full[2], t_done[2], last;
  uint32_t tmem_base;
  int abort_flag;
  float m[2][M], l[2][M];                     // FWD only (last: the other kernels do not allocate it)
};

// raw rows -> K-major A operand in shared memory: per 32 dimensions a TF32 plane and a plane of [bf16(hi) x32 | bf16(lo) x32] rows
template <int DP>
__device__ __forceinline__ void stage_own(uint32_t dst, const float* src, int row0, int rows, int d, int tid, int threads) {
  for (int i = tid; i < M * (DP / 4); i += threads) {
    const int r = i / (DP / 4), c = i % (DP / 4) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f}, h[4], l[4];
    if (row0 + r < rows) {
      const float* p = src + (long long)(row0 + r) * d + c;
      if (c + 3 < d && (d & 3) == 0) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c + j < d) v[j] = __ldg(p + j);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) split_tf32(v[j], h[j], l[j]);
    const uint32_t plane = dst + (uint32_t)(c >> 5) * (M * 256u);
    const int k = c & 31;
    sts_f32x4(plane + sw128_offset(r, k), h[0], h[1], h[2], h[3]);
    sts_b32x2(plane + M * 128u + sw128_offset_bf16(r, k), pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
    sts_b32x2(plane + M * 128u + sw128_offset_bf16(r, 32 + k), pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
  }
}

// 64 values of a row -> T in tensor memory: 64 columns of TF32 values, 32 of bf16 pairs of the high parts, 32 of the low parts
__device__ __forceinline__ void store_t(uint32_t t, const float (&v)[64]) {
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint32_t hi[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float h, l;
      split_tf32_fast(v[half * 32 + i], h, l);
      hi[i] = __float_as_uint(h);
    }
    tmem_st32(t + half * 32, hi);
  }
#pragma unroll
  for (int part = 0; part < 2; ++part) {
    uint32_t w[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float h0, l0, h1, l1;
      split_tf32_fast(v[2 * i], h0, l0);
      split_tf32_fast(v[2 * i + 1], h1, l1);
      w[i] = part ? pack_bf16x2(l0, l1) : pack_bf16x2(h0, h1);
    }
    tmem_st32(t + 64 + part * 32, w);
  }
  tmem_wait_st();
}

template <int MODE, int DP>
__global__ void __launch_bounds__(THREADS, 1) attention_kernel(const Args a) {
  constexpr bool PAIR = MODE == DQ || MODE == DK;               // needs dP
  constexpr bool OWN_Q = MODE == FWD || MODE == DQ;             // rows are queries
  constexpr int CH = DP / 32, ACCS = MODE == FWD ? 2 : 1;
  constexpr uint32_t OWN_BYTES = M * 256u * CH, COL_BYTES = IMG_CHUNK * CH;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t own2 = base + OWN_BYTES, cols = base + (PAIR ? 2u : 1u) * OWN_BYTES;
  const uint32_t c_stage = (PAIR ? 2u : 1u) * COL_BYTES, colb = cols + (uint32_t)a.stages * c_stage;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (colb - raw) + a.stages * COL_BYTES);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row0 = blockIdx.x * M;
  const long long batch = blockIdx.y;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctrl->c_full[s]), 1);
      mbar_init(smem_u32(&ctrl->c_empty[s]), 1);
      mbar_init(smem_u32(&ctrl->b_full[s]), 1);
      mbar_init(smem_u32(&ctrl->b_empty[s]), 1);
      mbar_init(smem_u32(&ctrl->s_full[s]), 1);
      mbar_init(smem_u32(&ctrl->t_full[s]), STREAM_WARPS);
      mbar_init(smem_u32(&ctrl->t_done[s]), 1);
    }
    mbar_init(smem_u32(&ctrl->last), 1);
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
  stage_own<DP>(base, a.own1 + batch * a.rows * a.d, row0, a.rows, a.d, threadIdx.x, THREADS);
  if (PAIR) stage_own<DP>(own2, a.own2 + batch * a.rows * a.d, row0, a.rows, a.d, threadIdx.x, THREADS);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  const uint32_t acc = tmem + 256;                              // streams: 2 x 128 columns [S | dP], overwritten by T
  // blocks this tile needs: causal hides keys beyond the query
  const int b_begin = a.causal && !OWN_Q ? row0 / BC : 0;
  const int b_end = a.causal && OWN_Q ? min(a.blocks, (row0 + M - 1) / BC + 1) : a.blocks;
  const int nb = max(0, b_end - b_begin);

  if (warp == MMA_WARP) {
    const bool leader = elect_one();
    constexpr uint32_t id_s = make_idesc_tf32(M, BC), id_s16 = make_idesc_bf16(M, BC);
    constexpr uint32_t id_t = make_idesc_tf32(M, DP) | (1u << 16), id_t16 = make_idesc_bf16(M, DP) | (1u << 16);
    const uint64_t a1 = make_kmajor_sw128_desc(base), a2 = make_kmajor_sw128_desc(own2), b1 = make_kmajor_sw128_desc(cols);
    const uint64_t bt = tcdw::make_mn_desc(colb, IMG_CHUNK), bt16 = tcdw::make_mn_desc16(colb + BC * 128u, IMG_CHUNK);
    auto product = [&](uint32_t d, uint64_t da, uint64_t db) {   // 128 x 64 x DP, K-major operands
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const uint64_t ah = da + c * (M * 256 / 16), bh = db + c * (IMG_CHUNK / 16);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_tf32(d, ah + 2 * k, bh + 2 * k, id_s, (uint32_t)((c | k) != 0));
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(d, ah + M * 128 / 16 + 2 * k, bh + BC * 128 / 16 + 2 * k, id_s16, 1);
      }
    };
    bool alive = true;
    for (int i = 0; i <= nb && alive; ++i) {
      if (i < nb) {                                             // S (and dP) of block i
        const uint32_t st = (uint32_t)i & 1u, slot = a.stages == 2 ? st : 0u, round = (uint32_t)(a.stages == 2 ? i >> 1 : i);
        if (i >= 2 && !warp_wait(smem_u32(&ctrl->t_done[st]), (uint32_t)((i >> 1) - 1) & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
        if (!warp_wait(smem_u32(&ctrl->c_full[slot]), round & 1u, abort_flag, a.status, STATUS_TIMEOUT_FULL)) break;
        tc_fence_after();
        if (leader) {
          product(tmem + st * 128u, a1, b1 + slot * (c_stage >> 4));
          if (PAIR) product(tmem + st * 128u + 64u, a2, b1 + slot * (c_stage >> 4) + (COL_BYTES >> 4));
          umma_commit(smem_u32(&ctrl->s_full[st]));
          umma_commit(smem_u32(&ctrl->c_empty[slot]));
        }
      }
      if (i > 0) {                                              // T * colB of block i - 1
        const int j = i - 1;
        const uint32_t st = (uint32_t)j & 1u, slot = a.stages == 2 ? st : 0u, round = (uint32_t)(a.stages == 2 ? j >> 1 : j);
        if (!warp_wait(smem_u32(&ctrl->b_full[slot]), round & 1u, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        if (!warp_wait(smem_u32(&ctrl->t_full[st]), (uint32_t)(j >> 1) & 1u, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        tc_fence_after();
        if (leader) {
          const uint32_t t = tmem + st * 128u, d = acc + (MODE == FWD ? st * (uint32_t)DP : 0u);
          const uint32_t first = MODE == FWD ? (uint32_t)(j >= 2) : (uint32_t)(j > 0);
          const uint64_t bh = bt + slot * (COL_BYTES >> 4), b_h16 = bt16 + slot * (COL_BYTES >> 4), b_l16 = b_h16 + (BC * 64 >> 4);
#pragma unroll
          for (int k = 0; k < 8; ++k) umma_tf32_ts(d, t + 8 * k, bh + 64 * k, id_t, k == 0 ? first : 1u);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, t + 64 + 8 * k, b_l16 + 64 * k, id_t16, 1);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, t + 96 + 8 * k, b_h16 + 64 * k, id_t16, 1);
          umma_commit(smem_u32(&ctrl->t_done[st]));
          umma_commit(smem_u32(&ctrl->b_empty[slot]));
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
        const uint32_t slot = a.stages == 2 ? (uint32_t)i & 1u : 0u, round = (uint32_t)(a.stages == 2 ? i >> 1 : i);
        if (!(alive = mbar_wait(smem_u32(&ctrl->c_empty[slot]), (round & 1u) ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY))) break;
        mbar_expect_tx(smem_u32(&ctrl->c_full[slot]), c_stage);
        bulk_g2s(cols + slot * c_stage, a.col1 + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->c_full[slot]));
        if (PAIR) bulk_g2s(cols + slot * c_stage + COL_BYTES, a.col2 + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->c_full[slot]));
        ++issued_c;
        if (!(alive = mbar_wait(smem_u32(&ctrl->b_empty[slot]), (round & 1u) ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY))) break;
        mbar_expect_tx(smem_u32(&ctrl->b_full[slot]), COL_BYTES);
        bulk_g2s(colb + slot * COL_BYTES, a.colb + (first + i) * COL_BYTES, COL_BYTES, smem_u32(&ctrl->b_full[slot]));
        ++issued_b;
      }
      // after an abort nobody consumes the stages: wait (bounded) for the copies still in flight
      if (!alive)
        for (int k = 0; k < 2; ++k) {
          const int n = k ? issued_b : issued_c;
          for (int j = max(0, n - a.stages); j < n; ++j)
            mbar_wait(smem_u32(k ? &ctrl->b_full[j % a.stages] : &ctrl->c_full[j % a.stages]), (uint32_t)(j / a.stages) & 1u, nullptr, a.status, STATUS_TIMEOUT_FULL);
        }
    }
  } else {
    // ------------------------------ element-wise streams ------------------------------
    const int stream = warp >> 2, row = (warp & 3) * 32 + lane, own = row0 + row;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t t = tmem + (uint32_t)stream * 128u + lane_base, o = acc + (MODE == FWD ? (uint32_t)(stream * DP) : 0u) + lane_base;
    float m = -INFINITY, l = 0.f, lse2 = INFINITY, delta = 0.f;
    if (MODE == DQ) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (own < a.rows) { lse2 = a.lse2[batch * a.q_pad + own]; delta = a.delta[batch * a.q_pad + own]; }
    }
    if (MODE == DV || MODE == DK) asm volatile("griddepcontrol.wait;" ::: "memory");
    bool alive = true;
    int done = 0;                                               // blocks of this stream whose product has been waited for
    for (int i = stream, n = 0; i < nb && alive; i += 2, ++n) {
      const int c0 = (b_begin + i) * BC;                        // first column of the block
      if (!warp_wait(smem_u32(&ctrl->s_full[stream]), (uint32_t)n & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
      float v[64];
      {
        float h[32];
        tmem_ld32(t, h);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = h[j];
        tmem_ld32(t + 32, h);
#pragma unroll
        for (int j = 0; j < 32; ++j) v[32 + j] = h[j];
      }
      // columns that exist and are visible to this row: [lo, hi)
      int lo = 0, hi = a.cols - c0;
      if (a.causal) {
        if (OWN_Q) hi = min(hi, own - c0 + 1);
        else lo = own - c0;
      }
      const bool all = __all_sync(0xffffffffu, lo <= 0 && hi >= BC);
      if (MODE == FWD) {
        float bm = -INFINITY;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          v[j] = all || j < hi ? v[j] * a.scale2 : -INFINITY;
          bm = fmaxf(bm, v[j]);
        }
        // the maximum moves, and the accumulator is rescaled, only when it has to
        if (__any_sync(0xffffffffu, bm > m + 8.f)) {
          const float m_new = fmaxf(m, bm), alpha = m == -INFINITY ? 0.f : exp2f(m - m_new);
          if (n > 0) {
            if (done < n) {
              if (!warp_wait(smem_u32(&ctrl->t_done[stream]), (uint32_t)(n - 1) & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
              tc_fence_after();
              done = n;
            }
#pragma unroll 1
            for (int c = 0; c < DP; c += 32) {
              float x[32];
              uint32_t y[32];
              tmem_ld32(o + (uint32_t)c, x);
#pragma unroll
              for (int j = 0; j < 32; ++j) y[j] = __float_as_uint(x[j] * alpha);
              tmem_st32(o + (uint32_t)c, y);
            }
            tmem_wait_st();
          }
          m = m_new;
          l *= alpha;
        }
        const float mm = m == -INFINITY ? 0.f : m;
        float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          v[j] = exp2f(v[j] - mm);
          v[j + 1] = exp2f(v[j + 1] - mm);
          sum0 += v[j]; sum1 += v[j + 1];
        }
        l += sum0 + sum1;
      } else {
        float dp[PAIR ? 64 : 1];
        if (PAIR) {
          float h[32];
          tmem_ld32(t + 64, h);
#pragma unroll
          for (int j = 0; j < 32; ++j) dp[j % (PAIR ? 64 : 1)] = h[j];
          tmem_ld32(t + 96, h);
#pragma unroll
          for (int j = 0; j < 32; ++j) dp[(32 + j) % (PAIR ? 64 : 1)] = h[j];
        }
        const float4* lse4 = reinterpret_cast<const float4*>(a.lse2 + batch * a.q_pad + c0);
        const float4* del4 = reinterpret_cast<const float4*>(a.delta + batch * a.q_pad + c0);
#pragma unroll
        for (int j = 0; j < 64; j += 4) {
          float ls[4] = {lse2, lse2, lse2, lse2}, de[4] = {delta, delta, delta, delta};
          if (!OWN_Q) {                                         // per column: the same address for the whole warp
            const float4 f = __ldg(lse4 + j / 4);
            ls[0] = f.x; ls[1] = f.y; ls[2] = f.z; ls[3] = f.w;
            if (PAIR) {
              const float4 e = __ldg(del4 + j / 4);
              de[0] = e.x; de[1] = e.y; de[2] = e.z; de[3] = e.w;
            }
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float p = exp2f(fmaf(v[j + k], a.scale2, -ls[k]));  // 0 where the query has no key (ls = +inf)
            if (!all && (j + k < lo || j + k >= hi)) p = 0.f;
            v[j + k] = PAIR ? p * (dp[(j + k) % (PAIR ? 64 : 1)] - de[k]) * a.scale : p;
          }
        }
      }
      store_t(t, v);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->t_full[stream]));
    }
    // ------------------------------ results ------------------------------
    if (MODE == FWD) { ctrl->m[stream][row] = m; ctrl->l[stream][row] = l; }
    const bool complete = warp_wait(smem_u32(&ctrl->last), 0, abort_flag, a.status, STATUS_TIMEOUT_ACCUM);
    asm volatile("bar.sync 1, 256;" ::: "memory");              // every stream warp, also after an abort
    if (complete) {
      tc_fence_after();
      float w0 = 1.f, w1 = 0.f;
      if (MODE == FWD) {
        const float m0 = ctrl->m[0][row], m1 = ctrl->m[1][row], mx = fmaxf(m0, m1);
        const float a0 = m0 == -INFINITY ? 0.f : exp2f(m0 - mx), a1 = m1 == -INFINITY ? 0.f : exp2f(m1 - mx);
        const float sum = ctrl->l[0][row] * a0 + ctrl->l[1][row] * a1;
        const bool dead = !(sum > 0.f);
        w0 = dead ? 0.f : a0 / sum;
        w1 = dead ? 0.f : a1 / sum;
        if (stream == 0 && own < a.rows) a.lse[batch * a.rows + own] = dead ? -INFINITY : mx * 0.6931471805599453f + logf(sum);
      }
      // the two streams share the columns: 32 at a time
      float* dst = a.out + (batch * a.rows + own) * a.d;
#pragma unroll 1
      for (int c = stream * 32; c < DP; c += 64) {
        float x[32];
        if (nb > 0) {
          tmem_ld32(acc + (uint32_t)c + lane_base, x);
          if (MODE == FWD) {
#pragma unroll
            for (int j = 0; j < 32; ++j) x[j] *= w0;
            if (nb > 1) {
              float y[32];
              tmem_ld32(acc + (uint32_t)(DP + c) + lane_base, y);
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = w0 + w1 == 0.f ? 0.f : fmaf(y[j], w1, x[j]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = w0 == 0.f ? 0.f : x[j];
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = 0.f;
        }
        if (own < a.rows) {
          if (c + 32 <= a.d && (a.d & 3) == 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(dst + c)[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c + j < a.d) dst[c + j] = x[j];
          }
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

// ---- column images, log-sum-exp and delta ------------------------------------------------------------------------------
struct StageTask {
  const float* src;            // [batch][tokens][d]
  unsigned char *kmajor, *mn;  // images to write (null: not wanted), [batch][blocks][chunks]
  int tokens, blocks;
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
#pragma unroll
    for (int j = 0; j < 4; ++j) split_tf32(v[j], h[j], l[j]);
    const float4 hi = make_float4(h[0], h[1], h[2], h[3]);
    const uint2 h16 = make_uint2(pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3])), l16 = make_uint2(pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
    const int k = c & 31;
    const long long chunk = image + (long long)(c >> 5) * IMG_CHUNK;
    if (t.kmajor) {            // second plane [bf16(lo) | bf16(hi)], pairing with the rows' [hi | lo]
      unsigned char* p = t.kmajor + chunk;
      *reinterpret_cast<float4*>(p + sw128_offset(r, k)) = hi;
      *reinterpret_cast<uint2*>(p + BC * 128 + sw128_offset_bf16(r, k)) = l16;
      *reinterpret_cast<uint2*>(p + BC * 128 + sw128_offset_bf16(r, 32 + k)) = h16;
    }
    if (t.mn) {                // token-major planes: TF32, bf16(hi), bf16(lo)
      unsigned char* p = t.mn + chunk;
      *reinterpret_cast<float4*>(p + tcdw::sw32b_offset(r, k)) = hi;
      *reinterpret_cast<uint2*>(p + BC * 128 + tcdw::sw64_offset(r, k)) = h16;
      *reinterpret_cast<uint2*>(p + BC * 192 + tcdw::sw64_offset(r, k)) = l16;
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

template <int MODE, int DP>
static int launch(Args a, int64_t batch, bool dependent, cudaStream_t st) {
  constexpr int CH = DP / 32, PAIR = MODE == DQ || MODE == DK ? 2 : 1;
  const int own = PAIR * M * 256 * CH, stage = (PAIR + 1) * (int)IMG_CHUNK * CH;
  const int fixed = own + (MODE == FWD ? (int)sizeof(Ctrl) : (int)offsetof(Ctrl, m)) + 1024 + 64;
  a.stages = fixed + 2 * stage <= SMEM_MAX ? 2 : 1;
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(attention_kernel<MODE, DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((a.rows + M - 1) / M), (unsigned)batch); cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = (size_t)(fixed + a.stages * stage); cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  if (dependent) { cfg.attrs = &attr; cfg.numAttrs = 1; }
  B200_CUDA(cudaLaunchKernelEx(&cfg, attention_kernel<MODE, DP>, a));
  count_launch();
  return launch_check("attention_kernel");
}

template <int DP>
static int forward_dp(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* q, const float* k, const float* v, int causal, float scale,
                      float* out, float* lse, unsigned char* ws, cudaStream_t st) {
  const int kb = (int)((tk + BC - 1) / BC);
  StageArgs s{};
  s.d = (int)d; s.tasks = 2;
  s.task[0] = StageTask{k, ws, nullptr, (int)tk, kb};
  s.task[1] = StageTask{v, nullptr, ws + image_bytes(batch, tk, d), (int)tk, kb};
  stage_kernel<DP><<<dim3((unsigned)kb, (unsigned)batch, 2), 256, 0, st>>>(s);
  count_launch();
  if (int rc = launch_check("stage_kernel")) return rc;
  Args a{};
  a.own1 = q; a.col1 = s.task[0].kmajor; a.colb = s.task[1].mn; a.out = out; a.lse = lse;
  a.rows = (int)tq; a.cols = (int)tk; a.d = (int)d; a.blocks = kb;
  a.causal = causal; a.scale = scale; a.scale2 = scale * LOG2E;
  a.status = device_status_word();
  return launch<FWD, DP>(a, batch, true, st);
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
  s.task[0] = StageTask{grad, g_k, g_mn, (int)tq, qb};
  s.task[1] = StageTask{q, q_k, q_mn, (int)tq, qb};
  s.task[2] = StageTask{k, k_k, k_mn, (int)tk, kb};
  s.task[3] = StageTask{v, v_k, nullptr, (int)tk, kb};
  stage_kernel<DP><<<dim3((unsigned)std::max(kb, qb), (unsigned)batch, 4), 256, 0, st>>>(s);
  count_launch();
  if (int rc = launch_check("stage_kernel")) return rc;
  Args a{};
  a.d = (int)d; a.q_pad = s.q_pad; a.lse2 = s.lse2; a.delta = s.delta;
  a.causal = causal; a.scale = scale; a.scale2 = scale * LOG2E;
  a.status = device_status_word();
  Args p = a;                                     // dV: keys on the rows, P^T dO
  p.own1 = k; p.col1 = q_k; p.colb = g_mn; p.out = dv; p.rows = (int)tk; p.cols = (int)tq; p.blocks = qb;
  if (int rc = launch<DV, DP>(p, batch, true, st)) return rc;
  p = a;                                          // dK: dS^T Q
  p.own1 = k; p.own2 = v; p.col1 = q_k; p.col2 = g_k; p.colb = q_mn; p.out = dk; p.rows = (int)tk; p.cols = (int)tq; p.blocks = qb;
  if (int rc = launch<DK, DP>(p, batch, false, st)) return rc;
  p = a;                                          // dQ: dS K
  p.own1 = q; p.own2 = grad; p.col1 = k_k; p.col2 = v_k; p.colb = k_mn; p.out = dq; p.rows = (int)tq; p.cols = (int)tk; p.blocks = kb;
  return launch<DQ, DP>(p, batch, false, st);
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

// Persistent tcgen05 kernel for convolution forward passes with a SHORT reduction (input channels x taps up to a few
// hundred): a network's first layer (1, 3 or 4 input channels, 3x3 or 7x7 filters).  FP32 by three TF32 products (tc_common.cuh).
//
// These layers ran in plain FP32 before, so their sums are kept close to it.  The tensor core truncates every addition to the accumulator:
// with the BF16 cross terms of the other kernels in one chain of 48 steps, a 7x7 layer of 3 channels was off by 1.1e-6 against 2.2e-7
// in FP32.  Here the cross terms are TF32 too (their operands cost the same bytes, and the producers save the packing), and beyond
// two K blocks they go to an accumulator of their own, where they lose nothing that counts; the chain of the main products then has
// 48 steps at most (SEG_KB), and the epilogue adds the pieces in FP32: 5.6e-7 for that layer, 8.7e-7 for the longest reductions (3.5e-6 in
// one chain; FP32 4.4e-7).  The time is that of one BF16 chain within 2 %, but for 7x7 filters with more than 64 output channels, whose single
// pair of accumulators makes the next tile's products wait (5 images of 179x179, 3 -> 112 channels: 44.5 us, now 56.4).
//
// What bounds these layers and what follows from it.  A 3 -> 64 channel 7x7 layer has 147 products per output: the whole
// filter fits shared memory, so every CTA splits it once and keeps it (no staging kernel, no workspace), and the tensor
// work is small enough that feeding the tensor core is the problem: 1307 us on the CUDA-core kernel, 135 us here (batch 64,
// 224x224, stride 2), of which the loads are a fifth and the tensor-memory stores with their splits a third.  The im2col rows are therefore never written to shared
// memory: a producer thread owns one output pixel (one accumulator row), gathers 32 of its reduction values straight
// into registers (coalesced across the warp's consecutive pixels, L1 serving the overlap of the windows), splits them and
// writes them to TENSOR MEMORY with tcgen05.st, from where tcgen05.mma takes its A operand.  The MMA then reads only the
// filter from shared memory (2 KB for 64 columns), so a 128x64x8 step runs at the tensor pipe's 32 clocks instead of the 64
// that reading both operands from shared memory takes.
//
// CTA roles: warps 0-3 epilogue, GROUPS groups of four producer warps (a group stages one K block of 128 pixels x 32
// reduction values at a time), one MMA warp.  A K block is loads, a conversion and a store in one warp, so four groups are faster than three although
// they leave 80 registers a thread (some spills): 3 -> 64 channels, 7x7, stride 2, 64x224x224 126 -> 118 us; where a CTA has fewer than seven K
// blocks the larger CTA starts later than it gains (8 images of 120x120, 4 -> 32 channels, 3x3, 6.5 and 7.0 us).  Tensor memory: two accumulators, or pairs of them (main, cross; one pair where they have more than 64 columns), the
// rest operand stages of 64 columns (32 high parts, 32 low parts).
//
// Replaces csrc/shaders/conv2d_tiled_body.glsl:53-86 of the reference for these geometries.
#include "common.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace b200 {
namespace tcr {
using namespace tc;

constexpr int BLOCK_M = 128, KBLK = 32, EPI_WARPS = 4;
template <int GROUPS> constexpr int MMA_WARP_OF = EPI_WARPS + 4 * GROUPS;
template <int GROUPS> constexpr int THREADS_OF = (MMA_WARP_OF<GROUPS> + 1) * 32;
constexpr int MAX_STAGES = 6, MAX_RUNS = 1024;
constexpr int FOUR_GROUPS_FROM = 7;   // K blocks of a CTA
constexpr int SEG_KB = 12;      // K blocks (of four main steps) per accumulation chain
constexpr int SMEM_LIMIT = 232448 - 2048;
constexpr uint32_t STAGE_COLS = 64;

struct RowsArgs {
  ConvGeom g;
  View4 x, w;            // w: [cout][cin][kh][kw] (any strides)
  const float* bias;
  long long bias_stride;
  float* out;            // contiguous NCHW
  // The window of a pixel is `runs` runs of `run_len` values `run_step` elements apart (unit step where memory allows: the taps
  // of a filter row in NCHW, the taps x channels of a row in channels-last), each padded to LP reduction indices.
  int runs, run_len, nkb;
  int segs, seg_kb;      // accumulation chains of a tile, K blocks of one
  long long run_step;
  int channels_last;     // a run holds (kx, ci) rather than kx
  int bn, acc_cols, ntn; // columns per tile (multiple of 16), accumulator pitch in tensor memory, column tiles of a CTA
  int bufs;              // accumulators, or pairs of them
  int nt_split;          // CTAs that share a pixel tile, each with its own `ntn` column tiles (a filter too large for one CTA)
  int stages, tiles_m;
  uint32_t m_total;      // output pixels
  FastDiv img_div, row_div, div_nkb, div_kh, div_cin, div_jobs;
  int* status;
};

struct Ctrl {
  unsigned long long full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};
struct RunEntry {
  int offset;            // elements from the pixel's window origin
  int ky;                // filter row (its bit of the row mask)
};

// PAIR: the cross terms have an accumulator of their own
template <int LP, bool UNIT, bool PAIR, int GROUPS>
__global__ void __launch_bounds__(THREADS_OF<GROUPS>, 1) conv_rows_kernel(const RowsArgs a) {
  constexpr int MMA_WARP = MMA_WARP_OF<GROUPS>, THREADS = THREADS_OF<GROUPS>;
  wait_previous();
  extern __shared__ unsigned char smem_raw[];
  const ConvGeom& g = a.g;
  const uint32_t raw = smem_u32(smem_raw), w_base = (raw + 1023u) & ~1023u;
  const uint32_t w_plane = (uint32_t)a.bn * 128u, w_block = 2u * w_plane;   // one K block of one column tile: high parts, low parts
  unsigned char* w_smem = smem_raw + (w_base - raw);
  RunEntry* tab = reinterpret_cast<RunEntry*>(w_smem + (size_t)a.ntn * a.nkb * w_block);
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(tab + a.nkb * (KBLK / LP));
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int ch0 = (int)(blockIdx.x % (unsigned)a.nt_split) * a.ntn * a.bn;   // first output channel of this CTA
  const uint32_t cta = blockIdx.x / (unsigned)a.nt_split, ctas = gridDim.x / (unsigned)a.nt_split;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 4);     // one arrival per warp of the producing group
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctrl->acc_full[s]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[s]), EPI_WARPS * 32);
    }
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
  // run r -> where it starts from the window's origin
  for (int r = threadIdx.x; r < a.nkb * (KBLK / LP); r += THREADS) {
    RunEntry e{0, 31};                           // padding runs: no pixel has row bit 31
    if (r < a.runs) {
      const int ci = a.channels_last ? 0 : (int)a.div_kh.div((uint32_t)r);
      e.ky = r - ci * g.kh;
      e.offset = (int)(ci * a.x.s1 + (long long)(e.ky * g.dh) * a.x.s2);
    }
    tab[r] = e;
  }
  // the filter, split once per CTA: per (column tile, K block) a plane of the high parts and one of the low parts
  for (int i = threadIdx.x; i < a.ntn * a.nkb * a.bn * 8; i += THREADS) {
    const int piece = i & 7, rest = i >> 3, row_all = rest % (a.ntn * a.bn), kb = rest / (a.ntn * a.bn);
    const int nt = row_all / a.bn, row = row_all - nt * a.bn;
    const int run = kb * (KBLK / LP) + piece * 4 / LP, j0 = piece * 4 % LP;
    const int ci_run = a.channels_last ? 0 : (int)a.div_kh.div((uint32_t)run), ky = run - ci_run * g.kh;
    float hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v = 0.f;
      if (ch0 + row_all < g.cout && run < a.runs && j0 + j < a.run_len) {
        const int kx = a.channels_last ? (int)a.div_cin.div((uint32_t)(j0 + j)) : j0 + j, ci = a.channels_last ? j0 + j - kx * g.cin : ci_run;
        v = __ldg(a.w.ptr + (long long)(ch0 + row_all) * a.w.s0 + ci * a.w.s1 + ky * a.w.s2 + kx * a.w.s3);
      }
      split_tf32(v, hi[j], lo[j]);
    }
    const uint32_t plane = w_base + (uint32_t)(nt * a.nkb + kb) * w_block;
    sts_f32x4(plane + sw128_offset(row, piece * 4), hi[0], hi[1], hi[2], hi[3]);
    sts_f32x4(plane + w_plane + sw128_offset(row, piece * 4), lo[0], lo[1], lo[2], lo[3]);
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  const uint32_t acc_pitch = (uint32_t)a.acc_cols * (PAIR ? 2u : 1u), a_cols = tmem_base + (uint32_t)a.bufs * acc_pitch;   // a_cols: first operand stage
  const int my_tiles = a.tiles_m > (int)cta ? (a.tiles_m - (int)cta + (int)ctas - 1) / (int)ctas : 0;
  const int jobs_per_tile = a.ntn * a.nkb;

  if (warp == MMA_WARP) {
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_tf32(BLOCK_M, a.bn);
    const uint64_t w_desc = make_kmajor_sw128_desc(w_base);
    uint32_t s = 0, par = 0, ab = 0, acc_par = 1;
    bool alive = true;
    for (int t = 0; t < my_tiles && alive; ++t) {
      for (int nt = 0; nt < a.ntn && alive; ++nt) {
        for (int seg = 0; seg < a.segs && alive; ++seg) {
          if (!warp_wait(smem_u32(&ctrl->acc_empty[ab]), acc_par, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) { alive = false; break; }
          tc_fence_after();
          const uint32_t acc = tmem_base + ab * acc_pitch, cross = PAIR ? acc + (uint32_t)a.acc_cols : acc;
          const int kb0 = seg * a.seg_kb, kb1 = min(a.nkb, kb0 + a.seg_kb);
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!warp_wait(smem_u32(&ctrl->full[s]), par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
            tc_fence_after();
            const uint32_t ta = a_cols + s * STAGE_COLS, later = (uint32_t)(kb != kb0);
            const uint64_t bh = w_desc + (uint64_t)((uint32_t)(nt * a.nkb + kb) * (w_block >> 4)), bl = bh + (w_plane >> 4);
            if (leader) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32_ts(cross, ta + 8 * kk, bl + 2 * kk, idesc, kk ? 1u : later);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32_ts(cross, ta + 32 + 8 * kk, bh + 2 * kk, idesc, 1);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32_ts(acc, ta + 8 * kk, bh + 2 * kk, idesc, kk || !PAIR ? 1u : later);
              umma_commit(smem_u32(&ctrl->empty[s]));
            }
            if (++s == (uint32_t)a.stages) { s = 0; par ^= 1; }
          }
          if (alive && leader) umma_commit(smem_u32(&ctrl->acc_full[ab]));
          if (++ab == (uint32_t)a.bufs) { ab = 0; acc_par ^= 1u; }
        }
      }
    }
  } else if (warp >= EPI_WARPS) {
    // ------------------------------ producers: thread = pixel row, group = K block ------------------------------
    const int group = (warp - EPI_WARPS) >> 2, row = ((warp & 3) << 5) + lane;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const int total = my_tiles * jobs_per_tile;
    const float* base = a.x.ptr;       // window origin of this thread's pixel (may lie outside the image: then masked)
    uint32_t ymask = 0, xmask = 0;     // filter rows, and values of a run, that lie inside the image
    int tile = -1;
    auto enter_tile = [&](int t) {
      tile = t;
      const uint32_t m = (cta + (uint32_t)t * ctas) * BLOCK_M + row;
      ymask = xmask = 0;
      if (m < a.m_total) {
        const uint32_t n = a.img_div.div(m), rem = m - n * (uint32_t)(g.oh * g.ow), oy = a.row_div.div(rem), ox = rem - oy * (uint32_t)g.ow;
        const int y0 = (int)oy * g.sh - g.ph, x0 = (int)ox * g.sw - g.pw;
        base = a.x.ptr + n * a.x.s0 + (long long)y0 * a.x.s2 + (long long)x0 * a.x.s3;
        for (int k = 0; k < g.kh; ++k) ymask |= (uint32_t)(y0 + k * g.dh >= 0 && y0 + k * g.dh < g.h) << k;
        const int per_tap = a.channels_last ? g.cin : 1;
        const uint32_t tap = (1u << per_tap) - 1u;
        for (int k = 0; k < g.kw; ++k) xmask |= (x0 + k * g.dw >= 0 && x0 + k * g.dw < g.w ? tap : 0u) << (k * per_tap);
      }
    };
    auto load = [&](int job, float (&v)[KBLK]) {
      const int t = (int)a.div_jobs.div((uint32_t)job);
      if (t != tile) enter_tile(t);
      const int j = job - t * jobs_per_tile;
      const int kb = j - (int)a.div_nkb.div((uint32_t)j) * a.nkb;
#pragma unroll
      for (int r = 0; r < KBLK / LP; ++r) {
        const RunEntry e = tab[kb * (KBLK / LP) + r];
        const uint32_t m = (ymask >> e.ky) & 1u ? xmask : 0u;
        const float* p = base + e.offset;
#pragma unroll
        for (int i = 0; i < LP; ++i) v[r * LP + i] = (m >> i) & 1u ? __ldg(UNIT ? p + i : p + i * a.run_step) : 0.f;
      }
    };
    uint32_t s = (uint32_t)group % (uint32_t)a.stages, par = ((uint32_t)group / (uint32_t)a.stages & 1u) ^ 1u;
    auto store = [&](const float (&v)[KBLK]) -> bool {
      if (!warp_wait(smem_u32(&ctrl->empty[s]), par, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) return false;
      tc_fence_after();
      const uint32_t ta = a_cols + s * STAGE_COLS + lane_base;
      uint32_t r[32], c[32];
#pragma unroll
      for (int i = 0; i < KBLK; ++i) {
        float h, l;
        split_tf32_fast(v[i], h, l);
        r[i] = __float_as_uint(h);
        c[i] = __float_as_uint(l);
      }
      tmem_st32(ta, r);
      tmem_st32(ta + 32, c);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->full[s]));
      s += GROUPS;
      while (s >= (uint32_t)a.stages) { s -= (uint32_t)a.stages; par ^= 1u; }
      return true;
    };
    for (int job = group; job < total; job += GROUPS) {
      float v[KBLK];
      load(job, v);
      if (!store(v)) break;
    }
  } else {
    // ------------------------------ epilogue: lane = pixel, a warp stores 32 consecutive pixels of one channel ------------------------------
    const long long plane = (long long)g.oh * g.ow;
    uint32_t ab = 0, acc_par = 0;
    bool alive = true;
    for (int t = 0; t < my_tiles && alive; ++t) {
      const uint32_t m = (cta + (uint32_t)t * ctas) * BLOCK_M + (uint32_t)(warp * 32 + lane);
      const bool ok = m < a.m_total;
      long long obase = 0;
      if (ok) {
        const uint32_t n = a.img_div.div(m), rem = m - n * (uint32_t)plane;
        obase = (long long)n * g.cout * plane + rem;
      }
      for (int piece = 0; piece < a.ntn * a.segs; ++piece) {    // (column tile, chain)
        const int nt = a.segs == 1 ? piece : piece / a.segs, seg = piece - nt * a.segs;
        const int cols = min(a.bn, g.cout - ch0 - nt * a.bn);   // may be <= 0 in the last CTA of a split
        const uint32_t done = smem_u32(&ctrl->acc_empty[ab]);
        if (!warp_wait(smem_u32(&ctrl->acc_full[ab]), acc_par, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) { alive = false; break; }
        tc_fence_after();
        if (cols <= 0) {
          tc_fence_before();
          mbar_arrive(done);
        }
        const uint32_t acc = tmem_base + ab * acc_pitch + ((uint32_t)(warp * 32) << 16);
        if (++ab == (uint32_t)a.bufs) { ab = 0; acc_par ^= 1u; }
#pragma unroll 1
        for (int c0 = 0; c0 < cols; c0 += 32) {
          float v[32];
          if (PAIR) tmem_ld32_sum(acc + (uint32_t)c0, acc + (uint32_t)(a.acc_cols + c0), v);
          else tmem_ld32(acc + (uint32_t)c0, v);
          if (c0 + 32 >= cols) {
            tc_fence_before();
            mbar_arrive(done);
          }
          const int nvalid = min(32, cols - c0);
          const int ch = ch0 + nt * a.bn + c0;
          if (a.bias && seg == 0) {
            float bv = lane < nvalid ? __ldg(a.bias + (long long)(ch + lane) * a.bias_stride) : 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += __shfl_sync(0xffffffffu, bv, i);
          }
          if (ok) {
            float* p = a.out + obase + (long long)ch * plane;
            if (PAIR && seg > 0) {      // onto what this thread stored for the chain before: one writer per address, in program order
#pragma unroll
              for (int i = 0; i < 32; ++i, p += plane)
                if (i < nvalid) atomicAdd(p, v[i]);
            } else if (nvalid == 32) {
#pragma unroll
              for (int i = 0; i < 32; ++i, p += plane) *p = v[i];
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i, p += plane)
                if (i < nvalid) *p = v[i];
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

struct RowsPlan {
  bool ok = false;
  int runs = 0, run_len = 0, lp = 0, nkb = 0, ntn = 0, nt_split = 1, bn = 0, acc_cols = 0, pair = 0, bufs = 0, stages = 0, smem = 0;
};
// `channels_last`: the values of a filter row (taps x channels) are adjacent, so they form one run.
static RowsPlan plan_rows(const ConvGeom& g, bool channels_last) {
  RowsPlan p;
  if (g.groups != 1 || g.cout < 16 || g.kh > 31 || g.kw > 31) return p;
  p.runs = channels_last ? g.kh : g.cin * g.kh;
  p.run_len = channels_last ? g.kw * g.cin : g.kw;
  if (p.run_len > 31 || p.runs > MAX_RUNS) return p;
  p.lp = p.run_len <= 4 ? 4 : p.run_len <= 8 ? 8 : p.run_len <= 16 ? 16 : 32;
  p.nkb = (p.runs * p.lp + KBLK - 1) / KBLK;
  // all column tiles in every CTA while the filter fits; else one column tile per CTA, narrower until it fits
  const int tiles = (g.cout + 127) / 128, even = ((g.cout + tiles - 1) / tiles + 15) / 16 * 16;
  auto bytes = [&](int ntn, int bn) {
    return (long long)ntn * p.nkb * bn * 256 + (long long)p.nkb * (KBLK / p.lp) * sizeof(RunEntry) + 1024 + sizeof(Ctrl) + 64;
  };
  p.bn = even;
  p.ntn = bytes(tiles, even) <= SMEM_LIMIT ? tiles : 1;
  while (p.bn >= 16 && bytes(p.ntn, p.bn) > SMEM_LIMIT) p.bn = p.bn / 2 / 16 * 16;
  if (p.bn < 16) return p;
  p.nt_split = ((g.cout + p.bn - 1) / p.bn + p.ntn - 1) / p.ntn;
  if (p.nt_split > 8) return p;
  p.acc_cols = (p.bn + 31) / 32 * 32;
  p.pair = p.nkb > 2;
  p.bufs = p.pair && p.acc_cols > 64 ? 1 : 2;
  p.stages = std::min<int>(MAX_STAGES, (512 - (p.bufs * p.acc_cols << p.pair)) / (int)STAGE_COLS);
  const long long smem = bytes(p.ntn, p.bn);
  p.smem = (int)smem;
  p.ok = (long long)g.n * g.oh * g.ow < 2147483647ll - (1 << 20);
  return p;
}

template <int LP, bool UNIT, bool PAIR, int GROUPS>
static int launch_groups(const RowsArgs& a, unsigned ctas, int smem, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(conv_rows_kernel<LP, UNIT, PAIR, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  launch_next(conv_rows_kernel<LP, UNIT, PAIR, GROUPS>, ctas, THREADS_OF<GROUPS>, (size_t)smem, st, a);
  count_launch();
  return launch_check("conv_rows_kernel");
}
template <int LP, bool UNIT, bool PAIR>
static int launch_rows(const RowsArgs& a, int smem, cudaStream_t st) {
  const int share = std::min(a.tiles_m, std::max(1, sm_count() / a.nt_split));   // CTAs that share the pixel tiles
  const unsigned ctas = (unsigned)(share * a.nt_split);
  const bool many = div_up64(a.tiles_m, share) * a.ntn * a.nkb >= FOUR_GROUPS_FROM;
  return many ? launch_groups<LP, UNIT, PAIR, 4>(a, ctas, smem, st) : launch_groups<LP, UNIT, PAIR, 3>(a, ctas, smem, st);
}

}  // namespace tcr

// Fewer than sixteen input channels: the strip kernels would multiply mostly padding.
bool rows_supported(const ConvGeom& g) { return g.cig < 16 && tcr::plan_rows(g, false).ok; }

int rows_conv(const ConvGeom& g, View4 x, View4 w, const float* bias, long long bias_stride, float* y, cudaStream_t st) {
  using namespace tcr;
  // channels-last with dense pixels: a filter row's taps x channels are adjacent and form one run, where such a run has 31 values at most
  bool channels_last = g.cin > 1 && x.s1 == 1 && x.s3 == g.cin && g.dw == 1;
  RowsPlan plan = plan_rows(g, channels_last);
  if (channels_last && !plan.ok) plan = plan_rows(g, channels_last = false);
  if (!plan.ok) return fail(B200_EUNSUPPORTED, "row kernel does not take this geometry");
  // offsets inside a window are 32-bit
  if ((g.cin - 1) * std::llabs(x.s1) + (long long)(g.kh - 1) * g.dh * std::llabs(x.s2) + (long long)(g.kw - 1) * g.dw * std::llabs(x.s3) > 2147483647ll)
    return fail(B200_EUNSUPPORTED, "row kernel: window too large for 32-bit element offsets");
  RowsArgs a{};
  a.g = g; a.x = x; a.w = w; a.bias = bias; a.bias_stride = bias_stride; a.out = y;
  a.runs = plan.runs; a.run_len = plan.run_len; a.channels_last = channels_last ? 1 : 0;
  a.run_step = channels_last ? 1 : g.dw * x.s3;
  a.segs = (plan.nkb + SEG_KB - 1) / SEG_KB; a.seg_kb = (plan.nkb + a.segs - 1) / a.segs;
  a.nkb = plan.nkb; a.bn = plan.bn; a.acc_cols = plan.acc_cols; a.ntn = plan.ntn; a.nt_split = plan.nt_split; a.bufs = plan.bufs; a.stages = plan.stages;
  a.m_total = (uint32_t)((long long)g.n * g.oh * g.ow);
  a.tiles_m = (int)div_up64(a.m_total, BLOCK_M);
  if ((long long)a.tiles_m * plan.ntn * plan.nkb > 2147483647ll) return fail(B200_EUNSUPPORTED, "row kernel: job count exceeds 32 bits");
  a.img_div = FastDiv((uint32_t)(g.oh * g.ow)); a.row_div = FastDiv((uint32_t)g.ow);
  a.div_nkb = FastDiv((uint32_t)plan.nkb); a.div_kh = FastDiv((uint32_t)g.kh); a.div_cin = FastDiv((uint32_t)g.cin);
  a.div_jobs = FastDiv((uint32_t)(plan.ntn * plan.nkb));
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  const bool unit = a.run_step == 1;
  auto launch = [&](auto lp) {
    constexpr int LP = decltype(lp)::value;
    return plan.pair ? (unit ? launch_rows<LP, true, true>(a, plan.smem, st) : launch_rows<LP, false, true>(a, plan.smem, st))
                     : (unit ? launch_rows<LP, true, false>(a, plan.smem, st) : launch_rows<LP, false, false>(a, plan.smem, st));
  };
  switch (plan.lp) {
    case 4: return launch(std::integral_constant<int, 4>{});
    case 8: return launch(std::integral_constant<int, 8>{});
    case 16: return launch(std::integral_constant<int, 16>{});
    default: return launch(std::integral_constant<int, 32>{});
  }
}

}  // namespace b200

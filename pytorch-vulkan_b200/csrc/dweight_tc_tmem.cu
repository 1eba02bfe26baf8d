// tcgen05 dWeight kernel with the output gradient in TENSOR MEMORY, FP32 by split precision (TF32 hi*hi plus BF16 cross terms).
//
//   dW[co][ci][ky][kx] = sum over grid pixels q of  dY[q][co] * X_phase(ky,kx)[q + shift(ky,kx)][ci]
//
// What bounds this product and why it is arranged this way.  With both operands in shared memory (dweight_tc_strip.cu) every
// 128-row step is paced by its operand reads (85 clocks for a 128x128x8 step that computes for 64), and a 3-wide filter
// leaves one of the four 32-row tap blocks on the M side empty: 0.56 of the pipe at best, 211 TFLOP/s measured.  Here
//   * A = dY transposed, 128 output channels on the lanes of tensor memory, written once per K block with tcgen05.st: it is
//     the operand that no filter tap shifts, so it can live where descriptors cannot reach;
//   * B = the input strip, pixel-major in shared memory, N = taps x 32 channels: the taps kx of a row are the N blocks of ONE
//     operand, `dilation` rows apart through the descriptor's leading-dimension stride, so a 3-wide filter runs at N = 96
//     without an empty block, and a step reads 3 KB for its 48 clocks: the multipliers set the pace.
//   * Up to 384 accumulator columns (several channel blocks, or several ky) share every dY block, which keeps the bytes pulled
//     from L2 per step down: the next bound.
//   * 64 or fewer output channels fill only half of the lanes: the other half then holds dY `delta` grid rows further down, so
//     one strip serves two vertical taps (two strips instead of three for a 3x3 filter).
// The input strips are RINGS of 32-row chunks (32 channels of one stride phase each), tall enough for every vertical tap: a
// pixel is staged once, and each ky reads the ring `dilation` image rows further on, so that a K block of a 3x3 filter stages
// one input chunk and four dY blocks for 24 steps of N = 96.  The first 40 rows of a ring are repeated behind its end, so that
// a descriptor (32 rows and up to eight rows of horizontal taps) never has to wrap.  Images too wide for that take one ky per
// CTA.
//
// FOLD (fewer than sixteen input channels: a network's first layer): the (input channel, ky) pairs of a pixel take the place of the
// channels of a strip, 21 of 32 for 3 channels and a 7x7 filter, and the taps kx stay row offsets.  dW is then that of a
// one-row filter over cin * kh channels, whose layout it already has.  Four offsets of these channels come with one read, pieces of eight
// channels beyond the last are neither loaded nor stored, and filter rows are tested only where the image cuts some off (one read
// and test a value took 28 instructions for each; 186 -> 181 us on that layer).
//
// The pixel grid, the split of the contraction over CTAs, the chunked accumulation (the tensor core truncates: CHUNK_KB) and
// the partial layout [split][cout][kh*kw][cin/g] are those of dweight_tc_strip.cu.
//
// Measured step times (128 rows, tensor-memory A): N / 2 clocks from N = 32 on; with A in shared memory 32 + N / 4.
//
// CTA roles: two or three sets of four dY warps (set s stages K blocks = s mod sets, a warp the lanes of its quarter; they
// also fold the accumulator), then input warps up to warp 14, warp 15 MMA issue.  All waits are bounded.
// Where 64 or fewer output channels leave lanes 64-127 empty and no second tap fills them (folded layers, 1x1 filters), the warps of those
// quarters stage input, and four sets of two warps stage dY: a dY block is a load from memory, a conversion and a store in one warp, so
// the number of warps that have one on its way sets the pace.  3 -> 64 channels, 7x7, stride 2, 64x224x224: 186 us, now 144.
//
// THREE (1x1 filters with 64 or fewer output channels): the cross terms are two TF32 products instead of one BF16 pass, in accumulator columns of
// their own.  dweight_tc_strip.cu, which takes these layers otherwise, runs three passes too, and the multipliers are idle here in any case: 432 -> 64
// channels of 5x 7x7 8.1 us and an error of 1.46e-6 against FP64 with the BF16 pass, 8.2 and 6.2e-7 with three (there 11.9 and 1.23e-6); 45 layers
// 0.99 of the BF16 form's time and 0.2 to 0.5 of its error.
//
// Replaces csrc/shaders/conv2d_backward_weight_tiled_body.glsl:42-70 of the reference for these geometries.
#include "common.cuh"
#include "plan_cache.cuh"
#include "dweight_stage.cuh"
#include "dweight_plan.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

namespace b200 {
namespace tcdt {
using namespace tc;
using tcdw::BlockPlanes;

constexpr int KP = 32;                       // pixels per K block
constexpr int HALO = 8;                      // rows that horizontal taps may reach beyond a K block's own
constexpr int MIRROR = KP + HALO;            // rows repeated behind the end of a ring
constexpr int MMA_WARP = 15, THREADS = 512;
constexpr int NARROW_X_WARPS = 7;            // warps 2, 3, 6, 7, 10, 11, 14
constexpr int MAX_RING = 24, MAX_A = 6, MAX_STRIPS = 8, MAX_GROUPS = 8, MAX_SLOTS = 12;
constexpr int ACC_COLS = 384;                // accumulator columns at most (two 64-column dY stages need the rest)
constexpr int SCRATCH = 32 * 36 * 4;         // transpose tile of a dY warp
constexpr int SMEM_LIMIT = 232448 - 2048;
constexpr int FOLD_MAX = 256;                // (input channel, filter row) pairs at most
constexpr int NO_PIXEL = -2147483647 - 1;    // an element offset that no admitted view has (strides may be negative, run() bounds their span)
constexpr int CHUNK_KB = 96;                 // K blocks per accumulation chain (see dweight_tc_strip.cu)
// ... of layers with fewer than 32 (input channel, tap) pairs per group, which ran in FP32 on the CUDA cores before: 49 images of 95x95, 3 -> 80
// channels, 3x3, off by 1.4e-5 in chains of 96, 1.0e-6 in chains of 4 (FP32 7.6e-7; in chains of 2 8e-7); 87 us, now 116 (FP32 613).
constexpr int CHUNK_KB_FP32 = 4;

struct Strip {       // one staged input strip
  signed char cblk;  // channel block within the CTA's tile
  signed char pa, pb;  // row and column phase of a strided input
  signed char dr, dc;  // whole-pixel row / column offset of its first row (pa, dr: of the CTA's own ky when ky_tiles > 1)
};
struct Group {       // one chain of MMAs: N = 32 * blocks
  uint32_t strip_off;  // bytes from the first strip's hi ring
  uint32_t lbo, lbo16; // bytes between N blocks in the hi ring / the bf16 rings
  uint32_t n_bits;     // N in instruction-descriptor position
  int row;             // row offset of its first tap within the ring
  int col;             // first accumulator column
};
struct Slot {        // 32 accumulator columns: 32 input channels of one tap
  signed char cblk, ky, kx, upper_ky;   // upper_ky: vertical tap of lanes 64-127 in shift mode, -1 = none
};

struct Args {
  ConvGeom g;
  View4 x, dy;
  float* out;                 // partials [split][cout][kh*kw][cig], or dW itself
  int partial_layout;
  int H, W, pr, pc;           // padded pixel grid
  int q_first, q_total;       // contraction range [q_first, q_total); q_first < 0 in shift mode
  FastDiv img_div, row_div, div_strips, div_ring;
  int dy_sets, ahead;         // sets of dY warps; chunks a K block reads beyond its own
  int narrow;                 // 64 or fewer output channels and no shift: a set is two warps, the warps of the other quarters stage input
  int span, splits;
  int shift_rows;             // shift mode: lanes 64-127 hold dY this many grid pixels ahead (0: off)
  int nci, ci_tiles, ky_tiles, co_tiles;
  int n_strips, n_groups, n_slots;
  int ring, a_stages, chunk_kb;
  int sph, spw, in_h, in_w, out_h, out_w;
  Strip strips[MAX_STRIPS];
  Group groups[MAX_GROUPS];
  Slot slots[MAX_SLOTS];
  int fold_kh, fold_sh, fold_dh, fold_ph, fold_h;   // FOLD: the real filter height and what places its rows (g describes the folded layer)
  int* status;
  int three;                  // THREE: as many accumulator columns again for the cross terms
};

struct Ctrl {
  unsigned long long x_full[MAX_RING], x_empty[MAX_RING], a_full[MAX_A], a_empty[MAX_A], accum, drained;
  uint32_t tmem_base;
  int abort_flag;
};

constexpr int FOLD_AT = ((int)sizeof(Ctrl) + 15) / 16 * 16;   // the fold table behind Ctrl, in 16-byte pieces

// whether the phase has completed, without the suspension of try_wait
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t desc64(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}

// NG groups of NB N-blocks each where the plan has that shape (0: as the arguments say): with the loop bounds and the step width
// known, the issuing warp needs 175 clocks less per K block of a 3x3 filter.
template <int NG, int NB, bool FOLD, bool THREE>
__global__ void __launch_bounds__(THREADS, 1) dweight_tmem_kernel(const Args a) {
  wait_previous();
  constexpr int GROUPS = NG ? NG : MAX_GROUPS;
  extern __shared__ unsigned char smem_raw[];
  if (a.partial_layout) asm volatile("griddepcontrol.launch_dependents;");
  const ConvGeom& g = a.g;
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t ring_pixels = (uint32_t)(a.ring * KP), ring_rows = ring_pixels + MIRROR;
  const uint32_t strip_bytes = ring_rows * 256u;                 // hi ring (128-byte rows), then bf16(hi) and bf16(lo) rings (64-byte rows)
  unsigned char* scratch_all = smem_raw + (base - raw) + a.n_strips * strip_bytes;
  const int dy_quarters = a.narrow ? 2 : 4, dy_warps = dy_quarters * a.dy_sets;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(scratch_all + dy_warps * SCRATCH);
  int* fold_off = reinterpret_cast<int*>(scratch_all + dy_warps * SCRATCH + FOLD_AT);   // [cig up to a multiple of 32] elements from the window's first row
  int* fold_ky = fold_off + FOLD_MAX;                                                   // filter row
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_RING; ++s) {
      mbar_init(smem_u32(&ctrl->x_full[s]), (uint32_t)a.n_strips);
      mbar_init(smem_u32(&ctrl->x_empty[s]), 1);
    }
    for (int s = 0; s < MAX_A; ++s) {
      mbar_init(smem_u32(&ctrl->a_full[s]), (uint32_t)dy_quarters);
      mbar_init(smem_u32(&ctrl->a_empty[s]), 1);
    }
    mbar_init(smem_u32(&ctrl->accum), 1);
    mbar_init(smem_u32(&ctrl->drained), (uint32_t)dy_warps);
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (FOLD)
    for (int c = threadIdx.x; c < (g.cig + 31) / 32 * 32; c += THREADS) {
      const int ci = c / a.fold_kh, ky = c - ci * a.fold_kh;
      fold_off[c] = c < g.cig ? (int)(ci * a.x.s1 + (long long)(ky * a.fold_dh) * a.x.s2) : 0;
      fold_ky[c] = c < g.cig ? ky : 31;                           // 31: no pixel has that row
    }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  const uint32_t acc_cols = (uint32_t)a.n_slots * 32u, a_cols = tmem + (THREE ? 2u : 1u) * acc_cols;   // dY stages of 64 columns behind the accumulators

  // ---- which piece of dW this CTA owns ----
  int id = blockIdx.x;
  const int ci_tile = id % a.ci_tiles; id /= a.ci_tiles;
  const int ky_tile = id % a.ky_tiles; id /= a.ky_tiles;
  const int co_tile = id % a.co_tiles; id /= a.co_tiles;
  const int group = id, split = blockIdx.y;
  const int ci0 = ci_tile * a.nci * 32;
  const int ky0 = a.ky_tiles > 1 ? ky_tile : -1;                 // this CTA's only vertical tap, -1: all of them
  const int co0 = co_tile * (a.shift_rows ? 64 : 128);
  const int row_pitch = a.W + a.pc, img_pitch = (a.H + a.pr) * row_pitch;
  const int k_begin = a.q_first + split * a.span;
  const int k_end = a.q_total - k_begin > a.span ? k_begin + a.span : a.q_total;
  const int kblocks = (k_end - k_begin + KP - 1) / KP;
  const int fold_chunks = (kblocks + a.chunk_kb - 1) / a.chunk_kb;

  if (warp == MMA_WARP) {
    const bool leader = elect_one();
    // A (tensor memory) is K-major by nature; B is MN-major (bit 16).  All control flow and descriptor arithmetic stays uniform over
    // the warp; only the tcgen05 instructions themselves are predicated on the elected lane.
    // The steps are short (48 clocks at N = 96) and the tensor pipe takes only a few of them ahead, so every instruction between two
    // of them counts, all the more beside busy staging warps: descriptors advance by additions to their low words, the group
    // parameters are indexed with constants, and the next K block's barriers are polled before the last group of the current one.
    const uint32_t idesc = make_idesc_tf32(128, 0) | (1u << 16), idesc16 = make_idesc_bf16(128, 0) | (1u << 16);
    const uint64_t hi_tmpl = tcdw::make_mn_desc(base, 0), b16_tmpl = tcdw::make_mn_desc16(base + ring_rows * 128u, 0);
    const uint32_t hi_top = (uint32_t)(hi_tmpl >> 32), b16_top = (uint32_t)(b16_tmpl >> 32), l16_d = (ring_rows * 64u) >> 4, lo_d = (ring_rows * 128u) >> 4;
    uint32_t lo_h[GROUPS], lo_16[GROUPS], pos[GROUPS];   // low descriptor words and ring position of every group
#pragma unroll
    for (int i = 0; i < GROUPS; ++i) {
      const uint32_t off = a.groups[i].strip_off >> 4;
      pos[i] = (uint32_t)a.groups[i].row;
      lo_h[i] = (uint32_t)hi_tmpl + off + pos[i] * 8u + ((a.groups[i].lbo >> 4) << 16);
      lo_16[i] = (uint32_t)b16_tmpl + off + pos[i] * 4u + ((a.groups[i].lbo16 >> 4) << 16);
    }
    uint32_t sa = 0, a_par = 0, slot = 0;
    uint32_t newest = 0, newest_slot = 0, newest_par = 0;   // chunks waited for so far
    int in_chunk = 0, chunk = 0;
    bool alive = true, ready = false;
    for (int kb = 0; kb < kblocks; ++kb, ++in_chunk) {
      if (in_chunk == a.chunk_kb) {   // hand the accumulator to the fold and wait until it has been read
        if (leader) umma_commit(smem_u32(&ctrl->accum));
        if (!warp_wait(smem_u32(&ctrl->drained), (uint32_t)chunk & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
        ++chunk;
        in_chunk = 0;
      }
      if (!ready) {
        for (; newest <= (uint32_t)(kb + a.ahead); ++newest) {
          if (!warp_wait(smem_u32(&ctrl->x_full[newest_slot]), newest_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
          if (++newest_slot == (uint32_t)a.ring) { newest_slot = 0; newest_par ^= 1u; }
        }
        if (!alive) break;
        if (!warp_wait(smem_u32(&ctrl->a_full[sa]), a_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) break;
      }
      tc_fence_after();
      const uint32_t ta = a_cols + sa * 64u, a_done = smem_u32(&ctrl->a_empty[sa]), x_done = smem_u32(&ctrl->x_empty[slot]);
      if (++sa == (uint32_t)a.a_stages) { sa = 0; a_par ^= 1u; }
      if (++slot == (uint32_t)a.ring) slot = 0;
#pragma unroll
      for (int i = 0; i < GROUPS; ++i) {
        if (!NG && i >= a.n_groups) break;
        const bool last = NG ? i + 1 == NG : i + 1 == a.n_groups;
        if (last)
          ready = __all_sync(0xffffffffu, mbar_test(smem_u32(&ctrl->x_full[newest_slot]), newest_par) & mbar_test(smem_u32(&ctrl->a_full[sa]), a_par));
        const uint32_t n = NB ? (uint32_t)NB << 19 : a.groups[i].n_bits, acc = tmem + (uint32_t)a.groups[i].col;
        if (leader) {
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32_ts(acc, ta + 8 * k, desc64(lo_h[i] + 64 * k, hi_top), idesc | n, (uint32_t)((in_chunk | k) != 0));
          if (THREE) {
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_tf32_ts(acc + acc_cols, ta + 8 * k, desc64(lo_h[i] + lo_d + 64 * k, hi_top), idesc | n, (uint32_t)((in_chunk | k) != 0));
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_tf32_ts(acc + acc_cols, ta + 32 + 8 * k, desc64(lo_h[i] + 64 * k, hi_top), idesc | n, 1);
          } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) umma_bf16_ts(acc, ta + 32 + 8 * k, desc64(lo_16[i] + l16_d + 64 * k, b16_top), idesc16 | n, 1);
#pragma unroll
            for (int k = 0; k < 2; ++k) umma_bf16_ts(acc, ta + 48 + 8 * k, desc64(lo_16[i] + 64 * k, b16_top), idesc16 | n, 1);
          }
          if (last) {
            umma_commit(a_done);
            umma_commit(x_done);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < GROUPS; ++i) {
        pos[i] += KP; lo_h[i] += KP * 8; lo_16[i] += KP * 4;
        if (pos[i] >= ring_pixels) { pos[i] -= ring_pixels; lo_h[i] -= ring_pixels * 8u; lo_16[i] -= ring_pixels * 4u; }
      }
      if (ready) {
        ++newest;
        if (++newest_slot == (uint32_t)a.ring) { newest_slot = 0; newest_par ^= 1u; }
      }
    }
    if (leader) umma_commit(smem_u32(&ctrl->accum));
  } else if (a.narrow ? (warp & 3) >= 2 : warp >= dy_warps) {
    // ---- input chunks: job j = (chunk, strip) goes to warp j mod (warps in use) ----
    const bool vec = channel_quads_aligned(a.x, g.cig, g.groups);
    const int jobs = (kblocks + a.ahead) * a.n_strips;
    // consecutive jobs of a warp stay within `ring` chunks of each other (a waiter must not skip a phase of a slot's barrier)
    const int active = min(a.narrow ? NARROW_X_WARPS : MMA_WARP - dy_warps, a.n_strips * a.ring);
    const int xw = a.narrow ? (warp >> 2) * 2 + (warp & 1) : warp - dy_warps;
    int dr0 = 0, pa0 = 0;
    if (ky0 >= 0) {
      const int oy = ky0 * g.dh - g.ph;
      dr0 = oy >= 0 ? oy / a.sph : -((-oy + a.sph - 1) / a.sph);
      pa0 = oy - dr0 * a.sph;
    }
    auto load = [&](int job, float (&val)[32]) -> bool {   // returns which register pattern stage_block used
      const int c = (int)a.div_strips.div((uint32_t)job), strip = job - c * a.n_strips;
      const Strip st = a.strips[strip];
      const int c0 = ci0 + st.cblk * 32;
      if (FOLD) {
        const int q = k_begin + c * KP + st.dc + lane;
        uint32_t rows = 0;                         // filter rows of this pixel that lie inside the image
        const uint32_t whole = (1u << a.fold_kh) - 1u;
        const float* p = a.x.ptr;
        if (q >= 0 && q < a.q_total) {
          const int n = (int)a.img_div.div((uint32_t)q), rem = q - n * img_pitch;
          const int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch, iy = y * a.fold_sh - a.fold_ph, ix = x * a.spw + st.pb;
          if (x < a.W && ix < a.in_w) {
            for (int k = 0; k < a.fold_kh; ++k) rows |= (uint32_t)(iy + k * a.fold_dh >= 0 && iy + k * a.fold_dh < a.fold_h) << k;
            p += n * a.x.s0 + (long long)iy * a.x.s2 + (long long)ix * a.x.s3;
          }
        }
        const int sw = ((lane >> 2) & 1) << 2;     // store_block's register order
        const bool inside = rows != 0;
        const bool all_rows = __all_sync(0xffffffffu, rows == whole || !inside);   // no row cut off by the image: one predicate for the pixel
#pragma unroll
        for (int m = 0; m < 32; m += 4) {
          if (c0 + (m & ~7) >= g.cig) break;       // the columns of these channels are never read
          const int at = c0 + (m ^ sw);
          const int4 o = *reinterpret_cast<const int4*>(fold_off + at);
          if (all_rows) {
            val[m] = inside ? __ldg(p + o.x) : 0.f; val[m + 1] = inside ? __ldg(p + o.y) : 0.f;
            val[m + 2] = inside ? __ldg(p + o.z) : 0.f; val[m + 3] = inside ? __ldg(p + o.w) : 0.f;
          } else {
            const int4 k = *reinterpret_cast<const int4*>(fold_ky + at);
            val[m] = (rows >> k.x) & 1u ? __ldg(p + o.x) : 0.f; val[m + 1] = (rows >> k.y) & 1u ? __ldg(p + o.y) : 0.f;
            val[m + 2] = (rows >> k.z) & 1u ? __ldg(p + o.z) : 0.f; val[m + 3] = (rows >> k.w) & 1u ? __ldg(p + o.w) : 0.f;
          }
        }
        return false;
      }
      return tcdw::stage_block(a.x, (long long)group * g.cig + c0, max(0, min(32, g.cig - c0)), a.H, a.W, row_pitch, img_pitch, a.img_div,
                               a.row_div, k_begin + c * KP + (ky0 >= 0 ? dr0 : st.dr) * row_pitch + st.dc, 0, a.q_total, 32, lane, vec, val,
                               a.sph, a.spw, ky0 >= 0 ? pa0 : st.pa, st.pb, a.in_h, a.in_w);
    };
    for (int job = xw; job < jobs && xw < active; job += active) {
      const int c = (int)a.div_strips.div((uint32_t)job), strip = job - c * a.n_strips;
      const uint32_t round = a.div_ring.div((uint32_t)c);
      const int slot = c - (int)round * a.ring;
      float val[32];
      const bool chunked = load(job, val);
      if (!warp_wait(smem_u32(&ctrl->x_empty[slot]), (round & 1u) ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) break;
      BlockPlanes pl;
      pl.hi = base + (uint32_t)strip * strip_bytes;
      pl.lo = pl.h16 = pl.hi + ring_rows * 128u;
      pl.l16 = pl.h16 + ring_rows * 64u;
      const int copies = slot * KP < MIRROR ? 2 : 1;        // the first rows of the ring once more behind its end
#pragma unroll 1
      for (int i = 0; i < copies; ++i) {
        const int row0 = slot * KP + i * (int)ring_pixels, rows = i ? min(KP, MIRROR - slot * KP) : KP;
        if (chunked) tcdw::store_block_chunks<!THREE>(val, rows, row0, pl, lane);
        else tcdw::store_block<!THREE>(val, rows, row0, pl, lane, FOLD ? g.cig - ci0 - a.strips[strip].cblk * 32 : 32);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->x_full[slot]));
    }
  } else if (!a.narrow || (warp >> 2) < a.dy_sets) {
    // ---- dY: lane = output channel (tensor-memory lane quarter * 32 + lane), columns = pixels ----
    const int set = warp >> 2, quarter = warp & 3;
    float* scratch = reinterpret_cast<float*>(scratch_all + (set * dy_quarters + quarter) * SCRATCH);
    const bool shift = a.shift_rows != 0;
    const int cq = co0 + (shift ? (quarter & 1) : quarter) * 32;           // first channel of this warp
    const int dq = shift && quarter >= 2 ? a.shift_rows : 0;
    const int chans = max(0, min(32, g.cog - cq));
    const bool channels_inner = a.dy.s1 == 1 && a.dy.s3 != 1;
    const long long chan_off = ((long long)group * g.cog + cq) * a.dy.s1;
    const long long s1 = a.dy.s1;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int taps = g.kh * g.kw;
    const long long cols = (long long)g.cig * taps;
    float* out = a.out + ((long long)split * g.cout + (long long)group * g.cog + cq) * cols;
    bool alive = true;
    int kb = set;
    uint32_t sa = (uint32_t)set, a_par = 1;        // a_stages >= sets
    const float* src = a.dy.ptr + chan_off;
    // lane = pixel (channels apart in memory) or lane = channel (channels adjacent)
    auto load = [&](int k, float (&v)[32]) {
      int off = NO_PIXEL;                          // element offset of this lane's pixel, NO_PIXEL where the contraction has nothing
      {
        const int qx = k_begin + k * KP + lane, q = qx + dq;
        if (qx < k_end && q >= 0 && q < a.q_total) {
          const int n = (int)a.img_div.div((uint32_t)q), rem = q - n * img_pitch;
          const int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch;
          if (y < a.out_h && x < a.out_w) off = (int)(n * a.dy.s0 + (long long)y * a.dy.s2 + (long long)x * a.dy.s3);
        }
      }
      if (channels_inner) {
        int* offs = reinterpret_cast<int*>(scratch);
        const float* mine = src + lane;
        __syncwarp();
        offs[lane] = off;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; i += 4) {            // four pixels' offsets per read
          const int4 o = *reinterpret_cast<const int4*>(offs + i);
          v[i] = o.x != NO_PIXEL && lane < chans ? __ldg(mine + o.x) : 0.f;
          v[i + 1] = o.y != NO_PIXEL && lane < chans ? __ldg(mine + o.y) : 0.f;
          v[i + 2] = o.z != NO_PIXEL && lane < chans ? __ldg(mine + o.z) : 0.f;
          v[i + 3] = o.w != NO_PIXEL && lane < chans ? __ldg(mine + o.w) : 0.f;
        }
      } else {
        const float* p = src + (off != NO_PIXEL ? off : 0);
#pragma unroll
        for (int i = 0; i < 32; ++i, p += s1) v[i] = off != NO_PIXEL && i < chans ? __ldg(p) : 0.f;
      }
    };
    auto advance = [&] {
      sa += (uint32_t)a.dy_sets;
      if (sa >= (uint32_t)a.a_stages) { sa -= (uint32_t)a.a_stages; a_par ^= 1u; }
    };
    auto store = [&](const float (&v)[32]) -> bool {
      if (!channels_inner) {                       // through shared memory to lane = channel
        __syncwarp();                              // the previous use of the tile is over
#pragma unroll
        for (int i = 0; i < 32; ++i) scratch[i * 36 + lane] = v[i];
        __syncwarp();
      }
      if (!warp_wait(smem_u32(&ctrl->a_empty[sa]), a_par, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) return false;
      tc_fence_after();
      const uint32_t ta = a_cols + sa * 64u + lane_base;
      uint32_t hi[32], cr[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float w[4];
        if (channels_inner) {
          w[0] = v[4 * i]; w[1] = v[4 * i + 1]; w[2] = v[4 * i + 2]; w[3] = v[4 * i + 3];
        } else {
          const float4 f = *reinterpret_cast<const float4*>(scratch + lane * 36 + 4 * i);
          w[0] = f.x; w[1] = f.y; w[2] = f.z; w[3] = f.w;
        }
        float h[4], l[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          split_tf32_fast(w[j], h[j], l[j]);
          hi[4 * i + j] = __float_as_uint(h[j]);
        }
        if (THREE) {
#pragma unroll
          for (int j = 0; j < 4; ++j) cr[4 * i + j] = __float_as_uint(l[j]);
        } else {
          cr[2 * i] = pack_bf16x2(h[0], h[1]);
          cr[2 * i + 1] = pack_bf16x2(h[2], h[3]);
          cr[16 + 2 * i] = pack_bf16x2(l[0], l[1]);
          cr[17 + 2 * i] = pack_bf16x2(l[2], l[3]);
        }
      }
      tmem_st32(ta, hi);
      tmem_st32(ta + 32, cr);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->a_full[sa]));
      advance();
      return true;
    };
    for (int chunk = 0; chunk < fold_chunks && alive; ++chunk) {
      // the first dY stages of the next chunk are staged before this chunk is folded: their slots depend on nothing the fold waits
      // for, and the MMA warp then finds them ready when the fold hands the accumulator back
      const int kb_end = chunk + 1 < fold_chunks ? min(kblocks, (chunk + 1) * a.chunk_kb + a.a_stages) : kblocks;
      for (; kb < kb_end; kb += a.dy_sets) {
        if (chans == 0 && kb >= a.a_stages) {      // lanes without channels hold zeros since the first round
          if (!(alive = warp_wait(smem_u32(&ctrl->a_empty[sa]), a_par, abort_flag, a.status, STATUS_TIMEOUT_EMPTY))) break;
          if (lane == 0) mbar_arrive(smem_u32(&ctrl->a_full[sa]));
          advance();
          continue;
        }
        float v[32];
        load(kb, v);
        if (!(alive = store(v))) break;
      }
      if (!alive) break;
      // ---- fold the chunk: slot i of the accumulator is read by set i mod sets; a warp turns its 32 channels x 32 input channels in
      // shared memory so that every store or reduction instruction covers 128 contiguous bytes ----
      if (!warp_wait(smem_u32(&ctrl->accum), (uint32_t)chunk & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
      const bool add = chunk > 0;
#pragma unroll 1
      for (int i = set; i < a.n_slots; i += a.dy_sets) {
        const Slot sl = a.slots[i];
        float v[32];
        const uint32_t at = tmem + (uint32_t)(i * 32) + lane_base;
        if (THREE) tmem_ld32_sum(at, at + acc_cols, v);
        else tmem_ld32(at, v);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) scratch[lane * 33 + j] = v[j];
        __syncwarp();
        const int ky = ky0 >= 0 ? ky0 : shift && quarter >= 2 ? sl.upper_ky : sl.ky;
        const int ci = ci0 + sl.cblk * 32 + lane, tap = ky * g.kw + sl.kx;
        if (ky < 0 || ky >= g.kh || chans == 0) continue;
        float* p = out + (a.partial_layout ? (long long)tap * g.cig + ci : (long long)ci * taps + tap);
        if (ci >= g.cig) continue;                 // no warp-wide instruction below
        auto emit = [&](auto full) {               // eight rows' reads are issued before the first store: one row at a time took 2000 clocks a slot
#pragma unroll 1
          for (int r = 0; r < 32; r += 8) {
            float t[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) t[j] = scratch[(r + j) * 33 + lane];
#pragma unroll
            for (int j = 0; j < 8; ++j, p += cols) {
              if (!full.value && r + j >= chans) continue;
              if (add) atomicAdd(p, t[j]);         // one writer per address, in program order: the same sums from run to run
              else *p = t[j];
            }
          }
        };
        if (chans == 32) emit(std::true_type{});
        else emit(std::false_type{});
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0 && chunk + 1 < fold_chunks) mbar_arrive(smem_u32(&ctrl->drained));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

static inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

struct Plan {
  bool ok = false;
  Args a{};                 // everything but the tensors
  int smem = 0;
  long long tiles = 0;
  size_t bytes = 0;
};

// Strips, MMA groups and accumulator slots of a CTA that owns `nci` channel blocks and the vertical taps of ky_list (one entry
// with ky_list null: the kernel takes the tap from its tile index).  Returns the rows a K block reads beyond its own, or -1.
static int layout(const ConvGeom& g, int nci, int nky, const int* ky_list, const int* upper, int row_pitch, Args& a) {
  a.nci = nci;
  a.n_strips = a.n_groups = a.n_slots = 0;
  const bool merge = g.kw == 1 && nky == 1;        // one tap: the N blocks of a group are channel blocks
  int reach = 0;
  struct Pending { int strip, row, blocks, step; } pend[MAX_GROUPS];
  // row phases in use and the smallest row offset of each
  int dr_of[8], pa_of[8];
  for (int i = 0; i < nky; ++i) {
    const int oy = ky_list ? ky_list[i] * g.dh - g.ph : 0;
    dr_of[i] = ky_list ? floor_div(oy, g.sh) : 0;
    pa_of[i] = ky_list ? oy - dr_of[i] * g.sh : 0;
  }
  for (int pa = 0; pa < g.sh; ++pa) {
    int dr_min = 1 << 30;
    for (int i = 0; i < nky; ++i)
      if (pa_of[i] == pa) dr_min = std::min(dr_min, dr_of[i]);
    if (dr_min == 1 << 30) continue;
    for (int pb = 0; pb < g.sw; ++pb) {
      int kxs[8], dcs[8], n = 0;
      for (int kx = 0; kx < g.kw; ++kx) {
        const int ox = kx * g.dw - g.pw, dc = floor_div(ox, g.sw);
        if (ox - dc * g.sw != pb) continue;
        kxs[n] = kx; dcs[n++] = dc;
      }
      if (!n) continue;
      if (dcs[n - 1] - dcs[0] > HALO || dcs[0] < -127 || dcs[0] > 127 || dr_min < -127 || dr_min > 127) return -1;
      for (int t = 2; t < n; ++t)
        if (dcs[t] - dcs[t - 1] != dcs[1] - dcs[0]) return -1;
      for (int c = 0; c < nci; ++c) {
        if (a.n_strips == MAX_STRIPS) return -1;
        a.strips[a.n_strips] = Strip{(signed char)c, (signed char)pa, (signed char)pb, (signed char)dr_min, (signed char)dcs[0]};
        for (int i = 0; i < nky; ++i) {
          if (pa_of[i] != pa) continue;
          if (a.n_slots + n > MAX_SLOTS) return -1;
          const int row = (dr_of[i] - dr_min) * row_pitch;
          if (merge && c > 0) {
            ++pend[a.n_groups - 1].blocks;
          } else {
            if (a.n_groups == MAX_GROUPS) return -1;
            a.groups[a.n_groups].row = row;
            a.groups[a.n_groups].col = a.n_slots * 32;
            pend[a.n_groups++] = Pending{a.n_strips, row, n, merge ? 0 : n > 1 ? dcs[1] - dcs[0] : 1};
          }
          reach = std::max(reach, row + dcs[n - 1] - dcs[0]);
          for (int t = 0; t < n; ++t)
            a.slots[a.n_slots++] = Slot{(signed char)c, (signed char)(ky_list ? ky_list[i] : 0), (signed char)kxs[t], (signed char)upper[i]};
        }
        ++a.n_strips;
      }
    }
  }
  a.ahead = (reach + KP - 1) / KP;
  for (int i = 0; i < a.n_groups; ++i) {          // strip_off, lbo of a merged group: filled in with the ring size (finish_groups)
    a.groups[i].strip_off = (uint32_t)pend[i].strip;
    a.groups[i].lbo = (uint32_t)pend[i].step;
    a.groups[i].n_bits = (uint32_t)pend[i].blocks << 19;   // (32 * blocks / 8) << 17
  }
  return reach;
}
static void finish_groups(Args& a) {
  const uint32_t strip_bytes = (uint32_t)(a.ring * KP + MIRROR) * 256u;
  for (int i = 0; i < a.n_groups; ++i) {
    Group& gr = a.groups[i];
    const uint32_t step = gr.lbo;
    gr.strip_off *= strip_bytes;
    gr.lbo = step ? step * 128u : strip_bytes;
    gr.lbo16 = step ? step * 64u : strip_bytes;
  }
}

static Plan make_plan(const ConvGeom& real, size_t budget) {
  Plan best;
  // fewer than sixteen input channels: fold the filter rows into the channels (see above)
  ConvGeom g = real;
  const bool fold = real.cig < 16;
  if (fold) {
    if (real.groups != 1 || real.kh > 31 || real.cig * real.kh > FOLD_MAX || real.cig * real.kh * real.kw < 9) return best;
    g.cin = g.cig = real.cig * real.kh;
    g.kh = 1; g.ph = 0; g.dh = 1; g.sh = 1; g.h = g.oh;
  }
  if ((!fold && g.cig < 16) || g.kw > 8 || g.cog < 16 || g.sh > 127 || g.sw > 127) return best;
  const int gh = std::max(g.oh, (g.h + g.sh - 1) / g.sh), gw = std::max(g.ow, (g.w + g.sw - 1) / g.sw);
  int pr = 0, pc = 0;
  for (int ky = 0; ky < g.kh; ++ky) pr = std::max(pr, std::abs(floor_div(ky * g.dh - g.ph, g.sh)));
  for (int kx = 0; kx < g.kw; ++kx) pc = std::max(pc, std::abs(floor_div(kx * g.dw - g.pw, g.sw)));
  const long long q_total = (long long)g.n * (gh + pr) * (gw + pc);
  if (q_total > 2147483647ll - (1 << 20)) return best;
  // 1x1 filters are bound by the staging of both operands, for which dweight_tc_strip.cu has more warps but needs long splits to fill its
  // pipeline.  Measured, that kernel against this one: 256 -> 512 channels of 32 x 14x14 38.7 and 28.4 us, 96 -> 131 of 42 x 7x7 31.9 and
  // 11.9, 32 -> 128 of 64 x 56x56 57 and 45; 512 -> 96 of 64 x 14x14 28.0 and 29.4, 512 -> 128 of 32 x 28x28 34 and 44, 64 -> 64 of
  // 64 x 56x56 42 and 53: the line is at five million input values, or one block of input channels.
  // Fewer than 64 input channels leave that kernel's rows half empty, with one value to a load in the ragged block: where wide outputs repeat it,
  // this one is faster at any size (48 -> 256 of 33 x 92x92 233 and 125 us, 61 -> 400 of 20 x 88x88 211 and 138; 64 -> 192 of 27 x 77x77 69 and 73).
  // Its BF16 cross terms cost them nothing: such sums are long, and that kernel's chains are as long with more steps to a K block (the same layers
  // 1.31e-5 and 8.9e-6 off, 1.46e-5 and 9.9e-6).
  if (!fold && g.kh * g.kw == 1 && g.cig > 32 && !(g.cig < 64 && g.cog > 128) && q_total * g.cig > (5ll << 20)) return best;
  const int row_pitch = gw + pc;
  // shift mode: vertical taps m apart lie a whole number of grid rows apart
  int m = 1;
  while (m * g.dh % g.sh) ++m;
  const bool shift = g.cog <= 64 && g.kh > m && g.kh <= 8;
  const int shift_rows = shift ? m * g.dh / g.sh * row_pitch : 0;
  int ky_list[8], upper[8], n_list = 0;
  if (shift) {
    bool done[8] = {};
    for (int ky = g.kh - 1; ky >= 0; --ky)
      if (!done[ky]) {
        done[ky] = true;
        ky_list[n_list] = ky;
        upper[n_list] = ky >= m && !done[ky - m] ? ky - m : -1;
        if (ky >= m) done[ky - m] = true;
        ++n_list;
      }
  }
  // 32 and more (input channel, tap) pairs, as with CHUNK_KB_FP32: below, chains of four K blocks
  const bool three = !fold && g.kh * g.kw == 1 && g.cog <= 64 && g.cig >= 32;
  const int q_first = -((shift_rows + KP - 1) / KP * KP);
  const int cib = (g.cig + 31) / 32;
  const size_t dw_bytes = sizeof(float) * (size_t)g.cout * g.cig * g.kh * g.kw;
  const long long kb_total = div_up64(q_total - q_first, KP);
  int limit = real.cig * real.kh * real.kw < 32 ? CHUNK_KB_FP32 : CHUNK_KB;
  if (const char* e = getenv("B200_DW_CHUNK_KB")) limit = std::max(1, atoi(e));   // testing aid: chain length in K blocks
  double best_cost = 0;
  for (int nci : {1, 2, 3, 4, 6, 8}) {
    if (nci > cib && nci > 1) break;
    for (int all = 1; all >= (g.kh > 1 && !shift ? 0 : 1); --all) {   // every vertical tap in one CTA, or one per CTA
      Plan p;
      Args& a = p.a;
      int list[64], up[64];
      const int nky = shift ? n_list : all ? g.kh : 1;
      if (nky > 8) continue;
      for (int i = 0; i < nky; ++i) { list[i] = shift ? ky_list[i] : i; up[i] = shift ? upper[i] : -1; }
      if (layout(g, nci, nky, all ? list : nullptr, up, row_pitch, a) < 0) continue;
      a.three = three;
      if ((three ? 64 : 32) * a.n_slots > ACC_COLS) continue;
      a.a_stages = std::min(MAX_A, (512 - (three ? 64 : 32) * a.n_slots) / 64);
      // dY sets against input warps: whichever split lets the slower side keep up best
      a.dy_sets = 1;
      auto slower = [&](int sets) { return std::max(1.0 / sets, (double)a.n_strips / (MMA_WARP - 4 * sets)); };
      for (int sets = 2; sets <= std::min(3, a.a_stages); ++sets)
        if (slower(sets) < slower(a.dy_sets)) a.dy_sets = sets;
      // lanes 64-127 have no channels: their warps stage input instead
      a.narrow = g.cog <= 64 && !shift;
      if (a.narrow) a.dy_sets = std::min(4, a.a_stages);
      const int fixed_smem = (a.narrow ? 2 : 4) * a.dy_sets * SCRATCH + (int)sizeof(Ctrl) + (fold ? 2 * FOLD_MAX * (int)sizeof(int) + 16 : 0) + 1024 + 64;
      a.ring = std::min({MAX_RING, a.ahead + 6, (SMEM_LIMIT - fixed_smem - a.n_strips * MIRROR * 256) / (a.n_strips * KP * 256)});
      if (a.ring < a.ahead + 3 || a.a_stages < 2) continue;
      a.ci_tiles = (cib + nci - 1) / nci;
      a.ky_tiles = all ? 1 : g.kh;
      a.co_tiles = shift ? 1 : (g.cog + 127) / 128;
      p.tiles = (long long)a.ci_tiles * a.ky_tiles * a.co_tiles * g.groups;
      p.smem = fixed_smem + a.n_strips * (a.ring * KP + MIRROR) * 256;
      // clocks of a K block: the MMAs (16 per N block and step, and what issuing
      // them beside the staging warps costs), the bytes pulled from L2 (about 22 per clock and SM), the work
      // of the staging warps (about 2400 clocks per job and warp)
      const int dy_jobs = shift ? 2 * std::min(2, (g.cog + 31) / 32) : std::min(4, (g.cog + 31) / 32);
      const double mma = (three ? 192.0 : 128.0) * a.n_slots + 100.0 + 60.0 * a.n_groups + 30.0 * (a.n_strips + dy_jobs);
      const double kb_clk = std::max({mma, 4096.0 * (a.n_strips + dy_jobs) / 22.0,
                                      2400.0 * (a.narrow ? std::max(1.0 / a.dy_sets, (double)a.n_strips / NARROW_X_WARPS) : slower(a.dy_sets))});
      for (int w = 0; w <= 3; ++w) {
        long long sp = w == 0 ? 1 : w * (long long)sm_count() / p.tiles;
        sp = std::min<long long>({sp, std::max<long long>(1, kb_total / 6), 65535, std::max<long long>(1, (long long)(budget / dw_bytes))});
        if (sp < 1) continue;
        const double per = (double)div_up64(kb_total, sp), waves = (double)div_up64(p.tiles * sp, sm_count());
        const double cost = waves * (per * kb_clk + per / limit * 2500.0 + 6000.0 + 150.0 * a.n_slots) +
                            (sp > 1 ? 3000.0 + (double)(sp + 1) * dw_bytes / 2200.0 : 0.0);
        if (!best.ok || cost < best_cost) {
          best_cost = cost;
          const long long span = div_up64(div_up64(q_total - q_first, sp), KP) * KP;
          a.span = (int)span;
          a.splits = (int)div_up64(q_total - q_first, span);
          p.bytes = a.splits > 1 ? (size_t)a.splits * dw_bytes : 0;
          p.ok = true;
          best = p;
        }
      }
    }
  }
  if (!best.ok) return best;
  Args& a = best.a;
  finish_groups(a);
  a.H = gh; a.W = gw; a.pr = pr; a.pc = pc;
  a.q_first = q_first; a.q_total = (int)q_total;
  a.shift_rows = shift_rows;
  a.img_div = FastDiv((uint32_t)((gh + pr) * row_pitch)); a.row_div = FastDiv((uint32_t)row_pitch);
  a.div_strips = FastDiv((uint32_t)a.n_strips); a.div_ring = FastDiv((uint32_t)a.ring);
  a.sph = g.sh; a.spw = g.sw; a.in_h = g.h; a.in_w = g.w; a.out_h = g.oh; a.out_w = g.ow;
  const int kblocks = a.span / KP, chunks = (kblocks + limit - 1) / limit;
  a.chunk_kb = (kblocks + chunks - 1) / chunks;
  a.g = g;
  a.fold_kh = fold ? real.kh : 0;
  a.fold_sh = real.sh; a.fold_dh = real.dh; a.fold_ph = real.ph; a.fold_h = real.h;
  return best;
}
static const Plan& cached_plan(const ConvGeom& g, size_t budget) {
  thread_local PlanCache<Plan> cache, pinned;
  if (getenv("B200_DW_CHUNK_KB")) return pinned.get(g, budget + (size_t)atoi(getenv("B200_DW_CHUNK_KB")) * 7919, [&] { return make_plan(g, budget); });
  return cache.get(g, budget, [&] { return make_plan(g, budget); });
}

bool plan_info(const ConvGeom& g, size_t budget, PlanInfo* info) {
  const Plan& p = cached_plan(g, budget);
  if (p.ok) *info = PlanInfo{p.bytes, p.a.span / KP, p.a.n_strips, p.a.n_slots, p.a.shift_rows != 0};
  return p.ok;
}

template <int NG, int NB, bool FOLD = false, bool THREE = false>
static int launch(const Args& a, const Plan& p, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(dweight_tmem_kernel<NG, NB, FOLD, THREE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  launch_next(dweight_tmem_kernel<NG, NB, FOLD, THREE>, dim3((unsigned)p.tiles, (unsigned)a.splits), THREADS, (size_t)p.smem, st, a);
  count_launch();
  return launch_check("dweight_tmem_kernel");
}

int run(const ConvGeom& g, View4 x, View4 dy, float* dw, void* ws, size_t ws_bytes, cudaStream_t st) {
  Plan p = cached_plan(g, ws ? ws_bytes : 0);
  if (!p.ok) return B200_EUNSUPPORTED;
  // element offsets inside a tensor are 32-bit in the kernel
  auto span = [](const View4& v, long long n, long long c, long long h, long long w) {
    return (n - 1) * std::llabs(v.s0) + (c - 1) * std::llabs(v.s1) + (h - 1) * std::llabs(v.s2) + (w - 1) * std::llabs(v.s3);
  };
  if (span(x, g.n, g.cin, g.h, g.w) > 2147483647ll - 64 * std::llabs(x.s1) || span(dy, g.n, g.cout, g.oh, g.ow) > 2147483647ll - 64 * std::llabs(dy.s1))
    return B200_EUNSUPPORTED;
  Args& a = p.a;
  a.x = x; a.dy = dy;
  a.out = a.splits > 1 ? (float*)ws : dw;
  a.partial_layout = a.splits > 1 ? 1 : 0;
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  if (p.tiles > 2147483647ll) return fail(B200_ERANGE, "dWeight kernel: grid exceeds launch limits");
  const bool threes = [&] {
    for (int i = 0; i < a.n_groups; ++i)
      if (a.groups[i].n_bits != 3u << 19) return false;
    return true;
  }();
  const int rc = a.three ? launch<1, 0, false, true>(a, p, st) : a.fold_kh ? (a.n_groups == 2 ? launch<2, 0, true>(a, p, st) : a.n_groups == 1 ? launch<1, 0, true>(a, p, st) : launch<0, 0, true>(a, p, st)) : threes && a.n_groups == 3 ? launch<3, 3>(a, p, st) : threes && a.n_groups == 4 ? launch<4, 3>(a, p, st)
               : a.n_groups == 1 ? launch<1, 0>(a, p, st) : a.n_groups == 6 ? launch<6, 0>(a, p, st) : launch<0, 0>(a, p, st);
  if (rc) return rc;
  if (a.splits > 1) return tcdw::finalize_partials((const float*)ws, dw, a.g, a.splits, st);
  return B200_OK;
}

}  // namespace tcdt
}  // namespace b200

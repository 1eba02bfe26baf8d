// Persistent tcgen05 implicit-GEMM kernel for convolution forward and dInput (any stride, padding,
// dilation and grouping; reduction channels in blocks of 32), FP32 by split precision (one TF32 pass
// for hi x hi, one BF16 pass for the cross terms: tc_common.cuh).  The same kernel is
// the GEMM behind mm/addmm and the plane product of the Winograd path.
//
// Idea: the kh*kw filter taps of one 32-channel block all read the same activations, shifted by
// whole pixels.  The activations of a tile are therefore staged ONCE per channel block as a
// "strip" in shared memory -- one 128-byte row (32 channels, TF32 hi and lo planes) per pixel of
// a zero-padded pixel grid -- and every tap's tcgen05.mma reads that strip through a matrix
// descriptor whose start address is moved by `shift(tap)` rows.  (The 128-byte swizzle is a
// function of the absolute shared-memory address, so a descriptor may start at any row.)
// Compared with gathering an operand tile per tap this issues kh*kw times fewer global loads,
// TF32 splits and shared-memory stores, which is what lets the tensor pipe stay busy.
//
// Padded pixel grid: `pc` zero columns after every row and `pr` zero rows after every image,
// q = (n*(H+pr) + y)*(W+pc) + x.  A tap offset (dr, dc) is then the constant row shift
// dr*(W+pc) + dc for every pixel, and reads that leave the image land on zero rows of the strip.
// Accumulator rows that fall on padding (or outside a smaller output) are discarded.
//
// Strides: with stride s the taps are grouped by the phase (row mod s, column mod s) of the pixels
// they touch -- input phases in forward (channel blocks are enumerated per phase, each with its own
// taps), output phases in dInput (column tiles are enumerated per phase; all read one dY strip).
// See TapTable and plan_strip.
//
// CTA roles (448 threads, persistent over tiles of 128 grid pixels x BN output channels):
//   warps 0-3    epilogue: tcgen05.ld of a finished accumulator, bias, coalesced stores
//   warps 4-11   strip producers: gather from the caller's strided view, TF32 split, swizzled stores
//   warp 12      (one thread) weight stages: one bulk copy (cp.async.bulk -> mbarrier complete_tx)
//                of a pre-split, pre-swizzled image per stage; stage_weights_kernel writes the
//                images once per call
//   warp 13      TMEM allocation; one thread issues the tcgen05.mma stream
// The accumulator is double-buffered in TMEM, so the epilogue of tile i overlaps the main loop of
// tile i+1.  All hand-offs are mbarriers with bounded waits.
//
// Replaces csrc/shaders/conv2d_tiled_body.glsl:53-86 and
// csrc/shaders/conv2d_backward_input_tiled_body.glsl:49-93 of the reference.
#include <cuda_bf16.h>

#include "common.cuh"
#include "gemm_tmem.cuh"
#include "plan_cache.cuh"
#include "strip_plan.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace b200 {
namespace tcs {
using namespace tc;

constexpr int BLOCK_M = 128, KBLK = 32;
// Warp roles: 4 epilogue warps, AW strip producers, the weight-copy warp, the MMA warp.  AW is 8, or 12 for layers
// whose producers set the pace (one tap per staged strip: 1x1 filters), which fetch a job ahead; sixteen had no registers for that.
constexpr int EPI_WARPS = 4, W_WARPS = 1;
constexpr int strip_threads(int aw) { return (EPI_WARPS + aw + W_WARPS + 1) * 32; }
constexpr int MAX_STAGES = 4;
constexpr int SMEM_LIMIT = 232448 - 2048;  // 227 KB per CTA minus the control block and alignment slack

struct StripArgs {
  ConvGeom g;
  View4 act;              // forward: x.  dInput: dy
  const float* wp;        // weight stage images [groups][tiles_n][phase][cblock][tap of phase] of BN*256 bytes
  const float* bias;
  long long bias_stride;
  float* out;             // contiguous NCHW [n][out_channels][out_h][out_w] (or row-major, see below)
  int H, W, pr, pc;       // pixel grid shared by the strip and the accumulator rows, and its zero padding
  int act_h, act_w;       // extent of the activation tensor; grid pixel (r, c) of phase (a, b) reads (r*sph + a, c*spw + b)
  int out_h, out_w;       // extent of the output tensor (grid pixels beyond it are discarded)
  int sph, spw;           // forward: phases live on the reduction side (channel block -> phase)
  int osh, osw;           // dInput: phases live on the output side: column tile -> phase (a, b), grid pixel (r, c)
                          // is the output pixel (r*osh + a, c*osw + b); all phases read the same dY strip
  int phase_on_n;         // 1 in the dInput arrangement
  int tiles_pp;           // column tiles per phase (dInput), else tiles_n
  int kc, nc, out_channels;
  // batched GEMM (groups used as the batch): extra element offsets per group on top of the grouped
  // convolution's own (group * kc channels in, group * nc columns out); 0 / out_channels / nc otherwise
  long long act_group_extra, out_pitch, out_group;
  int k_total;            // reduction channels of all groups (the last group may have fewer than kc)
  int cb_per_phase;       // kc / 32
  int cblocks;            // strips per tile: forward n_phase * cb_per_phase, dInput cb_per_phase
  int images_per_tile;    // forward: weight stages per tile = cb_per_phase * taps_total
  int tiles_n;
  int q_total;            // grid pixels incl. padding (below 2^31 - 2^20)
  FastDiv img_div, row_div;
  int tiles_m, tiles_total;
  int unit, units;        // tiles per scheduling unit, number of units (tiles_total = unit * units)
  int m_fastest;          // tile order (tile_coord)
  FastDiv div_tiles_n, div_tiles_m, div_tiles_pp, div_chunks, div_cblocks, div_cbpp, div_a_stages, div_unit;
  int halo, strip_rows;   // rows staged before the tile's first pixel; strip_rows is a multiple of 8
  int a_stages, w_stages;
  int out_rowmajor;       // 0: NCHW planes.  1: [pixel][channel] rows (channels-last / GEMM C)
  int out_vec4;           // row-major rows may be written with 16-byte stores
  int wide_producers;     // 1: the kernel instance with twelve producer warps
  float alpha, beta;      // out = alpha * acc + beta * bias
  View4 res;              // optional residual added after the bias (logical shape of the output), ptr null = none
  int relu;               // clamp at zero last
  int wait_for_images;    // launched with programmatic stream serialisation behind stage_weights_kernel
  int* status;
  unsigned long long* prof;  // optional cycle counters of CTA 0 (B200_STRIP_PROFILE=1), else null
  TapTable tt;
};

struct Ctrl {  // lives behind the operand stages in shared memory
  unsigned long long a_full[MAX_STAGES], a_empty[MAX_STAGES], w_full[MAX_STAGES], w_empty[MAX_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int shift[MAX_TAPS];
  unsigned char ph_a[MAX_PHASES], ph_b[MAX_PHASES], tap_start[MAX_PHASES + 1];
};

// Cycle accounting for one thread of each role in CTA 0 (diagnostics only).  The probes sit in the
// issuing loops, where every extra instruction costs tensor time, so they are compiled in only with
// -DB200_ROLE_PROFILE=1 (then B200_STRIP_PROFILE=1 in the environment prints them).
#ifndef B200_ROLE_PROFILE
#define B200_ROLE_PROFILE 0
#endif
#define PROF_ON(leader) (B200_ROLE_PROFILE && a.prof != nullptr && blockIdx.x == 0 && (leader))
#define PROF_T0(on) const long long prof_t0__ = (on) ? clock64() : 0
#define PROF_ADD(on, slot) do { if (on) atomicAdd(a.prof + (slot), (unsigned long long)(clock64() - prof_t0__)); } while (0)

// Tiles are dealt to CTAs in units of `unit` consecutive tiles, unit u to CTA u mod gridDim.  At any
// moment the CTAs then work on neighbouring pixel rows (their strips share DRAM pages and L2 lines),
// and with unit = all column tiles of a pixel-row tile a strided dInput gives every CTA the same mix
// of output phases, whose tap counts differ.
struct TileIter {
  int u, t, unit, units, step;
  __device__ explicit TileIter(const StripArgs& a) : u(blockIdx.x), t(0), unit(a.unit), units(a.units), step(gridDim.x) {}
  __device__ bool valid() const { return u < units; }
  __device__ int tile() const { return u * unit + t; }
  __device__ void next() { if (++t == unit) { t = 0; u += step; } }
};

// tile index -> (pixel-row tile, column tile, group).  Column tile fastest when tiles are dealt in
// units (see TileIter); otherwise the pixel-row tile runs fastest, so that the CTAs working at the same
// time share their weight stages (the heavier operand: BN*256 bytes per stage against 16 KB of raw
// activations) and L2 serves them as one stream.
struct TileCoord {
  int m_tile, n_tile, group;
};
__device__ __forceinline__ TileCoord tile_coord(const StripArgs& a, int tile) {
  TileCoord c;
  if (a.m_fastest) {
    const int rest = (int)a.div_tiles_m.div((uint32_t)tile);
    c.m_tile = tile - rest * a.tiles_m;
    c.group = (int)a.div_tiles_n.div((uint32_t)rest);
    c.n_tile = rest - c.group * a.tiles_n;
  } else {
    const int tn = (int)a.div_tiles_n.div((uint32_t)tile);
    c.n_tile = tile - tn * a.tiles_n;
    c.group = (int)a.div_tiles_m.div((uint32_t)tn);
    c.m_tile = tn - c.group * a.tiles_m;
  }
  return c;
}

// 32 consecutive floats of each lane's row (row = null: nothing to store): lanes l, l+4, ..., l+28 exchange 16-byte pieces so that a
// store instruction covers whole 128-byte lines of four rows instead of 16 bytes of 32 rows, which kept the load/store unit busy for
// 8000 of the 32000 cycles of a 128x256 tile's products and slowed the producers' loads beside it.
__device__ __forceinline__ void store_rows32(float (&v)[32], float* row, int lane) {
  const int i = lane >> 2;
#pragma unroll
  for (int s = 1; s < 8; s <<= 1) {
    const bool upper = (i & s) != 0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if ((j & s) == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float &lo = v[4 * j + e], &hi = v[4 * (j | s) + e];
          const float other = __shfl_xor_sync(0xffffffffu, upper ? lo : hi, s << 2);
          if (upper) lo = other; else hi = other;
        }
      }
  }
  const unsigned long long mine = reinterpret_cast<unsigned long long>(row);
#pragma unroll
  for (int j = 0; j < 8; ++j) {  // piece i of row 4j + lane % 4
    float* p = reinterpret_cast<float*>(__shfl_sync(0xffffffffu, mine, 4 * j + (lane & 3)));
    if (p) reinterpret_cast<float4*>(p)[i] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
}

template <int BN, int AW>
__global__ void __launch_bounds__(strip_threads(AW), 1) conv_strip_kernel(const StripArgs a) {
  constexpr int A_WARPS = AW, MMA_WARP = EPI_WARPS + AW + W_WARPS;
  extern __shared__ unsigned char smem_raw[];
  const unsigned long long prof_start = a.prof ? global_ns() : 0;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles_base = (raw + 1023u) & ~1023u;
  const uint32_t a_stage_bytes = (uint32_t)a.strip_rows * 256u, a_plane = (uint32_t)a.strip_rows * 128u;
  constexpr uint32_t w_stage_bytes = BN * 256u, w_plane = BN * 128u;
  const uint32_t w_base = tiles_base + a.a_stages * a_stage_bytes;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (w_base - raw) + a.w_stages * w_stage_bytes);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  // For BN <= 128 the weight stage's hi and lo planes (adjacent in shared memory) are fed to the
  // tensor core as ONE operand of 2*BN rows: a single MMA of width 2*BN yields a_hi*b_hi in columns
  // [0,BN) and a_hi*b_lo in [BN,2BN), a second one of width BN adds a_lo*b_hi to [0,BN); the epilogue
  // sums the two halves.  Two MMAs read 14/18 of the shared-memory bytes that three do.
  constexpr bool FUSE_HILO = BN <= 128 && !CROSS_BF16;
  constexpr uint32_t ACC_COLS = FUSE_HILO ? 2 * BN : BN;
  constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->a_full[s]), (uint32_t)((a.strip_rows + 31) / 32) * 32u);
      mbar_init(smem_u32(&ctrl->a_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctrl->acc_full[s]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[s]), EPI_WARPS * 32);
    }
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->w_full[s]), 1);  // the issuing thread's arrive.expect_tx; the copy completes the bytes
      mbar_init(smem_u32(&ctrl->w_empty[s]), 1);
    }
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  // the tap table moves to shared memory: kernel parameters are not indexed dynamically
  if (threadIdx.x < MAX_TAPS) ctrl->shift[threadIdx.x] = a.tt.shift[threadIdx.x];
  if (threadIdx.x < MAX_PHASES) { ctrl->ph_a[threadIdx.x] = a.tt.a[threadIdx.x]; ctrl->ph_b[threadIdx.x] = a.tt.b[threadIdx.x]; }
  if (threadIdx.x <= MAX_PHASES) ctrl->tap_start[threadIdx.x] = a.tt.start[threadIdx.x];
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);

  const int row_pitch = a.W + a.pc;
  const int img_pitch = (a.H + a.pr) * row_pitch;

  if (warp == MMA_WARP) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp runs the loop and waits on the barriers; one elected lane issues the tcgen05 instructions.
    // With uniform control flow the descriptors live in uniform registers, which is where tcgen05.mma reads its
    // operands (issued from one divergent thread, every operand crossed over from the vector registers first, and
    // that crossing paced the kernel).  Stage indices and parities are counted, not divided, and descriptors are
    // the stage's base plus an offset.
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_tf32(BLOCK_M, BN);
      constexpr uint32_t idesc_wide = make_idesc_tf32(BLOCK_M, FUSE_HILO ? 2 * BN : BN);
      constexpr uint32_t idesc_cross = make_idesc_bf16(BLOCK_M, BN);
      const uint64_t da_base = make_kmajor_sw128_desc(tiles_base + (uint32_t)a.halo * 128u);
      const uint64_t db_base = make_kmajor_sw128_desc(w_base);
      const uint32_t a_stage_d = a_stage_bytes >> 4, a_plane_d = a_plane >> 4;
      constexpr uint32_t w_stage_d = w_stage_bytes >> 4, w_plane_d = w_plane >> 4;
      uint32_t as = 0, a_par = 0, ws = 0, w_par = 0, t_count = 0;
      const bool pm = PROF_ON(lane == 0);
      bool alive = true;
      for (TileIter it(a); it.valid() && alive; it.next(), ++t_count) {
        const int tile = it.tile();
        const uint32_t ab = t_count & 1;
        { PROF_T0(pm);
        if (!warp_wait(smem_u32(&ctrl->acc_empty[ab]), ((t_count >> 1) & 1) ^ 1, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
        PROF_ADD(pm, 0); }
        tc_fence_after();
        const uint32_t tmem_acc = tmem_base + ab * ACC_COLS;
        const int n_tile = tile_coord(a, tile).n_tile;
        int phase = a.phase_on_n ? (int)a.div_tiles_pp.div((uint32_t)n_tile) : 0;  // dInput: the phase of this column tile
        int cbl = 0;
        uint32_t accumulate = 0;  // the tile's first MMA overwrites the accumulator
        for (int cb = 0; cb < a.cblocks && alive; ++cb) {
          { PROF_T0(pm);
          if (!warp_wait(smem_u32(&ctrl->a_full[as]), a_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
          PROF_ADD(pm, 1); }
          const uint64_t da_strip = da_base + as * a_stage_d;
          const int tap_end = ctrl->tap_start[phase + 1];
          for (int tap = ctrl->tap_start[phase]; tap < tap_end; ++tap) {
            const int sh = ctrl->shift[tap];
            { PROF_T0(pm);
            if (!warp_wait(smem_u32(&ctrl->w_full[ws]), w_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
            PROF_ADD(pm, 2); }
            PROF_T0(pm);
            const uint64_t da_hi = da_strip + (uint64_t)(long long)(sh * 8), da_lo = da_hi + a_plane_d;
            const uint64_t db_hi = db_base + ws * w_stage_d, db_lo = db_hi + w_plane_d;
            const uint32_t first = accumulate;
            accumulate = 1;
            if (!leader) {
            } else if (CROSS_BF16) {  // hi x hi in TF32, then both cross terms as one BF16 product over the second planes
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_hi + 2 * kk, db_hi + 2 * kk, idesc, first | (uint32_t)(kk != 0));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_bf16(tmem_acc, da_lo + 2 * kk, db_lo + 2 * kk, idesc_cross, 1);
            } else if (FUSE_HILO) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_hi + 2 * kk, db_hi + 2 * kk, idesc_wide, first | (uint32_t)(kk != 0));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_lo + 2 * kk, db_hi + 2 * kk, idesc, 1);
            } else {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_lo + 2 * kk, db_hi + 2 * kk, idesc, first | (uint32_t)(kk != 0));
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_hi + 2 * kk, db_lo + 2 * kk, idesc, 1);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_tf32(tmem_acc, da_hi + 2 * kk, db_hi + 2 * kk, idesc, 1);
            }
            if (leader) umma_commit(smem_u32(&ctrl->w_empty[ws]));
            if (++ws == (uint32_t)a.w_stages) { ws = 0; w_par ^= 1; }
            PROF_ADD(pm, 3);
          }
          if (alive && leader) umma_commit(smem_u32(&ctrl->a_empty[as]));
          if (++as == (uint32_t)a.a_stages) { as = 0; a_par ^= 1; }
          if (!a.phase_on_n && ++cbl == a.cb_per_phase) { cbl = 0; ++phase; }
        }
        if (alive && leader) umma_commit(smem_u32(&ctrl->acc_full[ab]));
      }
    }
  } else if (warp == EPI_WARPS + A_WARPS) {
    // ------------------------------ weight stages ------------------------------
    // One thread: each stage is a single bulk copy of a ready-made (split, swizzled) image.
    if (lane == 0) {
      uint32_t ws = 0, w_par = 1, issued = 0;
      bool alive = true;
      const bool pw = PROF_ON(true);
      // The kernel may have started while the staging kernel ahead of it was still running: only
      // this thread reads what that kernel writes, so only it waits for that kernel to finish.
      if (a.wait_for_images) asm volatile("griddepcontrol.wait;" ::: "memory");
      for (TileIter it(a); it.valid() && alive; it.next()) {
        const int tile = it.tile();
        const TileCoord tc_ = tile_coord(a, tile);
        const int n_tile = tc_.n_tile;
        const long long group = tc_.group;
        long long first_image;
        int images;
        if (a.phase_on_n) {  // images of a group: [phase][tile of the phase][channel block][tap of the phase]
          const int phase = (int)a.div_tiles_pp.div((uint32_t)n_tile), in_phase = n_tile - phase * a.tiles_pp;
          const int t0 = ctrl->tap_start[phase], ntap = ctrl->tap_start[phase + 1] - t0;
          images = a.cb_per_phase * ntap;
          first_image = ((group * a.tt.taps_total + t0) * a.tiles_pp + (long long)in_phase * ntap) * a.cb_per_phase;
        } else {
          images = a.images_per_tile;
          first_image = (group * a.tiles_n + n_tile) * a.images_per_tile;
        }
        const float* img = a.wp + first_image * (long long)(BN * 64);
        for (int i = 0; i < images; ++i, img += BN * 64) {
          { PROF_T0(pw);
          if (!mbar_wait(smem_u32(&ctrl->w_empty[ws]), w_par, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) { alive = false; break; }
          PROF_ADD(pw, 4); }
          const uint32_t full = smem_u32(&ctrl->w_full[ws]);
          mbar_expect_tx(full, w_stage_bytes);
          bulk_g2s(w_base + ws * w_stage_bytes, img, w_stage_bytes, full);
          ++issued;
          if (++ws == (uint32_t)a.w_stages) { ws = 0; w_par ^= 1; }
        }
      }
      // After an abort the MMA thread no longer consumes stages: wait (bounded) for the copies still
      // in flight so that none lands in shared memory of a finished CTA.
      if (!alive)
        for (uint32_t j = issued > (uint32_t)a.w_stages ? issued - a.w_stages : 0; j < issued; ++j)
          mbar_wait(smem_u32(&ctrl->w_full[j % a.w_stages]), (j / a.w_stages) & 1, nullptr, a.status, STATUS_TIMEOUT_FULL);
    }
  } else if (warp >= EPI_WARPS) {
    // ------------------------------ strip producers ------------------------------
    // A stage is staged as chunks of 32 rows, one warp per chunk (lane = row); chunk c of stage n
    // goes to warp (n*chunks + c) % 8, so short strips (1x1 filters) keep several stages in flight.
    const int aw = warp - EPI_WARPS;
    const int chunks = (a.strip_rows + 31) / 32;
    const bool vec_layout = a.act.s1 == 1 && a.kc % 4 == 0 && ((reinterpret_cast<uintptr_t>(a.act.ptr) & 15) == 0) &&
                        (a.act.s0 % 4 == 0) && (a.act.s2 % 4 == 0) && (a.act.s3 % 4 == 0) && (a.act_group_extra % 4 == 0);
    const int s1 = (int)a.act.s1;
    const int my_units = a.units > (int)blockIdx.x ? (a.units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int my_tiles = my_units * a.unit;
    const int total_jobs = my_tiles * a.cblocks * chunks;  // below 2^31 (checked by the host)
    // A warp's consecutive jobs must not be more than a_stages stages apart: a waiter that skips a
    // whole phase of a stage's mbarrier would see the parity of an older phase and run ahead.
    const int a_warps = min(A_WARPS, chunks * a.a_stages);
    // A job's loads are issued before the previous job is converted and stored: a warp that waited for its own loads first
    // left the tensor core idle for a third of the time where one strip feeds one tap (16384x1024 x 1024x1024: 155 -> 144 us).
    struct Job { int chunk; uint32_t as, round; bool chunked; };
    auto fetch = [&](auto wide, int job, float (&v)[KBLK]) -> Job {
      const uint32_t a_count = a.div_chunks.div((uint32_t)job);
      const int chunk = job - (int)a_count * chunks;
      const uint32_t tile_iter = a.div_cblocks.div(a_count);
      const int cb = (int)(a_count - tile_iter * a.cblocks);
      const uint32_t unit_iter = a.div_unit.div(tile_iter);
      const uint32_t tile = (blockIdx.x + unit_iter * gridDim.x) * a.unit + (tile_iter - unit_iter * a.unit);
      const TileCoord tc_ = tile_coord(a, (int)tile);
      const int group = tc_.group, m_tile = tc_.m_tile;
      const uint32_t a_round = a.div_a_stages.div(a_count);
      const uint32_t as = a_count - a_round * a.a_stages;
      const int r = chunk * 32 + lane;
      const int q = m_tile * BLOCK_M - a.halo + r;
      bool ok = r < a.strip_rows && q >= 0 && q < a.q_total;
      const float* src = a.act.ptr;
      const int phase = a.phase_on_n ? 0 : (int)a.div_cbpp.div((uint32_t)cb), cbl = cb - phase * a.cb_per_phase;
      // the last channel block of a group may be ragged (channel counts that are no multiple of 32):
      // it takes the masked one-value-per-load path, channels beyond the group read as zero
      const int nvalid = min(KBLK, min(a.kc, a.k_total - group * a.kc) - cbl * KBLK);
      const bool chunked = wide.value && nvalid == KBLK;
      if (ok) {
        const int n = (int)a.img_div.div((uint32_t)q);
        const int rem = q - n * img_pitch;
        const int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch;
        const int iy = a.phase_on_n ? y : y * a.sph + ctrl->ph_a[phase], ix = a.phase_on_n ? x : x * a.spw + ctrl->ph_b[phase];
        ok = y < a.H && x < a.W && iy < a.act_h && ix < a.act_w;
        src += n * a.act.s0 + ((long long)group * a.kc + cbl * KBLK) * a.act.s1 + (long long)iy * a.act.s2 + (long long)ix * a.act.s3 +
               (long long)group * a.act_group_extra;
      }
      if (chunked) {
        // Channels-last: the 32 channels of a pixel are 128 contiguous bytes.  Eight lanes fetch one
        // pixel (16 bytes each), so a load instruction covers four whole rows; lane r computed row r's
        // address above and hands it to the lanes that fetch it.
        const unsigned long long mine = ok ? reinterpret_cast<unsigned long long>(src) : 0ull;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4* ps = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, mine, 4 * i + (lane >> 3)));
          const float4 f = ps ? __ldg(ps + (lane & 7)) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[4 * i] = f.x; v[4 * i + 1] = f.y; v[4 * i + 2] = f.z; v[4 * i + 3] = f.w;
        }
      } else {
#pragma unroll
        for (int j = 0; j < KBLK; ++j) v[j] = (ok && j < nvalid) ? __ldg(src + j * s1) : 0.f;  // 32-bit offsets: two instructions per value
      }
      return Job{chunk, as, a_round, chunked};
    };
    auto place = [&](const Job& j, const float (&v)[KBLK]) {
      const uint32_t p_hi = tiles_base + j.as * a_stage_bytes, p_lo = p_hi + a_plane;
      const int r = j.chunk * 32 + lane;
      if (j.chunked) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int ri = j.chunk * 32 + 4 * i + (lane >> 3);  // strip_rows is a multiple of 8
          if (ri < a.strip_rows) {
            float h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split_tf32_fast(v[4 * i + e], h[e], l[e]);
            const int c4 = (lane & 7) * 4;  // first of this lane's four channels
            sts_f32x4(p_hi + sw128_offset(ri, c4), h[0], h[1], h[2], h[3]);
            if (CROSS_BF16) {
              sts_b32x2(p_lo + sw128_offset_bf16(ri, c4), pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
              sts_b32x2(p_lo + sw128_offset_bf16(ri, 32 + c4), pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
            } else {
              sts_f32x4(p_lo + sw128_offset(ri, c4), l[0], l[1], l[2], l[3]);
            }
          }
        }
      } else if (r < a.strip_rows) {
        if (CROSS_BF16) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {  // eight channels: two 16-byte chunks of the hi plane, one each of bf16(hi), bf16(lo)
            float h[8], l[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) split_tf32_fast(v[c * 8 + e], h[e], l[e]);
            sts_f32x4(p_hi + sw128_offset(r, c * 8), h[0], h[1], h[2], h[3]);
            sts_f32x4(p_hi + sw128_offset(r, c * 8 + 4), h[4], h[5], h[6], h[7]);
            sts_b32x4(p_lo + sw128_offset_bf16(r, c * 8), pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]),
                      pack_bf16x2(h[4], h[5]), pack_bf16x2(h[6], h[7]));
            sts_b32x4(p_lo + sw128_offset_bf16(r, 32 + c * 8), pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]),
                      pack_bf16x2(l[4], l[5]), pack_bf16x2(l[6], l[7]));
          }
        } else {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            float h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split_tf32_fast(v[c * 4 + e], h[e], l[e]);
            const uint32_t o = sw128_offset(r, c * 4);
            sts_f32x4(p_hi + o, h[0], h[1], h[2], h[3]);
            sts_f32x4(p_lo + o, l[0], l[1], l[2], l[3]);
          }
        }
      }
    };
    // The loop twice, by layout: with both ways of loading in one, the values of a pixel in one lane (NCHW, transposed matrices) paid for the uniform
    // tests of the other (products of 7 to 17 us with a transposed left matrix 2-3 % slower than with tests of every lane, now 1-3 % faster; 1x1 layers
    // of NCHW 0.98 of the time on average).
    auto produce = [&](auto wide) {
      if (aw < a_warps && aw < total_jobs) {
        constexpr bool AHEAD = AW > 8;  // eight warps serve layers of many taps, where the first strip is wanted at once
        float v[KBLK], ahead[AHEAD ? KBLK : 1];
        Job j = fetch(wide, aw, v), next = j;
#pragma unroll 1
        for (int job = aw;;) {
          const bool more = job + a_warps < total_jobs;
          if constexpr (AHEAD) if (more) next = fetch(wide, job + a_warps, ahead);
          const bool pa = PROF_ON(threadIdx.x == EPI_WARPS * 32);
          PROF_T0(pa);
          if (!mbar_wait(smem_u32(&ctrl->a_empty[j.as]), (j.round & 1) ^ 1, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) break;
          PROF_ADD(pa, 6);
          place(j, v);
          fence_proxy_async();
          mbar_arrive(smem_u32(&ctrl->a_full[j.as]));
          if (!more) break;
          job += a_warps;
          if constexpr (AHEAD) {
            j = next;
#pragma unroll
            for (int e = 0; e < KBLK; ++e) v[e] = ahead[e];
          } else {
            j = fetch(wide, job, v);
          }
        }
      }
    };
    if (vec_layout) produce(std::true_type{});
    else produce(std::false_type{});
  } else {
    // ------------------------------ epilogue ------------------------------
    // A warp reads the TMEM lane quarter (warp & 3); with 8 warps the 32-column chunks alternate
    // between warps w and w + 4.  One warp per scheduler runs at the latency of its dependent
    // instructions, so the per-element work is kept to a multiply-add and a store through a
    // running pointer; everything uniform (bias present, ragged last tile) is decided per chunk.
    const int quarter = warp & 3, half = warp >> 2;
    constexpr int HALVES = EPI_WARPS / 4;
    uint32_t t_count = 0;
    for (TileIter it(a); it.valid(); it.next(), ++t_count) {
      const int tile = it.tile();
      const TileCoord tc_ = tile_coord(a, tile);
      const int n_tile = tc_.n_tile, group = tc_.group, m_tile = tc_.m_tile;
      const int phase_n = (int)a.div_tiles_pp.div((uint32_t)n_tile);
      const int n0 = (n_tile - phase_n * a.tiles_pp) * BN;
      const int cols_valid = min(BN, a.nc - n0);
      const uint32_t ab = t_count & 1;
      const bool pe = PROF_ON(threadIdx.x == 0);
      // a dInput phase that no tap reaches (e.g. 1x1 filter with stride 2) gets zeros
      const bool has_taps = !a.phase_on_n || ctrl->tap_start[phase_n + 1] > ctrl->tap_start[phase_n];
      const int q = m_tile * BLOCK_M + quarter * 32 + lane;
      bool ok = q < a.q_total;
      long long obase = 0, res_off = 0;
      if (ok) {
        const long long n = a.img_div.div((uint32_t)q);
        const int rem = q - (int)n * img_pitch;
        int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch;
        ok = y < a.H && x < a.W;
        if (a.phase_on_n) { y = y * a.osh + ctrl->ph_a[phase_n]; x = x * a.osw + ctrl->ph_b[phase_n]; }
        ok = ok && y < a.out_h && x < a.out_w;
        res_off = n * a.res.s0 + ((long long)group * a.nc + n0) * a.res.s1 + (long long)y * a.res.s2 + (long long)x * a.res.s3;
        obase = a.out_rowmajor ? (((n * a.out_h + y) * a.out_w + x) * a.out_pitch + (long long)group * a.out_group + n0)
                               : (((n * a.out_channels + (long long)group * a.nc + n0) * a.out_h + y) * a.out_w + x);
      }
      const long long col_stride = a.out_rowmajor ? 1 : (long long)a.out_h * a.out_w;
      { PROF_T0(pe);
      if (!mbar_wait(smem_u32(&ctrl->acc_full[ab]), (t_count >> 1) & 1, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      PROF_ADD(pe, 8); }
      PROF_T0(pe);
      tc_fence_after();
      const uint32_t tmem_acc = tmem_base + ab * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      const int chunks = (cols_valid + 31) / 32;
      bool released = false;
#pragma unroll 1
      for (int ch = half; ch < chunks; ch += HALVES) {
        const int c0 = ch * 32;
        float v[32];
        tmem_ld32(tmem_acc + (uint32_t)c0, v);
        if (FUSE_HILO) {
          float v2[32];
          tmem_ld32(tmem_acc + (uint32_t)(BN + c0), v2);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += v2[j];
        }
        if (ch + HALVES >= chunks) {  // this warp's last read of the accumulator: hand it back early
          tc_fence_before();
          mbar_arrive(smem_u32(&ctrl->acc_empty[ab]));
          released = true;
        }
        const int nvalid = min(32, cols_valid - c0);
        if (!has_taps) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.f;
        }
        if (a.bias) {
          float bv = 0.f;  // lane j holds the bias of column c0 + j
          if (lane < nvalid) bv = a.beta * __ldg(a.bias + ((long long)group * a.nc + n0 + c0 + lane) * a.bias_stride);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaf(a.alpha, v[j], __shfl_sync(0xffffffffu, bv, j));
        } else if (a.alpha != 1.f) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= a.alpha;
        }
        if (a.res.ptr && ok) {
          // all loads of the chunk are issued before the first add (one warp per scheduler runs at
          // the latency of its dependent instructions)
          const float* rp = a.res.ptr + res_off + c0 * a.res.s1;
          float r[32];
          if (nvalid == 32 && a.res.s1 == 1 && ((reinterpret_cast<uintptr_t>(rp) & 15) == 0)) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 f = __ldg(reinterpret_cast<const float4*>(rp) + j);
              r[4 * j] = f.x; r[4 * j + 1] = f.y; r[4 * j + 2] = f.z; r[4 * j + 3] = f.w;
            }
          } else if (nvalid == 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = __ldg(rp + j * a.res.s1);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] = j < nvalid ? __ldg(rp + j * a.res.s1) : 0.f;
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += r[j];
        }
        if (a.relu) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
        }
        if (a.out_rowmajor && a.out_vec4 && nvalid == 32) {
          store_rows32(v, ok ? a.out + obase + c0 : nullptr, lane);
        } else if (ok) {
          float* p = a.out + obase + c0 * col_stride;
          if (nvalid == 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j, p += col_stride) *p = v[j];
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j, p += col_stride)
              if (j < nvalid) *p = v[j];
          }
        }
      }
      if (!released) {  // no chunk for this warp in a narrow last tile
        tc_fence_before();
        mbar_arrive(smem_u32(&ctrl->acc_empty[ab]));
      }
      PROF_ADD(pe, 9);
      if (pe) atomicAdd(a.prof + 10, 1ull);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (a.prof && threadIdx.x == 0) {  // spread of CTA start times and lifetimes (ns)
    const unsigned long long now = global_ns();
    atomicMin(a.prof + 11, prof_start);
    atomicMax(a.prof + 12, prof_start);
    atomicMax(a.prof + 13, now);
    atomicMin(a.prof + 14, now - prof_start);
    atomicMax(a.prof + 15, now - prof_start);
  }
}

// Split W[cout][cin/g][kh][kw] (any strides) into TF32 hi/lo parts laid out as the shared-memory
// images the MMA reads: image = [hi: bn rows x 128 B, SWIZZLE_128B][lo: same], row = output column of
// the tile (forward: co, dInput: ci; zero beyond nc), 32 reduction channels per row.  Images are
// ordered as the main loop consumes them: [group][n_tile][phase][channel block][tap of the phase],
// so a weight stage of the main kernel is one bulk copy from a running pointer.
//
// A thread takes four adjacent reduction channels of one row (a 16-byte piece of the swizzled row) and `per_thread` taps: the taps of a
// filter are adjacent in memory, and one tap per thread fetched every line once per tap (512 x 512 filters of 3x3 in the sibling kernel of conv_tc_tstrip.cu: 14.6 us, now 9.5).
// Neighbouring threads take neighbouring pieces of a row, or neighbouring rows where those are the adjacent values.
__global__ void __launch_bounds__(256) stage_weights_kernel(ConvGeom g, View4 w, int is_dx, int bn, int tiles_pp,
                                                            TapTable tt, float* __restrict__ out, long long total,
                                                            long long w_group_extra, int k_total, int rows_first, int per_thread) {
  // let the convolution kernel behind this one start its prologue and its activation strips now
  wait_previous();
  asm volatile("griddepcontrol.launch_dependents;");
  const long long i = blockIdx.x * 256ll + threadIdx.x;  // [group][tile][channel block][row, piece]
  if (i >= total) return;
  const int kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog;
  const int cpp = (kc + KBLK - 1) / KBLK;
  const int block = (int)(i / ((KBLK / 4) * bn)), in_block = (int)(i - (long long)block * ((KBLK / 4) * bn));
  // rows first: eight adjacent rows (32 bytes read) by four pieces (64 bytes written) to a warp; with a warp along the rows alone the
  // writes were 16 bytes of 32 lines (weight gradient of a 4096x512 -> 2048 linear layer 46.5 us, now 43.4)
  const int k = (rows_first ? in_block >> 3 & 7 : in_block % (KBLK / 4)) * 4;
  const int row = rows_first ? (in_block & 7) | in_block >> 6 << 3 : in_block / (KBLK / 4);
  const int tile_of_all = block / cpp, cbl = block - tile_of_all * cpp, grp = tile_of_all / tiles_pp, n_tile = tile_of_all - grp * tiles_pp;
  const int r = n_tile * bn + row, c = cbl * KBLK + k;
  // rows beyond the column count and channels beyond a ragged last block are zero
  const int valid = r < nc ? min(4, (int)min((long long)(kc - c), k_total - ((long long)grp * kc + c))) : 0;
  // forward: r is the output channel, c the input channel; dInput: the other way round
  const long long step = is_dx ? w.s0 : w.s1;
  const float* src = w.ptr + ((long long)grp * g.cog + (is_dx ? c : r)) * w.s0 + (long long)(is_dx ? r : c) * w.s1 + grp * w_group_extra;
  const int t0 = blockIdx.y * per_thread, t1 = min(tt.taps_total, t0 + per_thread);
  int phase = 0;
#pragma unroll 3
  for (int tap = t0; tap < t1; ++tap) {
    while (tap >= tt.start[phase + 1]) ++phase;
    const int ntap = tt.start[phase + 1] - tt.start[phase], rel = tap - tt.start[phase];
    // forward: [group][tile][phase][channel block][tap of the phase]; dInput: [group][phase][tile of the phase][channel block][tap of the phase]
    const long long image = is_dx ? (long long)(grp * tt.taps_total + tt.start[phase]) * tiles_pp * cpp + ((long long)n_tile * cpp + cbl) * ntap + rel
                                  : ((long long)tile_of_all * tt.taps_total + tt.start[phase]) * cpp + cbl * ntap + rel;
    const float* p = src + tt.ky[tap] * w.s2 + tt.kx[tap] * w.s3;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = j < valid ? __ldg(p + j * step) : 0.f;
    float hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) split_tf32(v[j], hi[j], lo[j]);
    float* plane = out + image * (bn * 64ll);
    *reinterpret_cast<float4*>(plane + sw128_offset(row, k) / 4) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    if (CROSS_BF16) {  // second plane: [bf16(lo) x32 | bf16(hi) x32] per row, pairing with the activations' [hi | lo]
      unsigned char* cross = reinterpret_cast<unsigned char*>(plane + bn * 32);
      *reinterpret_cast<uint2*>(cross + sw128_offset_bf16(row, k)) = make_uint2(pack_bf16x2(lo[0], lo[1]), pack_bf16x2(lo[2], lo[3]));
      *reinterpret_cast<uint2*>(cross + sw128_offset_bf16(row, 32 + k)) = make_uint2(pack_bf16x2(hi[0], hi[1]), pack_bf16x2(hi[2], hi[3]));
    } else {
      *reinterpret_cast<float4*>(plane + bn * 32 + sw128_offset(row, k) / 4) = make_float4(lo[0], lo[1], lo[2], lo[3]);
    }
  }
}

static inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }


// Any stride / padding / dilation in both directions; the reduction channels must come in blocks of
// 32 and there must be at least 16 output columns.  Forward groups the taps by the phase of the
// INPUT pixel they read; dInput by the phase of the OUTPUT (dX) pixel they contribute to: dX pixel
// s*r + a receives tap ky iff (ky*d - pad) = a (mod s), from dY row r - floor((ky*d - pad) / s).
StripPlan plan_strip_geometry(const ConvGeom& g, bool is_dx) {
  StripPlan p;
  const int kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog;
  // a ragged last channel block is padded with zeros; below 16 channels the padding would more than
  // double the work and the CUDA-core kernels are the better choice
  if (kc < 16 || nc < 16 || g.kh * g.kw > MAX_TAPS) return p;
  if (g.sh * g.sw > MAX_PHASES || g.sh > 255 || g.sw > 255) return p;
  p.sph = g.sh; p.spw = g.sw;
  p.act_h = is_dx ? g.oh : g.h; p.act_w = is_dx ? g.ow : g.w;
  p.out_h = is_dx ? g.h : g.oh; p.out_w = is_dx ? g.w : g.ow;
  // the grid covers the unstrided tensor and every phase sub-image of the strided one
  p.gh = std::max(g.oh, (g.h + p.sph - 1) / p.sph);
  p.gw = std::max(g.ow, (g.w + p.spw - 1) / p.spw);
  // taps -> (phase, whole-pixel offset); forward reads x at s*o - pad + k*d, dInput reads dy at i + pad - k*d
  struct Tap { int phase, dr, dc, ky, kx; };
  Tap taps[MAX_TAPS];
  int ntaps = 0, dr_lo = 0, dr_hi = 0, dc_lo = 0, dc_hi = 0;
  for (int ky = 0; ky < g.kh; ++ky)
    for (int kx = 0; kx < g.kw; ++kx) {
      const int oy = ky * g.dh - g.ph, ox = kx * g.dw - g.pw;
      const int fr = floor_div(oy, p.sph), fc = floor_div(ox, p.spw);
      const int dr = is_dx ? -fr : fr, dc = is_dx ? -fc : fc;
      taps[ntaps++] = Tap{(oy - fr * p.sph) * p.spw + (ox - fc * p.spw), dr, dc, ky, kx};
      dr_lo = std::min(dr_lo, dr); dr_hi = std::max(dr_hi, dr);
      dc_lo = std::min(dc_lo, dc); dc_hi = std::max(dc_hi, dc);
    }
  p.pr = std::max(-dr_lo, dr_hi);
  p.pc = std::max(-dc_lo, dc_hi);
  if ((long long)g.n * (p.gh + p.pr) * (p.gw + p.pc) > 2147483647ll - (1 << 20)) return p;  // 32-bit pixel indices
  const int row_pitch = p.gw + p.pc;
  TapTable& tt = p.tt;
  memset(&tt, 0, sizeof tt);
  int lo = 0, hi = 0;
  for (int phase = 0; phase < p.sph * p.spw; ++phase) {
    int count = 0;
    for (int t = 0; t < ntaps; ++t)
      if (taps[t].phase == phase) {
        const int i = tt.taps_total++;
        tt.ky[i] = (unsigned char)taps[t].ky; tt.kx[i] = (unsigned char)taps[t].kx;
        tt.shift[i] = taps[t].dr * row_pitch + taps[t].dc;
        lo = std::min(lo, tt.shift[i]); hi = std::max(hi, tt.shift[i]);
        ++count;
      }
    if (count == 0 && !is_dx) continue;  // forward: a phase no tap reads is never staged (dInput: it is zero-filled)
    tt.a[tt.n_phase] = (unsigned char)(phase / p.spw); tt.b[tt.n_phase] = (unsigned char)(phase % p.spw);
    tt.start[tt.n_phase + 1] = (unsigned char)tt.taps_total;
    ++tt.n_phase;
  }
  p.shift_lo = lo; p.shift_hi = hi;
  p.halo = -lo;
  p.ok = true;
  return p;
}

// Modelled time of `tiles` tiles of `bn` columns, in arbitrary units: a narrow tile feeds the tensor core less per shared-memory byte,
// and with one tap per strip stages as many activations for fewer products (4096 rows: 1.25, 0.95 and 0.63 us per 32-column block).
static double width_cost(long long tiles, int bn, bool single_tap) {
  const double eff = bn == 256 ? 1.0 : bn == 128 ? (single_tap ? 0.66 : 0.85) : (single_tap ? 0.5 : 0.55);
  return (double)div_up64(tiles, sm_count()) * bn / eff;
}

static StripPlan make_plan(const ConvGeom& g, bool is_dx) {
  StripPlan p = plan_strip_geometry(g, is_dx);
  if (!p.ok) return p;
  p.ok = false;
  const int nc = is_dx ? g.cig : g.cog;
  p.strip_rows = (BLOCK_M + p.shift_hi - p.shift_lo + 7) / 8 * 8;
  const int a_stage = p.strip_rows * 256;
  // Column tile: the widest tile makes the best use of shared-memory bandwidth per MMA, but a small
  // image gives few 128-pixel row tiles; pick the width with the lowest modelled time
  // waves(tiles / SMs) * width / efficiency(width).
  const long long tiles_m = div_up64((long long)g.n * (p.gh + p.pr) * (p.gw + p.pc), BLOCK_M);
  double best_cost = 0.0;
  bool single_tap = true;  // no phase has more than one tap (1x1 filters): every staged strip feeds one tap's MMAs only
  for (int ph = 0; ph < p.tt.n_phase; ++ph) single_tap = single_tap && p.tt.start[ph + 1] - p.tt.start[ph] <= 1;
  for (int bn : {256, 128, 64}) {
    if (bn > 64 && nc <= bn / 2) continue;  // do not pad the column tile by more than 2x
    const int w_stage = bn * 256;
    for (int a_stages : {4, 3, 2, 1}) {
      if (a_stages > 2 && a_stages * a_stage > SMEM_LIMIT / 2 && !single_tap) continue;  // deep strip pipelines only while cheap
                                                                                          // (or while the producers set the pace)
      const int left = SMEM_LIMIT - a_stages * a_stage;
      if (left < 2 * w_stage) continue;
      const long long tiles = tiles_m * ((nc + bn - 1) / bn) * g.groups * (is_dx ? p.sph * p.spw : 1);
      const double cost = width_cost(tiles, bn, single_tap);
      if (!p.ok || cost < best_cost) {
        best_cost = cost;
        p.ok = true;
        p.bn = bn;
        p.a_stages = a_stages;
        p.w_stages = std::min(MAX_STAGES, left / w_stage);
        p.smem = a_stages * a_stage + p.w_stages * w_stage + 1024 + (int)sizeof(Ctrl) + 64;
      }
      break;  // the deepest strip pipeline that fits is the one to use for this width
    }
  }
  return p;
}
static const StripPlan& plan_strip(const ConvGeom& g, bool is_dx) {
  thread_local PlanCache<StripPlan> cache;
  return cache.get(g, is_dx, [&] { return make_plan(g, is_dx); });
}

}  // namespace tcs

bool strip_supported(const ConvGeom& g, int phase) {
  if (phase != B200_PHASE_FORWARD && phase != B200_PHASE_DINPUT) return false;
  return tcs::plan_strip(g, phase == B200_PHASE_DINPUT).ok;
}
int strip_column_tile(const ConvGeom& g, bool is_dx) {
  const tcs::StripPlan& p = tcs::plan_strip(g, is_dx);
  return p.ok ? p.bn : 0;
}
// Waves of tiles times filter stages of a tile times the measured time of a stage at that width (layers of a few waves), and the
// prologue and epilogue of a wave.
double strip_time(const ConvGeom& g, bool is_dx, long long* tiles) {
  const tcs::StripPlan& p = tcs::plan_strip(g, is_dx);
  if (!p.ok) return 1e30;
  const int kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog, phases = is_dx ? std::max(1, p.tt.n_phase) : 1;
  const long long count = div_up64((long long)g.n * (p.gh + p.pr) * (p.gw + p.pc), tcs::BLOCK_M) * ((nc + p.bn - 1) / p.bn) * g.groups * phases;
  if (tiles) *tiles = count;
  const double stages = (double)((kc + 31) / 32) * p.tt.taps_total / phases;
  return (double)div_up64(count, sm_count()) * (stages * (p.bn == 256 ? 0.70 : p.bn == 128 ? 0.48 : 0.38) + 2.0) + 5.0;
}
// Bytes of the weight stage images: hi and lo planes with the column count padded to the tile width.
// The width depends on the image count, so take the largest over the widths the plan may pick.
size_t strip_workspace(const ConvGeom& g, int phase) {
  const bool is_dx = phase == B200_PHASE_DINPUT;
  const size_t kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog;
  size_t cols = 0;
  for (size_t bn : {256, 128, 64}) cols = std::max(cols, (nc + bn - 1) / bn * bn);
  return 2 * sizeof(float) * (size_t)g.groups * cols * ((kc + 31) / 32 * 32) * g.kh * g.kw;  // ragged last channel block padded
}

template <int BN, int AW>
static int launch_strip_aw(const tcs::StripArgs& a, int grid, int smem, cudaStream_t st) {
  // opt in once (thread-safe) to the full 227 KB of dynamic shared memory for this instantiation
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(tcs::conv_strip_kernel<BN, AW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(tcs::strip_threads(AW)); cfg.dynamicSmemBytes = (size_t)smem; cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  if (a.wait_for_images) { cfg.attrs = &attr; cfg.numAttrs = 1; }
  B200_CUDA(cudaLaunchKernelEx(&cfg, tcs::conv_strip_kernel<BN, AW>, a));
  count_launch();
  return launch_check("conv_strip_kernel");
}
template <int BN>
static int launch_strip(const tcs::StripArgs& a, int grid, int smem, cudaStream_t st) {
  return a.wide_producers ? launch_strip_aw<BN, 12>(a, grid, smem, st) : launch_strip_aw<BN, 8>(a, grid, smem, st);
}

// The kernel forms element offsets inside the activation tensor in 32 bits: true when the view's
// extent (with the 64 channels a ragged block may look ahead) stays below 2^31 elements.
bool strip_view_addressable(const ConvGeom& g, bool is_dx, const View4& act, const StripBatch* batch) {
  const long long an = g.n, ac = is_dx ? g.cout : g.cin, ah = is_dx ? g.oh : g.h, aw = is_dx ? g.ow : g.w;
  const long long span = (an - 1) * std::llabs(act.s0) + (ac - 1) * std::llabs(act.s1) +
                         (ah - 1) * std::llabs(act.s2) + (aw - 1) * std::llabs(act.s3) +
                         (batch ? (g.groups - 1) * std::llabs(batch->act_group_extra) : 0);
  return span <= 2147483647ll - 64 * std::llabs(act.s1);
}

int strip_conv(const ConvGeom& g, bool is_dx, View4 act, View4 w, const float* bias, long long bias_stride, float* out,
               void* ws, size_t ws_bytes, cudaStream_t st, bool rowmajor, float alpha, float beta, const float* staged_images,
               const StripPostOps* post, const StripBatch* batch) {
  using namespace tcs;
  const StripPlan& plan = plan_strip(g, is_dx);
  if (!plan.ok) return fail(B200_EUNSUPPORTED, "strip kernel does not take this geometry");
  const int kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog;
  const int tiles_pp = (nc + plan.bn - 1) / plan.bn;  // column tiles (per output phase in dInput)
  const int tiles_n = is_dx ? tiles_pp * plan.tt.n_phase : tiles_pp;
  const int cpp = (kc + KBLK - 1) / KBLK;  // channel blocks per group, the last one possibly ragged
  const int k_total = batch && batch->k_total ? (int)batch->k_total : g.groups * kc;
  const long long wcount = (long long)g.groups * tiles_pp * plan.bn * cpp * KBLK * plan.tt.taps_total;  // per plane
  const float* wp = staged_images;
  bool staged_here = false;
  if (!wp) {
    if (!ws || ws_bytes < 2 * sizeof(float) * (size_t)wcount || (reinterpret_cast<uintptr_t>(ws) & 15))
      return fail(B200_EWORKSPACE, "tcgen05 convolution needs a 16-byte aligned workspace of %zu bytes (got %zu)",
                  2 * sizeof(float) * (size_t)wcount, ws_bytes);
    const int taps = plan.tt.taps_total;
    const long long threads = wcount / taps / 4;
    const int per_thread = staged_taps(threads, taps);
    launch_next(stage_weights_kernel, dim3((unsigned)div_up64(threads, 256), (unsigned)((taps + per_thread - 1) / per_thread)), 256, 0, st, 
        g, w, is_dx ? 1 : 0, plan.bn, tiles_pp, plan.tt, (float*)ws, threads, batch ? batch->w_group_extra : 0, k_total,
        std::llabs(is_dx ? w.s1 : w.s0) < std::llabs(is_dx ? w.s0 : w.s1) ? 1 : 0, per_thread);
    count_launch();
    if (int rc = launch_check("stage_weights_kernel")) return rc;
    wp = (const float*)ws;
    staged_here = true;
  }
  if (reinterpret_cast<uintptr_t>(wp) & 15) return fail(B200_EINVAL, "weight stage images must be 16-byte aligned");
  if (!strip_view_addressable(g, is_dx, act, batch))
    return fail(B200_EUNSUPPORTED, "strip kernel: activation tensor too large for 32-bit element offsets");
  StripArgs a{};
  a.g = g; a.act = act; a.wp = wp; a.bias = bias; a.bias_stride = bias_stride; a.out = out;
  a.H = plan.gh; a.W = plan.gw; a.pr = plan.pr; a.pc = plan.pc;
  a.act_h = plan.act_h; a.act_w = plan.act_w; a.out_h = plan.out_h; a.out_w = plan.out_w;
  a.sph = is_dx ? 1 : plan.sph; a.spw = is_dx ? 1 : plan.spw;
  a.osh = is_dx ? plan.sph : 1; a.osw = is_dx ? plan.spw : 1;
  a.phase_on_n = is_dx ? 1 : 0;
  a.tiles_pp = tiles_pp;
  a.tt = plan.tt;
  a.kc = kc;
  a.nc = nc;
  a.out_channels = is_dx ? g.cin : g.cout;
  a.k_total = k_total;
  a.act_group_extra = batch ? batch->act_group_extra : 0;
  a.out_pitch = batch ? batch->out_pitch : a.out_channels;
  a.out_group = batch ? batch->out_group : nc;
  a.cb_per_phase = cpp;
  a.cblocks = (is_dx ? 1 : plan.tt.n_phase) * a.cb_per_phase;
  a.images_per_tile = a.cb_per_phase * plan.tt.taps_total;
  a.tiles_n = tiles_n;
  a.q_total = (int)((long long)g.n * (a.H + a.pr) * (a.W + a.pc));
  a.img_div = FastDiv((uint32_t)((a.H + a.pr) * (a.W + a.pc)));
  a.row_div = FastDiv((uint32_t)(a.W + a.pc));
  a.tiles_m = (int)div_up64(a.q_total, BLOCK_M);
  a.halo = plan.halo; a.strip_rows = plan.strip_rows; a.a_stages = plan.a_stages; a.w_stages = plan.w_stages;
  {
    // one tap per staged strip (1x1 filters): the MMAs wait for the producers, so twelve of them run
    int most = 0;
    for (int ph = 0; ph < plan.tt.n_phase; ++ph) most = std::max(most, (int)plan.tt.start[ph + 1] - (int)plan.tt.start[ph]);
    // ... and only while the reduction side is the larger one (256 -> 64 channels forward: 90 -> 69 us); with more output
    // than input (its dInput) the epilogue's stores set the pace and the extra warps only take registers from it (61 -> 80 us)
    // (row-major stores are whole lines and cost less: 1024 -> 1024 columns of a GEMM 198 -> 157 us, but 80 -> 1024 is faster with eight)
    a.wide_producers = most <= 1 && (kc > nc || (rowmajor && a.cblocks >= 16)) ? 1 : 0;
  }
  const int chunks = (a.strip_rows + 31) / 32;
  const long long tiles_total = (long long)a.tiles_m * a.tiles_n * g.groups;
  if (tiles_total * a.cblocks * chunks > 2147483647ll - (1 << 20))
    return fail(B200_EUNSUPPORTED, "strip kernel: tile count exceeds 32-bit job indices");
  a.tiles_total = (int)tiles_total;
  // units of all column tiles of a pixel-row tile while that still leaves every SM two or more units
  a.unit = (tiles_total / a.tiles_n >= 2ll * sm_count()) ? a.tiles_n : 1;
  a.units = a.tiles_total / a.unit;
  a.m_fastest = (a.unit == 1 && a.tiles_n > 1) ? 1 : 0;
  a.div_unit = FastDiv((uint32_t)a.unit);
  a.div_tiles_n = FastDiv((uint32_t)a.tiles_n); a.div_tiles_m = FastDiv((uint32_t)a.tiles_m);
  a.div_tiles_pp = FastDiv((uint32_t)a.tiles_pp); a.div_chunks = FastDiv((uint32_t)chunks);
  a.div_cblocks = FastDiv((uint32_t)a.cblocks); a.div_cbpp = FastDiv((uint32_t)a.cb_per_phase);
  a.div_a_stages = FastDiv((uint32_t)a.a_stages);
  a.wait_for_images = staged_here ? 1 : 0;
  if (post && !is_dx) { a.res = post->residual; a.relu = post->relu; }
  a.out_rowmajor = rowmajor ? 1 : 0;
  a.alpha = alpha; a.beta = beta;
  a.out_vec4 = rowmajor && a.out_pitch % 4 == 0 && a.out_group % 4 == 0 && plan.bn % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 &&
               a.nc % 4 == 0;
  // a plain product with wide column tiles: one tap per strip leaves shared memory as the bound, which the kernel with A in tensor memory
  // relieves (16384x1024 x 1024x1024: 144 -> 131 us); below 65 columns its tiles would be half empty
  if (rowmajor && !is_dx && !post && g.n == 1 && g.h == 1 && g.kh * g.kw == 1 && plan.bn >= 128) {
    gt::GemmArgs m{};
    m.A = act.ptr; m.a_m = act.s3; m.a_k = act.s1; m.a_group = kc * act.s1 + a.act_group_extra;
    m.images = wp; m.bias = bias; m.bias_stride = bias_stride;
    m.C = out; m.c_pitch = a.out_pitch; m.c_group = a.out_group;
    m.M = g.w; m.N = nc; m.kc = kc; m.k_total = k_total; m.kblocks = cpp;
    m.tiles_m = a.tiles_m; m.tiles_n = a.tiles_n; m.tiles = a.tiles_total; m.m_fastest = a.unit == 1;
    const bool lines = act.s1 == 1 || act.s3 == 1;
    m.along_k = act.s1 == 1;
    m.pieces16 = (m.along_k ? act.s3 : act.s1) % 4 == 0 && (!m.along_k || kc % 4 == 0) && m.a_group % 4 == 0 && (reinterpret_cast<uintptr_t>(act.ptr) & 15) == 0;
    m.vec_out = a.out_vec4; m.wait_for_images = a.wait_for_images; m.alpha = alpha; m.beta = beta;
    // rows of A along m that are not 16-byte aligned are better read straight into the strip producers' registers (51 against 66 us for
    // 1111x16000 x 16000x77), as is A without a contiguous dimension
    if (lines && (m.along_k || m.pieces16)) return gt::run(m, plan.bn, st);
  }
  // 1x1 layers of whole planes whose filter fits shared memory, large enough for two waves of tiles and with little of a tile empty (134 channels in
  // a tile of 256 from 32: 12.8 us in the strip kernel, 13.9 in the other)
  const int pixels = a.H * a.W;
  if (!rowmajor && !batch && (!post || (!post->residual.ptr && !post->relu)) && g.groups == 1 && g.kh * g.kw == 1 && g.sh == 1 && g.sw == 1 && g.ph == 0 && g.pw == 0 &&
      tiles_n == 1 && 4 * nc >= (plan.bn == 256 ? 3 : 2) * plan.bn && (long long)cpp * plan.bn * 256 <= gt::PLANES_B && act.s3 == 1 && (act.s2 == a.W || a.H == 1) && act.s1 % 4 == 0 && act.s0 % 4 == 0 &&
      (reinterpret_cast<uintptr_t>(act.ptr) & 15) == 0 && pixels >= 512 && (long long)g.n * ((pixels + 127) / 128) >= 2ll * sm_count() &&
      !getenv("B200_CONV_TC_VARIANT")) {
    note_kernel(is_dx ? "tc_planes_dinput" : "tc_planes_forward");
    gt::GemmArgs m{};
    m.planes = 1;
    m.A = act.ptr; m.a_m = 1; m.a_k = act.s1; m.a_group = act.s0;
    m.images = wp; m.bias = bias; m.bias_stride = bias_stride;
    m.C = out; m.c_pitch = pixels; m.c_group = (long long)nc * pixels;
    m.M = pixels; m.N = nc; m.kc = kc; m.k_total = kc; m.kblocks = cpp;
    m.tiles_m = (pixels + 127) / 128; m.tiles_n = 1; m.tiles = g.n * m.tiles_m; m.m_fastest = 1;
    m.pieces16 = 1; m.wait_for_images = a.wait_for_images; m.alpha = 1.f; m.beta = 1.f;
    return gt::run(m, plan.bn, st);
  }
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  static unsigned long long* prof_buf = nullptr;
  const char* prof_env = getenv("B200_STRIP_PROFILE");
  const bool profiling = B200_ROLE_PROFILE && prof_env && prof_env[0] == '1';
  if (profiling) {
    if (!prof_buf) B200_CUDA(cudaMalloc(&prof_buf, 16 * sizeof(unsigned long long)));
    B200_CUDA(cudaMemsetAsync(prof_buf, 0, 16 * sizeof(unsigned long long), st));
    B200_CUDA(cudaMemsetAsync(prof_buf + 11, 0xFF, sizeof(unsigned long long), st));
    B200_CUDA(cudaMemsetAsync(prof_buf + 14, 0xFF, sizeof(unsigned long long), st));
    a.prof = prof_buf;
  }
  const int grid = std::min(a.units, sm_count());
  if (profiling) {
    const int rc = plan.bn == 64 ? launch_strip<64>(a, grid, plan.smem, st)
                 : plan.bn == 128 ? launch_strip<128>(a, grid, plan.smem, st) : launch_strip<256>(a, grid, plan.smem, st);
    unsigned long long h[16];
    B200_CUDA(cudaStreamSynchronize(st));
    B200_CUDA(cudaMemcpy(h, prof_buf, sizeof h, cudaMemcpyDeviceToHost));
    fprintf(stderr, "[strip profile, CTA 0, cycles] bn=%d a_stages=%d w_stages=%d tiles=%llu | mma: wait_acc %llu wait_a %llu wait_w %llu issue %llu | "
            "w: wait_empty %llu convert %llu | a: wait_empty %llu stage_total %llu | epi: wait_acc %llu drain %llu | ns: CTA starts spread %llu, first start to last end %llu, CTA lifetime min %llu max %llu\n",
            plan.bn, plan.a_stages, plan.w_stages, h[10], h[0], h[1], h[2], h[3], h[4], h[5], h[6], h[7], h[8], h[9], h[12] - h[11], h[13] - h[11], h[14], h[15]);
    return rc;
  }
  if (plan.bn == 64) return launch_strip<64>(a, grid, plan.smem, st);
  if (plan.bn == 128) return launch_strip<128>(a, grid, plan.smem, st);
  return launch_strip<256>(a, grid, plan.smem, st);
}


// C = alpha * the sum of the split-K partial products (in order) + beta * bias[column]; V adjacent values per thread
template <int V>
__global__ void __launch_bounds__(256) gemm_finalize_kernel(const float* partial, int splits, long long count, int N, FastDiv by_n, float alpha,
                                                            const float* __restrict__ bias, float beta, float* __restrict__ C) {
  const long long i = (blockIdx.x * 256ll + threadIdx.x) * V;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (i >= count) return;
  float v[V] = {};
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float* p = partial + s * count + i;
    if (V == 4) {
      const float4 f = *reinterpret_cast<const float4*>(p);
      v[0] += f.x; v[1 % V] += f.y; v[2 % V] += f.z; v[3 % V] += f.w;
    } else {
      v[0] += *p;
    }
  }
#pragma unroll
  for (int j = 0; j < V; ++j) v[j] *= alpha;
  if (bias) {
    const long long row = count < (1ll << 31) ? by_n.div((uint32_t)i) : i / N;
    const int col = (int)(i - row * N);
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] = fmaf(beta, __ldg(bias + col + j), v[j]);
  }
  if (V == 4) *reinterpret_cast<float4*>(C + i) = make_float4(v[0], v[1 % V], v[2 % V], v[3 % V]);
  else C[i] = v[0];
}

int gemm_finalize(const float* parts, int splits, long long M, long long N, float alpha, const float* bias, float beta, float* C, cudaStream_t st) {
  const long long count = M * N;
  const bool vec = N % 4 == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)div_up64(vec ? count / 4 : count, 256)); cfg.blockDim = dim3(256); cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  B200_CUDA(cudaLaunchKernelEx(&cfg, vec ? gemm_finalize_kernel<4> : gemm_finalize_kernel<1>, parts, splits, count, (int)N, FastDiv((uint32_t)N), alpha, bias, beta, C));
  count_launch();
  return launch_check("gemm_finalize_kernel");
}

static ConvGeom gemm_geometry(long long M, long long N, long long K, int groups) {
  ConvGeom g{};
  g.n = 1; g.cin = (int)(groups * K); g.cout = (int)(groups * N); g.h = 1; g.w = (int)M; g.kh = g.kw = 1; g.oh = 1; g.ow = (int)M;
  g.sh = g.sw = 1; g.ph = g.pw = 0; g.dh = g.dw = 1; g.groups = groups; g.cig = (int)K; g.cog = (int)N;
  return g;
}

// Slices of the reduction for a product whose tiles leave SMs idle.  Modelled time in microseconds: waves of (32-column blocks of the
// reduction x the measured time of one at that tile width + prologue and last stores), and for two slices and more a second launch
// that moves the partial products.  4096x2048 x 2048x512: 74 us as 128 tiles of 128 columns, 57 as two slices of 64 tiles of 256;
// 2048x4096 x 4096x512: 84 -> 53 with four; 320x8000 x 8000x320: 147 -> 45.
static int gemm_splits(long long M, long long N, long long K, long long* k_slice) {
  int best = 1;
  double best_time = 0.0;
  *k_slice = K;
  const long long tiles_m = div_up64(M, tcs::BLOCK_M);
  for (int splits = 1; splits <= 32 && (splits == 1 || (tiles_m * (splits - 1) < 2ll * sm_count() && K >= 64ll * splits)); ++splits) {
    const long long slice = splits == 1 ? K : (div_up64(K, splits) + 31) / 32 * 32;
    if (splits > 1 && (div_up64(K, slice) != splits || splits * std::max(N, slice) > 2147483647ll)) continue;
    double cost = 0.0, time = 0.0;  // of the width that plan_strip takes
    for (int bn : {256, 128, 64}) {
      if (bn > 64 && N <= bn / 2) continue;
      const long long tiles = tiles_m * div_up64(N, bn) * splits;
      const double c = tcs::width_cost(tiles, bn, true);
      if (cost != 0.0 && c >= cost) continue;
      cost = c;
      time = (double)div_up64(tiles, sm_count()) * ((double)div_up64(slice, 32) * (bn == 256 ? 1.25 : bn == 128 ? 0.95 : 0.63) + 4.0);
    }
    if (splits > 1) time += 3.0 + splits * 2e-6 * (double)M * (double)N;
    if (best_time == 0.0 || time < best_time) { best_time = time; best = splits; *k_slice = slice; }
  }
  return best;
}

// C[M,N] = alpha * A*B + beta * bias[n] as a 1x1 convolution over an M-pixel image with K input and N
// output channels, written row-major; slices of K ride on the kernel's group dimension, each with its own partial product.  Takes
// K >= 16 and N >= 16 (a ragged last block of K is padded with zeros); anything else is the caller's CUDA-core kernel.  The staged copy
// of B and the partial products come from the caching allocator and are released on `st`.
int tc_gemm(long long M, long long N, long long K, const float* A, long long sa0, long long sa1, const float* B,
            long long sb0, long long sb1, const float* bias, float alpha, float beta, float* C, cudaStream_t st) {
  if (K < 16 || N < 16 || M > 2147483647ll || N > 2147483647ll || K > 2147483647ll)
    return fail(B200_EUNSUPPORTED, "tcgen05 GEMM is incompatible with this shape (needs K >= 16 and N >= 16)");
  long long slice;
  int splits = gemm_splits(M, N, K, &slice);
  ConvGeom g = gemm_geometry(M, N, slice, splits);
  if (!tcs::plan_strip(g, false).ok) return fail(B200_EUNSUPPORTED, "tcgen05 GEMM is incompatible with this shape");
  const View4 act{A, 0, sa1, 0, sa0};   // [n=1][c=k][h=1][w=m]
  const View4 wv{B, sb1, sb0, 0, 0};    // [co=n][ci=k][1][1]
  void* ws = nullptr;
  size_t images = (strip_workspace(g, B200_PHASE_FORWARD) + 255) & ~(size_t)255;
  int status = b200_malloc(&ws, images + (splits > 1 ? (size_t)splits * M * N * sizeof(float) : 0), st);
  if (status && splits > 1) {           // no room for the partial products: one slice
    splits = 1;
    slice = K;
    g = gemm_geometry(M, N, K, 1);
    if (!tcs::plan_strip(g, false).ok) return status;
    images = (strip_workspace(g, B200_PHASE_FORWARD) + 255) & ~(size_t)255;
    status = b200_malloc(&ws, images, st);
  }
  if (status) return status;
  StripBatch sb;
  sb.w_group_extra = slice * sb0 - N * sb1;  // slice s starts s*slice rows down B
  sb.out_pitch = N;
  sb.out_group = M * N;
  sb.k_total = K;
  if (!bias || beta == 0.f) { bias = nullptr; beta = 0.f; }
  int rc;
  if (splits == 1) {
    rc = strip_conv(g, false, act, wv, bias, 1, C, ws, images, st, true, alpha, beta);
  } else {
    float* parts = reinterpret_cast<float*>(static_cast<char*>(ws) + images);
    rc = strip_conv(g, false, act, wv, nullptr, 1, parts, ws, images, st, true, alpha, 0.f, nullptr, nullptr, &sb);
    if (!rc) rc = gemm_finalize(parts, splits, M, N, 1.f, bias, beta, C, st);
  }
  b200_free(ws, st);
  return rc;
}

// C[b] = A[b] * B[b] for every batch in ONE launch pair: the batch rides on the kernel's group
// dimension (each group has its own weight images and its own block of reduction channels), with the
// three per-group offsets of StripBatch standing in for the grouped convolution's channel arithmetic.
int tc_bmm(long long batch, long long M, long long N, long long K, const float* A, long long sa_b, long long sa0, long long sa1,
           const float* B, long long sb_b, long long sb0, long long sb1, float* C, cudaStream_t st) {
  if (K < 16 || N < 16 || M > 2147483647ll || batch * N > 2147483647ll || batch * K > 2147483647ll || batch > 65535)
    return fail(B200_EUNSUPPORTED, "tcgen05 batched GEMM is incompatible with this shape (needs K >= 16 and N >= 16)");
  const ConvGeom g = gemm_geometry(M, N, K, (int)batch);
  if (!tcs::plan_strip(g, false).ok) return fail(B200_EUNSUPPORTED, "tcgen05 batched GEMM is incompatible with this shape");
  const View4 act{A, 0, sa1, 0, sa0};   // [n=1][c=(b,k)][h=1][w=m]
  const View4 wv{B, sb1, sb0, 0, 0};    // [co=(b,n)][ci=k][1][1]
  StripBatch sb;
  sb.act_group_extra = sa_b - K * sa1;  // group b starts b*K channels in: b*K*sa1 of the way to A[b]
  sb.w_group_extra = sb_b - N * sb1;
  sb.out_pitch = N;
  sb.out_group = M * N;
  void* ws = nullptr;
  const size_t ws_bytes = strip_workspace(g, B200_PHASE_FORWARD);
  if (int rc = b200_malloc(&ws, ws_bytes, st)) return rc;
  const int rc = strip_conv(g, false, act, wv, nullptr, 1, C, ws, ws_bytes, st, true, 1.f, 0.f, nullptr, nullptr, &sb);
  b200_free(ws, st);
  return rc;
}

}  // namespace b200

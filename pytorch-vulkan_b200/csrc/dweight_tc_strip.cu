// tcgen05 dWeight kernel for filters up to eight taps wide (any stride, padding, dilation, groups;
// at least 16 channels on both sides), FP32 via 3xTF32, with both operands in shared memory: 1x1 filters, and what the
// tensor-memory kernel (dweight_tc_tmem.cu), which is tried first, does not take.
//
//   dW[co][ci][ky][kx] = sum over grid pixels q of  dY[q][co] * X_phase(ky,kx)[q + shift(ky,kx)][ci]
//
// The contraction runs over pixels, so both operands are staged pixel-major ("MN-major" for the
// tensor core): one 128-byte shared-memory row per pixel holding 32 channels, TF32 hi and lo
// planes, written in the 128-byte/32-byte-base swizzle that tcgen05 requires for 32-bit MN-major
// operands.  The M dimension of the MMA (4 blocks of 32 rows, at a programmable byte stride) is
// filled in one of two ways (plan_dw_strip):
//   strip   stride 1, output as large as the input: the vertical tap (ky) is a start-address
//           offset of ONE staged input strip and, with a block stride of `dilation_w` rows, its
//           four M blocks are the horizontal taps kx = 0..3: a single tcgen05.mma of shape
//           128 x BN x 8 accumulates up to four taps of a 32-channel block at once.  Two channel
//           blocks per CTA (two accumulators in TMEM) share every staged dY block.
//   blocks  everything else: four exact 32-pixel blocks per K block, the taps kx of one channel
//           block (each read from its own column phase and offset of a strided input) or four
//           channel blocks of a 1x1 filter.
// Every CTA owns one (channel tile, ky, column tile, pixel split); its 16 producer warps stream the
// input and dY blocks straight from the caller's strided views, one 32-row block per warp, several
// K blocks in flight.  Split partials land in [split][cout][kh*kw][cin/g] (channel fastest: the
// epilogue's lanes store neighbouring floats) and finalize_partials_kernel sums them in ascending
// split order (no atomics, run-to-run identical) while transposing into dW.
//
// Replaces csrc/shaders/conv2d_backward_weight_tiled_body.glsl:42-70 and
// conv2d_backward_weight_finalize.comp:9-18 of the reference for these geometries.
#include "common.cuh"
#include "plan_cache.cuh"
#include "dweight_plan.cuh"
#include "dweight_stage.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <mutex>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace b200 {
namespace tcdw {
using namespace tc;

// BF16 cross terms (tc_common.cuh) in this kernel: bf16 planes of 64-byte rows (SWIZZLE_64B) with the
// same row-shift and block-stride tricks as the TF32 planes.  The kernel is bound by what its producers
// pull from L2 (about 15-20 bytes per clock and SM for 128-byte pieces, loads or bulk copies alike), so
// the cross terms pay only where they cut that traffic: an accumulator then takes BN instead of 2*BN
// TMEM columns, and FOUR channel blocks can share every staged dY block.  Measured: 128/256/512-channel
// 3x3 layers 12-20 % faster, 64-channel, 1x1 and strided ones 2-8 % slower -- so the plan turns them
// on exactly when it can use four accumulators (plan_dw_strip); everything else runs 3xTF32.

constexpr int KP = 32;          // pixels per K block (four K=8 MMA steps)
constexpr int XR = 40;          // rows of one staged input strip: KP + margin for the horizontal taps
constexpr int XOFF = 4;         // row of the strip that corresponds to the first pixel of the K block
constexpr int PRODUCER_WARPS = 16;
constexpr int MMA_WARP = PRODUCER_WARPS;
constexpr int THREADS = (PRODUCER_WARPS + 1) * 32;
constexpr int MAX_STAGES = 6;
constexpr int SMEM_LIMIT = 232448 - 2048;
// The tensor core adds into its FP32 accumulator with truncation, so the error of one accumulation chain
// grows linearly with its length (measured: 2e-4 relative after 32k pixels, i.e. 8k accumulation steps).
// A CTA therefore keeps a chain to CHUNK_KB K blocks (3072 pixels, 768 steps: about 1.4e-5): after each
// chunk the epilogue warps fold the accumulator into the CTA's slot of `out` with ordinary FP32 adds
// (round to nearest; the first chunk is a store, later ones are global reductions with a single writer per
// address) and the next chunk starts from zero.  A long reduction then costs one pass over the CTA's own
// output tile every few thousand pixels (about 5 us per fold: the staging pipeline runs dry while the epilogue
// warps, which are also producers, read the accumulator) instead of more splits and more scratch.
constexpr int CHUNK_KB = 96;

struct DwStripArgs {
  ConvGeom g;
  View4 x, dy;
  float* out;            // dW (one split) or the partial buffer [split][cout][cig*taps]
  int H, W, pr, pc;      // padded pixel space (see conv_tc_strip.cu)
  int q_total;           // padded pixels (below 2^31 - 64)
  FastDiv img_div, row_div, div_tasks, div_stages;
  int span, splits;      // padded pixels per split (multiple of KP)
  int xblocks;           // staged input blocks per CTA: 1 (one strip, taps in M through the block stride) or 4
  int partial_layout;    // 1: `out` is the split buffer [split][cout][kh*kw][cig] (channel fastest, so the epilogue's
                         // lanes store neighbouring floats); 0: dW itself, [cout][cig][kh*kw]
  int nacc;              // accumulators per CTA (strip arrangement: 1 or 2 channel blocks sharing the dY operand)
  int xr;                // rows staged per input block: XR (strip with tap margin) or KP (exact blocks)
  int blocks_are_taps;   // xblocks == 4: block j is tap kx = j of one channel block (strided filters) rather than
                         // channel block j of a 1x1 filter
  int sph, spw;          // stride: grid pixel (r, c) of phase (a, b) is the input pixel (r*sph + a, c*spw + b)
  int in_h, in_w, out_h, out_w;  // extents of x and of dY (the grid H x W covers both)
  unsigned blk_b[2], blk_dc[2];  // per tap kx (up to 8): column phase and whole-pixel column offset (signed), 8 bits each
  int kx_groups;                 // filters wider than four taps take ceil(kw / 4) CTAs, four taps each
  int ci_tiles, co_tiles;
  int stages;
  int chunk_kb;          // K blocks accumulated in tensor memory before the sum is folded into `out` (see CHUNK_KB)
  int* status;
  unsigned long long* prof;  // optional cycle counters of CTA (0,0) (B200_STRIP_PROFILE=1), else null
};

// role cycle probes: compiled in only with -DB200_ROLE_PROFILE=1 (see conv_tc_strip.cu)
#ifndef B200_ROLE_PROFILE
#define B200_ROLE_PROFILE 0
#endif
#define DPROF_ON(leader) (B200_ROLE_PROFILE && a.prof != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && (leader))
#define DPROF_T0(on) const long long prof_t0__ = (on) ? clock64() : 0
#define DPROF_ADD(on, slot) do { if (on) atomicAdd(a.prof + (slot), (unsigned long long)(clock64() - prof_t0__)); } while (0)

struct Ctrl {
  unsigned long long full[MAX_STAGES], empty[MAX_STAGES], accum[2], drained[2];
  uint32_t tmem_base;
  int abort_flag;
};

struct FoldArgs {
  float* out;            // this thread's first output element
  long long cols;        // element stride between output channels
  uint32_t acc;          // tensor-memory address of this warp's accumulator rows (buffer 0)
  uint32_t acc_buffer_cols, nbuf;  // column distance between the two accumulator buffers; 1 or 2 buffers
  uint32_t accum_bar, drained_bar; // shared-memory addresses of accum[0] / drained[0] (buffer b: + 8 * b)
  int cols_valid;
  bool row_ok;
  int* abort_flag;
  int* status;
};

// Folds one warp's accumulator rows into `out` after chunk `c` of the reduction (see CHUNK_KB): the first chunk is
// stored, later ones are added to what the same thread stored before.  Out of line on purpose: it runs once per
// 2048 pixels, and inlined it costs the producers' loop registers (that loop runs at the 96-register limit of a
// 17-warp CTA).
template <int BN, bool FUSE_HILO>
__device__ __noinline__ bool fold_accumulator(FoldArgs f, int c, bool more) {
  // chunk c used accumulator buffer c % nbuf, for the (c / nbuf)-th time
  const uint32_t buf = f.nbuf == 2 ? (uint32_t)c & 1u : 0u, use = f.nbuf == 2 ? (uint32_t)c >> 1 : (uint32_t)c;
  if (!mbar_wait(f.accum_bar + 8u * buf, use & 1u, f.abort_flag, f.status, STATUS_TIMEOUT_ACCUM)) return false;
  tc_fence_after();
  const bool add = c > 0;
  f.acc += buf * f.acc_buffer_cols;
#pragma unroll 1
  for (int c0 = 0; c0 < BN; c0 += 32) {
    if (c0 >= f.cols_valid) break;
    float v[32];
    tmem_ld32(f.acc + (uint32_t)c0, v);
    if (FUSE_HILO) {
      float v2[32];
      tmem_ld32(f.acc + (uint32_t)(BN + c0), v2);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] += v2[j];
    }
    if (f.row_ok) {
      float* p = f.out + c0 * f.cols;
      const int nvalid = f.cols_valid - c0;
      if (add) {
        // Reductions without a return value: the thread does not wait for the old values, so the accumulator is
        // handed back after the tensor-memory reads alone.  Every address has exactly one writer (this thread,
        // in program order), so the sums are the same from run to run.
#pragma unroll
        for (int j = 0; j < 32; ++j, p += f.cols)
          if (j < nvalid) atomicAdd(p, v[j]);
      } else if (nvalid >= 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j, p += f.cols) *p = v[j];
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j, p += f.cols)
          if (j < nvalid) *p = v[j];
      }
    }
  }
  if (more) {  // the accumulator may be overwritten now
    tc_fence_before();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(f.drained_bar + 8u * buf);
  }
  return true;
}

template <int BN, bool DW_CROSS>
__global__ void __launch_bounds__(THREADS, 1) dweight_strip_kernel(const DwStripArgs a) {
  wait_previous();
  extern __shared__ unsigned char smem_raw[];
  const unsigned long long prof_start = a.prof ? global_ns() : 0;
  // the pass that sums the split partials may take its place on the SMs now (it waits for this grid to finish)
  if (a.partial_layout) asm volatile("griddepcontrol.launch_dependents;");
  const ConvGeom& g = a.g;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  constexpr int NB = BN / 32;                                  // dY blocks per stage
  const uint32_t x_plane = (uint32_t)a.xr * 128u, x_bytes = (uint32_t)(a.nacc * a.xblocks) * 2u * x_plane;
  constexpr uint32_t y_plane = NB * KP * 128u;                 // all dY blocks of one plane
  const uint32_t stage_bytes = x_bytes + 2u * y_plane;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (base - raw) + a.stages * stage_bytes);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x_halves = a.xr > 32 ? 2 : 1;                      // a strip = rows 0..31 and 32..47; an exact block = 32 rows
  const int kx0 = (int)(blockIdx.x % (unsigned)a.kx_groups) * 4;  // first horizontal tap of this CTA
  // taps beyond the filter width of a narrow filter are not staged (their accumulator rows are never
  // stored); the last group of a wide filter stages zeros for them so that every CTA has the same jobs
  const int x_tasks = a.nacc * (a.blocks_are_taps ? min(4, g.kw) : a.xblocks) * x_halves;
  const int tasks = x_tasks + NB;                              // warp-sized staging jobs per K block
  // BN <= 128: the dY hi and lo planes (their 32-channel blocks are equally spaced) form ONE operand
  // of 2*BN columns, so x_hi*[dy_hi | dy_lo] is a single MMA; the epilogue adds the two halves.
  constexpr bool FUSE_HILO = BN <= 128 && !DW_CROSS;
  constexpr uint32_t ACC_COLS = FUSE_HILO ? 2 * BN : BN;
  // Two accumulator buffers where tensor memory has room (512 columns): the MMA thread then moves on to the
  // other buffer at a chunk boundary while the epilogue warps fold the finished one, instead of waiting for them.
  const uint32_t acc_buffer_cols = ACC_COLS * (uint32_t)a.nacc;   // 64..512, a power of two
  const uint32_t nbuf = acc_buffer_cols <= 256 ? 2u : 1u;
  const uint32_t tmem_cols = acc_buffer_cols * nbuf;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), (uint32_t)tasks * 32u);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctrl->accum[b]), 1);
      mbar_init(smem_u32(&ctrl->drained[b]), (uint32_t)(4 * a.nacc));  // one arrival per epilogue warp
    }
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_acc = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);

  // ---- which piece of dW this CTA owns ----
  int id = blockIdx.x / a.kx_groups;
  const int ci_tile = id % a.ci_tiles; id /= a.ci_tiles;
  const int ky = id % g.kh;            id /= g.kh;
  const int co_tile = id % a.co_tiles; id /= a.co_tiles;
  const int group = id;
  const int split = blockIdx.y;
  const int ci_per_tile = a.blocks_are_taps ? 32 : a.nacc * a.xblocks * 32;
  const int ci0 = ci_tile * ci_per_tile, co0 = co_tile * BN;
  const int cols_valid = min(BN, g.cog - co0);
  const int row_pitch = a.W + a.pc;
  const int img_pitch = (a.H + a.pr) * row_pitch;
  const int k_begin = split * a.span;  // < q_total
  const int k_end = a.q_total - k_begin > a.span ? k_begin + a.span : a.q_total;
  const int kblocks = (k_end - k_begin + KP - 1) / KP;
  // vertical tap: input row sph*(r + dr) + pa
  const int oy = ky * g.dh - g.ph;
  const int dr = oy >= 0 ? oy / a.sph : -((-oy + a.sph - 1) / a.sph), pa = oy - dr * a.sph;
  const int yshift = dr * row_pitch;

  if (warp == MMA_WARP) {
    // The whole warp runs the loop and waits on the barriers; one elected lane issues the tcgen05 instructions.  With
    // uniform control flow the descriptors live in uniform registers, which is where tcgen05.mma reads its operands
    // (issued from one divergent thread, every operand crossed over from the vector registers first, and that
    // crossing, not the tensor pipe, paced the kernel).  Stage indices are counted and descriptors are base + offset.
    {
      const bool leader = elect_one();
      constexpr uint32_t idesc = make_idesc_tf32(128, BN) | (1u << 15) | (1u << 16);  // both operands MN-major
      constexpr uint32_t idesc_wide = make_idesc_tf32(128, FUSE_HILO ? 2 * BN : BN) | (1u << 15) | (1u << 16);
      const uint32_t a_lbo = a.xblocks == 1 ? (uint32_t)g.dw * 128u : 2u * x_plane;
      // input rows start at the pixel shifted by -pad_w; hi plane then lo plane of each block
      const uint64_t da_base = make_mn_desc(base + (a.xblocks == 1 ? (uint32_t)(XOFF - g.pw + kx0 * g.dw) * 128u : 0u), a_lbo);
      const uint64_t db_base = make_mn_desc(base + x_bytes, KP * 128u);
      const uint32_t stage_d = stage_bytes >> 4, x_plane_d = x_plane >> 4;
      constexpr uint32_t y_plane_d = y_plane >> 4;
      // BF16 cross terms: the second plane of every block is split into bf16(hi) and bf16(lo) halves
      // of 64-byte rows; x_hi16 pairs with dy_lo16 and x_lo16 with dy_hi16
      constexpr uint32_t idesc16 = make_idesc_bf16(128, BN) | (1u << 15) | (1u << 16);
      const uint32_t a_lbo16 = a.xblocks == 1 ? (uint32_t)g.dw * 64u : 2u * x_plane;
      const uint64_t da16_base = make_mn_desc16(base + x_plane + (a.xblocks == 1 ? (uint32_t)(XOFF - g.pw + kx0 * g.dw) * 64u : 0u), a_lbo16);
      const uint64_t db16_base = make_mn_desc16(base + x_bytes + y_plane, KP * 64u);
      const bool pm = DPROF_ON(lane == 0);
      uint32_t s = 0, par = 0;
      int kb_in_chunk = 0;
      uint32_t chunk = 0, buf = 0;
      for (int kb = 0; kb < kblocks; ++kb, ++kb_in_chunk) {
        if (kb_in_chunk == a.chunk_kb) {
          // chunk boundary: hand the accumulator to the epilogue warps; before the next buffer is overwritten its
          // previous chunk (nbuf chunks back) must have been read
          if (leader) umma_commit(smem_u32(&ctrl->accum[buf]));
          ++chunk;
          kb_in_chunk = 0;
          buf = nbuf == 2 ? chunk & 1u : 0u;
          if (chunk >= nbuf) {
            const uint32_t prev_use = (chunk - nbuf) / nbuf;
            if (!warp_wait(smem_u32(&ctrl->drained[buf]), prev_use & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
            tc_fence_after();
          }
        }
        { DPROF_T0(pm);
        if (!warp_wait(smem_u32(&ctrl->full[s]), par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) break;
        DPROF_ADD(pm, 0); }
        DPROF_T0(pm);
        const uint64_t da_hi = da_base + s * stage_d;
        const uint64_t db_hi = db_base + s * stage_d, db_lo = db_hi + y_plane_d;
        if (leader)
        for (int u = 0; u < a.nacc; ++u) {  // channel blocks that share this dY block
          const uint32_t acc = tmem_acc + buf * acc_buffer_cols + (uint32_t)u * ACC_COLS;
          const uint64_t ua_hi = da_hi + (uint64_t)u * (2 * x_plane_d), ua_lo = ua_hi + x_plane_d;
          if constexpr (DW_CROSS) {
#pragma unroll
            for (int kg = 0; kg < KP / 8; ++kg) umma_tf32(acc, ua_hi + kg * 64, db_hi + kg * 64, idesc, (kb_in_chunk | kg) != 0);
            const uint64_t a_h16 = da16_base + s * stage_d + (uint64_t)u * (2 * x_plane_d), a_l16 = a_h16 + (x_plane_d >> 1);
            const uint64_t b_l16 = db16_base + s * stage_d, b_h16 = b_l16 + (y_plane_d >> 1);
#pragma unroll
            for (int kg = 0; kg < KP / 16; ++kg) umma_bf16(acc, a_h16 + kg * 64, b_l16 + kg * 64, idesc16, 1);  // 16 rows of 64 bytes
#pragma unroll
            for (int kg = 0; kg < KP / 16; ++kg) umma_bf16(acc, a_l16 + kg * 64, b_h16 + kg * 64, idesc16, 1);
          } else {
#pragma unroll
            for (int kg = 0; kg < KP / 8; ++kg) {  // 8 pixels = 8 rows of 128 bytes per MMA
              if (FUSE_HILO) {
                umma_tf32(acc, ua_hi + kg * 64, db_hi + kg * 64, idesc_wide, (kb_in_chunk | kg) != 0);
                umma_tf32(acc, ua_lo + kg * 64, db_hi + kg * 64, idesc, 1);
              } else {
                umma_tf32(acc, ua_lo + kg * 64, db_hi + kg * 64, idesc, (kb_in_chunk | kg) != 0);
                umma_tf32(acc, ua_hi + kg * 64, db_lo + kg * 64, idesc, 1);
                umma_tf32(acc, ua_hi + kg * 64, db_hi + kg * 64, idesc, 1);
              }
            }
          }
        }
        if (leader) umma_commit(smem_u32(&ctrl->empty[s]));
        if (++s == (uint32_t)a.stages) { s = 0; par ^= 1; }
        DPROF_ADD(pm, 1);
      }
      if (leader) umma_commit(smem_u32(&ctrl->accum[buf]));
    }
  } else {
    // ---- producers: job j of K block kb goes to warp (kb*tasks + j) % 16 ----
    const bool x_vec = channel_quads_aligned(a.x, g.cig, g.groups), y_vec = channel_quads_aligned(a.dy, g.cog, g.groups);
    const int total_jobs = kblocks * tasks;  // kblocks <= 2^26, tasks <= 16
    // ---- folding the accumulator into `out` (warps 0 .. 4*nacc-1): lane = row of the accumulator = (block, channel) ----
    // Chunk c of the reduction is complete when the MMA thread's commit flips `accum` for the c-th time.  The first
    // chunk is stored, later ones are added to what this CTA stored before (same thread, same addresses: program order).
    const int chunks_total = (kblocks + a.chunk_kb - 1) / a.chunk_kb;
    const bool drains = warp < 4 * a.nacc;
    // what the fold needs, as plain values (the call is out of line: see fold_accumulator)
    FoldArgs fa;
    {
      const int taps = g.kh * g.kw;
      const int quarter = warp & 3, u = warp >> 2;
      // block index: horizontal tap (taps in M) or channel block (1x1 filter in the block arrangement)
      const bool taps_in_m = a.xblocks == 1 || a.blocks_are_taps;
      const int kx = taps_in_m ? kx0 + quarter : 0;
      const int ci = ci0 + u * 32 + (taps_in_m ? lane : quarter * 32 + lane);
      fa.cols = (long long)g.cig * taps;
      fa.row_ok = kx < g.kw && ci < g.cig;
      fa.out = a.out + ((long long)split * g.cout + (long long)group * g.cog + co0) * fa.cols +
               (a.partial_layout ? (long long)(ky * g.kw + kx) * g.cig + ci : (long long)ci * taps + ky * g.kw + kx);
      fa.acc = tmem_acc + (uint32_t)u * ACC_COLS + ((uint32_t)(quarter * 32) << 16);
      fa.cols_valid = cols_valid;
      fa.acc_buffer_cols = acc_buffer_cols;
      fa.nbuf = nbuf;
      fa.accum_bar = smem_u32(&ctrl->accum[0]);
      fa.drained_bar = smem_u32(&ctrl->drained[0]);
      fa.abort_flag = &ctrl->abort_flag;
      fa.status = a.status;
    }
    auto drain = [&](int c) -> bool { return fold_accumulator<BN, FUSE_HILO>(fa, c, c + (int)nbuf < chunks_total); };
    // consecutive jobs of a warp stay within `stages` K blocks of each other (a waiter that skipped
    // a whole phase of a stage's mbarrier would see the parity of an older phase and run ahead)
    const int warps_active = min(PRODUCER_WARPS, tasks * a.stages);
    const bool produces = warp < warps_active;
    bool alive = true;
    int job = warp;
    // chunk by chunk: this warp's staging jobs of the chunk (the inner loop is the hot one), then, for an
    // epilogue warp, the fold of that chunk -- so a warp never stages blocks of a later chunk before it has
    // folded the earlier one, and the MMA thread never waits for a fold that waits for this warp's blocks
    for (int chunk = 0; chunk < chunks_total && alive; ++chunk) {
    // ... except for the first `stages` K blocks of the next chunk, which it stages BEFORE folding: their slots
    // were last used by blocks of this chunk, so staging them depends on nothing the fold waits for, and the
    // MMA thread finds a full pipeline when the fold hands the accumulator back
    const int job_end = chunk + 1 < chunks_total ? min(total_jobs, ((chunk + 1) * a.chunk_kb + a.stages) * tasks) : total_jobs;
    for (; produces && job < job_end && alive; job += warps_active) {
      const int kb = (int)a.div_tasks.div((uint32_t)job), j = job - kb * tasks;
      const uint32_t round = a.div_stages.div((uint32_t)kb);
      const int s = kb - (int)round * a.stages;
      const int k0 = k_begin + kb * KP;
      const uint32_t xs = base + s * stage_bytes, ys = xs + x_bytes;
      float val[32];
      bool chunked;  // which register pattern stage_block used
      int rows, row0;
      BlockPlanes pl;
      const bool pp = DPROF_ON(threadIdx.x == 0);
      DPROF_T0(pp);
      if (j < x_tasks) {
        const int blk = x_halves == 2 ? j >> 1 : j, half = x_halves == 2 ? j & 1 : 0;
        rows = half ? XR - 32 : 32;
        row0 = half * 32;
        pl.hi = xs + (uint32_t)blk * 2u * x_plane;
        pl.lo = pl.hi + x_plane;
        pl.h16 = pl.lo;
        pl.l16 = pl.lo + x_plane / 2;
        if (a.xblocks == 1) {
          // one strip; the horizontal taps are its row offsets.  The input is needed wherever it
          // exists: no split-range clipping, only image bounds
          const int c0 = ci0 + blk * 32;  // strip blk of this CTA
          const int chans = max(0, min(32, g.cig - c0));
          chunked = stage_block(a.x, (long long)group * g.cig + c0, chans, a.H, a.W, row_pitch, img_pitch, a.img_div, a.row_div,
                      k0 + yshift - XOFF + row0, 0, a.q_total, rows, lane, x_vec, val);
        } else {
          // exact 32-pixel blocks: tap kx = blk of one channel block, or channel block blk of a 1x1 filter
          const int c0 = ci0 + (a.blocks_are_taps ? 0 : blk * 32);
          const int kx = kx0 + blk;  // tap of this block (blocks_are_taps)
          const int chans = (a.blocks_are_taps && kx >= g.kw) ? 0 : max(0, min(32, g.cig - c0));
          const unsigned tb = kx < 4 ? a.blk_b[0] >> (8 * kx) : a.blk_b[1] >> (8 * (kx - 4));
          const unsigned td = kx < 4 ? a.blk_dc[0] >> (8 * kx) : a.blk_dc[1] >> (8 * (kx - 4));
          const int pb = a.blocks_are_taps ? (int)(tb & 0xFFu) : 0;
          const int dc = a.blocks_are_taps ? (int)(signed char)(td & 0xFFu) : 0;
          chunked = stage_block(a.x, (long long)group * g.cig + c0, chans, a.H, a.W, row_pitch, img_pitch, a.img_div, a.row_div,
                      k0 + yshift + dc, 0, a.q_total, rows, lane, x_vec, val, a.sph, a.spw, pa, pb, a.in_h, a.in_w);
        }
      } else {
        const int blk = j - x_tasks;
        rows = 32;
        row0 = blk * KP;
        pl.hi = ys;
        pl.lo = ys + y_plane;
        pl.l16 = pl.lo;                 // [bf16(lo) blocks][bf16(hi) blocks]: x_hi16 meets dy_lo16
        pl.h16 = pl.lo + y_plane / 2;
        const int c0 = co0 + blk * 32;
        const int chans = max(0, min(32, g.cog - c0));
        // dY outside this split's pixel range must read as zero so that splits do not overlap
        chunked = stage_block(a.dy, (long long)group * g.cog + c0, chans, a.H, a.W, row_pitch, img_pitch, a.img_div, a.row_div,
                    k0, k_begin, k_end, rows, lane, y_vec, val, 1, 1, 0, 0, a.out_h, a.out_w);
      }
      DPROF_ADD(pp, 2);
      { const long long tw = pp ? clock64() : 0;
      if (!mbar_wait(smem_u32(&ctrl->empty[s]), (round & 1) ^ 1, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) { alive = false; break; }
      if (pp) atomicAdd(a.prof + 3, (unsigned long long)(clock64() - tw)); }
      { const long long tw = pp ? clock64() : 0;
      if (chunked) store_block_chunks<DW_CROSS>(val, rows, row0, pl, lane);
      else store_block<DW_CROSS>(val, rows, row0, pl, lane);
      fence_proxy_async();
      mbar_arrive(smem_u32(&ctrl->full[s]));
      if (pp) { atomicAdd(a.prof + 4, (unsigned long long)(clock64() - tw)); atomicAdd(a.prof + 5, 1ull); } }
    }
    if (drains && alive) {
      const bool pe = DPROF_ON(threadIdx.x == 0);
      DPROF_T0(pe);
      alive = drain(chunk);
      DPROF_ADD(pe, 7);
      if (pe) atomicAdd(a.prof + 8, 1ull);
    }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_acc, tmem_cols);
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

// Sum the split partials [split][cout][taps][cig] in a fixed order (run-to-run identical) and write dW[cout][cig][taps].
// A block owns 2^ch_log2 channels of one output channel with all their taps: it reads along the channels (16 bytes at a
// time when VEC is 4) and writes along the taps, both coalesced, with the transposition in shared memory (written straight
// from the reading order, each warp's stores touched 32 sectors).  `slices` threads share a value when a block has fewer
// values than threads; four splits are in flight per thread.
constexpr int FIN_SMEM = 48 << 10;
template <int VEC>
__global__ void __launch_bounds__(256) finalize_partials_kernel(const float* __restrict__ partial, float* __restrict__ dw,
                                                               long long count, int splits, int cig, int taps, int slices, int ch_log2,
                                                               FastDiv div_chunks, FastDiv div_units) {
  // launched with programmatic stream serialisation behind the kernel that writes the partials: its blocks may be
  // resident before that kernel has finished, and wait here until it has (and its stores are visible)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  extern __shared__ float part[];              // [slices][channel][tap]; not used by a block of one channel
  const int co = (int)div_chunks.div(blockIdx.x), chunk = (int)blockIdx.x - co * (int)div_chunks.d;
  const int ch = 1 << ch_log2, c0 = chunk << ch_log2, chans = min(ch, cig - c0), values = taps << ch_log2;
  const int units = values / VEC, per_tap = ch / VEC, ptl = ch_log2 - (VEC == 4 ? 2 : 0);
  const float* base = partial + (long long)co * taps * cig + c0;
  float* dst = dw + ((long long)co * cig + c0) * taps;
  for (int item = threadIdx.x; item < units * slices; item += 256) {
    const int slice = (int)div_units.div((uint32_t)item), e = item - slice * units, tap = e >> ptl, c = (e & (per_tap - 1)) * VEC;
    float sum[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) sum[k] = 0.f;
    if (c < chans) {                           // chans is a multiple of VEC
      const float* p = base + (long long)slice * count + tap * cig + c;
      const long long step = (long long)slices * count;
      for (int s = slice; s < splits; s += 4 * slices, p += 4 * step) {
        float v[4][VEC];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool ok = s + u * slices < splits;
          if (VEC == 4) {
            const float4 f = ok ? *reinterpret_cast<const float4*>(p + u * step) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[u][0] = f.x; v[u][1 % VEC] = f.y; v[u][2 % VEC] = f.z; v[u][3 % VEC] = f.w;
          } else {
            v[u][0] = ok ? p[u * step] : 0.f;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int k = 0; k < VEC; ++k) sum[k] += v[u][k];
      }
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      if (ch == 1) dst[tap] = sum[k];
      else part[slice * values + (c + k) * taps + tap] = sum[k];
    }
  }
  if (ch == 1) return;
  __syncthreads();
  for (int e = threadIdx.x; e < chans * taps; e += 256) {
    float sum = part[e];
    for (int k = 1; k < slices; ++k) sum += part[k * values + e];
    dst[e] = sum;
  }
}

int finalize_partials(const float* partial, float* dw, const ConvGeom& g, int splits, cudaStream_t st) {
  const long long count = (long long)g.cout * g.cig * g.kh * g.kw;
  cudaLaunchConfig_t cfg{};
  const int taps = g.kh * g.kw;
  const bool vec = g.cig % 4 == 0 && (reinterpret_cast<uintptr_t>(partial) & 15) == 0;   // the caller's workspace may start anywhere
  // channels per block: all of them if they fit the default shared memory, fewer while the blocks do not fill the SMs
  // twice (down to 16: shorter runs waste the sectors at their ends); a single channel needs no shared memory
  int ch_log2 = 0;
  while (ch_log2 < 9 && (1 << ch_log2) < g.cig && ((size_t)taps << (ch_log2 + 1)) * sizeof(float) <= FIN_SMEM) ++ch_log2;
  while (ch_log2 > 4 && (long long)g.cout * ((g.cig + (1 << ch_log2) - 1) >> ch_log2) < 2ll * sm_count()) --ch_log2;
  const bool v4 = vec && ch_log2 >= 2;
  const int chunks = (g.cig + (1 << ch_log2) - 1) >> ch_log2, units = (taps << ch_log2) / (v4 ? 4 : 1);
  const long long blocks = (long long)g.cout * chunks;
  const size_t values = ((size_t)taps << ch_log2) * sizeof(float);
  int slices = 1;
  while (ch_log2 > 0 && slices * 2 <= splits && units * slices < 256 && 2 * slices * values <= FIN_SMEM) slices *= 2;
  if (blocks > 2147483647ll) return fail(B200_ERANGE, "dWeight finalize: grid exceeds launch limits");
  cfg.gridDim = dim3((unsigned)blocks); cfg.blockDim = dim3(256); cfg.stream = st;
  cfg.dynamicSmemBytes = ch_log2 > 0 ? slices * values : 0;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  B200_CUDA(cudaLaunchKernelEx(&cfg, v4 ? finalize_partials_kernel<4> : finalize_partials_kernel<1>, partial, dw, count, splits,
                               g.cig, taps, slices, ch_log2, FastDiv((uint32_t)chunks), FastDiv((uint32_t)units)));
  count_launch();
  return launch_check("finalize_partials_kernel");
}

struct DwStripPlan {
  bool ok = false;
  bool cross = false;  // BF16 cross terms (four accumulators)
  int bn = 0, xblocks = 1, nacc = 1, xr = XR, blocks_are_taps = 0, stages = 0, smem = 0, ci_tiles = 0, co_tiles = 0, splits = 1, span = 0;
  int gh = 0, gw = 0, pr = 0, pc = 0;  // pixel grid (covers dY and every phase sub-image of x) and its zero padding
  unsigned blk_b[2] = {0, 0}, blk_dc[2] = {0, 0};
  int kx_groups = 1;
  size_t bytes = 0;
};

static inline int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// Two arrangements of the M dimension (4 blocks of 32 rows):
//   strip:  stride 1, output as large as the input, kw >= 2 (or few channels): one staged input
//           strip per K block, the horizontal taps are its row offsets;
//   blocks: everything else -- strides, any padding, 1x1: four exact 32-pixel blocks per K
//           block, either the taps kx = 0..3 of one channel block (each with its own column phase and
//           offset) or, for a 1x1 filter, four channel blocks.
static DwStripPlan make_plan(const ConvGeom& g, size_t budget) {
  DwStripPlan p;
  if (g.kw > 8 || g.cog < 16 || g.cig < 16) return p;
  p.kx_groups = (g.kw + 3) / 4;
  const bool same = g.sh == 1 && g.sw == 1 && g.oh == g.h && g.ow == g.w && 2 * g.ph == g.dh * (g.kh - 1) &&
                    2 * g.pw == g.dw * (g.kw - 1);
  // the last row a VALID tap's M block reads must be inside the strip (the unused blocks of the last
  // tap group read whatever follows in the stage; their accumulator rows are never stored)
  const bool strip_fits = same && g.pw <= XOFF && (g.kw - 1) * g.dw - g.pw + XOFF + KP <= XR;
  const bool pointwise = same && g.kh == 1 && g.kw == 1;
  if (strip_fits && !(pointwise && g.cig >= 64)) {
    p.xblocks = 1; p.xr = XR;
    p.gh = g.h; p.gw = g.w; p.pr = g.ph; p.pc = g.pw;
  } else {
    if (g.sh > 255 || g.sw > 255) return p;
    p.xblocks = 4; p.xr = KP;
    p.blocks_are_taps = pointwise ? 0 : 1;
    p.gh = std::max(g.oh, (g.h + g.sh - 1) / g.sh);
    p.gw = std::max(g.ow, (g.w + g.sw - 1) / g.sw);
    for (int ky = 0; ky < g.kh; ++ky) p.pr = std::max(p.pr, std::abs(floor_div(ky * g.dh - g.ph, g.sh)));
    for (int kx = 0; kx < g.kw; ++kx) {
      const int ox = kx * g.dw - g.pw, dc = floor_div(ox, g.sw);
      if (dc < -127 || dc > 127) return p;
      p.pc = std::max(p.pc, std::abs(dc));
      p.blk_b[kx / 4] |= (unsigned)(ox - dc * g.sw) << (8 * (kx % 4));
      p.blk_dc[kx / 4] |= ((unsigned)dc & 0xFFu) << (8 * (kx % 4));
    }
  }
  // Several channel blocks per CTA share every staged dY block (one TMEM accumulator each): less dY
  // staging per MMA.  The column tile then stays at 128 (TMEM holds 512 columns).
  if (p.xblocks == 1 && g.cig >= 64) {
    p.cross = g.cig >= 128;
    p.nacc = p.cross && g.cig > 64 ? 4 : 2;
    p.bn = g.cog <= 64 ? 64 : 128;
  } else {
    p.bn = g.cog <= 64 ? 64 : (g.cog <= 128 ? 128 : 256);
  }
  const int y_stage = 2 * (p.bn / 32) * KP * 128;
  const int stage = p.nacc * p.xblocks * 2 * p.xr * 128 + y_stage;
  p.stages = std::min(MAX_STAGES, SMEM_LIMIT / stage);
  if (p.stages < 2) return p;
  p.smem = p.stages * stage + 1024 + (int)sizeof(Ctrl) + 64;
  const int ci_per_tile = p.blocks_are_taps ? 32 : p.nacc * p.xblocks * 32;
  p.ci_tiles = (g.cig + ci_per_tile - 1) / ci_per_tile;
  p.co_tiles = (g.cog + p.bn - 1) / p.bn;
  const long long q_total = (long long)g.n * (p.gh + p.pr) * (p.gw + p.pc);
  const long long tiles = (long long)p.ci_tiles * g.kh * p.kx_groups * p.co_tiles * g.groups;
  const size_t dw_bytes = sizeof(float) * (size_t)g.cout * g.cig * g.kh * g.kw;
  // Number of pixel splits: the one that minimises a small model of the run time in K-block units --
  // waves of CTAs (one CTA per SM is resident) x (K blocks per split + a fixed cost per CTA for
  // pipeline fill and the epilogue) + the finalize pass over the partials.  Every split at least 16
  // K blocks long; partials within budget.
  const long long kblocks_total = div_up64(q_total, KP);
  long long most = std::max<long long>(1, kblocks_total / 16);
  most = std::min<long long>(most, 65535);
  most = std::min<long long>(most, (long long)(budget / dw_bytes));
  most = std::min<long long>(most, 4ll * sm_count() / tiles + 1);
  const double cta_fixed = 10.0, finalize_per_split = (double)dw_bytes / 3.3e6;  // ~3 TB/s against ~1.1 us per K block
  long long want = 1;
  double best = 0.0;
  for (long long sp = 1; sp <= std::max<long long>(1, most); ++sp) {
    const double waves = (double)div_up64(tiles * sp, sm_count());
    const double cost = waves * ((double)div_up64(kblocks_total, sp) + cta_fixed) + (sp > 1 ? finalize_per_split * (double)sp : 0.0);
    if (sp == 1 || cost < best) { best = cost; want = sp; }
  }
  long long span = div_up64(q_total, KP) * KP, splits = 1;
  if (want >= 2) {
    span = div_up64(div_up64(q_total, want), KP) * KP;
    splits = div_up64(q_total, span);
  }
  if (q_total > 2147483647ll - (1 << 20)) return p;  // pixel indices are 32-bit in the kernel
  p.splits = (int)splits;
  p.span = (int)span;
  p.bytes = splits > 1 ? (size_t)splits * dw_bytes : 0;
  p.ok = true;
  return p;
}
static const DwStripPlan& plan_dw_strip(const ConvGeom& g, size_t budget) {
  thread_local PlanCache<DwStripPlan> cache;
  return cache.get(g, budget, [&] { return make_plan(g, budget); });
}

}  // namespace tcdw

// B200_DW_VARIANT pins a kernel (testing aid): "strip" the one with both operands in shared memory, "tmem" the other where it takes the geometry.
enum class Variant { BY_RULE, STRIP, TMEM };
static Variant variant() {
  const char* e = getenv("B200_DW_VARIANT");
  return !e ? Variant::BY_RULE : !strcmp(e, "strip") ? Variant::STRIP : !strcmp(e, "tmem") ? Variant::TMEM : Variant::BY_RULE;
}
bool dweight_strip_supported(const ConvGeom& g) {
  tcdt::PlanInfo info;
  return tcdw::plan_dw_strip(g, 0).ok || (variant() != Variant::STRIP && tcdt::plan_info(g, 0, &info));
}
// The tensor-memory kernel gives a CTA of up to 64 output channels all vertical taps of an input block, where this one has a CTA for each
// tap.  That pays while the splits fill the machine; where they cannot (little or no scratch, few pixels) its CTAs are a third as many and
// do a third more per K block.  Per K block and for the rest of a CTA, measured: 0.74 us (six slots; 0.31 per strip of a strided input) and
// 6 against 0.51 (0.60 in four blocks) + 4.  (1x1 filters always gain by the tensor-memory kernel's idle warps, and run in three TF32
// passes there as here: 432 -> 64 channels of 5x 7x7 11.9 us here, 8.2 there.)  16 -> 62 channels of 7x 21x21, stride 2, no scratch: 45.6 and 25.3 us;
// 38 -> 32 of 5x 46x46, no scratch: 265 and 181; 16 -> 64 of 61x61 x 14 with all the scratch it wants: 27.4 and 28.9.
static bool strip_is_faster(const ConvGeom& g, const tcdt::PlanInfo& t, const tcdw::DwStripPlan& s) {
  if (!s.ok || g.cig * g.kh * g.kw < 32) return false;   // few products: short chains, which only the tensor-memory kernel has
  if (g.cog > 64 || s.nacc != 1 || !t.shift) return false;
  const double tmem = 6.0 + t.kblocks * std::max(0.74 * t.slots / 6, 0.31 * t.strips);
  const double strip = 4.0 + (double)(s.span / tcdw::KP) * (s.xblocks == 1 ? 0.51 : 0.60);
  return strip < 0.85 * tmem;
}
// Whether the tensor-memory kernel takes the call.
static bool tmem_takes(const ConvGeom& g, size_t budget, const tcdw::DwStripPlan& s, tcdt::PlanInfo* t) {
  const Variant pinned = variant();
  return pinned != Variant::STRIP && tcdt::plan_info(g, budget, t) && (pinned == Variant::TMEM || !strip_is_faster(g, *t, s));
}
size_t dweight_strip_workspace(const ConvGeom& g, size_t budget) {
  tcdt::PlanInfo t;
  const tcdw::DwStripPlan& s = tcdw::plan_dw_strip(g, budget);
  return tmem_takes(g, budget, s, &t) ? t.bytes : s.bytes;
}

template <int BN, bool CROSS>
static int launch_dw_strip(const tcdw::DwStripArgs& a, dim3 grid, int smem, cudaStream_t st) {
  // opt in once (thread-safe) to the full 227 KB of dynamic shared memory for this instantiation
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(tcdw::dweight_strip_kernel<BN, CROSS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  launch_next(tcdw::dweight_strip_kernel<BN, CROSS>, grid, tcdw::THREADS, smem, st, a);
  count_launch();
  return launch_check("dweight_strip_kernel");
}

int dweight_strip(const ConvGeom& g, View4 x, View4 dy, float* dw, void* ws, size_t ws_bytes, cudaStream_t st) {
  using namespace tcdw;
  const DwStripPlan& plan = plan_dw_strip(g, ws ? ws_bytes : 0);
  tcdt::PlanInfo t;
  if (tmem_takes(g, ws ? ws_bytes : 0, plan, &t)) {
    const int rc = tcdt::run(g, x, dy, dw, ws, ws_bytes, st);
    if (rc != B200_EUNSUPPORTED) return rc;
  }
  if (!plan.ok) return fail(B200_EUNSUPPORTED, "dWeight strip kernel does not take this geometry");
  // the kernel forms element offsets inside a tensor in 32 bits
  auto span = [](const View4& v, long long n, long long c, long long h, long long w) {
    return (n - 1) * std::llabs(v.s0) + (c - 1) * std::llabs(v.s1) + (h - 1) * std::llabs(v.s2) + (w - 1) * std::llabs(v.s3);
  };
  if (span(x, g.n, g.cin, g.h, g.w) > 2147483647ll - 64 * std::llabs(x.s1) || span(dy, g.n, g.cout, g.oh, g.ow) > 2147483647ll - 64 * std::llabs(dy.s1))
    return fail(B200_EUNSUPPORTED, "dWeight strip kernel: tensor too large for 32-bit element offsets");
  DwStripArgs a{};
  a.g = g; a.x = x; a.dy = dy;
  a.H = plan.gh; a.W = plan.gw; a.pr = plan.pr; a.pc = plan.pc;
  a.xr = plan.xr; a.blocks_are_taps = plan.blocks_are_taps; a.nacc = plan.nacc;
  a.sph = g.sh; a.spw = g.sw; a.in_h = g.h; a.in_w = g.w; a.out_h = g.oh; a.out_w = g.ow;
  a.blk_b[0] = plan.blk_b[0]; a.blk_b[1] = plan.blk_b[1]; a.blk_dc[0] = plan.blk_dc[0]; a.blk_dc[1] = plan.blk_dc[1];
  a.kx_groups = plan.kx_groups;
  a.q_total = (int)((long long)g.n * (a.H + a.pr) * (a.W + a.pc));
  a.img_div = FastDiv((uint32_t)((a.H + a.pr) * (a.W + a.pc)));
  a.row_div = FastDiv((uint32_t)(a.W + a.pc));
  a.span = plan.span; a.splits = plan.splits; a.xblocks = plan.xblocks;
  a.ci_tiles = plan.ci_tiles; a.co_tiles = plan.co_tiles; a.stages = plan.stages;
  {  // equal chunks of at most CHUNK_KB K blocks per CTA (a CTA reduces span / KP of them)
    int limit = CHUNK_KB;
    if (const char* e = getenv("B200_DW_CHUNK_KB")) limit = std::max(1, atoi(e));  // testing aid: chain length in K blocks
    const int kblocks = plan.span / KP;
    const int chunks = (kblocks + limit - 1) / limit;
    a.chunk_kb = std::max(1, (kblocks + chunks - 1) / std::max(1, chunks));
  }
  a.div_tasks = FastDiv((uint32_t)(plan.nacc * (plan.blocks_are_taps ? std::min(4, g.kw) : plan.xblocks) * (plan.xr > 32 ? 2 : 1) + plan.bn / 32));
  a.div_stages = FastDiv((uint32_t)plan.stages);
  a.out = plan.splits > 1 ? (float*)ws : dw;
  a.partial_layout = plan.splits > 1 ? 1 : 0;
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  const long long gx = (long long)plan.ci_tiles * g.kh * plan.kx_groups * plan.co_tiles * g.groups;
  if (gx > 2147483647ll) return fail(B200_ERANGE, "dWeight strip kernel: grid exceeds launch limits");
  // rows of dW that no CTA writes (channel blocks beyond kw taps) do not exist: every (co, ci, ky, kx)
  // is covered: four taps per CTA, ceil(kw / 4) tap groups, and all ci tiles are enumerated
  const dim3 grid((unsigned)gx, (unsigned)plan.splits);
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
  int rc = plan.cross ? (plan.bn == 64 ? launch_dw_strip<64, true>(a, grid, plan.smem, st) : launch_dw_strip<128, true>(a, grid, plan.smem, st))
         : plan.bn == 64 ? launch_dw_strip<64, false>(a, grid, plan.smem, st)
         : plan.bn == 128 ? launch_dw_strip<128, false>(a, grid, plan.smem, st) : launch_dw_strip<256, false>(a, grid, plan.smem, st);
  if (rc) return rc;
  if (profiling) {
    unsigned long long h[16];
    B200_CUDA(cudaStreamSynchronize(st));
    B200_CUDA(cudaMemcpy(h, prof_buf, sizeof h, cudaMemcpyDeviceToHost));
    fprintf(stderr, "[dweight strip profile, CTA 0, cycles] bn=%d xblocks=%d stages=%d grid=%lldx%d kblocks/cta=%d | mma: wait_full %llu issue %llu | "
            "warp 0: jobs %llu load %llu wait_empty %llu store %llu | folds: %llu, cycles in them %llu (of which waiting for the accumulator %llu) | ns: last CTA start %llu, first start to last end %llu, CTA lifetime min %llu max %llu\n",
            plan.bn, plan.xblocks, plan.stages, gx, plan.splits, plan.span / KP, h[0], h[1], h[5], h[2], h[3], h[4], h[8], h[7], h[6], h[12] - h[11], h[13] - h[11], h[14], h[15]);
  }
  if (plan.splits > 1) return tcdw::finalize_partials((const float*)ws, dw, g, plan.splits, st);
  return B200_OK;
}

}  // namespace b200

// One-launch tcgen05 kernel for convolutions (stride 1, forward and dInput) whose tiles leave most SMs idle, FP32 by split precision
// (tc_common.cuh): one image through one layer, where launches and latency are all there is.
//
// What bounds these layers and what follows from it.  The strip kernel (conv_tc_strip.cu) needs a launch ahead of it that splits the
// filter, and a tile then walks (channel block, tap) after (channel block, tap): 64 -> 64 channels of one 28x28 image are 7 tiles of
// 18 steps on 148 SMs, 11.4 us.  Here the CTAs of a cluster share a tile: each takes some of its (channel block, tap) pairs, splits the
// filter pieces and the pixels of these itself, all at once and without a pipeline, and has one short chain of products; the partial
// sums are exchanged through distributed shared memory, every CTA adding (in rank order) and storing its share of the tile's columns.  No second
// launch, no scratch: 6.8 us.  90 random layers of one to four images took 0.75 of the time (7 to 16 us before; best 0.33, worst 1.02).
//
// The exchange costs about 1 us and a rank's pairs 0.5 us each (32 columns) or 1 (64), so the plan takes as many ranks, and as narrow tiles,
// as still run in one wave.  CTAs: 16 warps, all of which stage, then one issues the products and eight carry the sums away.
//
// Grid pixels, row shifts and operand images are those of the strip kernel: a tile is 128 pixels of the padded grid, a tap a constant
// row offset into the staged pixels, channels beyond a ragged last block are zero.
//
// Replaces csrc/shaders/conv2d_tiled_body.glsl:53-86 of the reference for these geometries.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "plan_cache.cuh"
#include "strip_plan.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace tsm {
using namespace tc;
namespace cg = cooperative_groups;

constexpr int BLOCK_M = 128, KBLK = 32, WARPS = 16, THREADS = WARPS * 32, MAX_RANKS = 8;
constexpr int SMEM_LIMIT = 232448 - 2048;

struct SmallArgs {
  ConvGeom g;
  View4 act, w, res;
  const float* bias;
  long long bias_stride;
  float* out;                 // contiguous NCHW
  int is_dx, relu;
  int H, W, pr, pc;           // pixel grid and its padding
  int act_h, act_w, out_h, out_w;
  int kc, nc;                 // reduction channels, result channels
  int units, per, taps;       // (channel block, tap) pairs: of the layer, of a rank at most; taps of the filter
  int tiles_n, q_total;
  int strips, strip_rows;     // room for staged pixels: channel blocks, rows (a multiple of 8)
  int share;                  // columns that a rank adds up
  int act_quads, rows_first;  // channels-last pixels in 16-byte pieces; filter rows are the adjacent values
  FastDiv img_div, row_div, tap_div, share_div;
  int shift[tcs::MAX_TAPS];
  unsigned char ky[tcs::MAX_TAPS], kx[tcs::MAX_TAPS];
  int* status;
};
struct Ctrl {
  unsigned long long done;
  uint32_t tmem_base;
};

__device__ __forceinline__ uint32_t remote(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_remote(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

template <int BN>
__global__ void __launch_bounds__(THREADS, 1) conv_small_kernel(const __grid_constant__ SmallArgs a) {
  cluster_announce();
  wait_previous();
  constexpr uint32_t W_BYTES = BN * 256u, TMEM_COLS = BN < 32 ? 32 : BN;
  extern __shared__ unsigned char smem_raw[];
  auto cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), ranks = (int)cluster.num_blocks();
  const uint32_t raw = smem_u32(smem_raw), w_base = (raw + 1023u) & ~1023u;
  const uint32_t strip_plane = (uint32_t)a.strip_rows * 128u, strip_base = w_base + (uint32_t)a.per * W_BYTES;
  const uint32_t recv = strip_base + (uint32_t)a.strips * 2u * strip_plane;   // [rank][column of this rank's share][pixel]
  float* recv_ptr = reinterpret_cast<float*>(smem_raw + (recv - raw));
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(recv_ptr + ranks * a.share * BLOCK_M);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_tile = (int)blockIdx.x % a.tiles_n, m_tile = (int)blockIdx.x / a.tiles_n;
  const int n0 = n_tile * BN, q0 = m_tile * BLOCK_M;
  const int u0 = rank * a.per, u1 = min(a.units, u0 + a.per);        // the host leaves no rank without a pair
  const int row_pitch = a.W + a.pc, img_pitch = (a.H + a.pr) * row_pitch;
  const int cb0 = (int)a.tap_div.div((uint32_t)u0), cb1 = (int)a.tap_div.div((uint32_t)(u1 - 1));

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctrl->done), 1);
    fence_barrier_init();
  }
  if (warp == 0) tmem_alloc(smem_u32(&ctrl->tmem_base), TMEM_COLS);

  // rows of the strip of channel block cb: those that this rank's taps of it reach
  auto reach = [&](int cb, int& lo, int& hi) {
    const int t0 = cb == cb0 ? u0 - cb0 * a.taps : 0, t1 = cb == cb1 ? u1 - cb1 * a.taps : a.taps;
    lo = hi = a.shift[t0];
    for (int t = t0 + 1; t < t1; ++t) {
      lo = min(lo, a.shift[t]);
      hi = max(hi, a.shift[t]);
    }
  };
  // ---- pixels: a warp takes 32 rows by 8 channels at a time ----
  for (int cb = cb0; cb <= cb1; ++cb) {
    int lo, hi;
    reach(cb, lo, hi);
    const int rows = BLOCK_M + hi - lo, jobs = (rows + 31) / 32 * 4;
    const uint32_t p_hi = strip_base + (uint32_t)(cb - cb0) * 2u * strip_plane, p_lo = p_hi + strip_plane;
    for (int job = warp; job < jobs; job += WARPS) {
      const int r = (job >> 2) * 32 + lane, c = (job & 3) * 8, valid = min(8, a.kc - cb * KBLK - c), q = q0 + lo + r;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = 0.f;
      if (r < rows && q >= 0 && q < a.q_total) {
        const int n = (int)a.img_div.div((uint32_t)q), rem = q - n * img_pitch;
        const int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch;
        if (y < a.act_h && x < a.act_w) {
          const float* src = a.act.ptr + n * a.act.s0 + (cb * KBLK + c) * a.act.s1 + y * a.act.s2 + x * a.act.s3;
          if (a.act_quads && valid == 8) {
            const float4 f0 = __ldg(reinterpret_cast<const float4*>(src)), f1 = __ldg(reinterpret_cast<const float4*>(src) + 1);
            v[0] = f0.x; v[1] = f0.y; v[2] = f0.z; v[3] = f0.w; v[4] = f1.x; v[5] = f1.y; v[6] = f1.z; v[7] = f1.w;
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = j < valid ? __ldg(src + j * a.act.s1) : 0.f;
          }
        }
      }
      if (r < rows) {
        float h[8], l[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) split_tf32_fast(v[j], h[j], l[j]);
        sts_f32x4(p_hi + sw128_offset(r, c), h[0], h[1], h[2], h[3]);
        sts_f32x4(p_hi + sw128_offset(r, c + 4), h[4], h[5], h[6], h[7]);
        sts_b32x4(p_lo + sw128_offset_bf16(r, c), pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]), pack_bf16x2(h[4], h[5]), pack_bf16x2(h[6], h[7]));
        sts_b32x4(p_lo + sw128_offset_bf16(r, 32 + c), pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]), pack_bf16x2(l[4], l[5]),
                  pack_bf16x2(l[6], l[7]));
      }
    }
  }
  // ---- filter: a thread takes four reduction channels of a result channel, pair after pair (the taps of a filter are adjacent in memory) ----
  {
    constexpr int ITEMS = BN * (KBLK / 4), AT_ONCE = THREADS / ITEMS;
    const int i = (int)threadIdx.x % ITEMS, first = (int)threadIdx.x / ITEMS;
    const int row = a.rows_first ? (i & 7) | (i >> 6) << 3 : i >> 3, k = (a.rows_first ? i >> 3 & 7 : i & 7) * 4;
    const long long step = a.is_dx ? a.w.s0 : a.w.s1;
    const float* w_row = a.w.ptr + (n0 + row) * (a.is_dx ? a.w.s1 : a.w.s0);
#pragma unroll 3
    for (int u = u0 + first; u < u1; u += AT_ONCE) {
      const int cb = (int)a.tap_div.div((uint32_t)u), tap = u - cb * a.taps, c = cb * KBLK + k;
      const int valid = n0 + row < a.nc ? min(4, a.kc - c) : 0;
      const float* src = w_row + c * step + a.ky[tap] * a.w.s2 + a.kx[tap] * a.w.s3;
      float h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split_tf32(j < valid ? __ldg(src + j * step) : 0.f, h[j], l[j]);
      const uint32_t plane = w_base + (uint32_t)(u - u0) * W_BYTES, cross = plane + BN * 128u;
      sts_f32x4(plane + sw128_offset(row, k), h[0], h[1], h[2], h[3]);
      sts_b32x2(cross + sw128_offset_bf16(row, k), pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
      sts_b32x2(cross + sw128_offset_bf16(row, 32 + k), pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  if (warp == 0) {
    const bool leader = elect_one();
    constexpr uint32_t id32 = make_idesc_tf32(BLOCK_M, BN), id16 = make_idesc_bf16(BLOCK_M, BN);
    const uint64_t da = make_kmajor_sw128_desc(strip_base), db = make_kmajor_sw128_desc(w_base);
    const uint32_t plane_d = strip_plane >> 4;
    int cb = cb0, lo, hi, tap = u0 - cb0 * a.taps;
    reach(cb, lo, hi);
    for (int u = u0; u < u1; ++u) {
      const uint64_t a_hi = da + (uint64_t)((uint32_t)(cb - cb0) * 2u * plane_d + (uint32_t)(a.shift[tap] - lo) * 8u), a_lo = a_hi + plane_d;
      const uint64_t b_hi = db + (uint64_t)((uint32_t)(u - u0) * (W_BYTES >> 4)), b_lo = b_hi + (BN * 128u >> 4);
      if (leader) {
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_tf32(tmem, a_hi + 2 * k, b_hi + 2 * k, id32, (uint32_t)((u - u0) | k) != 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16(tmem, a_lo + 2 * k, b_lo + 2 * k, id16, 1);
      }
      if (++tap == a.taps && u + 1 < u1) {
        tap = 0;
        reach(++cb, lo, hi);
      }
    }
    if (leader) umma_commit(smem_u32(&ctrl->done));
  }
  cluster_wait_started();
  // ---- every rank leaves its columns with the ranks that add them ----
  if (warp < 8) {
    constexpr int COLS = BN / 2;
    warp_wait(smem_u32(&ctrl->done), 0, nullptr, a.status, STATUS_TIMEOUT_ACCUM);   // on a timeout the status word tells; the barriers below stay matched
    tc_fence_after();
    const int quarter = warp & 3, c0 = (warp >> 2) * COLS;
    float v[COLS];
    if constexpr (COLS == 32) tmem_ld32(tmem + (uint32_t)c0 + ((uint32_t)(quarter * 32) << 16), v);
    else tmem_ld16(tmem + (uint32_t)c0 + ((uint32_t)(quarter * 32) << 16), v);
    int owner = (int)a.share_div.div((uint32_t)c0), at = c0 - owner * a.share;
    const uint32_t mine = recv + 4u * (uint32_t)(rank * a.share * BLOCK_M + quarter * 32 + lane);
    uint32_t to = remote(mine, (uint32_t)owner);
#pragma unroll
    for (int j = 0; j < COLS; ++j) {
      st_remote(to + 4u * (uint32_t)(at * BLOCK_M), v[j]);
      if (++at == a.share) {
        at = 0;
        if (++owner < ranks) to = remote(mine, (uint32_t)owner);
      }
    }
    tc_fence_before();
  }
  cluster.sync();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
  // ---- add and store this rank's columns: thread = pixel ----
  const int p = (int)threadIdx.x % BLOCK_M, q = q0 + p;
  if (q >= a.q_total) return;
  const int n = (int)a.img_div.div((uint32_t)q), rem = q - n * img_pitch;
  const int y = (int)a.row_div.div((uint32_t)rem), x = rem - y * row_pitch;
  if (y >= a.out_h || x >= a.out_w) return;
  const int cols = min(min(a.share, BN - rank * a.share), a.nc - n0 - rank * a.share);
  const long long plane = (long long)a.out_h * a.out_w;
  for (int c = (int)threadIdx.x / BLOCK_M; c < cols; c += THREADS / BLOCK_M) {
    const int ch = n0 + rank * a.share + c;
    const float bv = a.bias ? __ldg(a.bias + ch * a.bias_stride) : 0.f;
    const float rv = a.res.ptr ? __ldg(a.res.ptr + n * a.res.s0 + ch * a.res.s1 + y * a.res.s2 + x * a.res.s3) : 0.f;
    float s = 0.f;
    for (int r = 0; r < ranks; ++r) s += recv_ptr[(r * a.share + c) * BLOCK_M + p];
    s += bv;
    if (a.res.ptr) s += rv;
    a.out[((long long)n * a.nc + ch) * plane + (long long)y * a.out_w + x] = a.relu ? fmaxf(s, 0.f) : s;
  }
}

// Clusters of that many CTAs (one on an SM) that run at the same time.  They are placed within groups of SMs, so that sixteen clusters of seven or
// forty-eight of three need a second wave, which takes as long as the first (16 tiles of 7 ranks: 12.8 us against 7.5 for 3).
static int clusters_at_once(int ranks);
struct SmallPlan {
  double time = 0;            // modelled, us
  int bn = 0, ranks = 0, per = 0, share = 0, strips = 0, strip_rows = 0, smem = 0, tiles_m = 0, tiles_n = 0;
  tcs::StripPlan geo;
};
static SmallPlan make_plan(const ConvGeom& g, bool is_dx) {
  SmallPlan best;
  if (g.groups != 1 || g.sh != 1 || g.sw != 1) return best;
  const tcs::StripPlan geo = tcs::plan_strip_geometry(g, is_dx);
  if (!geo.ok || geo.tt.n_phase != 1) return best;
  const int kc = is_dx ? g.cog : g.cig, nc = is_dx ? g.cig : g.cog, taps = geo.tt.taps_total, units = (kc + KBLK - 1) / KBLK * taps;
  const long long tiles_m = div_up64((long long)g.n * (geo.gh + geo.pr) * (geo.gw + geo.pc), BLOCK_M);
  if (tiles_m > sm_count()) return best;
  double best_cost = 0;
  for (int bn : {64, 32}) {
    const int tiles_n = (nc + bn - 1) / bn;
    for (int s = 1; s <= MAX_RANKS; ++s) {
      const int per = (units + s - 1) / s;
      if ((units + per - 1) / per != s || tiles_m * tiles_n > clusters_at_once(s)) continue;
      int strips = 1, rows = 0;
      for (int u = 0; u < units; u += per) {
        const int last = std::min(units, u + per) - 1, cb0 = u / taps, cb1 = last / taps;
        strips = std::max(strips, cb1 - cb0 + 1);
        for (int cb = cb0; cb <= cb1; ++cb) {
          const int t0 = cb == cb0 ? u - cb0 * taps : 0, t1 = cb == cb1 ? last - cb1 * taps : taps - 1;
          const auto mm = std::minmax_element(geo.tt.shift + t0, geo.tt.shift + t1 + 1);
          rows = std::max(rows, BLOCK_M + *mm.second - *mm.first);
        }
      }
      rows = (rows + 7) / 8 * 8;
      const int share = (bn + s - 1) / s;
      const long long smem = (long long)per * bn * 256 + (long long)strips * rows * 256 + (long long)s * share * BLOCK_M * 4 + 1024 + sizeof(Ctrl) + 64;
      if (smem > SMEM_LIMIT) continue;
      // us, measured on 70 layers: staging of the pixels, then the pairs one after another; with little L1 beside the shared memory every tap
      // fetches the lines of its filters anew
      const double cost = 4.7 + 0.4 * strips * rows / 128.0 + per * (bn == 64 ? 1.05 : 0.5) * std::min(1.0, (double)nc / bn) * (smem > 140000 ? 1.6 : 1.0);
      if (best.ranks == 0 || cost < best_cost) {
        best_cost = best.time = cost;
        best.bn = bn; best.ranks = s; best.per = per; best.share = share; best.strips = strips; best.strip_rows = rows;
        best.smem = (int)smem; best.tiles_m = (int)tiles_m; best.tiles_n = tiles_n;
      }
    }
  }
  if (best.ranks) best.geo = geo;
  return best;
}
static const SmallPlan& plan_small(const ConvGeom& g, bool is_dx) {
  thread_local PlanCache<SmallPlan> cache;
  return cache.get(g, is_dx, [&] { return make_plan(g, is_dx); });
}

static cudaError_t opt_in() {
  static std::once_flag once;
  static cudaError_t err = cudaSuccess;
  std::call_once(once, [] {
    err = cudaFuncSetAttribute(conv_small_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
    if (err == cudaSuccess) err = cudaFuncSetAttribute(conv_small_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
  });
  return err;
}
static int clusters_at_once(int ranks) {
  static std::once_flag once;
  static int count[MAX_RANKS + 1] = {};
  std::call_once(once, [] {
    for (int r = 1; r <= MAX_RANKS; ++r) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3(1024, (unsigned)r); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = SMEM_LIMIT;
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim.x = 1; attr.val.clusterDim.y = (unsigned)r; attr.val.clusterDim.z = 1;
      cfg.attrs = &attr; cfg.numAttrs = 1;
      int n = 0;
      if (opt_in() == cudaSuccess && cudaOccupancyMaxActiveClusters(&n, conv_small_kernel<64>, &cfg) == cudaSuccess) count[r] = n;
    }
    (void)cudaGetLastError();
  });
  return count[ranks];
}

template <int BN>
static int launch(const SmallArgs& a, const SmallPlan& p, cudaStream_t st) {
  B200_CUDA(opt_in());
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(p.tiles_m * p.tiles_n), (unsigned)p.ranks); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = (size_t)p.smem; cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = (unsigned)p.ranks; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  B200_CUDA(cudaLaunchKernelEx(&cfg, conv_small_kernel<BN>, a));
  count_launch();
  return launch_check("conv_small_kernel");
}

}  // namespace tsm

// Whether the layer is better off here than on the strip kernels.  Their time model is about a fifth above what single images take, and
// with slices of the reduction they stay below 16 us.
bool conv_small_wanted(const ConvGeom& g, bool is_dx, bool allow_transposed) {
  const tsm::SmallPlan& p = tsm::plan_small(g, is_dx);
  if (!p.ranks || getenv("B200_CONV_TC_VARIANT")) return false;   // testing aid: a pinned kernel
  const bool transposed = allow_transposed && tstrip_supported(g, is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD);
  return p.time < 0.75 * std::min(16.0, transposed ? tstrip_time(g, is_dx, nullptr) : strip_time(g, is_dx, nullptr));
}

int conv_small(const ConvGeom& g, bool is_dx, View4 act, View4 w, const float* bias, long long bias_stride, const StripPostOps* post, float* out,
               cudaStream_t st) {
  using namespace tsm;
  const SmallPlan& p = plan_small(g, is_dx);
  if (!p.ranks) return fail(B200_EUNSUPPORTED, "one-launch convolution kernel does not take this geometry");
  SmallArgs a{};
  a.g = g; a.act = act; a.w = w; a.bias = bias; a.bias_stride = bias_stride; a.out = out;
  if (post) { a.res = post->residual; a.relu = post->relu; }
  a.is_dx = is_dx ? 1 : 0;
  a.H = p.geo.gh; a.W = p.geo.gw; a.pr = p.geo.pr; a.pc = p.geo.pc;
  a.act_h = p.geo.act_h; a.act_w = p.geo.act_w; a.out_h = p.geo.out_h; a.out_w = p.geo.out_w;
  a.kc = is_dx ? g.cog : g.cig; a.nc = is_dx ? g.cig : g.cog;
  a.taps = p.geo.tt.taps_total; a.units = (a.kc + KBLK - 1) / KBLK * a.taps; a.per = p.per;
  a.tiles_n = p.tiles_n; a.q_total = (int)((long long)g.n * (a.H + a.pr) * (a.W + a.pc));
  a.strips = p.strips; a.strip_rows = p.strip_rows; a.share = p.share;
  a.act_quads = channel_quads_aligned(act, a.kc, 1) ? 1 : 0;
  a.rows_first = std::llabs(is_dx ? w.s1 : w.s0) < std::llabs(is_dx ? w.s0 : w.s1) ? 1 : 0;
  a.img_div = FastDiv((uint32_t)((a.H + a.pr) * (a.W + a.pc))); a.row_div = FastDiv((uint32_t)(a.W + a.pc));
  a.tap_div = FastDiv((uint32_t)a.taps); a.share_div = FastDiv((uint32_t)a.share);
  for (int t = 0; t < a.taps; ++t) { a.shift[t] = p.geo.tt.shift[t]; a.ky[t] = p.geo.tt.ky[t]; a.kx[t] = p.geo.tt.kx[t]; }
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  return p.bn == 64 ? launch<64>(a, p, st) : launch<32>(a, p, st);
}

}  // namespace b200

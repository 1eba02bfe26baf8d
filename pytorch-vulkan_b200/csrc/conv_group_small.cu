// CUDA-core kernels for grouped 3x3 convolutions with FEW channels per group (4 or 8 in and out), stride 1,
// dilation 1, padding 1: forward, dInput and dWeight.
//
// These are the groups=32 layers of a U-Net block at 128 / 256 channels.  With 4 or 8 channels per group the
// contraction per output is 36 or 72 long: the layers move 8 bytes per 9 to 18 FLOP, so their roofline is HBM, and
// an implicit-GEMM tile of 64 rows per group (conv_simt.cu) would spend nine tenths of its multiply-adds on padding.
// Here the tile follows the group instead: a thread block owns (image, group, 16 rows x 64 columns), brings the
// group's input tile (with its one-pixel halo) into shared memory once, and every thread keeps a 1 x 4 pixel strip
// of ALL the group's output channels in registers, so an input value is loaded once for up to 3 x 8 multiply-adds.
//   forward / dInput   one kernel; dInput runs it on dy with the filter rotated by 180 degrees and its channel roles
//                      exchanged (prepared in shared memory while the tile loads)
//   dWeight            each thread accumulates a 4 x 2 block of channel pairs with their nine taps over its pixel strips in
//                      registers; a block reduces them with warp shuffles and writes one partial per block; a second kernel
//                      sums the partials in a fixed order (no atomics: results are identical from run to run)
// Inputs are read through their strides (NCHW: a warp reads consecutive pixels of a channel; channels-last: the
// channels of a pixel first); results are contiguous NCHW.
//
// Replaces csrc/shaders/conv2d_depthwise.comp:1-41 and the small-channel side of the heuristic
// (csrc/ops/convolution.cpp:459-463) of the reference for these geometries.
#include "common.cuh"

#include <algorithm>

namespace b200 {
namespace gcs {

constexpr int THREADS = 256;

struct GArgs {
  View4 in;            // forward: x.  dInput: dy.  Logical [n][c][h][w]
  View4 w;             // [cout][cin/g][3][3]
  const float* bias;   // forward only
  long long bias_stride;
  float* out;          // contiguous [n][c][h][w]
  int n, c, h, w_, groups;
  int tiles_y, tiles_x;
  int transposed;      // dInput: use w[ci][co][2-ky][2-kx]
};

__device__ __forceinline__ void cp_async(uint32_t dst, const float* src, int bytes, bool inside) {  // zeros where the source lies outside
  if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(inside ? 16 : 0) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(inside ? 4 : 0) : "memory");
}
// two FP32 multiply-adds in one instruction, each rounded as fmaf
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long both(float v) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}

// y[n, g*CPG + co, y, x] = bias + sum_{ci, ky, kx} in[n, g*CPG + ci, y + ky - 1, x + kx - 1] * W[co][ci][ky][kx]
// SX strips of 4 pixels per tile row: the tile is (256 / SX) rows x (4 * SX) columns (16 x 64 for wide images,
// 32 x 32 for maps up to 32 columns, so that no thread idles on padding).
// One CTA per tile and a few tiles per SM, all in step: a tile's loads are latency, so every one of them is issued before any is waited
// for (asynchronous copies; through registers four at a time where rows are not 16-byte aligned), and the multiply-adds run two to an
// instruction, paired over output channels.  256 channels of 16 images of 32x32: 35 us from a
// sliced view and 25 from a dense one, now 28 and 19.
template <int CPG, int SX>
__global__ void __launch_bounds__(THREADS, 4) gconv_fwd_kernel(const GArgs a) {
  wait_previous();
  constexpr int TWK = 4 * SX, THK = THREADS / SX;         // tile extent
  constexpr int IWK = TWK + 8, IHK = THK + 2;              // with halo; image column x0 + c at c + 4, so that 16-byte pieces stay aligned
  __shared__ __align__(16) float s_in[CPG][IHK][IWK];
  __shared__ __align__(16) float s_w[CPG][3][3][CPG];   // [ci][ky][kx][co]: the co of one tap are one vector
  const int tid = threadIdx.x;
  int b = blockIdx.x;
  const int tx_tile = b % a.tiles_x; b /= a.tiles_x;
  const int ty_tile = b % a.tiles_y; b /= a.tiles_y;
  const int g = b % a.groups;
  const int n = b / a.groups;
  const int y0 = ty_tile * THK, x0 = tx_tile * TWK;
  const long long chan0 = (long long)g * CPG;

  // filter of the group
  for (int i = tid; i < CPG * CPG * 9; i += THREADS) {
    const int co = i % CPG, kx = (i / CPG) % 3, ky = (i / (CPG * 3)) % 3, ci = i / (CPG * 9);
    // forward: W[g*CPG + co][ci][ky][kx].  dInput: the output channel of this pass is the filter's input channel:
    // W[g*CPG + ci][co][2 - ky][2 - kx]
    const float v = a.transposed ? a.w.ptr[(chan0 + ci) * a.w.s0 + co * a.w.s1 + (2 - ky) * a.w.s2 + (2 - kx) * a.w.s3]
                                 : a.w.ptr[(chan0 + co) * a.w.s0 + ci * a.w.s1 + ky * a.w.s2 + kx * a.w.s3];
    s_w[ci][ky][kx][co] = v;
  }
  // input tile with halo; out-of-image pixels are zero
  const float* src = a.in.ptr + n * a.in.s0 + chan0 * a.in.s1;
  const uint32_t tile = (uint32_t)__cvta_generic_to_shared(&s_in[0][0][0]);
  auto copy = [&](int ci, int r, int c, int bytes) {      // c: image column relative to x0
    const int y = y0 - 1 + r, x = x0 + c;
    const bool inside = y >= 0 && y < a.h && x >= 0 && x < a.w_;
    cp_async(tile + 4u * (uint32_t)((ci * IHK + r) * IWK + c + 4), inside ? src + (ci * a.in.s1 + y * a.in.s2 + x * a.in.s3) : a.in.ptr, bytes, inside);
  };
  const bool rows_vec = a.in.s3 == 1 && a.in.s2 % 4 == 0 && a.in.s1 % 4 == 0 && a.in.s0 % 4 == 0 &&
                        ((reinterpret_cast<uintptr_t>(a.in.ptr) & 15) == 0) && x0 + TWK <= a.w_;
  if (rows_vec) {              // planes with contiguous rows: 16 bytes at a time, the two halo columns alone
    for (int i = tid; i < CPG * IHK * SX; i += THREADS) copy(i / (SX * IHK), (i / SX) % IHK, 4 * (i % SX), 16);
    for (int i = tid; i < CPG * IHK * 2; i += THREADS) copy(i / (2 * IHK), (i >> 1) % IHK, i & 1 ? TWK : -1, 4);
  } else if (a.in.s1 == 1) {   // channels-last: the channels of a pixel are adjacent
    for (int i = tid; i < CPG * IHK * (TWK + 2); i += THREADS) copy(i % CPG, i / (CPG * (TWK + 2)), (i / CPG) % (TWK + 2) - 1, 4);
  } else {
    for (int i = tid; i < CPG * IHK * (TWK + 2); i += THREADS) copy(i / ((TWK + 2) * IHK), (i / (TWK + 2)) % IHK, i % (TWK + 2) - 1, 4);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  const int tx = tid % SX, ty = tid / SX;   // strip of 4 pixels: row ty, columns 4*tx .. 4*tx+3
  unsigned long long pair[CPG / 2][4];      // output channels 2q and 2q + 1 of four pixels
#pragma unroll
  for (int q = 0; q < CPG / 2; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) pair[q][j] = 0ull;
#pragma unroll
  for (int ci = 0; ci < CPG; ++ci) {
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      const float* row = &s_in[ci][ty + ky][4 * tx + 3];
      const float4 p = *reinterpret_cast<const float4*>(row + 1);
      const unsigned long long v[6] = {both(row[0]), both(p.x), both(p.y), both(p.z), both(p.w), both(row[5])};
#pragma unroll
      for (int kx = 0; kx < 3; ++kx) {
        unsigned long long wv[CPG / 2];
#pragma unroll
        for (int q = 0; q < CPG / 4; ++q) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&s_w[ci][ky][kx][4 * q]);
          wv[2 * q] = t.x; wv[2 * q + 1] = t.y;
        }
#pragma unroll
        for (int q = 0; q < CPG / 2; ++q)
#pragma unroll
          for (int j = 0; j < 4; ++j) pair[q][j] = fma2(v[j + kx], wv[q], pair[q][j]);
      }
    }
  }
  float acc[CPG][4];
#pragma unroll
  for (int q = 0; q < CPG / 2; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[2 * q][j]), "=f"(acc[2 * q + 1][j]) : "l"(pair[q][j]));
  const int y = y0 + ty, x = x0 + 4 * tx;
  if (y >= a.h || x >= a.w_) return;
  const long long plane = (long long)a.h * a.w_;
  float* out = a.out + (n * (long long)a.c + chan0) * plane + (long long)y * a.w_ + x;
  const bool vec = x + 3 < a.w_ && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) && (plane % 4 == 0);
#pragma unroll
  for (int co = 0; co < CPG; ++co) {
    const float bv = a.bias ? __ldg(a.bias + (chan0 + co) * a.bias_stride) : 0.f;
    float* p = out + co * plane;
    if (vec) {
      *reinterpret_cast<float4*>(p) = make_float4(acc[co][0] + bv, acc[co][1] + bv, acc[co][2] + bv, acc[co][3] + bv);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < a.w_) p[j] = acc[co][j] + bv;
    }
  }
}

// ---- dWeight -------------------------------------------------------------------------------------------------------
// dW[g*CPG + co][ci][ky][kx] = sum_{n, y, x} dy[n, g*CPG + co, y, x] * x[n, g*CPG + ci, y + ky - 1, x + kx - 1]
// Bound by the FP32 multiply-adds (CPG * 9 per dy value) and by the shared-memory reads that feed them.  A thread owns
// strips of 8 pixels and a 4 x 2 block of (output, input) channels: its 72 sums stay in registers, and the ten x values of
// a filter row feed 4 * 3 * 8 multiply-adds, so the reads take under half the time of the arithmetic (one output channel
// and 4 pixels per thread read as much for an eighth of the work: 151 us at 256 channels, 32x32, batch 16; 32 us now, the
// input a channel slice of a wider tensor).
// Tiles of (128 / NQ / SX) rows x 8*SX columns arrive by 4-byte cp.async (any strides; zero fill outside the image), one or
// two tiles ahead of the one being used.
struct GdwArgs {
  View4 x, dy;
  float* partial;      // [blocks per group][cout][CPG][9]
  int n, c, h, w_, groups;
  int tiles_y, tiles_x, tiles_per_block, blocks_per_group;
};
constexpr int DW_THREADS = 128, DW_PITCH = 36;   // the pitch keeps 8-float strips of two rows on distinct banks
template <int CPG> constexpr int dw_stages = CPG == 4 ? 2 : 3;   // within 48 KB
template <int CPG> constexpr int dw_rows = DW_THREADS / (CPG * CPG / 8) / 4;   // tile rows (4 strips of 8 per row)

__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool ok) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
}

template <int CPG>
__global__ void __launch_bounds__(DW_THREADS, 3) gconv_dw_kernel(const GdwArgs a) {
  wait_previous();
  constexpr int NQ = CPG * CPG / 8;             // 4 x 2 channel blocks of a group
  constexpr int STRIPS = DW_THREADS / NQ;       // strips per tile
  constexpr int SX = 4, TR = STRIPS / SX, TW = 8 * SX;   // strips per row, rows, columns
  constexpr int WARPS = DW_THREADS / 32, DW_STAGES = dw_stages<CPG>;
  __shared__ __align__(16) float s_x[DW_STAGES][CPG][TR + 2][DW_PITCH];
  __shared__ __align__(16) float s_dy[DW_STAGES][CPG][TR][DW_PITCH];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = blockIdx.x / a.blocks_per_group, pb = blockIdx.x % a.blocks_per_group;
  const long long chan0 = (long long)g * CPG;
  const int q = tid / STRIPS, strip = tid % STRIPS;
  const int co0 = (q / (CPG / 2)) * 4, ci0 = (q % (CPG / 2)) * 2;
  const int ty = strip / SX, sx = strip % SX;
  float acc[72];       // [co 4][ci 2][tap 9]
#pragma unroll
  for (int i = 0; i < 72; ++i) acc[i] = 0.f;
  const int tiles_img = a.tiles_y * a.tiles_x, tiles_all = a.n * tiles_img;
  const int t_begin = pb * a.tiles_per_block, t_end = min(tiles_all, t_begin + a.tiles_per_block);

  auto load_tile = [&](int t, int stage) {
    const int n = t / tiles_img, rem = t - n * tiles_img;
    const int tyi = rem / a.tiles_x, y0 = tyi * TR, x0 = (rem - tyi * a.tiles_x) * TW;
    const float* px = a.x.ptr + n * a.x.s0 + chan0 * a.x.s1;
    const float* pd = a.dy.ptr + n * a.dy.s0 + chan0 * a.dy.s1;
    if (a.x.s1 == 1) {   // channels-last: the channels of a pixel are adjacent
      for (int i = tid; i < CPG * (TR + 2) * (TW + 2); i += DW_THREADS) {
        const int ci = i % CPG, c = (i / CPG) % (TW + 2), r = i / (CPG * (TW + 2)), y = y0 - 1 + r, x = x0 - 1 + c;
        const bool ok = y >= 0 && y < a.h && x >= 0 && x < a.w_;
        cp_async4(&s_x[stage][ci][r][c], ok ? px + ci + (long long)y * a.x.s2 + (long long)x * a.x.s3 : a.x.ptr, ok);
      }
    } else {             // a warp copies one row of 32 columns at a time, then the two last columns of all rows
      const int x = x0 - 1 + lane;
      const bool xok = x >= 0 && x < a.w_;
#pragma unroll
      for (int i = warp; i < CPG * (TR + 2); i += WARPS) {
        const int ci = i / (TR + 2), r = i % (TR + 2), y = y0 - 1 + r;
        const bool ok = xok && y >= 0 && y < a.h;
        cp_async4(&s_x[stage][ci][r][lane], ok ? px + ci * a.x.s1 + (long long)y * a.x.s2 + (long long)x * a.x.s3 : a.x.ptr, ok);
      }
      for (int i = tid; i < CPG * (TR + 2) * 2; i += DW_THREADS) {
        const int c = 32 + (i & 1), r = (i >> 1) % (TR + 2), ci = (i >> 1) / (TR + 2), y = y0 - 1 + r, xe = x0 - 1 + c;
        const bool ok = xe < a.w_ && y >= 0 && y < a.h;
        cp_async4(&s_x[stage][ci][r][c], ok ? px + ci * a.x.s1 + (long long)y * a.x.s2 + (long long)xe * a.x.s3 : a.x.ptr, ok);
      }
    }
    if (a.dy.s1 == 1) {
#pragma unroll
      for (int i = tid; i < CPG * TR * TW; i += DW_THREADS) {
        const int co = i % CPG, c = (i / CPG) % TW, r = i / (CPG * TW), y = y0 + r, x = x0 + c;
        const bool ok = y < a.h && x < a.w_;
        cp_async4(&s_dy[stage][co][r][c], ok ? pd + co + (long long)y * a.dy.s2 + (long long)x * a.dy.s3 : a.dy.ptr, ok);
      }
    } else {
      const int x = x0 + lane;
#pragma unroll
      for (int i = warp; i < CPG * TR; i += WARPS) {
        const int co = i / TR, r = i % TR, y = y0 + r;
        const bool ok = x < a.w_ && y < a.h;
        cp_async4(&s_dy[stage][co][r][lane], ok ? pd + co * a.dy.s1 + (long long)y * a.dy.s2 + (long long)x * a.dy.s3 : a.dy.ptr, ok);
      }
    }
  };

#pragma unroll
  for (int s = 0; s < DW_STAGES - 1; ++s) {
    if (t_begin + s < t_end) load_tile(t_begin + s, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0;
  for (int t = t_begin; t < t_end; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DW_STAGES - 2) : "memory");
    __syncthreads();   // tile t has landed for every thread, and the stage of tile t - 1 has been consumed
    {
      const int ahead = t + DW_STAGES - 1;
      if (ahead < t_end) load_tile(ahead, stage == 0 ? DW_STAGES - 1 : stage - 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float d[4][8];
#pragma unroll
    for (int co = 0; co < 4; ++co) {
      const float4 lo = *reinterpret_cast<const float4*>(&s_dy[stage][co0 + co][ty][8 * sx]);
      const float4 hi = *reinterpret_cast<const float4*>(&s_dy[stage][co0 + co][ty][8 * sx + 4]);
      d[co][0] = lo.x; d[co][1] = lo.y; d[co][2] = lo.z; d[co][3] = lo.w;
      d[co][4] = hi.x; d[co][5] = hi.y; d[co][6] = hi.z; d[co][7] = hi.w;
    }
#pragma unroll
    for (int ci = 0; ci < 2; ++ci)
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const float* row = &s_x[stage][ci0 + ci][ty + ky][8 * sx];
        const float4 p0 = *reinterpret_cast<const float4*>(row), p1 = *reinterpret_cast<const float4*>(row + 4);
        const float2 p2 = *reinterpret_cast<const float2*>(row + 8);
        const float v[10] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w, p2.x, p2.y};
#pragma unroll
        for (int co = 0; co < 4; ++co)
#pragma unroll
          for (int kx = 0; kx < 3; ++kx)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[(co * 2 + ci) * 9 + ky * 3 + kx] = fmaf(d[co][j], v[j + kx], acc[(co * 2 + ci) * 9 + ky * 3 + kx]);
      }
    if (++stage == DW_STAGES) stage = 0;
  }
  // Sum over the strips of a channel block: three halving exchanges over lane bits 3, 2, 1 (after each, a lane keeps half of the
  // values, summed over the pair), then plain exchanges over the remaining lane bits, in a fixed order.
  {
    int keep = 36;
#pragma unroll
    for (int step = 0; step < 3; ++step, keep /= 2) {
      const int o = 8 >> step;
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < 36; ++i)
        if (i < keep) {
          const float mine = upper ? acc[keep + i] : acc[i], theirs = upper ? acc[i] : acc[keep + i];
          acc[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 1);
    if (STRIPS >= 32) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 16);
  }
  // lane bits 3..1 select nine adjacent values: piece = (co, ci) of the channel block
  const int piece = ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
  const int co = co0 + (piece >> 1), ci = ci0 + (piece & 1);
  float* out = a.partial + ((long long)pb * a.c + chan0 + co) * (CPG * 9) + ci * 9;
  if (STRIPS <= 32) {
    if ((lane & 1) == 0 && (STRIPS < 32 || lane < 16)) {
#pragma unroll
      for (int i = 0; i < 9; ++i) out[i] = acc[i];
    }
  } else {               // several warps hold the same channel block (4 channels per group: two)
    constexpr int WPQ = STRIPS / 32 > 0 ? STRIPS / 32 : 1;
    __shared__ float s_red[WARPS][72];
    if ((lane & 1) == 0 && lane < 16)
#pragma unroll
      for (int i = 0; i < 9; ++i) s_red[warp][piece * 9 + i] = acc[i];
    __syncthreads();
    if (warp % WPQ == 0 && (lane & 1) == 0 && lane < 16) {
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        float v = acc[i];
        for (int w = 1; w < WPQ; ++w) v += s_red[warp + w][piece * 9 + i];
        out[i] = v;
      }
    }
  }
}

}  // namespace gcs

// 3x3, stride 1, dilation 1, padding 1, the same small channel count (4 or 8) in and out of every group
bool group_small_supported(const ConvGeom& g) {
  return g.kh == 3 && g.kw == 3 && g.sh == 1 && g.sw == 1 && g.dh == 1 && g.dw == 1 && g.ph == 1 && g.pw == 1 && g.cig == g.cog &&
         (g.cig == 4 || g.cig == 8) && g.groups >= 2 && g.oh == g.h && g.ow == g.w;
}

static void dw_tiling(const ConvGeom& g, int* tiles_y, int* tiles_x, int* tiles_per_block, int* blocks_per_group) {
  const int th = g.cig == 4 ? gcs::dw_rows<4> : gcs::dw_rows<8>;
  *tiles_y = (g.h + th - 1) / th;
  *tiles_x = (g.w + 31) / 32;
  const long long tiles_all = (long long)g.n * *tiles_y * *tiles_x;
  // three blocks per SM are resident (registers); at least four tiles per block, so that the pipeline and the block's reduction
  // are a small part of it
  const long long bpg = std::max<long long>(1, std::min<long long>(tiles_all / 4, 3ll * sm_count() / g.groups));
  *tiles_per_block = (int)div_up64(tiles_all, bpg);
  *blocks_per_group = (int)div_up64(tiles_all, *tiles_per_block);
}

size_t group_small_dweight_workspace(const ConvGeom& g) {
  int ty, tx, tpb, bpg;
  dw_tiling(g, &ty, &tx, &tpb, &bpg);
  return (size_t)bpg * g.cout * g.cig * 9 * sizeof(float);
}

int group_small_conv(const ConvGeom& g, bool is_dx, View4 in, View4 w, const float* bias, long long bias_stride, float* out, cudaStream_t st) {
  gcs::GArgs a{};
  a.in = in; a.w = w; a.bias = is_dx ? nullptr : bias; a.bias_stride = bias_stride; a.out = out;
  a.n = g.n; a.c = g.cin; a.h = g.h; a.w_ = g.w; a.groups = g.groups;
  const bool narrow = g.w <= 32;   // 32 x 32 tiles for small maps, 16 x 64 otherwise
  const int th = narrow ? 32 : 16, tw = narrow ? 32 : 64;
  a.tiles_y = (g.h + th - 1) / th; a.tiles_x = (g.w + tw - 1) / tw;
  a.transposed = is_dx ? 1 : 0;
  const long long blocks = (long long)g.n * g.groups * a.tiles_y * a.tiles_x;
  if (blocks > 2147483647ll) return fail(B200_ERANGE, "grouped convolution: grid exceeds launch limits");
  const unsigned nb = (unsigned)blocks;
  if (g.cig == 4) {
    if (narrow) launch_next(gcs::gconv_fwd_kernel<4, 8>, nb, gcs::THREADS, 0, st, a);
    else launch_next(gcs::gconv_fwd_kernel<4, 16>, nb, gcs::THREADS, 0, st, a);
  } else {
    if (narrow) launch_next(gcs::gconv_fwd_kernel<8, 8>, nb, gcs::THREADS, 0, st, a);
    else launch_next(gcs::gconv_fwd_kernel<8, 16>, nb, gcs::THREADS, 0, st, a);
  }
  count_launch();
  return launch_check("gconv_fwd_kernel");
}

int group_small_dweight(const ConvGeom& g, View4 x, View4 dy, float* dw, float* ws, size_t ws_bytes, cudaStream_t st) {
  gcs::GdwArgs a{};
  a.x = x; a.dy = dy; a.n = g.n; a.c = g.cin; a.h = g.h; a.w_ = g.w; a.groups = g.groups;
  dw_tiling(g, &a.tiles_y, &a.tiles_x, &a.tiles_per_block, &a.blocks_per_group);
  const size_t need = group_small_dweight_workspace(g);
  const long long count = (long long)g.cout * g.cig * 9;
  if (a.blocks_per_group > 1 && (!ws || ws_bytes < need))
    return fail(B200_EWORKSPACE, "grouped dWeight needs a workspace of %zu bytes (got %zu)", need, ws_bytes);
  a.partial = a.blocks_per_group > 1 ? ws : dw;   // one block per group writes dW directly ([cout][cig][9])
  const long long blocks = (long long)g.groups * a.blocks_per_group;
  if (g.cig == 4) launch_next(gcs::gconv_dw_kernel<4>, (unsigned)blocks, gcs::DW_THREADS, 0, st, a);
  else launch_next(gcs::gconv_dw_kernel<8>, (unsigned)blocks, gcs::DW_THREADS, 0, st, a);
  count_launch();
  if (int rc = launch_check("gconv_dw_kernel")) return rc;
  if (a.blocks_per_group > 1) return finalize_splits(ws, dw, count, a.blocks_per_group, st);
  return B200_OK;
}

}  // namespace b200

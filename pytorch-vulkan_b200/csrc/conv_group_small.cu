// CUDA-core kernels for grouped 3x3 convolutions with FEW channels per group (4 or 8 in and out), stride 1,
// dilation 1, padding 1: forward, dInput and dWeight.
//
// These are the groups=32 layers of a U-Net block at 128 / 256 channels.  With 4 or 8 channels per group the
// contraction per output is 36 or 72 long: the layers move 8 bytes per 9 to 18 FLOP, so their roofline is HBM, and
// an implicit-GEMM tile of 64 rows per group (conv_simt.cu) would spend nine tenths of its multiply-adds on padding.
// Here the tile follows the group instead: a thread block owns (image, group, 16 rows x 64 columns), brings the
// group's input tile (with its one-pixel halo) into shared memory once, and every thread keeps a 2 x 4 pixel strip
// of all the group's output channels (or half of them) in registers, so an input value is loaded once for up to 3 x 8 multiply-adds.
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
#include <type_traits>

namespace b200 {
namespace gcs {

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
// A tile is 16 rows x (4 * SX) columns of one group (64 columns for wide images, 32 for maps up to 32); a thread keeps 2 rows x 4 columns
// of all the group's output channels.
// Bound by the FP32 multiply-adds, and before them by everything that does not run beside them:
//   * the tile's copies are issued at once and waited for two input channels at a time, so the arithmetic starts when the first two have landed;
//   * two rows a thread share the input rows between them: three reads of an input row feed up to 96 paired multiply-adds;
//   * tiles of 16 rows leave at most seven on an SM where tiles of 32 left four of 3.5 on average;
//   * every product of an input value follows one doubling of it, and the copies walk rows and channels by additions.
// 256 channels of 16 images of 32x32 in 32 groups: 28.1 us from a sliced view and 19.3 from a dense one, now 19.5 and 17.3 (the multiply-adds
// alone are 8.3), and with
//   * where all tiles run at once a thread keeps half of the group's eight channels (CO): twice the warps hide the latency of the one wave.
//     256 channels of 16 images of 32x32: 19.5 -> 18.8 and 17.3 -> 16.9.  Beyond a wave, and for the tiles of wide images, the doubled reads of
//     the input cost more than that (60 images of 20x20 51.2 -> 56.1, 33 of 43x43 87 -> 103).
template <int CPG, int SX, int CO>
__global__ void __launch_bounds__(8 * SX * (CPG / CO), CPG != CO ? 7 : SX == 8 ? 8 : 4) gconv_fwd_kernel(const GArgs a) {
  wait_previous();
  constexpr int STRIPS = 8 * SX;                           // SX strips x 8 row pairs
  constexpr int NT = STRIPS * (CPG / CO), WARPS = NT / 32;
  constexpr int TWK = 4 * SX, THK = 16;                    // tile extent
  constexpr int IWK = TWK + 8, IHK = THK + 2;              // with halo; image column x0 + c at c + 4, so that 16-byte pieces stay aligned
  constexpr int STAGES = CPG / 2;                          // of two input channels
  __shared__ __align__(16) float s_in[CPG][IHK][IWK];
  __shared__ __align__(16) float s_w[CPG][3][3][CPG];   // [ci][ky][kx][co]: the co of one tap are one vector
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = blockIdx.x;
  const int tx_tile = b % a.tiles_x; b /= a.tiles_x;
  const int ty_tile = b % a.tiles_y; b /= a.tiles_y;
  const int g = b % a.groups;
  const int n = b / a.groups;
  const int y0 = ty_tile * THK, x0 = tx_tile * TWK;
  const long long chan0 = (long long)g * CPG;

  // filter of the group, with the first stage: a thread copies the nine taps of a channel pair
  for (int i = tid; i < CPG * CPG; i += NT) {
    const int co = i % CPG, ci = i / CPG;
    // forward: W[g*CPG + co][ci][ky][kx].  dInput: the output channel of this pass is the filter's input channel:
    // W[g*CPG + ci][co][2 - ky][2 - kx]
    const float* src = a.w.ptr + (chan0 + (a.transposed ? ci : co)) * a.w.s0 + (a.transposed ? co : ci) * a.w.s1;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s_w[ci][0][0][co]);
#pragma unroll
    for (int t = 0; t < 9; ++t) cp_async(dst + 4 * CPG * (a.transposed ? 8 - t : t), src + (t / 3) * a.w.s2 + (t % 3) * a.w.s3, 4, true);
  }
  // Input tile with halo; out-of-image pixels are zero.  Every thread keeps its column and walks rows and channels by additions: with the
  // addresses computed for each copy, 40 instructions of a copy took twice the issue slots of the multiply-adds.
  const float* src = a.in.ptr + n * a.in.s0 + chan0 * a.in.s1;
  const uint32_t tile = (uint32_t)__cvta_generic_to_shared(&s_in[0][0][0]);
  const long long s1 = a.in.s1, s2 = a.in.s2;
  constexpr uint32_t ROW = 4 * IWK, PLANE = 4 * IHK * IWK;
  const bool rows_vec = a.in.s3 == 1 && a.in.s2 % 4 == 0 && a.in.s1 % 4 == 0 && a.in.s0 % 4 == 0 &&
                        ((reinterpret_cast<uintptr_t>(a.in.ptr) & 15) == 0) && x0 + TWK <= a.w_;
  const bool pixels = a.in.s1 == 1 && a.in.s3 != 1;        // channels-last: the channels of a pixel are adjacent
  // rows r0, r0 + STEP, ... of two channels at image column x (tile column x - x0 + 4)
  auto column = [&](int ci, int r0, int x, auto step, auto piece) {
    constexpr int STEP = decltype(step)::value, BYTES = decltype(piece)::value;
    const bool xin = x >= 0 && x < a.w_;
    const float* p = src + ci * s1 + (y0 - 1 + r0) * s2 + x * a.in.s3;
    uint32_t dst = tile + ci * PLANE + r0 * ROW + 4u * (uint32_t)(x - x0 + 4);
#pragma unroll
    for (int r = r0; r < IHK; r += STEP, p += STEP * s2, dst += STEP * ROW) {
      const int y = y0 - 1 + r;
      const bool in = xin && y >= 0 && y < a.h;
      cp_async(dst, in ? p : a.in.ptr, BYTES, in);
      cp_async(dst + PLANE, in ? p + s1 : a.in.ptr, BYTES, in);
    }
  };
  if (pixels) {                                            // a thread keeps its channel
    const int ci = tid % CPG;
    for (int i = tid / CPG; i < IHK * (TWK + 2); i += NT / CPG) {
      const int r = i / (TWK + 2), c = i - r * (TWK + 2), y = y0 - 1 + r, x = x0 - 1 + c;
      const bool in = x >= 0 && x < a.w_ && y >= 0 && y < a.h;
      cp_async(tile + ci * PLANE + r * ROW + 4u * (uint32_t)(c + 3), in ? src + ci + (y * s2 + x * a.in.s3) : a.in.ptr, 4, in);
    }
  }
#pragma unroll 1
  for (int s = 0; s < STAGES; ++s) {
    if (!pixels) {
      using std::integral_constant;
      if (rows_vec) {            // planes with contiguous rows: 16 bytes at a time
        column(2 * s, tid / SX, x0 + 4 * (tid % SX), integral_constant<int, NT / SX>{}, integral_constant<int, 16>{});
      } else {                   // a warp copies a row of 32 columns at a time
#pragma unroll
        for (int c = 0; c < TWK; c += 32) column(2 * s, warp, x0 + c + lane, integral_constant<int, WARPS>{}, integral_constant<int, 4>{});
      }
      if (tid < 2 * IHK) column(2 * s, tid >> 1, x0 + (tid & 1 ? TWK : -1), integral_constant<int, IHK>{}, integral_constant<int, 4>{});   // the halo columns
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  const int tx = tid % SX, ty = tid % STRIPS / SX, co0 = tid / STRIPS * CO;   // rows 2*ty and 2*ty + 1, columns 4*tx .. 4*tx+3
  unsigned long long pair[2][CO / 2][4];    // output channels co0 + 2q and co0 + 2q + 1 of four pixels in two rows
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < CO / 2; ++q)
#pragma unroll
      for (int j = 0; j < 4; ++j) pair[r][q][j] = 0ull;
#pragma unroll 1
  for (int ci = 0; ci < CPG; ++ci) {
    if ((ci & 1) == 0) {                    // this stage has landed for every thread
      if (ci == 0) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
      else if (ci == 2) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES > 2 ? STAGES - 2 : 0) : "memory");
      else if (ci == 4) asm volatile("cp.async.wait_group %0;" ::"n"(STAGES > 3 ? STAGES - 3 : 0) : "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float* row = &s_in[ci][2 * ty + r][4 * tx + 3];
      const float4 p = *reinterpret_cast<const float4*>(row + 1);
      const float v[6] = {row[0], p.x, p.y, p.z, p.w, row[5]};
#pragma unroll
      for (int out = 0; out < 2; ++out) {   // input row 2*ty - 1 + r is tap ky of output row 2*ty + out
        const int ky = r - out;
        if (ky < 0 || ky > 2) continue;
        unsigned long long wv[3][CO / 2];
#pragma unroll
        for (int kx = 0; kx < 3; ++kx)
#pragma unroll
          for (int q = 0; q < CO / 4; ++q) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&s_w[ci][ky][kx][co0 + 4 * q]);
            wv[kx][2 * q] = t.x; wv[kx][2 * q + 1] = t.y;
          }
#pragma unroll
        for (int i = 0; i < 6; ++i) {       // every product of one input value, so that it is doubled once
          const unsigned long long vv = both(v[i]);
#pragma unroll
          for (int kx = 0; kx < 3; ++kx)
            if (i - kx >= 0 && i - kx < 4) {
#pragma unroll
              for (int q = 0; q < CO / 2; ++q) pair[out][q][i - kx] = fma2(vv, wv[kx][q], pair[out][q][i - kx]);
            }
        }
      }
    }
  }
  const int x = x0 + 4 * tx;
  const long long plane = (long long)a.h * a.w_;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int y = y0 + 2 * ty + r;
    if (y >= a.h || x >= a.w_) break;
    float* out = a.out + (n * (long long)a.c + chan0) * plane + (long long)y * a.w_ + x;
    const bool vec = x + 3 < a.w_ && ((reinterpret_cast<uintptr_t>(out) & 15) == 0) && (plane % 4 == 0);
#pragma unroll
    for (int q = 0; q < CO / 2; ++q) {
      float acc[2][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[0][j]), "=f"(acc[1][j]) : "l"(pair[r][q][j]));
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int co = co0 + 2 * q + i;
        const float bv = a.bias ? __ldg(a.bias + (chan0 + co) * a.bias_stride) : 0.f;
        float* p = out + co * plane;
        if (vec) {
          *reinterpret_cast<float4*>(p) = make_float4(acc[i][0] + bv, acc[i][1] + bv, acc[i][2] + bv, acc[i][3] + bv);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (x + j < a.w_) p[j] = acc[i][j] + bv;
        }
      }
    }
  }
}

// ---- dWeight -------------------------------------------------------------------------------------------------------
// dW[g*CPG + co][ci][ky][kx] = sum_{n, y, x} dy[n, g*CPG + co, y, x] * x[n, g*CPG + ci, y + ky - 1, x + kx - 1]
// Bound by the FP32 multiply-adds (CPG * 9 per dy value) and by the shared-memory reads that feed them.  A thread owns
// strips of 8 pixels and a 4 x 2 block of (output, input) channels: its 72 sums stay in registers, and the ten x values of
// a filter row feed 4 * 3 * 8 multiply-adds, so the reads take under half the time of the arithmetic (one output channel
// and 4 pixels per thread read as much for an eighth of the work: 151 us at 256 channels, 32x32, batch 16, the
// input a channel slice of a wider tensor).  The multiply-adds run two to an instruction over pairs of output channels, which lie side by side in
// shared memory: pairs put together in registers were put together again for every use (33 us; 32 without pairs, 25.5 now).
// Tiles of (128 / NQ / SX) rows x 8*SX columns arrive by 4-byte cp.async (any strides; zero fill outside the image), one or
// two tiles ahead of the one being used.
struct GdwArgs {
  View4 x, dy;
  float* partial;      // [blocks per group][cout][CPG][9]
  int n, c, h, w_, groups;
  int tiles_y, tiles_x, tiles_per_block, blocks_per_group;
};
constexpr int DW_THREADS = 128, DW_PITCH = 36, DW_DY_PITCH = 68;   // the pitches keep the strips of neighbouring rows on distinct banks
template <int CPG> constexpr int dw_stages = CPG == 4 ? 2 : 3;   // within 48 KB
template <int CPG> constexpr int dw_rows = DW_THREADS / (CPG * CPG / 8) / 4;   // tile rows (4 strips of 8 per row)

template <int CPG>
__global__ void __launch_bounds__(DW_THREADS, 3) gconv_dw_kernel(const GdwArgs a) {
  wait_previous();
  constexpr int NQ = CPG * CPG / 8;             // 4 x 2 channel blocks of a group
  constexpr int STRIPS = DW_THREADS / NQ;       // strips per tile
  constexpr int SX = 4, TR = STRIPS / SX, TW = 8 * SX;   // strips per row, rows, columns
  constexpr int WARPS = DW_THREADS / 32, DW_STAGES = dw_stages<CPG>;
  __shared__ __align__(16) float s_x[DW_STAGES][CPG][TR + 2][DW_PITCH];
  __shared__ __align__(16) float s_dy[DW_STAGES][CPG / 2][TR][DW_DY_PITCH];   // two channels of a pixel side by side: operands of fma2
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = blockIdx.x / a.blocks_per_group, pb = blockIdx.x % a.blocks_per_group;
  const long long chan0 = (long long)g * CPG;
  const int q = tid / STRIPS, strip = tid % STRIPS;
  const int co0 = (q / (CPG / 2)) * 4, ci0 = (q % (CPG / 2)) * 2;
  const int ty = strip / SX, sx = strip % SX;
  unsigned long long sums[2][2][9];    // [co pair][ci][tap]: output channels 2p and 2p + 1
#pragma unroll
  for (int i = 0; i < 36; ++i) sums[i / 18][i / 9 % 2][i % 9] = 0ull;
  const int tiles_img = a.tiles_y * a.tiles_x, tiles_all = a.n * tiles_img;
  const int t_begin = pb * a.tiles_per_block, t_end = min(tiles_all, t_begin + a.tiles_per_block);

  // what a thread copies of every tile: places in shared memory and offsets from the tile's first pixel that never change, rows and
  // channels by additions (with every address computed anew, the copies took more issue slots than the multiply-adds)
  const bool x_pixels = a.x.s1 == 1 && a.x.s3 != 1, dy_pixels = a.dy.s1 == 1 && a.dy.s3 != 1;   // channels-last
  constexpr int HALO = CPG * (TR + 2) * 2, HALOS = (HALO + DW_THREADS - 1) / DW_THREADS;   // values of the last two columns, of a thread
  const int halo_c = 32 + (tid & 1);
  int halo_r[HALOS], halo_ci[HALOS];
  long long halo_off[HALOS];
#pragma unroll
  for (int k = 0; k < HALOS; ++k) {
    const int i = (tid + k * DW_THREADS) >> 1;
    halo_r[k] = i % (TR + 2); halo_ci[k] = i / (TR + 2);
    halo_off[k] = halo_ci[k] * a.x.s1 + (halo_r[k] - 1) * a.x.s2 + (halo_c - 1) * a.x.s3;
  }
  constexpr uint32_t ROW = 4 * DW_PITCH, X_PLANE = ROW * (TR + 2), DY_ROW = 4 * DW_DY_PITCH, DY_PAIR = DY_ROW * TR,
                     X_STAGE = CPG * X_PLANE, DY_STAGE = CPG / 2 * DY_PAIR;
  const uint32_t x_smem = (uint32_t)__cvta_generic_to_shared(&s_x[0][0][0][0]), dy_smem = (uint32_t)__cvta_generic_to_shared(&s_dy[0][0][0][0]);
  auto load_tile = [&](int t, int stage) {
    const int n = t / tiles_img, rem = t - n * tiles_img;
    const int tyi = rem / a.tiles_x, y0 = tyi * TR, x0 = (rem - tyi * a.tiles_x) * TW;
    const float* px = a.x.ptr + n * a.x.s0 + chan0 * a.x.s1 + y0 * a.x.s2 + x0 * a.x.s3;     // the tile's first pixel
    const float* pd = a.dy.ptr + n * a.dy.s0 + chan0 * a.dy.s1 + y0 * a.dy.s2 + x0 * a.dy.s3;
    const uint32_t xs = x_smem + stage * X_STAGE, ds = dy_smem + stage * DY_STAGE;
    if (x_pixels) {      // a thread keeps its channel
      const int ci = tid % CPG;
      for (int i = tid / CPG; i < (TR + 2) * (TW + 2); i += DW_THREADS / CPG) {
        const int r = i / (TW + 2), c = i - r * (TW + 2), y = y0 - 1 + r, x = x0 - 1 + c;
        const bool ok = y >= 0 && y < a.h && x >= 0 && x < a.w_;
        cp_async(xs + ci * X_PLANE + r * ROW + 4 * c, ok ? px + ci + ((r - 1) * a.x.s2 + (c - 1) * a.x.s3) : a.x.ptr, 4, ok);
      }
    } else {             // a warp copies the rows of a channel, 32 columns at a time, then every thread one value of the last two columns
      const int x = x0 - 1 + lane;
      const bool xok = x >= 0 && x < a.w_;
      const float* p0 = px + warp * a.x.s1 - a.x.s2 + (lane - 1) * a.x.s3;
      uint32_t d0 = xs + warp * X_PLANE + 4 * lane;
#pragma unroll
      for (int ci = 0; ci < CPG; ci += WARPS, p0 += WARPS * a.x.s1, d0 += WARPS * X_PLANE) {
        const float* p = p0;
#pragma unroll
        for (int r = 0; r < TR + 2; ++r, p += a.x.s2) {
          const bool ok = xok && y0 - 1 + r >= 0 && y0 - 1 + r < a.h;
          cp_async(d0 + r * ROW, ok ? p : a.x.ptr, 4, ok);
        }
      }
#pragma unroll
      for (int k = 0; k < HALOS; ++k) {
        if (tid + k * DW_THREADS >= HALO) break;
        const int y = y0 - 1 + halo_r[k], xe = x0 - 1 + halo_c;
        const bool ok = xe < a.w_ && y >= 0 && y < a.h;
        cp_async(xs + halo_ci[k] * X_PLANE + halo_r[k] * ROW + 4 * halo_c, ok ? px + halo_off[k] : a.x.ptr, 4, ok);
      }
    }
    if (dy_pixels) {
      const int co = tid % CPG;
#pragma unroll 4
      for (int i = tid / CPG; i < TR * TW; i += DW_THREADS / CPG) {
        const int r = i / TW, c = i % TW;
        const bool ok = y0 + r < a.h && x0 + c < a.w_;
        cp_async(ds + (co >> 1) * DY_PAIR + r * DY_ROW + 8 * c + 4 * (co & 1), ok ? pd + co + (r * a.dy.s2 + c * a.dy.s3) : a.dy.ptr, 4, ok);
      }
    } else {
      const bool xok = x0 + lane < a.w_;
      const float* p0 = pd + warp * a.dy.s1 + lane * a.dy.s3;
      static_assert(WARPS % 2 == 0, "a warp keeps its place in the channel pair");
      uint32_t d0 = ds + (warp >> 1) * DY_PAIR + 8 * lane + 4 * (warp & 1);
#pragma unroll
      for (int co = 0; co < CPG; co += WARPS, p0 += WARPS * a.dy.s1, d0 += WARPS / 2 * DY_PAIR) {
        const float* p = p0;
#pragma unroll
        for (int r = 0; r < TR; ++r, p += a.dy.s2) {
          const bool ok = xok && y0 + r < a.h;
          cp_async(d0 + r * DY_ROW, ok ? p : a.dy.ptr, 4, ok);
        }
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
    unsigned long long d[2][8];        // eight pixels of the channel pairs
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(&s_dy[stage][co0 / 2 + p][ty][2 * (8 * sx + j)]);
        d[p][j] = t.x; d[p][j + 1] = t.y;
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
        for (int i = 0; i < 10; ++i) {
          const unsigned long long vv = both(v[i]);
#pragma unroll
          for (int kx = 0; kx < 3; ++kx)
            if (i - kx >= 0 && i - kx < 8) {
#pragma unroll
              for (int p = 0; p < 2; ++p) sums[p][ci][ky * 3 + kx] = fma2(d[p][i - kx], vv, sums[p][ci][ky * 3 + kx]);
            }
        }
      }
    if (++stage == DW_STAGES) stage = 0;
  }
  float acc[72];       // [co 4][ci 2][tap 9]
#pragma unroll
  for (int i = 0; i < 36; ++i) {
    const int p = i / 18, rest = i % 18;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[p * 36 + rest]), "=f"(acc[p * 36 + 18 + rest]) : "l"(sums[p][rest / 9][rest % 9]));
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
  const bool narrow = g.w <= 32;   // tiles of 32 columns for small maps, so that no thread idles on padding, 64 otherwise
  const int th = 16, tw = narrow ? 32 : 64;
  a.tiles_y = (g.h + th - 1) / th; a.tiles_x = (g.w + tw - 1) / tw;
  a.transposed = is_dx ? 1 : 0;
  const long long blocks = (long long)g.n * g.groups * a.tiles_y * a.tiles_x;
  if (blocks > 2147483647ll) return fail(B200_ERANGE, "grouped convolution: grid exceeds launch limits");
  const unsigned nb = (unsigned)blocks;
  if (g.cig == 4) {
    if (narrow) launch_next(gcs::gconv_fwd_kernel<4, 8, 4>, nb, 64, 0, st, a);
    else launch_next(gcs::gconv_fwd_kernel<4, 16, 4>, nb, 128, 0, st, a);
  } else {
    if (narrow && blocks <= 7ll * sm_count()) launch_next(gcs::gconv_fwd_kernel<8, 8, 4>, nb, 128, 0, st, a);   // one wave: seven CTAs fit an SM
    else if (narrow) launch_next(gcs::gconv_fwd_kernel<8, 8, 8>, nb, 64, 0, st, a);
    else launch_next(gcs::gconv_fwd_kernel<8, 16, 8>, nb, 128, 0, st, a);
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

// Operand staging shared by the two tcgen05 dWeight kernels (dweight_tc_strip.cu, dweight_tc_tmem.cu): pixel-major blocks of
// 32 rows (pixels) x 32 channels gathered from a strided view, split into TF32 / BF16 planes and written in the swizzles that
// MN-major operands need.
#pragma once
#include "common.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace tcdw {
using namespace tc;

// byte offset of channel e (0..31) of row `row` in a plane using the 128B swizzle with 32-byte base
__device__ __forceinline__ uint32_t sw32b_offset(int row, int e) {
  return (uint32_t)(row * 128 + ((((e >> 3) ^ (row & 3)) << 5) | ((e & 7) << 2)));
}
// MN-major operand descriptor: blocks of 32 channels `lbo` bytes apart, 4-row groups 512 bytes apart
__device__ __forceinline__ uint64_t make_mn_desc(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1 << 46;   // descriptor version of sm_100
  d |= (uint64_t)1 << 61;   // SWIZZLE_128B with 32-byte base
  return d;
}

// byte offset of channel e (0..31) of row `row` in a bf16 plane of 64-byte rows, SWIZZLE_64B
__device__ __forceinline__ uint32_t sw64_offset(int row, int e) {
  return (uint32_t)(row * 64 + ((((e >> 3) ^ ((row >> 1) & 3)) << 4) | ((e & 7) << 1)));
}
// MN-major descriptor of a bf16 plane (64-byte rows): blocks of 32 channels `lbo` bytes apart, 8-row
// groups 512 bytes apart, SWIZZLE_64B
__device__ __forceinline__ uint64_t make_mn_desc16(uint32_t addr, uint32_t lbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;   // SWIZZLE_64B
  return d;
}

// One warp stages `rows` (<= 32, lane = row) x 32 channels of a pixel-major block: gather from
// the strided view, split into TF32 hi/lo, swizzled stores.  `q_first` is the padded pixel of row 0;
// rows outside [q_lo, q_hi) or on padding are written as zeros.
//
// With the 32-byte-base swizzle rows r and r+4 put the same 16-byte chunk into the same banks, so
// lanes 4-7 of every group of eight write the two chunks of a 32-byte pair in the opposite order
// (every 8-lane store wavefront is then conflict-free).  To keep that free of per-value selects the
// swapped lanes already LOAD their channels in swapped order: val[j] holds channel j ^ 4 there.
__device__ __forceinline__ bool stage_block(const View4& v, long long chan0, int chans, int H, int W, int row_pitch,
                                            int img_pitch, const FastDiv& img_div, const FastDiv& row_div, int q_first,
                                            int q_lo, int q_hi, int rows, int lane, bool vec_ok, float (&val)[32],
                                            int sph = 1, int spw = 1, int pa = 0, int pb = 0, int lim_h = 1 << 30,
                                            int lim_w = 1 << 30) {
  const int q = q_first + lane;
  bool ok = lane < rows && q >= q_lo && q < q_hi;
  const float* src = v.ptr;
  if (ok) {
    const int n = (int)img_div.div((uint32_t)q);
    const int rem = q - n * img_pitch;
    const int y = (int)row_div.div((uint32_t)rem), x = rem - y * row_pitch;
    const int ty = y * sph + pa, tx = x * spw + pb;  // position in the tensor
    ok = y < H && x < W && ty < lim_h && tx < lim_w;
    src += n * v.s0 + chan0 * v.s1 + (long long)ty * v.s2 + (long long)tx * v.s3;
  }
  const int sw = (lane >> 2) & 1;
  if (vec_ok && chans == 32) {
    // Channels-last: eight lanes fetch the 128 contiguous bytes of one pixel, four pixels per load
    // instruction; lane r computed the address of row r above and hands it to the lanes that fetch
    // it.  val[4i..4i+3] is then the 16-byte chunk (lane & 7) of row 4i + (lane >> 3): see
    // store_block_chunks.
    const unsigned long long mine = ok ? reinterpret_cast<unsigned long long>(src) : 0ull;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4* ps = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, mine, 4 * i + (lane >> 3)));
      const float4 f = ps ? __ldg(ps + (lane & 7)) : make_float4(0.f, 0.f, 0.f, 0.f);
      val[4 * i] = f.x; val[4 * i + 1] = f.y; val[4 * i + 2] = f.z; val[4 * i + 3] = f.w;
    }
    return true;
  } else if (chans == 32) {
    // lane = pixel, one coalesced load per channel; 32-bit element offsets (the host checks that the
    // tensor is addressable with them) keep this at two instructions per value
    const int s1 = (int)v.s1;
    const float* pa = src + 4 * sw * s1;  // for j with bit 2 clear
    const float* pb = src - 4 * sw * s1;  // for j with bit 2 set
    if (__all_sync(0xffffffffu, ok)) {  // the common case away from padding: no predication
#pragma unroll
      for (int j = 0; j < 32; ++j) val[j] = __ldg(((j & 4) ? pb : pa) + j * s1);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) val[j] = ok ? __ldg(((j & 4) ? pb : pa) + j * s1) : 0.f;
    }
  } else {
    const int s1 = (int)v.s1;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      const int c = j ^ (sw << 2);
      val[j] = (ok && c < chans) ? __ldg(src + c * s1) : 0.f;
    }
  }
  return false;
}
// Where one staged block lives: the TF32 hi plane (128-byte rows) and either the FP32 lo plane or,
// with BF16 cross terms, the two bf16 planes (64-byte rows) of bf16(hi) and bf16(lo).
struct BlockPlanes {
  uint32_t hi, lo, h16, l16;
};
// Store for the channels-last load pattern: eight lanes write the eight 16-byte chunks of one row
// (a whole row per quarter warp: conflict-free in any swizzle).
template <bool DW_CROSS>
__device__ __forceinline__ void store_block_chunks(const float (&val)[32], int rows, int row0, const BlockPlanes& pl, int lane) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = 4 * i + (lane >> 3);
    if (r < rows) {
      float h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split_tf32_fast(val[4 * i + j], h[j], l[j]);
      const int c4 = (lane & 7) * 4;
      sts_f32x4(pl.hi + sw32b_offset(row0 + r, c4), h[0], h[1], h[2], h[3]);
      if (DW_CROSS) {
        const uint32_t o = sw64_offset(row0 + r, c4);
        sts_b32x2(pl.h16 + o, pack_bf16x2(h[0], h[1]), pack_bf16x2(h[2], h[3]));
        sts_b32x2(pl.l16 + o, pack_bf16x2(l[0], l[1]), pack_bf16x2(l[2], l[3]));
      } else {
        sts_f32x4(pl.lo + sw32b_offset(row0 + r, c4), l[0], l[1], l[2], l[3]);
      }
    }
  }
}
// Store for the lane = row pattern; val[j] holds channel j ^ 4 in lanes 4-7 of every eight (see stage_block).
template <bool DW_CROSS>
__device__ __forceinline__ void store_block(const float (&val)[32], int rows, int row0, const BlockPlanes& pl, int lane, int chans = 32) {
  if (lane >= rows) return;
  const uint32_t sw = (uint32_t)((lane >> 2) & 1);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    if (8 * m >= chans) break;   // nothing reads what lies in these columns
    float h0[4], l0[4], h1[4], l1[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      split_tf32_fast(val[m * 8 + j], h0[j], l0[j]);
      split_tf32_fast(val[m * 8 + 4 + j], h1[j], l1[j]);
    }
    const uint32_t oa = sw32b_offset(row0 + lane, m * 8) ^ (sw << 4), ob = oa ^ 16u;
    sts_f32x4(pl.hi + oa, h0[0], h0[1], h0[2], h0[3]);
    sts_f32x4(pl.hi + ob, h1[0], h1[1], h1[2], h1[3]);
    if (DW_CROSS) {
      // the eight channels of this group are one 16-byte chunk of a bf16 row; its two 8-byte halves
      // go where this lane's channel order puts them (64-byte rows need no bank-conflict swap)
      const uint32_t qa = sw64_offset(row0 + lane, m * 8) ^ (sw << 3), qb = qa ^ 8u;
      sts_b32x2(pl.h16 + qa, pack_bf16x2(h0[0], h0[1]), pack_bf16x2(h0[2], h0[3]));
      sts_b32x2(pl.h16 + qb, pack_bf16x2(h1[0], h1[1]), pack_bf16x2(h1[2], h1[3]));
      sts_b32x2(pl.l16 + qa, pack_bf16x2(l0[0], l0[1]), pack_bf16x2(l0[2], l0[3]));
      sts_b32x2(pl.l16 + qb, pack_bf16x2(l1[0], l1[1]), pack_bf16x2(l1[2], l1[3]));
    } else {
      sts_f32x4(pl.lo + oa, l0[0], l0[1], l0[2], l0[3]);
      sts_f32x4(pl.lo + ob, l1[0], l1[1], l1[2], l1[3]);
    }
  }
}

}  // namespace tcdw
}  // namespace b200

// GEMM on tcgen05 with the left operand in tensor memory: C[g] = alpha * A[g] * B[g] + beta * bias, FP32 by split precision (tc_common.cuh).
//
// In the strip kernel (conv_tc_strip.cu) a staged strip of A feeds one tap when it runs as a GEMM, and shared memory sets the pace: a
// 128x256x32 step reads 96 KB of operands, takes in 64 KB of B and 32 KB of A, 1600 clocks at 128 bytes each, for 1024 clocks of
// products.  Here the producers convert their rows in registers and store them to tensor memory, which leaves 64 KB of B read and
// 64 KB written, and 16 KB of raw A in and out: asynchronous copies keep three jobs of a warp on their way (loads into registers
// one job ahead: 148 us; transposing in registers instead of through those lines: 162).  16384x1024 x 1024x1024: 144 us in the strip kernel,
// 131 here; without loads, 113.
//
// CTA roles (576 threads, persistent over tiles of 128 x BN): warps 0-7 epilogue, warps 8-15 producers (two sets of four; a warp
// serves the 32 rows of its quarter of the tensor memory), warp 16 one thread streaming the images of B
// that stage_weights_kernel wrote, warp 17 tensor-memory allocation and MMA issue.
// Tensor memory: columns 0-255 the accumulators (one of 256 columns, two of 128 or four of 64), 256-511 four stages of A: 32 columns of
// TF32 values, 16 of BF16 pairs of the high parts, 16 of the low parts.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "gemm_tmem.cuh"
#include "tc_common.cuh"

namespace b200 {
namespace gt {
using namespace tc;

constexpr int M_TILE = 128, KBLK = 32;
constexpr int EPI_WARPS = 8, SETS = 2, W_WARP = EPI_WARPS + 4 * SETS, MMA_WARP = W_WARP + 1, THREADS = (MMA_WARP + 1) * 32;
constexpr int DEPTH = 3;             // jobs of a producer warp on their way
constexpr uint32_t SLOT = 4096;      // one of them: 32 lines of 128 bytes
constexpr int A_STAGES = 4, MAX_W_STAGES = 8, MAX_ACC = 4;
template <int BN> constexpr int W_RING = BN == 256 ? 2 : 4;

struct Ctrl {
  unsigned long long a_full[A_STAGES], a_empty[A_STAGES], w_full[MAX_W_STAGES], w_empty[MAX_W_STAGES], acc_full[MAX_ACC], acc_empty[MAX_ACC];
  uint32_t tmem_base;
  int abort_flag;
};
struct Tile { int m, n, group; };
__device__ __forceinline__ Tile tile_of(const GemmArgs& a, int t) {
  Tile c;
  if (a.m_fastest) {
    const int rest = (int)a.div_m.div((uint32_t)t);
    c.m = t - rest * a.tiles_m;
    c.group = (int)a.div_n.div((uint32_t)rest);
    c.n = rest - c.group * a.tiles_n;
  } else {
    const int rest = (int)a.div_n.div((uint32_t)t);
    c.n = t - rest * a.tiles_n;
    c.group = (int)a.div_m.div((uint32_t)rest);
    c.m = rest - c.group * a.tiles_m;
  }
  return c;
}

// 8x8 transposition of 16-byte pieces between lanes l, l+4, ..., l+28: piece j of lane (i, q) becomes piece i of lane (j, q)
__device__ __forceinline__ void transpose_pieces(float (&v)[32], int lane) {
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
}

template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, int bytes) {   // the rest of BYTES becomes zero
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float lds_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void lds_f32x4(uint32_t addr, float& a, float& b, float& c, float& d) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "r"(addr) : "memory");
}

// PLANES: 1x1 convolutions of NCHW planes (a line of A is 32 pixels of a channel, a tile 128 pixels of an image) whose filter fits shared
// memory: it is fetched once and stays.  Such a layer is bound by HBM, so what counts is the bytes on their way: 96 KB of asynchronous copies a
// CTA against the 48 KB that the strip kernel's twelve producer warps hold in registers, and no filter traffic beside them.  64 images of 56x56:
// 256 -> 64 channels 71 us in the strip kernel, 57 here (4.5 TB/s), 64 -> 256 61 and 51.
template <int BN, bool PLANES>
__global__ void __launch_bounds__(THREADS, 1) gemm_tmem_kernel(const GemmArgs a) {
  constexpr int NACC = 256 / BN;
  static_assert(NACC <= MAX_ACC, "a barrier pair for every accumulator");
  const int W_STAGES = PLANES ? a.kblocks : W_RING<BN>;
  constexpr uint32_t W_BYTES = BN * 256u;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), w_base = (raw + 1023u) & ~1023u;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (w_base - raw) + W_STAGES * W_BYTES + 4 * SETS * DEPTH * SLOT);
  volatile int* abort_flag = &ctrl->abort_flag;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < A_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->a_full[s]), 4);
      mbar_init(smem_u32(&ctrl->a_empty[s]), 1);
    }
    for (int s = 0; s < W_STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->w_full[s]), 1);
      mbar_init(smem_u32(&ctrl->w_empty[s]), 1);
    }
    for (int s = 0; s < NACC; ++s) {
      mbar_init(smem_u32(&ctrl->acc_full[s]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[s]), EPI_WARPS);
    }
    ctrl->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&ctrl->tmem_base);
  const int my_tiles = a.tiles > (int)blockIdx.x ? (a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;

  if (warp == MMA_WARP) {
    const bool leader = elect_one();
    constexpr uint32_t id32 = make_idesc_tf32(M_TILE, BN), id16 = make_idesc_bf16(M_TILE, BN);
    const uint64_t b_base = make_kmajor_sw128_desc(w_base);
    uint32_t as = 0, a_par = 0, ws = 0, w_par = 0;
    bool alive = true;
    for (int i = 0; i < my_tiles && alive; ++i) {
      const uint32_t ab = (uint32_t)i % NACC, round = (uint32_t)i / NACC;
      if (!warp_wait(smem_u32(&ctrl->acc_empty[ab]), (round & 1u) ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
      const uint32_t d = tmem + ab * BN;
      for (int kb = 0; kb < a.kblocks; ++kb) {
        if (!warp_wait(smem_u32(&ctrl->w_full[ws]), w_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        if (!warp_wait(smem_u32(&ctrl->a_full[as]), a_par, abort_flag, a.status, STATUS_TIMEOUT_FULL)) { alive = false; break; }
        tc_fence_after();
        if (leader) {
          const uint32_t ta = tmem + 256u + as * 64u;
          const uint64_t bh = b_base + ws * (W_BYTES >> 4), bc = bh + (BN * 128u >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_tf32_ts(d, ta + 8 * k, bh + 2 * k, id32, (uint32_t)((kb | k) != 0));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16_ts(d, ta + 32 + 8 * k, bc + 2 * k, id16, 1);
          umma_commit(smem_u32(&ctrl->a_empty[as]));
          if (!PLANES) umma_commit(smem_u32(&ctrl->w_empty[ws]));
        }
        if (++as == A_STAGES) { as = 0; a_par ^= 1u; }
        if (++ws == (uint32_t)W_STAGES) { ws = 0; w_par ^= PLANES ? 0u : 1u; }
      }
      if (alive && leader) umma_commit(smem_u32(&ctrl->acc_full[ab]));
    }
  } else if (warp == W_WARP) {
    if (lane == 0) {
      if (a.wait_for_images) asm volatile("griddepcontrol.wait;" ::: "memory");  // only this thread reads what the kernel ahead writes
      uint32_t ws = 0, par = 1, issued = 0;
      bool alive = true;
      for (int i = 0; i < (PLANES ? min(my_tiles, 1) : my_tiles) && alive; ++i) {
        const Tile t = tile_of(a, (int)blockIdx.x + i * (int)gridDim.x);
        const unsigned char* img = reinterpret_cast<const unsigned char*>(a.images) + ((long long)(PLANES ? 0 : t.group) * a.tiles_n + t.n) * a.kblocks * (long long)W_BYTES;
        for (int kb = 0; kb < a.kblocks; ++kb, img += W_BYTES) {
          if (!mbar_wait(smem_u32(&ctrl->w_empty[ws]), par, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) { alive = false; break; }
          mbar_expect_tx(smem_u32(&ctrl->w_full[ws]), W_BYTES);
          bulk_g2s(w_base + ws * W_BYTES, img, W_BYTES, smem_u32(&ctrl->w_full[ws]));
          ++issued;
          if (++ws == (uint32_t)W_STAGES) { ws = 0; par ^= 1u; }
        }
      }
      // after an abort nobody consumes the stages: wait (bounded) for the copies still in flight
      if (!alive)
        for (uint32_t j = issued > (uint32_t)W_STAGES ? issued - W_STAGES : 0; j < issued; ++j)
          mbar_wait(smem_u32(&ctrl->w_full[j % W_STAGES]), (j / W_STAGES) & 1u, nullptr, a.status, STATUS_TIMEOUT_FULL);
    }
  } else if (warp >= EPI_WARPS) {
    // ------------------------------ producers ------------------------------
    const int quarter = warp & 3, set = (warp - EPI_WARPS) >> 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16, slots = w_base + (uint32_t)W_STAGES * W_BYTES + (uint32_t)(warp - EPI_WARPS) * (DEPTH * SLOT);
    const int total = my_tiles * a.kblocks;       // below 2^31 (checked by the host)
    struct Block { const float* src; int rows, valid; };        // rows of this warp inside the matrix, values of this K block
    auto locate = [&](int c) -> Block {
      const int it = (int)a.div_kblocks.div((uint32_t)c), kb = c - it * a.kblocks;
      const Tile t = tile_of(a, (int)blockIdx.x + it * (int)gridDim.x);
      const int row0 = t.m * M_TILE + quarter * 32, k0 = kb * KBLK;
      return Block{a.A + t.group * a.a_group + (long long)k0 * a.a_k + (long long)row0 * a.a_m, a.M - row0,
                   min(KBLK, (PLANES ? a.kc : min(a.kc, a.k_total - t.group * a.kc)) - k0)};
    };
    // the 32 x 32 values of a job as 32 lines of 128 bytes, eight lanes to a line; what lies outside is zero
    auto issue = [&](int n) {
      const int c = set + n * SETS;
      if (c < total) {
        const Block k = locate(c);
        const int lines = a.along_k ? k.rows : k.valid, length = a.along_k ? k.valid : k.rows;
        const long long pitch = a.along_k ? a.a_m : a.a_k;
        const uint32_t slot = slots + (uint32_t)(n % DEPTH) * SLOT;
        if (a.pieces16) {
          const int bytes = max(0, min(16, (length - (lane & 7) * 4) * 4));
          const float* p = k.src + (long long)(lane >> 3) * pitch + (lane & 7) * 4;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int r = 4 * j + (lane >> 3), size = r < lines ? bytes : 0;
            cp_async<16>(slot + (uint32_t)(r * 128 + (((lane & 7) ^ (r & 7)) << 4)), size ? p + 4ll * j * pitch : a.A, size);
          }
        } else {                     // lines along k that start anywhere: a value at a time, a warp to a line
          const float* p = k.src + lane;
#pragma unroll 8
          for (int r = 0; r < 32; ++r) {
            const int size = r < k.rows && lane < k.valid ? 4 : 0;
            cp_async<4>(slot + (uint32_t)(r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4), size ? p + r * a.a_m : a.A, size);
          }
        }
      }
      cp_async_commit();
    };
    if (set < total) {
      for (int n = 0; n < DEPTH; ++n) issue(n);
#pragma unroll 1
      for (int n = 0, c = set; c < total; ++n, c += SETS) {
        float v[32];
        cp_async_wait<DEPTH - 1>();
        __syncwarp();
        const uint32_t slot = slots + (uint32_t)(n % DEPTH) * SLOT;
        if (a.along_k) {             // lines are rows: 16 bytes at a time of this lane's line
#pragma unroll
          for (int j = 0; j < 8; ++j) lds_f32x4(slot + (uint32_t)(lane * 128 + ((j ^ (lane & 7)) << 4)), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {                     // lines are values of the reduction: this lane's row out of each
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = lds_f32(slot + (uint32_t)(j * 128 + (((lane >> 2) ^ (j & 7)) << 4) + (lane & 3) * 4));
        }
        __syncwarp();
        issue(n + DEPTH);
        const uint32_t as = (uint32_t)c % A_STAGES, round = (uint32_t)c / A_STAGES;
        if (!warp_wait(smem_u32(&ctrl->a_empty[as]), (round & 1u) ^ 1u, abort_flag, a.status, STATUS_TIMEOUT_EMPTY)) break;
        tc_fence_after();
        const uint32_t ta = tmem + 256u + as * 64u + lane_base;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t x[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float hi, lo;
            split_tf32_fast(v[16 * h + j], hi, lo);
            x[j] = __float_as_uint(hi);
          }
          tmem_st16(ta + 16 * h, x);
        }
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t x[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            float h0, l0, h1, l1;
            split_tf32_fast(v[2 * j], h0, l0);
            split_tf32_fast(v[2 * j + 1], h1, l1);
            x[j] = part ? pack_bf16x2(l0, l1) : pack_bf16x2(h0, h1);
          }
          tmem_st16(ta + 32 + 16 * part, x);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->a_full[as]));
      }
      cp_async_wait<0>();            // also after a wait that gave up: nothing may land in shared memory once the CTA has gone
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    // two warps to a quarter of the rows, every other 32 columns each
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    for (int i = 0; i < my_tiles; ++i) {
      const Tile t = tile_of(a, (int)blockIdx.x + i * (int)gridDim.x);
      const uint32_t ab = (uint32_t)i % NACC, round = (uint32_t)i / NACC;
      const int row = t.m * M_TILE + quarter * 32 + lane, n0 = t.n * BN, cols = min(BN, a.N - n0);
      float* out = a.C + t.group * a.c_group + (long long)row * a.c_pitch + n0;
      if (!warp_wait(smem_u32(&ctrl->acc_full[ab]), round & 1u, abort_flag, a.status, STATUS_TIMEOUT_ACCUM)) break;
      tc_fence_after();
      if (half * 32 >= cols) {      // nothing of a narrow last tile for this warp
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->acc_empty[ab]));
      }
      for (int c0 = half * 32; c0 < cols; c0 += 64) {
        float v[32];
        tmem_ld32(tmem + ab * BN + (uint32_t)c0 + lane_base, v);
        if (c0 + 64 >= cols) {      // this warp's last read of the accumulator: hand it back
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctrl->acc_empty[ab]));
        }
        const int left = min(32, cols - c0);
        if (a.bias) {
          const float b = lane < left ? a.beta * __ldg(a.bias + ((PLANES ? 0 : (long long)t.group * a.N) + n0 + c0 + lane) * a.bias_stride) : 0.f;
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = fmaf(a.alpha, v[j], __shfl_sync(0xffffffffu, b, j));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= a.alpha;
        }
        if (PLANES) {                 // lane = pixel: 32 pixels of a channel to a store
          float* p = a.C + t.group * a.c_group + (long long)(n0 + c0) * a.c_pitch + row;
          if (row < a.M) {
#pragma unroll
            for (int j = 0; j < 32; ++j, p += a.c_pitch)
              if (j < left) *p = v[j];
          }
        } else if (left == 32) {
          transpose_pieces(v, lane);  // whole lines: piece i of row 4j + lane % 4
          float* p = a.C + t.group * a.c_group + (long long)(t.m * M_TILE + quarter * 32 + (lane & 3)) * a.c_pitch + n0 + c0 + (lane >> 2) * 4;
          if (a.vec_out) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (t.m * M_TILE + quarter * 32 + 4 * j + (lane & 3) < a.M)
                *reinterpret_cast<float4*>(p + 4ll * j * a.c_pitch) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          } else {                    // rows of C that are not 16-byte aligned (a row to a lane: 151 us for 16000x77 x 77x1111, now 71)
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (t.m * M_TILE + quarter * 32 + (j & ~3) + (lane & 3) < a.M) p[(long long)(j & ~3) * a.c_pitch + (j & 3)] = v[j];
          }
        } else if (row < a.M) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < left) out[c0 + j] = v[j];
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

template <int BN, bool PLANES>
static int launch(const GemmArgs& a, cudaStream_t st) {
  static std::once_flag once;
  static cudaError_t opt_in = cudaSuccess;
  std::call_once(once, [] { opt_in = cudaFuncSetAttribute(gemm_tmem_kernel<BN, PLANES>, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
  B200_CUDA(opt_in);
  const size_t smem = (size_t)(PLANES ? a.kblocks : W_RING<BN>) * BN * 256 + 4 * SETS * DEPTH * SLOT + 1024 + sizeof(Ctrl) + 64;
  const dim3 grid((unsigned)std::min(a.tiles, sm_count()));
  if (a.wait_for_images) launch_next(gemm_tmem_kernel<BN, PLANES>, grid, THREADS, smem, st, a);
  else gemm_tmem_kernel<BN, PLANES><<<grid, THREADS, smem, st>>>(a);
  count_launch();
  return launch_check("gemm_tmem_kernel");
}

int run(GemmArgs a, int bn, cudaStream_t st) {
  a.status = device_status_word();
  if (!a.status) return fail(B200_ECUDA, "device status word is not allocated");
  a.div_m = FastDiv((uint32_t)a.tiles_m); a.div_n = FastDiv((uint32_t)a.tiles_n); a.div_kblocks = FastDiv((uint32_t)a.kblocks);
  if (a.planes) return bn == 256 ? launch<256, true>(a, st) : bn == 128 ? launch<128, true>(a, st) : launch<64, true>(a, st);
  return bn == 256 ? launch<256, false>(a, st) : launch<128, false>(a, st);
}

}  // namespace gt
}  // namespace b200

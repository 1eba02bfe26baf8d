// Bandwidth-bound FP32 sums in one launch: per-channel sums of a 4-D view (dBias) and column sums of a matrix (the bias
// gradient of a linear layer, reached through b200_sum_strided).
//
// A sum of a few channels has too few results to fill the machine with one CTA per result, and a second launch that adds
// slab partials costs as much as the sum itself (64x64x56x56 channels-last: 8.1 us for the sum, 12 us for the pass
// behind it).  Here the slabs of a result are the CTAs of one thread-block cluster: each CTA hands its partial to rank 0
// through distributed shared memory, and rank 0 adds them in rank order (no atomics, no scratch, the same result from
// run to run).  Every thread keeps eight independent loads in flight.
//
// Replaces csrc/shaders/conv2d_backward_bias_reduce.comp:9-24 of the reference.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace b200 {
namespace red {

constexpr int THREADS = 256, COL_THREADS = 512, UNROLL = 8, MAX_CLUSTER = 16;

struct Rows {            // how row / pixel index i maps to memory: i = (b, y, x) when `dense` is 0
  long long s0, s2, s3;  // dense: pixel i of image b sits at b * s0 + (i - b * img) * s3
  FastDiv img_div, row_div;
  int img, row;
};
template <bool DENSE>
__device__ __forceinline__ long long offset_of(const Rows& r, uint32_t i) {
  const uint32_t b = r.img_div.div(i), rem = i - b * (uint32_t)r.img;
  if (DENSE) return (long long)b * r.s0 + (long long)rem * r.s3;
  const uint32_t y = r.row_div.div(rem), x = rem - y * (uint32_t)r.row;
  return (long long)b * r.s0 + (long long)y * r.s2 + (long long)x * r.s3;
}

__device__ __forceinline__ float add4(const float4& v) { return (v.x + v.y) + (v.z + v.w); }

// out[c] = sum over images and pixels of channel c.  blockIdx.x = channel, the cluster's ranks share its `count` units
// (a unit is four adjacent pixels of a dense plane when VEC, else one pixel).
template <bool VEC, bool DENSE>
__global__ void __launch_bounds__(THREADS) reduce_planes_kernel(const float* __restrict__ src, long long chan_stride, Rows rows, uint32_t count,
                                                                float* __restrict__ out, int accumulate) {
  cluster_announce();
  wait_previous();
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t ranks = cluster.num_blocks(), rank = cluster.block_rank();
  const float* base = src + (long long)blockIdx.x * chan_stride;
  const uint32_t step = ranks * THREADS;
  float sum = 0.f;
  uint32_t i = rank * THREADS + threadIdx.x;
  auto load = [&](uint32_t u) -> float {
    if (VEC) return add4(__ldg(reinterpret_cast<const float4*>(base + offset_of<true>(rows, u))));
    return __ldg(base + offset_of<DENSE>(rows, u));
  };
  for (; (unsigned long long)i + (UNROLL - 1ull) * step < count; i += UNROLL * step) {
    float v[UNROLL];
#pragma unroll
    for (int k = 0; k < UNROLL; ++k) v[k] = load(i + k * step);
    sum += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  for (; i < count; i += step) sum += load(i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  __shared__ float warp_part[THREADS / 32];
  __shared__ float slab_part[MAX_CLUSTER];
  if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = sum;
  __syncthreads();
  cluster_wait_started();
  if (threadIdx.x == 0) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) v += warp_part[w];
    *cluster.map_shared_rank(&slab_part[rank], 0) = v;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    float v = accumulate ? out[blockIdx.x] : 0.f;
    for (uint32_t r = 0; r < ranks; ++r) v += slab_part[r];
    out[blockIdx.x] = v;
  }
}

// out[c] = sum over rows of column c, columns adjacent in memory.  A CTA owns 4 * LPR columns (LPR lanes of 16 bytes per
// row); blockIdx.x = column block, the cluster's ranks share the rows; with gridDim.z > 1 clusters share them and write one
// partial row each.
template <int LPR, bool VEC, bool DENSE>
__global__ void __launch_bounds__(COL_THREADS) reduce_columns_kernel(const float* __restrict__ src, Rows rows, uint32_t count, int cols,
                                                                 float* __restrict__ out, int accumulate) {
  cluster_announce();
  wait_previous();
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cluster_ranks = cluster.num_blocks(), cluster_rank = cluster.block_rank();
  const uint32_t ranks = cluster_ranks * gridDim.z, rank = blockIdx.z * cluster_ranks + cluster_rank;   // shares of the rows
  constexpr uint32_t ROWS = COL_THREADS / LPR;        // rows per CTA pass
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = (int)blockIdx.x * 4 * LPR + (threadIdx.x % LPR) * 4;
  const float* base = src + c0;
  const uint32_t step = ranks * ROWS;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load = [&](uint32_t r) -> float4 {
    const float* p = base + offset_of<DENSE>(rows, r);
    if (VEC) return __ldg(reinterpret_cast<const float4*>(p));
    return make_float4(c0 < cols ? __ldg(p) : 0.f, c0 + 1 < cols ? __ldg(p + 1) : 0.f, c0 + 2 < cols ? __ldg(p + 2) : 0.f,
                       c0 + 3 < cols ? __ldg(p + 3) : 0.f);
  };
  if (!VEC || c0 < cols) {
    uint32_t r = rank * ROWS + threadIdx.x / LPR;
    for (; (unsigned long long)r + (UNROLL - 1ull) * step < count; r += UNROLL * step) {
      float4 v[UNROLL];
#pragma unroll
      for (int k = 0; k < UNROLL; ++k) v[k] = load(r + k * step);
#pragma unroll
      for (int k = 0; k < UNROLL; k += 4) {
        sum.x += (v[k].x + v[k + 1].x) + (v[k + 2].x + v[k + 3].x); sum.y += (v[k].y + v[k + 1].y) + (v[k + 2].y + v[k + 3].y);
        sum.z += (v[k].z + v[k + 1].z) + (v[k + 2].z + v[k + 3].z); sum.w += (v[k].w + v[k + 1].w) + (v[k + 2].w + v[k + 3].w);
      }
    }
    for (; r < count; r += step) {
      const float4 v = load(r);
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
  }
#pragma unroll
  for (int o = 16; o >= LPR; o >>= 1) {           // the lanes of a warp that hold the same columns
    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o); sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
    sum.z += __shfl_xor_sync(0xffffffffu, sum.z, o); sum.w += __shfl_xor_sync(0xffffffffu, sum.w, o);
  }
  __shared__ float4 warp_part[COL_THREADS / 32][LPR];
  __shared__ float slab_part[MAX_CLUSTER][4 * LPR];
  if (lane < LPR) warp_part[warp][lane] = sum;
  __syncthreads();
  cluster_wait_started();
  if (threadIdx.x < 4 * LPR) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < COL_THREADS / 32; ++w) v += reinterpret_cast<const float*>(&warp_part[w][0])[threadIdx.x];
    *cluster.map_shared_rank(&slab_part[cluster_rank][threadIdx.x], 0) = v;
  }
  cluster.sync();
  const int c = (int)blockIdx.x * 4 * LPR + (int)threadIdx.x;
  if (cluster_rank == 0 && threadIdx.x < 4 * LPR && c < cols) {
    float v = accumulate ? out[c] : 0.f;
    for (uint32_t r = 0; r < cluster_ranks; ++r) v += slab_part[r][threadIdx.x];
    out[(long long)blockIdx.z * cols + c] = v;
  }
}

template <int KERNEL_THREADS, typename... P, typename... A>
static int launch_cluster(void (*kernel)(P...), unsigned blocks, int ranks, int slabs, cudaStream_t st, A... args) {
  if (ranks > 8) B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks, (unsigned)ranks, (unsigned)slabs); cfg.blockDim = dim3(KERNEL_THREADS); cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = (unsigned)ranks; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_next()
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  count_launch();
  return launch_check("reduce kernel");
}

// Ranks of a cluster: enough that a thread has about one batch of eight loads, and no more CTAs than fit the machine
// twice over (a channel count in the thousands needs no help).
static int ranks_for(long long units_per_result, long long units_per_pass, long long results, int most) {
  int ranks = 1;
  while (ranks < most && units_per_result > ranks * units_per_pass * UNROLL && results * ranks < 4ll * sm_count()) ranks *= 2;
  return ranks;
}

}  // namespace red

// Bytes of partial sums that reduce_channels can use for a channels-last view (few channels and many pixels: sixteen CTAs per
// column block do not fill the machine, and a second small launch is then the cheaper way to add the clusters' sums).
constexpr int MAX_SLABS = 8;
constexpr long long SLAB_MIN_VALUES = 4ll << 20;   // below 16 MB one cluster per column block is as fast as two launches
size_t reduce_channels_workspace(long long n, int channels, int h, int w) {
  return (long long)n * h * w * channels >= SLAB_MIN_VALUES && div_up64(channels, 16) * red::MAX_CLUSTER < 2ll * sm_count()
             ? (size_t)MAX_SLABS * channels * sizeof(float) : 0;
}

// Sums a [n][channels][h][w] view over everything but the channel.
int reduce_channels(View4 v, long long n, int channels, int h, int w, float* out, float* partial, size_t partial_bytes, cudaStream_t st) {
  using namespace red;
  const long long plane = (long long)h * w;
  const long long images_per_call = std::max<long long>(1, (1ll << 30) / plane);
  if (plane >= 1ll << 31) return fail(B200_ERANGE, "channel sum: plane too large");
  const bool columns = v.s1 == 1 && v.s3 != 1;
  for (long long b0 = 0; b0 < n; b0 += images_per_call) {  // pixel indices are 32-bit inside a launch
    const long long images = std::min(images_per_call, n - b0);
    const float* src = v.ptr + b0 * v.s0;
    const int acc = b0 > 0;
    Rows r{};
    r.s0 = v.s0; r.s2 = v.s2; r.s3 = v.s3;
    r.img = (int)plane; r.row = w;
    r.img_div = FastDiv((uint32_t)plane); r.row_div = FastDiv((uint32_t)w);
    const uint32_t count = (uint32_t)(images * plane);
    const bool aligned = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    const bool dense = h == 1 || v.s2 == (long long)w * v.s3;
    int rc;
    if (columns) {
      const bool vec = aligned && channels % 4 == 0 && v.s0 % 4 == 0 && v.s2 % 4 == 0 && v.s3 % 4 == 0;
      // 128 bytes of a row per CTA where the column blocks (times sixteen ranks) fill the machine, else 64 bytes
      const bool wide = div_up64(channels, 32) * MAX_CLUSTER >= sm_count();
      const int lpr = wide ? 8 : 4;
      const unsigned blocks = (unsigned)div_up64(channels, 4 * lpr);
      const int ranks = ranks_for(count, COL_THREADS / lpr, blocks, MAX_CLUSTER);
      int slabs = 1;
      if (partial && n <= images_per_call && reduce_channels_workspace(n, channels, h, w) > 0)
        while (slabs < MAX_SLABS && blocks * (unsigned)(ranks * slabs) < 2u * (unsigned)sm_count() && 2 * slabs * sizeof(float) * channels <= partial_bytes) slabs *= 2;
      float* dst = slabs > 1 ? partial : out;
      auto go = [&](auto kernel) { return launch_cluster<COL_THREADS>(kernel, blocks, ranks, slabs, st, src, r, count, channels, dst, acc); };
      rc = wide ? (vec ? (dense ? go(reduce_columns_kernel<8, true, true>) : go(reduce_columns_kernel<8, true, false>))
                       : (dense ? go(reduce_columns_kernel<8, false, true>) : go(reduce_columns_kernel<8, false, false>)))
                : (vec ? (dense ? go(reduce_columns_kernel<4, true, true>) : go(reduce_columns_kernel<4, true, false>))
                       : (dense ? go(reduce_columns_kernel<4, false, true>) : go(reduce_columns_kernel<4, false, false>)));
      if (!rc && slabs > 1) rc = finalize_splits(partial, out, channels, slabs, st);
    } else {
      const bool vec = dense && v.s3 == 1 && aligned && plane % 4 == 0 && v.s0 % 4 == 0 && v.s1 % 4 == 0;
      uint32_t units = count;
      if (vec) {
        r.img = (int)(plane / 4); r.img_div = FastDiv((uint32_t)(plane / 4)); r.s3 = 4;
        units = count / 4;
      }
      const int ranks = ranks_for(units, THREADS, channels, 8);
      auto go = [&](auto kernel) { return launch_cluster<THREADS>(kernel, (unsigned)channels, ranks, 1, st, src, v.s1, r, units, out, acc); };
      rc = vec ? go(reduce_planes_kernel<true, true>) : dense ? go(reduce_planes_kernel<false, true>) : go(reduce_planes_kernel<false, false>);
    }
    if (rc) return rc;
  }
  return B200_OK;
}

}  // namespace b200

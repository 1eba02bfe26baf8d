// Normalisation rows held in registers: what batch_norm.cu (a row = the planes of one channel) and group_norm.cu (a row = the
// planes of one sample and group) share.
//
// A row that is read for its sums and again for its result costs a second trip to L2 or HBM and, with one CTA a row, leaves the
// machine to a few hundred long chains.  Here the CTAs of a thread-block cluster share a row: every thread loads its units (16 bytes,
// or one value where planes are not whole 16-byte pieces) at once, keeps them in registers, the CTAs exchange one partial
// sum each through distributed shared memory, and the result is computed from the registers.  One trip to memory, one exchange.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "norm_plan.cuh"

namespace b200 {
namespace nres {
namespace cg = cooperative_groups;

constexpr int THREADS = PLAN_THREADS, WARPS = THREADS / 32, MAX_RANKS = PLAN_MAX_RANKS;

struct Rows {
  uint32_t units, per;        // units of a row; of one rank
  uint32_t plane_units;
  FastDiv plane_div;          // by plane_units
  long long plane_stride;     // floats
};

template <int VEC>
struct Unit {
  float v[VEC];
  __device__ __forceinline__ void load(const float* p, bool inside) {
    if (VEC == 4) {
      const float4 f = inside ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[0] = f.x; v[1 % VEC] = f.y; v[2 % VEC] = f.z; v[3 % VEC] = f.w;
    } else {
      v[0] = inside ? __ldg(p) : 0.f;
    }
  }
  __device__ __forceinline__ void store(float* p) const {
    if (VEC == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1 % VEC], v[2 % VEC], v[3 % VEC]);
    else *p = v[0];
  }
};

// Units that wait in shared memory instead of registers, each thread's own: unit k of a thread is unit k * THREADS + its index of the CTA.
template <int VEC>
struct Staged {
  float* v;
  __device__ __forceinline__ void load(int k, const float* p, bool inside) const {   // asynchronous: arrive() before the first read
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(v + (k * THREADS + threadIdx.x) * VEC);
    if (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(p), "r"(inside ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(p), "r"(inside ? 4 : 0) : "memory");
  }
  static __device__ __forceinline__ void arrive() { asm volatile("cp.async.wait_all;" ::: "memory"); }
  __device__ __forceinline__ Unit<VEC> at(uint32_t i) const {        // unit i of the CTA
    Unit<VEC> u;
    if (VEC == 4) {
      const float4 f = *reinterpret_cast<const float4*>(v + i * VEC);
      u.v[0] = f.x; u.v[1 % VEC] = f.y; u.v[2 % VEC] = f.z; u.v[3 % VEC] = f.w;
    } else {
      u.v[0] = v[i];
    }
    return u;
  }
  __device__ __forceinline__ Unit<VEC> unit(int k) const { return at(k * THREADS + threadIdx.x); }
};

template <int VEC>
__device__ __forceinline__ long long unit_offset(const Rows& r, uint32_t u, uint32_t& plane) {
  plane = r.plane_div.div(u);
  return plane * r.plane_stride + (long long)((u - plane * r.plane_units) * VEC);
}

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of C values over the cluster, in every thread and in the same order everywhere: each warp leaves its sums with every rank, so
// that there is one barrier and no second level inside the CTA.  `table` is used once per kernel.  A kernel's first sum follows its
// cluster_announce() and a cluster_wait_started().
template <int C>
using Table = float[MAX_RANKS * WARPS][C];
template <int C>
__device__ __forceinline__ void cluster_sum(float (&v)[C], Table<C>& table, cg::cluster_group& cluster) {
  const int ranks = (int)cluster.num_blocks(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < C; ++c) v[c] = warp_total(v[c]);
  if (lane < ranks) {
    float* to = cluster.map_shared_rank(&table[cluster.block_rank() * WARPS + warp][0], lane);
#pragma unroll
    for (int c = 0; c < C; ++c) to[c] = v[c];
  }
  cluster.sync();
#pragma unroll
  for (int c = 0; c < C; ++c) v[c] = 0.f;
  for (int i = lane; i < ranks * WARPS; i += 32) {
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] += table[i][c];
  }
#pragma unroll
  for (int c = 0; c < C; ++c) v[c] = warp_total(v[c]);
}

// Mean relative to `origin` and sum of squared deviations of the row whose units from u0 this thread holds.  A warp takes the mean of its own
// values and then their deviations from it (they are in registers); count, mean and deviations of all warps are merged after ONE exchange, so
// that neither a common offset nor an outlier costs precision.  With the mean exchanged first and the deviations after it, 64x256x14x14
// took 7.65 us (batch norm forward) and 16x512x32x32 in 32 groups 16.7 (group norm forward); now 7.24 and 15.3.
template <int VEC, int UNROLL, typename F>     // unit(k) for k < n: the thread's units
__device__ __forceinline__ float2 row_moments(const F& unit, int n, uint32_t u0, uint32_t end, float origin, float count, Table<3>& table,
                                              cg::cluster_group& cluster) {
  const int ranks = (int)cluster.num_blocks(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t mine = 0;
#pragma unroll UNROLL
  for (int k = 0; k < n; ++k) {
    const bool inside = u0 + k * THREADS < end;
    mine += inside ? VEC : 0;
    const Unit<VEC> in = unit(k);
#pragma unroll
    for (int j = 0; j < VEC; ++j) s[(k * VEC + j) & 3] += inside ? in.v[j] - origin : 0.f;
  }
  const float held = (float)__reduce_add_sync(0xffffffffu, mine);     // values of this warp
  const float own = held > 0.f ? warp_total((s[0] + s[1]) + (s[2] + s[3])) / held : 0.f;
  s[0] = s[1] = s[2] = s[3] = 0.f;
#pragma unroll UNROLL
  for (int k = 0; k < n; ++k) {
    const Unit<VEC> in = unit(k);
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      const float d = u0 + k * THREADS < end ? (in.v[j] - origin) - own : 0.f;
      s[(k * VEC + j) & 3] = fmaf(d, d, s[(k * VEC + j) & 3]);
    }
  }
  const float own_m2 = warp_total((s[0] + s[1]) + (s[2] + s[3]));
  cluster_wait_started();
  if (lane < ranks) {
    float* to = cluster.map_shared_rank(&table[cluster.block_rank() * WARPS + warp][0], lane);
    to[0] = held; to[1] = own; to[2] = own_m2;
  }
  cluster.sync();
  float mean = 0.f, m2 = 0.f;
  for (int i = lane; i < ranks * WARPS; i += 32) mean = fmaf(table[i][0], table[i][1], mean);
  mean = warp_total(mean) / count;
  for (int i = lane; i < ranks * WARPS; i += 32) {
    const float d = table[i][1] - mean;
    m2 += fmaf(table[i][0] * d, d, table[i][2]);
  }
  return make_float2(mean, warp_total(m2));
}

inline Rows make_rows(int planes, int plane, int vec, long long plane_stride, int ranks) {
  Rows r{};
  r.plane_units = (uint32_t)(plane / vec);
  r.units = (uint32_t)planes * r.plane_units;
  r.per = (r.units + (uint32_t)ranks - 1) / (uint32_t)ranks;
  r.plane_div = FastDiv(r.plane_units);
  r.plane_stride = plane_stride;
  return r;
}

// grid (rows, ranks), clusters of `ranks` along y
template <typename... P, typename... A>
int launch(void (*kernel)(P...), unsigned rows, int ranks, size_t smem, cudaStream_t st, A... args) {
  if (smem) B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PLAN_STAGED_BYTES));
  if (ranks > 8) B200_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(rows, (unsigned)ranks); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = (unsigned)ranks; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_next()
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  B200_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  count_launch();
  return launch_check("normalisation kernel");
}

}  // namespace nres
}  // namespace b200

// Group-norm rows (the planes of one sample and group) in the shared memory of a cluster's CTAs, forward and backward.
#pragma once
#include "norm_resident.cuh"

namespace b200 {
namespace nres {

constexpr int STAGED_CHANNELS = 64;      // most channels of a group in the backward kernel
struct GroupShape {
  int groups, cpg, hw, c;                // cpg: channels of a group
  float count;                           // cpg * hw
};

// Rows beyond the registers of sixteen CTAs: the CTAs' shares are fetched into shared memory asynchronously and each tensor is read once.  The kernels
// with a CTA for a row read it again for each pass and leave the chip to as many CTAs as there are rows; the rule and what it measured stand at
// forward_staged() and backward_plan() in group_norm.cu.  Bound by latency with few rows, by memory beyond two waves.  `n`: units of a thread.
template <int VEC>
__global__ void __launch_bounds__(THREADS, 4) gn_forward_staged_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                                                                          const float* __restrict__ beta, GroupShape sh, Rows rows, int n, float eps,
                                                                          float* __restrict__ y, float* __restrict__ means, float* __restrict__ rstds) {
  cluster_announce();
  wait_previous();
  auto cluster = cg::this_cluster();
  extern __shared__ __align__(16) float staged[];
  __shared__ Table<3> table;
  const Staged<VEC> in{staged};
  const int row = blockIdx.x, rank = (int)cluster.block_rank();
  const int ch0 = row % sh.groups * sh.cpg;
  const uint32_t end = min(rows.units, (uint32_t)(rank + 1) * rows.per), u0 = (uint32_t)rank * rows.per + threadIdx.x;
  const size_t base = (size_t)row * sh.cpg * sh.hw;
  const float origin = __ldg(x + base);
#pragma unroll 8
  for (int k = 0; k < n; ++k) in.load(k, x + base + (size_t)min(u0 + k * THREADS, rows.units - 1) * VEC, u0 + k * THREADS < end);
  in.arrive();
  const float2 total = row_moments<VEC, 8>([&](int k) { return in.unit(k); }, n, u0, end, origin, sh.count, table, cluster);
  const float mean_rel = total.x, rstd = 1.f / sqrtf(total.y / sh.count + eps);
  if (rank == 0 && threadIdx.x == 0) {
    means[row] = origin + mean_rel;
    rstds[row] = rstd;
  }
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const uint32_t u = u0 + k * THREADS;
    if (u >= end) break;
    const int ch = ch0 + (int)rows.plane_div.div(u);
    const float scale = rstd * (gamma ? __ldg(gamma + ch) : 1.f), shift = beta ? __ldg(beta + ch) : 0.f;
    Unit<VEC> v = in.unit(k);
#pragma unroll
    for (int j = 0; j < VEC; ++j) v.v[j] = ((v.v[j] - origin) - mean_rel) * scale + shift;
    v.store(y + base + (size_t)u * VEC);
  }
}

// As gn_backward_cluster_kernel; with both tensors in shared memory a warp adds a plane's units themselves, and where a rank has fewer planes than
// warps each plane is cut into parts.
template <int VEC>
__global__ void __launch_bounds__(THREADS, 4) gn_backward_staged_kernel(const float* __restrict__ dy, const float* __restrict__ x,
                                                                           const float* __restrict__ means, const float* __restrict__ rstds,
                                                                           const float* __restrict__ gamma, GroupShape sh, Rows rows, int n,
                                                                           float* __restrict__ dx, float* __restrict__ plane_sums) {
  cluster_announce();
  wait_previous();
  auto cluster = cg::this_cluster();
  extern __shared__ __align__(16) float staged[];
  __shared__ float2 part[STAGED_CHANNELS];                           // of this rank: planes, or parts of them
  __shared__ float2 all_part[MAX_RANKS][STAGED_CHANNELS];      // rank 0: planes of every rank
  __shared__ float2 rank_part[MAX_RANKS];
  const Staged<VEC> xs{staged}, gs{staged + n * THREADS * VEC};
  const int row = blockIdx.x, ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ch0 = row % sh.groups * sh.cpg;
  const uint32_t begin = min(rows.units, (uint32_t)rank * rows.per), end = min(rows.units, (uint32_t)(rank + 1) * rows.per), u0 = begin + threadIdx.x;
  const size_t base = (size_t)row * sh.cpg * sh.hw;
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const size_t at = base + (size_t)min(u0 + k * THREADS, rows.units - 1) * VEC;
    xs.load(k, x + at, u0 + k * THREADS < end);
    gs.load(k, dy + at, u0 + k * THREADS < end);
  }
  const float mean = __ldg(means + row), rstd = __ldg(rstds + row);
  xs.arrive();
  __syncthreads();
  cluster_wait_started();
  const int p0 = (int)rows.plane_div.div(begin), planes = begin < end ? (int)rows.plane_div.div(end - 1) + 1 - p0 : 0;
  const int cut = planes && planes < WARPS ? WARPS / planes : 1;
  for (int i = warp; i < planes * cut; i += WARPS) {
    const uint32_t p = (uint32_t)(p0 + i / cut), a = max(begin, p * rows.plane_units) - begin, b = min(end, (p + 1) * rows.plane_units) - begin;
    const uint32_t share = (b - a + cut - 1) / cut, first = a + (uint32_t)(i % cut) * share, last = min(b, first + share);
    float s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
    auto add = [&](uint32_t u, int slot) {
      const Unit<VEC> xu = xs.at(u), gu = gs.at(u);
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        s1[(slot + j) & 3] += gu.v[j];
        s2[(slot + j) & 3] = fmaf(gu.v[j], (xu.v[j] - mean) * rstd, s2[(slot + j) & 3]);
      }
    };
    uint32_t u = first + lane;
    for (; u + 96 < last; u += 128) {
#pragma unroll
      for (int q = 0; q < 4; ++q) add(u + 32 * q, q);
    }
    for (; u < last; u += 32) add(u, 0);
    const float t1 = warp_total((s1[0] + s1[1]) + (s1[2] + s1[3])), t2 = warp_total((s2[0] + s2[1]) + (s2[2] + s2[3]));
    if (lane == 0) part[i] = make_float2(t1, t2);
  }
  __syncthreads();
  if (warp == 0) {
    float a = 0.f, b = 0.f;
    for (int i = lane; i < planes; i += 32) {
      float s1 = 0.f, s2 = 0.f;
      for (int q = 0; q < cut; ++q) s1 += part[i * cut + q].x, s2 += part[i * cut + q].y;
      if (plane_sums) *cluster.map_shared_rank(&all_part[rank][p0 + i], 0) = make_float2(s1, s2);
      const float w = gamma ? __ldg(gamma + ch0 + p0 + i) : 1.f;
      a = fmaf(w, s1, a);
      b = fmaf(w, s2, b);
    }
    a = warp_total(a);
    b = warp_total(b);
    if (lane < ranks) *cluster.map_shared_rank(&rank_part[rank], lane) = make_float2(a, b);
  }
  cluster.sync();
  asm volatile("griddepcontrol.launch_dependents;");
  if (plane_sums && rank == 0)
    for (int p = threadIdx.x; p < sh.cpg; p += THREADS) {
      const int r0 = (int)((uint32_t)p * rows.plane_units / rows.per), r1 = (int)(((uint32_t)(p + 1) * rows.plane_units - 1) / rows.per);
      float s1 = 0.f, s2 = 0.f;
      for (int r = r0; r <= r1; ++r) s1 += all_part[r][p].x, s2 += all_part[r][p].y;
      reinterpret_cast<float2*>(plane_sums)[(size_t)(row / sh.groups) * sh.c + ch0 + p] = make_float2(s1, s2);
    }
  if (!dx) return;
  float avg = 0.f, avg_z = 0.f;
  for (int r = 0; r < ranks; ++r) avg += rank_part[r].x, avg_z += rank_part[r].y;
  avg /= sh.count;
  avg_z /= sh.count;
#pragma unroll 4
  for (int k = 0; k < n; ++k) {
    const uint32_t u = u0 + k * THREADS;
    if (u >= end) break;
    const float w = gamma ? __ldg(gamma + ch0 + (int)rows.plane_div.div(u)) : 1.f;
    const Unit<VEC> xu = xs.unit(k);
    Unit<VEC> gu = gs.unit(k);
#pragma unroll
    for (int j = 0; j < VEC; ++j) gu.v[j] = rstd * (gu.v[j] * w - avg - (xu.v[j] - mean) * rstd * avg_z);
    gu.store(dx + base + (size_t)u * VEC);
  }
}

}  // namespace nres
}  // namespace b200

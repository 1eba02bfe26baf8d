// Forward and dInput of dense layers whose tiles leave SMs idle: the reduction channels in slices.
//
// A small batch of a deep layer has few pixels and a long reduction: 512 -> 512 channels of one 7x7 image are 8 tiles of 144 filter
// stages each, 62 us on 8 of 148 SMs (now 21); 64 such images fill a wave only with narrow tiles, at 60 % of the tensor core's pace.  Slices of the
// reduction channels ride on the group dimension of the strip kernels (slice s of the input is a group of its own), each writes a partial
// result, and the second kernel here adds them in order with bias, residual and ReLU.
#include <algorithm>

#include "common.cuh"
#include "plan_cache.cuh"

namespace b200 {
namespace {

constexpr int MAX_SLICES = 16;

// out[n][c][p] = sum over s of part[n][s][c][p] + bias[c] + residual, clamped when relu; V adjacent values of an image per thread
// (a residual is added only where they are pixels of one row-major plane)
template <int V>
__global__ void __launch_bounds__(256) add_slices_kernel(const float* part, int slices, uint32_t count, uint32_t image, FastDiv image_div, FastDiv plane_div,
                                                         FastDiv row_div, const float* __restrict__ bias, long long bias_stride, View4 res, int relu,
                                                         float* __restrict__ out) {
  const uint32_t i = (blockIdx.x * 256u + threadIdx.x) * V;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (i >= count) return;
  const uint32_t n = image_div.div(i), in_image = i - n * image;
  const float* p = part + (long long)n * slices * image + in_image;
  float v[V] = {};
#pragma unroll 4
  for (int s = 0; s < slices; ++s) {
    const float* q = p + (long long)s * image;
    if (V == 4) {
      const float4 f = *reinterpret_cast<const float4*>(q);
      v[0] += f.x; v[1 % V] += f.y; v[2 % V] += f.z; v[3 % V] += f.w;
    } else {
      v[0] += *q;
    }
  }
  if (bias) {
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] += __ldg(bias + plane_div.div(in_image + j) * bias_stride);
  }
  if (res.ptr) {
    const uint32_t c = plane_div.div(in_image), at = in_image - c * plane_div.d, y = row_div.div(at), x = at - y * row_div.d;
    const float* q = res.ptr + n * res.s0 + c * res.s1 + y * res.s2 + x * res.s3;
#pragma unroll
    for (int j = 0; j < V; ++j) v[j] += __ldg(q + j);
  }
#pragma unroll
  for (int j = 0; j < V; ++j)
    if (relu) v[j] = fmaxf(v[j], 0.f);
  if (V == 4) *reinterpret_cast<float4*>(out + i) = make_float4(v[0], v[1 % V], v[2 % V], v[3 % V]);
  else out[i] = v[0];
}

// The layer as `slices` groups: group s reduces its share of the channels into a result of its own.
ConvGeom sliced(const ConvGeom& g, bool is_dx, int slices) {
  ConvGeom s = g;
  s.groups = slices;
  if (is_dx) { s.cog = g.cout / slices; s.cin = slices * g.cin; }
  else { s.cig = g.cin / slices; s.cout = slices * g.cout; }
  return s;
}
size_t image_bytes(const ConvGeom& g, bool is_dx, bool transposed) {
  const int phase = is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD;
  return ((transposed ? tstrip_workspace(g, phase) : strip_workspace(g, phase)) + 255) & ~(size_t)255;
}
long long out_count(const ConvGeom& g, bool is_dx) { return is_dx ? (long long)g.n * g.cin * g.h * g.w : (long long)g.n * g.cout * g.oh * g.ow; }

}  // namespace

// Slices by the kernels' own time models; 1 when one slice is as good.  A second launch costs about 3 us and the partial results a
// write and a read, so layers below 12 us, or with two waves of tiles and more, are not looked at further (64 -> 64 channels of one 28x28
// image, 13 us, gain nothing: half the stages against the second launch).
static int plan_slices(const ConvGeom& g, bool is_dx, bool transposed, double* time = nullptr) {
  const int kc = is_dx ? g.cout : g.cin, phase = is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD;
  if (!transposed && !strip_supported(g, phase)) return 1;
  const long long values = out_count(g, is_dx);
  if (values * MAX_SLICES >= 1ll << 31) return 1;
  long long tiles;
  const double whole = transposed ? tstrip_time(g, is_dx, &tiles) : strip_time(g, is_dx, &tiles);
  if (time) *time = whole;
  if (whole < 12.0 || tiles >= 2ll * sm_count()) return 1;
  int best = 1;
  double best_time = whole;
  for (int s = 2; s <= std::min(MAX_SLICES, kc / 32); ++s) {
    if (kc / 32 % s) continue;
    const ConvGeom gs = sliced(g, is_dx, s);
    const double t = (transposed ? tstrip_time(gs, is_dx, nullptr) : strip_time(gs, is_dx, nullptr)) + 3.0 + (double)values * (8.0 * s + 4.0) * 2e-7;
    if (t < 0.95 * best_time) { best = s; best_time = t; }
  }
  if (time) *time = best_time;
  return best;
}
double conv_slices_time(const ConvGeom& g, bool is_dx) {
  const int kc = is_dx ? g.cout : g.cin;
  double time = strip_time(g, is_dx, nullptr);
  if (g.groups == 1 && kc % 32 == 0 && kc >= 64) plan_slices(g, is_dx, false, &time);
  return time;
}
int conv_slices(const ConvGeom& g, bool is_dx, bool allow_transposed) {
  const int kc = is_dx ? g.cout : g.cin;
  if (g.groups != 1 || kc % 32 || kc < 64) return 1;
  const bool transposed = allow_transposed && tstrip_supported(g, is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD);
  thread_local PlanCache<int> cache;
  return cache.get(g, 2 * transposed + is_dx, [&] { return plan_slices(g, is_dx, transposed); });
}

// Bytes of workspace for that many slices: the filter images and the partial results.
size_t conv_slices_workspace(const ConvGeom& g, bool is_dx, int slices, bool allow_transposed) {
  const int phase = is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD;
  const bool transposed = allow_transposed && tstrip_supported(g, phase);
  return image_bytes(sliced(g, is_dx, slices), is_dx, transposed) + (size_t)slices * out_count(g, is_dx) * sizeof(float);
}

int conv_sliced(const ConvGeom& g, bool is_dx, int slices, bool allow_transposed, View4 act, View4 w, const float* bias, long long bias_stride,
                const StripPostOps* post, float* out, void* ws, cudaStream_t st) {
  const int phase = is_dx ? B200_PHASE_DINPUT : B200_PHASE_FORWARD;
  const bool transposed = allow_transposed && tstrip_supported(g, phase);
  const ConvGeom gs = sliced(g, is_dx, slices);
  const size_t images = image_bytes(gs, is_dx, transposed);
  float* part = reinterpret_cast<float*>(static_cast<char*>(ws) + images);
  StripBatch b;
  b.w_group_extra = is_dx ? 0 : gs.cig * w.s1 - g.cout * w.s0;   // slice s starts s * cig input channels into the same filters
  const int rc = transposed ? tstrip_conv(gs, is_dx, act, w, nullptr, 0, part, ws, images, st, b.w_group_extra)
                            : strip_conv(gs, is_dx, act, w, nullptr, 0, part, ws, images, st, false, 1.f, 1.f, nullptr, nullptr, &b);
  if (rc) return rc;
  const int channels = is_dx ? g.cin : g.cout, oh = is_dx ? g.h : g.oh, ow = is_dx ? g.w : g.ow;
  const View4 res = post ? post->residual : View4{};
  const uint32_t plane = (uint32_t)(oh * ow), image = plane * (uint32_t)channels, count = (uint32_t)out_count(g, is_dx);
  const bool vec = image % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (!res.ptr || (plane % 4 == 0 && res.s3 == 1 && res.s2 == ow));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((count / (vec ? 4 : 1) + 255) / 256); cfg.blockDim = dim3(256); cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  B200_CUDA(cudaLaunchKernelEx(&cfg, vec ? add_slices_kernel<4> : add_slices_kernel<1>, (const float*)part, slices, count, image, FastDiv(image),
                               FastDiv(plane), FastDiv((uint32_t)ow), bias, bias_stride, res, post ? post->relu : 0, out));
  count_launch();
  return launch_check("add_slices_kernel");
}

}  // namespace b200

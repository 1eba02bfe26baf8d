// The pass behind both tcgen05 dWeight kernels, and the entry points of the tensor-memory one (dweight_tc_tmem.cu).
#pragma once
#include "common.cuh"

namespace b200 {
namespace tcdw {
// dW = sum of `splits` partials [split][cout][kh*kw][cig] (dweight_tc_strip.cu)
int finalize_partials(const float* partial, float* dw, const ConvGeom& g, int splits, cudaStream_t st);
}  // namespace tcdw
namespace tcdt {
// What the tensor-memory kernel would do with this budget; false where it does not take the geometry.
struct PlanInfo {
  size_t bytes;       // scratch for the split partials
  int kblocks;        // K blocks of a CTA
  int strips, slots;  // input strips and accumulator slots of a CTA
  bool shift;         // two vertical taps to a strip (64 output channels and fewer)
};
bool plan_info(const ConvGeom& g, size_t budget, PlanInfo* info);
int run(const ConvGeom& g, View4 x, View4 dy, float* dw, void* ws, size_t ws_bytes, cudaStream_t st);
}  // namespace tcdt
}  // namespace b200

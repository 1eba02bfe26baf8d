// Fused attention without mask and dropout (attention_fused.cu); contiguous [batch][tokens][d] operands, 16-byte aligned workspace.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace b200 {
namespace fa {
bool supported(int64_t batch, int64_t tq, int64_t tk, int64_t d, int64_t dv);
bool aligned(std::initializer_list<const void*> pointers);
size_t workspace(int64_t batch, int64_t tq, int64_t tk, int64_t d, bool backward);
int forward(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* q, const float* k, const float* v, int causal, float scale, float* out,
            float* lse, void* ws, cudaStream_t st);
int backward(int64_t batch, int64_t tq, int64_t tk, int64_t d, const float* grad, const float* q, const float* k, const float* v, const float* out,
             const float* lse, int causal, float scale, float* dq, float* dk, float* dv, void* ws, cudaStream_t st);
}  // namespace fa
}  // namespace b200

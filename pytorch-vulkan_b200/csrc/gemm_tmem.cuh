// The GEMM kernel with its left operand in tensor memory (gemm_tc_tmem.cu), launched by conv_tc_strip.cu behind its staging kernel.
#pragma once
#include "common.cuh"

namespace b200 {
namespace gt {
struct GemmArgs {
  const float* A;            // A[g][m][k] at g * a_group + m * a_m + k * a_k
  long long a_m, a_k, a_group;
  const float* images;       // stage images of B for column tiles of bn: [group][column tile][K block]
  const float* bias;         // per group and column, or null
  long long bias_stride;
  float* C;                  // C[g][m][n] at g * c_group + m * c_pitch + n
  long long c_pitch, c_group;
  int M, N, kc, k_total;     // kc: reduction values of a group; k_total: of all groups (the last may have fewer)
  int kblocks, tiles_m, tiles_n, tiles;
  int m_fastest;             // tile order
  int along_k;               // A in lines along k, else along m
  int pieces16;              // the lines start at multiples of 16 bytes (always so along m)
  int vec_out;               // rows of C may be written 16 bytes at a time
  int wait_for_images;
  int planes;                // 1x1 convolution on pixel planes: a group is an image, all share B and the bias, C[g][n][m] at g * c_group + n * c_pitch + m
  float alpha, beta;
  int* status;
  FastDiv div_m, div_n, div_kblocks;
};
int run(GemmArgs a, int bn, cudaStream_t st);
constexpr int PLANES_B = 128 << 10;   // bytes of B's images that the planes form keeps in shared memory
}  // namespace gt
}  // namespace b200

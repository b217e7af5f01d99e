// What the fp32 projection kernels (sgemm.cu, sgemm_tc.cu) share.
#pragma once

#include "common.cuh"

namespace mintb {

struct SgemmParams {
  const float* x;
  const float *w[6], *bias[6];
  float* out[6];
  const float* resid;      // row-major [M][N] or null
  int M, N, K, gelu;
  int B, T, H, D;          // D > 0: head-major outputs, row m = t * B + b, column n = h * D + d
};

// sgemm_tc.cu: the same on the tensor cores
bool sgemm_tc_wins(int groups, int M, int N, int K);
size_t sgemm_tc_workspace_bytes(int groups, int M, int N, int K);
int launch_sgemm_tc(const SgemmParams& p, int groups, void* workspace, cudaStream_t s, int* status);

}  // namespace mintb

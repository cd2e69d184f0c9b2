// Host interface of the cluster split-K GEMM (gemm_splitk.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct SplitkCall {
  const void *A, *B;
  void* C;
  int M, N, K;
  int64_t lda, ldb, ldc;
  int a_mn, b_mn, out_fp32, accumulate;
};

struct SplitkPlan {
  int slices;   // 1: do not split
  double clocks = 0;   // estimate of the chosen way, a launch included
};

// Whether the product is better split along K than run on the persistent kernel of tile width `bn`
// (`pair`: 256-row tiles on CTA pairs, else 128-row tiles).
SplitkPlan plan_splitk(int M, int N, int K, bool pair, int bn);
int launch_splitk(const SplitkCall& c, bool pair, SplitkPlan plan, cudaStream_t stream);

}  // namespace b200

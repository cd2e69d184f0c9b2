// The two products of a SwiGLU MLP that carry the activation in their epilogue:
//
//   gemm_swiglu     : gate|up = x [gate; up]^T and act = silu(gate) * up, in one launch
//   gemm_swiglu_bwd : d(gate)|d(up) from d(act) = dy W_down and the saved gate|up, in one launch
//
// The weights are stored as two halves, gate over up, as a plain linear layer has them. A SwiGLU pass of its own reads
// gate|up again (forward), or d(act), which was written for it, and gate|up (backward): 352 and 587 MB for 4096 tokens
// of 14336, which memory bounds. Against two launches (CUDA events, L2 flushed), forward and backward: 4096 tokens x 14336 x
// 4096 663 -> 587 us and 394 -> 337; 8192 x 8192 x 2048 413 -> 339 and 276 -> 216; 2048 x 8192 x 1024 87 -> 65 and
// 73 -> 60; 8192 x 4096 x 256 99 -> 67 and 89 -> 81; 256 x 512 x 256 15 -> 13 and 15 -> 15. Both times of launches alone, in
// a graph: the gradient's product has tiles of two widths only and an epilogue that the last tile does not hide, and below about 8 M elements
// of d(act) it is up to 14 % slower than a product and a pass (300 x 5632 x 2048 23.5 us, 20.6; 2048 x 1376 x 512 17.0 and 15.1; 256 x 512 x
// 256 8.3 and 7.6), above 5 to 22 % faster. It keeps d(act) in 32 bits, which a pass would have to write and read; forward and backward
// together are as fast as three launches and two or faster at 110 of 112 sizes (256 to 8192 tokens, 128 to 28672 x 64 to 8192).
#include "b200ops.h"
#include "gemm_epilogues.cuh"
#include "gemm_plan.h"
#include "gemm_tcgen05_2cta.cuh"
#include "host_util.h"

namespace b200 {

// Epilogue warps of the gradient's kernel: 64 columns take a warp 5000 clocks, 1400 of them waiting for gate and up. Four
// warps are as fast where the products take longer than that (K from about 4096 on), and slower otherwise: 4096 tokens x
// 14336 x 1024 188 us, 142 with eight. The forward epilogue loads nothing and keeps four warps and the sixth stage.
constexpr int BWD_EW = 8;

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
    gemm_swiglu_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const __grid_constant__ CUtensorMap tmGate, const __grid_constant__ CUtensorMap tmUp,
                       const __grid_constant__ CUtensorMap tmAct, GemmShape shape, int F, int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SwiGluSplitEpilogue epi{&tmGate, &tmUp, &tmAct, F, {}, {}, {}, {}};
  epi.slab.init(smem_raw, Gemm2Smem<BN>::EPI_OFF);
  NoGate gate;
  gemm_mainloop_2cta<BN, false, false>(&tmA, &tmB, shape, epi, gate, err_word, smem_raw);
}

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Gemm2Smem<BN, BWD_EW>::THREADS, 1)
    gemm_swiglu_bwd_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                           const __grid_constant__ CUtensorMap tmGate, const __grid_constant__ CUtensorMap tmUp,
                           const __grid_constant__ CUtensorMap tmDGate, const __grid_constant__ CUtensorMap tmDUp, GemmShape shape,
                           int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SwiGluBwdEpilogue<BWD_EW> epi{&tmGate, &tmUp, &tmDGate, &tmDUp, 0, 0, 0, 0, nullptr, nullptr};
  epi.init(smem_raw, Gemm2Smem<BN, BWD_EW>::EPI_OFF);
  NoGate gate;
  gemm_mainloop_2cta<BN, false, true, SwiGluBwdEpilogue<BWD_EW>, NoGate, false, BWD_EW>(&tmA, &tmB, shape, epi, gate, err_word, smem_raw);
}

template <int BN>
static int launch_swiglu(const void* x, const void* w, void* gu, void* act, int M, int F, int K, int64_t ldx, PairTiles tiles,
                         cudaStream_t stream) {
  GemmShape shape{M, 2 * F, K, 0, 0};
  const int grid = pair_grid(shape, tiles, BN, sm_count());
  shape.b_second = F;
  CUtensorMap tmA, tmB, tmGate, tmUp, tmAct;
  __nv_bfloat16* g = static_cast<__nv_bfloat16*>(gu);
  int rc;
  if ((rc = make_tmap_2d(&tmA, x, M, K, ldx, 128, GEMM_BK, 2, true))) return rc;
  if ((rc = make_tmap_2d(&tmB, w, 2 * static_cast<uint64_t>(F), K, K, shape.b_box, GEMM_BK, 2, true))) return rc;
  if ((rc = make_tmap_2d(&tmGate, g, M, F, 2 * static_cast<uint64_t>(F), 32, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&tmUp, g + F, M, F, 2 * static_cast<uint64_t>(F), 32, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&tmAct, act, M, F, F, 32, 64, 2, true))) return rc;
  constexpr auto kern = gemm_swiglu_kernel<BN>;
  if ((rc = allow_smem<kern>(Gemm2Smem<BN>::TOTAL_EPI))) return rc;
  launch_dependent(kern, grid, GEMM_THREADS, Gemm2Smem<BN>::TOTAL_EPI, stream, tmA, tmB, tmGate, tmUp, tmAct, shape, F, device_status_word());
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int BN>
static int launch_swiglu_bwd(const void* dy, const void* w, const void* gu, void* dgu, int M, int F, int K, int64_t lddy,
                             PairTiles tiles, cudaStream_t stream) {
  using S = Gemm2Smem<BN, BWD_EW>;
  GemmShape shape{M, F, K, 0, 0};
  const int grid = pair_grid(shape, tiles, BN, sm_count());
  CUtensorMap tmA, tmB, tm[4];
  int rc;
  if ((rc = make_tmap_2d(&tmA, dy, M, K, lddy, 128, GEMM_BK, 2, true))) return rc;
  if ((rc = make_tmap_2d(&tmB, w, K, F, F, GEMM_BK, 64, 2, true))) return rc;
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat16* base = static_cast<const __nv_bfloat16*>(i < 2 ? gu : dgu) + (i & 1) * F;
    if ((rc = make_tmap_2d(&tm[i], base, M, F, 2 * static_cast<uint64_t>(F), 32, 64, 2, true))) return rc;
  }
  constexpr auto kern = gemm_swiglu_bwd_kernel<BN>;
  if ((rc = allow_smem<kern>(S::TOTAL_EPI))) return rc;
  launch_dependent(kern, grid, S::THREADS, S::TOTAL_EPI, stream, tmA, tmB, tm[0], tm[1], tm[2], tm[3], shape, device_status_word());
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

static bool mlp_args_ok(const void* a, const void* b, const void* c, const void* d, int M, int F, int K, int64_t lda) {
  if (!a || !b || !c || !d || M <= 0 || F <= 0 || K <= 0 || F % 8 || K % 8 || lda % 8) return false;
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
           reinterpret_cast<uintptr_t>(d)) & 15) == 0;
}

}  // namespace b200

extern "C" {
using namespace b200;

// gu[M,2F] = x[M,K] w[2F,K]^T, gate over up in w, and act[M,F] = silu(gate) * up; contiguous but for x's row pitch.
int b200_gemm_swiglu(const void* x, const void* w, void* gu, void* act, int M, int F, int K, long long ldx, void* stream) {
  ensure_context();
  if (!mlp_args_ok(x, w, gu, act, M, F, K, ldx)) return B200_ERR_BAD_ARG;
  PairTiles tiles;
  if (!runs_on_pairs(M, 2 * F, K, ldx, K, false, x, w, &tiles)) {
    const int rc = b200_gemm_bf16(x, w, gu, M, 2 * F, K, ldx, K, 2ll * F, 0, 0, 0, 0, 0, 0, stream);
    return rc ? rc : b200_swiglu_fwd(gu, act, M, F, stream);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (tiles.width == 128) return launch_swiglu<128>(x, w, gu, act, M, F, K, ldx, tiles, s);
  return launch_swiglu<256>(x, w, gu, act, M, F, K, ldx, tiles, s);
}

// dgu[M,2F] = the gradient of SwiGLU at gu[M,2F] for d(act) = dy[M,K] w[K,F]; contiguous but for dy's row pitch. `scratch`
// [M,F] bf16 holds d(act) where the product does not run whole on CTA pairs.
int b200_gemm_swiglu_bwd(const void* dy, const void* w, const void* gu, void* dgu, void* scratch, int M, int F, int K, long long lddy,
                         void* stream) {
  ensure_context();
  if (!mlp_args_ok(dy, w, gu, dgu, M, F, K, lddy)) return B200_ERR_BAD_ARG;
  PairTiles tiles;
  if (!runs_on_pairs(M, F, K, lddy, F, true, dy, w, &tiles)) {
    if (!scratch) return B200_ERR_BAD_ARG;
    const int rc = b200_gemm_bf16(dy, w, scratch, M, F, K, lddy, F, F, 0, 1, 0, 0, 0, 0, stream);
    return rc ? rc : b200_swiglu_bwd(scratch, gu, dgu, M, F, stream);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (tiles.width == 128) return launch_swiglu_bwd<128>(dy, w, gu, dgu, M, F, K, lddy, tiles, s);
  return launch_swiglu_bwd<256>(dy, w, gu, dgu, M, F, K, lddy, tiles, s);
}

// Kernels that the two calls launch: one on CTA pairs, otherwise two.
int b200_gemm_swiglu_launches(const void* x, const void* w, int M, int F, int K, long long ldx) {
  ensure_context();
  PairTiles tiles;
  return runs_on_pairs(M, 2 * F, K, ldx, K, false, x, w, &tiles) ? 1 : 2;
}
int b200_gemm_swiglu_bwd_launches(const void* dy, const void* w, int M, int F, int K, long long lddy) {
  ensure_context();
  PairTiles tiles;
  return runs_on_pairs(M, F, K, lddy, F, true, dy, w, &tiles) ? 1 : 2;
}

}  // extern "C"

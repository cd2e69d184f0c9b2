// Dispatch of the cluster split-K GEMM: when it is taken, with how many slices, and its launch.
#include <atomic>

#include "gemm_splitk.cuh"
#include "gemm_splitk.h"
#include "host_util.h"

namespace b200 {

int* device_status_word();

namespace {

template <bool PAIR, int BN, bool A_MN, bool B_MN, typename OutT>
cudaLaunchConfig_t config(cudaLaunchAttribute* attr, int tiles, int slices, cudaStream_t stream) {
  const int cluster = slices * (PAIR ? 2 : 1);
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = cluster;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * cluster);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = SplitkSmem<PAIR, BN>::TOTAL;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <bool PAIR, int BN, bool A_MN, bool B_MN, typename OutT>
int launch(const SplitkCall& c, int slices, cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  int rc = A_MN ? make_tmap_2d(&tmA, c.A, c.K, c.M, c.lda, GEMM_BK, 64, 2, true)
                : make_tmap_2d(&tmA, c.A, c.M, c.K, c.lda, 128, GEMM_BK, 2, true);
  if (rc) return rc;
  rc = B_MN ? make_tmap_2d(&tmB, c.B, c.K, c.N, c.ldb, GEMM_BK, 64, 2, true)
            : make_tmap_2d(&tmB, c.B, c.N, c.K, c.ldb, PAIR ? BN / 2 : BN, GEMM_BK, 2, true);
  if (rc) return rc;
  constexpr int BM = PAIR ? 256 : 128;
  GemmShape shape{c.M, c.N, c.K, (c.M + BM - 1) / BM, (c.N + BN - 1) / BN};
  auto kern = gemm_splitk_kernel<PAIR, BN, A_MN, B_MN, OutT>;
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitkSmem<PAIR, BN>::TOTAL));
    attr_set.store(true, std::memory_order_release);
  }
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = config<PAIR, BN, A_MN, B_MN, OutT>(&attr, shape.tiles_m * shape.tiles_n, slices, stream);
  B200_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, static_cast<OutT*>(c.C), static_cast<int64_t>(c.ldc), shape, slices,
                                  c.accumulate, device_status_word()));
  return 0;
}

template <bool PAIR, int BN, typename OutT>
int launch_major(const SplitkCall& c, int slices, cudaStream_t s) {
  if (!c.a_mn && !c.b_mn) return launch<PAIR, BN, false, false, OutT>(c, slices, s);
  if (!c.a_mn) return launch<PAIR, BN, false, true, OutT>(c, slices, s);
  if (!c.b_mn) return launch<PAIR, BN, true, false, OutT>(c, slices, s);
  return launch<PAIR, BN, true, true, OutT>(c, slices, s);
}

// Clusters of `slices` members that run at once. The variants of one (PAIR, BN) use the same shared
// memory and threads, so one of them stands for all.
template <bool PAIR, int BN>
int resident_clusters(int log2_slices) {
  static std::atomic<int> known[4] = {{-1}, {-1}, {-1}, {-1}};
  int n = known[log2_slices].load(std::memory_order_relaxed);
  if (n >= 0) return n;
  auto kern = gemm_splitk_kernel<PAIR, BN, false, false, __nv_bfloat16>;
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = config<PAIR, BN, false, false, __nv_bfloat16>(&attr, 1, 1 << log2_slices, nullptr);
  n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitkSmem<PAIR, BN>::TOTAL) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();   // not available: the persistent kernels serve every size
    n = 0;
  }
  known[log2_slices].store(n, std::memory_order_relaxed);
  return n;
}

int resident_clusters(bool pair, int bn, int log2_slices) {
  if (pair) return bn == 256 ? resident_clusters<true, 256>(log2_slices) : resident_clusters<true, 128>(log2_slices);
  return bn == 256 ? resident_clusters<false, 256>(log2_slices) : resident_clusters<false, 128>(log2_slices);
}

// SM clocks per 64-deep k-block of one CTA: the larger of the tensor pipe's time (4096 multiply-adds a
// clock and SM) and of the operand bytes at the 64 B a clock that an SM takes in from L2.
int kblock_clocks(bool pair, int bn) { return pair ? (bn == 256 ? 512 : 384) : (bn == 256 ? 768 : 512); }

}  // namespace

SplitkPlan plan_splitk(int M, int N, int K, bool pair, int bn) {
  constexpr int FIXED = 5000;        // clocks of a launch besides its k-blocks: ramp, pipeline fill, epilogue
  constexpr int JOIN = 2500;         // cluster barriers and the sum over the slices
  constexpr int MIN_KBLOCKS = 4;     // a slice shorter than this does not fill its pipeline
  constexpr double HBM_BYTES_PER_CLOCK = 3500;
  const int units = pair ? sm_count() / 2 : sm_count();
  const int64_t rows = pair ? (M + 255) / 256 : (M + 127) / 128;
  const int kb = (K + GEMM_BK - 1) / GEMM_BK;
  const double floor = 2.0 * (static_cast<double>(M) * K + static_cast<double>(N) * K + static_cast<double>(M) * N) / HBM_BYTES_PER_CLOCK;
  auto at_least_floor = [&](double t) { return t > floor ? t : floor; };
  const int64_t tiles = rows * ((N + bn - 1) / bn);
  const double whole = at_least_floor(static_cast<double>((tiles + units - 1) / units) * kb * kblock_clocks(pair, bn)) + FIXED;
  SplitkPlan best{0, 1};
  double best_t = 0.85 * whole;   // the model is rough: a split has to promise 15 %
  for (int b = 128; b <= 256; b *= 2) {
    if (b > 128 && N <= 128) continue;
    const int64_t t = rows * ((N + b - 1) / b);
    for (int l = 1; l <= 3; ++l) {
      const int slices = 1 << l;
      if (slices * (pair ? 2 : 1) > SPLITK_MAX_CLUSTER || kb < slices * MIN_KBLOCKS) break;
      if (t * slices > units || t > resident_clusters(pair, b, l)) break;   // one wave only
      const double est = at_least_floor(static_cast<double>((kb + slices - 1) / slices) * kblock_clocks(pair, b)) + FIXED + JOIN;
      if (est < best_t) {
        best_t = est;
        best = SplitkPlan{b, slices};
      }
    }
  }
  return best;
}

int launch_splitk(const SplitkCall& c, bool pair, SplitkPlan plan, cudaStream_t s) {
  const int n = plan.slices;
  if (pair) {
    if (plan.bn == 256) return c.out_fp32 ? launch_major<true, 256, float>(c, n, s) : launch_major<true, 256, __nv_bfloat16>(c, n, s);
    return c.out_fp32 ? launch_major<true, 128, float>(c, n, s) : launch_major<true, 128, __nv_bfloat16>(c, n, s);
  }
  if (plan.bn == 256) return c.out_fp32 ? launch_major<false, 256, float>(c, n, s) : launch_major<false, 256, __nv_bfloat16>(c, n, s);
  return c.out_fp32 ? launch_major<false, 128, float>(c, n, s) : launch_major<false, 128, __nv_bfloat16>(c, n, s);
}

}  // namespace b200

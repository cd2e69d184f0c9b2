// Dispatch of the cluster split-K GEMM: when it is taken, with how many slices, and its launch.
#include <atomic>

#include "gemm_splitk.cuh"
#include "gemm_splitk.h"
#include "host_util.h"

namespace b200 {

int* device_status_word();

namespace {

template <bool PAIR>
cudaLaunchConfig_t config(cudaLaunchAttribute* attr, int tiles, int slices, cudaStream_t stream) {
  const int cluster = slices * (PAIR ? 2 : 1);
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see dependent_launch.cuh
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * cluster);
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = SplitkSmem<PAIR>::TOTAL;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

template <bool PAIR, bool A_MN, bool B_MN, typename OutT>
int launch(const SplitkCall& c, int slices, cudaStream_t stream) {
  constexpr int BM = PAIR ? 256 : 128, BN = SPLITK_BN;
  CUtensorMap tmA, tmB;
  int rc = A_MN ? make_tmap_2d(&tmA, c.A, c.K, c.M, c.lda, GEMM_BK, 64, 2, true)
                : make_tmap_2d(&tmA, c.A, c.M, c.K, c.lda, 128, GEMM_BK, 2, true);
  if (rc) return rc;
  rc = B_MN ? make_tmap_2d(&tmB, c.B, c.K, c.N, c.ldb, GEMM_BK, 64, 2, true)
            : make_tmap_2d(&tmB, c.B, c.N, c.K, c.ldb, PAIR ? BN / 2 : BN, GEMM_BK, 2, true);
  if (rc) return rc;
  GemmShape shape{c.M, c.N, c.K, (c.M + BM - 1) / BM, (c.N + BN - 1) / BN};
  constexpr auto kern = gemm_splitk_kernel<PAIR, A_MN, B_MN, OutT>;
  if ((rc = allow_smem<kern>(SplitkSmem<PAIR>::TOTAL))) return rc;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config<PAIR>(attr, shape.tiles_m * shape.tiles_n, slices, stream);
  B200_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, static_cast<OutT*>(c.C), static_cast<int64_t>(c.ldc), shape, slices,
                                  c.accumulate, device_status_word()));
  return 0;
}

template <bool PAIR, typename OutT>
int launch_major(const SplitkCall& c, int slices, cudaStream_t s) {
  if (!c.a_mn && !c.b_mn) return launch<PAIR, false, false, OutT>(c, slices, s);
  if (!c.a_mn) return launch<PAIR, false, true, OutT>(c, slices, s);
  if (!c.b_mn) return launch<PAIR, true, false, OutT>(c, slices, s);
  return launch<PAIR, true, true, OutT>(c, slices, s);
}

// Clusters of `slices` members that run at once. The variants of one PAIR use the same shared memory and
// threads, so one of them stands for all.
template <bool PAIR>
int resident_clusters(int log2_slices) {
  static std::atomic<int> known[4] = {{-1}, {-1}, {-1}, {-1}};
  int n = known[log2_slices].load(std::memory_order_relaxed);
  if (n >= 0) return n;
  constexpr auto kern = gemm_splitk_kernel<PAIR, false, false, __nv_bfloat16>;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = config<PAIR>(attr, 1, 1 << log2_slices, nullptr);
  n = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitkSmem<PAIR>::TOTAL) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();   // not available: the persistent kernels serve every size
    n = 0;
  }
  known[log2_slices].store(n, std::memory_order_relaxed);
  return n;
}

// SM clocks per 64-deep k-block of a CTA when `ctas` of them run: a CTA alone waits for its own pipeline,
// many share what L2 delivers.
double kblock_clocks(bool pair, int bn, int64_t ctas) {
  if (pair) return 295 + 1.7 * ctas;
  if (bn == 256) return 690;
  const double shared = 300 + 4.6 * ctas;
  return shared > 390 ? shared : 390;
}

}  // namespace

// The constants are fitted to times of both kernels at 16 to 1024 rows, 64 to 4096 columns and K from 256 to
// 14336 (343 products, L2 flushed and warm): of the 143 that are split none is slower than the persistent
// kernel, and the mean of the times relative to it is 0.83, where the best choice at every size gives 0.82.
// From about K = 4096 on a split gains: 256 x 256 x 4096 19.4 -> 16.6 us, x 14336 46.1 -> 22.6; at K = 1024
// the join (4 to 6 us) costs more than it saves (13.2 -> 14.3).
SplitkPlan plan_splitk(int M, int N, int K, bool pair, int bn) {
  constexpr double FIXED = 10000;        // clocks of a launch besides its k-blocks: ramp, pipeline fill, epilogue
  constexpr double JOIN = 6500, JOIN_SLICE = 600;   // cluster barriers and the sum over the slices
  constexpr int MIN_KBLOCKS = 4;         // a slice shorter than this does not fill its pipeline
  constexpr double HBM_BYTES_PER_CLOCK = 3500;
  const int per_tile = pair ? 2 : 1;
  const int units = sm_count() / per_tile;
  const int64_t rows = pair ? (M + 255) / 256 : (M + 127) / 128;
  const int kb = (K + GEMM_BK - 1) / GEMM_BK;
  const double floor = 2.0 * (static_cast<double>(M) * K + static_cast<double>(N) * K + static_cast<double>(M) * N) / HBM_BYTES_PER_CLOCK;
  auto at_least_floor = [&](double t) { return t > floor ? t : floor; };
  const int64_t whole_tiles = rows * ((N + bn - 1) / bn);
  const int64_t busy = whole_tiles < units ? whole_tiles : units;
  const double whole =
      at_least_floor(static_cast<double>((whole_tiles + units - 1) / units) * kb * kblock_clocks(pair, bn, busy * per_tile)) + FIXED;
  const int64_t tiles = rows * ((N + SPLITK_BN - 1) / SPLITK_BN);
  int best = 1;
  double best_t = 0.9 * whole, clocks = whole;   // the model is rough: a split has to promise 10 %
  for (int l = 1; l <= 3; ++l) {
    const int slices = 1 << l;
    if (slices * per_tile > SPLITK_MAX_CLUSTER || kb < slices * MIN_KBLOCKS) break;
    // one wave only
    if (tiles * slices > units || tiles > (pair ? resident_clusters<true>(l) : resident_clusters<false>(l))) break;
    const double est = at_least_floor(static_cast<double>((kb + slices - 1) / slices) * kblock_clocks(pair, SPLITK_BN, tiles * slices * per_tile)) +
                       FIXED + JOIN + JOIN_SLICE * slices;
    if (est < best_t) {
      best_t = clocks = est;
      best = slices;
    }
  }
  return SplitkPlan{best, clocks};
}

int launch_splitk(const SplitkCall& c, bool pair, SplitkPlan plan, cudaStream_t s) {
  const int n = plan.slices;
  if (pair) return c.out_fp32 ? launch_major<true, float>(c, n, s) : launch_major<true, __nv_bfloat16>(c, n, s);
  return c.out_fp32 ? launch_major<false, float>(c, n, s) : launch_major<false, __nv_bfloat16>(c, n, s);
}

}  // namespace b200

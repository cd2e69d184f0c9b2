// The gradients of a linear layer: one launch for both products or one for each, and the plan that decides.
#include <algorithm>

#include "b200ops.h"
#include "gemm_grads.cuh"
#include "gemm_plan.h"
#include "host_util.h"

namespace b200 {

// What the joint kernel runs on.
struct GradsPlan {
  int width[2];   // columns of a tile of dx and of dw: 128, 192 or 256
  int first;      // the product that goes first
  int fill;
  int warps;      // epilogue warps
  double clocks;  // estimate
};

namespace {

struct GradsCall {
  const void *dy, *x, *w;
  void *dx, *dw;
  int M, N, K;
  int64_t lddy, ldx, ldw, lddx, lddw;
  int accumulate;
};

int64_t tiles_of(int rows, int cols, int width) {
  return static_cast<int64_t>((rows + GEMM2_BM - 1) / GEMM2_BM) * ((cols + width - 1) / width);
}

GradsPlan plan_with(const GradsCall& c, int w_dx, int w_dw, bool lines, int pairs) {
  GradsPlan p{{w_dx, w_dw}, 0, 0, c.M <= SHORT_K ? 8 : 4, 0};
  const double t[2] = {pair_tile_clocks(c.N, w_dx, lines, p.warps), pair_tile_clocks(c.M, w_dw, lines, p.warps)};
  const int64_t n[2] = {tiles_of(c.M, c.K, w_dx), tiles_of(c.N, c.K, w_dw)};
  p.first = t[1] > t[0];
  const double long_t = t[p.first], short_t = t[p.first ^ 1];
  const int64_t n_first = n[p.first], n_second = n[p.first ^ 1];
  const int64_t units = n_first + n_second < pairs ? n_first + n_second : pairs;
  const int64_t longer = n_first % units;
  const double ratio = long_t / short_t;
  p.fill = longer ? static_cast<int>(ratio < 1000 ? ratio + 0.5 : 1000) : 0;
  const int64_t base = std::min(n_second, longer ? (units - longer) * p.fill : 0), rest = n_second - base;
  const double each = static_cast<double>(n_first / units) * long_t + static_cast<double>((rest + units - 1) / units) * short_t;
  const double filled = longer ? static_cast<double>((base + units - longer - 1) / (units - longer)) * short_t : 0;
  p.clocks = each + std::max(longer ? long_t : 0.0, filled);
  return p;
}

bool on_lines(const GradsCall& c) {
  const uint64_t low = reinterpret_cast<uintptr_t>(c.dy) | reinterpret_cast<uintptr_t>(c.x) | reinterpret_cast<uintptr_t>(c.w) |
                       static_cast<uint64_t>(c.lddy | c.ldx | c.ldw) * 2;
  return low % 128 == 0;
}

// A layer whose narrow tiles all run at once, with reductions too short to be worth splitting, is one launch of those: the plan of
// anything larger would take such a layer as long on the host as the launch that it saves.
bool one_wave(const GradsCall& c) {
  return std::max(c.M, c.N) <= 2048 && tiles_of(c.M, c.K, 128) + tiles_of(c.N, c.K, 128) <= sm_count() / 2;
}

GradsPlan plan_joint(const GradsCall& c) {
  if (one_wave(c)) return {{128, 128}, c.M > c.N, 1, c.M <= SHORT_K ? 8 : 4, 0};   // one tile for every pair
  const bool lines = on_lines(c);
  const int pairs = sm_count() / 2;
  GradsPlan best{};
  best.clocks = 1e30;
  for (int w_dx = 256; w_dx >= 128; w_dx -= 64)
    for (int w_dw = 256; w_dw >= 128; w_dw -= 64) {
      if ((w_dx > 128 || w_dw > 128) && c.K <= std::max(w_dx, w_dw) - 64) continue;   // narrower ones cover the row as well
      const GradsPlan p = plan_with(c, w_dx, w_dw, lines, pairs);
      if (p.clocks < best.clocks * 0.99) best = p;
    }
  return best;
}

// One launch or two. Two win where one product is a few tiles with a long reduction, which a launch of its own splits
// over clusters, and for few rows through a weight that L2 does not hold: a single row of tiles takes the weight from memory
// at the pace of its own pipeline, and joint kernels got 3.8 TB/s there where dx alone gets 5.3 (128 x 4096 x 14336
// with cold weights 63 us, 58 in two). Of 128 layers (M 16 to 8192, N 64 to 28672, K 64 to 14336, and the 8B model's) the
// rule took one launch for 93; the mean of its times was 0.789 of two launches', the faster way's 0.785. Since the second of two launches comes up
// while the first one ends (EARLY clocks), of 920 layers (M 16 to 8192, most of them 16 to 384, N 64 to 28672, K 64 to 14336) it takes one for 753 where
// 743 would be faster so; the mean of its times is 1.004 of the faster way's, 1.002 over 315 layers of 257 to 384 rows, and 34 are slower by
// more than 3 % (192 x 9408 x 1984 44 us for 31, 88 x 8320 x 3072 42 and 33). Between 129 and 256 rows dx by itself is a single row of tiles as well, and takes longer than the
// estimate for a product by itself says: of 37 such layers over weights of 64 to 600 MB with N <= 3 K the rule takes one launch for 33; the mean of
// its times is 0.86 of two launches' and 1.008 of the faster way's, 1.089 with the line that fewer rows have (256 x 8192 x 8192 72 us for
// 86, 200 x 5120 x 13824 73 and 92, 256 x 6144 x 6144 47 and 59). A longer reduction is a chain that two launches split (136 x 28672 x 4096 126 us, 147 jointly).
// 256 x 768 x 256: 11 us for 20; 1000 x 2568 x 5160 58 for 75; 4096 x 4096 x 4096 158 for 169.
bool pays(const GradsCall& c, const GradsPlan& p) {
  if (!pairs_enabled()) return false;
  if (one_wave(c)) return true;
  const bool few_rows = c.M <= GEMM2_BM && 2.0 * c.N * c.K > 64e6;
  const bool one_pair_row = few_rows && c.M > GEMM_BM && c.N <= 3ll * c.K;   // a row of tiles on CTA pairs in either way
  double alone = pair_tile_clocks(c.N, p.width[0], on_lines(c), p.warps);
  if (few_rows) alone = std::max(alone, (one_pair_row ? 520.0 : 700.0) * ((c.N + GEMM_BK - 1) / GEMM_BK));
  const double moved = (one_pair_row ? 1.15 : few_rows ? 1.25 : 0.8) * (memory_clocks(c.M, c.K, c.N) + memory_clocks(c.N, c.K, c.M));
  constexpr double EARLY = 4000;
  const double joint = std::max({p.clocks, alone, moved}) + LAUNCH_CLOCKS + EARLY;
  return joint < (one_pair_row ? 1.08 : 1.0) * (product_clocks(c.M, c.K, c.N, c.lddy, c.ldw, true, c.dy, c.w) + product_clocks(c.N, c.K, c.M, c.lddy, c.ldx, true, c.dy, c.x));
}

GemmShape product_shape(int rows, int cols, int k, int width) {
  GemmShape s{rows, cols, k, (rows + GEMM2_BM - 1) / GEMM2_BM, (cols + width - 1) / width};
  s.group_m = pair_group_m(GRADS_BN);
  s.bn = width;
  plan_walk(s, 2);
  return s;
}

template <int EW>
int launch(const GradsCall& c, const GradsPlan& p, cudaStream_t stream) {
  using S = Gemm2Smem<GRADS_BN, EW>;
  CUtensorMap rows, cols, w, x, dx, dw;
  const int whole = c.K & ~7;   // columns that TMA stores: whole vectors
  const int out_cols = whole ? whole : 8;
  // a single row may come with any pitch
  const int64_t one = (static_cast<int64_t>(c.K) + 7) / 8 * 8;
  int rc;
  if ((rc = make_tmap_2d(&rows, c.dy, c.M, c.N, c.lddy, 128, GEMM_BK, 2, true))) return rc;
  if ((rc = make_tmap_2d(&cols, c.dy, c.M, c.N, c.lddy, GEMM_BK, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&w, c.w, c.N, c.K, c.ldw, GEMM_BK, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&x, c.x, c.M, c.K, c.ldx, GEMM_BK, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&dx, c.dx, c.M, out_cols, c.M == 1 ? one : c.lddx, 32, 64, 2, true))) return rc;
  if ((rc = make_tmap_2d(&dw, c.dw, c.N, out_cols, c.N == 1 ? one : c.lddw, 32, 64, 2, true))) return rc;
  GradsArgs a{};
  int64_t tiles = 0;
  for (int i = 0; i < 2; ++i) {
    a.shape[i] = i == 0 ? product_shape(c.M, c.K, c.N, p.width[0]) : product_shape(c.N, c.K, c.M, p.width[1]);
    tiles += static_cast<int64_t>(a.shape[i].tiles_m) * a.shape[i].tiles_n;
  }
  a.out[0] = static_cast<__nv_bfloat16*>(c.dx);
  a.out[1] = static_cast<__nv_bfloat16*>(c.dw);
  a.ld_out[0] = c.lddx;
  a.ld_out[1] = c.lddw;
  a.accumulate = c.accumulate;
  a.first = p.first;
  a.fill = p.fill;
  constexpr auto kern = gemm_grads_kernel<EW>;
  if ((rc = allow_smem<kern>(S::TOTAL_EPI))) return rc;
  const int pairs = sm_count() / 2;
  const int grid = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  launch_dependent(kern, grid, S::THREADS, S::TOTAL_EPI, stream, rows, cols, w, x, dx, dw, a, device_status_word());
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

bool grads_args_ok(const GradsCall& c) {
  if (!c.dy || !c.x || !c.w || !c.dx || !c.dw || c.M <= 0 || c.N <= 0 || c.K <= 0) return false;
  const uintptr_t at = reinterpret_cast<uintptr_t>(c.dy) | reinterpret_cast<uintptr_t>(c.x) | reinterpret_cast<uintptr_t>(c.w) |
                       reinterpret_cast<uintptr_t>(c.dx) | reinterpret_cast<uintptr_t>(c.dw);
  return at % 16 == 0 && (c.lddy | c.ldx | c.ldw | c.lddx | c.lddw) % 8 == 0;
}

}  // namespace
}  // namespace b200

extern "C" {
using namespace b200;

// Both products in one launch, with tiles of the given widths (0: chosen).
int b200_linear_grads_joint(const void* dy, const void* x, const void* w, void* dx, void* dw, int M, int N, int K, long long lddy,
                            long long ldx, long long ldw, long long lddx, long long lddw, int accumulate, int w_dx, int w_dw,
                            void* stream) {
  ensure_context();
  const GradsCall c{dy, x, w, dx, dw, M, N, K, lddy, ldx, ldw, lddx, lddw, accumulate};
  if (!grads_args_ok(c)) return B200_ERR_BAD_ARG;
  GradsPlan p;
  if (w_dx == 0 && w_dw == 0) {
    p = plan_joint(c);
  } else {
    if (w_dx < 128 || w_dx > 256 || w_dx % 64 || w_dw < 128 || w_dw > 256 || w_dw % 64) return B200_ERR_BAD_ARG;
    p = plan_with(c, w_dx, w_dw, on_lines(c), sm_count() / 2);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return p.warps == 8 ? launch<8>(c, p, s) : launch<4>(c, p, s);
}

// dx[M,K] = dy[M,N] w[N,K] and dw[N,K] (+)= dy^T x[M,K], bf16, in one launch or in two (*launches says which).
int b200_linear_grads(const void* dy, const void* x, const void* w, void* dx, void* dw, int M, int N, int K, long long lddy,
                      long long ldx, long long ldw, long long lddx, long long lddw, int accumulate, int* launches, void* stream) {
  ensure_context();
  const GradsCall c{dy, x, w, dx, dw, M, N, K, lddy, ldx, ldw, lddx, lddw, accumulate};
  if (!grads_args_ok(c)) return B200_ERR_BAD_ARG;
  const GradsPlan p = plan_joint(c);
  if (pays(c, p)) {
    *launches = 1;
    return p.warps == 8 ? launch<8>(c, p, static_cast<cudaStream_t>(stream)) : launch<4>(c, p, static_cast<cudaStream_t>(stream));
  }
  *launches = 2;
  const int rc = b200_gemm_bf16(dy, w, dx, M, K, N, lddy, ldw, lddx, 0, 1, 0, 0, 0, 0, stream);
  return rc ? rc : b200_gemm_bf16(dy, x, dw, N, K, M, lddy, ldx, lddw, 1, 1, 0, accumulate, 0, 0, stream);
}

// Whether that is one launch, for operands with contiguous rows on cache-line boundaries, and its tile widths.
int b200_linear_grads_plan(int M, int N, int K, int* joint, int* w_dx, int* w_dw) {
  ensure_context();
  if (M <= 0 || N <= 0 || K <= 0 || !joint || !w_dx || !w_dw) return B200_ERR_BAD_ARG;
  const GradsCall c{nullptr, nullptr, nullptr, nullptr, nullptr, M, N, K, N, K, K, K, K, 0};
  const GradsPlan p = plan_joint(c);
  *joint = pays(c, p);
  *w_dx = p.width[0];
  *w_dw = p.width[1];
  return 0;
}

// M tiles of 256 rows per raster group of the joint kernel.
int b200_linear_grads_group(int M, int N, int K) { return product_shape(M, K, N, 128).group_m; }

}  // extern "C"

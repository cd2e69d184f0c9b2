// bf16 GEMM entry points built on the tcgen05 mainloop.
//
//   C[M,N] (+)= op(A) * op(B)     fp32 accumulation in TMEM, bf16 or fp32 output
//
// Operand storage is described by two flags instead of BLAS transposes:
//   a_mn = 0 : A stored [M][K] (K contiguous)      a_mn = 1 : A stored [K][M] (M contiguous)
//   b_mn = 0 : B stored [N][K] (K contiguous)      b_mn = 1 : B stored [K][N] (N contiguous)
// so a linear layer's forward (x W^T), input gradient (dy W) and weight gradient (dy^T x) all run
// on the same kernel without materialising a transpose.
#include <cuda_fp8.h>

#include <algorithm>
#include <atomic>

#include "b200ops.h"
#include "gemm_epilogues.cuh"
#include "gemm_plan.h"
#include "gemm_splitk.h"
#include "gemm_tcgen05.cuh"
#include "gemm_tcgen05_2cta.cuh"
#include "host_util.h"

namespace b200 {

// Part of the library's image, zero when that is loaded: a first call may come while a stream is being captured, where nothing may be
// allocated or set, and from several threads at once.
__device__ int g_status_word;

int* device_status_word() {
  static std::atomic<int*> words[64];
  int dev = -1;
  cudaGetDevice(&dev);
  const bool known = dev >= 0 && dev < 64;
  if (int* w = known ? words[dev].load(std::memory_order_acquire) : nullptr) return w;
  void* w = nullptr;
  if (cudaGetSymbolAddress(&w, g_status_word) != cudaSuccess) return nullptr;
  if (known) words[dev].store(static_cast<int*>(w), std::memory_order_release);
  return static_cast<int*>(w);
}

// C as the epilogues store it: boxes of 32 rows x 128 bytes. A store clips a row at 16 bytes, not at an
// element, so the map ends at the last whole vector (a C narrower than one has no use for its map).
template <typename OutT>
static int make_tmap_out(CUtensorMap* tm, const void* C, int M, int N, int64_t ldc) {
  if (M == 1) ldc = (static_cast<int64_t>(N) + 7) / 8 * 8;   // a single row may come with any pitch
  const int cols = whole_vectors<OutT>(N);
  return make_tmap_2d(tm, C, M, cols ? cols : 16 / sizeof(OutT), ldc, 32, 128 / sizeof(OutT), sizeof(OutT), true);
}

template <int BN, bool A_MN, bool B_MN, typename OutT>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, OutT* C, int64_t ldc, GemmShape shape, int accumulate,
                     int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  StoreEpilogue<OutT> epi{&tmC, C, ldc, accumulate, {}};
  epi.slab.init(smem_raw, GemmSmem<BN>::EPI_OFF);
  NoGate gate;
  gemm_mainloop<BN, A_MN, B_MN>(&tmA, &tmB, shape, epi, gate, err_word, smem_raw);
}

static int group_m_override() {
  static const int value = [] {
    const char* e = getenv("B200_GEMM_GROUP_M");
    return e ? atoi(e) : -1;
  }();
  return value;
}

// M tiles per raster group: the CTAs of one wave (one per SM) then cover a patch of about
// group_m x (SMs / group_m) tiles, which is close to square in elements for the default value.
// B200_GEMM_GROUP_M overrides it (0 = plain column-major walk).
int gemm_group_m(int bn) {
  if (group_m_override() >= 0) return group_m_override();
  return bn == 256 ? 16 : 12;
}

// A group of M tiles reads its rows of A once and all of B, so several groups take B from memory as often. Where one operand
// stays in L2 beside the streams, all of its tiles are walked before the next tile of the other operand, which is then read
// once: 4096 x 28672 x 4096 takes 0.33 GB from memory where groups of eight took 0.52. What that gains is power, which these
// products are bound by: looped over rotating buffers at the 1000 W limit it takes 711 us for 729, its weight gradient (N
// tiles first) 4096 x 14336 x 4096 364 for 371, 8192 x 16384 x 2048 417 for 429, the fp8 product 4096 x 14336 x 4096 with its
// quantiser 205 for 211. An operand of 34 MB stays; with 50 MB (6144 x 16384 x 4096, 5120 x 13824 x 5120) products took up to 2 %
// longer so, with 67 MB 6 %: the two halves of L2 each hold what their own SMs read. Operands of no more tiles than a group are
// walked whole by the groups (28672 x 2048 x 1024: N tiles first 105 us, 103 in groups). Where both operands are small both stay, and nothing is left to gain:
// over 623 such products the walk takes 0.995 of the time of groups on average, but 0.85 to 1.21 with how their stores fall, short reductions above all
// (5632 x 3592 x 352 with SwiGLU 54 us for 44, fp8 6656 x 8704 x 416 60 for 52); with a larger operand beyond 15 MB 0.990 over 284, and at most 1.03 but for one.
void plan_walk(GemmShape& s, int elem_bytes) {
  constexpr int64_t ROOM = 40000000, BOTH_STAY = 15000000;
  if (group_m_override() >= 0) return;
  const int64_t a = static_cast<int64_t>(s.M) * s.K * elem_bytes, b = static_cast<int64_t>(s.N) * s.K * elem_bytes;
  if (a <= BOTH_STAY && b <= BOTH_STAY) return;
  if (a <= b && a <= ROOM && s.tiles_m > s.group_m) {
    s.one_group = 1;
    s.m_major = 0;
  } else if (b < a && b <= ROOM && s.tiles_n > s.group_m) {
    s.m_major = 1;
  }
}

// max_ctas keeps SMs free for other streams. Such a product is launched when the kernel before it has ended, and releases none before it ends itself: the
// CTAs of a dependent, which come up wherever there is room, would hold those SMs.
static bool keeps_room(int max_ctas) { return max_ctas > 0 && max_ctas < sm_count(); }

template <int BN, bool A_MN, bool B_MN, typename OutT>
static int launch_gemm(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                       int64_t ldc, int accumulate, int max_ctas, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC;
  int rc;
  if (!A_MN)
    rc = make_tmap_2d(&tmA, A, M, K, lda, GEMM_BM, GEMM_BK, 2, true);
  else
    rc = make_tmap_2d(&tmA, A, K, M, lda, GEMM_BK, 64, 2, true);
  if (rc) return rc;
  if (!B_MN)
    rc = make_tmap_2d(&tmB, B, N, K, ldb, BN, GEMM_BK, 2, true);
  else
    rc = make_tmap_2d(&tmB, B, K, N, ldb, GEMM_BK, 64, 2, true);
  if (rc) return rc;
  if ((rc = make_tmap_out<OutT>(&tmC, C, M, N, ldc))) return rc;
  GemmShape shape{M, N, K, (M + GEMM_BM - 1) / GEMM_BM, (N + BN - 1) / BN};
  shape.group_m = gemm_group_m(BN);
  constexpr auto kern = gemm_bf16_kernel<BN, A_MN, B_MN, OutT>;
  if ((rc = allow_smem<kern>(GemmSmem<BN>::TOTAL_EPI))) return rc;
  int grid = shape.tiles_m * shape.tiles_n;
  shape.keep_room = keeps_room(max_ctas);
  const int cap = shape.keep_room ? max_ctas : sm_count();
  if (grid > cap) grid = cap;
  int* err = device_status_word();
  launch_after(!shape.keep_room, kern, grid, GEMM_THREADS, GemmSmem<BN>::TOTAL_EPI, stream, tmA, tmB, tmC, static_cast<OutT*>(C), ldc, shape, accumulate, err);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------- CTA-pair variant (256 x 256 tile per cluster)
template <int BN, bool A_MN, bool B_MN, typename OutT, int EW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Gemm2Smem<BN, EW>::THREADS, 1)
    gemm_bf16_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                          const __grid_constant__ CUtensorMap tmC, OutT* C, int64_t ldc, GemmShape shape, int accumulate,
                          int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  StoreEpilogue<OutT> epi{&tmC, C, ldc, accumulate, {}};
  epi.slab.init(smem_raw, Gemm2Smem<BN, EW>::EPI_OFF);
  NoGate gate;
  gemm_mainloop_2cta<BN, A_MN, B_MN, StoreEpilogue<OutT>, NoGate, false, EW>(&tmA, &tmB, shape, epi, gate, err_word, smem_raw);
}

int pair_grid(GemmShape& shape, PairTiles tiles, int bn, int ctas, int elem_bytes) {
  const int pairs = ctas / 2;
  shape.tiles_m = (shape.M + GEMM2_BM - 1) / GEMM2_BM;
  shape.tiles_n = (shape.N + tiles.width - 1) / tiles.width;
  shape.group_m = pair_group_m(bn);
  shape.bn = tiles.width;
  const int all = shape.tiles_m * shape.tiles_n;
  int items = all;
  if (tiles.halves) {
    shape.halve_from = all / pairs * pairs;
    items = 2 * all - shape.halve_from;
  }
  shape.b_box = tiles.width / (tiles.halves ? 4 : 2);
  plan_walk(shape, elem_bytes);
  return 2 * (items < pairs ? items : pairs);
}

template <int BN, bool A_MN, bool B_MN, typename OutT, int EW>
static int launch_gemm_2cta(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                            int64_t ldc, int accumulate, PairTiles tiles, int max_ctas, cudaStream_t stream) {
  using S = Gemm2Smem<BN, EW>;
  CUtensorMap tmA, tmB, tmC;
  int rc;
  GemmShape shape{M, N, K, 0, 0};
  shape.keep_room = keeps_room(max_ctas);
  const int grid = pair_grid(shape, tiles, BN, shape.keep_room ? max_ctas : sm_count());
  // every CTA loads 128 rows of A and its half of the tile's rows of B per k-block
  if (!A_MN)
    rc = make_tmap_2d(&tmA, A, M, K, lda, 128, GEMM_BK, 2, true);
  else
    rc = make_tmap_2d(&tmA, A, K, M, lda, GEMM_BK, 64, 2, true);
  if (rc) return rc;
  if (!B_MN)
    rc = make_tmap_2d(&tmB, B, N, K, ldb, shape.b_box, GEMM_BK, 2, true);
  else
    rc = make_tmap_2d(&tmB, B, K, N, ldb, GEMM_BK, 64, 2, true);
  if (rc) return rc;
  if ((rc = make_tmap_out<OutT>(&tmC, C, M, N, ldc))) return rc;
  constexpr auto kern = gemm_bf16_2cta_kernel<BN, A_MN, B_MN, OutT, EW>;
  if ((rc = allow_smem<kern>(S::TOTAL_EPI))) return rc;
  int* err = device_status_word();
  launch_after(!shape.keep_room, kern, grid, S::THREADS, S::TOTAL_EPI, stream, tmA, tmB, tmC, static_cast<OutT*>(C), ldc, shape, accumulate, err);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int BN, typename OutT, int EW = 4>
static int dispatch_major_2cta(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                               int64_t ldc, int a_mn, int b_mn, int accumulate, PairTiles tiles, int max_ctas, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_gemm_2cta<BN, false, false, OutT, EW>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, tiles, max_ctas, stream);
  if (!a_mn && b_mn) return launch_gemm_2cta<BN, false, true, OutT, EW>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, tiles, max_ctas, stream);
  if (a_mn && !b_mn) return launch_gemm_2cta<BN, true, false, OutT, EW>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, tiles, max_ctas, stream);
  return launch_gemm_2cta<BN, true, true, OutT, EW>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, tiles, max_ctas, stream);
}

// The narrow kernel has more stages; tiles of any other width run on the wide one. Eight epilogue warps store one tile during the next one's
// products; where every pair has a single tile there is no next one, and four start sooner: 1504 x 1784 x 96 5.9 -> 5.5 us, 3200 x 1136
// x 128 6.1 -> 5.9, 4 to 8 % over products of 38 to 74 tiles. Four are slower from three waves on (4096 x 4096 x 128 by 8 %), with two it varies.
static int epilogue_warps(int M, int N, int K, int width, int out_fp32, int ctas) {
  const int64_t tiles = static_cast<int64_t>((M + GEMM2_BM - 1) / GEMM2_BM) * ((N + width - 1) / width);
  return width > 128 && K <= SHORT_K && !out_fp32 && tiles > ctas / 2 ? 8 : 4;
}
static int gemm_2cta(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc, int a_mn,
                     int b_mn, int out_fp32, int accumulate, PairTiles tiles, int max_ctas, cudaStream_t s) {
  if (tiles.width == 128)
    return out_fp32 ? dispatch_major_2cta<128, float>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, tiles, max_ctas, s)
                    : dispatch_major_2cta<128, __nv_bfloat16>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, tiles, max_ctas, s);
  if (epilogue_warps(M, N, K, tiles.width, out_fp32, keeps_room(max_ctas) ? max_ctas : sm_count()) == 8)
    return dispatch_major_2cta<256, __nv_bfloat16, 8>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, tiles, max_ctas, s);
  return out_fp32 ? dispatch_major_2cta<256, float>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, tiles, max_ctas, s)
                  : dispatch_major_2cta<256, __nv_bfloat16>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, tiles, max_ctas, s);
}

// ---------------------------------------------------------------- fp8 (e4m3) x fp8 -> bf16 with row / column scales
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
    gemm_fp8_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const __grid_constant__ CUtensorMap tmC, __nv_bfloat16* C, int64_t ldc, const float* row_scale,
                         const float* col_scale, GemmShape shape, int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  ScaledStoreEpilogue epi{&tmC, C, ldc, row_scale, col_scale, {}};
  epi.slab.init(smem_raw, Gemm2Smem<BN>::EPI_OFF);
  NoGate gate;
  gemm_mainloop_2cta<BN, false, false, ScaledStoreEpilogue, NoGate, true>(&tmA, &tmB, shape, epi, gate, err_word, smem_raw);
}

template <int BN>
static int launch_gemm_fp8(const void* A, const void* B, const float* a_scale, const float* b_scale, void* C, int M, int N,
                           int K, int64_t lda, int64_t ldb, int64_t ldc, PairTiles tiles, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC;
  GemmShape shape{M, N, K, 0, 0};
  const int grid = pair_grid(shape, tiles, BN, sm_count(), 1);
  int rc = make_tmap_2d(&tmA, A, M, K, lda, 128, 2 * GEMM_BK, 1, true);   // 128 one-byte elements = 128 B per row
  if (rc) return rc;
  rc = make_tmap_2d(&tmB, B, N, K, ldb, shape.b_box, 2 * GEMM_BK, 1, true);
  if (rc) return rc;
  if ((rc = make_tmap_out<__nv_bfloat16>(&tmC, C, M, N, ldc))) return rc;
  constexpr auto kern = gemm_fp8_2cta_kernel<BN>;
  if ((rc = allow_smem<kern>(Gemm2Smem<BN>::TOTAL_EPI))) return rc;
  launch_dependent(kern, grid, GEMM_THREADS, Gemm2Smem<BN>::TOTAL_EPI, stream, tmA, tmB, tmC, static_cast<__nv_bfloat16*>(C), ldc, a_scale, b_scale,
                                                                     shape, device_status_word());
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// One e4m3 row per bf16 row: scale = amax / 448 (fp32), q = x / scale.
__device__ __forceinline__ float amax8(uint4 raw, float amax) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fmaxf(fabsf(__low2float(p[j])), fabsf(__high2float(p[j]))));
  return amax;
}
__device__ __forceinline__ uint2 scaled_e4m3(uint4 raw, float inv) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
  uint32_t w[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 f0 = __bfloat1622float2(p[2 * h]), f1 = __bfloat1622float2(p[2 * h + 1]);
    w[h] = static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(f0.x * inv, f0.y * inv), __NV_SATFINITE, __NV_E4M3)) |
           (static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(f1.x * inv, f1.y * inv), __NV_SATFINITE, __NV_E4M3)) << 16);
  }
  return make_uint2(w[0], w[1]);
}
__device__ __forceinline__ float warp_max32(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// TPR threads hold a row in registers, VPT vectors each: it is read once and all its loads are in flight together,
// where a warp that goes over the row twice waits for each: 4096 x 4096 14 us (L2 flushed), 20 that way, 4096 x 14336 34 and 71.
constexpr int QUANT_THREADS = 256;
template <int TPR, int VPT>
__global__ void __launch_bounds__(QUANT_THREADS)
    quant_rows_fp8_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scale, int rows, int K,
                          int64_t ldx, int64_t ldq) {
  after_wait(x, q, scale);
  grid_release();
  __shared__ float red[QUANT_THREADS / 32];
  const int t = threadIdx.x % TPR, warp = threadIdx.x >> 5;
  const int64_t r = static_cast<int64_t>(blockIdx.x) * (QUANT_THREADS / TPR) + threadIdx.x / TPR;
  const bool live = r < rows;
  const int nvec = K / 8;
  const uint4* src = reinterpret_cast<const uint4*>(x + r * ldx);
  uint4 raw[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    raw[i] = live && t + i * TPR < nvec ? src[t + i * TPR] : make_uint4(0, 0, 0, 0);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) amax = amax8(raw[i], amax);
  amax = warp_max32(amax);
  if constexpr (TPR > 32) {
    if ((threadIdx.x & 31) == 0) red[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TPR / 32; ++i) amax = fmaxf(amax, red[(warp & ~(TPR / 32 - 1)) + i]);
  }
  if (!live) return;
  const float s = fmaxf(amax, 1e-12f) * (1.f / 448.f);
  const float inv = 1.f / s;
  if (t == 0) scale[r] = s;
  uint2* dst = reinterpret_cast<uint2*>(q + r * ldq);
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    if (t + i * TPR < nvec) dst[t + i * TPR] = scaled_e4m3(raw[i], inv);
}

// Rows that a CTA's registers do not hold: a warp per row, twice over it.
__global__ void __launch_bounds__(QUANT_THREADS)
    quant_wide_rows_fp8_kernel(const __nv_bfloat16* x, uint8_t* q, float* scale, int rows, int K, int64_t ldx, int64_t ldq) {
  after_wait(x, q, scale);
  grid_release();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int64_t r = blockIdx.x * warps + warp; r < rows; r += gridDim.x * warps) {
    const uint4* src = reinterpret_cast<const uint4*>(x + r * ldx);
    const int nvec = K / 8;
    float amax = 0.f;
    for (int v = lane; v < nvec; v += 32) amax = amax8(src[v], amax);
    amax = warp_max32(amax);
    const float s = fmaxf(amax, 1e-12f) * (1.f / 448.f);
    const float inv = 1.f / s;
    if (lane == 0) scale[r] = s;
    uint2* dst = reinterpret_cast<uint2*>(q + r * ldq);
    for (int v = lane; v < nvec; v += 32) dst[v] = scaled_e4m3(src[v], inv);
  }
}

// B200_GEMM_2CTA=0 keeps every bf16 GEMM on the one-CTA kernel, and with it the joint gradients of a linear layer and the MLP's
// products, which only exist on pairs, in two launches each. By default CTA pairs are used wherever they apply (M >= 256, N >= 128; joint
// gradients from one row on). The fp8 product has no other kernel.
static int gemm_pair_mode() {
  static int mode = -2;
  if (mode == -2) {
    const char* e = getenv("B200_GEMM_2CTA");
    mode = e ? atoi(e) : -1;
  }
  return mode;
}

template <int BN, typename OutT>
static int dispatch_major(const void* A, const void* B, void* C, int M, int N, int K, int64_t lda, int64_t ldb,
                          int64_t ldc, int a_mn, int b_mn, int accumulate, int max_ctas, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_gemm<BN, false, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, max_ctas, stream);
  if (!a_mn && b_mn) return launch_gemm<BN, false, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, max_ctas, stream);
  if (a_mn && !b_mn) return launch_gemm<BN, true, false, OutT>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, max_ctas, stream);
  return launch_gemm<BN, true, true, OutT>(A, B, C, M, N, K, lda, ldb, ldc, accumulate, max_ctas, stream);
}

static bool gemm_args_ok(const void* A, const void* B, const void* C, int M, int N, int K, int64_t lda, int64_t ldb, int64_t ldc,
                         int out_fp32) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return false;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return false;
  return lda % 8 == 0 && ldb % 8 == 0 && ldc % (out_fp32 ? 4 : 8) == 0;
}

bool pairs_enabled() { return gemm_pair_mode() != 0; }
static bool use_pairs(int M, int N, int max_ctas) {
  return pairs_enabled() && M >= 256 && N >= 128 && (max_ctas == 0 || max_ctas >= 2);
}

// Three rows of 128 x 128 tiles that all run at once, where pairs would compute four rows in wide tiles on two thirds of the SMs: 257 to 384 rows
// and 4737 to 6272 columns. 384 x 6144 x 4096 19.4 us, 22.4 on pairs; 340 x 5952 x 2816 14.2 and 16.8; 384 x 6208 x 1024 8.3 and 10.4; 300 x
// 5120 x 13824 51 and 58. Fewer columns fit narrow pair tiles (384 x 4096 x 4096 16.6 us, 18.5 so), more take these two waves. A k-block takes THREE_ROWS_KBLOCK
// clocks there.
constexpr double THREE_ROWS_KBLOCK = 395;
static bool three_tile_rows(int M, int N) {
  const int columns = (N + 127) / 128;
  return M > 2 * GEMM_BM && M <= 3 * GEMM_BM && 3 * columns <= sm_count() && 2 * columns > sm_count() / 2;
}

// What a product with bn = 0 runs on: CTA pairs or single CTAs, the tile width of the persistent kernel, or a split along K.
// `a_at`, `b_at`: the operands' addresses (their alignment counts).
struct GemmChoice {
  bool pairs;
  int bn;            // the plain width that fits better, 128 or 256
  PairTiles tiles;   // on CTA pairs: what the product runs on
  SplitkPlan split;
};

// Tiles of a product on CTA pairs, in steps of `step` columns, whose better plain width is `bn`; a_low, b_low: what decides how the operands' rows
// lie on cache lines. A wave of narrower tiles costs more than their share of a wide one: their loads bring the
// same rows of A for fewer columns. Rows off cache lines take the loads half as long again, and the boxes of an N-major B
// are 64 columns, so that 160 and 224 columns (80 and 112 for a CTA) load as much as 256. The costs are medians over
// 140 products of 256 to 8192 rows, 128 to 28672 columns and K from 64 to 16040 in three majors; the rule's choice
// took 0.977 of the plain width's time on average there, the best choice 0.969, and none more than 1.03. What it
// gains is the last wave: 4096 x 4096 x 14336, 256 tiles for 74 pairs, takes 354 to 366 us in four wide waves and 329 with
// the last of them halved; 2048 x 8192 x 4096 93 and 86; 1000 x 5160 x 2568 40 us in two wide waves, 34 in two of 160 columns.
static PairTiles fit_tiles(int M, int N, int K, bool b_mn, uint64_t a_low, uint64_t b_low, int units, int bn,
                           int step = 32) {
  struct Costs {
    double at[5];   // 128, 160, 192, 224, 256 columns
  };
  static constexpr double NO = 9;
  static constexpr Costs ON_LINES[2] = {{{.58, .70, .785, .90, 1}}, {{.58, .79, .81, .90, 1}}};
  static constexpr Costs BETWEEN[2] = {{{.60, .72, .80, .90, 1}}, {{.605, NO, .90, .95, 1}}};
  static constexpr Costs OFF_LINES[2] = {{{.72, .79, .86, .925, 1}}, {{.72, NO, NO, NO, 1}}};
  const bool a_lines = a_low % 128 == 0, b_lines = b_low % 128 == 0;
  const Costs& c = a_lines && b_lines ? ON_LINES[b_mn] : a_lines || b_lines || (a_low | b_low) % 64 == 0 ? BETWEEN[b_mn] : OFF_LINES[b_mn];
  const int64_t rows = (M + GEMM2_BM - 1) / GEMM2_BM;
  // A width that is not the plain one has to promise 3 %, halves of the last wave 1 %. From K = 4096 on, with rows on cache lines, 2 % are enough, and
  // halves behind a single wave cost .64 of one, where behind several the pairs' drift hides some of it. Of 55 such products that
  // this gives another width none took more than 1.003 of the halves' time, and they took 0.967 on average: 768 x 8192 x 8192 99 -> 89 us,
  // 433 x 12416 x 10112 0.95, 2403 x 7680 x 11456 416 -> 396; 40 of fp8 (K is half of theirs) 0.98, 1343 x 4608 x 11520 68.1 -> 65.6. A shorter
  // K gains less and loses up to 3 % as often.
  const bool long_k = step == 32 && a_lines && b_lines && K >= 4096;
  const double gain = long_k ? 1.02 : 1.03;
  PairTiles best{bn, false};
  double best_cost = 1e30;
  for (int i = 0; i < 5; i += step / 32) {
    const int width = 128 + 32 * i;
    if (width > 128 && N <= width - step) break;   // a narrower one covers the row as well
    if (width % 64 && K < 1024) continue;        // the last 32 columns of a tile leave as vectors, not by TMA: with few k-blocks that counts
    const int64_t tiles = rows * ((N + width - 1) / width);
    const double cost = static_cast<double>((tiles + units - 1) / units) * c.at[i] * (width == bn ? 1 : gain);
    if (cost < best_cost) {
      best_cost = cost;
      best = {width, false};
    }
  }
  const int64_t wide = rows * ((N + 255) / 256), last = wide % units;
  const double half_wave = long_k && wide / units == 1 ? .64 : c.at[0];
  if (wide > units && last > 0 && 2 * last <= units && (static_cast<double>(wide / units) + half_wave) * 1.01 <= best_cost) best = {256, true};
  return best;
}
// three_rows: whether three_tile_rows may have it.
static GemmChoice choose_gemm(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, uintptr_t a_at, uintptr_t b_at, int max_ctas,
                              bool three_rows = true) {
  const bool pairs = use_pairs(M, N, max_ctas);
  const auto split_on = [&](int width) { return max_ctas == 0 ? plan_splitk(M, N, K, pairs, width) : SplitkPlan{1}; };
  int bn;
  PairTiles tiles{};
  // Wider tiles re-read A less; fall back to the narrower tile when that fills the SMs better.
  const int units = pairs ? sm_count() / 2 : sm_count();
  const long rows = pairs ? (M + 255) / 256 : (M + 127) / 128;
  const long t256 = rows * ((N + 255) / 256);
  const long t128 = rows * ((N + 127) / 128);
  const long w256 = (t256 + units - 1) / units, w128 = (t128 + units - 1) / units;
  if (pairs) {
    // With CTA pairs the tile is 256 rows tall and a wave is one tile per pair of SMs. A wave of narrow
    // tiles costs about 0.58 of one of wide tiles (4096 x 4096 x 14336: seven waves 376 us, four wide ones
    // 365), but nearly as much where the 128-byte rows of the operand boxes straddle cache lines and L2
    // delivers the operands late (1000 x 5160 x 2568: three waves 43 us, two wide ones 40;
    // 4096 x 4096 x 16040: seven 692 us, four wide ones 515). Where one operand straddles none, or every
    // second row of both straddles none (rows on 64 bytes), it lies between: two wide waves for three
    // narrow ones are slower (1068 x 3832 x 6432: 68 us, 60), three for five faster (by 3 to 18 %). With a
    // short K what a tile costs besides its products weighs more, and there are half as many: four wide waves for seven narrow
    // ones gain up to K = 2048 (6286 x 2368 x 640: 20.4 us, 21.0). The lines below lie between the products of each kind that
    // gained and those that lost, before waits suspended; the sizes here, timed since, are on the same side.
    const uintptr_t a_low = a_at | (static_cast<uintptr_t>(lda) * 2), b_low = b_at | (static_cast<uintptr_t>(ldb) * 2);
    const bool a_lines = a_low % 128 == 0, b_lines = b_low % 128 == 0, halves = (a_low | b_low) % 64 == 0;
    const double narrow_wave = a_lines && b_lines ? (K <= 2048 ? 0.58 : 0.56) : a_lines || b_lines || halves ? 0.62 : 0.85;
    bn = (N >= 256 && w256 <= narrow_wave * w128) ? 256 : 128;
    tiles = max_ctas == 0 ? fit_tiles(M, N, K, b_mn, a_low, b_low, units, bn) : PairTiles{bn, false};
  } else {
    const double eff256 = static_cast<double>(t256) / (w256 * units);
    const double eff128 = static_cast<double>(t128) / (w128 * units);
    bn = (N >= 256 && eff256 + 0.08 >= eff128) ? 256 : 128;
    // Narrow tiles that need no more waves are done sooner: 16 x 624 x 256 8 us, 10 in wide ones. The split is weighed against the
    // width above all the same, which its model was fitted to: against narrow tiles it would leave 24 x 560 x 2032 whole (12.8 us, 8.5 split).
    if (w256 == w128) {
      const SplitkPlan split = split_on(bn);
      return split.slices > 1 ? GemmChoice{false, bn, tiles, split} : GemmChoice{false, 128, tiles, split_on(128)};
    }
  }
  // Few tiles and a long K: the chip is filled by splitting K over clusters.
  const SplitkPlan split = split_on(bn);
  if (pairs && max_ctas == 0 && split.slices == 1 && three_rows && three_tile_rows(M, N)) return {false, 128, {}, split};
  return {pairs, bn, tiles, split};
}

double product_clocks(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, const void* A, const void* B) {
  const uintptr_t a_at = reinterpret_cast<uintptr_t>(A), b_at = reinterpret_cast<uintptr_t>(B);
  const GemmChoice g = choose_gemm(M, N, K, lda, ldb, b_mn, a_at, b_at, 0);
  const double floor = memory_clocks(M, N, K);
  // what the split model was fitted to had slower waits
  if (g.split.slices > 1) return std::max((g.split.clocks - LAUNCH_CLOCKS) * 0.7, floor) + LAUNCH_CLOCKS;
  if (!g.pairs) {
    const double tiles = use_pairs(M, N, 0) ? (K + GEMM_BK - 1) / GEMM_BK * THREE_ROWS_KBLOCK : (g.split.clocks - LAUNCH_CLOCKS) * 0.8;
    return std::max(tiles, floor) + LAUNCH_CLOCKS;
  }
  const bool lines = (a_at | b_at | static_cast<uint64_t>(lda | ldb) * 2) % 128 == 0;
  const int64_t rows = (M + GEMM2_BM - 1) / GEMM2_BM, units = sm_count() / 2;
  double best = 1e30;
  for (int width = 128; width <= 256; width += 64) {
    const int64_t tiles = rows * ((N + width - 1) / width);
    best = std::min(best, static_cast<double>((tiles + units - 1) / units) * pair_tile_clocks(K, width, lines, epilogue_warps(M, N, K, width, 0, sm_count())));
  }
  return std::max(best, floor) + LAUNCH_CLOCKS;
}

bool runs_on_pairs(int M, int N, int K, int64_t lda, int64_t ldb, bool b_mn, const void* A, const void* B, PairTiles* tiles) {
  if (!use_pairs(M, N, 0)) return false;
  const uintptr_t a_at = reinterpret_cast<uintptr_t>(A), b_at = reinterpret_cast<uintptr_t>(B);
  const GemmChoice g = choose_gemm(M, N, K, lda, ldb, b_mn, a_at, b_at, 0, false);
  if (g.split.slices > 1) return false;
  *tiles = fit_tiles(M, N, K, b_mn, a_at | (static_cast<uint64_t>(lda) * 2), b_at | (static_cast<uint64_t>(ldb) * 2), sm_count() / 2,
                     g.bn, 128);
  return true;
}

}  // namespace b200

extern "C" {

// Returns 0 on success. Alignment: base pointers and row pitches must be multiples of 16 bytes.
// out_fp32 selects an fp32 C; accumulate adds to the existing C. bn is 128 or 256 (0 = choose).
int b200_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                   long long ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int bn, int max_ctas,
                   void* stream) {
  b200::ensure_context();
  using namespace b200;
  if (!gemm_args_ok(A, B, C, M, N, K, lda, ldb, ldc, out_fp32)) return B200_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  bool pairs = use_pairs(M, N, max_ctas);   // of a width that the caller chose
  PairTiles tiles{bn, false};
  if (bn == 0) {
    const GemmChoice g =
        choose_gemm(M, N, K, lda, ldb, b_mn != 0, reinterpret_cast<uintptr_t>(A), reinterpret_cast<uintptr_t>(B), max_ctas);
    pairs = g.pairs;
    if (g.split.slices > 1)
      return launch_splitk({A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate}, pairs, g.split, s);
    bn = g.bn;
    tiles = g.tiles;
  }
  if (pairs && (bn == 256 || bn == 128))
    return gemm_2cta(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, tiles, max_ctas, s);
  if (bn == 256) {
    return out_fp32 ? dispatch_major<256, float>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, max_ctas, s)
                    : dispatch_major<256, __nv_bfloat16>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate,
                                                         max_ctas, s);
  }
  return out_fp32 ? dispatch_major<128, float>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate, max_ctas, s)
                  : dispatch_major<128, __nv_bfloat16>(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, accumulate,
                                                       max_ctas, s);
}

// What b200_gemm_bf16 with bn = 0 and max_ctas = 0 starts from for operands on cache-line boundaries: CTA pairs
// or single CTAs, slices of K (1: the persistent kernel) and the better one of its plain tile widths
// (b200_gemm_tiles has the tiles that CTA pairs then run on).
int b200_gemm_plan(int M, int N, int K, long long lda, long long ldb, int* pair, int* bn, int* slices) {
  b200::ensure_context();
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || !pair || !bn || !slices) return B200_ERR_BAD_ARG;
  const GemmChoice g = choose_gemm(M, N, K, lda, ldb, false, 0, 0, 0);
  *pair = g.pairs;
  *slices = g.split.slices;
  *bn = g.split.slices > 1 ? 128 : g.bn;
  return 0;
}

// The tiles of the same call where it runs on the persistent kernel of CTA pairs: their width and whether those
// of the last wave are halved.
int b200_gemm_tiles(int M, int N, int K, long long lda, long long ldb, int b_mn, int* width, int* halves) {
  b200::ensure_context();
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || !width || !halves) return B200_ERR_BAD_ARG;
  const GemmChoice g = choose_gemm(M, N, K, lda, ldb, b_mn != 0, 0, 0, 0);
  if (!g.pairs) return B200_ERR_BAD_ARG;
  *width = g.tiles.width;
  *halves = g.tiles.halves;
  return 0;
}

// b200_gemm_bf16 on CTA pairs with tiles of `width` columns (128 to 256 in steps of 32), those of the last wave
// halved or not (width 256 only), whatever the plan says.
int b200_gemm_bf16_tiles(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                         int a_mn, int b_mn, int out_fp32, int accumulate, int width, int halves, void* stream) {
  b200::ensure_context();
  using namespace b200;
  if (!gemm_args_ok(A, B, C, M, N, K, lda, ldb, ldc, out_fp32)) return B200_ERR_BAD_ARG;
  if (width < 128 || width > 256 || width % 32 || (halves && width != 256)) return B200_ERR_BAD_ARG;
  return gemm_2cta(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, PairTiles{width, halves != 0}, 0,
                   static_cast<cudaStream_t>(stream));
}

// b200_gemm_bf16 on the split kernel whatever the plan says: slices 2, 4 or 8 (with pair at most 4) and no
// more than K has 64-deep blocks.
int b200_gemm_bf16_split(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, int a_mn, int b_mn, int out_fp32, int accumulate, int pair, int slices, void* stream) {
  b200::ensure_context();
  using namespace b200;
  if (!gemm_args_ok(A, B, C, M, N, K, lda, ldb, ldc, out_fp32)) return B200_ERR_BAD_ARG;
  if ((slices != 2 && slices != 4 && slices != 8) || slices * (pair ? 2 : 1) > 8 || (K + GEMM_BK - 1) / GEMM_BK < slices)
    return B200_ERR_BAD_ARG;
  return launch_splitk({A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate}, pair != 0, SplitkPlan{slices},
                       static_cast<cudaStream_t>(stream));
}

// C[M,N] (bf16) = (A8[M,K] * B8[N,K]^T) * a_scale[M] x b_scale[N]; A8, B8 e4m3, K-major, K % 16 == 0.
// CTA pairs only: M >= 256 and N >= 128.
int b200_gemm_fp8(const void* A, const void* B, const float* a_scale, const float* b_scale, void* C, int M, int N, int K,
                  long long lda, long long ldb, long long ldc, void* stream) {
  b200::ensure_context();
  using namespace b200;
  if (!A || !B || !C || !a_scale || !b_scale || M < 256 || N < 128 || K <= 0) return B200_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(b_scale)) & 15)
    return B200_ERR_BAD_ARG;
  if ((lda % 16) || (ldb % 16) || (ldc % 8) || (K % 16) || (N % 4)) return B200_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int units = sm_count() / 2;
  const long rows = (M + 255) / 256;
  const long t256 = rows * ((N + 255) / 256), t128 = rows * ((N + 127) / 128);
  const double eff256 = static_cast<double>(t256) / (((t256 + units - 1) / units) * units);
  const double eff128 = static_cast<double>(t128) / (((t128 + units - 1) / units) * units);
  const int bn = N >= 256 && eff256 + 0.08 >= eff128 ? 256 : 128;
  // a k-block is 128 elements here, the same bytes
  const PairTiles tiles = fit_tiles(M, N, K / 2, false, reinterpret_cast<uintptr_t>(A) | static_cast<uint64_t>(lda),
                                    reinterpret_cast<uintptr_t>(B) | static_cast<uint64_t>(ldb), units, bn);
  if (tiles.width == 128) return launch_gemm_fp8<128>(A, B, a_scale, b_scale, C, M, N, K, lda, ldb, ldc, tiles, s);
  return launch_gemm_fp8<256>(A, B, a_scale, b_scale, C, M, N, K, lda, ldb, ldc, tiles, s);
}

// q[rows,K] (e4m3) and scale[rows] (fp32) from x[rows,K] (bf16); K % 8 == 0, 16-byte aligned rows.
int b200_quant_rows_fp8(const void* x, void* q, float* scale, int rows, int K, long long ldx, long long ldq, void* stream) {
  b200::ensure_context();
  if (!x || !q || !scale || rows <= 0 || K <= 0 || K % 8 || ldx % 8 || ldq % 8) return b200::B200_ERR_BAD_ARG;
  using namespace b200;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto Q = static_cast<uint8_t*>(q);
  // up to four vectors per thread while a warp can hold the row, then eight and more threads
#define B200_QUANT(TPR, VPT)                                                                                                   \
  launch_dependent(quant_rows_fp8_kernel<TPR, VPT>, (rows + QUANT_THREADS / TPR - 1) / (QUANT_THREADS / TPR), QUANT_THREADS, 0, st, X, Q, scale, rows, K, ldx, ldq)
  if (K <= 256) B200_QUANT(32, 1);
  else if (K <= 512) B200_QUANT(32, 2);
  else if (K <= 1024) B200_QUANT(32, 4);
  else if (K <= 2048) B200_QUANT(64, 4);
  else if (K <= 4096) B200_QUANT(128, 4);
  else if (K <= 8192) B200_QUANT(256, 4);
  else if (K <= 16384) B200_QUANT(256, 8);
  else {
    int grid = (rows + 7) / 8;
    const int cap = sm_count() * 8;
    if (grid > cap) grid = cap;
    launch_dependent(quant_wide_rows_fp8_kernel, grid, QUANT_THREADS, 0, st, X, Q, scale, rows, K, ldx, ldq);
  }
#undef B200_QUANT
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// Reads and clears the device status word (0 = no kernel gave up on a wait). Synchronises the device.
int b200_read_status(int clear) {
  b200::ensure_context();
  int* w = b200::device_status_word();
  if (!w) return -1;
  int v = 0;
  if (cudaMemcpy(&v, w, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -2;
  if (clear && v) cudaMemset(w, 0, sizeof(int));
  return v;
}

}  // extern "C"

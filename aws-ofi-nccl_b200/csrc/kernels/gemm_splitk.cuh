// GEMM for outputs with too few tiles to occupy the chip: a thread-block cluster computes ONE output
// tile, each of its `slices` members (a CTA, or a CTA pair) multiplying its own range of K, and the
// fp32 partial sums meet in distributed shared memory.
//
// A tile's slices are in one cluster, so the sum needs no workspace, no counters and no second
// launch: every CTA drains its accumulator into its own shared memory (the operand stages are free by
// then), the cluster synchronises, and every CTA adds up 1/slices of the tile's rows, always in the
// order of the slices, and stores them as full rows. Calls on any number of streams and threads share
// nothing. 128 tokens through a 4096 x 14336 projection (32 tiles, 224 k-blocks) take 36 us in four
// slices, 62 us on the persistent kernel; the bound is reading the weight, 18 us.
//
// Barriers as in the persistent mainloops, except that a member's leader is CTA (rank & ~1) of the
// cluster when PAIR is set. Every wait is bounded; a CTA that gives up still takes part in the
// cluster barriers, so nobody waits for it. No load is multicast.
#pragma once
#include "gemm_tcgen05_2cta.cuh"

namespace b200 {

// commit to the same barrier offset in the CTAs of `mask` (ranks in the cluster)
__device__ __forceinline__ void umma_commit_pair_mask(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}

constexpr int SPLITK_MAX_CLUSTER = 8;   // portable cluster size
// Tile width. Wider tiles have half the CTAs and twice the partial sums to join: at no size of 16 to 1024
// rows, 64 to 4096 columns and K from 256 to 14336 were they the faster split.
constexpr int SPLITK_BN = 128;

// Operand stages of a member CTA: the same as the persistent kernels' (Gemm2Smem / GemmSmem).
template <bool PAIR>
struct SplitkSmem {
  static constexpr int BN = SPLITK_BN;
  static constexpr int STAGE_BYTES = PAIR ? Gemm2Smem<BN>::STAGE_BYTES : GemmSmem<BN>::STAGE_BYTES;
  static constexpr int STAGES = PAIR ? Gemm2Smem<BN>::STAGES : GemmSmem<BN>::STAGES;
  static constexpr int A_BYTES = 128 * GEMM_BK * 2;
  static constexpr int TOTAL = 1024 + STAGES * STAGE_BYTES + 256;
  // partial sums: 128 rows, 16 bytes of padding each so that 32 rows' stores hit all banks
  static constexpr int RED_PITCH = (BN + 4) * 4;
  static_assert(128 * RED_PITCH <= STAGES * STAGE_BYTES, "the partial sums lie over the operand stages");
};

// grid = tiles x cluster size, cluster size = slices x (PAIR ? 2 : 1); shape.tiles_m counts 128-row
// tiles (256-row tiles with PAIR). 1 <= slices <= number of 64-deep k-blocks.
template <bool PAIR, bool A_MN, bool B_MN, typename OutT>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_splitk_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OutT* C, int64_t ldc,
                       GemmShape shape, int slices, int accumulate, int* err_word) {
  using S = SplitkSmem<PAIR>;
  constexpr int BN = SPLITK_BN;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t half = PAIR ? (crank & 1u) : 0u;           // which 128 rows of the tile
  const uint32_t lead = PAIR ? (crank & ~1u) : crank;       // the CTA that issues this member's MMAs
  const int slice = static_cast<int>(PAIR ? crank >> 1 : crank);
  const int tile = static_cast<int>(blockIdx.x) / (slices * (PAIR ? 2 : 1));
  const int tm = tile % shape.tiles_m, tn = tile / shape.tiles_m;
  const int num_kb = (shape.K + GEMM_BK - 1) / GEMM_BK;
  const int kb0 = static_cast<int>(static_cast<int64_t>(num_kb) * slice / slices);
  const int kb1 = static_cast<int>(static_cast<int64_t>(num_kb) * (slice + 1) / slices);
  const int row0 = tm * (PAIR ? 256 : 128) + static_cast<int>(half) * 128;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + S::STAGES * S::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (S::STAGES + s); };
  const uint32_t tfull_bar = bar_base + 8u * (2 * S::STAGES);
  const uint32_t tmem_slot = tfull_bar + 8u;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + (tmem_slot - smem_u32(smem_raw)) + 8u);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull_bar, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, BN);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, BN);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  grid_wait();   // the operands may be the kernel before's

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      constexpr int B_ROWS = PAIR ? BN / 2 : BN;   // rows of B this CTA loads
      const int col0 = tn * BN + static_cast<int>(half) * B_ROWS;
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1, abort_flag, err_word, DEV_ERR_EMPTY_BAR_TIMEOUT, GEMM_WAIT_LIMIT_NS))
          break;
        const uint32_t a_dst = smem_base + stage * S::STAGE_BYTES;
        const uint32_t b_dst = a_dst + S::A_BYTES;
        const uint32_t bar = PAIR ? map_to_cta(full_bar(stage), lead) : full_bar(stage);
        auto load = [&](uint32_t dst, const CUtensorMap* m, int x, int y) {
          if constexpr (PAIR)
            tma_load_2d_pair(dst, m, x, y, bar);
          else
            tma_load_2d(dst, m, x, y, bar);
        };
        if (half == 0) mbar_expect_tx(full_bar(stage), (PAIR ? 2 : 1) * S::STAGE_BYTES);
        if constexpr (!A_MN) {
          load(a_dst, &tmA, kb * GEMM_BK, row0);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) load(a_dst + j * 8192, &tmA, row0 + j * 64, kb * GEMM_BK);
        }
        if constexpr (!B_MN) {
          load(b_dst, &tmB, kb * GEMM_BK, col0);
        } else {
#pragma unroll
          for (int j = 0; j < B_ROWS / 64; ++j) load(b_dst + j * 8192, &tmB, col0 + j * 64, kb * GEMM_BK);
        }
        if (++stage == S::STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      grid_release();
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (half == 0 && elect_one_sync()) {
      constexpr uint32_t idesc = make_instr_desc(1, 1, PAIR ? 256 : 128, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      const uint16_t mask = static_cast<uint16_t>(3u << lead);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_bounded(full_bar(stage), phase, abort_flag, err_word, DEV_ERR_FULL_BAR_TIMEOUT, GEMM_WAIT_LIMIT_NS)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t a_src = smem_base + stage * S::STAGE_BYTES;
        const uint32_t b_src = a_src + S::A_BYTES;
#pragma unroll
        for (int k = 0; k < GEMM_BK / 16; ++k) {
          const uint64_t adesc = A_MN ? make_smem_desc_sw128(a_src + k * 2048, 8192, 1024)
                                      : make_smem_desc_sw128(a_src + k * 32, 16, 1024);
          const uint64_t bdesc = B_MN ? make_smem_desc_sw128(b_src + k * 2048, 8192, 1024)
                                      : make_smem_desc_sw128(b_src + k * 32, 16, 1024);
          const uint32_t acc = (kb != kb0 || k != 0) ? 1u : 0u;
          if constexpr (PAIR)
            umma_f16_pair(tmem_base, adesc, bdesc, idesc, acc);
          else
            umma_f16(tmem_base, adesc, bdesc, idesc, acc);
        }
        if constexpr (PAIR)
          umma_commit_pair_mask(empty_bar(stage), mask);
        else
          umma_commit(empty_bar(stage));
        if (++stage == S::STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (ok) {
        if constexpr (PAIR)
          umma_commit_pair_mask(tfull_bar, mask);
        else
          umma_commit(tfull_bar);
      }
    }
  } else {
    // ------------------------------------------------------------ accumulator -> this CTA's shared memory
    const int quarter = warp & 3;
    if (mbar_wait_bounded(tfull_bar, 0, abort_flag, err_word, DEV_ERR_TMEM_FULL_TIMEOUT, GEMM_WAIT_LIMIT_NS)) {
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
      const uint32_t dst = smem_base + (quarter * 32 + lane) * S::RED_PITCH;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t acc[32];
        tmem_ld_32x32(taddr + c * 32, acc);
        tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 8; ++v)
          st_shared_v4(dst + c * 128 + v * 16, acc[4 * v], acc[4 * v + 1], acc[4 * v + 2], acc[4 * v + 3]);
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before shared memory is reused or released.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  cluster_sync_all();   // all partial sums of the tile are in place

  // ------------------------------------------------------------ this CTA's share of the rows, all slices in order
  const int rows = 128 / slices;
  constexpr int VEC = BN / 8;
  for (int i = threadIdx.x; i < rows * VEC; i += GEMM_THREADS) {
    const int r = slice * rows + i / VEC, c = (i % VEC) * 8;
    const int row = row0 + r, col = tn * BN + c;
    if (row >= shape.M || col >= shape.N) continue;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const uint32_t at = smem_base + r * S::RED_PITCH + c * 4;
#pragma unroll 4
    for (int p = 0; p < slices; ++p) {
      const uint32_t peer = map_to_cta(at, PAIR ? 2u * p + half : static_cast<uint32_t>(p));
      const float4 x = ld_cluster_f4(peer), y = ld_cluster_f4(peer + 16);
      f[0] += x.x; f[1] += x.y; f[2] += x.z; f[3] += x.w;
      f[4] += y.x; f[5] += y.y; f[6] += y.z; f[7] += y.w;
    }
    OutT* dst = C + static_cast<int64_t>(row) * ldc + col;
    const int n = min(8, shape.N - col);
    if (accumulate) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n) f[j] += static_cast<float>(dst[j]);
    }
    if (n == 8) {
      if constexpr (sizeof(OutT) == 2) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                                                    pack_bf16x2(f[6], f[7]));
      } else {
        reinterpret_cast<float4*>(dst)[0] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4*>(dst)[1] = make_float4(f[4], f[5], f[6], f[7]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < n) dst[j] = static_cast<OutT>(f[j]);
    }
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  cluster_sync_all();   // the peers have read this CTA's sums
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR)
      tmem_dealloc_pair(tmem_base, BN);
    else
      tmem_dealloc(tmem_base, BN);
  }
}

}  // namespace b200

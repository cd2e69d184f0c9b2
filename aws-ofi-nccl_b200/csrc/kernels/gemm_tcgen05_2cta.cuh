// Persistent bf16 GEMM mainloop on CTA pairs: one 256 x 256 (or 256 x 128) output tile per cluster
// of two CTAs, computed by `tcgen05.mma.cta_group::2` issued from the even ("leader") CTA.
//
// Each CTA loads its own 128 rows of A and its own half of the B tile (32 KB per 64-deep k-block
// instead of the 48 KB a lone CTA needs for a 128 x 256 tile), so six stages fit where the one-CTA
// kernel has four (eight instead of six for the narrow tile) and the L2 traffic per flop drops by
// a third. Each CTA's TMEM holds its
// 128 rows of the accumulator (all 256 columns, double-buffered) and its own epilogue warps store
// them.
//
// Synchronisation (all barriers are mbarriers in shared memory, every wait is bounded):
//   full[s]   leader only : both CTAs' TMA loads report their bytes here
//   empty[s]  both CTAs   : the leader's tcgen05.commit arrives on both (multicast commit)
//   tfull[b]  both CTAs   : accumulator b complete (multicast commit)
//   tempty[b] leader only : all epilogue warps of the pair have drained accumulator b
// None of the loads uses cluster multicast; only tcgen05.commit does.
#pragma once
#include "gemm_tcgen05.cuh"

namespace b200 {

// BN: 256 or 128 output columns per cluster tile; EW: epilogue warps of a CTA, 4 or 8
template <int BN, int EW = 4>
struct Gemm2Smem {
  static constexpr int A_BYTES = 128 * GEMM_BK * 2;
  static constexpr int B_BYTES = (BN / 2) * GEMM_BK * 2;   // this CTA's half of the B tile
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? (EW == 8 ? 5 : 6) : (EW == 8 ? 6 : 8);
  static constexpr int THREADS = 64 + 32 * EW;
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = 1024 + STAGES * STAGE_BYTES + BAR_BYTES;
  static constexpr int EPI_OFF = STAGES * STAGE_BYTES + 1024;
  static constexpr int TOTAL_EPI = 1024 + EPI_OFF + EW * GEMM_EPI_WARP_BYTES;
  static_assert(EW == 4 || EW == 8, "one or two epilogue warps per quarter of the accumulator's rows");
  static_assert(TOTAL_EPI <= 232448, "more than a CTA's shared memory");
};
constexpr int GEMM2_BM = 256;  // rows per cluster tile

// What a pair works on at a time: columns [col0, col0 + width) of tile row tm. The last, partly filled wave
// of tiles leaves pairs idle; where halving its tiles fills them (GemmShape::halve_from is then the number of
// tiles in whole waves) it takes the time of a narrow wave instead of a wide one.
struct TileSpan {
  int tm, tn, col0, width;
};
__device__ __forceinline__ int tile_items(const GemmShape& s) {
  const int tiles = s.tiles_m * s.tiles_n;
  return tiles <= s.halve_from ? tiles : 2 * tiles - s.halve_from;
}
template <int BN>
__device__ __forceinline__ TileSpan tile_span(const GemmShape& s, int item) {
  TileSpan t;
  const int bn = s.bn ? s.bn : BN;
  const bool half = item >= s.halve_from;
  const int beyond = item - s.halve_from;
  tile_coords(s, half ? s.halve_from + (beyond >> 1) : item, t.tm, t.tn);
  t.col0 = t.tn * bn + (half && (beyond & 1) ? bn / 2 : 0);
  t.width = half ? bn / 2 : bn;
  return t;
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Address of the same shared-memory location in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// Hands tensor memory back: what it orders are tcgen05 operations, by the tcgen05 fences on both sides, and no other
// memory. As a release at cluster scope it waited for everything that the warp had stored, 1600 clocks a tile: the
// weight gradient 4096 x 14336 of 128 tokens (two k-blocks per tile) takes 37 us, 47 with it (39
// and 60 in narrow tiles).
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Tiled load into this CTA's shared memory whose byte count is reported to a barrier of the pair's
// leader (`bar_cluster` is a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst_smem, const CUtensorMap* m, int x, int y,
                                                 uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// fp8 (e4m3 / e5m2) operands: kind::f8f6f4, K = 32 per instruction.
__device__ __forceinline__ void umma_f8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on `bar` (same offset) in both CTAs of the pair once every MMA issued so far has finished.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}

// Launch with cluster dimension (2,1,1), Gemm2Smem<BN, EW>::THREADS threads, its TOTAL (+ epilogue extras)
// bytes of dynamic shared memory and an even grid. shape.tiles_m counts 256-row tiles here.
// The gate and the epilogue hooks (tile_begin / tile_end) are called with the index of this CTA's
// 128-row tile (2 * pair tile + rank in the pair), so gates and epilogues written for the one-CTA
// mainloop work unchanged. shape.cta_first / num_ctas (both even) restrict the GEMM to a part of
// the grid.
// A tile is 256 rows and BN columns, or shape.bn of them (a multiple of 32, at most BN); its columns and
// those of the halves of the last wave come from tile_span.
// FP8: both operands are 1-byte e4m3, K-major only; a k-block is then 128 elements (the same 128
// bytes per row, so stages, swizzle and descriptors do not change) and one MMA covers K = 32.
template <int BN, bool A_MN, bool B_MN, class Epilogue, class LoadGate, bool FP8 = false, int EW = 4>
__device__ __forceinline__ void gemm_mainloop_2cta(const CUtensorMap* tmA, const CUtensorMap* tmB, GemmShape shape,
                                                   Epilogue& epi, LoadGate& gate, int* err_word, uint8_t* smem_raw) {
  using S = Gemm2Smem<BN, EW>;
  static_assert(BN == 128 || BN == 256, "cluster tile is 256 x 128 or 256 x 256");
  static_assert(!FP8 || (!A_MN && !B_MN), "fp8 operands are K-major");
  constexpr int BK_ELEMS = FP8 ? 2 * GEMM_BK : GEMM_BK;   // elements per 128-byte row of a stage
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();   // 0 = leader
  const bool leader = rank == 0;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + S::STAGES * S::STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (S::STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * S::STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * S::STAGES + 2 + b); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * S::STAGES + 4);
  volatile int* abort_flag =
      reinterpret_cast<volatile int*>(smem_raw + (bar_base - smem_u32(smem_raw)) + 8u * (2 * S::STAGES + 4) + 8);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), 2 * EW);
    }
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(tmA);
    tma_prefetch_desc(tmB);
  }
  constexpr uint32_t TMEM_COLS = 2 * BN;
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - smem_u32(smem_raw)));
  grid_wait();   // the operands may be the kernel before's

  const int num_items = tile_items(shape);
  const int num_kb = (shape.K + BK_ELEMS - 1) / BK_ELEMS;
  const int pair_id = (static_cast<int>(blockIdx.x) - shape.cta_first) >> 1;
  const int pair_stride = (shape.num_ctas > 0 ? shape.num_ctas : static_cast<int>(gridDim.x)) >> 1;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const int box = shape.b_box ? shape.b_box : BN / 2;
      for (int item = pair_id; item < num_items && ok; item += pair_stride) {
        const TileSpan t = tile_span<BN>(shape, item);
        const int half = t.width >> 1;
        const int row0 = t.tm * GEMM2_BM + static_cast<int>(rank) * 128;   // this CTA's rows of A
        const int col0 = shape.b_second ? (t.col0 >> 1) + static_cast<int>(rank) * shape.b_second   // this CTA's half of B
                                        : t.col0 + static_cast<int>(rank) * half;
        const int b_boxes = B_MN ? (half + 63) / 64 : half / box;
        const uint32_t pair_bytes = 2 * (S::A_BYTES + b_boxes * (B_MN ? 64 : box) * 128);
        if (!gate.wait_tile(2 * t.tm + static_cast<int>(rank), t.tn, abort_flag, err_word)) break;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1, abort_flag, err_word, DEV_ERR_EMPTY_BAR_TIMEOUT,
                                 GEMM_WAIT_LIMIT_NS)) {
            ok = false;
            break;
          }
          const uint32_t a_dst = smem_base + stage * S::STAGE_BYTES;
          const uint32_t b_dst = a_dst + S::A_BYTES;
          const uint32_t bar = map_to_cta(full_bar(stage), 0);
          if (leader) mbar_expect_tx(full_bar(stage), pair_bytes);  // both CTAs' bytes
          if constexpr (!A_MN) {
            tma_load_2d_pair(a_dst, tmA, kb * BK_ELEMS, row0, bar);
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) tma_load_2d_pair(a_dst + j * 8192, tmA, row0 + j * 64, kb * GEMM_BK, bar);
          }
          if constexpr (!B_MN) {
            for (int j = 0; j < b_boxes; ++j) tma_load_2d_pair(b_dst + j * box * 128, tmB, kb * BK_ELEMS, col0 + j * box, bar);
          } else {
            for (int j = 0; j < b_boxes; ++j) tma_load_2d_pair(b_dst + j * 8192, tmB, col0 + j * 64, kb * GEMM_BK, bar);
          }
          if (++stage == S::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!shape.keep_room) grid_release();   // what is left are the last stages' products and the last stores
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one_sync()) {
      // operand format field: 1 = bf16 for kind::f16, 0 = e4m3 for kind::f8f6f4
      int stage = 0;
      uint32_t phase = 0;
      int acc_buf = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int item = pair_id; item < num_items && ok; item += pair_stride) {
        const uint32_t idesc = make_instr_desc(FP8 ? 0 : 1, FP8 ? 0 : 1, GEMM2_BM, tile_span<BN>(shape, item).width, A_MN ? 1 : 0, B_MN ? 1 : 0);
        if (!mbar_wait_bounded(tempty_bar(acc_buf), acc_phase ^ 1, abort_flag, err_word, DEV_ERR_TMEM_EMPTY_TIMEOUT,
                               GEMM_WAIT_LIMIT_NS))
          break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc_buf * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(full_bar(stage), phase, abort_flag, err_word, DEV_ERR_FULL_BAR_TIMEOUT,
                                 GEMM_WAIT_LIMIT_NS)) {
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
            if constexpr (FP8)
              umma_f8_pair(d_tmem, adesc, bdesc, idesc, (kb | k) != 0 ? 1u : 0u);
            else
              umma_f16_pair(d_tmem, adesc, bdesc, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit_pair(empty_bar(stage));  // frees the stage in both CTAs once these MMAs have read it
          if (++stage == S::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(tfull_bar(acc_buf));  // accumulator complete -> both epilogues
        acc_buf ^= 1;
        if (acc_buf == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps from 2 on, both CTAs)
    const int quarter = warp & 3;
    // with eight warps the two of a quarter take every second 64 columns each
    constexpr int STEP = 64 * (EW / 4);
    const int first = EW == 4 ? 0 : 64 * ((warp - 2) >> 2);
    int acc_buf = 0;
    uint32_t acc_phase = 0;
    for (int item = pair_id; item < num_items; item += pair_stride) {
      const TileSpan t = tile_span<BN>(shape, item);
      if constexpr (Epilogue::kAhead)
        epi.tile_ahead(t.tm * GEMM2_BM + static_cast<int>(rank) * 128 + quarter * 32, t.col0 + first, shape, abort_flag, err_word);
      if (!mbar_wait_bounded(tfull_bar(acc_buf), acc_phase, abort_flag, err_word, DEV_ERR_TMEM_FULL_TIMEOUT,
                             GEMM_WAIT_LIMIT_NS))
        break;
      tc_fence_after();
      epi.tile_begin(2 * t.tm + static_cast<int>(rank), t.tn);
      const int row = t.tm * GEMM2_BM + static_cast<int>(rank) * 128 + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc_buf * BN;
      if constexpr (Epilogue::kSplit) {
        const int half = t.width >> 1;
#pragma unroll 1
        for (int c = first; c < half; c += STEP) {
          uint32_t a[32], b[32];
          tmem_ld_32x32(taddr + c, a);
          tmem_ld_32x32(taddr + half + c, b);
          tmem_ld_wait();
          epi.template part<0>(a, b);
          tmem_ld_32x32(taddr + c + 32, a);
          tmem_ld_32x32(taddr + half + c + 32, b);
          tmem_ld_wait();
          epi.template part<1>(a, b);
          epi.store(row, (t.col0 >> 1) + c, shape);
        }
      } else if constexpr (Epilogue::kPair) {
#pragma unroll 1
        for (int c = first; c < t.width; c += STEP) {
          uint32_t acc0[32], acc1[32];
          tmem_ld_32x32(taddr + c, acc0);
          tmem_ld_32x32(taddr + c + 32, acc1);
          tmem_ld_wait();
          epi(row, t.col0 + c, acc0, acc1, shape, t.width - c);
        }
      } else {
        static_assert(EW == 4 || Epilogue::kPair || Epilogue::kSplit, "two warps share a quarter 64 columns at a time");
#pragma unroll 1
        for (int c = 0; c < t.width; c += 32) {
          uint32_t acc[32];
          tmem_ld_32x32(taddr + c, acc);
          tmem_ld_wait();
          epi(row, t.col0 + c, acc, shape);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_cta(tempty_bar(acc_buf), 0));
      epi.tile_end(2 * t.tm + static_cast<int>(rank), t.tn);
      acc_buf ^= 1;
      if (acc_buf == 0) acc_phase ^= 1;
    }
    epi.drain();
  }

  // ------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before shared memory is released.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
  cluster_sync_all();   // neither CTA leaves while the other may still signal its barriers or read its tiles
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

}  // namespace b200

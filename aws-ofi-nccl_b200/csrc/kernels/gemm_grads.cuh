// Both gradients of a linear layer y = x W^T in one persistent kernel on CTA pairs:
//
//   dx[M,K] = dy[M,N] W[N,K]        dw[N,K] (+)= dy[M,N]^T x[M,K]
//
// Each product alone leaves pairs idle in its last wave of tiles, and a small one is little but a launch; together they
// share the waves. The product whose tiles take longer goes first; pairs that get one tile less of it are given `fill`
// tiles of the other one before the rest is dealt out, so that all pairs finish within a short tile of each other. Both
// take B from rows of K columns (W, x), and differ in A: rows of dy, or its columns. Barriers, stages and epilogue are those
// of gemm_mainloop_2cta; no load is multicast and every wait is bounded.
#pragma once
#include "gemm_epilogues.cuh"
#include "gemm_tcgen05_2cta.cuh"

namespace b200 {

constexpr int GRADS_BN = 256;   // widest tile; GemmShape::bn has the width

struct GradsArgs {
  GemmShape shape[2];         // dx, dw
  __nv_bfloat16* out[2];
  int64_t ld_out[2];
  int accumulate;             // dw only
  int first;                  // the product whose tiles come first
  int fill;
};

// The tiles of one pair, in order: which product, and which tile of it.
struct GradsWalk {
  int first, pairs, n_first, n_second, fill_pairs, fill, base, offset, at, step;
  int product, tile;
  __device__ __forceinline__ GradsWalk(const GradsArgs& a) {
    first = a.first;
    pairs = static_cast<int>(gridDim.x) >> 1;
    n_first = a.shape[first].tiles_m * a.shape[first].tiles_n;
    n_second = a.shape[first ^ 1].tiles_m * a.shape[first ^ 1].tiles_n;
    const int longer = n_first % pairs;   // pairs with one tile more of the first product
    const int pair = static_cast<int>(blockIdx.x) >> 1;
    fill_pairs = longer ? pairs - longer : 0;
    base = min(n_second, fill_pairs * a.fill);
    // this pair's place among those that are filled, none if it has the longer share
    fill = longer && pair >= longer ? a.fill : 0;
    at = pair;
    step = 0;
    offset = pair - longer;
  }
  __device__ __forceinline__ bool next() {
    if (at < n_first) {
      product = first;
      tile = at;
      at += pairs;
      return true;
    }
    product = first ^ 1;
    while (step < fill) {
      tile = offset + fill_pairs * step++;
      if (tile < base) return true;
    }
    tile = base + (static_cast<int>(blockIdx.x) >> 1) + (step++ - fill) * pairs;
    return tile < n_second;
  }
};

template <int EW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(Gemm2Smem<GRADS_BN, EW>::THREADS, 1)
    gemm_grads_kernel(const __grid_constant__ CUtensorMap tmDyRows, const __grid_constant__ CUtensorMap tmDyCols,
                      const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                      const __grid_constant__ CUtensorMap tmDx, const __grid_constant__ CUtensorMap tmDw,
                      const __grid_constant__ GradsArgs args, int* err_word) {
  using S = Gemm2Smem<GRADS_BN, EW>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
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
    tma_prefetch_desc(&tmDyRows);
    tma_prefetch_desc(&tmDyCols);
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  constexpr uint32_t TMEM_COLS = 2 * GRADS_BN;
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
  GradsWalk walk(args);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      while (ok && walk.next()) {
        const bool dw = walk.product == 1;
        const GemmShape& shape = args.shape[walk.product];
        int tm, tn;
        tile_coords(shape, walk.tile, tm, tn);
        const int half = shape.bn >> 1;
        const int row0 = tm * GEMM2_BM + static_cast<int>(rank) * 128;
        const int col0 = tn * shape.bn + static_cast<int>(rank) * half;
        const int b_boxes = (half + 63) / 64;
        const uint32_t pair_bytes = 2 * (S::A_BYTES + b_boxes * 8192);
        const CUtensorMap* tmB = dw ? &tmX : &tmW;
        const int num_kb = (shape.K + GEMM_BK - 1) / GEMM_BK;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1, abort_flag, err_word, DEV_ERR_EMPTY_BAR_TIMEOUT, GEMM_WAIT_LIMIT_NS)) {
            ok = false;
            break;
          }
          const uint32_t a_dst = smem_base + stage * S::STAGE_BYTES;
          const uint32_t b_dst = a_dst + S::A_BYTES;
          const uint32_t bar = map_to_cta(full_bar(stage), 0);
          if (leader) mbar_expect_tx(full_bar(stage), pair_bytes);  // both CTAs' bytes
          if (!dw) {
            tma_load_2d_pair(a_dst, &tmDyRows, kb * GEMM_BK, row0, bar);
          } else {
            tma_load_2d_pair(a_dst, &tmDyCols, row0, kb * GEMM_BK, bar);
            tma_load_2d_pair(a_dst + 8192, &tmDyCols, row0 + 64, kb * GEMM_BK, bar);
          }
          for (int j = 0; j < b_boxes; ++j) tma_load_2d_pair(b_dst + j * 8192, tmB, col0 + j * 64, kb * GEMM_BK, bar);
          if (++stage == S::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      grid_release();   // what is left are the last stages' products and the last stores
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader && elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      int acc_buf = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      while (ok && walk.next()) {
        const bool dw = walk.product == 1;
        const GemmShape& shape = args.shape[walk.product];
        const uint32_t idesc = make_instr_desc(1, 1, GEMM2_BM, shape.bn, dw ? 1 : 0, 1);
        const int num_kb = (shape.K + GEMM_BK - 1) / GEMM_BK;
        if (!mbar_wait_bounded(tempty_bar(acc_buf), acc_phase ^ 1, abort_flag, err_word, DEV_ERR_TMEM_EMPTY_TIMEOUT, GEMM_WAIT_LIMIT_NS))
          break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc_buf * GRADS_BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(full_bar(stage), phase, abort_flag, err_word, DEV_ERR_FULL_BAR_TIMEOUT, GEMM_WAIT_LIMIT_NS)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_src = smem_base + stage * S::STAGE_BYTES;
          const uint32_t b_src = a_src + S::A_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k) {
            const uint64_t adesc = dw ? make_smem_desc_sw128(a_src + k * 2048, 8192, 1024) : make_smem_desc_sw128(a_src + k * 32, 16, 1024);
            umma_f16_pair(d_tmem, adesc, make_smem_desc_sw128(b_src + k * 2048, 8192, 1024), idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit_pair(empty_bar(stage));
          if (++stage == S::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (ok) umma_commit_pair(tfull_bar(acc_buf));
        acc_buf ^= 1;
        if (acc_buf == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps from 2 on, both CTAs)
    const int quarter = warp & 3;
    constexpr int STEP = 64 * (EW / 4);
    const int first = EW == 4 ? 0 : 64 * ((warp - 2) >> 2);
    StoreEpilogue<__nv_bfloat16> epi{&tmDx, nullptr, 0, 0, {}};
    epi.slab.init(smem_raw, S::EPI_OFF);
    int acc_buf = 0;
    uint32_t acc_phase = 0;
    while (walk.next()) {
      const GemmShape& shape = args.shape[walk.product];
      int tm, tn;
      tile_coords(shape, walk.tile, tm, tn);
      epi.tmC = walk.product ? &tmDw : &tmDx;
      epi.C = args.out[walk.product];
      epi.ldc = args.ld_out[walk.product];
      epi.accumulate = walk.product && args.accumulate;
      if (!mbar_wait_bounded(tfull_bar(acc_buf), acc_phase, abort_flag, err_word, DEV_ERR_TMEM_FULL_TIMEOUT, GEMM_WAIT_LIMIT_NS)) break;
      tc_fence_after();
      const int row = tm * GEMM2_BM + static_cast<int>(rank) * 128 + quarter * 32 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc_buf * GRADS_BN;
#pragma unroll 1
      for (int c = first; c < shape.bn; c += STEP) {
        uint32_t acc0[32], acc1[32];
        tmem_ld_32x32(taddr + c, acc0);
        tmem_ld_32x32(taddr + c + 32, acc1);
        tmem_ld_wait();
        epi(row, tn * shape.bn + c, acc0, acc1, shape, shape.bn - c);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_cta(tempty_bar(acc_buf), 0));
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

// Softmax cross-entropy of wide rows, forward and backward: a CTA's rows stream through its shared memory, one after the other.
//
// A row is read twice, for its maximum and sum and for its gradient, and the second time most of it is still in the ring of
// shared memory that it came through; what is not comes from L2. A warp of its own issues bulk copies: chunks of the next rows
// are on their way while the present row's gradient is computed and stored. 2048 x 128256 takes 195 us (5.4 TB/s), 247 in two passes
// of a row per CTA whose threads have one vector in flight each (cross_entropy_two_pass_kernel); 2048 x 32776 71 and 84, 148 x 65544
// 11.8 and 14.9. What bounds it is memory, 160 us, and the exponential unit, two per element: 117 us at 1.9 GHz, and more than
// memory at the clocks that products beside it leave. 24 warps of four vectors each: 16 of four take 207 us, 24 of two 205, 28 of one 236.
//
// Chunks are loaded into the slots of the ring in turn, and let go in the same order: of a row of C chunks the first C - CES_SLOTS are
// let go once they have been summed, the others are kept for the second pass, where the first come again after them. `full` of a
// slot: its load has landed; `done`: every warp has read what it needs of it. Every wait is bounded; a CTA that gives up goes on
// without waiting.
#pragma once
#include "cross_entropy_math.cuh"
#include "sm100_common.cuh"

namespace b200 {

constexpr int CES_WARPS = 24;                     // that compute
constexpr int CES_THREADS = 32 * (CES_WARPS + 1);
constexpr int CES_VPT = 4;                        // 16-byte vectors of a chunk for every thread
constexpr int CES_CHUNK = CES_VPT * 32 * CES_WARPS;
constexpr int CES_SLOT_BYTES = CES_CHUNK * 16;
constexpr int CES_SLOTS = 4;
constexpr int CES_SMEM = 1024 + CES_SLOTS * CES_SLOT_BYTES;
constexpr uint64_t CES_WAIT_LIMIT_NS = 2000000000ull;
static_assert(CES_SMEM <= 232448, "more than a CTA's shared memory");

// The chunks of this CTA's rows in the order in which they are loaded.
struct CesWalk {
  int chunks, again;   // of a row: all, and those that are loaded a second time
  int at;              // of the row's chunks + again loads
  int64_t row, step;
  __device__ __forceinline__ CesWalk(int nvec) {
    chunks = (nvec + CES_CHUNK - 1) / CES_CHUNK;
    again = chunks > CES_SLOTS ? chunks - CES_SLOTS : 0;
    at = 0;
    row = blockIdx.x;
    step = gridDim.x;
  }
  __device__ __forceinline__ int chunk() const { return at < chunks ? at : at - chunks; }
  __device__ __forceinline__ void next() {
    if (++at == chunks + again) {
      at = 0;
      row += step;
    }
  }
};

__global__ void __launch_bounds__(CES_THREADS, 1)
    cross_entropy_stream_kernel(bf16* logits, const int64_t* targets, float* loss, int T, int V, int64_t ld, float grad_scale,
                                int* err_word) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ alignas(8) uint64_t bars[2 * CES_SLOTS];
  __shared__ float2 parts[2][CES_WARPS];   // maximum and sum of a warp's elements, for rows in turn
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ring = (smem_u32(smem_raw) + 127u) & ~127u;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto done_bar = [&](int s) { return bar0 + 8u * (CES_SLOTS + s); };
  if (threadIdx.x == 0) {
    for (int s = 0; s < CES_SLOTS; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(done_bar(s), CES_WARPS);
    }
    abort_word = 0;
    fence_barrier_init();
  }
  __syncthreads();
  grid_wait();
  const int nvec = V / 8;
  auto wait = [&](uint32_t bar, uint32_t parity, int code) {
    mbar_wait_bounded(bar, parity, abort_flag, err_word, code, CES_WAIT_LIMIT_NS);
  };

  if (warp == CES_WARPS) {
    // ------------------------------------------------------------ copies
    if (lane == 0) {
      int slot = 0;
      uint32_t phase = 1;   // of a slot that has not been used
      for (CesWalk in(nvec); in.row < T; in.next()) {
        wait(done_bar(slot), phase, DEV_ERR_EMPTY_BAR_TIMEOUT);
        const int c = in.chunk();
        const uint32_t bytes = static_cast<uint32_t>(min(CES_CHUNK, nvec - c * CES_CHUNK)) * 16u;
        mbar_expect_tx(full_bar(slot), bytes);
        bulk_load(ring + slot * CES_SLOT_BYTES, logits + in.row * ld + static_cast<int64_t>(c) * CES_CHUNK * 8, bytes, full_bar(slot));
        if (++slot == CES_SLOTS) {
          slot = 0;
          phase ^= 1;
        }
      }
      grid_release();
    }
  } else {
    // ------------------------------------------------------------ sums and gradients
    int slot = 0;
    uint32_t phase = 0;
    auto advance = [&]() {
      if (++slot == CES_SLOTS) {
        slot = 0;
        phase ^= 1;
      }
    };
    const CesWalk walk(nvec);
    const int first = static_cast<int>(threadIdx.x);   // vector of a chunk; the others follow 32 * CES_WARPS apart
    Bf16x8 x[CES_VPT];
    auto read = [&](int n) {
#pragma unroll
      for (int h = 0; h < CES_VPT; ++h) {
        uint32_t r[4];
        if (first + h * 32 * CES_WARPS < n) {
          ld_shared_v4(ring + slot * CES_SLOT_BYTES + (first + h * 32 * CES_WARPS) * 16, r);
          x[h] = *reinterpret_cast<const Bf16x8*>(r);
        }
      }
    };
    auto let_go = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(done_bar(slot));
    };
    int turn = 0;
    for (int64_t row = walk.row; row < T; row += walk.step, turn ^= 1) {
      bf16* lr = logits + row * ld;
      const int64_t tgt = targets[row];
      const bool counts = tgt >= 0 && tgt < V;   // other rows are ignored: no loss, zeros for a gradient whatever the logits hold
      float lt = 0.f;
      if (threadIdx.x == 0 && counts) lt = __bfloat162float(lr[tgt]);   // before anything is overwritten
      const int tail = nvec * 8 + static_cast<int>(threadIdx.x);       // the last elements are less than a vector
      const float ft = tail < V ? __bfloat162float(lr[tail]) : -INFINITY;
      // ---- maximum, and sum of the exponentials relative to it
      float m = -FLT_MAX, c = 0.f, s = 0.f;
      auto raise = [&](float to) {
        s *= exp_share(m, to);
        m = to;
        c = exp_base(m);
      };
      const int slot0 = slot;
      const uint32_t phase0 = phase;
      for (int k = 0; k < walk.chunks; ++k) {
        wait(full_bar(slot), phase, DEV_ERR_FULL_BAR_TIMEOUT);
        const int n = min(CES_CHUNK, nvec - k * CES_CHUNK);
        read(n);
        if (k < walk.again) let_go();
        float lm = -FLT_MAX;
#pragma unroll
        for (int h = 0; h < CES_VPT; ++h)
          if (first + h * 32 * CES_WARPS < n) lm = fmaxf(lm, max8(x[h]));
        if (lm > m) raise(lm);
        if (!huge_max(m)) {
          float part[CES_VPT];
#pragma unroll
          for (int h = 0; h < CES_VPT; ++h) part[h] = first + h * 32 * CES_WARPS < n ? exp_sum8(x[h], c) : 0.f;
#pragma unroll
          for (int h = 0; h < CES_VPT; ++h) s += part[h];
        } else {
#pragma unroll
          for (int h = 0; h < CES_VPT; ++h)
            if (first + h * 32 * CES_WARPS < n) s += exp_sum8_huge(*reinterpret_cast<const uint4*>(&x[h]), m);
        }
        advance();
      }
      if (tail < V) {
        if (ft > m) raise(ft);
        s += huge_max(m) ? __expf(ft - m) : exp2_approx(fmaf(ft, LOG2E, -c));
      }
      // ---- over the warp, then over the CTA
      float wm = m;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) wm = fmaxf(wm, __shfl_xor_sync(0xffffffffu, wm, o));
      s *= exp_share(m, wm);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) parts[turn][warp] = make_float2(wm, s);
      asm volatile("bar.sync 1, %0;" ::"n"(32 * CES_WARPS) : "memory");
      const float2 p = lane < CES_WARPS ? parts[turn][lane] : make_float2(-FLT_MAX, 0.f);
      float gm = p.x;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) gm = fmaxf(gm, __shfl_xor_sync(0xffffffffu, gm, o));
      float gs = p.y * exp_share(p.x, gm);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, o);
      if (threadIdx.x == 0) loss[row] = counts ? ce_loss(gm, gs, lt) : 0.f;
      // ---- gradients, in the order in which the chunks lie in the ring
      const float inv = grad_scale / gs;
      const bool huge = huge_max(gm), special = !counts || huge || small_powers_count(inv);
      c = exp_base(gm);
      if (walk.again == 0) {
        slot = slot0;
        phase = phase0;
      } else {   // kept: all slots, the oldest of which comes next
        phase ^= 1;
      }
      for (int i = 0; i < walk.chunks; ++i) {
        const bool kept = i < walk.chunks - walk.again;
        const int k = kept ? walk.again + i : i - (walk.chunks - walk.again);
        if (!kept) wait(full_bar(slot), phase, DEV_ERR_FULL_BAR_TIMEOUT);
        const int n = min(CES_CHUNK, nvec - k * CES_CHUNK);
        read(n);
        let_go();
        const int own = counts ? static_cast<int>(tgt) - (k * CES_CHUNK + first) * 8 : -1;   // the target's place from this thread's first element on
#pragma unroll
        for (int h = 0; h < CES_VPT; ++h) {
          const int v = first + h * 32 * CES_WARPS;
          if (v >= n) break;
          const int at = own - h * 256 * CES_WARPS;
          uint4 o = make_uint4(0, 0, 0, 0);
          if (!special) {
            const Bf16x8 g = ce_gradient8<false>(x[h], c, inv, at, grad_scale);
            o = *reinterpret_cast<const uint4*>(&g);
          } else if (counts) {
            o = ce_gradient8_special(*reinterpret_cast<const uint4*>(&x[h]), gm, inv, at, grad_scale);
          }
          *reinterpret_cast<uint4*>(lr + static_cast<int64_t>(k * CES_CHUNK + v) * 8) = o;
        }
        advance();
      }
      if (tail < V) {
        float f = (huge ? __expf(ft - gm) : exp2_approx(fmaf(ft, LOG2E, -c))) * inv;
        if (tail == tgt) f -= grad_scale;
        lr[tail] = __float2bfloat16(counts ? f : 0.f);
      }
    }
  }
  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before shared memory is released.
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
  }
}

}  // namespace b200

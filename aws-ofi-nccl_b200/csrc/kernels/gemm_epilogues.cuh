// Epilogue functors for the tcgen05 GEMM mainloops: plain store (bf16 / fp32, optional accumulate),
// the scaled store of the fp8 product, and SwiGLU and its gradient in the products of an MLP.
//
// A thread holds one accumulator row, so storing from registers writes 16 bytes to each of 32 rows
// per instruction: half a sector at a time, 32 lines in flight per warp, and the epilogue of a short
// K loop costs more than its products. All functors therefore turn their 32 rows x 64 columns through
// shared memory (16-byte chunks XOR-swizzled by row: no bank conflict) and hand the slab to a TMA
// store, which writes whole 128-byte row segments, clips the edges of C and leaves the warp free for
// the next slab while it drains. It clips a row at 16 bytes: a width that is no multiple of that has
// its last elements stored from registers (store_row). Kernel times from register stores to TMA stores: the weight gradient
// 4096 x 14336 of 128 tokens 95 -> 38 us (117 MB stored), the fp8 product 4096 x 14336 x 4096
// 192 -> 158 us, one 256 x 768 x 256 product 12 -> 7 us.
#pragma once
#include "gemm_tcgen05.cuh"
#include "swiglu_math.cuh"

namespace b200 {

// One epilogue warp's staging area (GEMM_EPI_WARP_BYTES, 1024-byte aligned): two 4 KiB buffers, the
// older of which is free again once all but the last store have read theirs.
struct SlabStore {
  uint32_t buf;
  uint32_t which;
  // Shared memory of this thread's warp; `tiles_end` is the end of the operand stages, relative to
  // the aligned base of the dynamic shared memory, plus room for the barriers (EPI_OFF).
  __device__ __forceinline__ void init(uint8_t* smem_raw, uint32_t epi_off) {
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t warp = threadIdx.x >> 5;
    buf = base + epi_off + (warp >= 2 ? warp - 2 : 0) * GEMM_EPI_WARP_BYTES;
    which = 0;
  }
  __device__ __forceinline__ void drain() {
    if ((threadIdx.x & 31) == 0) tma_store_wait<0>();
  }
  // The buffer that the next put128 fills, free of the store before the last.
  __device__ __forceinline__ uint32_t next() {
    if ((threadIdx.x & 31) == 0) tma_store_wait_read<1>();
    __syncwarp();
    return buf + which * 4096u;
  }
  // 32 rows x 128 bytes; lane i passes its row as 32 words. Returns where its row lies in shared memory
  // (16-byte chunk j at j ^ (lane & 7)); without `store` it only goes there.
  __device__ __forceinline__ uint32_t put128(const CUtensorMap* tm, int x, int y, const uint32_t (&w)[32], bool store) {
    const int lane = threadIdx.x & 31;
    const uint32_t slab = next();
#pragma unroll
    for (int j = 0; j < 8; ++j)
      st_shared_v4(slab + lane * 128 + ((j ^ (lane & 7)) << 4), w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (store) tma_store_2d(tm, slab, x, y);
      tma_store_commit();
    }
    which ^= 1u;
    return slab + lane * 128;
  }
};

// The columns that TMA stores: whole 16-byte vectors.
template <typename OutT>
__host__ __device__ __forceinline__ int whole_vectors(int N) {
  return N & ~static_cast<int>(16 / sizeof(OutT) - 1);
}

// The elements of one row from column nv on, less than 16 bytes; `chunk` is where they lie in shared memory.
// A call of its own, out of the loop that every other width runs.
template <typename OutT>
__device__ __noinline__ void store_tail(uint32_t chunk, OutT* dst, int n) {
  uint32_t v[4];
  ld_shared_v4(chunk, v);
#pragma unroll
  for (int e = 0; e < static_cast<int>(16 / sizeof(OutT)) - 1; ++e) {
    if (e >= n) break;
    if constexpr (sizeof(OutT) == 2)
      reinterpret_cast<uint16_t*>(dst)[e] = static_cast<uint16_t>(v[e / 2] >> (16 * (e % 2)));
    else
      reinterpret_cast<uint32_t*>(dst)[e] = v[e];
  }
}

// The first 32 columns of a slab of 16-bit elements that lies in shared memory at `slab` -> C: what a tile holds of
// its last 64 columns where its width ends inside them (a TMA store would write the next tile's columns too).
template <typename OutT>
__device__ __noinline__ void store_half_slab(uint32_t slab, OutT* C, int64_t ldc, int row0, int M) {
  const int lane = threadIdx.x & 31, v = lane & 3;
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * 8 + (lane >> 2);
    uint32_t x[4];
    ld_shared_v4(slab + r * 128 + ((v ^ (r & 7)) << 4), x);
    if (row0 + r < M) *reinterpret_cast<uint4*>(C + static_cast<int64_t>(row0 + r) * ldc + v * 8) = make_uint4(x[0], x[1], x[2], x[3]);
  }
  __syncwarp();
}

// A warp's 32 rows from `row0` on, 128 bytes of each from column col0 on (w: this lane's row), of which a bf16
// tile may hold the first 32 columns only (left < 64). The map of C ends at whole_vectors(N); what is left of
// a row beyond it each lane stores itself.
template <typename OutT>
__device__ __forceinline__ void store_row(SlabStore& slab, const CUtensorMap* tmC, OutT* C, int64_t ldc, int row0, int col0,
                                          const uint32_t (&w)[32], const GemmShape& s, int left) {
  const int nv = whole_vectors<OutT>(s.N);
  if constexpr (sizeof(OutT) == 2) {
    if (left < 64 && col0 + left < s.N) {   // 32 whole columns, others to their right
      const uint32_t mine = slab.put128(tmC, col0, row0, w, false);
      store_half_slab(mine - (threadIdx.x & 31) * 128, C + col0, ldc, row0, s.M);
      return;
    }
  }
  const uint32_t mine = slab.put128(tmC, col0, row0, w, col0 < nv);
  if (nv == s.N) return;
  const int lane = threadIdx.x & 31;
  const int chunk = (nv - col0) * static_cast<int>(sizeof(OutT)) / 16;
  if (nv < col0 || chunk >= 8 || row0 + lane >= s.M) return;
  store_tail(mine + ((chunk ^ (lane & 7)) << 4), C + static_cast<int64_t>(row0 + lane) * ldc + nv, s.N - nv);
}

__device__ __forceinline__ void pack_row64(uint32_t (&w)[32], const uint32_t (&a0)[32], const uint32_t (&a1)[32]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    w[j] = pack_bf16x2(__uint_as_float(a0[2 * j]), __uint_as_float(a0[2 * j + 1]));
    w[16 + j] = pack_bf16x2(__uint_as_float(a1[2 * j]), __uint_as_float(a1[2 * j + 1]));
  }
}

// lo, hi (fp32 bits) += the two bf16 of `old`
__device__ __forceinline__ void add_bf16x2(uint32_t& lo, uint32_t& hi, uint32_t old) {
  const __nv_bfloat162 o = *reinterpret_cast<const __nv_bfloat162*>(&old);
  lo = __float_as_uint(__uint_as_float(lo) + __low2float(o));
  hi = __float_as_uint(__uint_as_float(hi) + __high2float(o));
}

// The first n elements (fewer than a vector) at src, zeros behind them.
template <typename OutT>
__device__ __noinline__ uint4 part_vector(const OutT* src, int n) {
  uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
  for (int e = 0; e < static_cast<int>(16 / sizeof(OutT)) - 1; ++e) {
    if (e >= n) break;
    if constexpr (sizeof(OutT) == 2)
      w[e / 2] |= static_cast<uint32_t>(reinterpret_cast<const uint16_t*>(src)[e]) << (16 * (e % 2));
    else
      w[e] = reinterpret_cast<const uint32_t*>(src)[e];
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// C (+)= acc. The tensor map of C has boxes of 32 rows x 128 bytes (64 bf16 or 32 fp32 columns).
template <typename OutT>
struct StoreEpilogue {
  static constexpr bool kPair = true, kSplit = false, kAhead = false;
  const CUtensorMap* tmC;
  OutT* C;   // read when accumulating
  int64_t ldc;
  int accumulate;
  SlabStore slab;
  __device__ __forceinline__ void tile_begin(int, int) {}
  __device__ __forceinline__ void tile_end(int, int) {}
  __device__ __forceinline__ void drain() { slab.drain(); }
  __device__ __forceinline__ void store_fp32(uint32_t (&acc)[32], int row0, int col0, const GemmShape& s) {
    if (accumulate) {
      uint32_t v[32];
      old_row(v, row0, col0, s);
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(acc[j]));
    }
    store_row(slab, tmC, C, ldc, row0, col0, acc, s, 64);
  }
  // v = 128 bytes of old C from column col0 on, of this lane's row. They come in as they are stored, whole
  // row segments by eight lanes each, and turn through the buffer that put128 fills next. Loads of a lane's own
  // row, 16 bytes in each of 32 rows, thrash the little L1 that the operand stages leave: accumulating into
  // 4096 x 14336 of 128 tokens took 278 us (fp32) and 158 (bf16) that way, 187 and 109 so.
  __device__ __forceinline__ void old_row(uint32_t (&v)[32], int row0, int col0, const GemmShape& s) {
    constexpr int V = 16 / sizeof(OutT);
    const int lane = threadIdx.x & 31, j = lane & 7, col = col0 + j * V;
    const uint32_t slab_at = slab.next();
    uint4 o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = row0 + i * 4 + (lane >> 3);
      const OutT* src = C + static_cast<int64_t>(row) * ldc + col;
      o[i] = make_uint4(0, 0, 0, 0);
      if (row < s.M) {
        if (col + V <= s.N)
          o[i] = *reinterpret_cast<const uint4*>(src);
        else if (col < s.N)
          o[i] = part_vector(src, s.N - col);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      st_shared_v4(slab_at + r * 128 + ((j ^ (r & 7)) << 4), o[i].x, o[i].y, o[i].z, o[i].w);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t w[4];
      ld_shared_v4(slab_at + lane * 128 + ((c ^ (lane & 7)) << 4), w);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[4 * c + e] = w[e];
    }
  }
  __device__ __forceinline__ void operator()(int row, int col0, uint32_t (&a0)[32], uint32_t (&a1)[32], const GemmShape& s, int left) {
    const int row0 = row - static_cast<int>(threadIdx.x & 31);
    if (row0 >= s.M || col0 >= s.N) return;   // uniform over the warp
    if constexpr (sizeof(OutT) == 2) {
      uint32_t w[32];
      if (accumulate) {
        old_row(w, row0, col0, s);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          add_bf16x2(a0[2 * j], a0[2 * j + 1], w[j]);
          add_bf16x2(a1[2 * j], a1[2 * j + 1], w[16 + j]);
        }
      }
      pack_row64(w, a0, a1);
      store_row(slab, tmC, C, ldc, row0, col0, w, s, left);
    } else {
      store_fp32(a0, row0, col0, s);
      if (left > 32 && col0 + 32 < s.N) store_fp32(a1, row0, col0 + 32, s);
    }
  }
};

// bf16 store of acc * row_scale[row] * col_scale[col]: the dequantisation of an fp8 product whose
// operands were quantised per row (activations: one scale per token, weights: one per output
// channel). N is a multiple of 4.
struct ScaledStoreEpilogue {
  static constexpr bool kPair = true, kSplit = false, kAhead = false;
  const CUtensorMap* tmC;
  __nv_bfloat16* C;
  int64_t ldc;
  const float* row_scale;   // [M]
  const float* col_scale;   // [N]
  SlabStore slab;
  __device__ __forceinline__ void tile_begin(int, int) {}
  __device__ __forceinline__ void tile_end(int, int) {}
  __device__ __forceinline__ void drain() { slab.drain(); }
  __device__ __forceinline__ void scale32(uint32_t* w, const uint32_t (&acc)[32], float rs, int col0, int N) const {
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      float4 cs = make_float4(0.f, 0.f, 0.f, 0.f);
      if (col0 + 4 * v < N) cs = *reinterpret_cast<const float4*>(col_scale + col0 + 4 * v);
      w[2 * v] = pack_bf16x2(__uint_as_float(acc[4 * v]) * rs * cs.x, __uint_as_float(acc[4 * v + 1]) * rs * cs.y);
      w[2 * v + 1] = pack_bf16x2(__uint_as_float(acc[4 * v + 2]) * rs * cs.z, __uint_as_float(acc[4 * v + 3]) * rs * cs.w);
    }
  }
  __device__ __forceinline__ void operator()(int row, int col0, uint32_t (&a0)[32], uint32_t (&a1)[32], const GemmShape& s, int left) {
    const int row0 = row - static_cast<int>(threadIdx.x & 31);
    if (row0 >= s.M || col0 >= s.N) return;
    const float rs = row < s.M ? row_scale[row] : 0.f;
    uint32_t w[32];
    scale32(w, a0, rs, col0, s.N);
    scale32(w + 16, a1, rs, col0 + 32, s.N);
    store_row(slab, tmC, C, ldc, row0, col0, w, s, left);
  }
};

// silu(g) * u of 32 columns, two to a word
__device__ __forceinline__ void swiglu32(uint32_t* act, const uint32_t (&g)[32], const uint32_t (&u)[32]) {
  bool ordinary = true;
#pragma unroll
  for (int j = 0; j < 32; ++j) ordinary &= fabsf(__uint_as_float(g[j])) < ORDINARY_GATE;
  if (ordinary) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      act[j] = pack_bf16x2(silu_ordinary(__uint_as_float(g[2 * j])) * __uint_as_float(u[2 * j]),
                           silu_ordinary(__uint_as_float(g[2 * j + 1])) * __uint_as_float(u[2 * j + 1]));
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      act[j] = pack_bf16x2(silu_any(__uint_as_float(g[2 * j])) * __uint_as_float(u[2 * j]),
                           silu_any(__uint_as_float(g[2 * j + 1])) * __uint_as_float(u[2 * j + 1]));
  }
}

// SwiGLU fused into the up/gate GEMM. The weight rows are interleaved in blocks of 64 output
// columns: 32 gate columns followed by their 32 up columns, so one call sees a gate chunk and the
// matching up chunk and writes act = silu(gate) * up (and, optionally, the raw gate|up pair that
// the backward pass needs). The warp's staging area holds the pair (4 KiB, boxes of 64 columns) and
// behind it the activation (2 KiB, boxes of 32 columns, 64-byte swizzle).
struct SwiGluEpilogue {
  static constexpr bool kPair = true, kSplit = false, kAhead = false;
  const CUtensorMap* tmAct;   // [M][N/2]
  const CUtensorMap* tmGu;    // [M][N] interleaved as computed
  int keep_gu;
  SlabStore slab;
  __device__ __forceinline__ void tile_begin(int, int) {}
  __device__ __forceinline__ void tile_end(int, int) {}
  __device__ __forceinline__ void drain() { slab.drain(); }
  // col0 is the first column of the 64-wide (gate|up) block
  __device__ __forceinline__ void operator()(int row, int col0, uint32_t (&g)[32], uint32_t (&u)[32], const GemmShape& s, int) {
    const int lane = threadIdx.x & 31;
    const int row0 = row - lane;
    if (row0 >= s.M || col0 >= s.N) return;
    uint32_t act[16];
    swiglu32(act, g, u);
    if (lane == 0) tma_store_wait_read<0>();
    __syncwarp();
    if (keep_gu) {
      uint32_t w[32];
      pack_row64(w, g, u);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        st_shared_v4(slab.buf + lane * 128 + ((j ^ (lane & 7)) << 4), w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      st_shared_v4(slab.buf + 4096 + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4), act[4 * j], act[4 * j + 1], act[4 * j + 2],
                   act[4 * j + 3]);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (keep_gu) tma_store_2d(tmGu, slab.buf, col0, row0);
      tma_store_2d(tmAct, slab.buf + 4096, col0 / 2, row0);
      tma_store_commit();
    }
  }
};

// SwiGLU in the gate|up product of weights that are stored as two halves, [gate; up]: a tile's first half of
// columns are gates and its second the matching ups (GemmShape::b_second). Stores both, which the backward pass
// reads, and act = silu(gate) * up.
struct SwiGluSplitEpilogue {
  static constexpr bool kPair = false, kSplit = true, kAhead = false;
  const CUtensorMap *tmGate, *tmUp, *tmAct;   // [M][F] each, boxes of 32 rows x 64 columns
  int F;
  SlabStore slab;
  uint32_t gate[32], up[32], act[32];   // this lane's 64 columns of each, two to a word
  __device__ __forceinline__ void tile_begin(int, int) {}
  __device__ __forceinline__ void tile_end(int, int) {}
  __device__ __forceinline__ void drain() { slab.drain(); }
  template <int J>
  __device__ __forceinline__ void part(const uint32_t (&g)[32], const uint32_t (&u)[32]) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      gate[16 * J + j] = pack_bf16x2(__uint_as_float(g[2 * j]), __uint_as_float(g[2 * j + 1]));
      up[16 * J + j] = pack_bf16x2(__uint_as_float(u[2 * j]), __uint_as_float(u[2 * j + 1]));
    }
    swiglu32(act + 16 * J, g, u);
  }
  __device__ __forceinline__ void store(int row, int col, const GemmShape& s) {
    const int row0 = row - static_cast<int>(threadIdx.x & 31);
    if (row0 >= s.M || col >= F) return;   // uniform over the warp
    slab.put128(tmGate, col, row0, gate, true);
    slab.put128(tmUp, col, row0, up, true);
    slab.put128(tmAct, col, row0, act, true);
  }
};

// The gradient of SwiGLU in the product that makes d(act): stores d(gate) and d(up) from the sums and the saved
// gate and up, so that d(act) is neither rounded nor written and read back. Gate and up come through TMA into the
// warp's staging area, the gradients replace them there and leave the same way; the loads of a tile's first columns
// are under way while its products are computed. interleaved: gate and up alternate in blocks of 32 columns
// (one map, 64 columns of d(act) are 128 there, N is a multiple of 64); otherwise they are two halves with a map each.
template <int EW>   // epilogue warps of a CTA
struct SwiGluBwdEpilogue {
  static constexpr bool kPair = true, kSplit = false, kAhead = true;
  static constexpr int STEP = 64 * (EW / 4);   // from one of this warp's slabs of columns to the next
  const CUtensorMap *in0, *in1, *out0, *out1;   // boxes of 32 rows x 64 columns
  int interleaved;
  uint32_t buf, bar;   // this warp's 8 KiB and its barrier for the loads
  uint32_t phase;
  volatile int* abort_flag;
  int* err_word;
  __device__ __forceinline__ void init(uint8_t* smem_raw, uint32_t epi_off) {
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t warp = threadIdx.x >> 5, mine = warp >= 2 ? warp - 2 : 0;
    buf = base + epi_off + mine * GEMM_EPI_WARP_BYTES;
    bar = base + epi_off - 64 + 8 * mine;   // behind the mainloop's barriers
    phase = 0;
    if (warp >= 2 && (threadIdx.x & 31) == 0) {
      mbar_init(bar, 1);
      fence_barrier_init();
    }
    __syncwarp();
  }
  __device__ __forceinline__ void load(int row0, int col0, const GemmShape& s) {
    if (row0 >= s.M || col0 >= s.N || (threadIdx.x & 31) != 0) return;
    tma_store_wait_read<0>();
    mbar_expect_tx(bar, 8192);
    tma_load_2d(buf, in0, interleaved ? 2 * col0 : col0, row0, bar);
    tma_load_2d(buf + 4096, in1, interleaved ? 2 * col0 + 64 : col0, row0, bar);
  }
  __device__ __forceinline__ void tile_ahead(int row0, int col0, const GemmShape& s, volatile int* abort, int* err) {
    abort_flag = abort;
    err_word = err;
    load(row0, col0, s);
  }
  __device__ __forceinline__ void tile_begin(int, int) {}
  __device__ __forceinline__ void tile_end(int, int) {}
  __device__ __forceinline__ void drain() {
    if ((threadIdx.x & 31) == 0) tma_store_wait<0>();
  }
  // d: eight sums; g_at, u_at: the chunks of gate and up, replaced by their gradients
  __device__ __forceinline__ void chunk(const uint32_t* d, uint32_t g_at, uint32_t u_at) const {
    uint32_t g[4], u[4];
    ld_shared_v4(g_at, g);
    ld_shared_v4(u_at, u);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const __nv_bfloat162 gp = *reinterpret_cast<const __nv_bfloat162*>(&g[p]), up = *reinterpret_cast<const __nv_bfloat162*>(&u[p]);
      float dg[2], du[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float gf = e ? __high2float(gp) : __low2float(gp), uf = e ? __high2float(up) : __low2float(up);
        const float df = __uint_as_float(d[2 * p + e]), s = logistic(gf), si = gf * s;
        du[e] = df * si;
        dg[e] = df * uf * (s + si * (1.f - s));
      }
      g[p] = pack_bf16x2(dg[0], dg[1]);
      u[p] = pack_bf16x2(du[0], du[1]);
    }
    st_shared_v4(g_at, g[0], g[1], g[2], g[3]);
    st_shared_v4(u_at, u[0], u[1], u[2], u[3]);
  }
  __device__ __forceinline__ void operator()(int row, int col0, uint32_t (&a0)[32], uint32_t (&a1)[32], const GemmShape& s, int left) {
    const int lane = threadIdx.x & 31, row0 = row - lane;
    if (row0 >= s.M || col0 >= s.N) return;   // uniform over the warp
    const bool here = mbar_wait_bounded(bar, phase, abort_flag, err_word, DEV_ERR_FULL_BAR_TIMEOUT, GEMM_WAIT_LIMIT_NS);
    if (!__all_sync(0xffffffffu, here)) return;
    phase ^= 1;
    const uint32_t first = buf + lane * 128, second = first + 4096;
    auto at = [&](uint32_t slab, int j) { return slab + ((j ^ (lane & 7)) << 4); };
    if (interleaved) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        chunk(a0 + 8 * j, at(first, j), at(first, 4 + j));
        chunk(a1 + 8 * j, at(second, j), at(second, 4 + j));
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        chunk(a0 + 8 * j, at(first, j), at(second, j));
        chunk(a1 + 8 * j, at(first, 4 + j), at(second, 4 + j));
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d(out0, buf, interleaved ? 2 * col0 : col0, row0);
      tma_store_2d(out1, buf + 4096, interleaved ? 2 * col0 + 64 : col0, row0);
      tma_store_commit();
    }
    if (left > STEP) load(row0, col0 + STEP, s);
  }
};

}  // namespace b200

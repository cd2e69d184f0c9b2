// Memory-bound kernels of the Llama training step: RMSNorm (+residual), SwiGLU, RoPE, fused
// softmax-cross-entropy forward+backward, embedding gather/scatter, fused AdamW over flat buffers.
// All are bandwidth kernels: 16-byte vector accesses, one pass where the maths allows it.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <type_traits>

#include "b200ops.h"
#include "cross_entropy_math.cuh"
#include "cross_entropy_stream.cuh"
#include "dependent_launch.cuh"
#include "host_util.h"
#include "swiglu_math.cuh"

namespace b200 {

int* device_status_word();   // gemm.cu

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}
template <int THREADS>
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? red[threadIdx.x] : -INFINITY;
  if (w == 0) {
    t = warp_max(t);
    if (l == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// ------------------------------------------------------------------ RMSNorm
// Bound by memory traffic when its latencies are hidden: at 4096 x 4096 with a residual, forward 28 -> 26 us,
// backward 53 -> 29 us and the sum over its partial rows 14 -> 5 us against one row per CTA, loads behind the
// row's reduction and one chain of loads per column. TPR threads share a row and a CTA holds
// 256 / TPR rows, so that a narrow row does not leave most of the CTA idle; each thread holds VPT
// 16-byte vectors of it.
constexpr int NORM_THREADS = 256;
constexpr int NORM_RING_CTAS = 3;   // of an SM, forward; the backward kernel's partial sums are for two
constexpr int NORM_MAX_SLOTS = 8;
constexpr uint64_t NORM_WAIT_LIMIT_NS = 2000000000ull;

// Sum over the TPR threads of a row, the same in each. `parity` alternates between consecutive calls:
// the one barrier of the next call then separates this call's reads from that buffer's next writes.
template <int TPR>
__device__ __forceinline__ float row_sum(float v, float (&red)[2][NORM_THREADS / 32], int parity) {
  v = warp_sum(v);
  if constexpr (TPR > 32) {
    constexpr int W = TPR / 32;
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[parity][w] = v;
    __syncthreads();
    v = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) v += red[parity][(w & ~(W - 1)) + i];
  }
  return v;
}

// If `res` is given: h = x + res is written to h_out (the new residual stream) and normalised in the
// same pass, so the residual add costs no extra pass.
template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
    rmsnorm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, bf16* __restrict__ h_out,
                       const bf16* __restrict__ w, bf16* __restrict__ y, float* __restrict__ rstd, int T, int H, float eps) {
  after_wait(x, res, h_out, w, y, rstd);
  grid_release_at_start<VPT == 1 ? 8 : VPT == 2 ? 6 : 4>();
  __shared__ float red[2][NORM_THREADS / 32];
  const int lane = threadIdx.x % TPR;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (NORM_THREADS / TPR) + threadIdx.x / TPR;
  const bool live = row < T;
  const Bf16x8* xr = reinterpret_cast<const Bf16x8*>(x + row * H);
  Bf16x8* hr = reinterpret_cast<Bf16x8*>(h_out + row * H);
  const Bf16x8* rr = res ? reinterpret_cast<const Bf16x8*>(res + row * H) : nullptr;
  const Bf16x8* wr = reinterpret_cast<const Bf16x8*>(w);
  Bf16x8 xv[VPT], rv[VPT], wv[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {   // every load of the row is in flight before the first is used
    const int idx = lane + i * TPR;
    if (live && idx * 8 < H) {
      xv[i] = xr[idx];
      if (rr) rv[i] = rr[idx];
      wv[i] = wr[idx];
    }
  }
  float vals[VPT][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = lane + i * TPR;
    if (live && idx * 8 < H) {
      unpack8(xv[i], vals[i]);
      if (rr) {
        float r[8];
        unpack8(rv[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) vals[i][j] += r[j];
        const Bf16x8 h = pack8(vals[i]);
        hr[idx] = h;
        unpack8(h, vals[i]);  // normalise exactly what was stored
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += vals[i][j] * vals[i][j];
    }
  }
  ss = row_sum<TPR>(ss, red, 0);
  if (!live) return;
  const float r = rsqrtf(ss / H + eps);
  if (lane == 0 && rstd) rstd[row] = r;
  Bf16x8* yr = reinterpret_cast<Bf16x8*>(y + row * H);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = lane + i * TPR;
    if (idx * 8 < H) {
      float wf[8], o[8];
      unpack8(wv[i], wf);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = vals[i][j] * r * wf[j];
      yr[idx] = pack8(o);
    }
  }
}

// The groups' parts of dw are added up in shared memory, R - 1 rows of TPR * VPT * 8 floats, and make one row of the partial sums.
template <int TPR, int VPT>
__device__ __forceinline__ void norm_partial_row(float (&dw_acc)[VPT][8], float* group_dw, float* dw_partial, int H, int lane, int group) {
  constexpr int R = NORM_THREADS / TPR, ROW = TPR * VPT * 8;
  if constexpr (R > 1) {
    if (group > 0) {
#pragma unroll
      for (int i = 0; i < VPT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) group_dw[(group - 1) * ROW + (i * 8 + j) * TPR + lane] = dw_acc[i][j];
    }
    __syncthreads();
    if (group > 0) return;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        for (int q = 0; q < R - 1; ++q) dw_acc[i][j] += group_dw[q * ROW + (i * 8 + j) * TPR + lane];
  }
  float* out = dw_partial + static_cast<int64_t>(blockIdx.x) * H;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = lane + i * TPR;
    if (idx * 8 < H) {
      reinterpret_cast<float4*>(out)[2 * idx] = make_float4(dw_acc[i][0], dw_acc[i][1], dw_acc[i][2], dw_acc[i][3]);
      reinterpret_cast<float4*>(out)[2 * idx + 1] = make_float4(dw_acc[i][4], dw_acc[i][5], dw_acc[i][6], dw_acc[i][7]);
    }
  }
}

template <int VPT>
struct NormRow {
  Bf16x8 dy[VPT], x[VPT], dr[VPT];
  float r;
};

// dx = rstd * (dy*w - x * rstd^2 * mean(dy*w*x)); optionally dx += dres (gradient arriving through
// the residual branch). Each CTA walks its rows (blockIdx.x, + gridDim.x, ... in groups of 256 / TPR)
// and keeps their part of dw in registers; the groups are added up in shared memory at the end and
// the CTA writes one row of `dw_partial[gridDim.x][H]`. The loads of the next row are issued before
// the sum over the present one (VPT <= 2, where the registers allow it): otherwise nothing is in
// flight while the CTA waits in its reduction.
template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_THREADS, 2)
    rmsnorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                       const float* __restrict__ rstd, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                       float* __restrict__ dw_partial, int T, int H) {
  after_wait(dy, x, w, rstd, dres, dx, dw_partial);
  constexpr int R = NORM_THREADS / TPR;   // rows of a CTA at a time
  __shared__ float red[2][NORM_THREADS / 32];
  __shared__ float group_dw[R > 1 ? (R - 1) * TPR * VPT * 8 : 1];
  const int lane = threadIdx.x % TPR, group = threadIdx.x / TPR;
  float dw_acc[VPT][8];
  Bf16x8 wv[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = lane + i * TPR;
    if (idx * 8 < H) wv[i] = reinterpret_cast<const Bf16x8*>(w)[idx];
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[i][j] = 0.f;
  }
  auto load = [&](NormRow<VPT>& n, int64_t row) {
    if (row >= T) return;
    n.r = rstd[row];
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = lane + i * TPR;
      if (idx * 8 < H) {
        n.dy[i] = reinterpret_cast<const Bf16x8*>(dy + row * H)[idx];
        n.x[i] = reinterpret_cast<const Bf16x8*>(x + row * H)[idx];
        if (dres) n.dr[i] = reinterpret_cast<const Bf16x8*>(dres + row * H)[idx];
      }
    }
  };
  constexpr bool AHEAD = VPT <= 2;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * R;
  NormRow<VPT> cur, next;
  int64_t row = static_cast<int64_t>(blockIdx.x) * R + group;
  if (AHEAD) load(cur, row);
  int parity = 0;
  for (int64_t row0 = static_cast<int64_t>(blockIdx.x) * R; row0 < T; row0 += stride, row += stride, parity ^= 1) {
    const bool live = row < T;
    if (AHEAD)
      load(next, row + stride);
    else
      load(cur, row);
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (live && (lane + i * TPR) * 8 < H) {
        float d[8], xf[8], wf[8];
        unpack8(cur.dy[i], d);
        unpack8(cur.x[i], xf);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dw_acc[i][j] += d[j] * xf[j] * cur.r;
          dot += d[j] * wf[j] * xf[j];
        }
      }
    }
    dot = row_sum<TPR>(dot, red, parity);
    if (live) {
      const float c = dot * cur.r * cur.r / H;
      Bf16x8* dxr = reinterpret_cast<Bf16x8*>(dx + row * H);
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int idx = lane + i * TPR;
        if (idx * 8 < H) {
          float d[8], xf[8], wf[8], o[8];   // unpacked again: the packed row takes half the registers
          unpack8(cur.dy[i], d);
          unpack8(cur.x[i], xf);
          unpack8(wv[i], wf);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = cur.r * (d[j] * wf[j] - xf[j] * c);
          if (dres) {
            float e[8];
            unpack8(cur.dr[i], e);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += e[j];
          }
          dxr[idx] = pack8(o);
        }
      }
    }
    if (AHEAD) cur = next;
  }
  grid_release();
  norm_partial_row<TPR, VPT>(dw_acc, group_dw, dw_partial, H, lane, group);
}

// ---- The same for many rows: a persistent CTA's rows come through a ring of shared memory, groups of 256 / TPR of them at a time, by bulk
// copies that one thread issues as soon as a group has been read. With loads into registers nothing of a CTA's next row is in flight
// while it reduces (forward), or one row (backward): 16384 x 4096 forward 62 -> 48 us (5.6 TB/s), backward 86 -> 77; 4096 x 4096
// with a residual 27.0 -> 26.0 and 31.7 -> 29.9 with the sum of the partial rows. The weight is read once
// per CTA instead of once per row. What it costs is a barrier of the CTA for every group: norm_ring_slots has where that pays.
struct NormRing {
  uint32_t ring, bars;       // shared memory: slots, and a barrier for each
  int slots, slot;
  uint32_t phase, slot_bytes;
  int* err_word;
  volatile int* abort_flag;
  __device__ __forceinline__ NormRing(uint8_t* smem, uint64_t* bar_words, int* abort_word, int n, uint32_t bytes, int* err)
      : ring(smem_u32(smem)), bars(smem_u32(bar_words)), slots(n), slot(0), phase(0), slot_bytes(bytes), err_word(err), abort_flag(abort_word) {
    if (threadIdx.x == 0) {
      for (int s = 0; s < slots; ++s) mbar_init(bars + 8u * s, 1);
      *abort_word = 0;
      fence_barrier_init();
    }
    __syncthreads();
  }
  __device__ __forceinline__ uint32_t at() const { return ring + slot * slot_bytes; }
  // One thread: part `part` of N of a slot, `bytes` of them.
  template <int N, typename... P>
  __device__ __forceinline__ void load(int s, uint32_t bytes, const P*... from) const {
    mbar_expect_tx(bars + 8u * s, bytes * (0 + ... + (from ? 1 : 0)));
    uint32_t to = ring + s * slot_bytes;
    ((from ? bulk_load(to, from, bytes, bars + 8u * s) : void(), to += slot_bytes / N), ...);
  }
  __device__ __forceinline__ void wait() const {
    mbar_wait_bounded(bars + 8u * slot, phase, abort_flag, err_word, DEV_ERR_FULL_BAR_TIMEOUT, NORM_WAIT_LIMIT_NS);
  }
  __device__ __forceinline__ void next() {
    if (++slot == slots) {
      slot = 0;
      phase ^= 1;
    }
  }
  // After a wait that ran out copies may still be under way.
  __device__ __forceinline__ void leave() const {
    __syncthreads();
    if (*abort_flag) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
  }
};
__device__ __forceinline__ Bf16x8 ring_vector(uint32_t at) {
  uint32_t r[4];
  ld_shared_v4(at, r);
  return *reinterpret_cast<const Bf16x8*>(r);
}

template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_THREADS, NORM_RING_CTAS)
    rmsnorm_fwd_ring_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res, bf16* __restrict__ h_out, const bf16* __restrict__ w,
                            bf16* __restrict__ y, float* __restrict__ rstd, int T, int H, float eps, int slots, int* err_word) {
  constexpr int R = NORM_THREADS / TPR;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bar_words[NORM_MAX_SLOTS];
  __shared__ int abort_word;
  __shared__ float red[2][NORM_THREADS / 32];
  const uint32_t row_bytes = H * 2, part = R * row_bytes;
  NormRing ring(smem, bar_words, &abort_word, slots, res ? 2 * part : part, err_word);
  after_wait(x, res, h_out, w, y, rstd);
  const int lane = threadIdx.x % TPR, group = threadIdx.x / TPR;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * R;
  int64_t row0 = static_cast<int64_t>(blockIdx.x) * R, ahead = row0;
  auto load = [&](int s) {
    if (ahead < T) {
      const uint32_t bytes = static_cast<uint32_t>(T - ahead < R ? T - ahead : R) * row_bytes;
      if (res)
        ring.load<2>(s, bytes, x + ahead * H, res + ahead * H);
      else
        ring.load<1>(s, bytes, x + ahead * H);
    }
    ahead += stride;
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < slots; ++s) load(s);
  Bf16x8 wv[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i)
    if ((lane + i * TPR) * 8 < H) wv[i] = reinterpret_cast<const Bf16x8*>(w)[lane + i * TPR];
  for (int parity = 0; row0 < T; row0 += stride, parity ^= 1) {
    const int64_t row = row0 + group;
    const bool live = row < T;
    ring.wait();
    const uint32_t at = ring.at() + group * row_bytes;
    Bf16x8 hv[VPT];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = lane + i * TPR;
      if (live && idx * 8 < H) {
        hv[i] = ring_vector(at + idx * 16);
        float f[8];
        unpack8(hv[i], f);
        if (res) {
          float r[8];
          unpack8(ring_vector(at + part + idx * 16), r);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] += r[j];
          hv[i] = pack8(f);
          reinterpret_cast<Bf16x8*>(h_out + row * H)[idx] = hv[i];
          unpack8(hv[i], f);  // normalise exactly what was stored
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
      }
    }
    ss = row_sum<TPR>(ss, red, parity);
    if constexpr (TPR <= 32) __syncthreads();   // everybody has read the slot
    if (threadIdx.x == 0) load(ring.slot);
    ring.next();
    if (!live) continue;
    const float r = rsqrtf(ss / H + eps);
    if (lane == 0 && rstd) rstd[row] = r;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = lane + i * TPR;
      if (idx * 8 < H) {
        float f[8], wf[8];
        unpack8(hv[i], f);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = f[j] * r * wf[j];
        reinterpret_cast<Bf16x8*>(y + row * H)[idx] = pack8(f);
      }
    }
  }
  grid_release();
  ring.leave();
}

template <int TPR, int VPT>
__global__ void __launch_bounds__(NORM_THREADS, 2)
    rmsnorm_bwd_ring_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                            const float* __restrict__ rstd, const bf16* __restrict__ dres, bf16* __restrict__ dx,
                            float* __restrict__ dw_partial, int T, int H, int slots, int* err_word) {
  constexpr int R = NORM_THREADS / TPR;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ uint64_t bar_words[NORM_MAX_SLOTS];
  __shared__ int abort_word;
  __shared__ float red[2][NORM_THREADS / 32];
  const uint32_t row_bytes = H * 2, part = R * row_bytes;
  NormRing ring(smem, bar_words, &abort_word, slots, dres ? 3 * part : 2 * part, err_word);
  after_wait(dy, x, w, rstd, dres, dx, dw_partial);
  const int lane = threadIdx.x % TPR, group = threadIdx.x / TPR;
  const int64_t stride = static_cast<int64_t>(gridDim.x) * R;
  int64_t row0 = static_cast<int64_t>(blockIdx.x) * R, ahead = row0;
  auto load = [&](int s) {
    if (ahead < T) {
      const uint32_t bytes = static_cast<uint32_t>(T - ahead < R ? T - ahead : R) * row_bytes;
      if (dres)
        ring.load<3>(s, bytes, dy + ahead * H, x + ahead * H, dres + ahead * H);
      else
        ring.load<2>(s, bytes, dy + ahead * H, x + ahead * H);
    }
    ahead += stride;
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < slots; ++s) load(s);
  float dw_acc[VPT][8];
  Bf16x8 wv[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = lane + i * TPR;
    if (idx * 8 < H) wv[i] = reinterpret_cast<const Bf16x8*>(w)[idx];
#pragma unroll
    for (int j = 0; j < 8; ++j) dw_acc[i][j] = 0.f;
  }
  float r_next = row0 + group < T ? rstd[row0 + group] : 0.f;
  for (int parity = 0; row0 < T; row0 += stride, parity ^= 1) {
    const int64_t row = row0 + group;
    const bool live = row < T;
    const float r = r_next;
    if (row + stride < T) r_next = rstd[row + stride];
    ring.wait();
    const uint32_t at = ring.at() + group * row_bytes;
    Bf16x8 dv[VPT], xv[VPT], ev[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int idx = lane + i * TPR;
      if (live && idx * 8 < H) {
        dv[i] = ring_vector(at + idx * 16);
        xv[i] = ring_vector(at + part + idx * 16);
        if (dres) ev[i] = ring_vector(at + 2 * part + idx * 16);
        float d[8], xf[8], wf[8];
        unpack8(dv[i], d);
        unpack8(xv[i], xf);
        unpack8(wv[i], wf);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          dw_acc[i][j] += d[j] * xf[j] * r;
          dot += d[j] * wf[j] * xf[j];
        }
      }
    }
    dot = row_sum<TPR>(dot, red, parity);
    if constexpr (TPR <= 32) __syncthreads();   // everybody has read the slot
    if (threadIdx.x == 0) load(ring.slot);
    ring.next();
    if (live) {
      const float c = dot * r * r / H;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int idx = lane + i * TPR;
        if (idx * 8 < H) {
          float d[8], xf[8], wf[8], o[8];   // unpacked again: the packed row takes half the registers
          unpack8(dv[i], d);
          unpack8(xv[i], xf);
          unpack8(wv[i], wf);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = r * (d[j] * wf[j] - xf[j] * c);
          if (dres) {
            float e[8];
            unpack8(ev[i], e);
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] += e[j];
          }
          reinterpret_cast<Bf16x8*>(dx + row * H)[idx] = pack8(o);
        }
      }
    }
  }
  grid_release();
  ring.leave();   // the ring's memory is free: the groups' sums are added up in it
  float* group_dw = reinterpret_cast<float*>(smem);
  norm_partial_row<TPR, VPT>(dw_acc, group_dw, dw_partial, H, lane, group);
}

// dw[h] (+)= sum over partial rows. A CTA takes 32 columns; each of its warps adds up every COLSUM_WARPS-th row, so that a column's
// rows are not one chain of dependent loads: the backward pass of 4096 x 4096
// takes 29.4 us, 29.9 with eight warps, 37 x 5120 7.0 and 7.5.
constexpr int COLSUM_WARPS = 32;
__global__ void __launch_bounds__(32 * COLSUM_WARPS)
    colsum_partial_kernel(const float* __restrict__ partial, bf16* __restrict__ dw, int nrows, int H, int accumulate) {
  after_wait(partial, dw);
  grid_release();
  __shared__ float part[COLSUM_WARPS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int h = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (h < H) {
#pragma unroll 10
    for (int r = warp; r < nrows; r += COLSUM_WARPS) s += partial[static_cast<int64_t>(r) * H + h];
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || h >= H) return;
  s = 0.f;
#pragma unroll
  for (int i = 0; i < COLSUM_WARPS; ++i) s += part[i][lane];
  if (accumulate) s += __bfloat162float(dw[h]);
  dw[h] = __float2bfloat16(s);
}

// ------------------------------------------------------------------ SwiGLU on a fused [T, 2F] gate|up tensor
// Element vectors are spread over the grid as (row, vector in the row); the row comes from a 32-bit
// division where the number of vectors allows it (the launcher checks). One vector per thread and pass; carrying row and
// vector along instead of dividing takes as long. 4096 x 14336, L2 flushed, launches in a graph: 56 us (6.3 TB/s);
// 67 with IEEE divisions, cached accesses and a quarter of the CTAs.
// Read once, written once: neither is worth a place in the caches.
__device__ __forceinline__ Bf16x8 load_stream(const Bf16x8* p) {
  const uint4 r = __ldcs(reinterpret_cast<const uint4*>(p));
  return *reinterpret_cast<const Bf16x8*>(&r);
}
__device__ __forceinline__ void store_stream(Bf16x8* p, const Bf16x8& v) {
  __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(&v));
}
template <typename Index>
__global__ void __launch_bounds__(256) swiglu_fwd_kernel(const bf16* __restrict__ gu, bf16* __restrict__ out, int64_t T, int F) {
  after_wait(gu, out);
  grid_release_at_start<8>();
  const Index nvec = static_cast<Index>(T * F / 8), fv = F / 8;
  for (Index k = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; k < nvec; k += static_cast<Index>(gridDim.x) * blockDim.x) {
    const Index t = k / fv, c = k - t * fv;
    const Bf16x8* row = reinterpret_cast<const Bf16x8*>(gu) + static_cast<int64_t>(t) * 2 * fv;
    float g[8], u[8], o[8];
    unpack8(load_stream(row + c), g);
    unpack8(load_stream(row + fv + c), u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = silu(g[j]) * u[j];
    store_stream(reinterpret_cast<Bf16x8*>(out) + k, pack8(o));
  }
}
// dgu[T,2F] from dout[T,F] and the saved gate|up. INTERLEAVED: gate and up alternate in blocks of
// 32 columns (the layout the fused GEMM+SwiGLU epilogue produces) instead of two halves. One vector per
// thread and pass: three loads and two stores already. 4096 x 14336, timed as above: 91 us
// (6.4 TB/s); 96 as the forward kernel was.
template <bool INTERLEAVED, typename Index>
__global__ void __launch_bounds__(256)
    swiglu_bwd_kernel(const bf16* __restrict__ dout, const bf16* __restrict__ gu, bf16* __restrict__ dgu, int64_t T, int F) {
  after_wait(dout, gu, dgu);
  grid_release_at_start<6>();
  const Index nvec = static_cast<Index>(T * F / 8), fv = F / 8;
  for (Index k = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; k < nvec; k += static_cast<Index>(gridDim.x) * blockDim.x) {
    int64_t gi, ui;
    if (INTERLEAVED) {   // rows hold whole blocks: no division
      gi = static_cast<int64_t>(k >> 2) * 8 + (k & 3);
      ui = gi + 4;
    } else {
      const Index t = k / fv;
      gi = static_cast<int64_t>(t) * 2 * fv + (k - t * fv);
      ui = gi + fv;
    }
    const Bf16x8 gv = load_stream(reinterpret_cast<const Bf16x8*>(gu) + gi), uv = load_stream(reinterpret_cast<const Bf16x8*>(gu) + ui);
    const Bf16x8 dv = load_stream(reinterpret_cast<const Bf16x8*>(dout) + k);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(gv, g);
    unpack8(uv, u);
    unpack8(dv, d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = logistic(g[j]);
      const float silu = g[j] * s;
      du[j] = d[j] * silu;
      dg[j] = d[j] * u[j] * (s + silu * (1.f - s));
    }
    store_stream(reinterpret_cast<Bf16x8*>(dgu) + gi, pack8(dg));
    store_stream(reinterpret_cast<Bf16x8*>(dgu) + ui, pack8(du));
  }
}

// ------------------------------------------------------------------ RoPE (rotate-half convention), in place.
// x: [T, nheads, hd] with row pitch `pitch` elements between tokens; cos/sin: [T_pos, hd/2] fp32;
// position of token t is t % seq. sign = +1 forward, -1 backward (the inverse rotation).
__global__ void rope_kernel(bf16* __restrict__ x, const float* __restrict__ cs, const float* __restrict__ sn, int64_t T,
                            int nheads, int hd, int64_t pitch, int seq, float sign) {
  after_wait(x, cs, sn);
  grid_release_at_start<8>();
  const int half = hd / 2;
  const int64_t total = T * nheads * (half / 2);  // each thread rotates two adjacent pairs (bf162 loads)
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int p2 = static_cast<int>(i % (half / 2));
    const int64_t th = i / (half / 2);
    const int h = static_cast<int>(th % nheads);
    const int64_t t = th / nheads;
    const int pos = static_cast<int>(t % seq);
    bf16* base = x + t * pitch + static_cast<int64_t>(h) * hd;
    bf162* lo = reinterpret_cast<bf162*>(base) + p2;
    bf162* hi = reinterpret_cast<bf162*>(base + half) + p2;
    const float2 c = reinterpret_cast<const float2*>(cs + static_cast<int64_t>(pos) * half)[p2];
    float2 s = reinterpret_cast<const float2*>(sn + static_cast<int64_t>(pos) * half)[p2];
    s.x *= sign;
    s.y *= sign;
    const bf162 a = *lo, b = *hi;
    const float a0 = __low2float(a), a1 = __high2float(a), b0 = __low2float(b), b1 = __high2float(b);
    *lo = __floats2bfloat162_rn(a0 * c.x - b0 * s.x, a1 * c.y - b1 * s.y);
    *hi = __floats2bfloat162_rn(b0 * c.x + a0 * s.x, b1 * c.y + a1 * s.y);
  }
}

// Rotary embedding between the fused projection [T][pitch] (q heads, k heads, v heads of `hd` elements
// each) and the three tensors that attention takes, in one pass: forward reads the projection and
// writes q, k (rotated) and v; backward reads the three gradients, undoes the rotation and writes the
// projection's gradient, in place of a zero-filled slice per tensor and two sums over all of it: 22 us each
// way at 4096 tokens of 32 + 2 x 8 heads of 128, where the in-place rotation took 39 and its backward pass
// moved about 600 MB in eight kernels.
// Element (t, h, i) of q lies at q + (t / seq) * batch + (t % seq) * tok + h * head + i. A thread moves
// V elements of a head's lower half and the V that they rotate with; V = 8 needs 16-byte aligned rows
// and hd % 16 == 0.
struct HeadsView {
  bf16* p;
  int64_t batch, tok, head;
};
template <int V>
struct alignas(2 * V) Bf16Vec {
  bf162 v[V / 2];
};
template <int V, bool BACKWARD, typename Index>
__global__ void __launch_bounds__(256)
    rope_qkv_kernel(bf16* __restrict__ qkv, int64_t pitch, HeadsView q, HeadsView k, HeadsView v, const float* __restrict__ cs,
                    const float* __restrict__ sn, int64_t T, int nq, int nkv, int hd, int seq) {
  after_wait(qkv, cs, sn);
  grid_release_at_start<6>();
  using Vec = Bf16Vec<V>;
  const int half = hd / 2;
  const Index per_head = half / V, heads = nq + 2 * nkv;
  const Index total = static_cast<Index>(T) * heads * per_head;
  for (Index i = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; i < total; i += static_cast<Index>(gridDim.x) * blockDim.x) {
    const Index th = i / per_head;
    const int c = static_cast<int>(i - th * per_head) * V;   // first element of the lower half's piece
    const Index t = th / heads;
    int h = static_cast<int>(th - t * heads);
    const int64_t b = t / static_cast<Index>(seq);
    const int pos = static_cast<int>(t - b * seq);
    bf16* fused = qkv + static_cast<int64_t>(t) * pitch + static_cast<int64_t>(h) * hd + c;
    const bool rotate = h < nq + nkv;
    const HeadsView& view = h < nq ? q : h < nq + nkv ? k : v;
    h -= h < nq ? 0 : h < nq + nkv ? nq : nq + nkv;
    bf16* part = view.p + b * view.batch + pos * view.tok + h * view.head + c;
    const bf16* src = BACKWARD ? part : fused;
    bf16* dst = BACKWARD ? fused : part;
    Vec lo = *reinterpret_cast<const Vec*>(src), hi = *reinterpret_cast<const Vec*>(src + half);
    if (rotate) {
      const float* cp = cs + static_cast<int64_t>(pos) * half + c;
      const float* sp = sn + static_cast<int64_t>(pos) * half + c;
#pragma unroll
      for (int j = 0; j < V / 2; ++j) {
        const float2 co = *reinterpret_cast<const float2*>(cp + 2 * j);
        float2 si = *reinterpret_cast<const float2*>(sp + 2 * j);
        if (BACKWARD) si = make_float2(-si.x, -si.y);
        const float a0 = __low2float(lo.v[j]), a1 = __high2float(lo.v[j]), b0 = __low2float(hi.v[j]), b1 = __high2float(hi.v[j]);
        lo.v[j] = __floats2bfloat162_rn(a0 * co.x - b0 * si.x, a1 * co.y - b1 * si.y);
        hi.v[j] = __floats2bfloat162_rn(b0 * co.x + a0 * si.x, b1 * co.y + a1 * si.y);
      }
    }
    *reinterpret_cast<Vec*>(dst) = lo;
    *reinterpret_cast<Vec*>(dst + half) = hi;
  }
}

// ------------------------------------------------------------------ softmax cross-entropy, forward + backward fused
// The logits are overwritten with dlogits = (softmax - onehot) * grad_scale; loss[row] = logsumexp - logit[target].
// Eight elements of a row of V, or as many as are left of it
__device__ __forceinline__ void zero8(bf16* row, int at, int V) {
  if (at + 8 <= V)
    *reinterpret_cast<uint4*>(row + at) = make_uint4(0, 0, 0, 0);
  else
    for (; at < V; ++at) row[at] = __float2bfloat16(0.f);
}

// A cluster of up to eight CTAs takes a row and keeps it in registers, 8 * VPT elements per thread: all loads of the
// row are in flight at once, and maximum and sum of the CTAs' parts meet in shared memory. For rows of one CTA, and for
// few wider ones (ce_row): many stream through shared memory (2048 x 128256: 294 us in clusters, 195 streamed).
// 4096 x 16040 takes 57 us, 97 in two passes; 2048 x 1024 8 and 18; 64 x 128256, in clusters, 13 and 22.
constexpr int CE_ROW_THREADS = 256;
constexpr int CE_ROW_CTAS = 4;   // of an SM
constexpr int CE_MAX_CLUSTER = 8;
constexpr int CE_MAX_VPT = 8;

__device__ __forceinline__ float2 ld_cluster_f2(const float2* local, uint32_t rank) {
  const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(local));
  uint32_t there;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"(rank));
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(there) : "memory");
  return v;
}

template <int VPT>
__global__ void __launch_bounds__(CE_ROW_THREADS, CE_ROW_CTAS)
    cross_entropy_row_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ targets, float* __restrict__ loss, int V,
                             int64_t ld, float grad_scale, int cluster) {
  after_wait(logits, targets, loss);
  grid_release_at_start<CE_ROW_CTAS>();
  __shared__ float red[32];
  __shared__ float2 part;   // maximum of this CTA's elements, sum of their exponentials relative to it
  const int rank = static_cast<int>(blockIdx.x) % cluster;
  const int64_t row = blockIdx.x / cluster;
  bf16* lr = logits + row * ld;
  const int first = (rank * VPT * CE_ROW_THREADS + static_cast<int>(threadIdx.x)) * 8;   // this thread's first element
  constexpr int STEP = CE_ROW_THREADS * 8;
  const bf162 lowest = __halves2bfloat162(__float2bfloat16(-INFINITY), __float2bfloat16(-INFINITY));
  Bf16x8 x[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int at = first + i * STEP;
    if (at + 8 <= V) {
      x[i] = *reinterpret_cast<const Bf16x8*>(lr + at);
    } else {   // the row ends inside the vector or before it
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[i].v[j] = lowest;
        if (at + 2 * j < V) x[i].v[j].x = lr[at + 2 * j];
        if (at + 2 * j + 1 < V) x[i].v[j].y = lr[at + 2 * j + 1];
      }
    }
  }
  const int64_t tgt = targets[row];
  const bool counts = tgt >= 0 && tgt < V;   // other rows are ignored: no loss, zeros for a gradient whatever the logits hold
  float lt = 0.f;
  if (rank == 0 && threadIdx.x == 0 && counts) lt = __bfloat162float(lr[tgt]);   // before anything is overwritten
  float m = -FLT_MAX;
#pragma unroll
  for (int i = 0; i < VPT; ++i) m = fmaxf(m, max8(x[i]));
  m = block_max<CE_ROW_THREADS>(m, red);
  const float own_max = m;
  float c = exp_base(m), s = 0.f;
  if (huge_max(m)) {   // uniform over the CTA
    c = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) x[i].v[j] = __halves2bfloat162(from_huge(x[i].v[j].x, m), from_huge(x[i].v[j].y, m));
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) s += exp_sum8(x[i], c);
  s = block_sum<CE_ROW_THREADS>(s, red);
  if (cluster > 1) {
    if (threadIdx.x == 0) part = make_float2(m, s);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    float2 p[CE_MAX_CLUSTER];
#pragma unroll
    for (int r = 0; r < CE_MAX_CLUSTER; ++r)
      if (r < cluster) {
        p[r] = ld_cluster_f2(&part, r);
        m = fmaxf(m, p[r].x);
      }
    // beside a maximum elsewhere, and where either is huge, nothing here is left of the exponentials
    if (m != own_max) c = huge_max(m) || huge_max(own_max) ? FLT_MAX : exp_base(m);
    s = 0.f;
#pragma unroll
    for (int r = 0; r < CE_MAX_CLUSTER; ++r)
      if (r < cluster) s += p[r].y * exp_share(p[r].x, m);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // waited for below: `part` may be read until then
  }
  if (rank == 0 && threadIdx.x == 0) loss[row] = counts ? ce_loss(m, s, lt) : 0.f;
  const float inv = counts ? grad_scale / s : 0.f;
  if (!counts) {   // 0 * 2^0
    c = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) *reinterpret_cast<uint4*>(&x[i]) = make_uint4(0, 0, 0, 0);
  }
  const int own = counts ? static_cast<int>(tgt) - first : -1;   // the target's place from this thread's first element on
  auto store = [&](auto small) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int at = first + i * STEP;
      if (at >= V) break;
      const Bf16x8 o = ce_gradient8<decltype(small)::value>(x[i], c, inv, own - i * STEP, grad_scale);
      if (at + 8 <= V) {
        *reinterpret_cast<Bf16x8*>(lr + at) = o;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (at + 2 * j < V) lr[at + 2 * j] = o.v[j].x;
          if (at + 2 * j + 1 < V) lr[at + 2 * j + 1] = o.v[j].y;
        }
      }
    }
  };
  if (small_powers_count(inv))
    store(std::true_type{});
  else
    store(std::false_type{});
  if (cluster > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One CTA per token row (ce_two_passes). Pass 1: online max/sum. Pass 2: overwrite the logits. The maximum starts below all bf16 but -inf,
// so that masked elements ahead of the others count as nothing; a branch for them took 16 of 268 us for 2048 x 128256.
constexpr int CE_THREADS = 1024;
__global__ void __launch_bounds__(CE_THREADS)
    cross_entropy_two_pass_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ targets,
                                  float* __restrict__ loss, int V, int64_t ld, float grad_scale) {
  after_wait(logits, targets, loss);
  grid_release();
  __shared__ float red[32];
  const int64_t row = blockIdx.x;
  bf16* lr = logits + row * ld;
  const int nvec = V / 8;
  const Bf16x8* lv = reinterpret_cast<const Bf16x8*>(lr);
  float m = -FLT_MAX, s = 0.f;
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8];
    unpack8(lv[i], f);
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > m) {
      s *= __expf(m - lm);
      m = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    const float f = __bfloat162float(lr[i]);
    if (f > m) {
      s *= __expf(m - f);
      m = f;
    }
    s += __expf(f - m);
  }
  const float gm = block_max<CE_THREADS>(m, red);
  const float gs = block_sum<CE_THREADS>(s * __expf(m - gm), red);
  const int64_t tgt = targets[row];
  if (threadIdx.x == 0) {
    const float lt = (tgt >= 0 && tgt < V) ? __bfloat162float(lr[tgt]) : 0.f;
    loss[row] = (tgt >= 0 && tgt < V) ? logf(gs) + (gm - lt) : 0.f;
  }
  __syncthreads();
  if (tgt < 0 || tgt >= V) {   // an ignored row: zeros, whatever its logits hold
    for (int at = 8 * threadIdx.x; at < V; at += 8 * CE_THREADS) zero8(lr, at, V);
    return;
  }
  const float inv = grad_scale / gs;
  Bf16x8* ov = reinterpret_cast<Bf16x8*>(lr);
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8];
    unpack8(ov[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      f[j] = __expf(f[j] - gm) * inv;
      if (i * 8 + j == tgt) f[j] -= grad_scale;
    }
    ov[i] = pack8(f);
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    float f = __expf(__bfloat162float(lr[i]) - gm) * inv;
    if (i == tgt) f -= grad_scale;
    lr[i] = __float2bfloat16(f);
  }
}

// ------------------------------------------------------------------ embedding
// Bound by look-ups, each two loads one behind the other, of which a thread has one under way: there are as many threads as vectors, or several times
// as many as run at once. 4096 x 4096 takes 11.6 us, 12198 x 2048 15.1, 256 x 256 1.2. A loop over 16 CTAs per SM took 14.9, 19.9 and 1.9 while the
// compiler could batch its loads, and 21.5, 30.9 and 1.6 with pointers that are taken behind the wait and may be those of the stores.
template <typename Index>
__global__ void __launch_bounds__(256) embedding_fwd_kernel(const int64_t* ids, const uint4* table, uint4* out, int64_t T, int H) {
  grid_wait();
  grid_release();
  const Index hv = H / 8, nvec = static_cast<Index>(T) * hv;
  for (Index i = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; i < nvec; i += static_cast<Index>(gridDim.x) * blockDim.x) {
    const Index t = i / hv;
    out[i] = table[ids[t] * hv + (i - t * hv)];
  }
}
// dtable[ids[t]] += dout[t]  (bf16x2 atomics: repeated tokens accumulate)
template <typename Index>
__global__ void embedding_bwd_kernel(const int64_t* __restrict__ ids, const bf16* __restrict__ dout,
                                     bf16* __restrict__ dtable, int64_t T, int H) {
  after_wait(ids, dout, dtable);
  grid_release();
  const Index hv = H / 2, pairs = static_cast<Index>(T) * hv;
  for (Index i = blockIdx.x * static_cast<Index>(blockDim.x) + threadIdx.x; i < pairs; i += static_cast<Index>(gridDim.x) * blockDim.x) {
    const int64_t t = i / hv;
    const int c = static_cast<int>(i - t * hv);
    atomicAdd(reinterpret_cast<bf162*>(dtable + ids[t] * H) + c, reinterpret_cast<const bf162*>(dout + t * H)[c]);
  }
}

// ------------------------------------------------------------------ fused AdamW over flat buffers
// p (bf16) and g (bf16) are the model's flat parameter/gradient buffers; m, v (fp32) and the optional
// fp32 master copy are the optimizer state. One launch updates every parameter. The gradient is
// multiplied by grad_scale (loss scaling / clipping factor) on the way in and zeroed on the way out
// when zero_grad is set, so no separate memset pass is needed.
__global__ void adamw_kernel(bf16* __restrict__ p, bf16* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                             float* __restrict__ master, int64_t n, float lr, float beta1, float beta2, float eps,
                             float wd, float bc1, float bc2, float grad_scale, int zero_grad) {
  after_wait(p, g, m, v, master);
  grid_release_at_start<4>();
  const int64_t nvec = n / 8;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float gf[8], pf[8];
    unpack8(reinterpret_cast<const Bf16x8*>(g)[i], gf);
    if (master) {
      const float4 a = reinterpret_cast<const float4*>(master)[2 * i], b = reinterpret_cast<const float4*>(master)[2 * i + 1];
      pf[0] = a.x; pf[1] = a.y; pf[2] = a.z; pf[3] = a.w; pf[4] = b.x; pf[5] = b.y; pf[6] = b.z; pf[7] = b.w;
    } else {
      unpack8(reinterpret_cast<const Bf16x8*>(p)[i], pf);
    }
    float4 m0 = reinterpret_cast<float4*>(m)[2 * i], m1 = reinterpret_cast<float4*>(m)[2 * i + 1];
    float4 v0 = reinterpret_cast<float4*>(v)[2 * i], v1 = reinterpret_cast<float4*>(v)[2 * i + 1];
    float mf[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
    float vf[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float gr = gf[j] * grad_scale;
      mf[j] = beta1 * mf[j] + (1.f - beta1) * gr;
      vf[j] = beta2 * vf[j] + (1.f - beta2) * gr * gr;
      const float mh = mf[j] / bc1, vh = vf[j] / bc2;
      pf[j] = pf[j] * (1.f - lr * wd) - lr * mh / (sqrtf(vh) + eps);
    }
    reinterpret_cast<float4*>(m)[2 * i] = make_float4(mf[0], mf[1], mf[2], mf[3]);
    reinterpret_cast<float4*>(m)[2 * i + 1] = make_float4(mf[4], mf[5], mf[6], mf[7]);
    reinterpret_cast<float4*>(v)[2 * i] = make_float4(vf[0], vf[1], vf[2], vf[3]);
    reinterpret_cast<float4*>(v)[2 * i + 1] = make_float4(vf[4], vf[5], vf[6], vf[7]);
    if (master) {
      reinterpret_cast<float4*>(master)[2 * i] = make_float4(pf[0], pf[1], pf[2], pf[3]);
      reinterpret_cast<float4*>(master)[2 * i + 1] = make_float4(pf[4], pf[5], pf[6], pf[7]);
    }
    reinterpret_cast<Bf16x8*>(p)[i] = pack8(pf);
    if (zero_grad) reinterpret_cast<uint4*>(g)[i] = make_uint4(0, 0, 0, 0);
  }
}

// sum of squares of a bf16 buffer -> out[0] (fp32 atomics; out must be zeroed by the caller)
__global__ void sumsq_kernel(const bf16* __restrict__ x, int64_t n, float* __restrict__ out) {
  after_wait(x, out);
  grid_release();
  __shared__ float red[32];
  float s = 0.f;
  const int64_t nvec = n / 8;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < nvec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const Bf16x8*>(x)[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += f[j] * f[j];
  }
  s = block_sum<256>(s, red);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

// What holds a row of the cross-entropy in registers: CTAs of a cluster with `vpt` vectors per thread, the fewest that can; none where
// two passes or the stream are better or a cluster is too small. One CTA always pays. Clusters use the SMs that two passes leave idle, so they pay for few rows, and for more
// of them the fuller a row makes their registers. Of 240 pairs of 20 widths from 16392 to 131072 and 1 to 296 rows the rule takes clusters for 116, in
// 0.29 to 1.10 of the time of two passes (1 x 65536 5.7 us, 12.1; 74 x 131072 16.4 and 22.3; 200 x 32768 10.6 and 12.4), and leaves out the slower
// ones (148 x 65544 23.9 and 15.1, 74 x 32776 10.1 and 8.9, 1 x 16392 5.7 and 4.9); its times are 1.005 of the better ones'.
struct CeRow {
  int ctas, vpt;
};
static CeRow ce_row(int64_t T, int V) {
  if (T <= 0 || V <= 0) return {0, 0};
  const int64_t vecs = (static_cast<int64_t>(V) + 7) / 8, sms = sm_count();
  int vpt = 1, ctas = 1;
  while (vpt < CE_MAX_VPT && vpt * CE_ROW_THREADS < vecs) vpt *= 2;
  while (ctas < CE_MAX_CLUSTER && ctas * vpt * CE_ROW_THREADS < vecs) ctas *= 2;
  const int64_t held = ctas * vpt * CE_ROW_THREADS;
  if (held < vecs) return {0, 0};
  bool pays = true;
  if (ctas == 2) pays = 6 * vecs >= 5 * held ? 2 * T <= 3 * sms : 3 * vecs >= 2 * held && 2 * T <= sms;
  if (ctas > 2) pays = 10 * T * held <= 9 * sms * vecs && T * ctas <= CE_ROW_CTAS * sms;
  return pays ? CeRow{ctas, vpt} : CeRow{0, 0};
}

// Rows that no registers hold stream through shared memory, but for two rows for an SM of about a chunk's length (24576 elements), where two
// CTAs of many threads are ahead. The lines are fitted to 64 pairs of times (149 to 296 rows of 18000 to 32760): 240 x 24576 10.0 us, 10.7 streamed, 240 x 28672 11.1
// and 12.3; at 20000 to 22000 both are within 3 %, below 20000 and from 32768 on the stream is the faster one. Everywhere else of 18 numbers of rows from 1
// to 2048 and 12 widths from 16392 to 200000 the stream takes 0.68 to 1.00 of two passes. A row without elements has no chunk to stream.
static bool ce_two_passes(int64_t T, int V) { return V < 8 || (V >= 20000 && V < 32768 && T > sm_count() && T <= 2 * sm_count()); }

// Rows move as 16-byte vectors: null (an argument left out) or on a 16-byte boundary.
template <class... P>
static bool aligned16(const P*... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0;
}

// CTAs for a grid-stride loop over `work_items`, at most per_sm for every SM. With no more than run at once (8 of 256
// threads) the SMs that memory serves last finish last; several times as many even that out, until a thread
// has a single pass left: AdamW over 218 M parameters takes 1032 us with 16
// CTAs per SM, 1004 with 64, 975 with 256 and 1060 with one pass per thread (CUDA events, L2 flushed before).
static inline int grid_for(int64_t work_items, int threads, int per_sm = 16) {
  int64_t b = (work_items + threads - 1) / threads;
  const int64_t cap = static_cast<int64_t>(sm_count()) * per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

constexpr int NORM_RING_SMEM = 112 * 1024;   // what a ring takes at most
// Slots of `bytes` for each of `ctas` CTAs of an SM (228 KB, of which a CTA's own part takes 1 KB and the kernels' other arrays less than that).
static int norm_slots(int bytes, int ctas) {
  const int n = bytes > 0 ? (228 / ctas - 3) * 1024 / bytes : 0;
  return n < NORM_MAX_SLOTS ? n : NORM_MAX_SLOTS;
}

// Slots of the ring that T rows of H elements come through, of 256 / tpr rows each, or none where the kernels without one are as fast. A CTA with one group
// has nothing to read ahead. The lines below lie between those of 1394 pairs of times (330 to 262144 rows of 54 widths from 8 to 8192, up to 2^27
// elements, both kernels in one process, memory cold) where the ring gains and those where it loses, 0.75 to 1.5 of the time:
// - a group of a few hundred elements costs more in its barrier than in its loads (65536 x 64 forward 15.1 us for 12.9, backward 31.6 for 25.2);
// - a ring has to turn some times to gain (1500 x 2048 forward 5.3 for 4.6, 16384 x 2048 28 for 33), and rows that leave a quarter of the
//   threads' registers empty or more are bound by their groups' latency, which a ring makes longer (12000 x 2304 backward 64 us for 59);
// - with a residual many rows are bound by memory, and a ring's are slower there (4096 x 4096 26.0 for 27.0, 16384 x 4096 100 for 94) but for rows
//   that fill half of the threads (65536 x 1032 96 for 108);
// - backward rows wider than 4096 are not loaded ahead without a ring (4096 x 5120 34 for 41), narrower ones are (16384 x 2048 43 for 48, 4096 x 2048
//   17.9 for 17.1), and a fourth vector of a thread costs both more.
// What the rule takes is 1.002 of the better one's time on average forward, 1.003 with a residual, 1.001 and 1.002 backward, and at worst 1.09 (2200 x 1000); no rings
// would be 1.02 to 1.06, rings wherever there are two groups for a CTA 1.04 to 1.06. At 888 other sizes, which it was not drawn by, it is 1.005, 1.006, 1.001 and
// 1.003, at worst 1.12 (500 x 3400 with a residual 6.1 us for 5.5), no rings 1.02 to 1.06.
static int norm_ring_slots(int64_t T, int H, int tpr, int vpt, bool res, bool backward) {
  const int rows = NORM_THREADS / tpr, per_sm = backward ? 2 : NORM_RING_CTAS, room = tpr * vpt * 8;   // elements that a group's registers hold of a row
  const int slots = norm_slots(rows * H * 2 * (1 + backward + res), per_sm);
  if ((T + rows - 1) / rows <= sm_count() * per_sm || slots < (backward ? 3 : 2)) return 0;
  const int64_t millions = T * H / 1000000;
  const bool full = 8 * H >= 7 * room, half = 16 * H <= 9 * room;
  bool pays;
  if (backward)
    pays = H > 6144 ? millions >= (full ? 8 : 20) : H > 4096 ? true : full ? H >= 512 && millions >= (H < 896 ? 25 : 16)
                                                                            : H >= 640 && 16 * H >= 11 * room && millions >= 50;
  else if (!res)
    pays = H >= 256 && millions >= (H > 2048 && H <= 4096 ? 16 : 6);
  else if (H > 4096)
    pays = millions >= 5 && millions < 20;
  else
    pays = full ? H >= 448 && millions < 20 : H >= 256 && half && millions >= 16;
  return pays ? slots : 0;
}

// 32-bit indices hold while a grid's last pass, beyond the last item, stays below 2^32. What they gain is their divisions: rotary split of
// 4096 x 48 x 128 22.9 -> 22.2 us, its backward pass 23.8 -> 22.6, 2048 x 12 x 64 4.6 -> 4.2, the embedding's gradient of 4096 x 4096 28.7 -> 24.8.
static bool small_index(int64_t items) { return items < (1ll << 31); }
static bool swiglu_small(int64_t T, int F) { return small_index(T * F / 8); }

}  // namespace b200

extern "C" {
using namespace b200;

// Threads per row and vectors per thread for a row of H elements: two vectors per thread where a row
// is wide enough (the loads of one thread overlap), one CTA per row from 4096 elements on.
#define B200_NORM_DISPATCH(LAUNCH)        \
  do {                                    \
    if (H <= 256) LAUNCH(32, 1);          \
    else if (H <= 512) LAUNCH(32, 2);     \
    else if (H <= 1024) LAUNCH(64, 2);    \
    else if (H <= 2048) LAUNCH(128, 2);   \
    else if (H <= 4096) LAUNCH(256, 2);   \
    else if (H <= 6144) LAUNCH(256, 3);   \
    else LAUNCH(256, 4);                  \
  } while (0)

int b200_rmsnorm_fwd(const void* x, const void* res, void* h_out, const void* w, void* y, float* rstd, int T, int H,
                     float eps, void* stream) {
  b200::ensure_context();
  if (H % 8 || H > NORM_THREADS * 8 * 4) return B200_ERR_BAD_ARG;
  if (res && !h_out) return B200_ERR_BAD_ARG;
  if (!aligned16(x, res, h_out, w, y)) return B200_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto X = static_cast<const bf16*>(x);
  auto RES = static_cast<const bf16*>(res);
  auto HO = static_cast<bf16*>(h_out);
  auto W = static_cast<const bf16*>(w);
  auto Y = static_cast<bf16*>(y);
#define B200_NORM_FWD(TPR, VPT)                                                                                              \
  do {                                                                                                                       \
    constexpr int R = NORM_THREADS / TPR;                                                                                    \
    const int slots = norm_ring_slots(T, H, TPR, VPT, RES, false);                                                           \
    if (slots) {                                                                                                             \
      const int rc = allow_smem<rmsnorm_fwd_ring_kernel<TPR, VPT>>(NORM_RING_SMEM);                                          \
      if (rc) return rc;                                                                                                     \
      launch_dependent(rmsnorm_fwd_ring_kernel<TPR, VPT>, sm_count() * NORM_RING_CTAS, NORM_THREADS,                         \
                       slots * R * H * 2 * (RES ? 2 : 1), s, X, RES, HO, W, Y, rstd, T, H, eps, slots, device_status_word());\
    } else {                                                                                                                 \
      launch_dependent(rmsnorm_fwd_kernel<TPR, VPT>, (T + R - 1) / R, NORM_THREADS, 0, s, X, RES, HO, W, Y, rstd, T, H, eps);\
    }                                                                                                                        \
  } while (0)
  B200_NORM_DISPATCH(B200_NORM_FWD);
#undef B200_NORM_FWD
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// Whether the rows of those calls come through a ring of shared memory.
int b200_rmsnorm_ring(int T, int H, int with_res, int backward) {
  b200::ensure_context();
  if (H % 8 || H > NORM_THREADS * 8 * 4) return 0;
#define B200_NORM_RING(TPR, VPT) return norm_ring_slots(T, H, TPR, VPT, with_res, backward) > 0
  B200_NORM_DISPATCH(B200_NORM_RING);
#undef B200_NORM_RING
}

// Number of fp32 rows the caller must provide in dw_partial.
int b200_rmsnorm_bwd_partial_rows() {
  b200::ensure_context(); return sm_count() * 2; }

int b200_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                     float* dw_partial, void* dw, int accumulate_dw, int T, int H, void* stream) {
  b200::ensure_context();
  if (H % 8 || H > NORM_THREADS * 8 * 4 || !aligned16(dy, x, w, dres, dx, dw_partial)) return B200_ERR_BAD_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int grid = sm_count() * 2;
  auto DY = static_cast<const bf16*>(dy);
  auto X = static_cast<const bf16*>(x);
  auto W = static_cast<const bf16*>(w);
  auto DR = static_cast<const bf16*>(dres);
  auto DX = static_cast<bf16*>(dx);
#define B200_NORM_BWD(TPR, VPT)                                                                                              \
  do {                                                                                                                       \
    constexpr int R = NORM_THREADS / TPR;                                                                                    \
    const int slots = norm_ring_slots(T, H, TPR, VPT, DR, true);                                                             \
    if (slots) {                                                                                                             \
      const int ring = slots * R * H * 2 * (DR ? 3 : 2), parts = (R - 1) * TPR * VPT * 8 * 4;                                \
      const int rc = allow_smem<rmsnorm_bwd_ring_kernel<TPR, VPT>>(NORM_RING_SMEM);                                          \
      if (rc) return rc;                                                                                                     \
      launch_dependent(rmsnorm_bwd_ring_kernel<TPR, VPT>, grid, NORM_THREADS, ring > parts ? ring : parts, s, DY, X, W, rstd, DR, DX,\
                       dw_partial, T, H, slots, device_status_word());                                                       \
    } else {                                                                                                                 \
      const int groups = (T + R - 1) / R;                                                                                    \
      if (grid > groups) grid = groups;                                                                                      \
      launch_dependent(rmsnorm_bwd_kernel<TPR, VPT>, grid, NORM_THREADS, 0, s, DY, X, W, rstd, DR, DX, dw_partial, T, H);    \
    }                                                                                                                        \
  } while (0)
  B200_NORM_DISPATCH(B200_NORM_BWD);
#undef B200_NORM_BWD
  launch_dependent(colsum_partial_kernel, (H + 31) / 32, 32 * COLSUM_WARPS, 0, s, dw_partial, static_cast<bf16*>(dw), grid, H, accumulate_dw);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_swiglu_fwd(const void* gu, void* out, long long T, int F, void* stream) {
  b200::ensure_context();
  if (F % 8 || !aligned16(gu, out)) return B200_ERR_BAD_ARG;
  const int grid = grid_for(T * F / 8, 256, 64);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto GU = static_cast<const bf16*>(gu);
  auto O = static_cast<bf16*>(out);
  if (swiglu_small(T, F)) launch_dependent(swiglu_fwd_kernel<unsigned>, grid, 256, 0, s, GU, O, T, F);
  else launch_dependent(swiglu_fwd_kernel<int64_t>, grid, 256, 0, s, GU, O, T, F);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_swiglu_bwd(const void* dout, const void* gu, void* dgu, long long T, int F, void* stream) {
  b200::ensure_context();
  if (F % 8 || !aligned16(dout, gu, dgu)) return B200_ERR_BAD_ARG;
  auto kern = swiglu_small(T, F) ? swiglu_bwd_kernel<false, unsigned> : swiglu_bwd_kernel<false, int64_t>;
  launch_dependent(kern, grid_for(T * F / 8, 256, 64), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<const bf16*>(dout), static_cast<const bf16*>(gu), static_cast<bf16*>(dgu), T, F);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}
int b200_swiglu_bwd_interleaved(const void* dout, const void* gu, void* dgu, long long T, int F, void* stream) {
  b200::ensure_context();
  if (F % 32 || !aligned16(dout, gu, dgu)) return B200_ERR_BAD_ARG;
  auto kern = swiglu_small(T, F) ? swiglu_bwd_kernel<true, unsigned> : swiglu_bwd_kernel<true, int64_t>;
  launch_dependent(kern, grid_for(T * F / 8, 256, 64), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<const bf16*>(dout), static_cast<const bf16*>(gu), static_cast<bf16*>(dgu), T, F);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_rope(void* x, const float* cs, const float* sn, long long T, int nheads, int hd, long long pitch, int seq,
              int backward, void* stream) {
  b200::ensure_context();
  if (hd % 4 || reinterpret_cast<uintptr_t>(x) % 4 || (T > 1 && pitch % 2) ||
      (reinterpret_cast<uintptr_t>(cs) | reinterpret_cast<uintptr_t>(sn)) % 8)
    return B200_ERR_BAD_ARG;
  launch_dependent(rope_kernel, grid_for(T * nheads * (hd / 4), 256), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<bf16*>(x), cs, sn, T, nheads, hd, pitch, seq, backward ? -1.f : 1.f);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// q, k, v: element strides (batch, token, head) in `strides` as {q.batch, q.tok, q.head, k..., v...}; cs, sn
// [>= seq][hd / 2]; T = batches * seq rows of the fused projection. hd must be a multiple of 4.
int b200_rope_qkv(void* qkv, long long pitch, void* q, void* k, void* v, const long long* strides, const float* cs,
                  const float* sn, long long T, int nq, int nkv, int hd, int seq, int backward, void* stream) {
  b200::ensure_context();
  if (hd % 4 || T <= 0 || seq <= 0 || nq <= 0 || nkv <= 0) return B200_ERR_BAD_ARG;
  HeadsView w[3];
  bf16* base[3] = {static_cast<bf16*>(q), static_cast<bf16*>(k), static_cast<bf16*>(v)};
  uint64_t ptrs = reinterpret_cast<uint64_t>(qkv), steps = static_cast<uint64_t>(pitch);
  for (int i = 0; i < 3; ++i) {
    w[i] = HeadsView{base[i], strides[3 * i], strides[3 * i + 1], strides[3 * i + 2]};
    ptrs |= reinterpret_cast<uint64_t>(base[i]);
    steps |= static_cast<uint64_t>(w[i].batch) | static_cast<uint64_t>(w[i].tok) | static_cast<uint64_t>(w[i].head);
  }
  if (ptrs % 4 || steps % 2 || (reinterpret_cast<uintptr_t>(cs) | reinterpret_cast<uintptr_t>(sn)) % 8) return B200_ERR_BAD_ARG;
  const bool wide = hd % 16 == 0 && ptrs % 16 == 0 && steps % 8 == 0;
  const int64_t items = T * (nq + 2 * nkv) * (hd / 2 / (wide ? 8 : 2));
  const int grid = grid_for(items, 256);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  auto pick = [&](auto index) {
    using Index = decltype(index);
    return wide ? (backward ? rope_qkv_kernel<8, true, Index> : rope_qkv_kernel<8, false, Index>)
                : (backward ? rope_qkv_kernel<2, true, Index> : rope_qkv_kernel<2, false, Index>);
  };
  auto kern = small_index(items) ? pick(0u) : pick(int64_t{0});
  launch_dependent(kern, grid, 256, 0, s, static_cast<bf16*>(qkv), pitch, w[0], w[1], w[2], cs, sn, T, nq, nkv, hd, seq);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_cross_entropy(void* logits, const long long* targets, float* loss, int T, int V, long long ld,
                       float grad_scale, void* stream) {
  b200::ensure_context();
  if (ld % 8 || (V >= 8 && !aligned16(logits))) return B200_ERR_BAD_ARG;   // rows move as 16-byte vectors
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto L = static_cast<bf16*>(logits);
  auto TG = reinterpret_cast<const int64_t*>(targets);
  const CeRow r = ce_row(T, V);
  if (r.ctas) {
    auto kern = r.vpt == 1 ? cross_entropy_row_kernel<1> : r.vpt == 2 ? cross_entropy_row_kernel<2>
              : r.vpt == 4 ? cross_entropy_row_kernel<4> : cross_entropy_row_kernel<8>;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = r.ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see dependent_launch.cuh
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(T * r.ctas);
    cfg.blockDim = dim3(CE_ROW_THREADS);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    B200_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, L, TG, loss, V, static_cast<int64_t>(ld), grad_scale, r.ctas));
    return 0;
  }
  if (ce_two_passes(T, V)) {
    launch_dependent(cross_entropy_two_pass_kernel, T, CE_THREADS, 0, st, L, TG, loss, V, ld, grad_scale);
  } else {
    const int rc = allow_smem<cross_entropy_stream_kernel>(CES_SMEM);
    if (rc) return rc;
    launch_dependent(cross_entropy_stream_kernel, T < sm_count() ? T : sm_count(), CES_THREADS, CES_SMEM, st, L, TG, loss, T, V, ld,
                     grad_scale, device_status_word());
  }
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// CTAs that share a row of that call, 0 where a CTA goes over its row twice.
int b200_cross_entropy_ctas(int T, int V) { return ce_row(T, V).ctas; }

int b200_embedding_fwd(const long long* ids, const void* table, void* out, long long T, int H, void* stream) {
  b200::ensure_context();
  if (H % 8 || !aligned16(table, out)) return B200_ERR_BAD_ARG;
  launch_dependent(small_index(T * H / 8) ? embedding_fwd_kernel<unsigned> : embedding_fwd_kernel<int64_t>, grid_for(T * H / 8, 256, 256), 256, 0,
      static_cast<cudaStream_t>(stream), reinterpret_cast<const int64_t*>(ids), static_cast<const uint4*>(table), static_cast<uint4*>(out), T, H);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}
int b200_embedding_bwd(const long long* ids, const void* dout, void* dtable, long long T, int H, void* stream) {
  b200::ensure_context();
  // pairs of elements, and atomics on them
  if (H % 2 || (reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dtable)) % 4) return B200_ERR_BAD_ARG;
  launch_dependent(small_index(T * H / 2) ? embedding_bwd_kernel<unsigned> : embedding_bwd_kernel<int64_t>, grid_for(T * H / 2, 256), 256, 0, static_cast<cudaStream_t>(stream),
      reinterpret_cast<const int64_t*>(ids), static_cast<const bf16*>(dout), static_cast<bf16*>(dtable), T, H);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_adamw(void* p, void* g, float* m, float* v, float* master, long long n, float lr, float beta1, float beta2,
               float eps, float wd, int step, float grad_scale, int zero_grad, void* stream) {
  b200::ensure_context();
  if (n % 8) return B200_ERR_BAD_ARG;
  const float bc1 = 1.f - powf(beta1, static_cast<float>(step));
  const float bc2 = 1.f - powf(beta2, static_cast<float>(step));
  launch_dependent(adamw_kernel, grid_for(n / 8, 256, 256), 256, 0, static_cast<cudaStream_t>(stream),
      static_cast<bf16*>(p), static_cast<bf16*>(g), m, v, master, n, lr, beta1, beta2, eps, wd, bc1, bc2, grad_scale,
      zero_grad);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_sumsq(const void* x, long long n, float* out, void* stream) {
  b200::ensure_context();
  if (n % 8) return B200_ERR_BAD_ARG;
  launch_dependent(sumsq_kernel, grid_for(n / 8, 256), 256, 0, static_cast<cudaStream_t>(stream), static_cast<const bf16*>(x), n, out);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // extern "C"

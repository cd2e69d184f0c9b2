// Expert-parallel MoE dispatch / combine, device-initiated over the GIN primitives (peer stores,
// release-ordered remote atomics, bounded waits), fused with the routing permute and the
// block-scaled fp8 (e4m3, 1x128 groups) quantisation:
//
//  moe_route    : histogram of this rank's top-k choices per expert, all ranks exchange their
//                 histograms (puts + signals), and every rank derives from the full matrix where
//                 each (source rank, expert) segment starts in the owner's receive buffer. The
//                 receive buffer therefore comes out packed expert-major with no padding and is
//                 directly usable as the row-segmented operand of the expert GEMMs.
//  moe_dispatch : a team of warps per token: quantise (or copy) the row once, then store it into the
//                 receive buffer of every rank that owns one of its k experts, with its scales
//                 and a 16-byte record (token, slot, weight, source rank) used on the way back.
//  moe_combine  : every expert-output row travels back to its source token's (token, slot) cell;
//                 when all ranks have delivered, the source sums its k cells, gate-weighted.
//
// Rows that stay on their rank need not be read back from the window: dispatch can store them into the
// tensor that the experts read as well (moe_collect_rows adds what other ranks sent), and combine sums
// them from the expert outputs. The window holds every row and every cell after each call all the same,
// since its views are part of the interface.
//
// The reference moves such traffic as host-proxied RDMA writes with immediate data and signal
// atomics (reference: src/rdma/gin/nccl_ofi_gin.cpp, nccl_ofi_gin_resources.cpp); here the GPU
// threads that produce the bytes also put them.
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "dependent_launch.cuh"
#include "gin_device.cuh"
#include "host_util.h"

namespace b200 {

const GinDevHandle* comm_handle(int id);  // collectives.cu

constexpr int MOE_SIG_BASE = 3072;  // GIN signal slots [3072, 3072 + 3 * 8): phase x source rank
constexpr int MOE_MAX_EXPERTS = 1024;
constexpr int MOE_THREADS = 256;
constexpr int CTAS_PER_SM = 16;   // of a grid that has the work for them, see token_grid

struct MoeMeta {  // one per received row
  int32_t token, slot;
  float weight;
  int32_t src_rank;
};

__device__ __forceinline__ bool moe_wait_all(const GinDevHandle& h, int phase, uint64_t epoch) {
  // threads 0..nranks-1 each wait for one source
  bool ok = true;
  if (static_cast<int>(threadIdx.x) < h.nranks)
    ok = gin_spin_u64_ge(h, gin_signal_ptr(h, h.rank, MOE_SIG_BASE + phase * GIN_MAX_RANKS + threadIdx.x), 0, epoch,
                         DEV_ERR_SIGNAL_TIMEOUT);
  return __syncthreads_and(ok ? 1 : 0) != 0;
}

// The CTA that finishes last returns true (and rearms the counter for the next launch).
__device__ __forceinline__ bool last_cta_done(unsigned int* counter) {
  __shared__ int is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int prev = atomicAdd(counter, 1u);
    is_last = prev == gridDim.x - 1;
    if (is_last) *counter = 0;
    __threadfence();
  }
  __syncthreads();
  return is_last != 0;
}

// ------------------------------------------------------------------------------------------ route
struct RouteArgs {
  GinDevHandle h;
  const int32_t* topk_idx;  // [T][k]
  int T, k, E;
  size_t cnt_off;           // window: int32 [2][nranks][E] (call parity), row r written by rank r
  int32_t* cnt_local;       // [E] zero on entry, zero again on exit
  int32_t* dest_base;       // [E] out: first row, in the owner's receive buffer, of this rank's tokens for expert e
  int32_t* expert_offsets;  // [E/nranks + 1] out: row ranges of the local experts in this rank's receive buffer
  int32_t* cursor;          // [E] out: zeroed (next free position inside each of this rank's segments)
  unsigned int* done;
  uint64_t epoch;
};

__global__ void __launch_bounds__(MOE_THREADS) moe_route_kernel(RouteArgs a) {
  grid_wait();
  __shared__ int32_t hist[MOE_MAX_EXPERTS];
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int total = a.T * a.k;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int e = a.topk_idx[i];
    if (e >= 0 && e < a.E) atomicAdd(&hist[e], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x)
    if (hist[e]) atomicAdd(&a.cnt_local[e], hist[e]);
  if (!last_cta_done(a.done)) return;
  const GinDevHandle& h = a.h;
  // publish this rank's histogram in everybody's matrix, then signal
  for (int p = 0; p < h.nranks; ++p) {
    int32_t* row = reinterpret_cast<int32_t*>(h.window[p] + a.cnt_off) + ((a.epoch & 1) * h.nranks + h.rank) * a.E;
    for (int e = threadIdx.x; e < a.E; e += blockDim.x) row[e] = a.cnt_local[e];
  }
  __syncthreads();
  if (static_cast<int>(threadIdx.x) < h.nranks)
    gin_signal(h, threadIdx.x, MOE_SIG_BASE + 0 * GIN_MAX_RANKS + h.rank, 1, GIN_SIGNAL_INC);
  const bool ok = moe_wait_all(h, 0, a.epoch);
  const int32_t* mat = reinterpret_cast<const int32_t*>(h.window[h.rank] + a.cnt_off) + (a.epoch & 1) * h.nranks * a.E;
  const int el = a.E / h.nranks;  // experts per rank
  // Totals per expert and their exclusive prefix over all experts, PER of them to a thread; an owner's experts are neighbours, so
  // that a prefix among them is a difference. A loop over an expert's predecessors took up to 3 us (256 experts).
  constexpr int PER = MOE_MAX_EXPERTS / MOE_THREADS, WARPS = MOE_THREADS / 32;
  __shared__ int32_t before[MOE_MAX_EXPERTS], warp_total[WARPS];
  int tot[PER], sum = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x * PER + i;
    tot[i] = 0;
    for (int s = 0; s < h.nranks; ++s) tot[i] += ok && e < a.E ? mat[s * a.E + e] : 0;
    sum += tot[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int scan = sum;   // inclusive over the warp
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int left = __shfl_up_sync(0xffffffffu, scan, o);
    if (lane >= o) scan += left;
  }
  if (lane == 31) warp_total[warp] = scan;
  __syncthreads();
  int at = scan - sum;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) at += w < warp ? warp_total[w] : 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x * PER + i;
    hist[e] = tot[i];
    before[e] = at;
    at += tot[i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < a.E; e += blockDim.x) {
    const int owner_first = (e / el) * el;
    const int base = before[e] - before[owner_first];
    int before_me = 0;
    for (int s = 0; s < h.rank; ++s) before_me += ok ? mat[s * a.E + e] : 0;
    a.dest_base[e] = base + before_me;
    a.cursor[e] = 0;
    a.cnt_local[e] = 0;
    if (e / el == h.rank) {
      a.expert_offsets[e - owner_first] = base;
      if (e - owner_first == el - 1) a.expert_offsets[el] = base + hist[e];
    }
  }
}

// ------------------------------------------------------------------------------------------ dispatch
struct DispatchArgs {
  GinDevHandle h;
  const __nv_bfloat16* x;    // [T][H]
  const int32_t* topk_idx;   // [T][k]
  const float* topk_w;       // [T][k]
  int T, k, H, E;
  int team_warps;            // TokenTeam
  int fp8;                   // 1: payload e4m3 + fp32 scale per 128 elements; 0: payload bf16
  int use_saved_rows;        // 1: rows come from row_of (backward pass); 0: assigned here and saved there
  int scale_by_weight;       // 1: the row is multiplied by its gate weight before it is sent
  const int32_t* dest_base;  // [E]
  int32_t* cursor;           // [E]
  int32_t* row_of;           // [T][k] receive-buffer row of every (token, slot); -1 = dropped
  int32_t* local_row;        // [T][k] out: the same row where this rank owns the expert, else -1
  __nv_bfloat16* local_out;  // rows of this rank's own tokens go here as well (as the dequantised values), or null
  size_t recv_off, scale_off, meta_off;  // window offsets on the receiving side
  int capacity_rows;
  unsigned int* done;
  uint64_t epoch;
};

__device__ __forceinline__ float warp_half_max(float v) {  // max over each group of 16 lanes
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

constexpr int MOE_MAX_TOPK = 16;

// How the warps of a CTA share tokens in dispatch and in combine's sum: a team of them, the smallest power
// of two that covers a row, works on one token and synchronises on a barrier of its own, so that a wide row
// moves in pieces of several KiB and a narrow one leaves no warp idle. A warp takes 1024 elements of the
// row where that gives every SM 16 warps, and 256 where there are too few tokens for it: 4096 x 3072, top-2,
// sum 43 -> 38 us and dispatch 46 -> 40 against 256 elements a warp; 64 x 1024 sum 15 us, 17 with 1024.
struct TokenTeam {
  static constexpr int WARPS = MOE_THREADS / 32;
  int warps, teams;   // warps of a team, teams of the CTA
  int team, warp;     // this thread's team and its warp in the team
  static int warps_for(int T, int H) {
    const int64_t wide = static_cast<int64_t>(T) * ((H + 1023) / 1024);
    const int per_warp = wide >= 16ll * sm_count() ? 1024 : 256;
    int w = 1;
    while (w < WARPS && w * per_warp < H) w *= 2;
    return w;
  }
  __device__ __forceinline__ explicit TokenTeam(int team_warps) {
    warps = team_warps;
    teams = WARPS / warps;
    team = static_cast<int>(threadIdx.x >> 5) / warps;
    warp = static_cast<int>(threadIdx.x >> 5) % warps;
  }
  __device__ __forceinline__ void sync() const {
    if (warps == 1)
      __syncwarp();
    else
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(warps * 32) : "memory");
  }
  __device__ __forceinline__ int thread() const { return warp * 32 + static_cast<int>(threadIdx.x & 31); }
};

// Eight values of one lane (16 lanes share a 128-element scale group) -> eight e4m3 bytes.
__device__ __forceinline__ uint2 quantize8(const float (&v)[8], float w, float& scale) {
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j] * w));
  amax = warp_half_max(amax);
  scale = fmaxf(amax, 1e-12f) * (1.f / 448.f);
  const float m = w / scale;
  uint2 q;
  q.x = static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(v[0] * m, v[1] * m), __NV_SATFINITE, __NV_E4M3)) |
        (static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(v[2] * m, v[3] * m), __NV_SATFINITE, __NV_E4M3)) << 16);
  q.y = static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(v[4] * m, v[5] * m), __NV_SATFINITE, __NV_E4M3)) |
        (static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(v[6] * m, v[7] * m), __NV_SATFINITE, __NV_E4M3)) << 16);
  return q;
}

// Eight e4m3 bytes times their scale, as bf16.
__device__ __forceinline__ uint4 dequantize8(uint2 q, float scale) {
  const __nv_fp8x2_storage_t* p = reinterpret_cast<const __nv_fp8x2_storage_t*>(&q);
  __nv_bfloat162 o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2(p[j], __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hr));
    o[j] = __floats2bfloat162_rn(f.x * scale, f.y * scale);
  }
  return *reinterpret_cast<const uint4*>(o);
}

// A team per token: a wide one writes a destination row 2 KiB (fp8) or 4 KiB (bf16) at a time, where a warp
// per token left every row 256 or 512 bytes at a time among thousands of others (4096 tokens x 7168, top-8,
// routing included: fp8 95 -> 79 us, bf16 140 -> 120). Four CTAs per SM: with the registers of three the
// fp8 call took 101 us. local_out adds stores to the call and saves reading the window back.
__global__ void __launch_bounds__(MOE_THREADS, 4) moe_dispatch_kernel(DispatchArgs a) {
  grid_wait();
  const GinDevHandle& h = a.h;
  const TokenTeam team(a.team_warps);
  const int lane = threadIdx.x & 31;
  const int el = a.E / h.nranks;
  const int chunks = a.H / 256;      // 256 elements (two scale groups) per warp pass
  const int groups = a.H / 128;
  const size_t row_bytes = a.fp8 ? static_cast<size_t>(a.H) : static_cast<size_t>(a.H) * 2;
  const bool weighted = a.scale_by_weight != 0;
  constexpr int MAX_PASSES = 4;      // H / 128 <= 64 (the launcher checks): at most 32 chunks
  __shared__ float team_scale[TokenTeam::WARPS][64];
  __shared__ int team_rank[TokenTeam::WARPS][MOE_MAX_TOPK], team_row[TokenTeam::WARPS][MOE_MAX_TOPK];   // row < 0: goes nowhere
  __shared__ float team_w[TokenTeam::WARPS][MOE_MAX_TOPK];
  float* scale_buf = team_scale[team.team];
  int *slot_rank = team_rank[team.team], *slot_row = team_row[team.team];
  float* slot_w = team_w[team.team];
  for (int t0 = blockIdx.x * team.teams; t0 < a.T; t0 += gridDim.x * team.teams) {
    const int t = t0 + team.team;
    const bool live = t < a.T;
    // the token's row is on its way while the k copies find their places
    const uint4* src = reinterpret_cast<const uint4*>(a.x + static_cast<size_t>(t) * a.H);
    uint4 raws[MAX_PASSES];
#pragma unroll
    for (int i = 0; i < MAX_PASSES; ++i)
      if (live && team.warp + i * team.warps < chunks) raws[i] = src[(team.warp + i * team.warps) * 32 + lane];
    team.sync();   // the slots and scales of the token before have been read
    if (live && team.thread() < a.k) {
      const int slot = team.thread();
      int my_rank = -1, my_row = -1;
      const int e = a.topk_idx[t * a.k + slot];
      const float my_w = a.topk_w ? a.topk_w[t * a.k + slot] : 1.f;
      if (e >= 0 && e < a.E) {
        my_rank = e / el;
        if (a.use_saved_rows) {
          my_row = a.row_of[t * a.k + slot];
        } else {
          my_row = a.dest_base[e] + atomicAdd(&a.cursor[e], 1);
          if (my_row >= a.capacity_rows) {
            gin_record_error(h, DEV_ERR_CAPACITY);
            my_row = -1;
          }
          a.row_of[t * a.k + slot] = my_row;
        }
        if (my_row >= 0) {
          MoeMeta m{t, slot, my_w, h.rank};
          *reinterpret_cast<int4*>(h.window[my_rank] + a.meta_off + static_cast<size_t>(my_row) * sizeof(MoeMeta)) =
              *reinterpret_cast<const int4*>(&m);
        }
      } else if (!a.use_saved_rows) {
        a.row_of[t * a.k + slot] = -1;
      }
      // saved rows too: a program that keeps row_of of several routings puts back the one it continues with
      a.local_row[t * a.k + slot] = my_rank == h.rank ? my_row : -1;
      slot_rank[slot] = my_rank;
      slot_row[slot] = my_row;
      slot_w[slot] = my_w;
    }
    team.sync();
    // ---- the row itself; an unweighted row is quantised once and stored k times, a weighted one is
    // scaled and quantised per slot
#pragma unroll
    for (int i = 0; i < MAX_PASSES; ++i) {
      const int c = team.warp + i * team.warps;
      if (!live || c >= chunks) break;
      const uint4 raw = raws[i];
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&raw);
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[2 * j] = __low2float(p[j]);
        v[2 * j + 1] = __high2float(p[j]);
      }
      uint2 q = make_uint2(0, 0);
      float scale = 1.f;
      if (a.fp8 && !weighted) {
        q = quantize8(v, 1.f, scale);
        if ((lane & 15) == 0) scale_buf[2 * c + (lane >> 4)] = scale;
      }
      uint4 plain = make_uint4(0, 0, 0, 0);
      if (a.fp8 && !weighted && a.local_out) plain = dequantize8(q, scale);
      for (int s = 0; s < a.k; ++s) {
        const int drank = slot_rank[s], drow = slot_row[s];
        const float w = slot_w[s];
        if (drow < 0) continue;  // uniform over the team
        uint8_t* dst = h.window[drank] + a.recv_off + static_cast<size_t>(drow) * row_bytes;
        uint4* own = a.local_out && drank == h.rank
                         ? reinterpret_cast<uint4*>(a.local_out) + static_cast<size_t>(drow) * (a.H / 8)
                         : nullptr;
        if (a.fp8) {
          if (weighted) {
            q = quantize8(v, w, scale);
            if ((lane & 15) == 0)
              reinterpret_cast<float*>(h.window[drank] + a.scale_off)[static_cast<size_t>(drow) * groups + 2 * c + (lane >> 4)] = scale;
          }
          reinterpret_cast<uint2*>(dst)[c * 32 + lane] = q;
          if (own) own[c * 32 + lane] = weighted ? dequantize8(q, scale) : plain;
        } else {
          uint4 r = raw;
          if (weighted) {
            __nv_bfloat162* rp = reinterpret_cast<__nv_bfloat162*>(&r);
#pragma unroll
            for (int j = 0; j < 4; ++j) rp[j] = __floats2bfloat162_rn(v[2 * j] * w, v[2 * j + 1] * w);
          }
          reinterpret_cast<uint4*>(dst)[c * 32 + lane] = r;
          if (own) own[c * 32 + lane] = r;
        }
      }
    }
    if (a.fp8 && !weighted) {
      team.sync();
      for (int i = team.thread(); live && i < a.k * groups; i += team.warps * 32) {
        const int s = i / groups, g = i - s * groups;
        if (slot_row[s] >= 0)
          reinterpret_cast<float*>(h.window[slot_rank[s]] + a.scale_off)[static_cast<size_t>(slot_row[s]) * groups + g] = scale_buf[g];
      }
    }
  }
  grid_release();
  if (!last_cta_done(a.done)) return;
  // every row of this rank is on its way: tell all ranks, then wait until everybody's rows are here
  if (static_cast<int>(threadIdx.x) < h.nranks) {
    fence_acq_rel_sys();
    gin_signal(h, threadIdx.x, MOE_SIG_BASE + 1 * GIN_MAX_RANKS + h.rank, 1, GIN_SIGNAL_INC);
  }
  moe_wait_all(h, 1, a.epoch);
}

// What dispatch left in the window (rows from other ranks' tokens) -> out; rows past the last received
// one are zeroed. With `local_in_place` this rank's own rows are in `out` already, stored there by dispatch:
// 6 us for 32768 rows that are all local, where a copy of the window took 146.
__global__ void __launch_bounds__(MOE_THREADS)
    moe_collect_rows_kernel(GinDevHandle h, const int32_t* rows_ptr, size_t recv_off, size_t meta_off, int capacity_rows, int H,
                            int local_in_place, __nv_bfloat16* out) {
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int rows = min(*rows_ptr, capacity_rows);
  const int vec = H / 8;
  const MoeMeta* meta = reinterpret_cast<const MoeMeta*>(h.window[h.rank] + meta_off);
  const uint4* recv = reinterpret_cast<const uint4*>(h.window[h.rank] + recv_off);
  // A warp's lanes look their rows' records up together: one after the other they took 13 us for 32768 rows.
  const int all_warps = gridDim.x * warps, share = (capacity_rows + all_warps - 1) / all_warps, batch = share < 32 ? share : 32;
  for (int64_t r0 = static_cast<int64_t>(blockIdx.x * warps + warp) * batch; r0 < capacity_rows; r0 += static_cast<int64_t>(all_warps) * batch) {
    const int64_t mine = r0 + lane;
    const bool todo = lane < batch && mine < capacity_rows && !(local_in_place && mine < rows && meta[mine].src_rank == h.rank);
    for (unsigned left = __ballot_sync(0xffffffffu, todo); left; left &= left - 1) {
      const int r = static_cast<int>(r0) + __ffs(left) - 1;
      uint4* dst = reinterpret_cast<uint4*>(out) + static_cast<size_t>(r) * vec;
      if (r >= rows) {
        for (int v = lane; v < vec; v += 32) dst[v] = make_uint4(0, 0, 0, 0);
        continue;
      }
      const uint4* src = recv + static_cast<size_t>(r) * vec;
      constexpr int U = 4;
      for (int v0 = lane; v0 < vec; v0 += 32 * U) {
        uint4 tmp[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < vec) tmp[u] = src[v0 + 32 * u];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < vec) dst[v0 + 32 * u] = tmp[u];
      }
    }
  }
}

// ------------------------------------------------------------------------------------------ combine
struct CombineArgs {
  GinDevHandle h;
  const __nv_bfloat16* y;          // [rows][H] expert outputs in receive-buffer row order
  const int32_t* expert_offsets;   // [E/nranks + 1]; the last entry is the number of rows
  int experts_local;
  size_t meta_off, comb_off;       // window offsets: MoeMeta [rows] (local), bf16 [T][k][H] (on the source)
  const float* topk_w;             // [T][k] on the source, or null for an unweighted sum
  const int32_t* row_of;           // [T][k] on the source: cells whose row is < 0 were never sent
  const int32_t* local_row;        // [T][k] row of y for the cells whose expert is on the source itself, else -1
  __nv_bfloat16* cells_out;        // [T][k][H] a copy of every sent cell, or null
  int T, k, H;
  int team_warps;                  // TokenTeam
  __nv_bfloat16* out;              // [T][H]
  unsigned int senders;            // CTAs that send rows to other ranks, no more than run at once
  unsigned int* done;              // CTAs that have started, and 2^16 for every sender that is through
  uint64_t epoch;
};

__global__ void __launch_bounds__(MOE_THREADS, 4) moe_combine_kernel(CombineArgs a) {
  grid_wait();
  const GinDevHandle& h = a.h;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int rows = a.expert_offsets[a.experts_local];
  const int vec = a.H / 8;
  const MoeMeta* meta = reinterpret_cast<const MoeMeta*>(h.window[h.rank] + a.meta_off);
  // The CTAs that start first send, however they are numbered: whoever waits below waits for CTAs that are running.
  __shared__ unsigned int ticket;
  const unsigned int all_done = gridDim.x | (a.senders << 16);
  auto count = [&](unsigned int n) {   // rearmed by whoever counts last
    const unsigned int was = atomicAdd(a.done, n);
    if (was + n == all_done) *a.done = 0;
    return was;
  };
  if (threadIdx.x == 0) ticket = count(1) & 0xffffu;
  __syncthreads();
  const int cta = static_cast<int>(ticket);
  const bool sender = ticket < a.senders;
  for (int r = cta * warps + warp; sender && r < rows; r += a.senders * warps) {
    const MoeMeta m = meta[r];
    if (m.src_rank < 0 || m.src_rank >= h.nranks || m.token < 0 || m.token >= a.T || m.slot < 0 || m.slot >= a.k) {
      if (lane == 0) gin_record_error(h, DEV_ERR_BOUNDS);
      continue;
    }
    if (m.src_rank == h.rank) continue;   // summed from y below
    const uint4* src = reinterpret_cast<const uint4*>(a.y + static_cast<size_t>(r) * a.H);
    uint4* dst = reinterpret_cast<uint4*>(h.window[m.src_rank] + a.comb_off) +
                 (static_cast<size_t>(m.token) * a.k + m.slot) * vec;
    constexpr int U = 4;
    for (int v0 = lane; v0 < vec; v0 += 32 * U) {
      uint4 tmp[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + 32 * u < vec) tmp[u] = src[v0 + 32 * u];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + 32 * u < vec) dst[v0 + 32 * u] = tmp[u];
    }
  }
  // ---- all of this rank's rows are out: signal every source (the last sender does it) ...
  if (sender) {
    __shared__ int is_last;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      is_last = (count(1u << 16) >> 16) == a.senders - 1;
      __threadfence();
    }
    __syncthreads();
    if (is_last && static_cast<int>(threadIdx.x) < h.nranks) {
      fence_acq_rel_sys();
      gin_signal(h, threadIdx.x, MOE_SIG_BASE + 2 * GIN_MAX_RANKS + h.rank, 1, GIN_SIGNAL_INC);
    }
  }
  // ---- ... and every CTA waits for all ranks' rows before it reduces its share of the tokens
  if (!moe_wait_all(h, 2, a.epoch)) return;
  // A team per token: a wide one reads 4 KiB of each of the token's rows at a time. With a warp per
  // token every row is visited 512 bytes at a time by thousands of warps at once: 4096 tokens x 7168,
  // top-8, one rank took 194 us that way (314 with eight loads in flight per warp instead of four)
  // and 140 so, before the stores to the window's cells: 207 with them, on average over the forward call,
  // which copies the cells out as well, and the backward call, which does not; 299 (and 150 for the copy)
  // when every row was read back from its cell. Four cells' loads are issued together and added in the
  // order of the slots.
  uint4* comb = reinterpret_cast<uint4*>(h.window[h.rank] + a.comb_off);
  const TokenTeam team(a.team_warps);
  __shared__ float team_w[TokenTeam::WARPS][MOE_MAX_TOPK];
  __shared__ int team_row[TokenTeam::WARPS][MOE_MAX_TOPK];   // row of y, -1: the cell in the window, -2: never sent
  float* slot_w = team_w[team.team];
  int* slot_row = team_row[team.team];
  for (int t0 = cta * team.teams; t0 < a.T; t0 += gridDim.x * team.teams) {
    const int t = t0 + team.team;
    const bool on = t < a.T;
    team.sync();   // the slots of the token before have been read
    if (on && team.thread() < a.k) {
      const int i = t * a.k + team.thread();
      const int sent = a.row_of[i], own = a.local_row[i];
      int row = sent < 0 ? -2 : own;
      if (row >= rows) {
        gin_record_error(h, DEV_ERR_BOUNDS);
        row = -2;
      }
      slot_row[team.thread()] = row;
      slot_w[team.thread()] = a.topk_w ? a.topk_w[i] : 1.f;
    }
    team.sync();
    constexpr int U = 4;
    for (int v = team.thread(); on && v < vec; v += team.warps * 32) {
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (int s0 = 0; s0 < a.k; s0 += U) {
        uint4 q[U];
        int row[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          row[u] = s0 + u < a.k ? slot_row[s0 + u] : -2;
          if (row[u] == -2) continue;
          q[u] = row[u] >= 0 ? reinterpret_cast<const uint4*>(a.y)[static_cast<size_t>(row[u]) * vec + v]
                             : comb[(static_cast<size_t>(t) * a.k + s0 + u) * vec + v];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (row[u] == -2) continue;
          const size_t cell = (static_cast<size_t>(t) * a.k + s0 + u) * vec + v;
          if (row[u] >= 0) comb[cell] = q[u];   // what another rank sent is there already
          if (a.cells_out) reinterpret_cast<uint4*>(a.cells_out)[cell] = q[u];
          const float ws = slot_w[s0 + u];
          const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q[u]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc[2 * j] += ws * __low2float(p[j]);
            acc[2 * j + 1] += ws * __high2float(p[j]);
          }
        }
      }
      __nv_bfloat162 o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
      reinterpret_cast<uint4*>(a.out + static_cast<size_t>(t) * a.H)[v] = *reinterpret_cast<const uint4*>(o);
    }
  }
}

// d(weight)[t][s] = <d_out[t], cell[t][s]> over the combine buffer kept from the forward pass.
__global__ void __launch_bounds__(MOE_THREADS)
    moe_combine_wgrad_kernel(const __nv_bfloat16* dout, const __nv_bfloat16* comb, const int32_t* row_of, float* dw, int T,
                             int k, int H) {
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int vec = H / 8;
  for (int i = blockIdx.x * warps + warp; i < T * k; i += gridDim.x * warps) {
    const int t = i / k;
    float acc = 0.f;
    if (row_of[i] >= 0) {
      const uint4* a = reinterpret_cast<const uint4*>(dout + static_cast<size_t>(t) * H);
      const uint4* b = reinterpret_cast<const uint4*>(comb + static_cast<size_t>(i) * H);
      constexpr int U = 4;
      for (int v0 = lane; v0 < vec; v0 += 32 * U) {
        uint4 x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < vec) {
            x[u] = a[v0 + 32 * u];
            y[u] = __ldcs(b + v0 + 32 * u);   // the token's gradient is read k times, a cell once: 92 -> 87 us
          }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (v0 + 32 * u >= vec) break;
          const __nv_bfloat162* px = reinterpret_cast<const __nv_bfloat162*>(&x[u]);
          const __nv_bfloat162* py = reinterpret_cast<const __nv_bfloat162*>(&y[u]);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc += __low2float(px[j]) * __low2float(py[j]) + __high2float(px[j]) * __high2float(py[j]);
        }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) dw[i] = acc;
  }
}

// 8-element vectors of a row that a warp takes at a time: four per lane.
constexpr int DEQUANT_PIECE = 128;
__host__ __device__ inline int dequant_pieces(int H) { return (H / 8 + DEQUANT_PIECE - 1) / DEQUANT_PIECE; }

// fp8 (e4m3) rows with one fp32 scale per 128 elements -> bf16. A warp takes 1024 elements of a row at a time, a lane 8
// values, so that the warp's stores are 512 consecutive bytes, and four such loads are in flight: 32768 x
// 7168 in 125 us (5.6 TB/s), 175 with a grid-stride loop over single vectors; 128 rows 8 us, 16 with a warp
// for a whole row. With zero_tail the rows past
// the last received one are written as zeros, in place of a fill of the whole output before (120 us). With `meta`
// the rows of rank `here` are in `out` already. Dispatch and combine of 4096 x 7168, top-8, with their gradients on one
// rank: 814 us; reading every row back here cost 33 more.
__global__ void __launch_bounds__(MOE_THREADS)
    fp8_dequant_rows_kernel(const uint8_t* q, const float* scales, __nv_bfloat16* out, const int32_t* rows_ptr, int rows_max,
                            int H, int zero_tail, const MoeMeta* meta, int here) {
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int rows = rows_ptr ? min(*rows_ptr, rows_max) : rows_max;
  const int vec = H / 8, groups = H / 128, pieces = dequant_pieces(H);
  const int64_t items = static_cast<int64_t>(zero_tail ? rows_max : rows) * pieces;
  const int64_t all_warps = static_cast<int64_t>(gridDim.x) * warps;
  // Pieces of one warp at a time: its lanes look their rows up together, and the warp goes on to those it has to do.
  const int64_t share = (items + all_warps - 1) / all_warps;
  const int batch = !meta ? 1 : share < 32 ? static_cast<int>(share) : 32;
  for (int64_t i0 = (static_cast<int64_t>(blockIdx.x) * warps + warp) * batch; i0 < items; i0 += all_warps * batch) {
    const int64_t mine = i0 + lane;
    bool todo = lane < batch && mine < items;
    if (meta && todo) {
      const int64_t r = mine / pieces;
      todo = r >= rows || meta[r].src_rank != here;
    }
    for (unsigned left = __ballot_sync(0xffffffffu, todo); left; left &= left - 1) {
      const int64_t i = i0 + __ffs(left) - 1;
      const int r = static_cast<int>(i / pieces);
      const int v0 = static_cast<int>(i - static_cast<int64_t>(r) * pieces) * DEQUANT_PIECE + lane;
      uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(r) * H);
      constexpr int U = DEQUANT_PIECE / 32;
      if (r >= rows) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (v0 + 32 * u < vec) dst[v0 + 32 * u] = make_uint4(0, 0, 0, 0);
        continue;
      }
      const uint2* src = reinterpret_cast<const uint2*>(q + static_cast<size_t>(r) * H);
      const float* sc = scales + static_cast<size_t>(r) * groups;
      uint2 raw[U];
      float s[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (v0 + 32 * u < vec) {
          raw[u] = src[v0 + 32 * u];
          s[u] = sc[(v0 + 32 * u) / 16];
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (v0 + 32 * u >= vec) break;
        dst[v0 + 32 * u] = dequantize8(raw[u], s[u]);
      }
    }
  }
}

static uint64_t g_moe_epoch[64][3] = {};

// CTAs for T tokens, of which one works on per_cta at a time. Four run on an SM; with no more than that the SMs that memory serves
// last finish last, and with several times as many the others take their work: 4096 x 7168, top-8, fp8 dispatch 147 -> 134 us,
// combine 262 -> 246, in the backward pass 186 -> 165 and 169 -> 168, the weights' gradient (moe_grid) 98 -> 92 (8 per SM: 146 and
// 183 for the dispatches, 64: 134 and 166).
static int token_grid(int T, int per_cta) {
  return std::min((T + per_cta - 1) / per_cta, sm_count() * CTAS_PER_SM);
}
static int moe_grid(int64_t work_warps, int per_sm = 4) {
  const int per_cta = MOE_THREADS / 32;
  const int64_t grid = (work_warps + per_cta - 1) / per_cta;
  const int cap = sm_count() * per_sm;
  return grid > cap ? cap : grid < 1 ? 1 : static_cast<int>(grid);
}

}  // namespace b200

extern "C" {
using namespace b200;

// Collective over the communicator. `done` is a zero-initialised device word private to this call
// site; cnt_local must be zero on the first call (the kernel leaves it zero).
int b200_moe_route(int comm, const void* topk_idx, int T, int k, int E, size_t cnt_off, void* cnt_local, void* dest_base,
                   void* expert_offsets, void* cursor, void* done, void* stream) {
  ensure_context();
  const GinDevHandle* hp = comm_handle(comm);
  if (!hp || comm < 0 || comm >= 64) return B200_ERR_BAD_ARG;
  GinDevHandle h = *hp;
  if (E <= 0 || E > MOE_MAX_EXPERTS || E % h.nranks || k <= 0 || k > MOE_MAX_TOPK || T <= 0) return B200_ERR_BAD_ARG;
  if (cnt_off % 16 || cnt_off + 2ull * h.nranks * E * 4 > h.window_bytes) return B200_ERR_BAD_ARG;
  RouteArgs a{h, static_cast<const int32_t*>(topk_idx), T, k, E, cnt_off, static_cast<int32_t*>(cnt_local),
              static_cast<int32_t*>(dest_base), static_cast<int32_t*>(expert_offsets), static_cast<int32_t*>(cursor),
              static_cast<unsigned int*>(done), ++g_moe_epoch[comm][0]};
  int grid = (T * k + MOE_THREADS * 2 - 1) / (MOE_THREADS * 2);   // a thread's loads wait for one another
  if (grid > 128) grid = 128;
  launch_dependent(moe_route_kernel, grid, MOE_THREADS, 0, static_cast<cudaStream_t>(stream), a);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// Collective. Window layout on every rank: payload rows at recv_off (H bytes per row for fp8, 2H
// for bf16), fp32 scales at scale_off (H/128 per row, fp8 only), 16-byte records at meta_off.
int b200_moe_dispatch(int comm, const void* x, const void* topk_idx, const void* topk_w, int T, int k, int H, int E, int fp8,
                      int use_saved_rows, int scale_by_weight, const void* dest_base, void* cursor, void* row_of, void* local_row,
                      void* local_out, size_t recv_off, size_t scale_off, size_t meta_off, int capacity_rows, void* done, void* stream) {
  ensure_context();
  const GinDevHandle* hp = comm_handle(comm);
  if (!hp || comm < 0 || comm >= 64) return B200_ERR_BAD_ARG;
  GinDevHandle h = *hp;
  if (E <= 0 || E % h.nranks || k <= 0 || k > MOE_MAX_TOPK || H % 256 || T <= 0) return B200_ERR_BAD_ARG;
  if (H / 128 > 64) return B200_ERR_TOO_LARGE;
  const size_t row_bytes = fp8 ? static_cast<size_t>(H) : static_cast<size_t>(H) * 2;
  if (recv_off % 16 || meta_off % 16 || scale_off % 16) return B200_ERR_BAD_ARG;
  if (!local_row || reinterpret_cast<uintptr_t>(local_out) % 16) return B200_ERR_BAD_ARG;
  if (recv_off + row_bytes * capacity_rows > h.window_bytes || meta_off + 16ull * capacity_rows > h.window_bytes ||
      (fp8 && scale_off + 4ull * (H / 128) * capacity_rows > h.window_bytes))
    return B200_ERR_BAD_ARG;
  DispatchArgs a{h, static_cast<const __nv_bfloat16*>(x), static_cast<const int32_t*>(topk_idx),
                 static_cast<const float*>(topk_w), T, k, H, E, TokenTeam::warps_for(T, H), fp8, use_saved_rows, scale_by_weight,
                 static_cast<const int32_t*>(dest_base), static_cast<int32_t*>(cursor), static_cast<int32_t*>(row_of),
                 static_cast<int32_t*>(local_row), static_cast<__nv_bfloat16*>(local_out), recv_off, scale_off, meta_off, capacity_rows, static_cast<unsigned int*>(done), ++g_moe_epoch[comm][1]};
  const int per_cta = TokenTeam::WARPS / a.team_warps;
  launch_dependent(moe_dispatch_kernel, token_grid(T, per_cta), MOE_THREADS, 0, static_cast<cudaStream_t>(stream), a);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// Rows of the last dispatch (bf16 payload) -> out[capacity_rows][H], see moe_collect_rows_kernel.
int b200_moe_collect_rows(int comm, const void* rows_ptr, size_t recv_off, size_t meta_off, int capacity_rows, int H,
                          int local_in_place, void* out, void* stream) {
  ensure_context();
  const GinDevHandle* hp = comm_handle(comm);
  if (!hp || !rows_ptr || !out || H % 8 || capacity_rows <= 0 || recv_off % 16 || meta_off % 16) return B200_ERR_BAD_ARG;
  if (recv_off + 2ull * H * capacity_rows > hp->window_bytes || meta_off + 16ull * capacity_rows > hp->window_bytes)
    return B200_ERR_BAD_ARG;
  launch_dependent(moe_collect_rows_kernel, moe_grid(capacity_rows), MOE_THREADS, 0, static_cast<cudaStream_t>(stream),
      *hp, static_cast<const int32_t*>(rows_ptr), recv_off, meta_off, capacity_rows, H, local_in_place,
      static_cast<__nv_bfloat16*>(out));
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// Collective. Every CTA of this kernel waits for the other ranks' rows and for this rank's senders, which are the first CTAs to
// start: as many as run at once.
int b200_moe_combine(int comm, const void* y, const void* expert_offsets, int experts_local, size_t meta_off, size_t comb_off,
                     const void* topk_w, const void* row_of, const void* local_row, void* cells_out, int T, int k, int H,
                     void* out, void* done, void* stream) {
  ensure_context();
  const GinDevHandle* hp = comm_handle(comm);
  if (!hp || comm < 0 || comm >= 64) return B200_ERR_BAD_ARG;
  GinDevHandle h = *hp;
  if (H % 8 || k <= 0 || k > MOE_MAX_TOPK || T <= 0 || !local_row) return B200_ERR_BAD_ARG;
  if (comb_off % 16 || comb_off + static_cast<size_t>(T) * k * H * 2 > h.window_bytes) return B200_ERR_BAD_ARG;
  CombineArgs a{h, static_cast<const __nv_bfloat16*>(y), static_cast<const int32_t*>(expert_offsets), experts_local, meta_off,
                comb_off, static_cast<const float*>(topk_w), static_cast<const int32_t*>(row_of),
                static_cast<const int32_t*>(local_row), static_cast<__nv_bfloat16*>(cells_out), T, k, H, TokenTeam::warps_for(T, H),
                static_cast<__nv_bfloat16*>(out), 0, static_cast<unsigned int*>(done), ++g_moe_epoch[comm][2]};
  const int per_cta = TokenTeam::WARPS / a.team_warps;
  int per_sm = 0;
  B200_CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, moe_combine_kernel, MOE_THREADS, 0));
  if (per_sm < 1) return B200_ERR_BAD_ARG;
  if (per_sm > 4) per_sm = 4;
  a.senders = sm_count() * per_sm;
  const int grid = std::max(static_cast<int>(a.senders), token_grid(T, per_cta));
  launch_dependent(moe_combine_kernel, grid, MOE_THREADS, 0, static_cast<cudaStream_t>(stream), a);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

int b200_moe_combine_wgrad(const void* dout, const void* comb, const void* row_of, void* dw, int T, int k, int H, void* stream) {
  ensure_context();
  if (H % 8) return B200_ERR_BAD_ARG;
  launch_dependent(moe_combine_wgrad_kernel, moe_grid(T * k, CTAS_PER_SM), MOE_THREADS, 0, static_cast<cudaStream_t>(stream),
      static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(comb), static_cast<const int32_t*>(row_of),
      static_cast<float*>(dw), T, k, H);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// rows_ptr (device int32, may be null) limits the work to the rows actually received; with zero_tail the
// others are written as zeros.
int b200_fp8_dequant_rows(const void* q, const void* scales, void* out, const void* rows_ptr, int rows_max, int H, int zero_tail,
                          void* stream) {
  ensure_context();
  if (H % 128) return B200_ERR_BAD_ARG;
  launch_dependent(fp8_dequant_rows_kernel, moe_grid(static_cast<int64_t>(rows_max) * dequant_pieces(H)), MOE_THREADS, 0, static_cast<cudaStream_t>(stream),
      static_cast<const uint8_t*>(q), static_cast<const float*>(scales), static_cast<__nv_bfloat16*>(out),
      static_cast<const int32_t*>(rows_ptr), rows_max, H, zero_tail, nullptr, 0);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

// The fp8 rows of the last dispatch that other ranks sent -> out[capacity_rows][H]; this rank's own are there already
// (dispatch's local_out). Rows past the last received one become zeros.
int b200_moe_collect_rows_fp8(int comm, const void* rows_ptr, size_t recv_off, size_t scale_off, size_t meta_off, int capacity_rows,
                              int H, void* out, void* stream) {
  ensure_context();
  const GinDevHandle* hp = comm_handle(comm);
  if (!hp || !rows_ptr || !out || H % 128 || capacity_rows <= 0 || (recv_off | scale_off | meta_off) % 16) return B200_ERR_BAD_ARG;
  const size_t rows = capacity_rows;
  if (recv_off + H * rows > hp->window_bytes || scale_off + 4ull * (H / 128) * rows > hp->window_bytes ||
      meta_off + 16ull * rows > hp->window_bytes)
    return B200_ERR_BAD_ARG;
  const uint8_t* window = static_cast<const uint8_t*>(hp->window[hp->rank]);
  launch_dependent(fp8_dequant_rows_kernel, moe_grid(static_cast<int64_t>(rows) * dequant_pieces(H)), MOE_THREADS, 0, static_cast<cudaStream_t>(stream),
      window + recv_off, reinterpret_cast<const float*>(window + scale_off), static_cast<__nv_bfloat16*>(out),
      static_cast<const int32_t*>(rows_ptr), capacity_rows, H, 1, reinterpret_cast<const MoeMeta*>(window + meta_off), hp->rank);
  B200_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // extern "C"

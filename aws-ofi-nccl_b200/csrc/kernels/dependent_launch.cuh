// Kernels that start while the one before them in the stream ends (programmatic dependent launch).
//
// A kernel launched with launch_dependent may be scheduled once every CTA of the kernel before it has called grid_release (or
// has exited), so that its launch, its barriers, its tensor memory and its first instructions are under way while the last
// tiles of that kernel are stored. Every CTA of it calls grid_wait before it touches global memory: that returns when the
// kernel before it, and by the same rule everything before that, has ended and its writes are visible. Behind a kernel that
// never releases, or anything that is no kernel, such a launch is an ordinary one. What it gains is 2 to 2.5 us between two
// kernels: forward and both gradients of 128 x 4096 x 14336, three of them, take 82.6 us for 89.6, 1000 x 2568 x 5160 85 for 90
// (two), SwiGLU of 4096 x 14336 and its gradient 147.6 for 150.2. The products fused with a
// collective, whose CTAs wait for other ranks' tiles, are launched ordinarily.
//
// Where a kernel takes const __restrict__ pointers (or restrict ones that it only reads from) the compiler may move loads through
// them anywhere, before grid_wait too: such kernels use their pointers as after_wait returns them. What it then knows of them no longer is that stores leave
// the loads alone: a loop's loads are no longer batched across its stores.
//
// grid_release stands near the end of a kernel's work, or at the start of kernels of several waves, where the last CTA to start
// is what counts: from then on CTAs of the next kernel hold what room there is on an SM,
// which kernels of other streams could use. Kernels without shared memory, the collectives among them, fit beside a product's CTAs on an SM and are not
// held up (copies and sums beside a chain of 4096 x 4096 x 4096 take as long as before, 110 and 11 us); another product waits for an SM of its own, 87 us for
// 72 there. A product that leaves SMs free for others (max_ctas) is launched ordinarily and releases none, which costs it those 2 us: of
// 2048 x 2048 x 2048 on 100 or 74 SMs dependents came up 4.8 us before the end, one every 24.3 us, 27.5 so.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace b200 {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// grid_release at the start of a kernel of which CTAS run on an SM at once. Not where the grid is half to four fifths of what runs at once: the
// next kernel's CTAs then fill what is left of the SMs, unevenly, and the rest of them follows as CTAs end. The same kernel launched again and again,
// rotary split of 731 x 48 heads of 64 (548 CTAs of 888) 5.9 us so and 4.9 with the release at the end, RMSNorm of 1000 x 2048 (500 of 888) 4.6 and
// 4.0, AdamW of 686592 (336 of 592) 6.7 and 6.2, cross-entropy of 149 x 28672 (298 of 592) 10.8 and 9.5; with fewer or more CTAs the early release is up to 0.3 us ahead.
// One piece of assembly, since the compiler gave some kernels four registers more for the same in C++, and an SM a CTA of them less.
template <int CTAS>
__device__ __forceinline__ void grid_release_at_start() {
  asm volatile(
      "{\n"
      ".reg .pred few, many;\n"
      ".reg .u32 sms, ctas, half, most;\n"
      "mov.u32 sms, %%nsmid;\n"
      "mov.u32 ctas, %%nctaid.x;\n"
      "mul.lo.u32 ctas, ctas, 10;\n"
      "mul.lo.u32 half, sms, %0;\n"
      "mul.lo.u32 most, sms, %1;\n"
      "setp.lt.u32 few, ctas, half;\n"
      "setp.gt.or.u32 many, ctas, most, few;\n"
      "@many griddepcontrol.launch_dependents;\n"
      "}\n" ::"n"(5 * CTAS), "n"(8 * CTAS)
      : "memory");
}

template <typename P>
__device__ __forceinline__ void written_before(P& pointer) {
  asm volatile("" : "+l"(pointer)::"memory");
}
template <typename... P>
__device__ __forceinline__ void after_wait(P&... pointers) {
  grid_wait();
  (written_before(pointers), ...);
}

// With `dependent` false an ordinary launch, whose CTAs come up when the kernel before has ended. The launch error, if any, is left for
// cudaGetLastError.
template <typename... P, typename... A>
void launch_after(bool dependent, void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = dependent;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, static_cast<P>(std::forward<A>(args))...);
}
template <typename... P, typename... A>
void launch_dependent(void (*kern)(P...), int grid, int threads, size_t smem, cudaStream_t stream, A&&... args) {
  launch_after(true, kern, grid, threads, smem, stream, std::forward<A>(args)...);
}

}  // namespace b200

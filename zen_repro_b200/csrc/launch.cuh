// Kernels that may be set up while the previous kernel of the stream still runs (programmatic dependent launch).
//
// Between two dependent kernels of a stream the GPU idles: the first one drains, the second one is fetched and started on
// every SM, initialises barriers and allocates tensor memory.  Back to back, an 8192 x 768 x 768 product took 16.8 us of which
// the kernel itself ran 13.4, 0.9 of them for its setup (12 forward layers of 8192 x 768: 3640 -> 3555 us).  A kernel launched with `launch` starts as soon as every CTA of its
// predecessor has called `trigger` (or ended) and there is room for it, and stops at `wait` until the predecessor has
// ended and its writes are visible.
//
//  * Everything a kernel reads or writes in global memory comes after `wait`.  Since every kernel waits for its predecessor's
//    end, the end of a kernel implies the end of all earlier ones of the stream.
//  * A kernel that allocates tensor memory triggers after its allocation: a successor's CTA on the same SM could otherwise
//    allocate first and keep it until this kernel ends.
//  * Input pointers of such kernels are not `const __restrict__`: the compiler reads those through the read-only path, which
//    promises that nobody writes the data while the kernel runs, also before `wait`, and may move the loads across it.
//  * Kernels that wait for other GPUs are launched plainly.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace zen_pdl {

// Kernels launched by this library in this process (zen_launch_count; a captured launch counts when it is captured).  Every launch
// of the library goes through this file, which is what makes the count one.
inline std::atomic<long long> g_launched{0};
inline int counted(cudaError_t e) {
  if (e == cudaSuccess) g_launched.fetch_add(1, std::memory_order_relaxed);
  return (int)e;
}

__device__ __forceinline__ void trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// First statement of a kernel without a setup phase.
__device__ __forceinline__ void enter() {
  trigger();
  wait();
}

// `early` = false: an ordinary launch.
template <typename... P, typename... A>
inline int launch_if(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return counted(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}
template <typename K, typename... A>
inline int launch(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_if(true, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}
template <typename K, typename... A>
inline int plain(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_if(false, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}
// Kernels that stream memory through a grid of several CTAs per SM start early only when they are small (at most two CTAs per
// SM): waiting CTAs of a large grid settle unevenly over the SMs beside their predecessor's, which cost up to a third of a
// kernel's time (64 M x 8 sparse all-reduce 820 -> 1080 us), while the gap they hide is 2 to 3 us.
template <typename K, typename... A>
inline int launch_small(K kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  return launch_if((unsigned long long)grid.x * grid.y * grid.z <= 296, kernel, grid, block, smem, st, static_cast<A&&>(args)...);
}

}  // namespace zen_pdl

// Helpers shared by the kernel launchers.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace mdt {
// Kernels follow one another on a stream by programmatic dependent launch: a kernel may be set up on the GPU while its predecessor
// still runs, and waits itself (after_predecessor) before it reads or writes anything that other kernels touch, until the
// predecessor has finished and its writes are visible.  Every kernel launched with launch_after has to call after_predecessor first
// of all, or after set-up that stays in its own shared memory, TMEM and parameters; its own successor may then be set up in turn.
// TMEM is allocated before a successor is admitted: that one allocates too before it waits, and an allocation waits without limit.
// A two-layer training step is 600 to 900 launches of 2 to 400 microseconds with about 2 us between any two: 19.2 -> 18.7 ms with
// adapters on attention, 23.0 -> 21.9 with adapters everywhere; logits of a 77-token prompt (42 launches) 1.21 -> 1.14 ms.
// Grids of many rounds of CTAs keep plain launches: every CTA would pay for the wait, which small ones feel (attention backward of
// 19 120 tokens: the 4 900 CTAs before the main kernel 126 us plain, 141 so; the main kernel's 6 160 CTAs 3.0 to 3.2 ms either way).
// Kernels that wait for other GPUs or streams keep plain launches (csrc/comm.cu), or do not admit successors early: a successor's CTAs
// could take the place of those that are waited for.
inline int early_setup_pays(long long ctas) { return ctas <= 2048 ? 1 : 0; }
template <class... P, class... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = early_setup_pays((long long)grid.x * grid.y * grid.z);
  cfg.attrs = &attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void admit_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_predecessor() { wait_for_predecessor(); admit_successor(); }
#endif

// Number of SMs of the current device (grids are sized in multiples of it); cached per device ordinal.
inline int sm_count_of_current_device() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}
}  // namespace mdt

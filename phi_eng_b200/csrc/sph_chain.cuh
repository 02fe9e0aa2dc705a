// Launches of the substep chain: each kernel's launch is set up while the one
// before it in the stream drains, and it waits on the device for that one's end.
// A step is five short kernels: 20 steps of 32,499 particles 447 -> 434 us, 10
// steps of 2^18 403 -> 391 us, of 2^20 944 -> 933 us.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace phieng {

// First statement of every kernel that launch_chained starts: waits until the
// kernels before this one are complete and their writes visible. No memory is
// touched before it, and every thread calls it, so a kernel's end implies the
// end of all before it. The pointers are those it reads and an earlier kernel of
// the chain may write: passed through here they are no longer known to be
// unwritten during the kernel, so that no load through them moves to before the
// wait. No kernel lets the next one's blocks in before its own have ended: their
// registers are missing to the kernel at work (2^18 particles 391 -> 406 us,
// 47x41x42 in 3D 2912 -> 3031 us).
template <class... P>
__device__ __forceinline__ void chain_wait(P&... p) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (..., [](auto& q) { asm volatile("" : "+l"(q)::"memory"); }(p));
}

// <<<grid, block, smem, st>>> of a kernel that begins with chain_wait.
template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(a)...);
}

}  // namespace phieng

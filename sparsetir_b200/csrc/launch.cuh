// Launches that overlap with the end of the launch before them on the stream (programmatic dependent launch).
//
// Without it a kernel's blocks are scheduled only when the kernel before has ended and its writes are flushed,
// one to two microseconds in which the GPU does nothing (calls in a row, us, without / with: CSR SpMM 3,000 rows of 5
// entries, F = 32, 6.15 / 3.9; BSR 1,024^2, F = 128, 8.2 / 5.5; RGMS of 20,000 edges 19.5 / 14.4; hyb SpMM at F = 32 on
// 169 k nodes 19.1 / 17.5).  A kernel launched by launch_chained() is scheduled as the blocks of the one before leave
// their SMs, and calls chain_enter() before its first access to global memory:
//  - the wait holds every thread until all launches before this one on the stream have ended and their writes are
//    visible, whoever made them, so that the order of a stream is what it always was;
//  - the trigger allows the next launch to be scheduled once every block of this one has got that far.  A
//    block of the next launch that is resident early only waits; no block of this launch is still to be scheduled then,
//    so it takes nobody's place.
// Every block of such a kernel must call chain_enter(): a launch that ended without having waited would let the next
// one pass its wait while the one before is still running.
#ifndef SPARSETIR_B200_LAUNCH_CUH_
#define SPARSETIR_B200_LAUNCH_CUH_

#include <cuda_runtime.h>

#include <cstddef>

namespace sptir {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
  chain_wait();
  chain_trigger();
}

// Where a call of many stored entries starts (0.3 ms and more), chaining is not worth what it can cost: blocks of the
// next kernel that become resident early are placed by what the leaving ones make room for, not evenly over the SMs
// (attention over 20 M positions: 726 us without, 731 with; over 4.5 M: 102 without, 94 with).
constexpr int kChainEntries = 8 << 20;

// An error of the launch is the runtime's last error, which SPTIR_LAUNCH_OK reads, as behind <<<>>>.
template <class... Params, class... Args>
inline void launch_chained_if(bool chained, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = chained ? 1 : 0;
  (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <class... Params, class... Args>
inline void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  launch_chained_if(true, kernel, grid, block, smem, stream, args...);
}

}  // namespace sptir
#endif  // SPARSETIR_B200_LAUNCH_CUH_

// Launches that overlap with the end of the launch before them on the stream (programmatic dependent launch).
//
// Without it a kernel's blocks are scheduled only when the kernel before has ended and its writes are flushed,
// one to two microseconds in which the GPU does nothing (calls in a row, us, without / with: CSR SpMM 3,000 rows of 5
// entries, F = 32, 6.15 / 3.5; BSR 1,024^2, F = 128, 8.2 / 5.5; RGMS of 20,000 edges 19.5 / 14.4; hyb SpMM at F = 32 on
// 169 k nodes 19.1 / 17.4).  A kernel launched by launch_chained() calls chain_wait() before its first access to global
// memory: every thread waits until all launches before this one on the stream have ended and their writes are visible,
// whoever made them, so that the order of a stream is what it always was.  It is scheduled when every block of the launch
// before has ended or called chain_trigger().
//  - Kernels of many small blocks do not trigger: their ends come close together, and the next launch then finds the SMs
//    empty.  Scheduled earlier, its blocks fill the SMs that come free first, and a launch of less than a full
//    wave lies unevenly over them (us, triggered at the start / not: SDDMM 20 k rows, F = 512, 34.8 / 29.0, CSR SpMM
//    20 k rows, F = 512, 43.3 / 38.8, 4,096 rows 5.1 / 4.5).
//    The gather of rgms_f16.cu does so all the same: behind it comes one block per SM that sets up barriers and waits (20.7 /
//    21.3 at 64 -> 64 on 22 k nodes, 16.8 / 17.9 at 32 -> 32).
//  - Kernels of one wave of blocks, one or two to an SM, trigger behind the wait, so that the next one's set-up overlaps:
//    no block of this launch is still to be scheduled then, and a block of the next one only waits.
//  - A kernel that takes tensor memory triggers when its block has it (behind the barrier that publishes the address).
//    The next launch may take some before it waits, and would keep it until this one has ended: a block of this one that
//    had yet to take its own on the same SM would wait for it for good.
// Such a kernel lives while the one before it still writes what it is going to read, so it reads its operands with
// ld_global().  __ldg(), and what the compiler makes of a const __restrict__ pointer (ld.global.nc), promise that the
// memory does not change as long as the kernel lives: the load may be moved ahead of the wait, or be answered by
// what another block of the SM has brought before it.
// At least one block of every such kernel must have waited when the launch ends, or the next one could pass its wait
// while the one before is still running.  All blocks of all of them do, but for the gather of rgms_f16.cu, which runs
// beside the launch before it: there a flag, set by that launch behind its own wait (st_release) and read by this one
// (ld_acquire), stands for the wait, and one block waits in the end.
#ifndef SPARSETIR_B200_LAUNCH_CUH_
#define SPARSETIR_B200_LAUNCH_CUH_

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace sptir {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
  chain_wait();
  chain_trigger();
}

// Loads of 2, 4, 8 or 16 bytes that stay behind chain_wait().
template <class T>
__device__ __forceinline__ T ld_global(const T* p) {
  T v;
  if constexpr (sizeof(T) == 16) {
    uint4& r = reinterpret_cast<uint4&>(v);
    asm volatile("ld.global.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  } else if constexpr (sizeof(T) == 8) {
    uint2& r = reinterpret_cast<uint2&>(v);
    asm volatile("ld.global.v2.b32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
  } else if constexpr (sizeof(T) == 4) {
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(reinterpret_cast<uint32_t&>(v)) : "l"(p));
  } else {
    static_assert(sizeof(T) == 2, "2, 4, 8 or 16 bytes");
    asm volatile("ld.global.b16 %0, [%1];" : "=h"(reinterpret_cast<uint16_t&>(v)) : "l"(p));
  }
  return v;
}

// A flag between launches that run side by side: what happened before it was set is visible to who has read it.
__device__ __forceinline__ void st_release(int32_t* p, int32_t v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int32_t ld_acquire(const int32_t* p) {
  int32_t v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// From this many stored entries on (0.1 ms and more) CSR SpMM by entries, SDDMM and softmax are launched as usual: a
// microsecond is nothing to them.  The kernels with tensor memory, hyb, the condensed and the row-wise SpMM are chained
// whatever their size.
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

// The register-level matrix instruction (m16n8k16, fp16 operands, fp32 sums) for kernels whose right
// operand is a gather of rows: both operands are loaded from global memory in the layout that the
// instruction reads, nothing goes through shared memory.
//  - Which row of a group of 16 plays which k is free as long as both operands agree: the four k's of lane l
//    are rows 4(l%4) .. 4(l%4)+3 of the group, so a lane's part of a row of the left operand is 8 bytes.
//  - Which feature plays which column is free too: lane group l/4 holds 16 bytes (8 features, one "piece")
//    of each of its rows and instruction j takes the j-th feature of every piece.  64 features make
//    whole 128-byte lines per row, and a lane ends with 8 consecutive features of a result row.
#ifndef SPARSETIR_B200_MMA16_CUH_
#define SPARSETIR_B200_MMA16_CUH_

#include <cuda_fp16.h>

#include <cstdint>

namespace sptir {
namespace mma16 {

constexpr int kSlab = 64;  // features per warp

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc[mt][j][c]: instruction j = feature j of every piece; c = 0, 1: row 16 mt + lane/4, pieces 2(lane%4)
// and the next; c = 2, 3: row 16 mt + lane/4 + 8.
template <int MT>
__device__ __forceinline__ void clear(float (&acc)[MT][8][4]) {
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[mt][j][c] = 0.f;
}

// v: the lane's piece of its four rows; av[mt]: its 8 bytes of row lane/4 (words 0, 2) and lane/4 + 8 (1, 3)
template <int MT>
__device__ __forceinline__ void multiply(float (&acc)[MT][8][4], const uint4 (&v)[4], const uint32_t (&av)[MT][4]) {
  auto two = [&](int j, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    const uint32_t lo0 = __byte_perm(w0, w1, 0x5410), lo1 = __byte_perm(w2, w3, 0x5410);
    const uint32_t hi0 = __byte_perm(w0, w1, 0x7632), hi1 = __byte_perm(w2, w3, 0x7632);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) mma16816(acc[mt][j], av[mt], lo0, lo1);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) mma16816(acc[mt][j + 1], av[mt], hi0, hi1);
  };
  two(0, v[0].x, v[1].x, v[2].x, v[3].x);
  two(2, v[0].y, v[1].y, v[2].y, v[3].y);
  two(4, v[0].z, v[1].z, v[2].z, v[3].z);
  two(6, v[0].w, v[1].w, v[2].w, v[3].w);
}

}  // namespace mma16
}  // namespace sptir
#endif  // SPARSETIR_B200_MMA16_CUH_

// The register-level matrix instruction (m16n8k16, fp16 operands, fp32 sums) for kernels whose right operand is a gather of
// rows.  Which row of a group of 16 plays which k is free as long as both operands agree: the four k's of lane l are rows
// 4(l%4) .. 4(l%4)+3 of the group, so a lane's part of a row of the left operand is 8 bytes.  The rows come in one of two ways:
//  - Straight from global memory into the registers that the instruction reads, the shortest way for a few groups (tcspmm).  Which
//    feature plays which column is free too: lane group l/4 holds 16 bytes (8 features, one "piece") of each of its rows and
//    instruction j takes the j-th feature of every piece; a lane ends with 8 consecutive features of a result row.  Four
//    neighbouring lanes hold four rows, so a load takes 16 clocks of the L1 data path where whole lines take 6.
//  - Through shared memory of the warp, by asynchronous copies of whole lines a few groups ahead, read back transposed
//    (ldmatrix): where a warp walks many groups (bsrmm).
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

// ---- through shared memory

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {  // zeros where not live
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}

// A group of 16 rows of 64 features in shared memory: row k at 128 k, its 16-byte pieces exchanged by the row's number so that
// eight rows of one piece lie in all banks.
constexpr int kGroupBytes = 16 * 128;
__device__ __forceinline__ uint32_t piece_at(int k, int piece) { return static_cast<uint32_t>(k * 128 + ((piece ^ (k & 7)) << 4)); }
// where row c of the group, which multiplies column c of the left operand, lies
__device__ __forceinline__ int row_slot(int c) { return 2 * (c >> 2) + (c & 1) + 8 * ((c >> 1) & 1); }

// acc[mt][j][c]: features 8j + 2(lane%4) + (c & 1) of row 16 mt + lane/4 + 8 (c >> 1).  rows: shared address of the group; av[mt]: the lane's 8 bytes of row lane/4 (words 0, 2) and lane/4 + 8 (1, 3)
template <int MT>
__device__ __forceinline__ void multiply(float (&acc)[MT][8][4], uint32_t rows, int lane, const uint32_t (&av)[MT][4]) {
  const int k = (lane & 7) + (lane & 8), up = lane >> 4;
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    uint32_t b0, b1, b2, b3;
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                 : "r"(rows + piece_at(k, j + up))
                 : "memory");
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) mma16816(acc[mt][j], av[mt], b0, b1);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) mma16816(acc[mt][j + 1], av[mt], b2, b3);
  }
}

}  // namespace mma16
}  // namespace sptir
#endif  // SPARSETIR_B200_MMA16_CUH_

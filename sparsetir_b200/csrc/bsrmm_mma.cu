// BSR SpMM for block sizes that are multiples of 16 and feature counts that are multiples of 8, fp16
// operands, fp32 sums: calls of one wave on blocks of 32 (bsrmm.cu has the rule), and all shapes that the tcgen05 kernels of
// bsrmm_tc.cu (block size 32, features in steps of 128) do not take.  Those ran on CUDA cores at 11 TFLOP/s.
//
// A thread block owns 16 MT rows of a block row and 64 features; its four warps share the stored blocks, 16 columns ("a group")
// at a time.  The rows of B and the values of A of a warp's next three or four groups are on their way into shared memory
// by asynchronous copies (mma16.cuh).  The warps' sums meet there in a fixed order and every result is written once.
// MT = 2 halves the reads of B per result where the block size allows it.
//
// Bound: the L2-to-SM gather of B (each block reads the 16 rows of its groups once per 16 MT rows of C) and the copies' latency on
// small matrices.  10 % of the blocks stored, us, CUDA cores / operands straight into registers, where four rows per
// load met in the same banks of L1 / now: 8192 x 8192, block 16, F = 512 626 / 81 / 49; block 64 645 / 64 / 48; block 32, F = 496
// 630 / 56 / 45; 4096 x 4096, block 16, 5 %, F = 208 - / 11.2 / 8.1.
#include <cuda_fp16.h>

#include "common.h"
#include "launch.cuh"
#include "mma16.cuh"
#include "vec.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 128;

__host__ __device__ constexpr int stages(int mt) { return mt == 1 ? 4 : 3; }
template <int MT>
struct __align__(128) WarpRing {
  unsigned char rows[stages(MT)][mma16::kGroupBytes];
  unsigned char values[stages(MT)][MT * 512];
};

template <int MT>
__global__ void __launch_bounds__(kThreads, MT == 1 ? 5 : 4)
bsrmm_mma_kernel(const __half* a, const __half* b, float* __restrict__ c,
                 const int32_t* indptr, const int32_t* indices, int blk, int feat,
                 int slabs, int parts, int vec_out) {
  constexpr int S = stages(MT);
  __shared__ WarpRing<MT> s_ring[4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  const int slab = static_cast<int>(blockIdx.x) % slabs, rest = static_cast<int>(blockIdx.x) / slabs;
  const int part = rest % parts, i = rest / parts;
  const int f0 = slab * mma16::kSlab, row0 = part * 16 * MT;
  chain_wait();
  const int p0 = ld_global(indptr + i), p1 = ld_global(indptr + i + 1);
  const int per_blk = blk >> 4;  // groups per stored block
  const long long total = static_cast<long long>(p1 - p0) * per_blk;
  const long long g0 = total * warp / 4;
  const int groups = static_cast<int>(total * (warp + 1) / 4 - g0);

  float acc[MT][8][4];
  mma16::clear(acc);
  const int piece = lane & 7, first = (lane >> 3) * 4;  // of the rows of B that this lane copies
  const bool in = f0 + piece * 8 < feat;
  const __half* bl = b + static_cast<size_t>(first) * feat + (in ? f0 + piece * 8 : 0);
  const __half* al = a + static_cast<size_t>(row0 + (lane >> 1)) * blk + (lane & 1) * 8;
  WarpRing<MT>& ring = s_ring[warp];
  const uint32_t rows0 = static_cast<uint32_t>(__cvta_generic_to_shared(&ring.rows[0][0]));
  const uint32_t values0 = static_cast<uint32_t>(__cvta_generic_to_shared(&ring.values[0][0]));
  // the next group to copy: stored block, group inside it; lane k holds the column of block id0 + k
  int pc = p0 + static_cast<int>(g0 / per_blk), kc = static_cast<int>(g0 % per_blk);
  int id0 = pc, ids = 0;
  if (groups > 0) ids = ld_global(indices + min(id0 + lane, p1 - 1));
  auto copy_group = [&](int n) {
    if (n < groups) {
      if (pc - id0 == 32) {
        id0 = pc;
        ids = ld_global(indices + min(id0 + lane, p1 - 1));
      }
      const int col = __shfl_sync(0xffffffffu, ids, pc - id0), stage = n % S;
      const __half* p = bl + (static_cast<size_t>(col) * blk + kc * 16) * feat;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        mma16::copy16(rows0 + stage * mma16::kGroupBytes + mma16::piece_at(mma16::row_slot(first + k), piece),
                      p + static_cast<size_t>(k) * feat, in);
      const __half* at = al + static_cast<size_t>(pc) * blk * blk + kc * 16;
#pragma unroll
      for (int m = 0; m < MT; ++m)
        mma16::copy16(values0 + stage * (MT * 512) + (m * 32 + lane) * 16, at + static_cast<size_t>(m * 16) * blk, true);
      if (++kc == per_blk) {
        kc = 0;
        ++pc;
      }
    }
  };
#pragma unroll
  for (int n = 0; n < S; ++n) {
    copy_group(n);
    cp_async_commit();
  }
  for (int n = 0; n < groups; ++n) {
    cp_async_wait<S - 1>();
    __syncwarp();
    const unsigned char* v = ring.values[n % S];
    uint32_t av[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const uint2 lo = *reinterpret_cast<const uint2*>(v + (mt * 16 + r) * 32 + q * 8);
      const uint2 hi = *reinterpret_cast<const uint2*>(v + (mt * 16 + 8 + r) * 32 + q * 8);
      av[mt][0] = lo.x; av[mt][1] = hi.x; av[mt][2] = lo.y; av[mt][3] = hi.y;
    }
    mma16::multiply(acc, rows0 + n % S * mma16::kGroupBytes, lane, av);
    __syncwarp();
    copy_group(n + S);
    cp_async_commit();
  }
  cp_async_wait<0>();
  __syncwarp();
  // the warps' sums meet, row by row, in place of their rings
  constexpr int kRow = mma16::kSlab + 8;  // floats; rows of four neighbours lie in all banks
  static_assert(MT * 16 * kRow * 4 <= sizeof(WarpRing<MT>), "fits the ring");
  float* mine = reinterpret_cast<float*>(&ring) + r * kRow + 2 * q;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<float2*>(mine + (mt * 16 + h * 8) * kRow + j * 8) = make_float2(acc[mt][j][2 * h], acc[mt][j][2 * h + 1]);
  __syncthreads();
  // a warp finishes every fourth row, 16 bytes per lane: whole lines
  const int f = (lane & 15) * 4;
  if (f0 + f >= feat) return;
#pragma unroll
  for (int k = 0; k < 2 * MT; ++k) {
    const int row = (k * 4 + warp) * 2 + (lane >> 4);  // of 16 MT
    const auto of = [&](int w) { return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(&s_ring[w]) + row * kRow + f); };
    const float4 s0 = of(0), s1 = of(1), s2 = of(2), s3 = of(3);
    const float4 v = make_float4((s0.x + s1.x) + (s2.x + s3.x), (s0.y + s1.y) + (s2.y + s3.y), (s0.z + s1.z) + (s2.z + s3.z),
                                 (s0.w + s1.w) + (s2.w + s3.w));
    float* dst = c + (static_cast<size_t>(i) * blk + row0 + row) * feat + f0 + f;
    if (vec_out) {
      __stcs(reinterpret_cast<float4*>(dst), v);
    } else {
      dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
    }
  }
}

}  // namespace

// 0 when launched, 1 when this path cannot take the call (caller falls back), -1 on error
int bsrmm_mma_launch(const __half* a, const __half* b, float* c, const int32_t* indptr, const int32_t* indices,
                     int nb, int blk, int feat, cudaStream_t st) {
  if (blk % 16 != 0 || feat % 8 != 0 || !aligned16(a) || !aligned16(b)) return 1;
  const int mt = blk % 32 == 0 ? 2 : 1, parts = blk / (16 * mt), slabs = ceil_div(feat, mma16::kSlab);
  const long long blocks = static_cast<long long>(nb) * parts * slabs;
  if (blocks > INT32_MAX) return 1;
  const int vec_out = aligned16(c) ? 1 : 0;
  if (mt == 2)
    launch_chained(bsrmm_mma_kernel<2>, static_cast<unsigned>(blocks), kThreads, 0, st, a, b, c, indptr, indices, blk, feat, slabs, parts, vec_out);
  else
    launch_chained(bsrmm_mma_kernel<1>, static_cast<unsigned>(blocks), kThreads, 0, st, a, b, c, indptr, indices, blk, feat, slabs, parts, vec_out);
  SPTIR_LAUNCH_OK("bsrmm_mma_kernel");
  return 0;
}

}  // namespace sptir

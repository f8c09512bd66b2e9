// BSR SpMM for block sizes that are multiples of 16 and feature counts that are multiples of 8, fp16
// operands, fp32 sums: the shapes that the tcgen05 kernels of bsrmm_tc.cu (block size 32, features in
// steps of 128) do not take.  They ran on CUDA cores at 11 TFLOP/s.
//
// A thread block owns 16 MT rows of a block row and 64 features; its four warps share the stored blocks,
// 16 columns ("a group") at a time, two groups in flight per warp, operands straight into the registers
// of the matrix instruction (mma16.cuh).  The warps' sums meet in shared memory in a fixed order and every
// result is written once.  MT = 2 halves the reads of B per result where the block size allows it.
//
// Bound: the L2-to-SM gather of B (each block reads the 16 rows of its groups once per 16 MT rows of C).
// 10 % of the blocks stored, us, before / now: 8192 x 8192, block 16, F = 512 626 / 84; block 64 645 / 66; block
// 32, F = 496 630 / 57; 4096 x 4096, block 16, F = 64 68 / 11; 1024 x 1024, block 64, F = 64 31 / 7.
#include <cuda_fp16.h>

#include "common.h"
#include "launch.cuh"
#include "mma16.cuh"
#include "vec.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 128;

template <int MT>
__global__ void __launch_bounds__(kThreads, MT == 1 ? 5 : 3)
bsrmm_mma_kernel(const __half* a, const __half* b, float* __restrict__ c,
                 const int32_t* indptr, const int32_t* indices, int blk, int feat,
                 int slabs, int parts, int vec_out) {
  __shared__ float s_sum[4][MT][4][8][32];  // [warp][row tile][c][j][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r = lane >> 2;
  const int slab = static_cast<int>(blockIdx.x) % slabs, rest = static_cast<int>(blockIdx.x) / slabs;
  const int part = rest % parts, i = rest / parts;
  const int f0 = slab * mma16::kSlab, row0 = part * 16 * MT;
  chain_wait();
  const int p0 = ld_global(indptr + i), p1 = ld_global(indptr + i + 1);
  const int per_blk = blk >> 4;  // groups per stored block
  const long long total = static_cast<long long>(p1 - p0) * per_blk;
  const long long g0 = total * warp / 4, g1 = total * (warp + 1) / 4;

  float acc[MT][8][4];
  mma16::clear(acc);
  const bool in = f0 + r * 8 < feat;
  const __half* bl = b + static_cast<size_t>(4 * q) * feat + (in ? f0 + r * 8 : 0);
  const __half* al = a + static_cast<size_t>(row0 + r) * blk + 4 * q;
  auto rows_of = [&](int col, int kk, uint4 (&v)[4]) {
    const __half* p = bl + (static_cast<size_t>(col) * blk + kk * 16) * feat;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = make_uint4(0u, 0u, 0u, 0u);
      if (in) v[k] = ld_global(reinterpret_cast<const uint4*>(p + static_cast<size_t>(k) * feat));
    }
  };
  auto values_of = [&](int p, int kk, uint32_t (&av)[MT][4]) {
    const __half* at = al + static_cast<size_t>(p) * blk * blk + kk * 16;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const uint2 lo = ld_global(reinterpret_cast<const uint2*>(at + static_cast<size_t>(mt * 16) * blk));
      const uint2 hi = ld_global(reinterpret_cast<const uint2*>(at + static_cast<size_t>(mt * 16 + 8) * blk));
      av[mt][0] = lo.x; av[mt][1] = hi.x; av[mt][2] = lo.y; av[mt][3] = hi.y;
    }
  };
  // (block, group inside it) of the next two groups; their column ids are requested one pair ahead
  int pa = p0 + static_cast<int>(g0 / per_blk), ka = static_cast<int>(g0 % per_blk);
  auto next = [&](int& p, int& k) {
    if (++k == per_blk) { k = 0; ++p; }
  };
  int pb = pa, kb = ka;
  next(pb, kb);
  auto id_of = [&](int p) { return ld_global(indices + min(p, p1 - 1)); };  // past the last block: not used
  int ca = 0, cb = 0;
  if (p0 < p1) {
    ca = id_of(pa);
    cb = id_of(pb);
  }
  for (long long g = g0; g < g1; g += 2) {
    const bool two = g + 1 < g1;
    uint4 va[4], vb[4];
    uint32_t aa[MT][4], ab[MT][4];
    rows_of(ca, ka, va);
    if (two) rows_of(cb, kb, vb);
    values_of(pa, ka, aa);
    if (two) values_of(pb, kb, ab);
    next(pa, ka); next(pa, ka);
    next(pb, kb); next(pb, kb);
    ca = id_of(pa);
    cb = id_of(pb);
    mma16::multiply(acc, va, aa);
    if (two) mma16::multiply(acc, vb, ab);
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int j = 0; j < 8; ++j) s_sum[warp][mt][k][j][lane] = acc[mt][j][k];
  __syncthreads();
  // warp w finishes the pieces c = w
  const int f = f0 + (2 * q + (warp & 1)) * 8;
  if (f >= feat) return;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      v[j] = (s_sum[0][mt][warp][j][lane] + s_sum[1][mt][warp][j][lane]) +
             (s_sum[2][mt][warp][j][lane] + s_sum[3][mt][warp][j][lane]);
    float* dst = c + (static_cast<size_t>(i) * blk + row0 + mt * 16 + r + (warp >> 1) * 8) * feat + f;
    if (vec_out) {
      __stcs(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
      __stcs(reinterpret_cast<float4*>(dst) + 1, make_float4(v[4], v[5], v[6], v[7]));
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) dst[j] = v[j];
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

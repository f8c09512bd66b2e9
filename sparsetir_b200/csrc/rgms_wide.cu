// The transform and scatter of RGMS for feature counts that are multiples of 128, in fp32:
//   Y[I[i], fo] += sum_fi Z[i, fi] * W[r, fo, fi]      for the CSF rows i of relation r
// Z holds the aggregated rows (a launch of the SpMM kernel).  Tensor cores would need the operands split
// into TF32 parts, whose truncated sums leave more error than fp32 does (5e-7 against 2e-7 of the norm at
// F = 128), so this stays on the FMA units and is bound by them.
//
// A block walks consecutive tiles of 128 rows of one relation x 128 outputs.  Slices of 16 features of
// both operands are stored transposed in shared memory (two buffers, the next slice - of the next tile
// too - in registers meanwhile), four lanes to the 64 bytes of a row; a thread owns 8 x 8 results as 2 x 2 pieces of 4 x 4, so
// that its operands are four 16-byte reads per 64 FMAs, and these 32 two-wide instructions.  Sums run over ascending fi.  Two
// blocks per SM.  100 k nodes, 46 relations, 1 M edges, F = 128 / 256, the call: single FMAs and two lanes to a row 527 / 1830 us, two-wide
// ones, and the sums of rgms_pairs.cu in front, 490 / 1727, four lanes 471 / 1647 (a lane to a row, without conflicts in
// the transposed stores, 561 / 2025).
//
// It replaces a kernel that gathered, multiplied and scattered tile by tile with one block of 256
// threads per SM (131 KB of shared memory) at F = 128, and one warp per row at other sizes.  With the
// aggregation, 100 k nodes, 46 relations, 1 M edges: F = 128 1602 / 471 us, F = 256 125 / 1.65 ms.
#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "rgms_common.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;
constexpr int kTile = 128;
constexpr int kK = 16;
constexpr int kStride = kTile + 4;  // padded: the transposed stores of a warp spread over the banks

__global__ void __launch_bounds__(kThreads, 2)
rgms_wide_kernel(const float* w, float* __restrict__ y, const int32_t* indptr_i,
                 const int32_t* indices_i, const float* z, int num_rels, int nnz_i,
                 int feat, int tiles_per_block) {
  __shared__ __align__(16) float s_z[2][kK][kStride];
  __shared__ __align__(16) float s_w[2][kK][kStride];
  const int tid = threadIdx.x, lane = tid & 31;
  TileWalk tw;
  chain_wait();
  if (!locate_tile_warp(indptr_i, num_rels, static_cast<int>(blockIdx.x) * tiles_per_block, lane, &tw.rel, &tw.row0,
                        &tw.row1))
    return;  // the same in all warps
  tw.rel_end = ld_global(indptr_i + tw.rel + 1);
  const int o0 = static_cast<int>(blockIdx.y) * kTile;
  const int lr = tid >> 2, lk = (tid & 3) * 4;  // rows (and outputs) lr and lr + 64 of the slice: 4 features of each
  const int ty = tid >> 4, tx = tid & 15;
  const int slices = feat / kK;

  float4 nz[2], nw[2];
  auto fetch = [&](const TileWalk& t, int s) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      nz[h] = ld_global(reinterpret_cast<const float4*>(z + static_cast<size_t>(min(t.row0 + lr + h * 64, nnz_i - 1)) * feat + s * kK + lk));
      nw[h] = ld_global(reinterpret_cast<const float4*>(w + (static_cast<size_t>(t.rel) * feat + o0 + lr + h * 64) * feat + s * kK + lk));
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = lr + h * 64;
      s_z[buf][lk + 0][r] = nz[h].x; s_z[buf][lk + 1][r] = nz[h].y; s_z[buf][lk + 2][r] = nz[h].z; s_z[buf][lk + 3][r] = nz[h].w;
      s_w[buf][lk + 0][r] = nw[h].x; s_w[buf][lk + 1][r] = nw[h].y; s_w[buf][lk + 2][r] = nw[h].z; s_w[buf][lk + 3][r] = nw[h].w;
    }
  };

  fetch(tw, 0);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k = 0; k < tiles_per_block; ++k) {
    TileWalk ahead = tw;
    const bool more = k + 1 < tiles_per_block && ahead.next(indptr_i, num_rels);
    unsigned long long acc[8][4];  // results (i, 2j) and (i, 2j + 1)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    for (int s = 0; s < slices; ++s) {
      const bool last = s + 1 == slices;
      if (!last) fetch(tw, s + 1);
      else if (more) fetch(ahead, 0);
#pragma unroll
      for (int f = 0; f < kK; ++f) {
        float zr[8];
        ulonglong2 wr[2];
        *reinterpret_cast<float4*>(zr) = *reinterpret_cast<const float4*>(&s_z[buf][f][ty * 4]);
        *reinterpret_cast<float4*>(zr + 4) = *reinterpret_cast<const float4*>(&s_z[buf][f][64 + ty * 4]);
        wr[0] = *reinterpret_cast<const ulonglong2*>(&s_w[buf][f][tx * 4]);
        wr[1] = *reinterpret_cast<const ulonglong2*>(&s_w[buf][f][64 + tx * 4]);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const unsigned long long zz = pack_pair(zr[i], zr[i]);
          fma_pair(acc[i][0], zz, wr[0].x);
          fma_pair(acc[i][1], zz, wr[0].y);
          fma_pair(acc[i][2], zz, wr[1].x);
          fma_pair(acc[i][3], zz, wr[1].y);
        }
      }
      // the other buffer was last read before the previous barrier
      if (!last || more) put(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
    const int nrows = tw.row1 - tw.row0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = (i >> 2) * 64 + ty * 4 + (i & 3);
      if (t < nrows) {
        float* dst = y + static_cast<size_t>(ld_global(indices_i + tw.row0 + t)) * feat + o0 + tx * 4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float4 v;
          unpack_pair(acc[i][2 * h], v.x, v.y);
          unpack_pair(acc[i][2 * h + 1], v.z, v.w);
          atomicAdd(reinterpret_cast<float4*>(dst + h * 64), v);
        }
      }
    }
    if (!more) break;
    tw = ahead;
  }
}

}  // namespace

// z, w and y 16-byte aligned, feat a multiple of 128, nnz_i > 0
int rgms_wide_launch(const float* w, float* y, const int32_t* indptr_i, const int32_t* indices_i, const float* z,
                     int num_rels, int nnz_i, int feat, cudaStream_t stream) {
  // upper bound on the number of tiles: every relation can add one partly filled tile
  const long long tiles = static_cast<long long>(nnz_i) / kTile + num_rels;
  const int ny = feat / kTile;
  const long long want = std::max(1ll, 2ll * kNumSMs * 4 / ny);  // four runs of tiles per resident block: even ends
  const long long per = (tiles + want - 1) / want;
  const dim3 grid(static_cast<unsigned>((tiles + per - 1) / per), ny);
  launch_chained(rgms_wide_kernel, grid, kThreads, 0, stream, w, y, indptr_i, indices_i, z, num_rels, nnz_i, feat,
                 static_cast<int>(per));
  SPTIR_LAUNCH_OK("rgms_wide_kernel");
  return 0;
}

}  // namespace sptir

// BSR SpMM, fp16 blocks and dense operand, fp32 accumulation and output:
//   C[i*blk+bi, f] = sum_{p in block-row i} sum_bj A[p,bi,bj] * B[indices[p]*blk+bj, f]
// Semantics: tests/python/sparsetir/sparse_tir_lowered_buffer_scripts.py:192-249 of the
// reference; generated kernel being replaced: examples/blocksparse/bsr_spmm.py:359-425 (wmma,
// fp16 accumulate).  Block-rows without blocks are written as zeros (T.init of the reference).
//
// This file holds the CUDA-core kernel that works for every block size; bsrmm_tc.cu (block size 32,
// features in steps of 128) and bsrmm_mma.cu (block sizes in steps of 16, features in steps of 8) hold
// the tensor-core kernels and are tried first.
#include <cuda_fp16.h>

#include <cstdlib>

#include "common.h"

namespace sptir {

// defined in bsrmm_tc.cu; returns 1 when the shape is not supported by the tensor-core path
int bsrmm_tc_launch(const __half* a, const __half* b, float* c, const int32_t* indptr,
                    const int32_t* indices, int nb, int mb, int nnzb, int blk, int feat,
                    cudaStream_t stream);
// defined in bsrmm_mma.cu
int bsrmm_mma_launch(const __half* a, const __half* b, float* c, const int32_t* indptr, const int32_t* indices,
                     int nb, int blk, int feat, cudaStream_t st);

namespace {

constexpr int kThreads = 128;
constexpr int kBi = 8;  // output rows of the block handled per thread block pass

// One thread block per (block-row, tile of 128 features, group of kBi rows inside the block).
// Thread t owns feature f = tile*128 + t and kBi accumulators; the A sub-block is staged in
// shared memory, B rows are read coalesced.
__global__ void __launch_bounds__(kThreads)
bsrmm_simt_kernel(const __half* __restrict__ a, const __half* __restrict__ b,
                  float* __restrict__ c, const int32_t* __restrict__ indptr,
                  const int32_t* __restrict__ indices, int blk, int feat) {
  extern __shared__ float a_s[];  // [kBi][blk]
  const int i = blockIdx.x;
  const int f = blockIdx.y * kThreads + threadIdx.x;
  const int bi0 = blockIdx.z * kBi;
  const int nbi = min(kBi, blk - bi0);
  float acc[kBi];
#pragma unroll
  for (int r = 0; r < kBi; ++r) acc[r] = 0.f;
  const int p0 = __ldg(indptr + i), p1 = __ldg(indptr + i + 1);
  for (int p = p0; p < p1; ++p) {
    __syncthreads();
    for (int t = threadIdx.x; t < nbi * blk; t += kThreads) {
      int r = t / blk, bj = t % blk;
      a_s[r * blk + bj] = __half2float(a[(static_cast<size_t>(p) * blk + bi0 + r) * blk + bj]);
    }
    __syncthreads();
    if (f < feat) {
      const __half* brow = b + static_cast<size_t>(__ldg(indices + p)) * blk * feat + f;
      for (int bj = 0; bj < blk; ++bj) {
        float bv = __half2float(brow[static_cast<size_t>(bj) * feat]);
#pragma unroll
        for (int r = 0; r < kBi; ++r)
          if (r < nbi) acc[r] = fmaf(a_s[r * blk + bj], bv, acc[r]);
      }
    }
  }
  if (f < feat) {
#pragma unroll
    for (int r = 0; r < kBi; ++r)
      if (r < nbi) c[(static_cast<size_t>(i) * blk + bi0 + r) * feat + f] = acc[r];
  }
}

}  // namespace
}  // namespace sptir

extern "C" int sparsetir_bsrmm_raw(const void* a_f16, const void* b_f16, float* c,
                                   const int32_t* indptr, const int32_t* indices, int nb, int mb,
                                   int nnzb, int blk, int feat, int device_id, void* stream) {
  using namespace sptir;
  if (nb < 0 || mb < 0 || nnzb < 0 || blk < 1 || feat < 0)
    return fail("sparsetir_bsrmm: invalid size");
  if (nb == 0 || feat == 0) return 0;
  if (!c || !indptr || (nnzb > 0 && (!a_f16 || !b_f16 || !indices)))
    return fail("sparsetir_bsrmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled() && validate_csr("sparsetir_bsrmm", indptr, nb, indices, nnzb, mb, st) != 0) return -1;
  const __half* a = static_cast<const __half*>(a_f16);
  const __half* b = static_cast<const __half*>(b_f16);
  // Blocks of 32 and features in steps of 128 could take either tensor-core kernel.  bsrmm_mma.cu has the shorter chain in front of
  // the first product and is the faster one as long as all its thread blocks, 64 features of a block row each, are resident at
  // once; where whole pairs of feature tiles share the loads of A, less than that.  How many blocks are stored moves both alike.
  // us, tcgen05 / mma, at 2, 10, 50 and 100 % stored: 1024^2, F = 256 4.0 / 3.0, 5.3 / 3.2, 9.9 / 5.7, 13.0 / 7.3; 4096^2, F = 128 5.3 / 4.1, 10.5 / 7.0,
  // 32.6 / 18.9, 48.8 / 30.6; F = 256 5.4 / 5.2, 9.8 / 9.4, 31.3 / 27.6, 47.3 / 47.5; in more than one wave F = 384 5.8 / 7.3, 10.2 / 13.6, 31.5 / 39.9,
  // 47.9 / 70.7; pairs of tiles, 1536^2, F = 512 4.5 / 4.1, 6.7 / 5.8, 13.7 / 11.5, 19.0 / 15.9, 2048^2 4.5 / 4.6, 6.8 / 7.2, 16.6 / 15.9, 25.1 / 25.5.
  // One row of 2,000 blocks among rows of 10, F = 256, 64 block rows 873 / 312.
  const long long units = static_cast<long long>(nb) * ceil_div(feat, 64);
  static const bool chosen = [] {  // a comparison switch of bsrmm_tc.cu
    const char* e = std::getenv("SPARSETIR_BSR_PATH");
    return e != nullptr && e[0] != '\0';
  }();
  int rc = 1;
  if (!chosen && blk == 32 && units <= (feat > 256 && feat % 256 == 0 ? 400 : 4 * kNumSMs)) {
    rc = bsrmm_mma_launch(a, b, c, indptr, indices, nb, blk, feat, st);
    if (rc <= 0) return rc;
  }
  rc = bsrmm_tc_launch(a, b, c, indptr, indices, nb, mb, nnzb, blk, feat, st);
  if (rc <= 0) return rc;
  rc = bsrmm_mma_launch(a, b, c, indptr, indices, nb, blk, feat, st);
  if (rc <= 0) return rc;
  dim3 grid(nb, ceil_div(feat, kThreads), ceil_div(blk, kBi));
  if (grid.y > 65535 || grid.z > 65535) return fail("sparsetir_bsrmm: shape exceeds the grid limits");
  size_t smem = static_cast<size_t>(kBi) * blk * sizeof(float);
  if (smem > 48 * 1024) return fail("sparsetir_bsrmm: block size %d is too large", blk);
  bsrmm_simt_kernel<<<grid, kThreads, smem, st>>>(a, b, c, indptr, indices, blk, feat);
  SPTIR_LAUNCH_OK("bsrmm_simt_kernel");
  return 0;
}

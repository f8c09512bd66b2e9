// The small operators either side of SpMM / SDDMM in the reference's script collection, fp32:
//   csr_reduce / segment_reduce  B[i] = sum_j A[i,j]                  (sparse_tir_scripts.py:74-110)
//   sparse_softmax               B[i,j] = exp(A[i,j]) / sum_j exp(A[i,j] - max_j A[i,j])   (:503-528)
//   csr2bsr                      scatter of CSR entries into the blocks of a BSR matrix      (:532-557)
//   ellmm                        block-ELL SpMM C[i,bi,f] = sum_j sum_bj A[i,j,bi,bj] B[ind[i,j],bj,f] (:150-181)
// All four stream their operands once: a sub-warp per row (4 lanes for short rows, a warp for
// long ones) for the row-wise ones, a thread per entry for the scatter, a block per block row
// and 128 features for the block-ELL product.
#include <cfloat>

#include "common.h"
#include "launch.cuh"
#include "vec.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;

template <int LPR>
__device__ __forceinline__ float group_sum(float v, unsigned mask) {
#pragma unroll
  for (int o = LPR / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(mask, v, o, LPR);
  return v;
}
template <int LPR>
__device__ __forceinline__ float group_max(float v, unsigned mask) {
#pragma unroll
  for (int o = LPR / 2; o >= 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(mask, v, o, LPR));
  return v;
}

template <int LPR>
__global__ void __launch_bounds__(kThreads)
csr_reduce_kernel(const float* __restrict__ a, float* __restrict__ b, const int32_t* __restrict__ indptr,
                  int n) {
  const int lane = threadIdx.x % LPR;
  const unsigned mask = group_mask<LPR>();
  const long long row = static_cast<long long>(blockIdx.x) * (kThreads / LPR) + threadIdx.x / LPR;
  if (row >= n) return;
  const int p0 = __ldg(indptr + row), p1 = __ldg(indptr + row + 1);
  float s = 0.f;
  for (int p = p0 + lane; p < p1; p += LPR) s += __ldg(a + p);
  s = group_sum<LPR>(s, mask);
  if (lane == 0) b[row] = s;
}

// Each lane keeps the first CACHE of its entries of the row in registers (LPR * CACHE entries
// per row: the whole row in the common case), so the row is read from memory once instead of
// three times; exp(a) = exp(a - max) * exp(max) saves the second exponential per entry.
template <int LPR, int CACHE>
__global__ void __launch_bounds__(kThreads)
sparse_softmax_kernel(const float* a, float* b,
                      const int32_t* indptr, int n) {
  const int lane = threadIdx.x % LPR;
  const unsigned mask = group_mask<LPR>();
  const long long row = static_cast<long long>(blockIdx.x) * (kThreads / LPR) + threadIdx.x / LPR;
  chain_wait();
  if (row >= n) return;
  const int p0 = ld_global(indptr + row), p1 = ld_global(indptr + row + 1);
  const int len = p1 - p0, left = len - lane;  // left: entries from the thread's first one on
  const float* at = a + p0 + lane;
  float* to = b + p0 + lane;
  // Ordinary loads, which the compiler keeps behind the wait like ld_global and makes predicated ones of; four at a time,
  // of which those behind the row's end are skipped by all.
  float v[CACHE];
#pragma unroll
  for (int k0 = 0; k0 < CACHE; k0 += 4) {
#pragma unroll
    for (int k = k0; k < k0 + 4; ++k) v[k] = -FLT_MAX;
    if (k0 * LPR < len) {
#pragma unroll
      for (int k = k0; k < k0 + 4; ++k)
        if (k * LPR < left) v[k] = at[k * LPR];
    }
  }
  // The entries beyond the cached ones, four at a time: a load may not pass the store of an entry before it (5.6 M entries,
  // 10,000 in the longest row: 16 us, one at a time 19; a power-law graph, 13,000 in the longest: 208, 369).
  auto beyond = [&](auto&& take) {
    int e = CACHE * LPR;
    for (; left - e > 3 * LPR; e += 4 * LPR) {
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = at[e + u * LPR];
#pragma unroll
      for (int u = 0; u < 4; ++u) take(e + u * LPR, x[u]);
    }
    for (; e < left; e += LPR) take(e, at[e]);
  };
  float mx = -FLT_MAX;
#pragma unroll
  for (int k = 0; k < CACHE; ++k) mx = fmaxf(mx, v[k]);
  beyond([&](int, float x) { mx = fmaxf(mx, x); });
  mx = group_max<LPR>(mx, mask);
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < CACHE; ++k) {
    v[k] = k * LPR < left ? __expf(v[k] - mx) : 0.f;
    s += v[k];
  }
  beyond([&](int, float x) { s += expf(x - mx); });
  s = group_sum<LPR>(s, mask);
  // the reference divides exp(A) — not exp(A - max) — by the shifted sum
  const float scale = expf(mx) / s;
#pragma unroll
  for (int k = 0; k < CACHE; ++k)
    if (k * LPR < left) to[k * LPR] = v[k] * scale;
  beyond([&](int e, float x) { to[e] = expf(x - mx) * scale; });
}

// Rows of any length, a block per 8 of them.  A warp takes a row of up to kWarpRow entries, 32 * kCache of which stay in
// its registers between the three passes; longer rows wait until the block's other ones are done and are then shared by its
// eight warps, 256 * kCache entries in registers.  Bound: instructions, about 20 per 32 entries.  So addresses are a
// pointer and a constant, and the entries are taken kBatch to a thread, of which those behind the row's end are skipped
// by all.  20 M entries in 40 k rows of 245 in the median and 10,000 at most: 64 us; a warp that walks its row alone, with
// the launch as long as the longest row: 79.  Smaller matrices keep that form (softmax_by_blocks).
// Eight rows that are all shared are taken one after the other, two barriers each, so a row is shared only where a warp
// alone would be the launch's tail (us, a warp per row at any length / shared from 512 / 2048 / 4096 entries on: 13 M entries in rows
// of 600 29 / 58 / 27 / 27, of 1,000 27 / 45 / 25 / 25, of 2,000 28 / 39 / 34 / 29; 20 M as above 79 / 66 / 64 / 76).
// b may be a: an entry is read for the last time by the thread that then writes it.
constexpr int kWarpRow = 2048;
constexpr int kCache = 16, kBatch = 4;

// Maximum, sum and store over the entries a[0], a[STRIDE], ... of which the thread has those below `left` (the
// row's length less the thread's first entry, which may be negative); `len` is the row's length.  all_max / all_sum
// combine the threads' values.
template <int STRIDE, class AllMax, class AllSum>
__device__ __forceinline__ void softmax_row(const float* a, float* b, int left, int len, AllMax&& all_max, AllSum&& all_sum) {
  float v[kCache];
  float mx = -FLT_MAX;
#pragma unroll
  for (int k0 = 0; k0 < kCache; k0 += kBatch)
    if (k0 * STRIDE < len) {
#pragma unroll
      for (int k = k0; k < k0 + kBatch; ++k) {
        v[k] = -FLT_MAX;
        if (k * STRIDE < left) v[k] = a[k * STRIDE];
      }
    }
#pragma unroll
  for (int k0 = 0; k0 < kCache; k0 += kBatch)
    if (k0 * STRIDE < len) {
#pragma unroll
      for (int k = k0; k < k0 + kBatch; ++k) mx = fmaxf(mx, v[k]);
    }
  // the entries beyond the cached ones, kCache at a time
  auto batch = [&](int at, float (&x)[kCache]) {
#pragma unroll
    for (int u = 0; u < kCache; ++u) {
      x[u] = -FLT_MAX;
      if (u * STRIDE < left - at) x[u] = a[static_cast<size_t>(at) + u * STRIDE];
    }
  };
  constexpr int kStep = kCache * STRIDE;
  for (int at = kStep; at < len; at += kStep) {
    float x[kCache];
    batch(at, x);
#pragma unroll
    for (int u = 0; u < kCache; ++u) mx = fmaxf(mx, x[u]);
    if (len - at <= kStep) break;  // before `at` could pass the largest int
  }
  mx = all_max(mx);
  float s = 0.f;
#pragma unroll
  for (int k0 = 0; k0 < kCache; k0 += kBatch)
    if (k0 * STRIDE < len) {
#pragma unroll
      for (int k = k0; k < k0 + kBatch; ++k) {
        v[k] = expf(v[k] - mx);
        if (k * STRIDE < left) s += v[k];
      }
    }
  for (int at = kStep; at < len; at += kStep) {
    float x[kCache];
    batch(at, x);
#pragma unroll
    for (int u = 0; u < kCache; ++u)
      if (u * STRIDE < left - at) s += expf(x[u] - mx);
    if (len - at <= kStep) break;
  }
  s = all_sum(s);
  // the reference divides exp(A) — not exp(A - max) — by the shifted sum
  const float scale = expf(mx) / s;
#pragma unroll
  for (int k0 = 0; k0 < kCache; k0 += kBatch)
    if (k0 * STRIDE < len) {
#pragma unroll
      for (int k = k0; k < k0 + kBatch; ++k)
        if (k * STRIDE < left) b[k * STRIDE] = v[k] * scale;
    }
  for (int at = kStep; at < len; at += kStep) {
    float x[kCache];
    batch(at, x);
#pragma unroll
    for (int u = 0; u < kCache; ++u)
      if (u * STRIDE < left - at) b[static_cast<size_t>(at) + u * STRIDE] = expf(x[u] - mx) * scale;
    if (len - at <= kStep) break;
  }
}

__global__ void __launch_bounds__(kThreads, 5)
sparse_softmax_rows_kernel(const float* a, float* b, const int32_t* indptr, int n) {
  constexpr int kWarps = kThreads / 32;
  __shared__ int s_begin[kWarps], s_len[kWarps];  // the long rows; others: length 0
  __shared__ float s_max[kWarps], s_sum[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long row = static_cast<long long>(blockIdx.x) * kWarps + warp;
  int p0 = 0, len = 0;
  if (row < n) {
    p0 = ld_global(indptr + row);
    len = ld_global(indptr + row + 1) - p0;
  }
  const bool is_long = len > kWarpRow;
  if (!is_long && len > 0)
    softmax_row<32>(a + p0 + lane, b + p0 + lane, len - lane, len, [](float v) { return group_max<32>(v, 0xffffffffu); },
                    [](float v) { return group_sum<32>(v, 0xffffffffu); });
  if (lane == 0) {
    s_begin[warp] = p0;
    s_len[warp] = is_long ? len : 0;
  }
  if (!__syncthreads_or(is_long)) return;
  for (int w = 0; w < kWarps; ++w) {
    const int long_len = s_len[w];
    if (long_len == 0) continue;
    const size_t at = static_cast<size_t>(s_begin[w]) + threadIdx.x;
    softmax_row<kThreads>(a + at, b + at, long_len - static_cast<int>(threadIdx.x), long_len,
                          [&](float v) {
                            v = group_max<32>(v, 0xffffffffu);
                            if (lane == 0) s_max[warp] = v;
                            __syncthreads();
#pragma unroll
                            for (int j = 0; j < kWarps; ++j) v = fmaxf(v, s_max[j]);
                            return v;
                          },
                          [&](float v) {
                            v = group_sum<32>(v, 0xffffffffu);
                            if (lane == 0) s_sum[warp] = v;
                            __syncthreads();  // the next row's maxima are written behind this barrier
                            v = 0.f;
#pragma unroll
                            for (int j = 0; j < kWarps; ++j) v += s_sum[j];
                            return v;
                          });
  }
}

// row of entry p by the search of the lowered code; position of the block by lower bound
__global__ void __launch_bounds__(kThreads)
csr2bsr_kernel(const float* __restrict__ a, float* __restrict__ b, const int32_t* __restrict__ indptr_in,
               const int32_t* __restrict__ indices_in, const int32_t* __restrict__ indptr_out,
               const int32_t* __restrict__ indices_out, int m_in, int nnz_in, int blk) {
  const long long p = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  if (p >= nnz_in) return;
  int lo = 0, hi = m_in + 1;  // row(p) = upper_bound(indptr_in, p) - 1
  while (lo < hi) {
    const int mid = lo + (hi - lo) / 2;
    if (__ldg(indptr_in + mid) > p) hi = mid; else lo = mid + 1;
  }
  const int i = lo - 1;
  const int j = __ldg(indices_in + p);
  const int bo = __ldg(indptr_out + i / blk);
  int low = 0, high = __ldg(indptr_out + i / blk + 1) - bo;
  const int key = j / blk;
  while (low < high) {
    const int mid = low + (high - low) / 2;
    if (__ldg(indices_out + mid + bo) < key) low = mid + 1; else high = mid;
  }
  b[(static_cast<size_t>(low + bo) * blk + i % blk) * blk + j % blk] = __ldg(a + p);
}

// block (block row i, 128 features): the row's A blocks go through shared memory one at a time;
// a thread owns feature f of 128 and walks the block's rows
constexpr int kTileF = 128;
__global__ void __launch_bounds__(kTileF)
ellmm_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ c,
             const int32_t* __restrict__ indices, int col, int blk, int feat) {
  extern __shared__ float s_a[];  // blk x blk
  const int i = blockIdx.x;
  const int f = blockIdx.y * kTileF + threadIdx.x;
  const bool live = f < feat;
  for (int bi0 = 0; bi0 < blk; bi0 += 8) {  // 8 output rows per pass keep the accumulators in registers
    float acc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = 0.f;
    for (int j = 0; j < col; ++j) {
      const float* ab = a + (static_cast<size_t>(i) * col + j) * blk * blk;
      __syncthreads();
      for (int e = threadIdx.x; e < blk * blk; e += kTileF) s_a[e] = __ldg(ab + e);
      __syncthreads();
      const float* bb = b + static_cast<size_t>(__ldg(indices + static_cast<size_t>(i) * col + j)) * blk * feat;
      if (live) {
        for (int bj = 0; bj < blk; ++bj) {
          const float x = __ldg(bb + static_cast<size_t>(bj) * feat + f);
#pragma unroll
          for (int r = 0; r < 8; ++r)
            if (bi0 + r < blk) acc[r] = fmaf(s_a[(bi0 + r) * blk + bj], x, acc[r]);
        }
      }
    }
    if (live) {
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (bi0 + r < blk) c[(static_cast<size_t>(i) * blk + bi0 + r) * feat + f] = acc[r];
    }
  }
}

}  // namespace
}  // namespace sptir

namespace sptir {
// Whether the softmax of such a matrix is formed by sparse_softmax_rows_kernel, in place if the caller wants it so.  For
// matrices of long rows that are many: where a launch is two or three waves of blocks, rows that a block takes one after the
// other are the longer chain (attention, us, a warp per row / a block per 8: 1 M entries in 2 k rows 35.3 / 36.2, 4.5 M in
// 10 k 93.8 / 96.7, 9 M in 20 k 559 / 557 at F = 128, 20 M in 40 k 726 / 706).
bool softmax_by_blocks(int n, int nnz) { return nnz >= (12 << 20) && static_cast<double>(nnz) / n >= 24.0; }
}  // namespace sptir

extern "C" int sparsetir_csr_reduce_raw(const float* a, float* b, const int32_t* indptr, int n, int nnz,
                                        int device_id, void* stream) {
  using namespace sptir;
  if (n < 0 || nnz < 0) return fail("sparsetir_csr_reduce: negative size");
  if (n == 0) return 0;
  if (!b || !indptr || (nnz > 0 && !a)) return fail("sparsetir_csr_reduce: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled() && validate_indptr("sparsetir_csr_reduce", "indptr", indptr, n, nnz, st) != 0) return -1;
  if (static_cast<double>(nnz) / n >= 24.0) {
    csr_reduce_kernel<32><<<ceil_div(n, kThreads / 32), kThreads, 0, st>>>(a, b, indptr, n);
  } else {
    csr_reduce_kernel<4><<<ceil_div(n, kThreads / 4), kThreads, 0, st>>>(a, b, indptr, n);
  }
  SPTIR_LAUNCH_OK("csr_reduce_kernel");
  return 0;
}

extern "C" int sparsetir_sparse_softmax_raw(const float* a, float* b, const int32_t* indptr, int n,
                                            int nnz, int device_id, void* stream) {
  using namespace sptir;
  if (n < 0 || nnz < 0) return fail("sparsetir_sparse_softmax: negative size");
  if (n == 0 || nnz == 0) return 0;
  if (!a || !b || !indptr) return fail("sparsetir_sparse_softmax: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled() && validate_indptr("sparsetir_sparse_softmax", "indptr", indptr, n, nnz, st) != 0) return -1;
  if (softmax_by_blocks(n, nnz)) {
    sparse_softmax_rows_kernel<<<ceil_div(n, kThreads / 32), kThreads, 0, st>>>(a, b, indptr, n);
  } else if (static_cast<double>(nnz) / n >= 24.0) {
    launch_chained_if(nnz < kChainEntries, sparse_softmax_kernel<32, 16>, ceil_div(n, kThreads / 32), kThreads, 0, st, a, b, indptr, n);
  } else {
    launch_chained_if(nnz < kChainEntries, sparse_softmax_kernel<4, 4>, ceil_div(n, kThreads / 4), kThreads, 0, st, a, b, indptr, n);
  }
  SPTIR_LAUNCH_OK("sparse_softmax_kernel");
  return 0;
}

extern "C" int sparsetir_csr2bsr_raw(const float* a, float* b, const int32_t* indptr_in,
                                     const int32_t* indices_in, const int32_t* indptr_out,
                                     const int32_t* indices_out, int m_in, int nnz_in, int blk,
                                     int device_id, void* stream) {
  using namespace sptir;
  if (m_in < 0 || nnz_in < 0 || blk < 1) return fail("sparsetir_csr2bsr: invalid size");
  if (nnz_in == 0) return 0;
  if (!a || !b || !indptr_in || !indices_in || !indptr_out || !indices_out)
    return fail("sparsetir_csr2bsr: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  csr2bsr_kernel<<<ceil_div(nnz_in, kThreads), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      a, b, indptr_in, indices_in, indptr_out, indices_out, m_in, nnz_in, blk);
  SPTIR_LAUNCH_OK("csr2bsr_kernel");
  return 0;
}

extern "C" int sparsetir_ellmm_raw(const float* a, const float* b, float* c, const int32_t* indices,
                                   int nb, int mb, int feat, int col, int blk, int device_id,
                                   void* stream) {
  using namespace sptir;
  (void)mb;
  if (nb < 0 || feat < 0 || col < 0 || blk < 1) return fail("sparsetir_ellmm: invalid size");
  if (nb == 0 || feat == 0) return 0;
  if (!c || (col > 0 && (!a || !b || !indices))) return fail("sparsetir_ellmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  const size_t smem = static_cast<size_t>(blk) * blk * sizeof(float);
  if (smem > 48 * 1024) return fail("sparsetir_ellmm: block size %d is too large", blk);
  if (ceil_div(feat, kTileF) > 65535) return fail("sparsetir_ellmm: feat_size %d is too large", feat);
  dim3 grid(nb, ceil_div(feat, kTileF));
  ellmm_kernel<<<grid, kTileF, smem, static_cast<cudaStream_t>(stream)>>>(a, b, c, indices, col, blk, feat);
  SPTIR_LAUNCH_OK("ellmm_kernel");
  return 0;
}

// The first launch of RGMS at 64 features where many (relation, destination) pairs have one edge: those need no sum, and the
// transform (rgms_tc.cu) can take their row straight from X.
//   Z[t,:] = sum_{p in CSF row t} A[p] * X[J[p],:]   for rows of two entries and more, and zeros for rows without;
// rows of one are left out.
//
// 100 k nodes, 46 relations, 1.5 M edges: 530 k of the 690 k pairs have one edge.  With a row of Z for each of them the SpMM kernel
// gathered 401 MB and wrote 177 in 57 us; 248 and 41 MB are left, 34 us.
//
// A group of LPR lanes takes LPR consecutive rows: lane j looks at row j, and the entries of the rows of two and more are one
// stream, LPR at a time (the row of an entry by a search in the running sum of the lengths, in registers), with the ids of
// the next batch on their way and 8 (16-byte lanes) or 4 (32-byte lanes) rows of X in flight.  The groups of a warp run in step:
// with branches of their own they executed 20.2 M instructions and took 47 us instead of 14.5 M and 37 (counters of one launch).
// What bounds it is the latency of the gathers (10 of 16 waiting warps; L1 data path 49 %, issue slots 34 %, L2 35 %); twice the rows
// in flight on half the warps is slower (the call 112 us against 99).
#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "row_walk.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;

// The rows of a block that one group would walk alone while the rest of the call waits (more than 64 entries, or four times the average: a
// destination with 1,000 edges of one relation): all groups share each of them, and their sums are added in a fixed order.  s_long: a bit for each
// such row of a group.  us, alone / so, 1.5 M edges on 100 k nodes, destinations drawn as the square, the fourth and the eighth power of a uniform number:
// 46 relations F = 64 360 / 107, 4361 / 253, 16054 / 739; 80 k edges on 10 k nodes, F = 128 86 / 57, 386 / 57, 1064 / 97; uniform ones 98.4 / 98.6
// and 51 / 51.  The sums of the groups of a warp meet by shuffles: with 8 KB of shared memory for all of them, off L1, uniform ones took 99.6.
template <int LPR, int W>
__device__ __forceinline__ void long_rows(const float* a, const float* x, float* z, const int32_t* indptr, const int32_t* indices, int rpi,
                                       const unsigned* s_long) {
  using LV = LaneVec<W>;
  constexpr int SUBS = kThreads / LPR;
  constexpr unsigned kRowBytes = LPR * W * 4;
  constexpr int WARPS = kThreads / 32;
  __shared__ __align__(32) float s_part[WARPS][LPR * W];
  const int lane = threadIdx.x % LPR, sub = threadIdx.x / LPR;
  const char* xl = reinterpret_cast<const char*>(x) + lane * (W * 4);
  for (int owner = 0; owner < SUBS; ++owner) {
    for (unsigned todo = s_long[owner]; todo != 0u; todo &= todo - 1u) {
      const long long row = (static_cast<long long>(blockIdx.x) * SUBS + owner) * rpi + __ffs(todo) - 1;
      const int begin = ld_global(indptr + row), end = ld_global(indptr + row + 1);
      typename LV::type acc = LV::zero();
      add_entries<LPR, W>(a, indices, xl, kRowBytes, begin + sub * LPR, end, SUBS * LPR, lane, group_mask<LPR>(), acc);
#pragma unroll
      for (int o = LPR; o < 32; o <<= 1) LV::add_xor(acc, o);
      if (threadIdx.x % 32 < LPR) LV::sts(&s_part[threadIdx.x / 32][lane * W], acc);
      __syncthreads();
      if (sub == 0) {
        for (int j = 1; j < WARPS; ++j) LV::add(acc, LV::lds(&s_part[j][lane * W]));
        LV::stcg(reinterpret_cast<char*>(z) + row * kRowBytes + lane * (W * 4), acc);
      }
      __syncthreads();
    }
  }
}

// ALL: rows of one entry as well.
template <int LPR, int W, bool ALL>
__global__ void __launch_bounds__(kThreads, 4)
rgms_pairs_kernel(const float* a, const float* x, float* __restrict__ z,
                  const int32_t* indptr, const int32_t* indices, int m, int rpi, int long_row) {
  constexpr int kF = LPR * W;
  using LV = LaneVec<W>;
  constexpr int SUBS = kThreads / LPR;
  constexpr int U = 32 / W;
  const int lane = threadIdx.x % LPR, shift = (threadIdx.x & 31) / LPR * LPR;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr unsigned kGroup = LPR == 32 ? kAll : (1u << LPR) - 1u;
  const long long r0l = (static_cast<long long>(blockIdx.x) * SUBS + threadIdx.x / LPR) * rpi;
  chain_wait();
  const int r0 = static_cast<int>(min(r0l, static_cast<long long>(m))), row = r0 + lane;
  const bool there = lane < rpi && row < m;
  const int begin = ld_global(indptr + min(row, m)), len = there ? ld_global(indptr + min(row + 1, m)) - begin : -1;
  __shared__ unsigned s_long[SUBS];
  const unsigned own_long = (__ballot_sync(kAll, len > long_row) >> shift) & kGroup;
  if (lane == 0) s_long[threadIdx.x / LPR] = own_long;
  const bool any_long = __syncthreads_or(own_long != 0u);
  const int own = len >= (ALL ? 1 : 2) && len <= long_row ? len : 0;
  int upto = own;  // entries of the rows up to this lane's
#pragma unroll
  for (int o = 1; o < LPR; o <<= 1) {
    const int v = __shfl_up_sync(kAll, upto, o, LPR);
    if (lane >= o) upto += v;
  }
  const int total = __shfl_sync(kAll, upto, LPR - 1, LPR);
  const int steps = __reduce_max_sync(kAll, total);  // the groups of a warp run in step
  const int base = begin - (upto - own);  // position of entry e of the stream, if it is in this lane's row: base + e
  char* zl = reinterpret_cast<char*>(z) + static_cast<size_t>(r0) * (kF * 4) + lane * (W * 4);
  const char* xl = reinterpret_cast<const char*>(x) + lane * (W * 4);

  for (unsigned empty = (__ballot_sync(kAll, len == 0) >> shift) & kGroup; empty != 0u; empty &= empty - 1u)
    LV::stcg(zl + (__ffs(empty) - 1) * (kF * 4), LV::zero());

  int cid = 0, at = 0;   // of the batch to come: column, row inside the group
  float av = 0.f;
  unsigned ends = 0;     // bit k: the row of entry k ends with it
  auto request = [&](int e0) {  // lanes past the group's last entry repeat it: it is added to a sum that nobody stores
    const int e = min(e0 + lane, total - 1);
    int pos = 0;
#pragma unroll
    for (int step = LPR / 2; step >= 1; step >>= 1)
      if (__shfl_sync(kAll, upto, pos + step - 1, LPR) <= e) pos += step;
    const int p = __shfl_sync(kAll, base, pos, LPR) + e;
    const bool last = __shfl_sync(kAll, upto, pos, LPR) == e + 1 && e0 + lane < total;
    at = pos * (kF * 4);
    ends = (__ballot_sync(kAll, last) >> shift) & kGroup;
    if (total > 0) {
      cid = ld_global(indices + p);
      av = ld_global(a + p);
    }
  };
  if (steps > 0) request(0);
  typename LV::type acc = LV::zero();
  for (int e0 = 0; e0 < steps; e0 += LPR) {
    const int cid_now = cid, at_now = at, left = total - e0;
    const float av_now = av;
    const unsigned ends_now = ends, any_ends = __reduce_or_sync(kAll, ends);
    if (e0 + LPR < steps) request(e0 + LPR);
#pragma unroll
    for (int k0 = 0; k0 < LPR; k0 += U) {
      if (k0 < steps - e0) {
        typename LV::type v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned col = static_cast<unsigned>(__shfl_sync(kAll, cid_now, k0 + u, LPR));
          v[u] = LV::zero();
          if (k0 + u < left) v[u] = LV::ldg(xl + static_cast<unsigned long long>(col) * (kF * 4));
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          LV::fma(acc, __shfl_sync(kAll, av_now, k0 + u, LPR), v[u]);
          if ((any_ends >> (k0 + u)) & 1u) {  // a row ends here in some group of the warp
            const int to = __shfl_sync(kAll, at_now, k0 + u, LPR);
            const bool end = (ends_now >> (k0 + u)) & 1u;
            if (end) LV::stcg(zl + to, acc);
            LV::zero_if(acc, end);
          }
        }
      }
    }
  }
  if (any_long) long_rows<LPR, W>(a, x, z, indptr, indices, rpi, s_long);
}

template <int LPR, int W, bool ALL>
int launch(const float* a, const float* x, float* z, const int32_t* indptr, const int32_t* indices, int m, int nnz, cudaStream_t st) {
  // fewer rows per group where the groups would not fill the SMs
  constexpr int kGroups = kThreads / LPR;
  int rpi = LPR;
  while (rpi > 1 && ceil_div(m, rpi) < kNumSMs * 4 * kGroups) rpi /= 2;
  launch_chained(rgms_pairs_kernel<LPR, W, ALL>, ceil_div(ceil_div(m, rpi), kGroups), kThreads, 0, st, a, x, z, indptr, indices, m, rpi, std::max(64, 4 * (nnz / m)));
  SPTIR_LAUNCH_OK("rgms_pairs_kernel");
  return 0;
}

}  // namespace

int rgms_pairs_launch(const float* a, const float* x, float* z, const int32_t* indptr, const int32_t* indices, int m,
                      int nnz, cudaStream_t st) {
  // 32-byte lanes lose where there are too few rows for the groups (3 k nodes, 12 k edges, the call 12.3 us with 16 bytes, 13.9 with 32)
  if (m >= (1 << 15) && aligned32(x) && aligned32(z)) return launch<8, 8, false>(a, x, z, indptr, indices, m, nnz, st);
  return launch<16, 4, false>(a, x, z, indptr, indices, m, nnz, st);
}

// All rows, 128 or 256 features, x and z 32-byte aligned.
int rgms_rows_launch(const float* a, const float* x, float* z, const int32_t* indptr, const int32_t* indices, int m, int nnz,
                     int feat, cudaStream_t st) {
  if (feat == 128) return launch<16, 8, true>(a, x, z, indptr, indices, m, nnz, st);
  return launch<32, 8, true>(a, x, z, indptr, indices, m, nnz, st);
}

}  // namespace sptir

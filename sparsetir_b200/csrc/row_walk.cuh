// Finding the row of a stored position, for kernels that split a CSR matrix by stored entries
// instead of by rows (equal work per warp whatever the row lengths).
#ifndef SPARSETIR_B200_ROW_WALK_CUH_
#define SPARSETIR_B200_ROW_WALK_CUH_

#include "vec.cuh"

namespace sptir {

// row(p) = upper_bound(indptr[0..m], p) - 1, the search of
// tests/python/sparsetir/sparse_tir_lowered_buffer_scripts.py:530-549 of the reference
__device__ __forceinline__ int edge_row_search(const int32_t* indptr, int lo_row,
                                               int m, int p) {
  int low = lo_row, high = m + 1;
  while (low < high) {
    int mid = low + (high - low) / 2;
    if (ld_global(indptr + mid) > p) high = mid; else low = mid + 1;
  }
  return low - 1;
}

// First index of [lo, hi) whose pointer lies behind p, or hi, found by a whole warp: 32-ary steps, every
// level is one load per lane (4 dependent reads instead of 18 at 2^18 rows).  Reads stay in [lo, hi).
__device__ __forceinline__ int warp_upper_bound(const int32_t* indptr, int lo, int hi, int p, int wlane) {
  while (hi - lo >= 32) {
    const int step = (hi - lo + 31) / 32;
    const long long probe = static_cast<long long>(lo) + static_cast<long long>(wlane + 1) * step;
    const bool in = probe < hi;
    const bool gt = !in || ld_global(indptr + (in ? probe : 0)) > p;
    const int first = __ffs(__ballot_sync(0xffffffffu, gt)) - 1;  // lane 31 probes >= hi: always set
    const int q = lo + (first + 1) * step;
    if (first > 0) lo = q - step + 1;
    hi = min(hi, q);
  }
  const int idx = lo + wlane;
  const bool in = idx < hi;
  const bool gt = !in || ld_global(indptr + (in ? idx : 0)) > p;  // lane hi - lo (< 32) has idx == hi
  return lo + __ffs(__ballot_sync(0xffffffffu, gt)) - 1;
}

// Row of position p, clamped into [0, m - 1], found by a whole warp: 32 probes around a first
// guess (position x rows / entries), at distances that double, then 32-ary steps inside the
// bracket.  Two or three memory round trips where the rows are
// roughly equally long in the large, four or five for any other matrix of 2^18 rows (a binary
// search: 18).  Every read stays inside indptr whatever p says.
__device__ __forceinline__ int warp_row_of(const int32_t* indptr, int m, int p,
                                           float rows_per_entry, int wlane) {
  int lo = 0, hi = m + 1;  // the answer + 1: first index whose pointer lies behind p
  if (m >= 64) {
    const int guess = static_cast<int>(min(static_cast<float>(m), static_cast<float>(p) * rows_per_entry));
    const long long at = wlane < 16 ? static_cast<long long>(guess) - (16ll << (15 - wlane))
                                    : static_cast<long long>(guess) + (16ll << (wlane - 16));
    const bool in = at >= 0 && at <= m;
    const bool gt = at > m || (in && ld_global(indptr + (in ? at : 0)) > p);
    const unsigned bits = __ballot_sync(0xffffffffu, gt);
    const int first = bits != 0u ? __ffs(bits) - 1 : 32;
    const int idx = static_cast<int>(max(-1ll, min(at, static_cast<long long>(m) + 1)));
    const int above = __shfl_sync(0xffffffffu, idx, min(first, 31)), below = __shfl_sync(0xffffffffu, idx, max(first - 1, 0));
    if (first < 32) hi = above;
    if (first > 0) lo = below + 1;
  }
  return max(0, min(m - 1, warp_upper_bound(indptr, lo, hi, p, wlane) - 1));
}

// Rows of N ascending positions, found by a whole warp: the first by the search, the others by
// counting the row ends among the next 128 rows that lie at or before them (by a search each where
// the rows are so short, or empty, that 128 of them end before the last position).
template <int N>
__device__ __forceinline__ void warp_rows_of(const int32_t* indptr, int m,
                                             const int (&p)[N], float rows_per_entry, int wlane,
                                             int (&row)[N]) {
  row[0] = warp_row_of(indptr, m, p[0], rows_per_entry, wlane);
  if constexpr (N > 1) {
    constexpr int kWin = 4;
    int end[kWin];
#pragma unroll
    for (int k = 0; k < kWin; ++k) end[k] = ld_global(indptr + min(row[0] + 1 + k * 32 + wlane, m));
    if (__shfl_sync(0xffffffffu, end[kWin - 1], 31) > p[N - 1]) {
#pragma unroll
      for (int i = 1; i < N; ++i) {
        int before = 0;
#pragma unroll
        for (int k = 0; k < kWin; ++k) before += __popc(__ballot_sync(0xffffffffu, end[k] <= p[i]));
        row[i] = min(m - 1, row[0] + before);
      }
    } else {
#pragma unroll
      for (int i = 1; i < N; ++i) row[i] = warp_row_of(indptr, m, p[i], rows_per_entry, wlane);
    }
  }
}

// A group of LPR lanes walks consecutive positions.  `wend` of lane j is the end of row r + j (the
// window), loaded with row_window(); row_in_window() gives the row of position e (each lane its
// own e, ascending over the lanes and at or after the first position of row r) and that row's end,
// with log2(LPR) + 1 shuffles and no memory access as long as the row lies in the window (always,
// unless rows are empty).  All 32 lanes of the warp take part, every group for itself.
template <int LPR>
__device__ __forceinline__ int row_window(const int32_t* indptr, int m, int r, int lane) {
  return ld_global(indptr + min(r + 1 + lane, m));
}
template <int LPR>
__device__ __forceinline__ int row_in_window(const int32_t* indptr, int m, int r, int wend,
                                             int e, int& row_end) {
  int pos = 0;
#pragma unroll
  for (int step = LPR / 2; step >= 1; step >>= 1)
    if (__shfl_sync(0xffffffffu, wend, pos + step - 1, LPR) <= e) pos += step;
  row_end = __shfl_sync(0xffffffffu, wend, pos, LPR);
  int row = r + pos;
  if (row_end <= e) {  // past the window (empty rows): search the rest
    row = min(m - 1, edge_row_search(indptr, min(row, m), m, e));
    row_end = ld_global(indptr + row + 1);
  }
  return row;
}

// acc += the entries [p0, p1) of a row, taken LPR at a time, `stride` apart
template <int LPR, int W>
__device__ __forceinline__ void add_entries(const float* a, const int32_t* indices,
                                            const char* bl, unsigned row_bytes, int p0, int p1, int stride,
                                            int lane, unsigned mask, typename LaneVec<W>::type& acc) {
  using LV = LaneVec<W>;
  constexpr int U = (32 / W) < LPR ? (32 / W) : LPR;
  for (int e0 = p0; e0 < p1; e0 += stride) {
    const bool live = lane < p1 - e0;
    const int cid = live ? ld_global(indices + e0 + lane) : 0;
    const float av = live ? ld_global(a + e0 + lane) : 0.f;
    const int cnt = min(LPR, p1 - e0);
#pragma unroll
    for (int k0 = 0; k0 < LPR; k0 += U) {
      if (k0 < cnt) {
        typename LV::type x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const unsigned col = static_cast<unsigned>(__shfl_sync(mask, cid, k0 + u, LPR));
          x[u] = LV::ldg(bl + static_cast<unsigned long long>(col) * row_bytes);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float ak = __shfl_sync(mask, av, k0 + u, LPR);
          if (k0 + u < cnt) LV::fma(acc, ak, x[u]);
        }
      }
    }
  }
}

}  // namespace sptir
#endif  // SPARSETIR_B200_ROW_WALK_CUH_

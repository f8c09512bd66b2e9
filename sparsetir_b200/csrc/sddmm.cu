// SDDMM, fp32:  C[p] = sum_k A[row(p),k] * B[indices[p],k]   (optionally times scale[p])
// Semantics: tests/python/sparsetir/sparse_tir_lowered_buffer_scripts.py:458-507 (sddmm) and
// :510-569 (fused_sddmm with the edge->row binary search) of the reference; generated kernel
// being replaced: examples/sddmm/bench_sddmm.py:97-167.
//
// The reference runs a separate preprocess kernel that stores row(p) for every stored position and
// then gives every (ty, group) slot one edge with the dot product split over tx lanes and reduced
// across threads.  Here one kernel does both: a warp owns a contiguous range of stored positions and
// finds their rows itself, a sub-warp loads the B row of one position at a time (several positions
// in flight) and keeps one partial sum per position, and the partial sums of several positions are
// reduced together by a transposing butterfly, so that the warp stores 32 consecutive results with
// one coalesced store.
#include <cstdint>
#include <cstdlib>

#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "row_walk.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;

// General kernel: any feature count and alignment, rows of any length.
//
// A warp owns `chunk` consecutive positions and takes them 32 at a time; their rows come out of a
// register window of row ends (row_walk.cuh).  Its sub-warps of LPR lanes take LPR positions each,
// eight at a time: the rows of B of U positions and, where the row changes, their rows of A are
// requested together, so that a matrix of short rows does not wait for A once per row (169 k-node
// power-law graph, 5 entries per row, F = 64: 66 us when it did).  The feature tiles are walked
// inside the kernel, the eight sums staying in registers; seven shuffles transpose and add them
// over eight lanes, one more per doubling of the group adds the rest.
//
// What bounds it on short rows is the latency of the gathers (169 k rows of 5 entries, F = 64, counters of one launch: 17 of
// the 23 warps per issued instruction wait for memory, L1 data path 35 %, L2 32 %, issue slots 22 %, DRAM 30 %).  Groups of
// 8 lanes of 32 bytes have as many bytes in flight as 16 lanes of 16 bytes and four positions where those had two: power-law graphs, us, before / with them: 169 k rows, F = 64 43.1 / 31.9, 200 k rows
// F = 192 131 / 102, F = 128 72 / 67, 20 k rows F = 128 10.1 / 8.6.  Groups of 16 such lanes gain nothing (F = 256 137 / 141).
//
// Five blocks per SM with one position in flight per group, where four had two (BLOCKS): B in L2 far from the SMs is waited for longer, and
// a fifth more warps bring more than the second position (us, two on four blocks / one on five: 169 k power-law rows, F = 64 31 / 28.6,
// 110 k rows of 12 F = 64 28.9 / 26.3, F = 256 164 / 149, 130 k of 20 F = 64 55.4 / 49.5, 80 k of 11 F = 512 219 / 205).  Only where that spares a round
// of positions (five_blocks(); 20 k of 11, F = 512, 41.1 / 45.1, 50 k of 12 125 / 137, 40 k of 11 92 / 102 spare none).  Four positions on three or two
// blocks: 42.7, 52.2 on the first of these; two on five and one on six blocks spill (35.9, 31.4).  16-byte lanes spill on four, 36 features and
// 100, 20 k rows of 11, a warp or half of one to a row / four blocks / five 8.7 / 13.2 / 7.3 and 14.1 / 21.3 / 11.7, 3 k of 11 4.3 / 5.1 / 4.0
// and 6.0 / 7.7 / 5.9.
constexpr size_t kFarBytes = size_t{24} << 20;
template <int LPR, int W, int VPL, bool PEERS, int BLOCKS>
__global__ void __launch_bounds__(kThreads, BLOCKS)
sddmm_kernel(const float* a, const float* b, float* __restrict__ c,
             const int32_t* indptr, const int32_t* indices,
             const float* scale, int m, int feat, int nnz, int chunk, float rows_per_entry,
             const __grid_constant__ PeerOut po) {
  using LT = LaneTile<LPR, W, VPL, false>;
  using V = typename LT::Piece;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int U = BLOCKS == 5 ? 1 : W == 8 || VPL == 4 ? 2 : VPL * W >= 4 ? 4 : 8;  // positions in flight; four of four single floats spill
  const int wlane = threadIdx.x & 31;
  const int lane = wlane % LPR;
  const int sub = wlane / LPR;
  const long long warp = static_cast<long long>(blockIdx.x) * (kThreads / 32) + threadIdx.x / 32;
  const long long begin = warp * chunk;
  chain_wait();
  if (begin >= nnz) return;
  const int e0 = static_cast<int>(begin);
  const int count = static_cast<int>(min(static_cast<long long>(chunk), nnz - begin));
  const unsigned row_bytes = static_cast<unsigned>(feat) * 4u;
  const char* ab = reinterpret_cast<const char*>(a);
  const char* bb = reinterpret_cast<const char*>(b);
  const int tiles = (feat + LT::kFloats - 1) / LT::kFloats;

  int col = wlane < count ? ld_global(indices + e0 + wlane) : 0;
  int r = warp_row_of(indptr, m, e0, rows_per_entry, wlane);
  int wend = row_window<32>(indptr, m, r, wlane);
  for (int s0 = 0; s0 < count; s0 += 32) {
    const bool live = wlane < count - s0;
    const int e = e0 + min(s0 + wlane, count - 1);  // lanes past the last position repeat its row
    int col_next = 0;
    if (s0 + 32 + wlane < count) col_next = ld_global(indices + e0 + s0 + 32 + wlane);
    const float mul = live && scale != nullptr ? ld_global(scale + e) : 1.f;
    int row_end;
    const int row = row_in_window<32>(indptr, m, r, wend, e, row_end);
    r = __shfl_sync(kAll, row, 31);
    wend = row_window<32>(indptr, m, r, wlane);
    // bit k: position k of this sub-warp is in another row than position k - 1
    const int row_before = __shfl_up_sync(kAll, row, 1, LPR);
    const unsigned changes = __ballot_sync(kAll, lane == 0 || row != row_before) >> (sub * LPR);
    float out = 0.f;
#pragma unroll
    for (int g = 0; g < LPR / 8; ++g) {
      float part[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) part[k] = 0.f;
      for (int t = 0; t < tiles; ++t) {
        const LT lt(feat, t, lane);
        V arow = LT::zero();
#pragma unroll
        for (int h = 0; h < 8; h += U) {
          V x[U], ar[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int k = g * 8 + h + u;
            const unsigned ck = static_cast<unsigned>(__shfl_sync(kAll, col, k, LPR));
            const unsigned rk = static_cast<unsigned>(__shfl_sync(kAll, row, k, LPR));
            x[u] = lt.ldg(bb + static_cast<unsigned long long>(ck) * row_bytes);
            if (h + u == 0 || ((changes >> k) & 1u)) ar[u] = lt.ldg(ab + static_cast<unsigned long long>(rk) * row_bytes);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int k = g * 8 + h + u;
            if (h + u == 0 || ((changes >> k) & 1u)) arow = ar[u];
            part[h + u] += lt.dot(arow, x[u]);
          }
        }
      }
#pragma unroll
      for (int off = 4, n = 8; off >= 1; off >>= 1, n >>= 1) {  // afterwards part[0] is position lane % 8
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
          const float send = upper ? part[i] : part[i + n / 2];
          const float keep = upper ? part[i + n / 2] : part[i];
          part[i] = keep + __shfl_xor_sync(kAll, send, off);
        }
      }
#pragma unroll
      for (int off = 8; off < LPR; off <<= 1) part[0] += __shfl_xor_sync(kAll, part[0], off);
      if (lane / 8 == g) out = part[0];
    }
    if (live) {
      const float v = out * mul;
      c[e] = v;
      if constexpr (PEERS)
        for (int k = 0; k < po.n; ++k)
          *reinterpret_cast<float*>(reinterpret_cast<char*>(c + e) + po.delta[k]) = v;
    }
    col = col_next;
  }
}

// A product that came out as a NaN, feature by feature.
__device__ __noinline__ float plain_dot(const float* a, const float* b, int feat) {
  float s = 0.f;
  for (int f = 0; f < feat; ++f) s = fmaf(ld_global(a + f), ld_global(b + f), s);
  return s;
}

// ---------------------------------------------------------------------------------------------
// Lean variant for feature counts that are multiples of 32, or of 8 and below 128 (PART), with 32-byte aligned operands.
//
// One launch covers a tile of 8*LPR consecutive features [foff, foff + 8*LPR) of every stored
// position; the host walks the tiles with one launch each, the first storing C and the others
// adding to it, and picks the tile so that the slice of B a launch gathers from stays in L2.
// A lane owns 8 consecutive features: one 256-bit load per gathered row, the dot product as
// packed two-wide fp32 FMAs.  A warp owns `chunk` consecutive positions, finds the row of its
// first position together (row(p) = upper bound - 1, the search of
// sparse_tir_lowered_buffer_scripts.py:530-549), and loads the column ids of the next batch before it
// gathers for this one.  It keeps the row of A that it is in: for matrices of 10 entries per row and more (sddmm_run).
//
// Batches in which rows end.  Rows that are short beside the average make most batches such ones, and a matrix whose rows vary has
// many of them whatever its average is.  Tiles of 64 features, and PART, find the rows of a batch in a register window of row ends
// (kWindow; up to four ends are counted, more are searched), and tiles of 64 ask for up to four rows of A together with those of B
// (kTogether).  A walk along the row pointers, lane by lane, and a row of A when it is met took, us, log-normal rows of sigma 2 and their mean,
// walk / so (groups of sddmm_kernel): 100 k rows of 30, F = 256 409 / 280, 20 k of 80, F = 64 29.1 / 25.8, 20 k of 30, F = 24 12.1 / 9.0
// (10.5), F = 40 21.5 / 18.3; rows of one length within 2 %.  Tiles of 32, 128 and 256 keep the walk (the window on 60 k rows of 15 to 70
// entries: F = 96 102 to 105 %, F = 128 97 to 101 %, F = 256 from 40 k rows 102 to 105 %, 60 k rows of log-normal lengths F = 32 and rows of A
// together 250 / 239), PART and tiles of 32 ask for rows of A one by one (together: 20 k of 30, F = 40 16.2 / 21.9, F = 24 9.1 / 10.3).
// With PEERS the finished value of every position (the last feature tile's pass) is also stored
// into the peers' copies of c: 128 contiguous bytes per warp and peer, over NVLink.
template <int LPR, bool PEERS, bool PART>
__global__ void __launch_bounds__(kThreads, LPR == 4 ? 4 : 2)
sddmm_lean_kernel(const float* a, const float* b, float* __restrict__ c,
                  const int32_t* indptr, const int32_t* indices,
                  const float* scale, int m, int nnz, int ld, int foff, int accumulate,
                  int chunk, int last_tile, const __grid_constant__ PeerOut po) {
  // Gathered rows in flight per lane (8 registers each).  Tiles of 64 features keep the eight of a batch in flight on half the blocks
  // (us, four on four blocks per SM / eight on two: 20 M positions in 40 k rows F = 64 366 / 317, 10 M in 100 k rows F = 128,
  // two tiles, 413 / 353, F = 256 827 / 704); tiles of 32 with two batches at once lose (117 M, F = 128 3720 / 4150), and so do wider
  // ones with eight (F = 128 558 / 721).
  constexpr int U = LPR == 8 ? 8 : 4;
  constexpr bool kWindow = LPR == 8 || PART, kTogether = LPR == 8 && !PART;
  const int wlane = threadIdx.x & 31;
  const int lane = wlane % LPR;
  const unsigned mask = group_mask<LPR>();
  const long long warp = static_cast<long long>(blockIdx.x) * (kThreads / 32) + threadIdx.x / 32;
  const long long e_begin = warp * chunk;
  chain_wait();
  if (e_begin >= nnz) return;
  const int e_end = static_cast<int>(min(static_cast<long long>(nnz), e_begin + chunk));
  // PART: lanes past the row load its first piece once more.  Groups of 8 and 16 multiply it by zeros, and what that makes a NaN is
  // formed again; those of 4, which have no registers for that, mask their products (20 M positions, F = 72, a select that
  // became a branch around each product 910 us, a mask, which spills, 800, zeros 595; F = 24 a mask 166, zeros 242).
  constexpr bool kMask = PART && LPR == 4, kAgain = PART && !kMask;
  const bool in = !PART || lane * 8 < ld - foff;
  const unsigned keep_bits = in ? 0xffffffffu : 0u;
  const float* a_lane = a + foff + (in ? lane * 8 : 0);
  const float* b_lane = b + foff + (in ? lane * 8 : 0);
  auto product = [&](const Pack4& p, const Pack4& q) {
    const float d = dot8(p, q);
    return kMask ? __uint_as_float(__float_as_uint(d) & keep_bits) : d;
  };
  auto row_of_a = [&](int r) { return in || kMask ? ldg256(a_lane + static_cast<size_t>(r) * ld) : pack4_zero(); };

  int warp_row = max(0, min(m - 1, warp_upper_bound(indptr, 0, m + 1, static_cast<int>(e_begin), wlane) - 1));
  // end of the warp's current row; kWindow: in lane j that of the row j behind it
  int wend = kWindow ? row_window<32>(indptr, m, warp_row, wlane) : ld_global(indptr + warp_row + 1);
  int cur_row = -1;
  Pack4 arow = pack4_zero();

  int col_next = (static_cast<int>(e_begin) + wlane < e_end) ? ld_global(indices + e_begin + wlane) : 0;
  for (int base = static_cast<int>(e_begin); base < e_end; base += 32) {
    const int e = base + wlane;
    const bool live = e < e_end;
    const int col = col_next;
    if (e + 32 < e_end) col_next = ld_global(indices + e + 32);
    float mul = 1.f, old = 0.f;
    if (live) {
      if (scale != nullptr) mul = ld_global(scale + e);
      if (accumulate) old = c[e];
    }
    float part[LPR];
    int row = warp_row;
    if (base + 32 <= min(kWindow ? __shfl_sync(0xffffffffu, wend, 0) : wend, e_end)) {
      // every position of the batch lies in the warp's current row
      if (cur_row != warp_row) {
        cur_row = warp_row;
        arow = row_of_a(cur_row);
      }
#pragma unroll
      for (int k0 = 0; k0 < LPR; k0 += U) {
        Pack4 x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          x[u] = ldg256(b_lane + static_cast<size_t>(__shfl_sync(mask, col, k0 + u, LPR)) * ld);
#pragma unroll
        for (int u = 0; u < U; ++u) part[k0 + u] = product(arow, x[u]);
      }
    } else {
      if constexpr (kWindow) {
        const int last = min(e, e_end - 1);  // dead positions: the last live one's row
        const int over = __popc(__ballot_sync(0xffffffffu, wend <= min(base + 31, e_end - 1)));  // rows that end before the batch does
        if (over <= 4) {
#pragma unroll
          for (int k = 0; k < 4; ++k) row += __shfl_sync(0xffffffffu, wend, k) <= last ? 1 : 0;
          row = min(row, m - 1);
        } else {
          int row_end;
          row = row_in_window<32>(indptr, m, warp_row, wend, last, row_end);
        }
        warp_row = __shfl_sync(0xffffffffu, row, 31);
        wend = row_window<32>(indptr, m, warp_row, wlane);
      } else {
        if (live) {
          int steps = 0;
          // row < m - 1 keeps every read inside indptr even if nnz disagrees with indptr[m]
          while (row < m - 1 && ld_global(indptr + row + 1) <= e) {
            ++row;
            if (++steps == 8) {  // long run of empty rows: finish with a search
              row = min(m - 1, edge_row_search(indptr, row, m, e));
              break;
            }
          }
        }
        // the next batch starts from the row of this batch's last live position
        warp_row = __shfl_sync(0xffffffffu, row, min(31, e_end - 1 - base));
        wend = ld_global(indptr + warp_row + 1);
      }
      if constexpr (kTogether) {
        constexpr int UM = 4;  // rows of B in flight beside as many of A
#pragma unroll
        for (int k0 = 0; k0 < LPR; k0 += UM) {
          Pack4 x[UM], ar[UM];
          bool other[UM];  // uniform inside the sub-warp
#pragma unroll
          for (int u = 0; u < UM; ++u) {  // dead positions carry column 0
            const int rk = __shfl_sync(mask, row, k0 + u, LPR);
            x[u] = ldg256(b_lane + static_cast<size_t>(__shfl_sync(mask, col, k0 + u, LPR)) * ld);
            other[u] = rk != cur_row;
            if (other[u]) ar[u] = ldg256(a_lane + static_cast<size_t>(rk) * ld);
            cur_row = rk;
          }
#pragma unroll
          for (int u = 0; u < UM; ++u) {
            if (other[u]) arow = ar[u];
            part[k0 + u] = product(arow, x[u]);
          }
        }
      } else {
#pragma unroll
        for (int k0 = 0; k0 < LPR; k0 += U) {
          Pack4 x[U];
          int rk[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {  // dead positions carry column 0 and the warp's row
            rk[u] = __shfl_sync(mask, row, k0 + u, LPR);
            x[u] = ldg256(b_lane + static_cast<size_t>(__shfl_sync(mask, col, k0 + u, LPR)) * ld);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (rk[u] != cur_row) {  // uniform inside the sub-warp
              cur_row = rk[u];
              arow = row_of_a(cur_row);
            }
            part[k0 + u] = product(arow, x[u]);
          }
        }
      }
    }
    // transposing butterfly: afterwards part[0] of lane l is the dot product of position l
#pragma unroll
    for (int offl = LPR / 2, n = LPR; offl >= 1; offl >>= 1, n >>= 1) {
      const bool upper = (lane & offl) != 0;
#pragma unroll
      for (int i = 0; i < n / 2; ++i) {
        const float send = upper ? part[i] : part[i + n / 2];
        const float keep = upper ? part[i + n / 2] : part[i];
        part[i] = keep + __shfl_xor_sync(mask, send, offl, LPR);
      }
    }
    if (live) {
      if constexpr (kAgain) {
        if (part[0] != part[0]) part[0] = plain_dot(a + static_cast<size_t>(row) * ld, b + static_cast<size_t>(col) * ld, ld);
      }
      const float v = fmaf(part[0], mul, old);
      c[e] = v;
      if constexpr (PEERS) {
        if (last_tile)
          for (int k = 0; k < po.n; ++k)
            *reinterpret_cast<float*>(reinterpret_cast<char*>(c + e) + po.delta[k]) = v;
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads)
edge_to_row_kernel(const int32_t* indptr, int32_t* __restrict__ mid, int m, int nnz) {
  const long long p = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  if (p < nnz) mid[p] = edge_row_search(indptr, 0, m, static_cast<int>(p));
}

template <int LPR, int W, int VPL, int BLOCKS = 4>
int launch(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
           const float* scale, int m, int feat, int nnz, const PeerOut& po, cudaStream_t stream) {
  // one wave of resident blocks; two for the narrow vectors, whose positions take longer (50 k-node
  // power-law graph, F = 299: 88 against 97 us), but one of them, with more positions per warp, where the second would be filled to less than 0.6
  // (pairs, two waves / one, 1.06 of them, 80 k rows of 5, F = 298 131 / 105 us, 1.16, 20 k of 11, F = 190 26.3 / 22.7; 1.69, 80 k of 8,
  // F = 46 25.6 / 26.9)
  const long long wave = static_cast<long long>(kNumSMs) * BLOCKS * (kThreads / 32);
  auto chunk_of = [&](long long warps) { return (static_cast<int>((nnz + warps - 1) / warps) + 31) & ~31; };
  int chunk = chunk_of(W < 4 ? 2 * wave : wave);
  if (W < 4 && BLOCKS == 5) {
    const long long last = ceil_div(nnz, chunk) - wave;  // warps of the second
    if (last > 0 && last * 10 < wave * 6) chunk = chunk_of(wave);
  }
  const int blocks = ceil_div(ceil_div(nnz, chunk), kThreads / 32);
  const float rows_per_entry = static_cast<float>(m) / static_cast<float>(nnz);
  if constexpr (W >= 4 && BLOCKS == 4) {
    if (po.n > 0) {
      launch_chained_if(nnz < kChainEntries, sddmm_kernel<LPR, W, VPL, true, BLOCKS>, blocks, kThreads, 0, stream, a, b, c, indptr, indices, scale, m,
                        feat, nnz, chunk, rows_per_entry, po);
      SPTIR_LAUNCH_OK("sddmm_kernel");
      return 0;
    }
  }
  launch_chained_if(nnz < kChainEntries, sddmm_kernel<LPR, W, VPL, false, BLOCKS>, blocks, kThreads, 0, stream, a, b, c, indptr, indices, scale, m, feat,
                    nnz, chunk, rows_per_entry, po);
  SPTIR_LAUNCH_OK("sddmm_kernel");
  return 0;
}

// Blocks of sddmm_lean_kernel<LPR> that fit one SM at a time (asked of the runtime once per device).
template <int LPR, bool PART>
int lean_blocks_per_sm() {
  static thread_local int cached_device = -1, cached = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 4;
  if (dev != cached_device) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sddmm_lean_kernel<LPR, false, PART>, kThreads, 0) != cudaSuccess || n < 1)
      n = 4;
    cached = n;
    cached_device = dev;
  }
  return cached;
}

template <int LPR, bool PART>
int launch_lean_tile(const float* a, const float* b, float* c, const int32_t* indptr,
                     const int32_t* indices, const float* scale, int m, int feat, int nnz, int foff,
                     int last_tile, const PeerOut& po, cudaStream_t stream) {
  // About 1024 positions per warp amortise the row search, in whole waves of resident blocks: a
  // launch of a few waves ends with a partly filled one otherwise (3.02 waves cost as much as 4;
  // 1.7 M positions, F = 64: 59 us in 1.4 waves of 256 positions per warp).
  const int wpb = kThreads / 32;
  const long long resident = static_cast<long long>(kNumSMs) * lean_blocks_per_sm<LPR, PART>() * wpb;
  const long long waves = std::max<long long>(1, (nnz / 1024 + resident / 2) / resident);
  int chunk = 1024;
  if (waves < 8) chunk = static_cast<int>((nnz + waves * resident - 1) / (waves * resident) + 31) & ~31;
  const int blocks = ceil_div(ceil_div(nnz, chunk), wpb);
  if constexpr (!PART) {
    if (po.n > 0) {
      launch_chained_if(nnz < kChainEntries, sddmm_lean_kernel<LPR, true, false>, blocks, kThreads, 0, stream, a, b, c, indptr, indices, scale, m,
                        nnz, feat, foff, foff != 0, chunk, last_tile, po);
      SPTIR_LAUNCH_OK("sddmm_lean_kernel");
      return 0;
    }
  }
  launch_chained_if(nnz < kChainEntries, sddmm_lean_kernel<LPR, false, PART>, blocks, kThreads, 0, stream, a, b, c, indptr, indices, scale, m, nnz, feat,
                   foff, foff != 0, chunk, last_tile, po);
  SPTIR_LAUNCH_OK("sddmm_lean_kernel");
  return 0;
}

// What stays resident in L2 of data that every SM reads (about half of the 126 MB);
// SPARSETIR_L2_BUDGET_MB overrides it for tuning on other parts.
size_t l2_budget_bytes() {
  static const size_t budget = [] {
    const char* e = std::getenv("SPARSETIR_L2_BUDGET_MB");
    const long mb = e ? std::atol(e) : 0;
    return static_cast<size_t>(mb > 0 ? mb : 48) << 20;
  }();
  return budget;
}

// feat is a multiple of 32: the widest tile (32..256 features) that divides feat and whose
// slice of B (n rows) fits the L2 budget.
int lean_tile(int n, int feat) {
  for (int t = 256; t > 32; t /= 2)
    if (feat % t == 0 && static_cast<size_t>(n) * t * 4 <= l2_budget_bytes()) return t;
  return 32;
}

// Whether a call of whole 32-feature tiles takes the general kernel in groups of 8 lanes of 32 bytes.  It reads the
// whole row of B and of A at every position, so it wants B in L2 as a whole, where the lean kernel needs a slice of it
// and keeps the row of A.  All figures: us, lean / groups, of 60 matrices of equal and of log-normal rows.
//  - Rows of less than 10 entries: always (power-law graphs, the header of sddmm_kernel).
//  - 64 features in one launch of the lean one: rows of up to 64 entries, 100 where B is far (20 k of 24 12.7 / 12.4, of 40 17.1 / 17.4, of 80 26.8 /
//    30.1, 60 k of 40 44.1 / 43.3, of 80 84 / 86, 150 k of 40 128 / 112, 100 k of 80, log-normal of sigma 1 149 / 138, 140 k of 70 186 / 177).
//  - In place of several launches: rows of up to 50 entries (F = 96: 60 k of 24 56 / 49, 20 k of 80 49.4 / 49.5; F = 64: 233 k of 50
//    248 / 235, of 80 349 / 363, of 500 1734 / 2241), and B up to a share of the L2 budget that grows with the launches
//    saved: F = 512, two, 20 k of 30 87 / 77, 30 k 136 / 141; F = 256, two, 50 k of 30 109 / 103, 80 k 182 / 225; F = 96,
//    three narrow ones, 100 k of 30 108 / 99, 150 k 162 / 167, 200 k 219 / 270; F = 64, two, 200 k of 30 147 / 121, 300 k
//    of 45 at 0.91; F = 128, two, 150 k of 24 186 / 171, of 40 267 / 266; F = 192, three, 60 k of 24 108 / 78, 150 k 277 / 308.
//  - In place of three launches and more over tiles of 32 or 64, which read and add to C once for each, if the groups fill seven eighths of
//    their tiles of 64: rows of any length while B fits (20 k rows of 200 F = 192 179 / 177, F = 224 231 / 222, F = 288 299 / 275, F = 320 306 / 288,
//    F = 448 431 / 400; 60 k of 200 F = 192 610 / 549; F = 160, five sixths, 165 / 168, and F = 96 99 / 117 do not).
bool in_groups(int m, int n, int feat, int nnz) {
  const int per_row = nnz / m, tile = lean_tile(n, feat);
  if (feat < 64) return false;
  if (per_row < 10) return true;
  const size_t b_bytes = static_cast<size_t>(n) * feat * 4;
  if (feat == tile) return feat == 64 && per_row < (b_bytes >= kFarBytes ? 100 : 64);
  if (tile <= 64 && feat / tile >= 3 && feat * 8 >= ceil_div(feat, 64) * 64 * 7 && b_bytes <= l2_budget_bytes()) return true;
  const int eighths = tile == 256 || feat == 96 ? 8 : tile == 128 ? 9 : feat == 64 ? 11 : 13;
  return per_row < (feat == 64 ? 64 : 50) && b_bytes <= l2_budget_bytes() / 8 * eighths;
}

// Whether groups of 32-byte lanes run on five blocks per SM: where the positions make fewer rounds of 32 per warp of them (us, four / five, 160 k
// positions, F = 64 6.1 / 5.2, F = 256 15.6 / 12.3, 80 k power-law rows F = 128 33.1 / 25.8, 120 k 44.5 / 37.4, 200 k 67.5 / 61.1; as many rounds, 200 k
// positions 6.4 / 6.7 and 16.3 / 17.8, power-law rows 101 k F = 128 34.8 / 35.4, F = 256 65.9 / 67.3, 60 k F = 512 82.6 / 84.5), of few rounds, where
// one counts, or with a large B (40 k rows of 20, F = 256 59 / 57, 50 k of 30, F = 512 295 / 262, but 20 k of 30, F = 64 12.3 / 12.7).
bool five_blocks(int n, int feat, int nnz) {
  const int round = kNumSMs * (kThreads / 32) * 32;
  const int four = ceil_div(nnz, 4 * round), five = ceil_div(nnz, 5 * round);
  return five < four && (four <= 3 || static_cast<size_t>(n) * feat * 4 >= kFarBytes);
}

// Feature counts in steps of 8 below 128 whose lanes the lean kernel fills better than the groups fill their tiles of 64, on rows long
// enough for it and with a B that stays in L2 (us, groups / lean: 40 k rows of 500 F = 40 461 / 397, F = 104 711 / 611, F = 72 572 / 605,
// F = 136 815 / 1146; 60 k of 60 F = 88 126 / 138; 20 k of 11 F = 40 7.9 / 8.7, of 30 16.6 / 16.2, F = 104 24.5 / 23.9; F = 24, a group of 8 / lean, 20 k
// of 11 5.4 / 5.6, 60 k of 30 26.2 / 21.6).  The lean kernel has half the blocks: not where the positions make one round of the groups
// (10 k of 11 F = 40 4.9 / 6.5, 3 k of 30 4.7 / 5.9).
bool lean_part(int m, int n, int feat, int nnz) {
  if (feat % 8 != 0 || feat % 32 == 0 || feat >= 128 || (feat > 64 && feat < 96)) return false;
  if (feat > 32 && nnz < 120000) return false;
  return nnz / m >= (feat < 64 ? 16 : 24) && static_cast<size_t>(n) * feat * 4 <= l2_budget_bytes();
}

// One launch per tile, in stream order.
int launch_lean(const float* a, const float* b, float* c, const int32_t* indptr,
                const int32_t* indices, const float* scale, int m, int n, int feat, int nnz,
                const PeerOut& po, cudaStream_t stream) {
  const int tile = lean_tile(n, feat);
  for (int foff = 0; foff < feat; foff += tile) {
    int rc;
    const int last = foff + tile >= feat;
    switch (tile) {
      case 256: rc = launch_lean_tile<32, false>(a, b, c, indptr, indices, scale, m, feat, nnz, foff, last, po, stream); break;
      case 128: rc = launch_lean_tile<16, false>(a, b, c, indptr, indices, scale, m, feat, nnz, foff, last, po, stream); break;
      case 64: rc = launch_lean_tile<8, false>(a, b, c, indptr, indices, scale, m, feat, nnz, foff, last, po, stream); break;
      default: rc = launch_lean_tile<4, false>(a, b, c, indptr, indices, scale, m, feat, nnz, foff, last, po, stream); break;
    }
    if (rc != 0) return rc;
  }
  return 0;
}

// Other feature counts in steps of 8, in one launch whose last lanes are idle.
int launch_lean_part(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices, const float* scale,
                     int m, int feat, int nnz, cudaStream_t stream) {
  const PeerOut none{};
  if (feat > 64) return launch_lean_tile<16, true>(a, b, c, indptr, indices, scale, m, feat, nnz, 0, 1, none, stream);
  if (feat > 32) return launch_lean_tile<8, true>(a, b, c, indptr, indices, scale, m, feat, nnz, 0, 1, none, stream);
  return launch_lean_tile<4, true>(a, b, c, indptr, indices, scale, m, feat, nnz, 0, 1, none, stream);
}

}  // namespace
}  // namespace sptir

namespace sptir {
namespace {
int sddmm_run(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
              const float* scale, int m, int n, int feat, int nnz, int device_id, void* stream,
              const PeerOut& po) {
  if (m < 0 || n < 0 || feat < 0 || nnz < 0) return fail("sparsetir_sddmm: negative size");
  if (nnz == 0) return 0;
  if (m < 1) return fail("sparsetir_sddmm: %d stored entries but no rows", nnz);
  if (!c || !indptr || !indices || (feat > 0 && (!a || !b)))
    return fail("sparsetir_sddmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled() && validate_csr("sparsetir_sddmm", indptr, m, indices, nnz, n, st) != 0) return -1;
  const bool lean = feat > 0 && feat % 32 == 0 && aligned32(a) && aligned32(b);
  if (po.n > 0 && !lean)
    return fail("sparsetir_sddmm_peers: needs feat_size a positive multiple of 32 and 32-byte aligned a and b; "
                "run sparsetir_sddmm and sparsetir_peer_scatter instead");
  if (feat == 0) {
    SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, static_cast<size_t>(nnz) * sizeof(float), st));
    return 0;
  }
  if (lean && in_groups(m, n, feat, nnz)) {
    if (po.n == 0 && five_blocks(n, feat, nnz)) return launch<8, 8, 1, 5>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
    return launch<8, 8, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  }
  // The lean kernel where rows are long enough for it: it asks for a row of A when it meets one.
  if (lean && nnz / m >= 10) return launch_lean(a, b, c, indptr, indices, scale, m, n, feat, nnz, po, st);
  if (lean_part(m, n, feat, nnz) && aligned32(a) && aligned32(b)) return launch_lean_part(a, b, c, indptr, indices, scale, m, feat, nnz, st);
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b);
  // Groups of 8 lanes with 64 features between them, of 16 where a lane holds single floats.  With a warp to a row of more than 64
  // features, and two positions of more than 32 (us, power-law graphs of 80 k rows, that / now: F = 72 21.1 / 15.6, F = 136 44 / 27, F = 100
  // 29.2 / 18.7, F = 260 75 / 55, F = 46 21.5 / 17.9, F = 190 71 / 47, F = 41 27.7 / 21.4, F = 189 96 / 83).
  if (feat % 8 == 0 && feat > 32 && bits % 32 == 0) {
    if (five_blocks(n, feat, nnz)) return launch<8, 8, 1, 5>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
    return launch<8, 8, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  }
  if (feat % 4 == 0 && bits % 16 == 0) {
    if (feat <= 32) return launch<8, 4, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
    return launch<8, 4, 2, 5>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  }
  if (feat % 2 == 0 && bits % 8 == 0) {
    if (feat <= 16) return launch<8, 2, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
    if (feat <= 32) return launch<16, 2, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
    return launch<8, 2, 4, 5>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  }
  if (feat <= 8) return launch<8, 1, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  if (feat <= 16) return launch<16, 1, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  if (feat <= 32) return launch<32, 1, 1>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
  return launch<16, 1, 4>(a, b, c, indptr, indices, scale, m, feat, nnz, po, st);
}
}  // namespace
}  // namespace sptir

extern "C" int sparsetir_sddmm_raw(const float* a, const float* b, float* c, const int32_t* indptr,
                                   const int32_t* indices, const float* scale, int m, int n,
                                   int feat, int nnz, int device_id, void* stream) {
  return sptir::sddmm_run(a, b, c, indptr, indices, scale, m, n, feat, nnz, device_id, stream, sptir::PeerOut{});
}

extern "C" int sparsetir_sddmm_peers_raw(const float* a, const float* b, float* c, const int32_t* indptr,
                                         const int32_t* indices, const float* scale, int m, int n,
                                         int feat, int nnz, int n_peers, void* const* peer_c,
                                         int device_id, void* stream) {
  sptir::PeerOut po{};
  if (sptir::peer_table("sparsetir_sddmm_peers", c, n_peers, peer_c, 4, &po) != 0) return -1;
  return sptir::sddmm_run(a, b, c, indptr, indices, scale, m, n, feat, nnz, device_id, stream, po);
}

extern "C" int sparsetir_sddmm_edge_to_row_raw(const int32_t* indptr, int32_t* mid, int m, int nnz,
                                               int device_id, void* stream) {
  using namespace sptir;
  if (m < 0 || nnz < 0) return fail("sparsetir_sddmm_edge_to_row: negative size");
  if (nnz == 0) return 0;
  if (!indptr || !mid) return fail("sparsetir_sddmm_edge_to_row: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  edge_to_row_kernel<<<ceil_div(nnz, kThreads), kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      indptr, mid, m, nnz);
  SPTIR_LAUNCH_OK("edge_to_row_kernel");
  return 0;
}

// Decomposed hyb SpMM, fp32: for every (partition, bucket) array q, ELL row r, slot s
//     C[rows_q[r], :] (+)= W_q[r,s] * B[cols_q[r,s], :]
// Replaces the horizontally fused kernel the reference generates in
// examples/spmm/bench_spmm.py:116-199 (argument list :207-222).  As there, ONE launch covers
// all buckets: the blockIdx.x range is the concatenation of the buckets' block ranges
// (the idea of src/tir/transforms/horizontal_fusion.cc:80-171), described by a small table
// passed by value in the kernel parameters — no device-side scratch, no host->device copy.
//
// Differences from the reference schedule, all invisible in the results:
//  - a work item (one sub-warp) covers about item_slots() stored slots whatever the bucket:
//    several ELL rows of a narrow bucket, or one item_slots()-slot piece of an ELL row of a wide
//    bucket.  Equal-sized items keep every SM busy until the end of the launch; the reference
//    equalises per block instead (8 * maxBucket slots per block, bench_spmm.py:187-189).
//    Wide buckets are scheduled first.
//  - the reference marks whole buckets atomic (bench_spmm.py:170,174-177).  Here the main (lean)
//    kernel gives every output row one writer: the pieces of a wide ELL row meet in shared memory,
//    the ELL rows of a row that the format split (src/sparse/format.cc:110-116: consecutive ELL
//    rows of the widest bucket repeating the row id) meet in a scratch buffer and are added in
//    order by the last one to finish — no atomics on the output, the same bits on every run.
//    The fallback kernels for odd shapes decide from the data instead: pieces of a chunked wide
//    ELL row and ELL rows whose id equals a neighbour's are added with vector atomics.
//    With several column partitions the same output row appears in several arrays, which the
//    kernels cannot see; the caller says so with SPARSETIR_HYB_ALL_ATOMIC.
#include <algorithm>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "common.h"
#include "launch.cuh"
#include "spmm_core.cuh"

namespace sptir {
namespace {

#ifndef SPTIR_HYB_MIN_BLOCKS
#define SPTIR_HYB_MIN_BLOCKS 3  // resident blocks per SM the register budget is sized for
#endif
constexpr int kThreads = 128;
constexpr int kMaxB = SPARSETIR_HYB_MAX_BUCKETS;

// Stored slots covered by one work item (one sub-warp of `lpr` lanes): four id batches, so that
// the per-item set-up is amortised and the id prefetch of spmm_core.cuh has something to hide.
constexpr int item_slots(int lpr) { return 4 * lpr; }
// lean kernel: lpr lanes of w floats each, `tiles` feature tiles (blockIdx.y), `slots` stored
// slots in all buckets.  Batches of ids per item, measured on the 169,343-node power-law graph
// (945,629 slots): with four feature tiles or more, 8 batches of 16-byte lanes (step over
// F = 32..512 0.385 ms; 4 batches 0.394, 12 batches 0.425, 16 batches 0.448; F = 128 59 against
// 64 us, F = 512 183 against 188 us) — longer items hide more of the id loads; with fewer tiles 4
// batches (F = 32: 26.0 against 27.3 us).  Row shards of that graph (half or a quarter of the
// slots) lose 5-9 % with 8 batches (F = 512 on half: 115 against 109 us): a pass over one feature
// tile then has too few blocks, so the longer items are for launches of 3/4 M slots or more.
// 32-byte lanes: 8 batches (the row ids of an item's rows of 8 slots or more travel in one
// register per lane, which caps an item at lpr such rows).
inline int lean_item_slots(int lpr, int w, int tiles, long long slots) {
  return lpr * w * ((w == 4 && tiles >= 4 && slots >= 3 * (1ll << 18)) ? 2 : 1);
}

struct HybTable {
  const float* w[kMaxB];
  const int32_t* rows[kMaxB];
  const int32_t* cols[kMaxB];
  int32_t nrows[kMaxB];
  int32_t width[kMaxB];
  int32_t rows_per_item[kMaxB];    // >= 1; 1 for chunked buckets
  int32_t chunks_per_row[kMaxB];   // 1 unless width > item_slots (lean kernel: sub-warps per ELL row)
  int32_t block_start[kMaxB + 1];
  int32_t row_base[kMaxB];         // buckets without a row-id array: ELL row r -> output row base + r
  int32_t part_base[kMaxB];        // lean kernel: scratch row of ELL row 0, or -1 (bucket has no split rows)
  int32_t nb;
};

__device__ __forceinline__ int find_bucket(const HybTable& tb, int block) {
  int q = 0;
  while (q + 1 < tb.nb && block >= tb.block_start[q + 1]) ++q;
  return q;
}

// A bucket without a row-id array (`rows == nullptr`) writes ELL row r to output row base + r.
__device__ __forceinline__ int row_id(const int32_t* rows, int r, int base) {
  return rows != nullptr ? ld_global(rows + r) : base + r;
}

__device__ __forceinline__ bool is_split_row(const int32_t* rows, int r, int nrows,
                                             int row) {
  if (rows == nullptr) return false;
  return (r > 0 && ld_global(rows + r - 1) == row) || (r + 1 < nrows && ld_global(rows + r + 1) == row);
}

template <int LPR, int VPL, int VEC>
__global__ void __launch_bounds__(kThreads, SPTIR_HYB_MIN_BLOCKS)
hyb_spmm_kernel(const __grid_constant__ HybTable tb, const float* b,
                float* __restrict__ c, int feat, int all_atomic) {
  using V = typename Vec<VEC>::type;
  constexpr int SUBS = kThreads / LPR;
  constexpr int ITEM = item_slots(LPR);
  // row ids of the item's ELL rows and of the two neighbouring ELL rows (-1 outside the
  // bucket): read at every row end, so they must not cost a trip to global memory there
  __shared__ int32_t s_rows[SUBS][ITEM + 2];
  const int lane = threadIdx.x % LPR;
  const int sub = threadIdx.x / LPR;
  const unsigned mask = group_mask<LPR>();
  const int q = find_bucket(tb, blockIdx.x);
  const int width = tb.width[q], nrows = tb.nrows[q];
  const int rpi = tb.rows_per_item[q], cpr = tb.chunks_per_row[q];
  const long long item = static_cast<long long>(blockIdx.x - tb.block_start[q]) * SUBS + sub;
  // slot range [first, first + nslots) of the bucket's flat slot array; `per_row` slots
  // complete one output contribution
  long long r0l;
  int nslots, per_row, nr;
  size_t first;
  if (cpr == 1) {
    r0l = item * rpi;
    if (r0l >= nrows) return;
    nr = static_cast<int>(min(static_cast<long long>(nrows), r0l + rpi) - r0l);
    nslots = nr * width;
    per_row = width;
    first = static_cast<size_t>(r0l) * width;
  } else {
    r0l = item / cpr;
    if (r0l >= nrows) return;
    const int s0 = static_cast<int>(item % cpr) * ITEM;
    nr = 1;
    nslots = min(ITEM, width - s0);
    per_row = nslots;
    first = static_cast<size_t>(r0l) * width + s0;
  }
  const int r0 = static_cast<int>(r0l);
  const int32_t* rows = tb.rows[q];
  for (int j = lane; j < nr + 2; j += LPR) {
    const int idx = r0 - 1 + j;
    s_rows[sub][j] = (idx >= 0 && idx < nrows) ? row_id(rows, idx, tb.row_base[q]) : -1;
  }
  __syncwarp(mask);
  const FeatLane<LPR, VPL, VEC> fl(feat, blockIdx.y, lane);
  V* cv = reinterpret_cast<V*>(c);
  const bool always_atomic = all_atomic || cpr > 1;

  V acc[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) acc[v] = Vec<VEC>::zero();
  int j = 1, left = per_row;  // s_rows[sub][j] is the id of the ELL row being accumulated
  auto on_done = [&](V(&)[VPL], int n) {
    left -= n;
    if (left != 0) return;
    const int row = s_rows[sub][j];
    const bool atomic = always_atomic || s_rows[sub][j - 1] == row || s_rows[sub][j + 1] == row;
    V* dst = cv + static_cast<size_t>(row) * fl.row_vecs;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (fl.valid[v]) {
        if (atomic) Vec<VEC>::atomic_add(dst + fl.off[v], acc[v]);
        else __stcs(dst + fl.off[v], acc[v]);  // written once: do not displace B rows in L2
      }
      acc[v] = Vec<VEC>::zero();
    }
    ++j;
    left = per_row;
  };
  const int32_t* cols = tb.cols[q] + first;
  const float* wts = tb.w[q] + first;
  const V* bv = reinterpret_cast<const V*>(b);
  // Row ends fall on chunk boundaries when the row length is a multiple of the chunk: then the
  // row-end test runs once per chunk instead of once per slot.
  const bool per_slot = per_row % ChunkOf<LPR, VPL>::value != 0;
  const bool full = feat % (LPR * VPL * VEC) == 0;
  if (per_slot) {
    if (full) stream_slots<LPR, VPL, VEC, true, true>(cols, wts, nslots, bv, fl, lane, mask, acc, on_done);
    else stream_slots<LPR, VPL, VEC, true, false>(cols, wts, nslots, bv, fl, lane, mask, acc, on_done);
  } else {
    if (full) stream_slots<LPR, VPL, VEC, false, true>(cols, wts, nslots, bv, fl, lane, mask, acc, on_done);
    else stream_slots<LPR, VPL, VEC, false, false>(cols, wts, nslots, bv, fl, lane, mask, acc, on_done);
  }
}

// ---------------------------------------------------------------------------------------------
// Lean kernel: ELL widths of 1, 2, 4 or a multiple of 8 (every power-of-two bucket list), any
// feature count and alignment.  Feature counts that are not whole tiles and rows that are not whole
// 16-byte vectors run it with predicated or narrower vectors instead of the kernels below (F = 100
// on a 100 k-node power-law graph 58 -> 35 us, F = 41 on 60 k nodes 50 -> 16 us, F = 184 on 194 k
// nodes with 36 entries per row in two column partitions 1065 -> 566 us).  Written for instruction
// economy — the gathers come from L2 at well over 10 TB/s if, and only if, the warp spends its
// issue slots on loads: per stored slot the loop executes one address + one 16-byte load and four
// FMAs, and between them two shuffles or half a read of shared memory (enum Hand below); row ends sit at compile-time positions of the
// unrolled batch (narrow rows) or are tested once per 8 slots (wide rows); row ids travel in
// registers with two flag bits, so a row end costs one shuffle and a store.
//
// Every output row has ONE writer, so results are bit-identical from run to run and nothing has
// to be cleared between calls:
//  - an ELL row wider than a work item is cut into equal spans, one per sub-warp of the SAME
//    block; the partial sums meet in shared memory and are added in span order;
//  - a row that the format split into several ELL rows (consecutive ELL rows of the widest
//    bucket repeating the row id, src/sparse/format.cc:110-116) is reduced across blocks: each
//    piece stores its partial sum in a scratch row of its own and counts itself in; the piece that
//    counts in last adds all of them in ELL-row order and writes the output row.  The counter is
//    back at zero when the launch ends.
// With SPARSETIR_HYB_ALL_ATOMIC (several column partitions: the same row in several arrays, which
// the kernel cannot see) every contribution is added atomically into the zero-filled output.
// W = floats per lane: 4 (16-byte vectors) or 8 (32-byte vectors, two-wide FMAs)
constexpr int kFlagAtomic = static_cast<int>(0x80000000u);  // add atomically instead of storing

// Ids and weights of two batches of a sub-warp, written by its lanes and read by all of them four at a time.
template <int LPR>
struct __align__(16) SlotBuffer {
  static constexpr int kWords = 2 * LPR + 4;  // the sub-warps of a warp read from different banks
  int32_t cols[kWords];
  float wts[kWords];
};
// Volatile, so that the weights are not read, and held in registers, long before they are used.
__device__ __forceinline__ int4 lds4(const int32_t* from) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(from))) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds4(const float* from) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(from))) : "memory");
  return v;
}

// How ids and weights come to all lanes of a sub-warp: by shuffles, or four at a time by way of shared memory, which spares the data
// path of L1, the busiest unit, three of four of these steps.  us, shuffles / shared: 20 k rows of 30 F = 128 28.7 / 27.3, F = 256 46.1 /
// 40.5, F = 512 89.7 / 77.3; rows of 500 F = 300 420 / 387, F = 512 558 / 528; the 169 k-node power-law graph F = 256 100.6 / 98.4, F = 512
// 187 / 182.  kChunks: shuffles in the loop that kShared has, for long rows in one tile of 8 lanes (3 k rows of 30, F = 32 4.4, so 4.0, shared 4.2; 60 k
// of them 20.3, 19.1, 19.8), but not for the spans of wide rows (log-normal rows, 60 k of 60, F = 32 so 51.7, shared 47.6).
enum Hand : int { kShuffles, kChunks, kShared };

// Walks the slots of an item's ELL rows.  WM = 1, 2, 4: their width itself; 8: a multiple of 8.
// row_flag(g): flag word of ELL row g (called by the lane that will hold it)
// row_end(acc, flag word): all lanes of the sub-warp, after the last slot of an ELL row
template <int LPR, int WM, int W, int VPL, bool WHOLE, Hand HAND, class RowFlag, class RowEnd>
__device__ __forceinline__ void lean_item(const int32_t* cols,
                                          const float* wts, int r0, int nr, int nslots,
                                          int per_row, const char* bl,
                                          unsigned row_bytes, const LaneTile<LPR, W, VPL, WHOLE>& lt, int lane,
                                          unsigned mask, SlotBuffer<LPR>& sb, RowFlag&& row_flag, RowEnd&& row_end) {
  using LT = LaneTile<LPR, W, VPL, WHOLE>;
  using V = typename LT::Piece;
  constexpr int kU = W == 8 ? 4 : W == 4 ? 8 : VPL == 1 ? 16 : VPL == 2 ? 8 : 4;  // gathered rows in flight
  constexpr int U = WM == 8 && kU > 8 ? 8 : (kU < LPR ? kU : LPR);
  // address of dense row `col`: one 32x32->64 multiply-add
  auto vec_of = [&](const char* base, int col) -> const char* {
    return base + static_cast<unsigned long long>(static_cast<unsigned>(col)) * row_bytes;
  };
  static_assert(LPR % U == 0, "a batch is a whole number of chunks");
  static_assert(HAND == kShuffles || (WM == 8 && U % 4 == 0), "read four at a time");
  constexpr int RPB = WM < 8 ? LPR / WM : 0;  // ELL rows that end inside one batch (narrow rows)

  V acc = LT::zero();
  int c = 0, rf = 0;
  float a = 0.f;
  if (lane < nslots) {
    c = ld_global(cols + lane);
    a = ld_global(wts + lane);
  }
  if (WM < 8) {
    if (lane < RPB && lane < nr) rf = row_flag(r0 + lane);   // rows ending in batch 0
  } else {
    if (lane < nr) rf = row_flag(r0 + lane);                  // all rows of the item (nr <= LPR)
  }
  int left = per_row, jrow = 0;  // wide rows only

  for (int s0 = 0; s0 < nslots; s0 += LPR) {
    int cn = 0, rfn = 0;
    float an = 0.f;
    if (s0 + LPR + lane < nslots) {  // ids, weights (and row ids) of the next batch
      cn = ld_global(cols + s0 + LPR + lane);
      an = ld_global(wts + s0 + LPR + lane);
    }
    if (WM < 8 && lane < RPB && (s0 + LPR) / WM + lane < nr) rfn = row_flag(r0 + (s0 + LPR) / WM + lane);
    const int cnt = nslots - s0;  // live slots of this batch if < LPR
    if constexpr (HAND != kShuffles) {
      const int at = s0 / LPR % 2 * LPR;
      if constexpr (HAND == kShared) {
        sb.cols[at + lane] = c;
        sb.wts[at + lane] = a;
        __syncwarp(mask);  // and every lane is done with the batch before, which lies where the next one will
      }
      auto chunk = [&](int k0) {  // U live slots: nslots and per_row are multiples of 8
        V x[U];
#pragma unroll
        for (int u = 0; u < U; u += 4) {
          if constexpr (HAND == kShared) {
            const int4 id = lds4(sb.cols + at + k0 + u);
            x[u] = lt.ldg(vec_of(bl, id.x));
            x[u + 1] = lt.ldg(vec_of(bl, id.y));
            x[u + 2] = lt.ldg(vec_of(bl, id.z));
            x[u + 3] = lt.ldg(vec_of(bl, id.w));
          } else {
#pragma unroll
            for (int k = u; k < u + 4; ++k) x[k] = lt.ldg(vec_of(bl, __shfl_sync(mask, c, k0 + k, LPR)));
          }
        }
#pragma unroll
        for (int u = 0; u < U; u += 4) {
          if constexpr (HAND == kShared) {
            const float4 ak = lds4(sb.wts + at + k0 + u);
            LT::fma(acc, ak.x, x[u]);
            LT::fma(acc, ak.y, x[u + 1]);
            LT::fma(acc, ak.z, x[u + 2]);
            LT::fma(acc, ak.w, x[u + 3]);
          } else {
#pragma unroll
            for (int k = u; k < u + 4; ++k) LT::fma(acc, __shfl_sync(mask, a, k0 + k, LPR), x[k]);
          }
        }
        left -= U;
        if (left == 0) {
          row_end(acc, __shfl_sync(mask, rf, jrow, LPR));
          ++jrow;
          left = per_row;
        }
      };
      if (cnt >= LPR) {
#pragma unroll
        for (int k0 = 0; k0 < LPR; k0 += U) chunk(k0);
      } else {
#pragma unroll
        for (int k0 = 0; k0 < LPR; k0 += U)
          if (k0 < cnt) chunk(k0);
      }
    } else if (cnt >= LPR) {
#pragma unroll
      for (int k0 = 0; k0 < LPR; k0 += U) {
        V x[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          x[u] = lt.ldg(vec_of(bl, __shfl_sync(mask, c, k0 + u, LPR)));
#pragma unroll
        for (int u = 0; u < U; ++u) {
          LT::fma(acc, __shfl_sync(mask, a, k0 + u, LPR), x[u]);
          if (WM < 8 && (k0 + u + 1) % WM == 0)
            row_end(acc, __shfl_sync(mask, rf, (k0 + u) / WM, LPR));
        }
        if (WM == 8) {
          left -= U;
          if (left == 0) {
            row_end(acc, __shfl_sync(mask, rf, jrow, LPR));
            ++jrow;
            left = per_row;
          }
        }
      }
    } else {  // last, partly filled batch: slots past the end are neither added nor stored
#pragma unroll
      for (int k0 = 0; k0 < LPR; k0 += U) {
        if (k0 < cnt) {
          V x[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            x[u] = lt.ldg(vec_of(bl, __shfl_sync(mask, c, k0 + u, LPR)));  // dead slots: column 0
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float ak = __shfl_sync(mask, a, k0 + u, LPR);
            const int rfe = (WM < 8) ? __shfl_sync(mask, rf, (k0 + u) / WM, LPR) : 0;
            if (k0 + u < cnt) {
              LT::fma(acc, ak, x[u]);
              if (WM < 8 && (k0 + u + 1) % WM == 0) row_end(acc, rfe);
            }
          }
          if (WM == 8) {  // wide rows: nslots is a multiple of 8, so the chunk was whole
            left -= U;
            if (left == 0) {
              row_end(acc, __shfl_sync(mask, rf, jrow, LPR));
              ++jrow;
              left = per_row;
            }
          }
        }
      }
    }
    c = cn;
    a = an;
    if (WM < 8) rf = rfn;
  }
}

// What the lean kernel needs besides the bucket table.
struct LeanArgs {
  const float* b;
  float* c;
  float* part;          // scratch rows for the pieces of split rows (same row stride as c)
  unsigned* counters;   // [scratch rows][feature tiles], zero before and after every launch
  int feat;
  int all_atomic;
  PeerOut peers;
};

// The one store of a finished piece of an output row: into this GPU's C and, when the call has
// peers, into every peer's copy (plain stores over NVLink; nothing waits on them).
template <int LPR, int W, int VPL, bool WHOLE>
__device__ __forceinline__ void store_out(const LaneTile<LPR, W, VPL, WHOLE>& lt, char* row, const LanePiece<W, VPL>& v,
                                          const PeerOut* po) {
  lt.stcs(row, v);
  if (po != nullptr)
    for (int k = 0; k < po->n; ++k) lt.stcg(row + po->delta[k], v);
}

// Bits of `pred` over the LPR lanes of this thread's sub-warp, lane 0 of the sub-warp in bit 0.
template <int LPR>
__device__ __forceinline__ unsigned sub_ballot(unsigned mask, bool pred) {
  const unsigned all = __ballot_sync(mask, pred);
  if constexpr (LPR == 32) {
    return all;
  } else {
    return (all >> ((threadIdx.x & 31) / LPR * LPR)) & ((1u << LPR) - 1u);
  }
}

// The last ELL row `g` of a piece of a split row has been accumulated into `acc` by this
// sub-warp.  A piece is the part of a run of equal row ids that lies inside one work item
// (items hold `rpi` consecutive ELL rows; rpi = 1 for wide buckets).  Pieces are numbered in
// ELL-row order; piece k keeps its partial sum in the scratch row of its first ELL row.
template <int LPR, int W, int VPL, bool WHOLE>
__device__ __noinline__ void finish_split_row(const LaneTile<LPR, W, VPL, WHOLE> lt, LanePiece<W, VPL> acc,
                                              const int32_t* rows, int nrows, int g,
                                              int rpi, int rid, int part_base, char* part, char* c,
                                              unsigned* counters, unsigned row_bytes, int lane,
                                              unsigned mask, const PeerOut* po) {
  using LT = LaneTile<LPR, W, VPL, WHOLE>;
  constexpr unsigned kFull = LPR == 32 ? 0xffffffffu : ((1u << LPR) - 1u);
  int first = g, last = g;
  while (true) {  // LPR ELL rows per step, backwards then forwards
    const int idx = first - 1 - lane;
    const unsigned bits = sub_ballot<LPR>(mask, idx >= 0 && ld_global(rows + max(idx, 0)) == rid);
    const int n = bits == kFull ? LPR : __ffs(~bits) - 1;
    first -= n;
    if (n < LPR) break;
  }
  while (true) {
    const int idx = last + 1 + lane;
    const unsigned bits = sub_ballot<LPR>(mask, idx < nrows && ld_global(rows + min(idx, nrows - 1)) == rid);
    const int n = bits == kFull ? LPR : __ffs(~bits) - 1;
    last += n;
    if (n < LPR) break;
  }
  const int item0 = first / rpi;
  const int npieces = last / rpi - item0 + 1;
  char* dst = c + static_cast<unsigned long long>(static_cast<unsigned>(rid)) * row_bytes;
  if (npieces == 1) {  // the whole run lies inside this item
    store_out(lt, dst, acc, po);
    return;
  }
  const int mine = max(first, g / rpi * rpi);
  auto part_of = [&](int ell_row) -> char* {
    return part + static_cast<unsigned long long>(static_cast<unsigned>(part_base + ell_row)) * row_bytes;
  };
  lt.stcg(part_of(mine), acc);
  __threadfence();
  __syncwarp(mask);
  unsigned* counter = counters + static_cast<size_t>(part_base + first) * gridDim.y + blockIdx.y;
  unsigned seen = 0;
  if (lane == 0) seen = atomicAdd(counter, 1u);
  seen = __shfl_sync(mask, seen, 0, LPR);
  if (seen + 1 != static_cast<unsigned>(npieces)) return;
  // last piece to arrive: every other piece's partial sum is visible
  if (lane == 0) *counter = 0u;
  __threadfence();
  typename LT::Piece sum = lt.ldcg(part_of(first));
  for (int k = 1; k < npieces; ++k) LT::add(sum, lt.ldcg(part_of((item0 + k) * rpi)));
  store_out(lt, dst, sum, po);
}

// The same for an ELL row wide enough to be shared by all the sub-warps of this warp (one ELL row
// per piece): the whole warp takes part.  `before` and `behind` are the row ids of the 32 ELL rows
// on either side, requested before the row was gathered, so that the run of equal ids is known
// without another trip to memory; the partial sums of the run are read by all sub-warps at once.
// On the 169 k-node power-law graph at F = 32 the two serial walks (over the ids, over the 26
// pieces of the largest row) were the last 8 us of a 21 us launch.
template <int LPR, int W, int VPL, bool WHOLE>
__device__ __noinline__ void finish_split_row_warp(const LaneTile<LPR, W, VPL, WHOLE> lt, LanePiece<W, VPL> acc,
                                                   const int32_t* rows, int nrows, int g,
                                                   int rid, int before, int behind, int part_base,
                                                   char* part, char* c, unsigned* counters,
                                                   unsigned row_bytes, const PeerOut* po) {
  using LT = LaneTile<LPR, W, VPL, WHOLE>;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NW = 32 / LPR;
  const int wlane = threadIdx.x & 31, lane = wlane % LPR, sub = wlane / LPR;
  int first = g, last = g;
  while (true) {
    const unsigned bits = __ballot_sync(kAll, first - 1 - wlane >= 0 && before == rid);
    const int n = bits == kAll ? 32 : __ffs(~bits) - 1;
    first -= n;
    if (n < 32) break;
    before = ld_global(rows + max(first - 1 - wlane, 0));
  }
  while (true) {
    const unsigned bits = __ballot_sync(kAll, last + 1 + wlane < nrows && behind == rid);
    const int n = bits == kAll ? 32 : __ffs(~bits) - 1;
    last += n;
    if (n < 32) break;
    behind = ld_global(rows + min(last + 1 + wlane, nrows - 1));
  }
  char* dst = c + static_cast<unsigned long long>(static_cast<unsigned>(rid)) * row_bytes;
  if (first == last) {  // not split after all
    if (sub == 0) store_out(lt, dst, acc, po);
    return;
  }
  auto part_of = [&](int ell_row) -> char* {
    return part + static_cast<unsigned long long>(static_cast<unsigned>(part_base + ell_row)) * row_bytes;
  };
  if (sub == 0) lt.stcg(part_of(g), acc);
  __threadfence();
  __syncwarp();
  unsigned* counter = counters + static_cast<size_t>(part_base + first) * gridDim.y + blockIdx.y;
  unsigned seen = 0;
  if (wlane == 0) seen = atomicAdd(counter, 1u);
  seen = __shfl_sync(kAll, seen, 0);
  if (seen != static_cast<unsigned>(last - first)) return;
  // last piece to arrive: every other piece's partial sum is visible
  if (wlane == 0) *counter = 0u;
  __threadfence();
  typename LT::Piece sum = LT::zero();
  constexpr int G = VPL * W >= 8 ? 4 : 8;
  for (int k0 = first + sub; k0 <= last; k0 += NW * G) {
    typename LT::Piece x[G];
#pragma unroll
    for (int u = 0; u < G; ++u) x[u] = lt.ldcg(part_of(min(k0 + u * NW, last)));
#pragma unroll
    for (int u = 0; u < G; ++u)
      if (k0 + u * NW <= last) LT::add(sum, x[u]);
  }
#pragma unroll
  for (int o = LPR; o < 32; o *= 2)
#pragma unroll
    for (int v = 0; v < VPL; ++v) LaneVec<W>::add_xor(sum.v[v], o);
  if (sub == 0) store_out(lt, dst, sum, po);
}

// A narrow item of the widest bucket that holds ELL rows of a split row (rare: only bucket lists
// whose last width is small put split rows into a narrow bucket).  Plain loop, one ELL row at a
// time; consecutive ELL rows of the same output row inside the item are added up first.
template <int LPR, int W, int VPL, bool WHOLE>
__device__ __noinline__ void split_item(const LaneTile<LPR, W, VPL, WHOLE> lt, const int32_t* cols,
                                        const float* wts, const int32_t* rows,
                                        int nrows, int r0, int nr, int width, int rpi, int part_base,
                                        const char* b, char* part, char* c,
                                        unsigned* counters, unsigned row_bytes, int lane, unsigned mask,
                                        const PeerOut* po) {
  using LT = LaneTile<LPR, W, VPL, WHOLE>;
  typename LT::Piece acc = LT::zero();
  for (int j = 0; j < nr; ++j) {
    const int g = r0 + j;
    for (int s = 0; s < width; ++s) {
      const int col = ld_global(cols + j * width + s);
      const float a = ld_global(wts + j * width + s);
      LT::fma(acc, a, lt.ldg(b + static_cast<unsigned long long>(static_cast<unsigned>(col)) * row_bytes));
    }
    const int rid = ld_global(rows + g);
    const bool next_same = g + 1 < nrows && ld_global(rows + g + 1) == rid;
    if (next_same && j + 1 < nr) continue;  // the next ELL row of this item continues the row
    if (next_same || (g > 0 && ld_global(rows + g - 1) == rid))
      finish_split_row(lt, acc, rows, nrows, g, rpi, rid, part_base, part, c, counters, row_bytes, lane, mask, po);
    else
      store_out(lt, c + static_cast<unsigned long long>(static_cast<unsigned>(rid)) * row_bytes, acc, po);
    acc = LT::zero();
  }
}

// blockIdx.y = feature tile of LPR * W * VPL floats; the last one may be partly filled
// HAND: of rows of 8 slots and more
template <int LPR, int W, int VPL, bool WHOLE, bool PEERS, Hand HAND>
__global__ void __launch_bounds__(kThreads, 8)
hyb_spmm_lean_kernel(const __grid_constant__ HybTable tb, const __grid_constant__ LeanArgs la) {
  using LT = LaneTile<LPR, W, VPL, WHOLE>;
  using V = typename LT::Piece;
  const PeerOut* po = PEERS ? &la.peers : nullptr;
  constexpr int SUBS = kThreads / LPR;
  constexpr int NW = 32 / LPR;
  __shared__ union __align__(32) {  // of a sub-warp: its batches, then, in wide rows, the partial sum of its span
    SlotBuffer<LPR> slots;
    float part[LT::kFloats];
  } s_sub[SUBS];
  const int lane = threadIdx.x % LPR;
  const int sub = threadIdx.x / LPR;
  const unsigned mask = group_mask<LPR>();
  const int q = find_bucket(tb, blockIdx.x);
  const int width = tb.width[q], nrows = tb.nrows[q];
  const int rpi = tb.rows_per_item[q], spr = tb.chunks_per_row[q];
  const int part_base = tb.part_base[q];
  const unsigned stride = static_cast<unsigned>(la.feat) * 4u;  // bytes per dense row
  const LT lt(la.feat, blockIdx.y, lane);
  const char* bl = reinterpret_cast<const char*>(la.b);
  char* cl = reinterpret_cast<char*>(la.c);
  char* pl = reinterpret_cast<char*>(la.part);
  const int32_t* rows = tb.rows[q];
  if (rows == nullptr) cl += static_cast<size_t>(tb.row_base[q]) * stride;
  const bool all_atomic = la.all_atomic != 0;
  auto y_of = [&](int rid) -> char* {
    return cl + static_cast<unsigned long long>(static_cast<unsigned>(rid)) * stride;
  };
  chain_wait();

  if (spr == 1) {
    // ---- narrow bucket: a sub-warp owns rpi whole ELL rows
    const long long item = static_cast<long long>(blockIdx.x - tb.block_start[q]) * SUBS + sub;
    const long long r0l = item * rpi;
    if (r0l >= nrows) return;
    const int r0 = static_cast<int>(r0l);
    const int nr = min(nrows, r0 + rpi) - r0;
    const size_t first = static_cast<size_t>(r0) * width;
    if (!all_atomic && part_base >= 0) {
      // the widest bucket: an item that holds an ELL row of a split row takes the careful path
      bool any = false;
      for (int j = lane; j < nr; j += LPR) any = any || is_split_row(rows, r0 + j, nrows, ld_global(rows + r0 + j));
      if (sub_ballot<LPR>(mask, any) != 0u) {
        split_item(lt, tb.cols[q] + first, tb.w[q] + first, rows, nrows, r0, nr, width, rpi, part_base,
                   bl, pl, cl, la.counters, stride, lane, mask, po);
        return;
      }
    }
    auto row_flag = [&](int g) -> int {
      // a bucket without row ids has its base folded into cl
      return row_id(rows, g, 0) | (all_atomic ? kFlagAtomic : 0);
    };
    auto row_end = [&](V& acc, int rf) {
      if (rf < 0) lt.atomic_add(y_of(rf & 0x7fffffff), acc);
      else store_out(lt, y_of(rf), acc, po);  // written once: do not displace B rows in L2
      acc = LT::zero();
    };
    const int32_t* cols = tb.cols[q] + first;
    const float* wts = tb.w[q] + first;
    const int nslots = nr * width;
    if (width == 1) lean_item<LPR, 1, W, VPL, WHOLE, kShuffles>(cols, wts, r0, nr, nslots, width, bl, stride, lt, lane, mask, s_sub[sub].slots, row_flag, row_end);
    else if (width == 2) lean_item<LPR, 2, W, VPL, WHOLE, kShuffles>(cols, wts, r0, nr, nslots, width, bl, stride, lt, lane, mask, s_sub[sub].slots, row_flag, row_end);
    else if (width == 4) lean_item<LPR, 4, W, VPL, WHOLE, kShuffles>(cols, wts, r0, nr, nslots, width, bl, stride, lt, lane, mask, s_sub[sub].slots, row_flag, row_end);
    else lean_item<LPR, 8, W, VPL, WHOLE, HAND>(cols, wts, r0, nr, nslots, width, bl, stride, lt, lane, mask, s_sub[sub].slots, row_flag, row_end);
    return;
  }

  // ---- wide bucket: spr sub-warps of this block share one ELL row, each takes one span of it
  const int rpb = SUBS / spr;  // ELL rows per block
  const int part = sub % spr;
  const long long rl = static_cast<long long>(blockIdx.x - tb.block_start[q]) * rpb + sub / spr;
  const bool live = rl < nrows;
  const int r = live ? static_cast<int>(rl) : 0;
  const int span = ((width + spr - 1) / spr + 7) & ~7;  // slots per span, a multiple of 8
  // all sub-warps of the first warp of an ELL row belong to it: that warp finishes the row
  const bool by_warp = spr >= NW && !all_atomic && part_base >= 0;
  int rid = 0, before = 0, behind = 0;
  if (live && part < NW) {
    rid = row_id(rows, r, 0);
    if (by_warp) {
      before = ld_global(rows + max(r - 1 - static_cast<int>(threadIdx.x & 31), 0));
      behind = ld_global(rows + min(r + 1 + static_cast<int>(threadIdx.x & 31), nrows - 1));
    }
  }
  V total = LT::zero();
  if (live && part * span < width) {
    const int s0 = part * span;
    const int nslots = min(span, width - s0);
    const size_t first = static_cast<size_t>(r) * width + s0;
    auto no_flag = [](int) -> int { return 0; };
    auto keep = [&](V& acc, int) { total = acc; };
    lean_item<LPR, 8, W, VPL, WHOLE, HAND == kShuffles ? kShuffles : kShared>(tb.cols[q] + first, tb.w[q] + first, r, 1, nslots, nslots, bl, stride, lt, lane, mask,
                                             s_sub[sub].slots, no_flag, keep);
  }
  __syncwarp(mask);  // every lane is done with the batches
  if (part != 0) LT::sts(s_sub[sub].part, lane, total);
  __syncthreads();
  if (!live || part >= NW || (part != 0 && !by_warp)) return;
  if (part == 0)
    for (int k = 1; k < spr; ++k) LT::add(total, LT::lds(s_sub[sub + k].part, lane));
  if (by_warp) {
    finish_split_row_warp(lt, total, rows, nrows, r, rid, before, behind, part_base, pl, cl, la.counters, stride, po);
  } else if (all_atomic) {
    lt.atomic_add(y_of(rid), total);
  } else if (part_base >= 0 && is_split_row(rows, r, nrows, rid)) {
    finish_split_row(lt, total, rows, nrows, r, 1, rid, part_base, pl, cl, la.counters, stride, lane, mask, po);
  } else {
    store_out(lt, y_of(rid), total, po);
  }
}

// The main kernel for 16-byte aligned operands: B rows are staged through per-lane rings in
// shared memory by asynchronous copies (see stream_slots_async), ids / weights / row ids of the
// item are read into shared memory once, with coalesced loads, before the pipeline starts.
// One lane covers one 16-byte vector of a 4*LPR-float feature tile; blockIdx.y walks the tiles.
constexpr int kRing = 12;  // slots in flight per lane

template <int LPR>
struct AsyncSmem {
  static constexpr int SUBS = kThreads / LPR;
  static constexpr int ITEM = item_slots(LPR);
  static constexpr size_t ring_bytes = sizeof(float4) * SUBS * kRing * LPR;
  static constexpr size_t bytes = ring_bytes + sizeof(int32_t) * SUBS * (ITEM + ITEM + ITEM + 2);
};

template <int LPR>
__global__ void __launch_bounds__(kThreads, 3)
hyb_spmm_async_kernel(const __grid_constant__ HybTable tb, const float* b,
                      float* __restrict__ c, int feat, int all_atomic) {
  using S = AsyncSmem<LPR>;
  constexpr int SUBS = S::SUBS, ITEM = S::ITEM;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x % LPR;
  const int sub = threadIdx.x / LPR;
  float4* ring = reinterpret_cast<float4*>(smem_raw) + sub * (kRing * LPR) + lane;
  int32_t* s_ids = reinterpret_cast<int32_t*>(smem_raw + S::ring_bytes) + sub * ITEM;
  float* s_wts = reinterpret_cast<float*>(smem_raw + S::ring_bytes) + SUBS * ITEM + sub * ITEM;
  int32_t* s_rows = reinterpret_cast<int32_t*>(smem_raw + S::ring_bytes) + 2 * SUBS * ITEM +
                    sub * (ITEM + 2);
  const unsigned mask = group_mask<LPR>();
  const int q = find_bucket(tb, blockIdx.x);
  const int width = tb.width[q], nrows = tb.nrows[q];
  const int rpi = tb.rows_per_item[q], cpr = tb.chunks_per_row[q];
  const long long item = static_cast<long long>(blockIdx.x - tb.block_start[q]) * SUBS + sub;
  long long r0l;
  int nslots, per_row, nr;
  size_t first;
  if (cpr == 1) {
    r0l = item * rpi;
    if (r0l >= nrows) return;
    nr = static_cast<int>(min(static_cast<long long>(nrows), r0l + rpi) - r0l);
    nslots = nr * width;
    per_row = width;
    first = static_cast<size_t>(r0l) * width;
  } else {
    r0l = item / cpr;
    if (r0l >= nrows) return;
    const int s0 = static_cast<int>(item % cpr) * ITEM;
    nr = 1;
    nslots = min(ITEM, width - s0);
    per_row = nslots;
    first = static_cast<size_t>(r0l) * width + s0;
  }
  const int r0 = static_cast<int>(r0l);
  {
    const int32_t* cols = tb.cols[q] + first;
    const float* wts = tb.w[q] + first;
    const int32_t* rows = tb.rows[q];
    for (int s = lane; s < nslots; s += LPR) {
      s_ids[s] = ld_global(cols + s);
      s_wts[s] = ld_global(wts + s);
    }
    for (int j = lane; j < nr + 2; j += LPR) {
      const int idx = r0 - 1 + j;
      s_rows[j] = (idx >= 0 && idx < nrows) ? row_id(rows, idx, tb.row_base[q]) : -1;
    }
  }
  __syncwarp(mask);
  const int row_vecs = feat / 4;
  const int off = blockIdx.y * LPR + lane;
  const bool valid = off < row_vecs;
  float4* cv = reinterpret_cast<float4*>(c) + off;
  const bool always_atomic = all_atomic || cpr > 1;

  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  int j = 1, left = per_row;
  auto on_done = [&](float4&, int n) {
    left -= n;
    if (left != 0) return;
    const int row = s_rows[j];
    const bool atomic = always_atomic || s_rows[j - 1] == row || s_rows[j + 1] == row;
    float4* dst = cv + static_cast<size_t>(row) * row_vecs;
    if (valid) {
      if (atomic) atomicAdd(dst, acc);
      else __stcs(dst, acc);  // written once: do not displace B rows in L2
    }
    acc = make_float4(0.f, 0.f, 0.f, 0.f);
    ++j;
    left = per_row;
  };
  const float4* bl = reinterpret_cast<const float4*>(b) + off;
  // Row ends fall on group boundaries when the row length is a multiple of 4: then the row-end
  // test runs once per group instead of once per slot.
  if (per_row % 4 != 0)
    stream_slots_async<LPR, kRing, true>(s_ids, s_wts, nslots, bl, static_cast<size_t>(row_vecs),
                                         valid, ring, acc, on_done);
  else
    stream_slots_async<LPR, kRing, false>(s_ids, s_wts, nslots, bl, static_cast<size_t>(row_vecs),
                                          valid, ring, acc, on_done);
}

// Zeroes the output rows that are accumulated into atomically, so that repeated calls on the same C stay
// correct without a full memset and rows that no bucket names stay as they are: with `all` every row of the
// buckets, else what the fallback kernels add to (chunked wide rows and split rows).  One thread inspects
// one ELL row (coalesced reads of the row ids); each row to be cleared is then cleared by the whole warp.
__global__ void __launch_bounds__(kThreads)
hyb_rearm_kernel(const __grid_constant__ HybTable tb, float* __restrict__ c, int feat, bool all) {
  const int q = find_bucket(tb, blockIdx.x);
  const int nrows = tb.nrows[q];
  const int32_t* rows = tb.rows[q];
  const long long r = static_cast<long long>(blockIdx.x - tb.block_start[q]) * kThreads + threadIdx.x;
  int row = -1;
  bool clear = false;
  if (r < nrows) {
    row = row_id(rows, static_cast<int>(r), tb.row_base[q]);
    clear = all || tb.chunks_per_row[q] > 1 || is_split_row(rows, static_cast<int>(r), nrows, row);
    // of a run of equal ids only the first ELL row clears
    if (clear && r > 0 && rows != nullptr && ld_global(rows + r - 1) == row) clear = false;
  }
  unsigned todo = __ballot_sync(0xffffffffu, clear);
  const int lane = threadIdx.x & 31;
  while (todo != 0) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int rr = __shfl_sync(0xffffffffu, row, src);
    float* dst = c + static_cast<size_t>(rr) * feat;
    for (int f = lane; f < feat; f += 32) dst[f] = 0.f;
  }
}

// Scratch (bytes) the lean kernel may use for the pieces of split rows before it falls back to
// atomic accumulation; SPARSETIR_HYB_SCRATCH_MB overrides the default of 1 GiB.
size_t hyb_scratch_limit() {
  static const size_t v = [] {
    const char* e = std::getenv("SPARSETIR_HYB_SCRATCH_MB");
    const long mb = e ? std::atol(e) : -1;
    return static_cast<size_t>(mb >= 0 ? mb : 1024) << 20;
  }();
  return v;
}

void plan_items(HybTable& tb, int item) {
  for (int q = 0; q < tb.nb; ++q) {
    tb.rows_per_item[q] = std::max(1, item / tb.width[q]);
    tb.chunks_per_row[q] = tb.width[q] > item ? ceil_div(tb.width[q], item) : 1;
  }
}

// Lean kernel: a bucket wider than an item gives each ELL row a power-of-two number of sub-warps of
// one block (all of them from SUBS * item slots on; a sub-warp then walks a longer span).  Returns the number of blocks or -1.
long long plan_lean(HybTable& tb, int item, int subs) {
  long long blocks = 0;
  for (int q = 0; q < tb.nb; ++q) {
    tb.rows_per_item[q] = std::max(1, item / tb.width[q]);
    // rows of 8 slots or more: the row ids of an item travel in one register per lane
    if (tb.width[q] >= 8) tb.rows_per_item[q] = std::min(tb.rows_per_item[q], kThreads / subs);
    int spr = 1;
    while (spr < subs && spr * item < tb.width[q]) spr *= 2;
    tb.chunks_per_row[q] = spr;
    if (spr > 1) tb.rows_per_item[q] = 1;
    tb.block_start[q] = static_cast<int32_t>(blocks);
    const long long per_block = spr > 1 ? subs / spr : static_cast<long long>(subs) * tb.rows_per_item[q];
    blocks += (tb.nrows[q] + per_block - 1) / per_block;
    if (blocks > INT32_MAX) return -1;
  }
  tb.block_start[tb.nb] = static_cast<int32_t>(blocks);
  return blocks;
}

// Lanes per dense row, the first template argument of the kernel used: one lane per 16-byte
// vector, at most a warp.  Rows wider than the lanes cover are walked feature tile by feature
// tile (blockIdx.y, the slowest grid dimension).  A pass gathers from an n x tile slice of B; the
// tile is narrowed until that slice fits the part of L2 that stays resident for data every SM
// reads (measured: about half of the 126 MB), because re-reading the index arrays once per tile
// costs little next to re-fetching B rows from HBM.
int lanes_per_row_impl(int feat, bool vec4, int n, int lane_w) {
  const int units = vec4 ? ceil_div(feat, lane_w) : feat;
  const int min_lanes = lane_w == 8 ? 4 : 8;
  int lanes = units <= min_lanes ? min_lanes : (units <= 8 ? 8 : (units <= 16 ? 16 : 32));
  if (vec4) {
    // SPARSETIR_L2_BUDGET_MB overrides the default for tuning on other parts
    static const size_t l2_budget = [] {
      const char* e = std::getenv("SPARSETIR_L2_BUDGET_MB");
      const long mb = e ? std::atol(e) : 0;
      return static_cast<size_t>(mb > 0 ? mb : 48) << 20;
    }();
    while (lanes > min_lanes && static_cast<size_t>(n) * lanes * lane_w * 4 > l2_budget) lanes /= 2;
    // Up to `narrow_passes` passes over the index arrays the narrowest tile wins even when a
    // wider slice would fit L2: twice the independent sub-warps per block keep more gathers in
    // flight (measured on B200: F = 64 38 vs 41 us, F = 128 60 vs 66 us, F = 256 equal, F = 512
    // 211 vs 197 us, where the 16 passes re-read 120 MB of ids).
    static const int narrow_passes = [] {
      const char* e = std::getenv("SPARSETIR_HYB_NARROW_PASSES");
      const int v = e ? std::atoi(e) : -1;
      return v >= 0 ? v : 4;
    }();
    if (lanes > min_lanes && ceil_div(feat, min_lanes * lane_w) <= narrow_passes) lanes = min_lanes;
    // narrower too where a quarter of the lanes would lie past the end of the row
    while (lanes > min_lanes && ceil_div(units, lanes) * lanes * 4 > units * 5) lanes /= 2;
  }
  return lanes;
}

// Fills block_start for SUBS items per block; returns the number of blocks or -1.
long long plan_blocks(HybTable& tb, int subs) {
  long long blocks = 0;
  for (int q = 0; q < tb.nb; ++q) {
    tb.block_start[q] = static_cast<int32_t>(blocks);
    const long long items = tb.chunks_per_row[q] > 1
                                ? static_cast<long long>(tb.nrows[q]) * tb.chunks_per_row[q]
                                : ceil_div(tb.nrows[q], tb.rows_per_item[q]);
    blocks += (items + subs - 1) / subs;
    if (blocks > INT32_MAX) return -1;
  }
  tb.block_start[tb.nb] = static_cast<int32_t>(blocks);
  return blocks;
}

template <int LPR, int W, int VPL, bool WHOLE>
int launch_lean_as(HybTable& tb, const LeanArgs& la, cudaStream_t stream) {
  const int tiles = ceil_div(la.feat, W * LPR * VPL);
  long long slots = 0, rows = 0, wide = 0;  // wide: slots of rows of 8 and more
  for (int q = 0; q < tb.nb; ++q) {
    const long long of = static_cast<long long>(tb.nrows[q]) * tb.width[q];
    rows += tb.nrows[q];
    slots += of;
    if (tb.width[q] >= 8) wide += of;
  }
  const int item = lean_item_slots(LPR, W, tiles, slots);
  long long blocks = plan_lean(tb, item, kThreads / LPR);
  if (blocks < 0) return fail("sparsetir_hyb_spmm: too many thread blocks");
  // A second wave of a few blocks costs as much as a full one: items up to half longer where that makes one of both (us, 1.06 waves / one: 10 k rows of
  // 12, F = 512 25.5 / 17.7, 20 k of 8, F = 128 10.3 / 7.7; 1.34 waves, 19 k of 8, F = 512 32.4 / 29.5).  Up to 1.1 waves where rows of 1 and 2 slots are many,
  // which end the more often the longer the item is: power-law rows, 1.05 waves, 59 k, F = 64 14.0 / 11.7, but 1.2, 62 k, F = 64 15.2 / 16.2, 31 k, F = 512 38.9 / 44.0.
  // Twice the item takes half the blocks away that wider rows would have (rows of 1 and 20 slots, 18 k, F = 100 12.2 / 14.3).  Single floats per lane lose by it (14 k
  // power-law rows, F = 299 19.4 / 21.5).  Over 313 matrices of 1 to 1.35 waves, among them rows of 1 and 10 and power-law rows in pieces of 32, 179 take it:
  // the mean of these gains 11 %, seven lose 2 to 6.
  constexpr long long kResident = 8ll * kNumSMs;
  if (W > 1 && blocks * tiles > kResident && blocks * tiles * 100 <= kResident * (slots >= 7 * rows ? 135 : 110)) {
    long long fit = blocks;
    for (int more = item + 8; fit * tiles > kResident && more <= item + item / 2; more += 8) fit = plan_lean(tb, more, kThreads / LPR);
    blocks = fit * tiles > kResident ? plan_lean(tb, item, kThreads / LPR) : fit;
  }
  dim3 grid(static_cast<unsigned>(blocks), tiles);
  // 32-byte lanes and rows of 34, 38, 42... features, one pair to a lane, lose by it (20 k-node power-law graph, F = 34 8.9 / 10.7 us).
  constexpr bool kMay = W <= 4 && !(W == 2 && VPL == 1);
  // Shared memory is written and waited for once per batch, whatever its rows: where most slots are in rows of 1, 2 and 4, which keep the shuffles, the
  // kernel with both loops only has fewer registers for theirs (20 k rows of 3, F = 299 13.3 / 14.5, F = 256 10.8 / 11.3).  Tiles of 8 lanes: not on
  // short rows either, where they wait for chains of loads and not for L1 (169 k-node power-law graph, F = 100 59.8 / 61.1, F = 128 53.9 / 54.5; F = 32 among
  // other work 19.3 / 19.6; tiles that rows do not fill, 40 k rows of 8, F = 100 16.5 / 17.6; one tile, 40 k rows of 9, F = 32 8.3 / 8.6).  One tile that adds its
  // results atomically, F = 32, two partitions, shuffles / chunks: 105 k rows of 37 61.6 / 57.5, 40 k of 100 57.6 / 55.5, of 20 19.6 / 19.4.
  const bool long_rows = slots >= (tiles == 1 ? 16 * rows : WHOLE ? 8 * rows : 8 * rows + 1);
  const bool shared = kMay && (LPR > 8 ? 4 * wide >= slots : long_rows);
  auto go = [&](auto hand) -> int {
    constexpr Hand S = decltype(hand)::value;
    if (la.peers.n > 0) {
      if constexpr (W == 4 && WHOLE)
        launch_chained(hyb_spmm_lean_kernel<LPR, W, VPL, WHOLE, true, S>, grid, kThreads, 0, stream, tb, la);
      else
        return fail("sparsetir_hyb_spmm_peers: whole tiles of 16-byte lanes only");  // the dispatcher picks them
    } else {
      launch_chained(hyb_spmm_lean_kernel<LPR, W, VPL, WHOLE, false, S>, grid, kThreads, 0, stream, tb, la);
    }
    return 0;
  };
  using Shuffles = std::integral_constant<Hand, kShuffles>;
  int rc;
  if constexpr (!kMay) {
    rc = go(Shuffles{});
  } else {
    using InChunks = std::integral_constant<Hand, LPR == 8 ? kChunks : kShared>;
    rc = !shared ? go(Shuffles{}) : LPR == 8 && tiles == 1 ? go(InChunks{}) : go(std::integral_constant<Hand, kShared>{});
  }
  if (rc != 0) return -1;
  SPTIR_LAUNCH_OK("hyb_spmm_lean_kernel");
  return 0;
}

// Whole tiles get a kernel of their own: with predicated vectors F = 512 takes 195 us on the
// 169 k-node graph instead of 186.
template <int LPR, int W, int VPL>
int launch_lean(HybTable& tb, const LeanArgs& la, cudaStream_t stream) {
  if constexpr (W >= 4)
    if (la.feat % (LPR * W * VPL) == 0) return launch_lean_as<LPR, W, VPL, true>(tb, la, stream);
  return launch_lean_as<LPR, W, VPL, false>(tb, la, stream);
}

// lane_w = 1 or 2 (rows that are not whole 16-byte vectors): a warp per row, up to 128 floats of it
// per pass over the ids
inline int lean_tile_floats(int feat, int lanes, int lane_w) {
  if (lane_w >= 4) return lanes * lane_w;
  return feat <= 32 * lane_w ? 32 * lane_w : (feat <= 64 ? 64 : 128);
}

int dispatch_lean(HybTable& tb, const LeanArgs& la, int lanes, int lane_w, cudaStream_t st) {
  if (lane_w == 8) {
    if (lanes == 4) return launch_lean<4, 8, 1>(tb, la, st);
    if (lanes == 8) return launch_lean<8, 8, 1>(tb, la, st);
    if (lanes == 16) return launch_lean<16, 8, 1>(tb, la, st);
    return launch_lean<32, 8, 1>(tb, la, st);
  }
  if (lane_w == 4) {
    if (lanes == 8) return launch_lean<8, 4, 1>(tb, la, st);
    if (lanes == 16) return launch_lean<16, 4, 1>(tb, la, st);
    return launch_lean<32, 4, 1>(tb, la, st);
  }
  const int tile = lean_tile_floats(la.feat, 32, lane_w);
  if (lane_w == 2) return tile == 64 ? launch_lean<32, 2, 1>(tb, la, st) : launch_lean<32, 2, 2>(tb, la, st);
  if (tile == 32) return launch_lean<32, 1, 1>(tb, la, st);
  if (tile == 64) return launch_lean<32, 1, 2>(tb, la, st);
  return launch_lean<32, 1, 4>(tb, la, st);
}

template <int LPR>
int launch_async(HybTable& tb, const float* b, float* c, int feat, int all_atomic,
                 cudaStream_t stream) {
  using S = AsyncSmem<LPR>;
  const long long blocks = plan_blocks(tb, S::SUBS);
  if (blocks < 0) return fail("sparsetir_hyb_spmm: too many thread blocks");
  static thread_local int configured_device = -1;
  int dev = 0;
  SPTIR_CUDA_OK(cudaGetDevice(&dev));
  if (configured_device != dev) {
    SPTIR_CUDA_OK(cudaFuncSetAttribute(hyb_spmm_async_kernel<LPR>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(S::bytes)));
    configured_device = dev;
  }
  dim3 grid(static_cast<unsigned>(blocks), ceil_div(feat / 4, LPR));
  hyb_spmm_async_kernel<LPR><<<grid, kThreads, S::bytes, stream>>>(tb, b, c, feat, all_atomic);
  SPTIR_LAUNCH_OK("hyb_spmm_async_kernel");
  return 0;
}

template <int LPR, int VPL, int VEC>
int launch(HybTable& tb, const float* b, float* c, int feat, int all_atomic, cudaStream_t stream) {
  const long long blocks = plan_blocks(tb, kThreads / LPR);
  if (blocks < 0) return fail("sparsetir_hyb_spmm: too many thread blocks");
  const int tile_feat = LPR * VPL * VEC;
  dim3 grid(static_cast<unsigned>(blocks), ceil_div(feat, tile_feat));
  hyb_spmm_kernel<LPR, VPL, VEC><<<grid, kThreads, 0, stream>>>(tb, b, c, feat, all_atomic);
  SPTIR_LAUNCH_OK("hyb_spmm_kernel");
  return 0;
}

}  // namespace
}  // namespace sptir

namespace sptir {
size_t hyb_scratch_limit_bytes() { return hyb_scratch_limit(); }
int lanes_per_row(int feat, bool vec4, int n, int lane_w) { return lanes_per_row_impl(feat, vec4, n, lane_w); }

// The launcher behind sparsetir_hyb_spmm_raw.  row_bases (may be null): for buckets whose `rows`
// array is null, ELL row r of bucket q is written to output row row_bases[q] + r.
int hyb_spmm_run(const float* b, float* c, const SparsetirEllBucket* buckets, const int32_t* row_bases,
                 int num_buckets, int m, int n, int feat, int flags, int device_id, void* stream,
                 const PeerOut* peers) {
  if (num_buckets < 0 || num_buckets > kMaxB)
    return fail("sparsetir_hyb_spmm: %d buckets exceed the maximum of %d", num_buckets, kMaxB);
  if (m < 0 || feat < 0) return fail("sparsetir_hyb_spmm: negative size");
  if (num_buckets > 0 && !buckets) return fail("sparsetir_hyb_spmm: null bucket table");
  if (feat == 0 || m == 0) return 0;
  if (!b || !c) return fail("sparsetir_hyb_spmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int all_atomic = (flags & SPARSETIR_HYB_ALL_ATOMIC) ? 1 : 0;

  // Table in launch order: widest bucket first, empty buckets dropped.
  std::vector<int> order;
  for (int q = 0; q < num_buckets; ++q) {
    const SparsetirEllBucket& bk = buckets[q];
    if (bk.nrows < 0 || bk.width < 0) return fail("sparsetir_hyb_spmm: negative bucket size");
    if (bk.nrows == 0) continue;
    if (bk.width == 0) return fail("sparsetir_hyb_spmm: bucket %d has rows but width 0", q);
    // rows may be null: ELL row r then belongs to output row r
    if (!bk.w || !bk.cols) return fail("sparsetir_hyb_spmm: null bucket array");
    order.push_back(q);
  }
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return buckets[x].width > buckets[y].width; });
  HybTable tb{};
  tb.nb = static_cast<int32_t>(order.size());
  for (int k = 0; k < tb.nb; ++k) {
    const SparsetirEllBucket& bk = buckets[order[k]];
    tb.w[k] = bk.w; tb.rows[k] = bk.rows; tb.cols[k] = bk.cols;
    tb.nrows[k] = bk.nrows; tb.width[k] = bk.width;
    tb.row_base[k] = row_bases ? row_bases[order[k]] : 0;
  }
  if (validate_enabled()) {
    for (int k = 0; k < tb.nb; ++k) {
      const long long slots = static_cast<long long>(tb.nrows[k]) * tb.width[k];
      if (validate_range("sparsetir_hyb_spmm", "a bucket's row_indices", tb.rows[k], tb.nrows[k], m, st) != 0 ||
          validate_range("sparsetir_hyb_spmm", "a bucket's col_indices", tb.cols[k], slots, n, st) != 0)
        return -1;
    }
  }
  const bool vec4 = (feat % 4 == 0) && aligned16(b) && aligned16(c);
  // the lean kernel takes ELL widths of 1, 2, 4 or a multiple of 8; its lanes own 16-byte vectors
  // (32-byte ones on request, for 32-byte aligned operands and a multiple of 32 features), or 8- and
  // 4-byte ones where the row length or the alignment allows no more
  bool lean = static_cast<long long>(feat) * 4 < (1ll << 32);
  for (int q = 0; q < tb.nb; ++q) {
    const int w = tb.width[q];
    lean = lean && (w == 1 || w == 2 || w == 4 || w % 8 == 0);
  }
  const bool to_peers = peers != nullptr && peers->n > 0;
  // the form that stores to peers exists for 16-byte lanes only (the library's default)
  int lane_w = (lean && !to_peers && feat % 32 == 0 && aligned32(b) && aligned32(c)) ? max_lane_floats() : 4;
  int lanes = lanes_per_row_impl(feat, vec4, n, lane_w);
  if (lane_w == 8 && feat % (lane_w * lanes) != 0) {  // no whole tiles of 8-float lanes
    lane_w = 4;
    lanes = lanes_per_row_impl(feat, vec4, n, lane_w);
  }
  if (!vec4) {
    lane_w = feat % 2 == 0 && (reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) % 8 == 0 ? 2 : 1;
    if (lean) lanes = 32;
  }
  const size_t c_bytes = static_cast<size_t>(m) * feat * sizeof(float);
  if (to_peers && (!lean || !vec4 || feat % (lane_w * lanes) != 0 || all_atomic || (flags & SPARSETIR_HYB_ZERO_C)))
    return fail("sparsetir_hyb_spmm_peers: needs the one-writer kernel (feat_size a multiple of its tile, "
                "16-byte aligned b and c, bucket widths 1, 2, 4 or multiples of 8, no ALL_ATOMIC or ZERO_C "
                "flag); run sparsetir_hyb_spmm and sparsetir_peer_scatter instead");
  if (tb.nb == 0) {
    if (flags & SPARSETIR_HYB_ZERO_C) SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, c_bytes, st));
    return 0;
  }

  auto clear_rows = [&](bool all) -> int {
    long long blocks = 0;
    for (int q = 0; q < tb.nb; ++q) {
      tb.block_start[q] = static_cast<int32_t>(blocks);
      blocks += ceil_div(tb.nrows[q], kThreads);
    }
    tb.block_start[tb.nb] = static_cast<int32_t>(blocks);
    if (blocks > INT32_MAX) return fail("sparsetir_hyb_spmm: too many thread blocks");
    hyb_rearm_kernel<<<static_cast<unsigned>(blocks), kThreads, 0, st>>>(tb, c, feat, all);
    SPTIR_LAUNCH_OK("hyb_rearm_kernel");
    return 0;
  };

  if (lean) {
    // ---- one writer per output row (or everything atomic when the caller asks for it)
    LeanArgs la{b, c, nullptr, nullptr, feat, all_atomic, PeerOut{}};
    if (to_peers) la.peers = *peers;
    bool clear = (flags & SPARSETIR_HYB_ZERO_C) || (all_atomic && (flags & SPARSETIR_HYB_REARM));
    CallScratch cs;
    for (int q = 0; q < tb.nb; ++q) tb.part_base[q] = -1;
    if (!all_atomic) {
      // split rows live in the widest bucket(s) that carry row ids: one scratch row per ELL row
      int maxw = 0;
      for (int q = 0; q < tb.nb; ++q)
        if (tb.rows[q] != nullptr) maxw = std::max(maxw, tb.width[q]);
      long long part_rows = 0;
      for (int q = 0; q < tb.nb; ++q)
        if (tb.rows[q] != nullptr && tb.width[q] == maxw) {
          tb.part_base[q] = static_cast<int32_t>(part_rows);
          part_rows += tb.nrows[q];
        }
      const int tiles = ceil_div(feat, lean_tile_floats(feat, lanes, lane_w));
      const size_t part_bytes = static_cast<size_t>(part_rows) * feat * sizeof(float);
      const size_t counter_bytes = static_cast<size_t>(part_rows) * tiles * sizeof(unsigned);
      if (part_rows > INT32_MAX || part_bytes > hyb_scratch_limit()) {
        // a bucket list whose widest bucket holds most of the matrix: adding atomically into
        // cleared rows of C costs less memory than a scratch copy of that size
        if (to_peers)
          return fail("sparsetir_hyb_spmm_peers: the split rows need %zu bytes of scratch, beyond the limit; "
                      "run sparsetir_hyb_spmm and sparsetir_peer_scatter instead", part_bytes);
        for (int q = 0; q < tb.nb; ++q) tb.part_base[q] = -1;
        la.all_atomic = 1;
        if (!clear && clear_rows(true) != 0) return -1;
      } else if (part_rows > 0) {
        // Whole tiles are captured with the stream's own buffers where these have been reserved; everything
        // else that is being captured gets memory of the graph (ragged feature counts and unaligned
        // operands need no reservation: the kernels that they took before this one had no scratch).
        if (vec4 && feat % (lane_w * lanes) == 0 && workspace_fits(device_id, st, part_bytes, counter_bytes)) {
          cs.scratch = static_cast<char*>(workspace(device_id, st, part_bytes));
          cs.counters = static_cast<unsigned*>(zeroed_workspace(device_id, st, counter_bytes));
        } else if (take_scratch(device_id, st, part_bytes, counter_bytes, &cs) != 0) {
          return -1;
        }
        la.part = reinterpret_cast<float*>(cs.scratch);
        la.counters = cs.counters;
      }
    }
    if (clear) SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, c_bytes, st));
    if (dispatch_lean(tb, la, lanes, lane_w, st) != 0) return -1;
    return return_scratch(cs, st);
  }

  // ---- fallback kernels for ELL widths other than 1, 2, 4 and multiples of 8
  plan_items(tb, item_slots(lanes));
  if (flags & SPARSETIR_HYB_ZERO_C) {
    SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, c_bytes, st));
  } else if (flags & SPARSETIR_HYB_REARM) {
    if (all_atomic) {
      SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, c_bytes, st));
    } else {
      if (clear_rows(false) != 0) return -1;
    }
  }

  if (vec4) {
    if (lanes == 8) return launch_async<8>(tb, b, c, feat, all_atomic, st);
    if (lanes == 16) return launch_async<16>(tb, b, c, feat, all_atomic, st);
    return launch_async<32>(tb, b, c, feat, all_atomic, st);
  }
  if (feat <= 8) return launch<8, 1, 1>(tb, b, c, feat, all_atomic, st);
  if (feat <= 16) return launch<16, 1, 1>(tb, b, c, feat, all_atomic, st);
  if (feat <= 32) return launch<32, 1, 1>(tb, b, c, feat, all_atomic, st);
  return launch<32, 4, 1>(tb, b, c, feat, all_atomic, st);
}

int hyb_spmm_impl(const float* b, float* c, const SparsetirEllBucket* buckets, const int32_t* row_bases,
                  int num_buckets, int m, int n, int feat, int flags, int device_id, void* stream) {
  return hyb_spmm_run(b, c, buckets, row_bases, num_buckets, m, n, feat, flags, device_id, stream, nullptr);
}
}  // namespace sptir

extern "C" int sparsetir_hyb_spmm_tile(int n, int feat, int* lanes, int* lane_floats) {
  if (!lanes || !lane_floats || feat <= 0 || feat % 4 != 0)
    return sptir::fail("sparsetir_hyb_spmm_tile: feat_size must be a positive multiple of 4");
  int lane_w = feat % 32 == 0 ? sptir::max_lane_floats() : 4;
  int l = sptir::lanes_per_row(feat, true, n, lane_w);
  if (lane_w == 8 && feat % (lane_w * l) != 0) {
    lane_w = 4;
    l = sptir::lanes_per_row(feat, true, n, lane_w);
  }
  *lanes = l;
  *lane_floats = lane_w;
  return 0;
}

extern "C" int sparsetir_hyb_spmm_workspace(const SparsetirEllBucket* buckets, int num_buckets,
                                            int feat, size_t* scratch_bytes,
                                            size_t* counter_bytes) {
  if (num_buckets < 0 || (num_buckets > 0 && !buckets) || feat < 0 || !scratch_bytes || !counter_bytes)
    return sptir::fail("sparsetir_hyb_spmm_workspace: bad argument");
  int maxw = 0;
  for (int q = 0; q < num_buckets; ++q)
    if (buckets[q].nrows > 0 && buckets[q].rows != nullptr) maxw = std::max(maxw, buckets[q].width);
  size_t rows = 0;
  for (int q = 0; q < num_buckets; ++q)
    if (buckets[q].nrows > 0 && buckets[q].rows != nullptr && buckets[q].width == maxw)
      rows += static_cast<size_t>(buckets[q].nrows);
  const size_t part = rows * static_cast<size_t>(feat) * sizeof(float);
  const bool fits = part <= sptir::hyb_scratch_limit_bytes();
  *scratch_bytes = fits ? part : 0;
  // a feature tile is at least 32 floats wide
  *counter_bytes = fits ? rows * static_cast<size_t>((feat + 31) / 32) * sizeof(unsigned) : 0;
  return 0;
}

extern "C" int sparsetir_hyb_spmm_peers_raw(const float* b, float* c, const SparsetirEllBucket* buckets,
                                            int num_buckets, int m, int n, int feat, int flags,
                                            int n_peers, void* const* peer_c, int device_id, void* stream) {
  sptir::PeerOut po{};
  if (sptir::peer_table("sparsetir_hyb_spmm_peers", c, n_peers, peer_c, 32, &po) != 0) return -1;
  return sptir::hyb_spmm_run(b, c, buckets, nullptr, num_buckets, m, n, feat, flags, device_id, stream, &po);
}

extern "C" int sparsetir_hyb_spmm_raw(const float* b, float* c, const SparsetirEllBucket* buckets,
                                      int num_buckets, int m, int n, int feat, int flags,
                                      int device_id, void* stream) {
  return sptir::hyb_spmm_impl(b, c, buckets, nullptr, num_buckets, m, n, feat, flags, device_id, stream);
}

// CSR SpMM, fp32, split by stored entries:  C[i,:] = sum_{p in row i} A[p] * B[indices[p],:]
//
// A block owns a contiguous range of stored entries (SUBS sub-warps of LPR lanes, `span` entries
// each), so a hub row of thousands of entries is spread over many sub-warps and a run of short
// rows costs what its entries cost: one launch, whatever the row lengths.  It replaces a row-wise
// kernel with two more launches for the rows of more than 32 entries (169 k-node power-law graph,
// F = 32 / 512: 74 / 358 us against 26.6 / 229 us) and a row-wise kernel for the feature counts
// that are not whole tiles, where one sub-warp walked a hub row alone (100 k-node power-law
// graph, F = 100: 2302 us against 33.5 us).
//
// Rows are found without a plan: a 32-ary search of `indptr` for the first entry of a sub-warp,
// then a register window of row ends (row_walk.cuh).  Every output row has one writer and one
// order of summation, so results repeat bit by bit:
//  - a row inside one sub-warp is written by it;
//  - the pieces of a row that crosses sub-warps meet in shared memory and are added in order by
//    the sub-warp in which the row (or the block's part of it) starts;
//  - the pieces of a row that crosses blocks meet in a scratch buffer; the block that counts in
//    last adds them in order.  Nobody waits: counters are back at zero when the launch ends.
// Rows without entries are cleared by the block that owns that share of the rows.
//
// Bound: latency of the dependent chain (search, ids, rows of B) on small matrices, the L2-to-SM
// gather rate (about 17 TB/s) on large ones.
#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "row_walk.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;

struct SplitArgs {
  const float* a;
  const float* b;
  float* c;
  const int32_t* indptr;
  const int32_t* indices;
  float* part;         // two scratch rows per block with entries: the piece of a row that began before it, and
                       // of a row that goes on behind it
  unsigned* counters;  // [blocks with entries][feature tiles], zero before and after every launch
  int m, nnz, feat, span;
  float rows_per_entry;
};

template <int LPR>
__device__ __forceinline__ unsigned group_ballot(unsigned mask, bool pred) {
  const unsigned all = __ballot_sync(mask, pred);
  if constexpr (LPR == 32) {
    return all;
  } else {
    return (all >> ((threadIdx.x & 31) / LPR * LPR)) & ((1u << LPR) - 1u);
  }
}

// Resident blocks.  The widest pieces per lane spill at 64 registers: three blocks of 80 hold them (50 k-node
// power-law graph, F = 299: 80 against 77.6 us; 100 k nodes, F = 222: 76 against 70; 30 k rows of 38 entries,
// F = 151: 104 against 99; two single floats per lane: F = 41, 49 against 53).
// Two 16-byte vectors per lane hold eight rows each in flight: two blocks of 128 (40 k rows of 20 entries, F = 64, four rows
// in flight at 80 registers 21.7 us, eight 19.0).
__host__ __device__ constexpr int blocks_per_sm(int w, int vpl) { return vpl == 1 || vpl * w <= 2 ? 4 : w == 4 ? 2 : 3; }

// A lane owns VPL vectors of W floats of the feature tile (VPL * LPR * W floats), LPR * W apart: one
// 16-byte vector where rows allow it, several 4- or 8-byte ones where their length or alignment
// does not (odd feature counts: tiles of up to 160 floats instead of 32, so that ids are read that
// much less often: 30 k rows, F = 299, 104 us with one vector, 66 with four, 59 with five).
template <int LPR, int W, int VPL>
__global__ void __launch_bounds__(kThreads, blocks_per_sm(W, VPL))
csr_split_kernel(const SplitArgs s) {
  using LV = LaneVec<W>;
  using V = typename LV::type;
  constexpr int SUBS = kThreads / LPR;
  constexpr int NW = 32 / LPR;                       // sub-warps of a warp
  constexpr int kU = W == 4 ? 8 : VPL <= 4 ? 16 / VPL : 4;  // more rows spill registers
  constexpr int U = kU < LPR ? kU : LPR;             // gathered rows in flight per lane
  constexpr int TILE = LPR * W * VPL;
  __shared__ __align__(16) float s_lead[SUBS][TILE];  // piece of a row that began before the sub-warp
  __shared__ __align__(16) float s_tail[SUBS][TILE];  // piece of a row that goes on behind it
  __shared__ int s_state[SUBS];                          // kLead, kOpen, kTail
  __shared__ int s_bounds[2];                            // first stored entry, end of the last
  constexpr int kLead = 1, kOpen = 2, kTail = 4;         // kOpen: the lead piece is the whole span

  const int wlane = threadIdx.x & 31;
  const int lane = threadIdx.x % LPR;
  const int sub = threadIdx.x / LPR;
  const unsigned mask = group_mask<LPR>();
  const long long block_entries = static_cast<long long>(SUBS) * s.span;
  const unsigned row_bytes = static_cast<unsigned>(s.feat) * 4u;
  const long long warp_at = blockIdx.x * block_entries + static_cast<long long>((threadIdx.x / 32) * NW) * s.span;
  chain_wait();
  // The stored entries are those between the first and the last row pointer: of a slice of a larger
  // matrix, or of arrays with room behind, not all nnz.  The two pointers are not waited for: ids and
  // row of the first entry are requested as if they were 0 and nnz, and once more where they are not.
  int lo = 0, hi = s.nnz;
  const int ptr_first = ld_global(s.indptr), ptr_last = ld_global(s.indptr + s.m);
  int p0 = 0, count = 0, steps = 0, cid = 0;  // of the sub-warp: first entry, entries; entries of the warp's first sub-warp
  float av = 0.f;
  auto first_ids = [&]() {
    cid = 0;
    av = 0.f;
    if (lane < count) {
      cid = ld_global(s.indices + p0 + lane);
      av = ld_global(s.a + p0 + lane);
    }
  };
  int first_row = 0;
  bool first_lead = false;  // the first row of the sub-warp began before it
#pragma unroll 1
  while (true) {
    const long long w0 = lo + warp_at;  // first entry of the warp
    const long long p0l = w0 + static_cast<long long>(wlane / LPR) * s.span;
    p0 = static_cast<int>(min(p0l, static_cast<long long>(hi)));
    count = static_cast<int>(min(p0l + s.span, static_cast<long long>(hi))) - p0;
    first_ids();  // on their way while the row is searched
    steps = static_cast<int>(max(0ll, min(static_cast<long long>(s.span), hi - w0)));
    if (steps > 0) {
      int pos[NW], row[NW];
#pragma unroll
      for (int i = 0; i < NW; ++i)
        pos[i] = static_cast<int>(min(w0 + static_cast<long long>(i) * s.span, static_cast<long long>(hi) - 1));
      warp_rows_of<NW>(s.indptr, s.m, pos, s.rows_per_entry, wlane, row);
      first_row = row[0];
#pragma unroll
      for (int i = 1; i < NW; ++i)
        if (wlane / LPR == i) first_row = row[i];
      first_lead = count > 0 && ld_global(s.indptr + first_row) < p0;
    }
    const int lo_now = max(0, min(ptr_first, s.nnz)), hi_now = max(lo_now, min(ptr_last, s.nnz));
    if (lo == lo_now && hi == hi_now) break;
    lo = lo_now;
    hi = hi_now;
  }
  if (threadIdx.x == 0) {  // read behind a barrier: they need no registers in the loops
    s_bounds[0] = lo;
    s_bounds[1] = hi;
  }

  const int tiles = (s.feat + TILE - 1) / TILE;
  for (int tile = blockIdx.y; tile < tiles; tile += gridDim.y) {
    const int f0 = tile * TILE + lane * W;
    // vectors past the row read the tile's first vector once more and store nothing
    bool inside[VPL];
    unsigned at[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      inside[v] = f0 + v * (LPR * W) < s.feat;
      at[v] = (inside[v] ? f0 + v * (LPR * W) : tile * TILE) * 4u;
    }
    const char* bl = reinterpret_cast<const char*>(s.b);
    char* cl = reinterpret_cast<char*>(s.c);
    auto c_row = [&](int r) -> char* {
      return cl + static_cast<unsigned long long>(static_cast<unsigned>(r)) * row_bytes;
    };
    if (tile > static_cast<int>(blockIdx.y)) {
      first_ids();
      __syncthreads();  // the pieces of the tile before have been collected
    }
    int r = first_row, state = 0;
    if (steps > 0) {  // the whole warp, its sub-warps in step
      int wend = row_window<LPR>(s.indptr, s.m, r, lane);
      bool lead = first_lead;
      if (lead) state = kLead;
      bool pending = false;  // entries of an unfinished row in acc
      V acc[VPL];
#pragma unroll
      for (int v = 0; v < VPL; ++v) acc[v] = LV::zero();
      for (int s0 = 0; s0 < steps; s0 += LPR) {
        int cidn;
        float avn;
        auto next_ids = [&]() {  // ids and values of the next batch; past the last one that of the last entry, not added
          const int at_next = max(p0 + min(s0 + LPR + lane, count - 1), 0);
          cidn = ld_global(s.indices + at_next);
          avn = ld_global(s.a + at_next);
        };
        const int cnt = max(0, min(LPR, count - s0));
        auto rows_of_b = [&](int k0, V (&x)[U][VPL]) {
#pragma unroll
          for (int u = 0; u < U; ++u) {  // entries past the end are not added
            const unsigned col = static_cast<unsigned>(__shfl_sync(0xffffffffu, cid, k0 + u, LPR));
            const char* src = bl + static_cast<unsigned long long>(col) * row_bytes;
#pragma unroll
            for (int v = 0; v < VPL; ++v) x[u][v] = LV::ldg(src + at[v]);
          }
        };
        // Most batches of a matrix of long rows lie inside one row for every sub-warp of the warp: a loop of
        // their own without tests per entry (10 M entries in rows of 500 on average, F = 128: 322 -> 277 us).
        // Groups of 8 lanes, whose batch is one step, take all that are left of the row in it: one step at a time 9.3 M
        // entries, F = 32, take 84 us, so 78.6.  Others gain nothing by it (F = 64 135, with the vote once per step 134).
        const int batches = lane != 0 ? INT32_MAX : min(count - s0, wend - (p0 + s0) - 1) / LPR;  // inside the sub-warp's row
        int inside_row = LPR == 8 ? __reduce_min_sync(0xffffffffu, batches) : __all_sync(0xffffffffu, batches > 0);
        if (inside_row > 0) {
          pending = true;
          while (true) {
#pragma unroll
            for (int k0 = 0; k0 < LPR; k0 += U) {
              V x[U][VPL];
              rows_of_b(k0, x);
              if (k0 == 0) next_ids();
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const float ak = __shfl_sync(0xffffffffu, av, k0 + u, LPR);
#pragma unroll
                for (int v = 0; v < VPL; ++v) LV::fma(acc[v], ak, x[u][v]);
              }
            }
            if (LPR != 8 || --inside_row == 0) break;
            s0 += LPR;
            cid = cidn;
            av = avn;
          }
        } else {
          next_ids();
          const int e = p0 + min(s0 + lane, count - 1);  // lanes past the last entry repeat it
          int row_end;
          const int row = row_in_window<LPR>(s.indptr, s.m, r, wend, e, row_end);
          const unsigned ends = group_ballot<LPR>(0xffffffffu, lane < cnt && row_end == e + 1);
          const unsigned any_ends = NW == 1 ? ends : __reduce_or_sync(0xffffffffu, ends);
          r = __shfl_sync(0xffffffffu, row, LPR - 1, LPR);
          if (cnt > 0) pending = ((ends >> (cnt - 1)) & 1u) == 0u;
          if (!pending && cnt > 0) r = min(r + 1, s.m - 1);
          // where the sum up to this entry goes if a row ends here; -1: the lead piece
          const int to = lead && (ends & ((1u << lane) - 1u)) == 0u ? -1 : row;
          if (ends != 0u) lead = false;
          wend = row_window<LPR>(s.indptr, s.m, r, lane);
#pragma unroll
          for (int k0 = 0; k0 < LPR; k0 += U) {
            if (k0 < steps - s0) {
              V x[U][VPL];
              rows_of_b(k0, x);
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const float ak = __shfl_sync(0xffffffffu, av, k0 + u, LPR);
                if (k0 + u < cnt) {
#pragma unroll
                  for (int v = 0; v < VPL; ++v) LV::fma(acc[v], ak, x[u][v]);
                }
                if ((any_ends >> (k0 + u)) & 1u) {  // a row ends here in some sub-warp of the warp
                  const int rk = __shfl_sync(0xffffffffu, to, k0 + u, LPR);
                  const bool end = (ends >> (k0 + u)) & 1u;
                  // one store instruction for both destinations: no branch among the sub-warps
                  char* dst = rk < 0 ? reinterpret_cast<char*>(&s_lead[sub][0]) - tile * (TILE * 4) : c_row(rk);
#pragma unroll
                  for (int v = 0; v < VPL; ++v) {
                    if (end && inside[v]) LV::st(dst + at[v], acc[v]);
                    LV::zero_if(acc[v], end);
                  }
                }
              }
            }
          }
        }
        cid = cidn;
        av = avn;
      }
      if (pending) {
        float* piece = lead ? s_lead[sub] : s_tail[sub];
#pragma unroll
        for (int v = 0; v < VPL; ++v) LV::sts(piece + v * (LPR * W) + lane * W, acc[v]);
        state |= lead ? kOpen : kTail;
      }
    }
    if (lane == 0) s_state[sub] = state;
    __syncthreads();

    // ---- rows that cross sub-warps
    auto finish = [&](V (&sum)[VPL], int row, bool from_before, bool goes_on) {
      if (from_before || goes_on) {
        const int begin = ld_global(s.indptr + row) - s_bounds[0];
        const int end = min(ld_global(s.indptr + row + 1), s_bounds[1]) - s_bounds[0];
        const int b0 = static_cast<int>(begin / block_entries), b1 = static_cast<int>((end - 1) / block_entries);
        char* pl = reinterpret_cast<char*>(s.part);
        auto piece = [&](int b) -> char* {
          return pl + (2ull * static_cast<unsigned>(b) + (b == b0 ? 1u : 0u)) * row_bytes;
        };
#pragma unroll
        for (int v = 0; v < VPL; ++v)
          if (inside[v]) LV::stcg(piece(blockIdx.x) + at[v], sum[v]);
        __threadfence();
        __syncwarp(mask);
        unsigned* counter = s.counters + static_cast<size_t>(b0) * tiles + tile;
        unsigned seen = 0;
        if (lane == 0) seen = atomicAdd(counter, 1u);
        seen = __shfl_sync(mask, seen, 0, LPR);
        if (seen != static_cast<unsigned>(b1 - b0)) return;
        if (lane == 0) *counter = 0u;  // last piece to arrive: all of them are visible
        __threadfence();
        constexpr int G = VPL < 5 ? 8 / VPL : 2;
#pragma unroll
        for (int v = 0; v < VPL; ++v) sum[v] = LV::zero();
        for (int b = b0; b <= b1; b += G) {
          V x[G][VPL];
#pragma unroll
          for (int u = 0; u < G; ++u)
#pragma unroll
            for (int v = 0; v < VPL; ++v) x[u][v] = LV::ldcg(piece(min(b + u, b1)) + at[v]);
#pragma unroll
          for (int u = 0; u < G; ++u)
            if (b + u <= b1) {
#pragma unroll
              for (int v = 0; v < VPL; ++v) LV::add(sum[v], x[u][v]);
            }
        }
      }
#pragma unroll
      for (int v = 0; v < VPL; ++v)
        if (inside[v]) LV::stcs(c_row(row) + at[v], sum[v]);  // written once: keep B rows in L2
    };
    // adds the lead pieces of sub-warps k, k + 1, ... until the row ends; true if it leaves the block
    auto collect = [&](V (&sum)[VPL], int k) -> bool {
      for (; k < SUBS; ++k) {
#pragma unroll
        for (int v = 0; v < VPL; ++v) LV::add(sum[v], LV::lds(&s_lead[k][v * (LPR * W) + lane * W]));
        if ((s_state[k] & kOpen) == 0) return false;
      }
      return true;
    };
    const bool more_blocks = s_bounds[0] + (blockIdx.x + 1) * block_entries < s_bounds[1];
    if (sub == 0 && (state & kLead)) {
      V sum[VPL];
#pragma unroll
      for (int v = 0; v < VPL; ++v) sum[v] = LV::zero();
      const bool goes_on = collect(sum, 0);
      finish(sum, first_row, true, goes_on && more_blocks);
    }
    if (state & kTail) {
      V sum[VPL];
#pragma unroll
      for (int v = 0; v < VPL; ++v) sum[v] = LV::lds(&s_tail[sub][v * (LPR * W) + lane * W]);
      const bool goes_on = collect(sum, sub + 1);
      finish(sum, r, false, goes_on && more_blocks);
    }
  }  // feature tiles

  // ---- rows without entries: this block's share of the rows
  if (blockIdx.y == 0) {
    const int per = static_cast<int>((static_cast<long long>(s.m) + gridDim.x - 1) / gridDim.x);
    const long long ra = static_cast<long long>(blockIdx.x) * per;
    const long long rb = min(static_cast<long long>(s.m), ra + per);
    for (long long r0 = ra + threadIdx.x - wlane; r0 < rb; r0 += kThreads) {
      const long long rr = r0 + wlane;
      const bool empty = rr < rb && ld_global(s.indptr + rr) == ld_global(s.indptr + rr + 1);
      unsigned todo = __ballot_sync(0xffffffffu, empty);
      while (todo != 0u) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1u;
        char* dst = reinterpret_cast<char*>(s.c) + static_cast<unsigned long long>(r0 + k) * row_bytes;
        for (unsigned at = wlane * (W * 4u); at < row_bytes; at += 32u * W * 4u) LV::stcs(dst + at, LV::zero());
      }
    }
  }
}

// Lanes per row, floats per vector, vectors per lane.
struct SplitShape {
  int lanes, w, vpl;
};

// Two vectors per lane on half the lanes, us, one vector / two (rows of about equal length unless said otherwise):
//  - up to 64 features: 30 k rows of 12 15.3 / 12.1, 9 k of 60 15.9 / 13.8, 200 k of 30 117 / 109, power-law graphs (4.5 per row)
//    70 k 18.1 / 15.8, 200 k 34.7 / 34.7; 36 features, 20 k of 40 24.2 / 19.5, 40 k of 200 161 / 146.
//  - up to 64, no whole tile, long rows: equal ones lose by it and uneven ones gain, more by the fewer of the lanes' second vectors are in use:
//    20 k rows of 500 / 20 k log-normal ones of that mean, F = 36 180 / 192 and 173 / 153, F = 48 180 / 186 and 170 / 147, F = 52 181 / 200 and
//    172 / 162, F = 60 183 / 205 and 176 / 167; 40 k of 300 F = 36 213 / 223, F = 60 213 / 239; 40 k of 200 F = 52 153 / 153, F = 60 154 / 157, 20 k of 200 F = 60
//    77 / 72.  Sizes do not tell the two apart; uneven rows, which graphs of that density have, decide (attention over 40 k of
//    them, F = 56, one vector from 250 entries per row on 806, two 789).
//  - more: 30 k of 8 F = 128 18.1 / 17.5, of 12 21.8 / 21.1, F = 512 70.8 / 68.1, 20 k of 10 F = 68 14.7 / 13.1; where a slice of B is more than a share of L2, from 10
//    entries per row on (60 k of 10 F = 128 31.5 / 31.1, 75 k of 12 42.9 / 42.1, 60 k of 20 F = 512 186 / 176; 60 k of 8 F = 100 28.1 / 29.6, F = 512 97 / 103, 90 k of 6
//    F = 256 62.9 / 66.9); where it is more than L2 keeps they bring nothing (200 k of 16 F = 128 148 / 161), nor on power-law graphs (100 k
//    F = 128 28.4 / 29.5).
//  - whole tiles on long rows are at the L2-to-SM rate with either (200 per row and more, F = 64 and 128: within the 15 % by which
//    one kernel's time moves there with the share of a sub-warp): not taken.
//  - less than a batch for each of the resident blocks, half as many here: not taken (3 k of 30 F = 128 9.4 / 10.0).
bool two_vectors(int m, int n, int feat, int nnz, bool whole) {
  const int per_row = nnz / m;
  if (whole && per_row >= 100) return false;
  if (feat <= 64) return nnz >= 80000;
  const size_t slice = static_cast<size_t>(n) * std::min(feat * 4, 512);
  return nnz >= 100000 && per_row >= (slice <= (size_t{22} << 20) ? 6 : 10) && slice <= (size_t{48} << 20);
}

SplitShape split_shape(uintptr_t bits, int m, int n, int feat, int nnz) {
  if (feat % 4 == 0 && bits % 16 == 0) {
    // The narrowest group that covers a row, a warp at most: several sub-warps per warp keep more
    // rows in flight (4.5 M entries, F = 64: 16 lanes 93, 32 lanes 160, 8 lanes 107 us), a second
    // pass over the entries costs more than it brings (169 k-node power-law graph, F = 128: 32
    // lanes 56, 16 lanes 68 us) unless every row of B is gathered so often that a slice of B that
    // stays in L2 pays for it.
    int lanes = feat <= 32 ? 8 : (feat <= 64 ? 16 : 32);
    while (lanes > 8 && n > 0 && nnz / n >= 64 &&
           static_cast<size_t>(n) * std::min(lanes * 16, feat * 4) > (size_t{48} << 20))
      lanes /= 2;
    // Half the lanes with two vectors each: half the shuffles per entry.
    if (lanes > 8 && two_vectors(m, n, feat, nnz, feat % (lanes * 4) == 0)) return {lanes / 2, 4, 2};
    return {lanes, 4, 1};
  }
  if (feat % 2 == 0 && bits % 8 == 0) return {feat <= 16 ? 8 : (feat <= 32 ? 16 : 32), 2, feat <= 64 ? 1 : 2};
  if (feat <= 32) return {feat <= 8 ? 8 : (feat <= 16 ? 16 : 32), 1, 1};
  return {32, 1, feat <= 64 ? 2 : (feat <= 128 ? 4 : 5)};
}

struct SplitPlan {
  int gy, span, blocks;
  size_t part_bytes, counter_bytes;
};

SplitPlan split_plan(const SplitShape& sh, int m, int feat, int nnz) {
  const int subs = kThreads / sh.lanes;
  const int tiles = ceil_div(feat, sh.lanes * sh.w * sh.vpl);
  // One wave of resident blocks with equal shares of the entries: a block's fixed cost (search,
  // meeting of the pieces) is paid once, 4.5 M entries, F = 64: 94 us against 109 with four waves.
  // A block walks the feature tiles one after the other, all blocks roughly in step, which keeps
  // the slice of B that they gather from in L2; matrices too small to give every resident block
  // three batches of entries for each of its sub-warps deal the tiles to more blocks, equal shares of them.
  //
  // Shares of a few batches are made up to a multiple of 8 entries and not to whole batches: of 32 entries, 40 k of them, F = 512, took 628
  // blocks, 1.06 waves, or a third of the blocks for four tiles (us, four tiles side by side in 1.06 waves / three in one / four in one with
  // shares of 40 entries: 10 k rows of 4 16.5 / 17.8 / 13.9, 10 k power-law rows 16.4 / 19.0 / 14.8; other calls of up to two waves, two waves / one
  // with such shares: 20 k power-law rows F = 256 16.8 / 15.0, 9 k rows of 9 F = 384 18.0 / 15.3, 30 k of 5, F = 299 32.4 / 29.5; one tile, 40 k
  // power-law rows, F = 100 16.9 / 15.4).  Two tiles on one block and one on the next: 14 k rows of 7, F = 384 20.2 / 23.5, three side by side 17.0.
  const long long resident = static_cast<long long>(blocks_per_sm(sh.w, sh.vpl)) * kNumSMs, batch = static_cast<long long>(subs) * sh.lanes;
  const long long fewest = (nnz + batch - 1) / batch;
  SplitPlan p;
  p.gy = static_cast<int>(std::min<long long>(tiles, std::max<long long>(1, resident * 3 / fewest)));
  int even = p.gy;
  while (tiles % even != 0) ++even;
  if (even <= resident) p.gy = even;  // a prime number of tiles is not a number of blocks that a grid can have
  const long long want = std::max<long long>(1, resident / p.gy) * subs, share = (nnz + want - 1) / want;
  const long long step = share < 4 * sh.lanes ? 8 : sh.lanes;
  p.span = static_cast<int>(std::max<long long>(sh.lanes, (share + step - 1) / step * step));
  const long long per_block = static_cast<long long>(subs) * p.span;
  const long long with_entries = (nnz + per_block - 1) / per_block;  // the first blocks; the others clear rows
  p.blocks = static_cast<int>(std::max(with_entries, (static_cast<long long>(m) + 8 * kThreads - 1) / (8 * kThreads)));
  p.part_bytes = 2 * static_cast<size_t>(with_entries) * feat * sizeof(float);
  p.counter_bytes = static_cast<size_t>(with_entries) * tiles * sizeof(unsigned);
  return p;
}

template <int LPR, int W, int VPL>
int launch_split(const SplitArgs& s, const SplitPlan& p, cudaStream_t st) {
  launch_chained_if(s.nnz < kChainEntries, csr_split_kernel<LPR, W, VPL>, dim3(p.blocks, p.gy), kThreads, 0, st, s);
  SPTIR_LAUNCH_OK("csr_split_kernel");
  return 0;
}

int dispatch_split(const SplitArgs& s, const SplitShape& sh, const SplitPlan& p, cudaStream_t st) {
  if (sh.w == 4) {
    if (sh.vpl == 2) return sh.lanes == 8 ? launch_split<8, 4, 2>(s, p, st) : launch_split<16, 4, 2>(s, p, st);
    if (sh.lanes == 8) return launch_split<8, 4, 1>(s, p, st);
    if (sh.lanes == 16) return launch_split<16, 4, 1>(s, p, st);
    return launch_split<32, 4, 1>(s, p, st);
  }
  if (sh.w == 2) {
    if (sh.lanes == 8) return launch_split<8, 2, 1>(s, p, st);
    if (sh.lanes == 16) return launch_split<16, 2, 1>(s, p, st);
    if (sh.vpl == 1) return launch_split<32, 2, 1>(s, p, st);
    return launch_split<32, 2, 2>(s, p, st);
  }
  if (sh.lanes == 8) return launch_split<8, 1, 1>(s, p, st);
  if (sh.lanes == 16) return launch_split<16, 1, 1>(s, p, st);
  if (sh.vpl == 1) return launch_split<32, 1, 1>(s, p, st);
  if (sh.vpl == 2) return launch_split<32, 1, 2>(s, p, st);
  if (sh.vpl == 4) return launch_split<32, 1, 4>(s, p, st);
  return launch_split<32, 1, 5>(s, p, st);
}

inline uintptr_t low_bits(const float* b, const float* c) {
  return reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
}

}  // namespace

// Bytes of scratch that the pieces of this call need.
size_t csr_split_scratch(const float* b, const float* c, int m, int n, int feat, int nnz) {
  if (nnz == 0) return 0;
  return split_plan(split_shape(low_bits(b, c), m, n, feat, nnz), m, feat, nnz).part_bytes;
}

// The most that a call of these sizes needs, whatever its operands' alignment.
void csr_split_scratch_bound(int m, int n, int feat, int nnz, size_t* part_bytes, size_t* counter_bytes) {
  *part_bytes = *counter_bytes = 0;
  if (m == 0 || feat == 0 || nnz == 0) return;
  for (const uintptr_t bits : {16, 8, 4}) {
    const SplitPlan p = split_plan(split_shape(bits, m, n, feat, nnz), m, feat, nnz);
    *part_bytes = std::max(*part_bytes, p.part_bytes);
    *counter_bytes = std::max(*counter_bytes, p.counter_bytes);
  }
}

// pieces: csr_split_scratch() bytes, 16-byte aligned, from a caller that holds the stream's scratch buffer; null:
// the call takes its scratch itself.
int csr_split_run(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
                  int m, int n, int feat, int nnz, void* pieces, int device_id, cudaStream_t st) {
  if (nnz == 0) {
    SPTIR_CUDA_OK(cudaMemsetAsync(c, 0, static_cast<size_t>(m) * feat * sizeof(float), st));
    return 0;
  }
  const SplitShape sh = split_shape(low_bits(b, c), m, n, feat, nnz);
  const SplitPlan p = split_plan(sh, m, feat, nnz);
  CallScratch cs;
  if (pieces != nullptr) {
    cs.scratch = static_cast<char*>(pieces);
    cs.counters = static_cast<unsigned*>(zeroed_workspace(device_id, st, p.counter_bytes));
    if (cs.counters == nullptr) return -1;
  } else if (take_scratch(device_id, st, p.part_bytes, p.counter_bytes, &cs) != 0) {
    return -1;
  }
  const SplitArgs s{a, b, c, indptr, indices, reinterpret_cast<float*>(cs.scratch), cs.counters, m, nnz, feat, p.span,
                    static_cast<float>(m) / static_cast<float>(nnz)};
  if (dispatch_split(s, sh, p, st) != 0) return -1;
  return return_scratch(cs, st);
}

}  // namespace sptir

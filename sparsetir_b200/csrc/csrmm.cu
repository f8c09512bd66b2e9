// CSR SpMM, fp32:  C[i,:] = sum_{p in row i} A[p] * B[indices[p],:]
// Semantics: tests/python/sparsetir/sparse_tir_lowered_buffer_scripts.py:22-68 of the reference;
// like the reference's scheduled GPU kernel (examples/spmm/bench_spmm_naive.py:102-119) rows
// without entries are written as zeros.
//
// Two kernels.  Matrices of a few thousand rows, and callers that promise short rows (the
// sums of RGMS in the forms that rgms_pairs.cu does not take), take the row-wise kernel below: row
// pointer -> ids -> rows of B is the shortest chain of memory round trips there is.  All others take the kernel that splits the
// matrix by stored entries (csr_split.cu).
#include <algorithm>
#include <cstdlib>

#include "common.h"
#include "launch.cuh"
#include "row_walk.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 256;

// ---------------------------------------------------------------------------------------------
// Lean kernel: fast path for 16-byte aligned operands and whole feature tiles.
// A sub-warp of LPR lanes owns `rpi` consecutive rows (rpi < LPR).  Short rows are the hard
// case for CSR: row pointer -> ids -> dense rows is a chain of three dependent memory round
// trips, and a row of two or three entries gives nothing to overlap them with.  So the chain is
// paid once per ITEM, not per row: the rpi+1 row pointers are read with one coalesced load and
// kept in registers (lane j holds indptr[r0+j], fetched by shuffle at row ends), the item's
// entries are one contiguous slot stream whose ids/values are read a batch of LPR ahead, and the
// dense rows are gathered 8 at a time.  One writer per output row, CSR summation order, rows
// without entries written as zeros.
//
// HUBS: a row of more than `long_row` entries, which one sub-warp would walk alone (a 2,000-entry row
// of an 8,000-row graph: 100 us beside 5 us for all the others), is left to the end of its block
// and then shared by all sub-warps; their partial sums are added in order.  long_row is 64, or four
// times the average row where that is more: rows that are all about as long are spread over the sub-warps
// as they are (1,000 rows of 60 entries, F = 64: 13 us, taken one after the other by the block 18).  Blocks
// without long rows pay for one barrier behind the row pointers; what the others need inline, or the barrier
// at the end, cost up to a tenth (8,191 rows of 3 entries, F = 512: 16.4 against 18.0 us).
constexpr int kLongRow = 64;

// All of a block whose items hold long rows: the other rows one after the other by their sub-warps, then
// the long ones by all sub-warps.  It starts from the kernel's arguments: nothing is kept for it elsewhere.
template <int LPR, int W>
__device__ __noinline__ void block_with_long_rows(const float* a, const float* b, float* c, const int32_t* indptr,
                                                  const int32_t* indices, int m, int feat, int rpi, int long_row) {
  using LV = LaneVec<W>;
  constexpr int SUBS = kThreads / LPR;
  __shared__ unsigned s_long[SUBS];  // the long rows of every sub-warp's item, a bit each
  __shared__ __align__(32) float s_part[SUBS][LPR * W];
  const int lane = threadIdx.x % LPR, sub = threadIdx.x / LPR;
  const unsigned mask = group_mask<LPR>();
  const long long item0 = static_cast<long long>(blockIdx.x) * SUBS;
  const int r0 = static_cast<int>(min((item0 + sub) * rpi, static_cast<long long>(m)));
  const int nr = min(rpi, m - r0);
  const unsigned row_bytes = static_cast<unsigned>(feat) * 4u;
  const unsigned off = (blockIdx.y * LPR + lane) * (W * 4u);
  const char* bl = reinterpret_cast<const char*>(b) + off;
  char* cl = reinterpret_cast<char*>(c) + off;
  auto c_row = [&](int r) -> char* { return cl + static_cast<unsigned long long>(static_cast<unsigned>(r)) * row_bytes; };
  unsigned long_rows = 0;
  for (int j = 0; j < nr; ++j) {
    const int begin = ld_global(indptr + r0 + j), end = ld_global(indptr + r0 + j + 1);
    if (end - begin > long_row) {
      long_rows |= 1u << j;
      continue;
    }
    typename LV::type acc = LV::zero();
    add_entries<LPR, W>(a, indices, bl, row_bytes, begin, end, LPR, lane, mask, acc);
    LV::stcs(c_row(r0 + j), acc);
  }
  if (lane == 0) s_long[sub] = long_rows;
  __syncthreads();
  for (int owner = 0; owner < SUBS; ++owner) {
    for (unsigned todo = s_long[owner]; todo != 0u; todo &= todo - 1u) {
      const int row = static_cast<int>((item0 + owner) * rpi) + __ffs(todo) - 1;
      const int begin = ld_global(indptr + row), end = ld_global(indptr + row + 1);
      typename LV::type acc = LV::zero();
      add_entries<LPR, W>(a, indices, bl, row_bytes, begin + sub * LPR, end, SUBS * LPR, lane, mask, acc);
      LV::sts(&s_part[sub][lane * W], acc);
      __syncthreads();
      if (sub == 0) {
        for (int j = 1; j < SUBS; ++j) LV::add(acc, LV::lds(&s_part[j][lane * W]));
        LV::stcs(c_row(row), acc);
      }
      __syncthreads();
    }
  }
}

template <int LPR, int W, bool HUBS>  // W floats per lane: 4 (16-byte vectors) or 8 (32-byte vectors)
__global__ void __launch_bounds__(kThreads, 4)
csrmm_lean_kernel(const float* a, const float* b, float* __restrict__ c,
                  const int32_t* indptr, const int32_t* indices, int m,
                  int feat, int rpi, int long_row) {
  using LV = LaneVec<W>;
  using V = typename LV::type;
  constexpr int SUBS = kThreads / LPR;
  constexpr int U = (32 / W) < LPR ? (32 / W) : LPR;  // gathered rows in flight: 32 registers
  const int lane = threadIdx.x % LPR;
  const unsigned mask = group_mask<LPR>();
  const long long item = static_cast<long long>(blockIdx.x) * SUBS + threadIdx.x / LPR;
  const long long r0l = item * rpi;
  chain_wait();
  if (!HUBS && r0l >= m) return;
  const int r0 = static_cast<int>(min(r0l, static_cast<long long>(m)));
  const int nr = min(rpi, m - r0);  // 0 past the last row
  const int ptr = ld_global(indptr + r0 + min(lane, nr));  // lane j: start of row r0+j (j <= nr)
  const unsigned row_bytes = static_cast<unsigned>(feat) * 4u;
  const unsigned off = (blockIdx.y * LPR + lane) * (W * 4u);
  const char* bl = reinterpret_cast<const char*>(b) + off;
  char* cl = reinterpret_cast<char*>(c) + off +
             static_cast<unsigned long long>(static_cast<unsigned>(r0)) * row_bytes;

  if (HUBS) {
    const int len = __shfl_down_sync(mask, ptr, 1, LPR) - ptr;
    if (__syncthreads_or(lane < nr && len > long_row)) {
      block_with_long_rows<LPR, W>(a, b, c, indptr, indices, m, feat, rpi, long_row);
      return;
    }
  }
  if (nr > 0) {
    // ---- the rows of the item: one contiguous slot stream
    const int p0s = __shfl_sync(mask, ptr, 0, LPR);
    const int nslots_s = __shfl_sync(mask, ptr, nr, LPR) - p0s;
    const int32_t* cols_s = indices + p0s;
    const float* wts_s = a + p0s;
    V acc = LV::zero();
    int j = 0;                                             // row being accumulated
    int row_end = __shfl_sync(mask, ptr, 1, LPR) - p0s;  // its end, as a slot number
    int s = 0;                                              // slots consumed so far
    auto finish_rows = [&]() {  // store every row whose last entry has been consumed
      while (j < nr && s >= row_end) {
        LV::stcs(cl, acc);  // written once: keep B rows in L2
        acc = LV::zero();
        cl += row_bytes;
        ++j;
        row_end = __shfl_sync(mask, ptr, min(j + 1, nr), LPR) - p0s;
      }
    };
    finish_rows();  // rows without entries at the front

    int cid = 0, cidn = 0;
    float av = 0.f, avn = 0.f;
    if (lane < nslots_s) {
      cid = ld_global(cols_s + lane);
      av = ld_global(wts_s + lane);
    }
    for (int s0 = 0; s0 < nslots_s; s0 += LPR) {
      cidn = 0;
      avn = 0.f;
      if (s0 + LPR + lane < nslots_s) {  // ids and values of the next batch
        cidn = ld_global(cols_s + s0 + LPR + lane);
        avn = ld_global(wts_s + s0 + LPR + lane);
      }
      const int cnt = min(LPR, nslots_s - s0);
#pragma unroll
      for (int k0 = 0; k0 < LPR; k0 += U) {
        if (k0 < cnt) {
          V x[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {  // slots past the end ask for column 0: never consumed
            const unsigned col = static_cast<unsigned>(__shfl_sync(mask, cid, k0 + u, LPR));
            x[u] = LV::ldg(bl + static_cast<unsigned long long>(col) * row_bytes);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const float ak = __shfl_sync(mask, av, k0 + u, LPR);
            if (k0 + u < cnt) {
              LV::fma(acc, ak, x[u]);
              ++s;
              if (s >= row_end) finish_rows();
            }
          }
        }
      }
      cid = cidn;
      av = avn;
    }
  }
}

}  // namespace
}  // namespace sptir

namespace sptir {
int csr_split_run(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
                  int m, int n, int feat, int nnz, void* pieces, int device_id, cudaStream_t st);
size_t csr_split_scratch(const float* b, const float* c, int m, int n, int feat, int nnz);
void csr_split_scratch_bound(int m, int n, int feat, int nnz, size_t* part_bytes, size_t* counter_bytes);

namespace {
// Whether a call takes the row-wise kernel, and with which lanes.
bool row_wise(const float* b, const float* c, int m, int n, int feat, int nnz, bool hub_rows, int* lane_w, int* lanes_per_row) {
  const bool vec4 = (feat % 4 == 0) && aligned16(b) && aligned16(c);
  // The row-wise kernel needs whole feature tiles.  Its share ends where the split by entries is
  // the faster one although it has to search for its rows: 4,096 rows of 10 entries, F = 64, 4.8
  // against 7.1 us; 16,886 power-law rows, F = 32, 23.4 (with the two launches for hub rows that
  // it needed there) against 9.6 us.
  const bool small = m < 8192 && nnz < 65536;
  if (!vec4 || (!small && hub_rows)) return false;
  // lanes per row: one per 32-byte vector when the operands allow it, else one per 16-byte
  // vector; narrowed until the n x tile slice of B that a pass over the rows gathers from fits
  // the resident part of L2 (see hyb_spmm.cu)
  const int w = (feat % 32 == 0 && aligned32(b) && aligned32(c)) ? max_lane_floats() : 4;
  const int nv = feat / w;
  int lanes = nv <= 4 ? 4 : (nv <= 8 ? 8 : (nv <= 16 ? 16 : 32));
  if (w == 4 && lanes < 8) lanes = 8;
  const size_t l2_budget = 48u << 20;
  const int min_lanes = w == 8 ? 4 : 8;
  while (lanes > min_lanes && static_cast<size_t>(n) * lanes * w * 4 > l2_budget) lanes /= 2;
  *lane_w = w;
  *lanes_per_row = lanes;
  return feat % (w * lanes) == 0;
}
}  // namespace

// Scratch that a csrmm call over these operands needs (0: none), for callers that hold the stream's buffer.
size_t csrmm_scratch(const float* b, const float* c, int m, int n, int feat, int nnz) {
  int w = 0, lanes = 0;
  return row_wise(b, c, m, n, feat, nnz, true, &w, &lanes) ? 0 : csr_split_scratch(b, c, m, n, feat, nnz);
}

// The launcher behind sparsetir_csrmm_raw.  hub_rows = false: the caller knows that its rows are
// short, and that b and c are 16-byte aligned with feat a multiple of 64 that makes whole tiles; such a
// call never touches the per-stream workspace (the caller may hold it).
// pieces: csrmm_scratch() bytes from a caller that holds the stream's scratch buffer, null from others.
int csrmm_run(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
              int m, int n, int feat, int nnz, int device_id, void* stream, bool hub_rows, void* pieces) {
  if (m < 0 || feat < 0 || nnz < 0) return fail("sparsetir_csrmm: negative size");
  if (m == 0 || feat == 0) return 0;
  if (!b || !c || !indptr || (nnz > 0 && (!a || !indices)))
    return fail("sparsetir_csrmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled() && validate_csr("sparsetir_csrmm", indptr, m, indices, nnz, n, st) != 0) return -1;
  int w = 0, lanes = 0;
  if (row_wise(b, c, m, n, feat, nnz, hub_rows, &w, &lanes)) {
    const int subs = kThreads / lanes;
    // about four id batches per item, but never so few items that SMs sit idle
    const double avg = m > 0 ? static_cast<double>(nnz) / m : 0.0;
    int rpi = static_cast<int>(4.0 * lanes / (avg > 1.0 ? avg : 1.0));
    rpi = rpi < 1 ? 1 : (rpi > lanes - 1 ? lanes - 1 : rpi);
    const long long want_items = 4ll * kNumSMs * 4 * subs;
    while (rpi > 1 && (m + rpi - 1) / rpi < want_items) rpi /= 2;
    const int long_row = std::max(kLongRow, static_cast<int>(4.0 * avg));
    dim3 grid(ceil_div(ceil_div(m, rpi), subs), feat / (w * lanes));
#define SPTIR_CSR_LEAN(L, WW)                                                                                   \
  if (hub_rows)                                                                                                 \
    launch_chained(csrmm_lean_kernel<L, WW, true>, grid, kThreads, 0, st, a, b, c, indptr, indices, m, feat, rpi, long_row); \
  else                                                                                                          \
    launch_chained(csrmm_lean_kernel<L, WW, false>, grid, kThreads, 0, st, a, b, c, indptr, indices, m, feat, rpi, 0)
    if (w == 8) {
      if (lanes == 4) { SPTIR_CSR_LEAN(4, 8); }
      else if (lanes == 8) { SPTIR_CSR_LEAN(8, 8); }
      else if (lanes == 16) { SPTIR_CSR_LEAN(16, 8); }
      else { SPTIR_CSR_LEAN(32, 8); }
    } else {
      if (lanes == 8) { SPTIR_CSR_LEAN(8, 4); }
      else if (lanes == 16) { SPTIR_CSR_LEAN(16, 4); }
      else { SPTIR_CSR_LEAN(32, 4); }
    }
#undef SPTIR_CSR_LEAN
    SPTIR_LAUNCH_OK("csrmm_lean_kernel");
    return 0;
  }
  if (!hub_rows) return fail("sparsetir_csrmm: short-row call with operands that are not whole tiles");
  return csr_split_run(a, b, c, indptr, indices, m, n, feat, nnz, pieces, device_id, st);
}

int csrmm_impl(const float* a, const float* b, float* c, const int32_t* indptr, const int32_t* indices,
               int m, int n, int feat, int nnz, int device_id, void* stream, bool hub_rows) {
  return csrmm_run(a, b, c, indptr, indices, m, n, feat, nnz, device_id, stream, hub_rows, nullptr);
}

// For matrices of very short rows: the sums of RGMS where rgms_pairs.cu does not take them, which is under its comparison switch at 64
// features, and at 128 and 256 where X is not 32-byte aligned.
int csrmm_short_rows_impl(const float* a, const float* b, float* c, const int32_t* indptr,
                          const int32_t* indices, int m, int n, int feat, int nnz, int device_id,
                          void* stream) {
  return csrmm_run(a, b, c, indptr, indices, m, n, feat, nnz, device_id, stream, false, nullptr);
}
}  // namespace sptir

extern "C" int sparsetir_csrmm_workspace(int m, int n, int feat, int nnz, size_t* scratch_bytes, size_t* counter_bytes) {
  if (m < 0 || n < 0 || feat < 0 || nnz < 0 || !scratch_bytes || !counter_bytes)
    return sptir::fail("sparsetir_csrmm_workspace: bad argument");
  sptir::csr_split_scratch_bound(m, n, feat, nnz, scratch_bytes, counter_bytes);
  return 0;
}

extern "C" int sparsetir_csrmm_raw(const float* a, const float* b, float* c, const int32_t* indptr,
                                   const int32_t* indices, int m, int n, int feat, int nnz,
                                   int device_id, void* stream) {
  return sptir::csrmm_impl(a, b, c, indptr, indices, m, n, feat, nnz, device_id, stream, true);
}

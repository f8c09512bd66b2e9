// Condensed tensor-core SpMM ("tcspmm"), fp16 operands, fp32 accumulation:
//   C[io*t + ii, f] = sum_{jo in [indptr[io], indptr[io+1])} sum_{ji < g} A[jo,ii,ji] * B[indices[jo*g+ji], f]
// Semantics: examples/spmm/bench_tc_spmm.py:537-565 of the reference (operator `tcspmm`; the
// wmma schedule it replaces: :591-640); the condensed operands come from ConDense
// (src/sparse/format.cc:353-429): every t-row tile keeps the sorted distinct columns it touches,
// g at a time; A holds the t x g values (mask) of a group, `indices` its g source rows.
//
// Tensor-core form (g = 16, t = 8, 16 or 32, feat a multiple of 8).  Of a group's work the gather of
// 16 rows of B is what costs: 2 KB per 64 features against 8 instructions of m16n8k16.  So the
// operands never touch shared memory: a warp owns 64 features of a row tile and loads both
// operands straight into the registers that the instruction reads (mma16.cuh); its four source rows are
// 16 bytes of `indices`.
// Two groups are in flight per warp.  Row tiles of up to kLight groups are one warp's work; longer
// ones (hub rows) are cut at multiples of a window of groups of the whole matrix: a block owns a window,
// its four warps share the part of each long tile that lies in it and meet in shared memory; parts
// of a tile in several windows meet in a scratch buffer, where the block that counts in last adds them in
// order.  One launch, no plan, every output written once, the same bits on every call.
//
// It replaces a tcgen05 kernel (one block per tile and 128 features, operands through shared memory,
// atomics for hub tiles) whose steps waited for one another, and CUDA-core code for the feature counts
// that are not multiples of 128.  Power-law graphs, float16 result, us, before / now: 169 k rows (57,508
// groups) F = 64 6010 / 32, F = 128 137 / 61, F = 512 422 / 222; 20 k rows F = 128 52 / 14; 3 k rows 39 / 9.
// Bound: the round trips indptr -> indices -> B of a short tile, with 20 warps of two groups per SM in
// flight; at F = 128 the 57,508 groups load 4.6 KB each, 4.4 TB/s (counters of one launch: L1 data path 61 % of the elapsed
// time, issue slots 29 %, L2 20 %, DRAM 18 %, 25 % of the warp slots in use).  Slower: neighbouring short tiles as one stream per
// warp (72 us at F = 128), 16 or 24 warps per SM (66, 111), windows of 32 groups at this size (68).
// Other shapes run on CUDA cores.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "mma16.cuh"
#include "row_walk.cuh"
#include "vec.cuh"

namespace sptir {
namespace {

constexpr int kThreads = 128;
constexpr int kG = 16;
constexpr int kLight = 16;    // longest tile of a single warp, in groups

template <typename OutT> __device__ __forceinline__ OutT to_out(float v);
template <> __device__ __forceinline__ float to_out<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_out<__half>(float v) { return __float2half_rn(v); }

struct TcArgs {
  const __half* a;
  const __half* b;
  void* c;
  const int32_t* indptr;
  const int32_t* indices;
  float* part;         // two pieces per window and slab: of a tile that began before it, of one that goes on behind it
  unsigned* counters;  // [windows][slabs], zero before and after every launch
  int mb, nnzb, t, feat, slabs, windows;
  int window_log;      // groups per block of the long tiles: 2^window_log
  float tiles_per_group;
  bool vec_indices;    // `indices` is 16-byte aligned
  bool vec_out;        // rows of C are made of whole 16-byte pieces
  bool wide_out;       // ... and, 16 results at a time, of whole 32-byte sectors
};

// 8 consecutive results of row `ii` (inside the tile) from feature f on
__device__ __forceinline__ void store8(const TcArgs& s, float* c, int io, int ii, int f, const float (&v)[8]) {
  float* dst = c + (static_cast<size_t>(io) * s.t + ii) * s.feat + f;
  if (s.vec_out) {
    __stcs(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
    __stcs(reinterpret_cast<float4*>(dst) + 1, make_float4(v[4], v[5], v[6], v[7]));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[j] = v[j];
  }
}
__device__ __forceinline__ void store8(const TcArgs& s, __half* c, int io, int ii, int f, const float (&v)[8]) {
  __half* dst = c + (static_cast<size_t>(io) * s.t + ii) * s.feat + f;
  if (s.vec_out) {
    uint4 o;
    __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
    __stcs(reinterpret_cast<uint4*>(dst), o);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) dst[j] = __float2half_rn(v[j]);
  }
}

// 16 consecutive results, which a lane of a short tile holds: whole sectors in one instruction.  As two stores of 16
// bytes every sector of a float16 result went to L2 in halves (169 k rows, F = 128 57.7 / 56.3 us, F = 512 222 / 216).
__device__ __forceinline__ void store16(const TcArgs& s, float* c, int io, int ii, int f, const float (&v)[8], const float (&w)[8]) {
  float* dst = c + (static_cast<size_t>(io) * s.t + ii) * s.feat + f;
  Pack4 a, b;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a.q[j] = pack_pair(v[2 * j], v[2 * j + 1]);
    b.q[j] = pack_pair(w[2 * j], w[2 * j + 1]);
  }
  stcs256(dst, a);
  stcs256(dst + 8, b);
}
__device__ __forceinline__ void store16(const TcArgs& s, __half* c, int io, int ii, int f, const float (&v)[8], const float (&w)[8]) {
  __half* dst = c + (static_cast<size_t>(io) * s.t + ii) * s.feat + f;
  Pack4 a;
  __half2* h = reinterpret_cast<__half2*>(&a);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    h[j] = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
    h[4 + j] = __floats2half2_rn(w[2 * j], w[2 * j + 1]);
  }
  stcs256(dst, a);
}

// A slot that a row does not use has a zero in A, and 0 * B is NaN where B is not finite.  Results that
// came out as NaN are formed again from the slots that the row does use: out[j * stride] = the sum over
// the groups [g0, g1) for feature f + j of row ii.  Apart from the main loop, so that it costs no
// registers there.
template <typename OutT>
__device__ __noinline__ void by_slots(const TcArgs& s, int g0, int g1, int ii, int f, OutT* out, int stride) {
  float sum[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sum[j] = 0.f;
  for (int g = g0; g < g1; ++g)
    for (int ji = 0; ji < kG; ++ji) {
      const float av = __half2float(s.a[(static_cast<size_t>(g) * s.t + ii) * kG + ji]);
      if (av == 0.f) continue;
      const __half* br = s.b + static_cast<size_t>(s.indices[static_cast<size_t>(g) * kG + ji]) * s.feat + f;
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[j] = fmaf(av, __half2float(br[j]), sum[j]);
    }
#pragma unroll
  for (int j = 0; j < 8; ++j) out[j * stride] = to_out<OutT>(sum[j]);
}

// acc = the groups [g0, g1) of a tile (MT = tiles of 16 rows; layout of acc: mma16.cuh).  True if a
// result of this lane is a NaN.
template <int MT>
__device__ __forceinline__ bool accumulate(const TcArgs& s, int g0, int g1, int f0, int lane, float (&acc)[MT][8][4]) {
  mma16::clear(acc);
  const int q = lane & 3, r = lane >> 2;
  const bool in = f0 + r * 8 < s.feat;
  const __half* bl = s.b + (in ? f0 + r * 8 : 0);
  auto ids_of = [&](int g) {
    const int32_t* p = s.indices + static_cast<size_t>(g) * kG + q * 4;
    if (s.vec_indices) return ld_global(reinterpret_cast<const int4*>(p));
    return make_int4(ld_global(p), ld_global(p + 1), ld_global(p + 2), ld_global(p + 3));
  };
  auto rows_of = [&](const int4& id, uint4 (&v)[4]) {
    const int row[4] = {id.x, id.y, id.z, id.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = make_uint4(0u, 0u, 0u, 0u);
      if (in) v[k] = ld_global(reinterpret_cast<const uint4*>(bl + static_cast<size_t>(row[k]) * s.feat));
    }
  };
  auto values_of = [&](int g, uint32_t (&av)[MT][4]) {
    const __half* p = s.a + (static_cast<size_t>(g) * s.t + r) * kG + q * 4;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const uint2 lo = ld_global(reinterpret_cast<const uint2*>(p + mt * 16 * kG));
      uint2 hi = make_uint2(0u, 0u);
      if (s.t >= 16) hi = ld_global(reinterpret_cast<const uint2*>(p + (mt * 16 + 8) * kG));
      av[mt][0] = lo.x; av[mt][1] = hi.x; av[mt][2] = lo.y; av[mt][3] = hi.y;
    }
  };
  int4 id0 = make_int4(0, 0, 0, 0), id1 = id0;
  if (g0 < g1) id0 = ids_of(g0);
  if (g0 + 1 < g1) id1 = ids_of(g0 + 1);
  for (int g = g0; g < g1; g += 2) {
    const bool two = g + 1 < g1;
    uint4 v0[4], v1[4];
    uint32_t a0[MT][4], a1[MT][4];
    rows_of(id0, v0);
    if (two) rows_of(id1, v1);
    values_of(g, a0);
    if (two) values_of(g + 1, a1);
    if (g + 2 < g1) id0 = ids_of(g + 2);
    if (g + 3 < g1) id1 = ids_of(g + 3);
    mma16::multiply(acc, v0, a0);
    if (two) mma16::multiply(acc, v1, a1);
  }
  bool nan = false;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) nan |= acc[mt][j][c] != acc[mt][j][c];
  return nan;
}

template <int MT, typename OutT>
__global__ void __launch_bounds__(kThreads, MT == 1 ? 5 : 2)
tcspmm_mma_kernel(const __grid_constant__ TcArgs s) {
  __shared__ float s_sum[4][MT][4][8][32];  // [warp][row tile][c][j][lane]
  __shared__ unsigned s_seen;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slab = static_cast<int>(blockIdx.x) % s.slabs, unit = static_cast<int>(blockIdx.x) / s.slabs;
  const int f0 = slab * mma16::kSlab;
  const int q = lane & 3, r = lane >> 2;
  OutT* c = static_cast<OutT*>(s.c);
  float acc[MT][8][4];
  chain_wait();

  if (unit >= s.windows) {  // ---- a short tile per warp
    const int io = (unit - s.windows) * 4 + warp;
    if (io >= s.mb) return;
    const int g0 = ld_global(s.indptr + io), g1 = ld_global(s.indptr + io + 1);
    if (g1 - g0 > kLight) return;
    const bool nan = accumulate<MT>(s, g0, g1, f0, lane, acc);
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const int ii = mt * 16 + r + (k >> 1) * 8, f = f0 + 2 * q * 8;
        float v[8], w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          v[j] = acc[mt][j][k];
          w[j] = acc[mt][j][k + 1];
        }
        if (ii < s.t) {
          if (s.wide_out) {
            if (f < s.feat) store16(s, c, io, ii, f, v, w);
          } else {
            if (f < s.feat) store8(s, c, io, ii, f, v);
            if (f + 8 < s.feat) store8(s, c, io, ii, f + 8, w);
          }
        }
      }
    if (nan) {
      for (int k = 0; k < 4 * MT; ++k) {
        const int ii = (k >> 2) * 16 + r + (k >> 1 & 1) * 8, f = f0 + (2 * q + (k & 1)) * 8;
        if (ii < s.t && f < s.feat) by_slots(s, g0, g1, ii, f, c + (static_cast<size_t>(io) * s.t + ii) * s.feat + f, 1);
      }
    }
    return;
  }

  // ---- a window: the long tiles that reach into it, one after the other
  const int w0 = unit << s.window_log, w1 = w0 + min(1 << s.window_log, s.nnzb - w0);
  int cur = warp_row_of(s.indptr, s.mb, w0, s.tiles_per_group, lane);
  while (cur < s.mb) {
    const int start = ld_global(s.indptr + min(cur + lane, s.mb)), end = ld_global(s.indptr + min(cur + lane + 1, s.mb));
    unsigned todo = __ballot_sync(0xffffffffu, end - start > kLight && start < w1 && end > w0);
    while (todo != 0u) {  // the same in all four warps
      const int k = __ffs(todo) - 1;
      todo &= todo - 1u;
      const int io = cur + k;
      const int g0 = __shfl_sync(0xffffffffu, start, k), g1 = __shfl_sync(0xffffffffu, end, k);
      const int p0 = max(g0, w0), p1 = min(g1, w1), per = (p1 - p0 + 3) / 4;
      const int q0 = min(p1, p0 + warp * per), q1 = min(p1, q0 + per);
      const bool nan = accumulate<MT>(s, q0, q1, f0, lane, acc);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
#pragma unroll
          for (int j = 0; j < 8; ++j) s_sum[warp][mt][cc][j][lane] = acc[mt][j][cc];
      if (nan) {
        for (int k = 0; k < 4 * MT; ++k) {
          const int ii = (k >> 2) * 16 + r + (k >> 1 & 1) * 8, f = f0 + (2 * q + (k & 1)) * 8;
          if (ii < s.t && f < s.feat) by_slots(s, q0, q1, ii, f, &s_sum[warp][k >> 2][k & 3][0][lane], 32);
        }
      }
      __syncthreads();
      // warp w finishes the pieces c = w: row (lane/4 + 8 (w/2)), 8 features
      const int e0 = g0 >> s.window_log, e1 = (g1 - 1) >> s.window_log;
      float v[MT][8];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[mt][j] = (s_sum[0][mt][warp][j][lane] + s_sum[1][mt][warp][j][lane]) +
                     (s_sum[2][mt][warp][j][lane] + s_sum[3][mt][warp][j][lane]);
      bool mine = true;
      if (e0 != e1) {
        // a piece: 8 floats per (row tile, warp, lane), the layout of v
        auto piece = [&](int e, int mt) {
          const size_t slot = (static_cast<size_t>(2 * e + (e == e0 ? 1 : 0)) * s.slabs + slab) * MT + mt;
          return reinterpret_cast<float4*>(s.part) + (slot * kThreads + threadIdx.x) * 2;
        };
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          __stcg(piece(unit, mt), make_float4(v[mt][0], v[mt][1], v[mt][2], v[mt][3]));
          __stcg(piece(unit, mt) + 1, make_float4(v[mt][4], v[mt][5], v[mt][6], v[mt][7]));
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
          unsigned* counter = s.counters + static_cast<size_t>(e0) * s.slabs + slab;
          s_seen = atomicAdd(counter, 1u);
          if (s_seen == static_cast<unsigned>(e1 - e0)) *counter = 0u;  // last piece to arrive
        }
        __syncthreads();
        mine = s_seen == static_cast<unsigned>(e1 - e0);
        if (mine) {
          __threadfence();
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[mt][j] = 0.f;
#pragma unroll 4
            for (int e = e0; e <= e1; ++e) {
              const float4 x = __ldcg(piece(e, mt)), y = __ldcg(piece(e, mt) + 1);
              v[mt][0] += x.x; v[mt][1] += x.y; v[mt][2] += x.z; v[mt][3] += x.w;
              v[mt][4] += y.x; v[mt][5] += y.y; v[mt][6] += y.z; v[mt][7] += y.w;
            }
          }
        }
      }
      if (mine) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int ii = mt * 16 + r + (warp >> 1) * 8, f = f0 + (2 * q + (warp & 1)) * 8;
          if (ii < s.t && f < s.feat) store8(s, c, io, ii, f, v[mt]);
        }
      }
      __syncthreads();  // the meeting place is free for the next tile
    }
    const int last = __shfl_sync(0xffffffffu, end, 31);
    if (last >= w1) break;
    // 32 tiles on; over a run of empty tiles with a search
    const bool empty = last == __shfl_sync(0xffffffffu, start, 0);
    const int next = empty ? warp_row_of(s.indptr, s.mb, last, s.tiles_per_group, lane) : 0;
    cur = max(cur + 32, next);
  }
}

// CUDA-core form for every other shape: a block per row tile; a thread owns output elements
// (ii, f) and walks the groups.
template <typename OutT>
__global__ void __launch_bounds__(256)
tcspmm_simt_kernel(const __half* __restrict__ a, const __half* __restrict__ b, OutT* __restrict__ c,
                   const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices, int t,
                   int g, int feat) {
  const int io = blockIdx.x;
  const int g0 = __ldg(indptr + io), g1 = __ldg(indptr + io + 1);
  for (int e = threadIdx.x; e < t * feat; e += blockDim.x) {
    const int ii = e / feat, f = e % feat;
    float acc = 0.f;
    for (int jo = g0; jo < g1; ++jo) {
      const __half* ar = a + (static_cast<size_t>(jo) * t + ii) * g;
      const int32_t* ix = indices + static_cast<size_t>(jo) * g;
      for (int ji = 0; ji < g; ++ji) {
        const float av = __half2float(__ldg(ar + ji));
        if (av != 0.f) acc = fmaf(av, __half2float(__ldg(b + static_cast<size_t>(__ldg(ix + ji)) * feat + f)), acc);
      }
    }
    c[(static_cast<size_t>(io) * t + ii) * feat + f] = to_out<OutT>(acc);
  }
}

struct TcPlan {
  int slabs, window_log, windows;
  size_t part_bytes, counter_bytes;
};

TcPlan tc_plan(int nnzb, int t, int feat) {
  TcPlan p;
  p.slabs = ceil_div(feat, mma16::kSlab);
  // Windows of 128 groups keep the scratch small; down to 32 where there would not be enough blocks
  // (20 k rows, 6,118 groups, F = 64: 12.4 against 18.9 us).
  p.window_log = 5;
  while (p.window_log < 7 && (static_cast<long long>(nnzb) * p.slabs >> p.window_log) > 4 * kNumSMs) ++p.window_log;
  p.windows = ceil_div(nnzb, 1 << p.window_log);
  // Longer windows where the pieces would take more than 64 MB (there are thousands of blocks by then): with
  // windows of 128 groups they grow with the matrix, at 512 features to the size of its values.
  const size_t window_bytes = 2 * static_cast<size_t>(p.slabs) * (t > 16 ? 2 : 1) * kThreads * 8 * sizeof(float);
  while (p.windows > 1 && p.windows * window_bytes > (size_t{64} << 20)) p.windows = ceil_div(nnzb, 1 << ++p.window_log);
  p.part_bytes = p.windows * window_bytes;
  p.counter_bytes = static_cast<size_t>(std::max(p.windows, 1)) * p.slabs * sizeof(unsigned);
  return p;
}

template <int MT, typename OutT>
int launch_mma(TcArgs s, int device_id, cudaStream_t st) {
  const TcPlan p = tc_plan(s.nnzb, s.t, s.feat);
  s.slabs = p.slabs;
  s.window_log = p.window_log;
  s.windows = p.windows;
  s.tiles_per_group = s.nnzb > 0 ? static_cast<float>(s.mb) / static_cast<float>(s.nnzb) : 0.f;
  const long long blocks = (static_cast<long long>(s.windows) + ceil_div(s.mb, 4)) * s.slabs;
  if (blocks > INT32_MAX) return fail("sparsetir_tcspmm: too many thread blocks");
  CallScratch cs;
  if (take_scratch(device_id, st, p.part_bytes, p.counter_bytes, &cs) != 0) return -1;
  s.part = reinterpret_cast<float*>(cs.scratch);
  s.counters = cs.counters;
  launch_chained(tcspmm_mma_kernel<MT, OutT>, static_cast<unsigned>(blocks), kThreads, 0, st, s);
  SPTIR_LAUNCH_OK("tcspmm_mma_kernel");
  return return_scratch(cs, st);
}

// Whether the operands' shape, alignment aside, is one that the matrix instruction takes.
inline bool mma_shape(int t, int g, int feat) { return g == kG && (t == 8 || t == 16 || t == 32) && feat % 8 == 0; }

template <typename OutT>
int launch_all(const __half* a, const __half* b, OutT* c, const int32_t* indptr, const int32_t* indices,
               int mb, int nnzb, int t, int g, int feat, int device_id, cudaStream_t st) {
  if (mma_shape(t, g, feat) && aligned16(a) && aligned16(b)) {
    const TcArgs s{a, b, c, indptr, indices, nullptr, nullptr, mb, nnzb, t, feat, 0, 0, 0, 0.f, aligned16(indices), aligned16(c),
                   feat % 16 == 0 && aligned32(c)};
    if (t == 32) return launch_mma<2, OutT>(s, device_id, st);
    return launch_mma<1, OutT>(s, device_id, st);
  }
  tcspmm_simt_kernel<OutT><<<mb, 256, 0, st>>>(a, b, c, indptr, indices, t, g, feat);
  SPTIR_LAUNCH_OK("tcspmm_simt_kernel");
  return 0;
}

}  // namespace
}  // namespace sptir

extern "C" int sparsetir_tcspmm_workspace(int nnzb, int feat, int tile_size, int group_size, size_t* scratch_bytes,
                                          size_t* counter_bytes) {
  using namespace sptir;
  if (nnzb < 0 || feat < 0 || tile_size < 1 || group_size < 1 || !scratch_bytes || !counter_bytes)
    return fail("sparsetir_tcspmm_workspace: bad argument");
  *scratch_bytes = *counter_bytes = 0;
  if (feat == 0 || !mma_shape(tile_size, group_size, feat)) return 0;
  const TcPlan p = tc_plan(nnzb, tile_size, feat);
  *scratch_bytes = p.part_bytes;
  *counter_bytes = p.counter_bytes;
  return 0;
}

extern "C" int sparsetir_tcspmm_raw(const void* a_f16, const void* b_f16, void* c, int c_is_f16,
                                    const int32_t* indptr, const int32_t* indices, int mb, int nb,
                                    int nnzb, int feat, int tile_size, int group_size, int device_id,
                                    void* stream) {
  using namespace sptir;
  (void)nb;
  if (mb < 0 || nnzb < 0 || feat < 0 || tile_size < 1 || group_size < 1)
    return fail("sparsetir_tcspmm: invalid size");
  if (mb == 0 || feat == 0) return 0;
  if (!c || !indptr || (nnzb > 0 && (!a_f16 || !b_f16 || !indices)))
    return fail("sparsetir_tcspmm: null pointer argument");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* a = static_cast<const __half*>(a_f16);
  const __half* b = static_cast<const __half*>(b_f16);
  if (c_is_f16)
    return launch_all<__half>(a, b, static_cast<__half*>(c), indptr, indices, mb, nnzb, tile_size, group_size, feat,
                              device_id, st);
  return launch_all<float>(a, b, static_cast<float*>(c), indptr, indices, mb, nnzb, tile_size, group_size, feat,
                           device_id, st);
}

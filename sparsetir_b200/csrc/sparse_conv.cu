// Sparse convolution with the neighbour map of a layer laid out once, fp16 operands, fp32 sums:
//   Y[d, :] (+)= sum over kernel offsets r with a pair (s, d):  X[s, :] * W[r, :, :]
// for layers in which an (offset, output) pair never repeats (examples/sparse_conv of the
// reference: examples/rgms/sparse_conv/sparse_conv.py:93-125).  map holds, for tiles of 128 outputs,
// map[(tile * R + r) * 128 + t] = s, or -1 where output tile * 128 + t has no pair of offset r.
//
// The product is one GEMM per tile with K = R * feat_in: row t of the left operand is the
// concatenation of the X rows of its pairs (zeros where there is none), the right operand is W as
// it lies in memory.  A persistent block per SM walks the tiles, one at a time or two side by side (TPS); per
// 64-wide slice of K
//  - six groups of four warps fetch the left operand with 16-byte asynchronous copies into the
//    swizzled stage (a slice may straddle offsets, so channel counts that are not multiples of 64
//    waste nothing; a missing pair is a copy of no bytes, which fills in zeros);
//  - one thread brings the slice of W with TMA, one issues the MMAs into one of two accumulators;
//  - four warps take finished tiles out of TMEM and write (or add to) Y, each row once.
//
// No unit is at its limit (100,000 points, 27 offsets, 64 -> 128, counters of one launch: tensor pipe 39 %, L1 data pipe
// 47 %, issue slots 35 %, L2 25 %, DRAM 5 % of the elapsed time): a step of the ring costs the gathering warps'
// instructions and their waits for map entries and stages, whatever the share of pairs (64 -> 32: a layer with 2 % of
// them takes as long as one with 95 %).  What was cut is therefore instructions and what passes the data pipe: no divisions in the loops and MMAs from an elected thread 97 -> 64 us (64 ->
// 128), asynchronous copies instead of loads and stores 64 -> 58; then (us, 64 -> 128 / 64 -> 32, 54.7 / 48.6 before) one
// slice of W for two tiles and copies that arrive at the stage's barrier themselves, 51.5 / 44.2, the copies of a step
// written out, 50.3 / 41.2, an epilogue of a third of the instructions, 47.2 / 39.7.  Rows loaded into registers and
// stored took 54.9, gathering by TMA (four rows per copy) 215 us.  The map replaces one built, checked and cleared on
// every call: together with the cleared Y that took 37 us of 122.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.h"
#include "launch.cuh"
#include "tc05.cuh"
#include "tmap.h"
#include "vec.cuh"

namespace sptir {
namespace {

constexpr int kTM = 128;                // outputs per tile
constexpr int kKC = 64;                 // slice of K per stage: one 128-byte swizzled row
constexpr int kZBytes = kTM * kKC * 2;  // 16 KB
constexpr int kWBox = kKC * 64 * 2;     // 8 KB: 64 rows of K x 64 outputs
constexpr int kMaxOut = 256;
constexpr int kMaxStages = 8;
constexpr int kGroups = 6;              // gather groups of four warps
constexpr int kFirstGather = 8;         // warp 0 loads W, 1 issues MMAs, 4-7 epilogue, 8-31 gather
constexpr int kThreads = (kFirstGather + 4 * kGroups) * 32;
constexpr int kOutStride = 128 + 16;    // padded row of 32 floats: rows spread over all banks
constexpr int kOutBytes = kTM * kOutStride;
// byte offset of 16-byte piece q of a row of 32 halves: unpadded rows, whose pieces are exchanged so that eight rows
// written at once, or two read, touch every bank once
__device__ __forceinline__ int half_piece(int row, int q) { return row * 64 + ((q ^ ((row >> 1) & 3)) << 4); }
constexpr int kSmemLimit = 226 * 1024;  // dynamic part: the static barriers count against the 227 KB too

__device__ unsigned int g_conv_timeouts = 0;

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc05::smem_u32(bar)) : "memory");
}

// 32 columns of a lane's row of a finished tile go to the warp's part of the staging buffer, rounded to the result's type.
// True if a value may be a NaN: 0 * v is one for every v that is not finite.  (A comparison per value is twice
// the instructions, and the epilogue's instructions share the issue slots with those of the gathering warps.)
__device__ __forceinline__ bool stage32(const float*, unsigned char* wbase, int lane, const uint32_t (&r)[32]) {
  unsigned long long t[2] = {0ull, 0ull};
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    *reinterpret_cast<uint4*>(wbase + lane * kOutStride + q * 16) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const unsigned long long v = static_cast<unsigned long long>(r[4 * q + 2 * j + 1]) << 32 | r[4 * q + 2 * j];
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t[j]) : "l"(v), "l"(0ull));
    }
  }
  float lo, hi, lo2, hi2;
  unpack_pair(t[0], lo, hi);
  unpack_pair(t[1], lo2, hi2);
  const float any = (lo + hi) + (lo2 + hi2);
  return any != any;
}
__device__ __forceinline__ bool stage32(const __half*, unsigned char* wbase, int lane, const uint32_t (&r)[32]) {
  const __half2 zero = __floats2half2_rn(0.f, 0.f);
  __half2 t[2] = {zero, zero};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 o;
    __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      h[j] = __floats2half2_rn(__uint_as_float(r[8 * q + 2 * j]), __uint_as_float(r[8 * q + 2 * j + 1]));
      t[j & 1] = __hfma2(h[j], zero, t[j & 1]);
    }
    *reinterpret_cast<uint4*>(wbase + half_piece(lane, q)) = o;
  }
  const __half2 any = __hadd2(t[0], t[1]);
  return __hisnan(__low2half(any)) || __hisnan(__high2half(any));
}
__device__ __forceinline__ void stage1(const float*, unsigned char* wbase, int row, int col, float v) {
  *reinterpret_cast<float*>(wbase + row * kOutStride + col * 4) = v;
}
__device__ __forceinline__ void stage1(const __half*, unsigned char* wbase, int row, int col, float v) {
  *reinterpret_cast<__half*>(wbase + half_piece(row, col >> 3) + (col & 7) * 2) = __float2half_rn(v);
}

// The warp's 32 staged rows go to Y with whole 128-byte (fp32) or 64-byte (fp16) row pieces; y points at the first of
// the 32 columns in the warp's first row.  With `add` all old values are read before the first store.
__device__ __forceinline__ void write32(float* y, const unsigned char* wbase, int nrows, int feat_out, int lane, bool add) {
  const unsigned char* from = wbase + (lane >> 3) * kOutStride + (lane & 7) * 16;
  float4* to = reinterpret_cast<float4*>(y + static_cast<size_t>(lane >> 3) * feat_out) + (lane & 7);
  const size_t step = static_cast<size_t>(feat_out);  // four rows, in 16-byte pieces
  if (!add) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (4 * i + (lane >> 3) < nrows) __stcs(to + i * step, *reinterpret_cast<const float4*>(from + 4 * i * kOutStride));
    return;
  }
  float4 old[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (4 * i + (lane >> 3) < nrows) old[i] = __ldcs(to + i * step);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (4 * i + (lane >> 3) < nrows) {
      const float4 v = *reinterpret_cast<const float4*>(from + 4 * i * kOutStride);
      __stcs(to + i * step, make_float4(old[i].x + v.x, old[i].y + v.y, old[i].z + v.z, old[i].w + v.w));
    }
  }
}
__device__ __forceinline__ void write32(__half* y, const unsigned char* wbase, int nrows, int feat_out, int lane, bool add) {
  const unsigned char* from = wbase + half_piece(lane >> 2, lane & 3);  // rows 8 apart have their pieces in the same order
  uint4* to = reinterpret_cast<uint4*>(y + static_cast<size_t>(lane >> 2) * feat_out) + (lane & 3);
  const size_t step = static_cast<size_t>(feat_out);  // eight rows, in 16-byte pieces
  if (!add) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (8 * i + (lane >> 2) < nrows) __stcs(to + i * step, *reinterpret_cast<const uint4*>(from + 8 * i * 64));
    return;
  }
  uint4 old[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    old[i] = make_uint4(0u, 0u, 0u, 0u);
    if (8 * i + (lane >> 2) < nrows) old[i] = __ldcs(to + i * step);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (8 * i + (lane >> 2) < nrows) {
      const uint4 v = *reinterpret_cast<const uint4*>(from + 8 * i * 64);
      const __half2* vh = reinterpret_cast<const __half2*>(&v);
      uint4 o = old[i];
      __half2* h = reinterpret_cast<__half2*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = __hadd2(h[j], vh[j]);
      __stcs(to + i * step, o);
    }
  }
}

// One row's 32 outputs from its pairs alone, lane = output.  A row without a pair of some offset takes
// part in that offset's product with zeros, and 0 * W is NaN where W is not finite: rows that came
// out with a NaN are formed again here, from the terms of the sum and no others.
__device__ __noinline__ float row_by_pairs(const __half* x, const __half* w,
                                           const int32_t* entries, int num_rels, int feat_in,
                                           int feat_out, int col) {
  float sum = 0.f;
  for (int rel = 0; rel < num_rels; ++rel) {
    const int e = ld_global(entries + static_cast<size_t>(rel) * kTM);
    if (e < 0) continue;
    const __half* xr = x + static_cast<size_t>(e) * feat_in;
    const __half* wr = w + static_cast<size_t>(rel) * feat_in * feat_out + col;
#pragma unroll 8
    for (int fi = 0; fi < feat_in; ++fi)
      sum = fmaf(__half2float(ld_global(xr + fi)), __half2float(ld_global(wr + static_cast<size_t>(fi) * feat_out)), sum);
  }
  return sum;
}

// Eight rows' pieces of 16 bytes into shared memory: row i from xb + from[i] * row_bytes to at0 (even i) or at1 (odd i)
// + i / 2 * 1024; zeros where from[i] is negative, or everywhere with `skip`.  One statement, written out: what a
// step costs is the instructions of the gathering warps, and the selects and addresses that the compiler made of the
// same loop were more: 16 instructions a step and warp were 4 us of 45 (100,000 points, 27 offsets, 64 -> 32).
__device__ __forceinline__ void copy_rows(uint32_t at0, uint32_t at1, const int (&from)[8], uint32_t row_bytes, const char* xb, int skip) {
#define SPTIR_COPY_ROW(E, AT, OFF)              \
  "setp.lt.or.s32 p, " E ", 0, q;\n\t"          \
  "max.s32 f, " E ", 0;\n\t"                    \
  "mad.wide.u32 a, f, %10, %11;\n\t"            \
  "cp.async.cg.shared.global [" AT "+" OFF "], [a], 16, p;\n\t"
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 a;\n\t.reg .b32 f;\n\t"
      "setp.ne.s32 q, %12, 0;\n\t"
      SPTIR_COPY_ROW("%2", "%0", "0") SPTIR_COPY_ROW("%3", "%1", "0")
      SPTIR_COPY_ROW("%4", "%0", "1024") SPTIR_COPY_ROW("%5", "%1", "1024")
      SPTIR_COPY_ROW("%6", "%0", "2048") SPTIR_COPY_ROW("%7", "%1", "2048")
      SPTIR_COPY_ROW("%8", "%0", "3072") SPTIR_COPY_ROW("%9", "%1", "3072")
      "}"
      ::"r"(at0), "r"(at1), "r"(from[0]), "r"(from[1]), "r"(from[2]), "r"(from[3]), "r"(from[4]), "r"(from[5]), "r"(from[6]),
        "r"(from[7]), "r"(row_bytes), "l"(xb), "r"(skip)
      : "memory");
#undef SPTIR_COPY_ROW
}

template <typename OutT, int TPS>
__global__ void __launch_bounds__(kThreads, 1)
sparse_conv_kernel(const __grid_constant__ CUtensorMap tm_w, OutT* __restrict__ y, const __half* x,
                   const __half* w, const int32_t* map, int m, int num_rels, int feat_in,
                   int feat_out, int tmem_cols, int acc_cols, int nstages, int slots, int add) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];   // both operands of the stage are there
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];  // the tensor core has read the stage
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* base = smem_raw + ((1024u - (tc05::smem_u32(smem_raw) & 1023u)) & 1023u);
  const int nwb = (feat_out + 63) / 64;
  const int stride = TPS * kZBytes + nwb * kWBox;
  const int ktotal = num_rels * feat_in;
  const int steps = (ktotal + kKC - 1) / kKC;  // stages per unit of TPS tiles
  const int ntiles = (m + kTM - 1) / kTM;
  // tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the grid never exceeds the number of tiles
  const int my_tiles = (ntiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);

  const int units = (my_tiles + TPS - 1) / TPS;  // the last one may be a tile short

  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < nstages; ++s) {
        tc05::mbar_init(&bar_full[s], 1 + 128 * TPS);  // W, and the threads of a gather group per tile
        tc05::mbar_init(&bar_empty[s], 1);
      }
      for (int b = 0; b < 2; ++b) {
        tc05::mbar_init(&bar_acc_full[b], 1);
        tc05::mbar_init(&bar_acc_empty[b], 4);
      }
      tc05::fence_mbar_init();
      tc05::prefetch_tensormap(&tm_w);
    }
    __syncwarp();
    tc05::tmem_alloc(&s_tmem, tmem_cols);
  }
  chain_wait();
  tc05::fence_before_sync();
  __syncthreads();
  chain_trigger();
  tc05::fence_after_sync();
  const uint32_t tmem = s_tmem;
  bool ok = true;
  int armed = 0;

  if (warp == 0) {
    // ---- W: rows [64 s, 64 s + 64) of the (R * feat_in) x feat_out array; past its end zeros
    if (tc05::elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      unsigned char* st = base + TPS * kZBytes;
      for (int u = 0; u < units && ok; ++u) {
        for (int sidx = 0; sidx < steps; ++sidx) {
          if (!tc05::mbar_wait(&bar_empty[s], phase ^ 1u)) { ok = false; break; }
          tc05::mbar_arrive_expect_tx(&bar_full[s], nwb * kWBox);
          for (int j = 0; j < nwb; ++j) tc05::tma_load_2d(st + j * kWBox, &tm_w, j * 64, sidx * kKC, &bar_full[s]);
          ++armed;
          st += stride;
          if (++s == nstages) { s = 0; phase ^= 1u; st = base + TPS * kZBytes; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMAs: M = 128 outputs, N = feat_out, K = 16 per instruction
    if (tc05::elect_one()) {
      const uint32_t idesc = tc05::instr_desc(tc05::kFmtF16, kTM, feat_out, /*a_mn=*/0, /*b_mn=*/1);
      const uint64_t dz0 = tc05::smem_desc_swizzled(tc05::smem_u32(base), 0, 1024, tc05::kSwizzle128B);
      const uint64_t dw0 = tc05::smem_desc_swizzled(tc05::smem_u32(base) + TPS * kZBytes, kWBox, 1024, tc05::kSwizzle128B);
      const int last = (ktotal - (steps - 1) * kKC) / 16;  // instructions of the last slice
      int s = 0;
      uint32_t phase = 0;
      uint64_t dz = dz0, dw = dw0;
      for (int u = 0; u < units && ok; ++u) {
        const int buf = u & 1, buse = u >> 1;
        const bool both = TPS == 2 && u * TPS + 1 < my_tiles;
        if (!tc05::mbar_wait(&bar_acc_empty[buf], (buse & 1) ^ 1)) { ok = false; break; }
        const uint32_t acc = tmem + buf * (TPS * acc_cols);
        for (int sidx = 0; sidx < steps; ++sidx) {
          if (!tc05::mbar_wait(&bar_full[s], phase)) { ok = false; break; }
          // the rows come by cp.async, whose writes the barrier has made visible to this thread: on to the
          // proxy that the tensor core reads through
          tc05::fence_async_smem();
          tc05::fence_after_sync();
          const int ksteps = sidx + 1 < steps ? kKC / 16 : last;
#pragma unroll
          for (int ks = 0; ks < kKC / 16; ++ks)
            if (ks < ksteps)
              tc05::mma_f16(acc, tc05::desc_advance(dz, ks * 32), tc05::desc_advance(dw, ks * 2048), idesc,
                            (sidx > 0 || ks > 0) ? 1u : 0u);
          if (both) {
#pragma unroll
            for (int ks = 0; ks < kKC / 16; ++ks)
              if (ks < ksteps)
                tc05::mma_f16(acc + acc_cols, tc05::desc_advance(dz, kZBytes + ks * 32), tc05::desc_advance(dw, ks * 2048), idesc,
                              (sidx > 0 || ks > 0) ? 1u : 0u);
          }
          tc05::mma_commit(&bar_empty[s]);
          dz = tc05::desc_advance(dz, stride);
          dw = tc05::desc_advance(dw, stride);
          if (++s == nstages) { s = 0; phase ^= 1u; dz = dz0; dw = dw0; }
        }
        if (!ok) break;
        tc05::mma_commit(&bar_acc_full[buf]);
      }
    }
  } else if (warp >= kFirstGather) {
    // ---- gather: group g fills tile g % TPS of the steps g / TPS, g / TPS + slots, ...; warp gw of it rows
    // gw * 32 .. gw * 32 + 31 of the tile, eight lanes per row.  Nobody waits for the copies: they arrive at the
    // stage's barrier themselves.  No more slots than stages: the group that passes the wait of step n knows that the
    // tensor core is past step n - nstages, and may wait for the stage of step n + slots only if that puts it at most
    // one phase of the stage's barrier behind.  The map entries of a group's next step are requested before this
    // step's rows are copied.
    //
    // (offset, piece) of the lane move by whole rows of the ring: quotients and remainders are formed once.
    const int g = (warp - kFirstGather) >> 2, gw = (warp - kFirstGather) & 3;
    const int half = g % TPS, slot = g / TPS;
    const int cpr = feat_in / 8;  // 16-byte pieces per X row
    const uint32_t row_bytes = static_cast<uint32_t>(feat_in) * 2u;
    const int chunk = lane & 7;
    const int step_rel = slots * 8 / cpr, step_off = slots * 8 - step_rel * cpr;
    const int unit_rel = steps * 8 / cpr, unit_off = steps * 8 - unit_rel * cpr;
    int sidx = slot, rel = (slot * 8 + chunk) / cpr, off = slot * 8 + chunk - rel * cpr;
    int left = my_tiles;  // tiles from the unit of this step on
    const size_t tile_map = static_cast<size_t>(num_rels) * kTM;
    const int32_t* mp = map + (blockIdx.x + static_cast<size_t>(half) * gridDim.x) * tile_map + gw * 32 + (lane >> 3);
    auto into_unit = [&]() {  // steps past the end of a unit belong to the block's next ones
      while (left > 0 && sidx >= steps) {
        sidx -= steps;
        left -= TPS;
        mp += tile_map * (TPS * gridDim.x);
        rel -= unit_rel;
        off -= unit_off;
        if (off < 0) { off += cpr; --rel; }
      }
    };
    int entry[8];     // of the next step, as they come: looked at a step later, so that nobody waits for them here
    int none = 0;     // not 0: the next step has none for this lane
    auto entries_of_step = [&]() {
      const bool in = left > half && rel < num_rels;
      none = in ? 0 : 1;
      const int32_t* e = in ? mp + static_cast<size_t>(rel) * kTM : map;
#pragma unroll
      for (int i = 0; i < 8; ++i) entry[i] = ld_global(e + 4 * i);
    };
    // the lane's rows of the tile are 4 apart: two places in an atom of 8 swizzled rows, atoms 1024 bytes apart
    const int r4 = lane >> 3;
    const uint32_t at0 = tc05::smem_u32(base) + half * kZBytes + gw * 4096 + r4 * 128 + ((chunk ^ r4) << 4);
    const uint32_t at1 = tc05::smem_u32(base) + half * kZBytes + gw * 4096 + (4 + r4) * 128 + ((chunk ^ (4 + r4)) << 4);
    int s = slot;
    uint32_t phase = 0, stage = slot * stride;
    if (slot < slots) into_unit();
    if (slot < slots && left > 0) entries_of_step();
    while (slot < slots && left > 0) {
      const char* xb = reinterpret_cast<const char*>(x) + off * 16;
      const bool tile_there = left > half;
      const int skip = none;
      int from[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) from[i] = entry[i];
      sidx += slots;
      rel += step_rel;
      off += step_off;
      if (off >= cpr) { off -= cpr; ++rel; }
      into_unit();
      if (left > 0) entries_of_step();
      if (!tc05::mbar_wait(&bar_empty[s], phase ^ 1u)) { ok = false; break; }
      if (tile_there) copy_rows(at0 + stage, at1 + stage, from, row_bytes, xb, skip);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc05::smem_u32(&bar_full[s])) : "memory");
      s += slots;
      stage += slots * stride;
      if (s >= nstages) { s -= nstages; stage -= nstages * stride; phase ^= 1u; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // also when giving up: nothing may land later
  } else if (warp >= 4) {
    // ---- epilogue: thread = tile row = TMEM lane, 32 columns at a time
    unsigned char* wbase = base + nstages * stride + (warp & 3) * 32 * kOutStride;
    for (int u = 0; u < units && ok; ++u) {
      const int buf = u & 1, buse = u >> 1;
      if (!tc05::mbar_wait(&bar_acc_full[buf], buse & 1)) { ok = false; break; }
      tc05::fence_after_sync();
#pragma unroll 1
      for (int h = 0; h < TPS && u * TPS + h < my_tiles; ++h) {
        const int tile = static_cast<int>(blockIdx.x) + (u * TPS + h) * static_cast<int>(gridDim.x);
        const int row_base = tile * kTM + (warp & 3) * 32;
        const int nrows = min(32, m - row_base);  // live rows among the warp's 32 (may be <= 0)
        const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (buf * TPS + h) * acc_cols;
        for (int c0 = 0; c0 < feat_out; c0 += 32) {
          uint32_t r[32];
          tc05::tmem_ld32(taddr + c0, r);
          if (c0 + 32 >= feat_out && (h == TPS - 1 || u * TPS + h + 1 == my_tiles)) {
            // the unit's results are in registers: a later one may overwrite its accumulators
            tc05::fence_before_sync();
            __syncwarp();
            if (lane == 0) arrive(&bar_acc_empty[buf]);
          }
          __syncwarp();  // the warp's reads of the previous 32 columns are over
          bool nan = stage32(y, wbase, lane, r);
          __syncwarp();
          if (nan) {
            nan = false;
#pragma unroll
            for (int q = 0; q < 32; ++q) nan |= __uint_as_float(r[q]) != __uint_as_float(r[q]);
          }
          for (unsigned todo = __ballot_sync(0xffffffffu, nan && lane < nrows); todo != 0u; todo &= todo - 1u) {
            const int lr = __ffs(todo) - 1;
            const int32_t* entries = map + static_cast<size_t>(tile) * num_rels * kTM + (warp & 3) * 32 + lr;
            stage1(y, wbase, lr, lane, row_by_pairs(x, w, entries, num_rels, feat_in, feat_out, c0 + lane));
            __syncwarp();
          }
          write32(y + static_cast<size_t>(row_base) * feat_out + c0, wbase, nrows, feat_out, lane, add != 0);
        }
      }
    }
  }

  const bool all_ok = !__syncthreads_or(!ok);
  if (!all_ok) {
    if (tid == 0) atomicAdd(&g_conv_timeouts, 1u);
    // gave up: the loading thread lets the loads it has issued land (bounded) before the block's memory is released
    for (int it = max(0, armed - nstages); it < armed; ++it)
      tc05::mbar_wait(&bar_full[it % nstages], (it / nstages) & 1);
  }
  tc05::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc05::tmem_dealloc(tmem, tmem_cols);
}

template <typename OutT, int TPS>
int launch_units(const CUtensorMap& tm_w, OutT* y, const __half* x, const __half* w, const int32_t* map, int m, int num_rels,
                 int feat_in, int feat_out, int add, cudaStream_t st) {
  static thread_local int configured_device = -1;
  int dev = 0;
  SPTIR_CUDA_OK(cudaGetDevice(&dev));
  if (configured_device != dev) {
    SPTIR_CUDA_OK(cudaFuncSetAttribute(sparse_conv_kernel<OutT, TPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    configured_device = dev;
  }
  const int stride = TPS * kZBytes + ceil_div(feat_out, 64) * kWBox;
  const int nstages = std::min(kMaxStages, (kSmemLimit - kOutBytes - 1024) / stride);
  const int smem = nstages * stride + kOutBytes + 1024;
  const int acc_cols = (feat_out + 31) & ~31;
  int tmem_cols = 32;
  while (tmem_cols < 2 * TPS * acc_cols) tmem_cols *= 2;
  const int grid = std::min(ceil_div(m, kTM), kNumSMs);
  launch_chained(sparse_conv_kernel<OutT, TPS>, grid, kThreads, smem, st, tm_w, y, x, w, map, m, num_rels, feat_in, feat_out,
                 tmem_cols, acc_cols, nstages, std::min(kGroups / TPS, nstages), add);
  SPTIR_LAUNCH_OK("sparse_conv_kernel");
  return 0;
}

template <typename OutT>
int launch(const CUtensorMap& tm_w, OutT* y, const __half* x, const __half* w, const int32_t* map, int m, int num_rels, int feat_in,
           int feat_out, int add, cudaStream_t st) {
  // Two tiles side by side, where blocks have more than one and the accumulators fit twice: one slice of W and one round
  // of the ring for 256 outputs (us, one / two, 27 offsets: 100,000 points 64 -> 32 43.7 / 37.9, 64 -> 128 50.4 / 47.0,
  // 22,000 points 128 -> 64 31.0 / 28.3; 8 offsets, 40,000 points: 64 -> 64 11.6 / 11.7, 128 -> 128 18.5 / 18.2).
  if (feat_out <= kMaxOut / 2 && m > kNumSMs * kTM)
    return launch_units<OutT, 2>(tm_w, y, x, w, map, m, num_rels, feat_in, feat_out, add, st);
  return launch_units<OutT, 1>(tm_w, y, x, w, map, m, num_rels, feat_in, feat_out, add, st);
}

}  // namespace

int conv_timeouts(unsigned int* count) {
  SPTIR_CUDA_OK(cudaMemcpyFromSymbol(count, g_conv_timeouts, sizeof(unsigned int)));
  return 0;
}

}  // namespace sptir

extern "C" int sparsetir_sparse_conv_f16_raw(const void* w, const void* x, void* y, int y_is_f16, const int32_t* map,
                                             int m, int n, int num_rels, int feat_in, int feat_out, int add,
                                             int device_id, void* stream) {
  using namespace sptir;
  if (m < 0 || n < 0 || num_rels < 0 || feat_in < 0 || feat_out < 0)
    return fail("sparsetir_sparse_conv_f16: negative size");
  if (feat_in == 0 || feat_in % 16 != 0 || feat_out == 0 || feat_out % 32 != 0 || feat_out > kMaxOut)
    return fail("sparsetir_sparse_conv_f16: feat_in must be a multiple of 16 and feat_out a multiple of 32 up to %d "
                "(use sparsetir_rgms_ell3d_f16)", kMaxOut);
  if (static_cast<long long>(num_rels) * feat_in > INT32_MAX / 64 || num_rels == 0)
    return fail("sparsetir_sparse_conv_f16: %d kernel offsets", num_rels);
  if (m == 0) return 0;
  if (!w || !x || !y || !map) return fail("sparsetir_sparse_conv_f16: null pointer argument");
  if (!aligned16(w) || !aligned16(x) || !aligned16(y))
    return fail("sparsetir_sparse_conv_f16: w, x and y must be 16-byte aligned (use sparsetir_rgms_ell3d_f16)");
  const long long steps = static_cast<long long>(ceil_div(m, kTM)) / std::min(ceil_div(m, kTM), kNumSMs) + 1;
  if (steps * ceil_div(static_cast<long long>(num_rels) * feat_in, kKC) > INT32_MAX)
    return fail("sparsetir_sparse_conv_f16: the layer is too large for 32-bit indices");
  if (use_device(device_id) != 0) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (validate_enabled()) {
    const long long entries = static_cast<long long>(ceil_div(m, kTM)) * num_rels * kTM;
    if (validate_range("sparsetir_sparse_conv_f16", "map", map, entries, n, st, /*lowest=*/-1) != 0) return -1;
  }
  CUtensorMap tm_w;
  if (make_tmap_2d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, w, static_cast<uint64_t>(feat_out),
                   static_cast<uint64_t>(num_rels) * feat_in, static_cast<uint64_t>(feat_out) * 2, 64, kKC,
                   CU_TENSOR_MAP_SWIZZLE_128B) != 0)
    return -1;
  if (y_is_f16)
    return launch(tm_w, static_cast<__half*>(y), static_cast<const __half*>(x), static_cast<const __half*>(w), map, m,
                  num_rels, feat_in, feat_out, add, st);
  return launch(tm_w, static_cast<float*>(y), static_cast<const __half*>(x), static_cast<const __half*>(w), map, m,
                num_rels, feat_in, feat_out, add, st);
}

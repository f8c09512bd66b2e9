// Sparse convolution with the neighbour map of a layer laid out once, fp16 operands, fp32 sums:
//   Y[d, :] (+)= sum over kernel offsets r with a pair (s, d):  X[s, :] * W[r, :, :]
// for layers in which an (offset, output) pair never repeats (examples/sparse_conv of the
// reference: examples/rgms/sparse_conv/sparse_conv.py:93-125).  map holds, for tiles of 128 outputs,
// map[(tile * R + r) * 128 + t] = s, or -1 where output tile * 128 + t has no pair of offset r.
//
// The product is one GEMM per tile with K = R * feat_in: row t of the left operand is the
// concatenation of the X rows of its pairs (zeros where there is none), the right operand is W as
// it lies in memory.  A persistent block per SM walks the tiles; per 64-wide slice of K
//  - six groups of four warps fetch the left operand with 16-byte asynchronous copies into the
//    swizzled stage (a slice may straddle offsets, so channel counts that are not multiples of 64
//    waste nothing; a missing pair is a copy of no bytes, which fills in zeros);
//  - one thread brings the slice of W with TMA, one issues the MMAs into one of two accumulators;
//  - four warps take finished tiles out of TMEM and write (or add to) Y, each row once.
//
// Bound by the instructions and round trips of the ring, not by a unit (100,000 points, 27 offsets,
// 64 -> 128: tensor pipe 34 %, L1 data pipe 61 %, L2 22 %): the time goes with the steps and hardly
// depends on the share of pairs or on feat_out.  What the steps cost is therefore what was cut: no
// divisions in the loops and MMAs from an elected thread 97 -> 64 us, asynchronous copies instead of
// loads and stores 64 -> 61 us.  Gathering by TMA (four rows per copy) took 215 us.  The map replaces one
// built, checked and cleared on every call: together with the cleared Y that took 37 us of 122.
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
constexpr int kSmemLimit = 226 * 1024;  // dynamic part: the static barriers count against the 227 KB too

__device__ unsigned int g_conv_timeouts = 0;

__device__ __forceinline__ void arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc05::smem_u32(bar)) : "memory");
}

// 32 columns of 32 rows of a finished tile, staged in shared memory, go to Y with whole 128-byte
// (fp32) or 64-byte (fp16) row pieces; with `add` all old values are read before the first store
__device__ __forceinline__ void write32(float* y, const unsigned char* wbase, int row_base, int nrows, int feat_out,
                                        int c0, int lane, bool add) {
  float4 old[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int lr = 4 * i + (lane >> 3);
    old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (add && lr < nrows)
      old[i] = __ldcs(reinterpret_cast<const float4*>(y + static_cast<size_t>(row_base + lr) * feat_out + c0) + (lane & 7));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int lr = 4 * i + (lane >> 3);
    if (lr < nrows) {
      const float4 v = *reinterpret_cast<const float4*>(wbase + lr * kOutStride + (lane & 7) * 16);
      __stcs(reinterpret_cast<float4*>(y + static_cast<size_t>(row_base + lr) * feat_out + c0) + (lane & 7),
             make_float4(old[i].x + v.x, old[i].y + v.y, old[i].z + v.z, old[i].w + v.w));
    }
  }
}
__device__ __forceinline__ void write32(__half* y, const unsigned char* wbase, int row_base, int nrows, int feat_out,
                                        int c0, int lane, bool add) {
  uint4 old[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = 8 * i + (lane >> 2);
    old[i] = make_uint4(0u, 0u, 0u, 0u);
    if (add && lr < nrows)
      old[i] = __ldcs(reinterpret_cast<const uint4*>(y + static_cast<size_t>(row_base + lr) * feat_out + c0) + (lane & 3));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int lr = 8 * i + (lane >> 2);
    if (lr < nrows) {
      const float4 a = *reinterpret_cast<const float4*>(wbase + lr * kOutStride + (lane & 3) * 32);
      const float4 b = *reinterpret_cast<const float4*>(wbase + lr * kOutStride + (lane & 3) * 32 + 16);
      uint4 o = old[i];
      __half2* h = reinterpret_cast<__half2*>(&o);
      h[0] = __hadd2(h[0], __floats2half2_rn(a.x, a.y));
      h[1] = __hadd2(h[1], __floats2half2_rn(a.z, a.w));
      h[2] = __hadd2(h[2], __floats2half2_rn(b.x, b.y));
      h[3] = __hadd2(h[3], __floats2half2_rn(b.z, b.w));
      __stcs(reinterpret_cast<uint4*>(y + static_cast<size_t>(row_base + lr) * feat_out + c0) + (lane & 3), o);
    }
  }
}

// One row's 32 outputs from its pairs alone, lane = output.  A row without a pair of some offset takes
// part in that offset's product with zeros, and 0 * W is NaN where W is not finite: rows that came
// out with a NaN are formed again here, from the terms of the sum and no others.
__device__ __noinline__ float row_by_pairs(const __half* __restrict__ x, const __half* __restrict__ w,
                                           const int32_t* __restrict__ entries, int num_rels, int feat_in,
                                           int feat_out, int col) {
  float sum = 0.f;
  for (int rel = 0; rel < num_rels; ++rel) {
    const int e = __ldg(entries + static_cast<size_t>(rel) * kTM);
    if (e < 0) continue;
    const __half* xr = x + static_cast<size_t>(e) * feat_in;
    const __half* wr = w + static_cast<size_t>(rel) * feat_in * feat_out + col;
#pragma unroll 8
    for (int fi = 0; fi < feat_in; ++fi)
      sum = fmaf(__half2float(__ldg(xr + fi)), __half2float(__ldg(wr + static_cast<size_t>(fi) * feat_out)), sum);
  }
  return sum;
}

template <typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
sparse_conv_kernel(const __grid_constant__ CUtensorMap tm_w, OutT* __restrict__ y, const __half* __restrict__ x,
                   const __half* __restrict__ w, const int32_t* __restrict__ map, int m, int num_rels, int feat_in,
                   int feat_out, int tmem_cols, int acc_cols, int nstages, int groups, int add) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[kMaxStages];   // both operands of the stage are there
  __shared__ __align__(8) uint64_t bar_empty[kMaxStages];  // the tensor core has read the stage
  __shared__ __align__(8) uint64_t bar_acc_full[2];
  __shared__ __align__(8) uint64_t bar_acc_empty[2];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* base = smem_raw + ((1024u - (tc05::smem_u32(smem_raw) & 1023u)) & 1023u);
  const int nwb = (feat_out + 63) / 64;
  const int stride = kZBytes + nwb * kWBox;
  const int ktotal = num_rels * feat_in;
  const int steps = (ktotal + kKC - 1) / kKC;  // stages per tile
  const int ntiles = (m + kTM - 1) / kTM;
  // tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the grid never exceeds the number of tiles
  const int my_tiles = (ntiles - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);

  if (warp == 0) {
    if (lane == 0) {
      for (int s = 0; s < nstages; ++s) {
        tc05::mbar_init(&bar_full[s], 1 + 4);  // W, and the four warps of a gather group
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
  chain_enter();
  tc05::fence_before_sync();
  __syncthreads();
  tc05::fence_after_sync();
  const uint32_t tmem = s_tmem;
  bool ok = true;
  int armed = 0;

  if (warp == 0) {
    // ---- W: rows [64 s, 64 s + 64) of the (R * feat_in) x feat_out array; past its end zeros
    if (tc05::elect_one()) {
      int s = 0;
      uint32_t phase = 0;
      unsigned char* st = base + kZBytes;
      for (int k = 0; k < my_tiles && ok; ++k) {
        for (int sidx = 0; sidx < steps; ++sidx) {
          if (!tc05::mbar_wait(&bar_empty[s], phase ^ 1u)) { ok = false; break; }
          tc05::mbar_arrive_expect_tx(&bar_full[s], nwb * kWBox);
          for (int j = 0; j < nwb; ++j) tc05::tma_load_2d(st + j * kWBox, &tm_w, j * 64, sidx * kKC, &bar_full[s]);
          ++armed;
          st += stride;
          if (++s == nstages) { s = 0; phase ^= 1u; st = base + kZBytes; }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMAs: M = 128 outputs, N = feat_out, K = 16 per instruction
    if (tc05::elect_one()) {
      const uint32_t idesc = tc05::instr_desc(tc05::kFmtF16, kTM, feat_out, /*a_mn=*/0, /*b_mn=*/1);
      const uint64_t dz0 = tc05::smem_desc_swizzled(tc05::smem_u32(base), 0, 1024, tc05::kSwizzle128B);
      const uint64_t dw0 = tc05::smem_desc_swizzled(tc05::smem_u32(base) + kZBytes, kWBox, 1024, tc05::kSwizzle128B);
      const int last = (ktotal - (steps - 1) * kKC) / 16;  // instructions of the last slice
      int s = 0;
      uint32_t phase = 0;
      uint64_t dz = dz0, dw = dw0;
      for (int k = 0; k < my_tiles && ok; ++k) {
        const int buf = k & 1, buse = k >> 1;
        if (!tc05::mbar_wait(&bar_acc_empty[buf], (buse & 1) ^ 1)) { ok = false; break; }
        const uint32_t acc = tmem + buf * acc_cols;
        for (int sidx = 0; sidx < steps; ++sidx) {
          if (!tc05::mbar_wait(&bar_full[s], phase)) { ok = false; break; }
          tc05::fence_after_sync();
          const int ksteps = sidx + 1 < steps ? kKC / 16 : last;
#pragma unroll
          for (int ks = 0; ks < kKC / 16; ++ks)
            if (ks < ksteps)
              tc05::mma_f16(acc, tc05::desc_advance(dz, ks * 32), tc05::desc_advance(dw, ks * 2048), idesc,
                            (sidx > 0 || ks > 0) ? 1u : 0u);
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
    // ---- gather: group g fills the left operand of steps g, g + groups, ...; warp gw of it rows
    // gw * 32 .. gw * 32 + 31, eight lanes per row.  No more groups than stages: a group that has
    // written step n knows that the tensor core is past step n - nstages, and may wait for the stage
    // of step n + groups only if that puts it at most one phase of the stage's barrier behind.  The map
    // entries of a group's next step are requested before this step's rows are written.
    //
    // (offset, piece) of the lane move by whole rows of the ring: quotients and remainders are formed once.
    const int g = (warp - kFirstGather) >> 2, gw = (warp - kFirstGather) & 3;
    const int cpr = feat_in / 8;  // 16-byte pieces per X row
    const int chunk = lane & 7;
    const int step_rel = groups * 8 / cpr, step_off = groups * 8 - step_rel * cpr;
    const int tile_rel = steps * 8 / cpr, tile_off = steps * 8 - tile_rel * cpr;
    int sidx = g, rel = (g * 8 + chunk) / cpr, off = g * 8 + chunk - rel * cpr;
    int left = my_tiles;  // tiles from the one of this step on
    const size_t tile_map = static_cast<size_t>(num_rels) * kTM;
    const int32_t* mp = map + static_cast<size_t>(blockIdx.x) * tile_map + gw * 32 + (lane >> 3);
    auto into_tile = [&]() {  // steps past the end of a tile belong to the block's next ones
      while (left > 0 && sidx >= steps) {
        sidx -= steps;
        --left;
        mp += tile_map * gridDim.x;
        rel -= tile_rel;
        off -= tile_off;
        if (off < 0) { off += cpr; --rel; }
      }
    };
    int entry[8];
    auto entries_of_step = [&]() {
      const bool in = rel < num_rels;
      const int32_t* e = mp + static_cast<size_t>(in ? rel : 0) * kTM;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int v = __ldg(e + 4 * i);
        entry[i] = in ? v : -1;
      }
    };
    int s = g;
    uint32_t phase = 0;
    if (g < groups) into_tile();
    if (g < groups && left > 0) entries_of_step();
    while (g < groups && left > 0) {
      const int piece = off;
      int from[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) from[i] = entry[i];
      sidx += groups;
      rel += step_rel;
      off += step_off;
      if (off >= cpr) { off -= cpr; ++rel; }
      into_tile();
      if (left > 0) entries_of_step();
      if (!tc05::mbar_wait(&bar_empty[s], phase ^ 1u)) { ok = false; break; }
      const uint32_t st = tc05::smem_u32(base + s * stride);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = gw * 32 + 4 * i + (lane >> 3);
        const uint32_t dst = st + (row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4);
        const __half* src = x + static_cast<size_t>(max(from[i], 0)) * feat_in + piece * 8;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(from[i] >= 0 ? 16u : 0u)
                     : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      tc05::fence_async_smem();
      __syncwarp();
      if (lane == 0) arrive(&bar_full[s]);
      s += groups;
      if (s >= nstages) { s -= nstages; phase ^= 1u; }
    }
  } else if (warp >= 4) {
    // ---- epilogue: thread = tile row = TMEM lane, 32 columns at a time
    unsigned char* buf0 = base + nstages * stride;
    unsigned char* my_row = buf0 + ((warp & 3) * 32 + lane) * kOutStride;
    const unsigned char* wbase = buf0 + (warp & 3) * 32 * kOutStride;
    for (int k = 0; k < my_tiles; ++k) {
      const int buf = k & 1, buse = k >> 1;
      const int row_base = (static_cast<int>(blockIdx.x) + k * static_cast<int>(gridDim.x)) * kTM + (warp & 3) * 32;
      const int nrows = min(32, m - row_base);  // live rows among the warp's 32 (may be <= 0)
      if (!tc05::mbar_wait(&bar_acc_full[buf], buse & 1)) { ok = false; break; }
      tc05::fence_after_sync();
      const uint32_t taddr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + buf * acc_cols;
      for (int c0 = 0; c0 < feat_out; c0 += 32) {
        uint32_t r[32];
        tc05::tmem_ld32(taddr + c0, r);
        if (c0 + 32 >= feat_out) {  // the accumulator is in registers: a later tile may overwrite it
          tc05::fence_before_sync();
          __syncwarp();
          if (lane == 0) arrive(&bar_acc_empty[buf]);
        }
        __syncwarp();  // the warp's reads of the previous 32 columns are over
#pragma unroll
        for (int q = 0; q < 8; ++q)
          *reinterpret_cast<uint4*>(my_row + q * 16) = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
        __syncwarp();
        bool nan = false;
#pragma unroll
        for (int q = 0; q < 32; ++q) nan |= __uint_as_float(r[q]) != __uint_as_float(r[q]);
        for (unsigned todo = __ballot_sync(0xffffffffu, nan && lane < nrows); todo != 0u; todo &= todo - 1u) {
          const int lr = __ffs(todo) - 1;
          const int tile = static_cast<int>(blockIdx.x) + k * static_cast<int>(gridDim.x);
          const int32_t* entries = map + static_cast<size_t>(tile) * num_rels * kTM + (warp & 3) * 32 + lr;
          *reinterpret_cast<float*>(buf0 + ((warp & 3) * 32 + lr) * kOutStride + lane * 4) =
              row_by_pairs(x, w, entries, num_rels, feat_in, feat_out, c0 + lane);
          __syncwarp();
        }
        write32(y, wbase, row_base, nrows, feat_out, c0, lane, add != 0);
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

template <typename OutT>
int launch(const CUtensorMap& tm_w, OutT* y, const __half* x, const __half* w, const int32_t* map, int m, int num_rels, int feat_in,
           int feat_out, int add, cudaStream_t st) {
  static thread_local int configured_device = -1;
  int dev = 0;
  SPTIR_CUDA_OK(cudaGetDevice(&dev));
  if (configured_device != dev) {
    SPTIR_CUDA_OK(cudaFuncSetAttribute(sparse_conv_kernel<OutT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    configured_device = dev;
  }
  const int stride = kZBytes + ceil_div(feat_out, 64) * kWBox;
  const int nstages = std::min(kMaxStages, (kSmemLimit - kOutBytes - 1024) / stride);
  const int smem = nstages * stride + kOutBytes + 1024;
  const int acc_cols = (feat_out + 31) & ~31;
  int tmem_cols = 32;
  while (tmem_cols < 2 * acc_cols) tmem_cols *= 2;
  const int grid = std::min(ceil_div(m, kTM), kNumSMs);
  launch_chained(sparse_conv_kernel<OutT>, grid, kThreads, smem, st, tm_w, y, x, w, map, m, num_rels, feat_in, feat_out,
                 tmem_cols, acc_cols, nstages, std::min(kGroups, nstages), add);
  SPTIR_LAUNCH_OK("sparse_conv_kernel");
  return 0;
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

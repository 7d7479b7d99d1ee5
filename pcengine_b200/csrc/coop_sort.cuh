// A stable radix sort of (64-bit key, 32-bit value) pairs by all blocks of ONE cooperatively launched kernel.
//
// The arrays the engine sorts (a scan's points, the voxels of a level) are 10^4..10^6 entries that live in L2: there a
// library sort is bound by its launches, its memsets and the look-back latency of every pass (8 us a pass for 90 k
// entries, and one pass per 8 bits of the key TYPE unless the host knows the key range).  Inside a cooperative kernel
// a pass is a count, a grid barrier, a scatter and a grid barrier (about 4 us), the keys of a chunk stay in registers
// between the two halves, and the number of passes follows from key bits that only the device knows.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace pce {
namespace coop {

namespace cg = cooperative_groups;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

template <int BITS>
struct SortShared {
  static constexpr int kBins = 1 << BITS;  // 256 or 512
  int count[kWarps][kBins];  // per warp and digit: first the count, then the offset of the warp's first entry
  int base[kBins];           // where the block's entries of a digit go
  int part[2][kThreads - kBins > 0 ? kBins : 1];
  int warp_sum[kWarps];
};

// Exclusive scan of one value per thread over the block; `total` = the sum.
__device__ __forceinline__ int block_exclusive(int v, int* warp_sum, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d) incl += u;
  }
  __syncthreads();
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const int s = warp_sum[w];
    before += w < warp ? s : 0;
    total += s;
  }
  return before + incl - v;
}

// sh.base[d] = entries of lower digits + entries of digit d in earlier blocks, from hist [grid][bins] (256 bins: two
// threads per digit, half the blocks each).
template <int BITS>
__device__ __forceinline__ void block_offsets(SortShared<BITS>& sh, const int* hist) {
  constexpr int kBins = 1 << BITS, kHalves = kThreads / kBins;
  static_assert(kHalves == 1 || kHalves == 2, "256 or 512 bins");
  const int tid = threadIdx.x;
  const int d = tid & (kBins - 1), half = tid / kBins;
  const int g = static_cast<int>(gridDim.x), mid = kHalves == 2 ? (g + 1) / 2 : g;
  int pre = 0, all = 0;
  // (batches of loads in flight: one after the other they were half of the pass)
  for (int b0 = half ? mid : 0, end = half ? g : mid; b0 < end; b0 += 16) {
    int c[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) c[u] = b0 + u < end ? __ldcg(hist + (b0 + u) * kBins + d) : 0;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      all += c[u];
      pre += b0 + u < static_cast<int>(blockIdx.x) ? c[u] : 0;
    }
  }
  if (kHalves == 2) {
    if (half) {
      sh.part[0][d] = pre;
      sh.part[1][d] = all;
    }
    __syncthreads();
    if (!half) {
      pre += sh.part[0][d];
      all += sh.part[1][d];
    }
  }
  int total;
  const int lower = block_exclusive(half ? 0 : all, sh.warp_sum, total);
  if (!half) sh.base[d] = lower + pre;
  __syncthreads();
}

// One pass over the chunk of this block: entry j of a thread is element (warp's first + 32 j + lane), so that warps and
// then items and then lanes are in array order (stability).  `hist` is [grid][256].
template <int ITEMS>
__device__ __forceinline__ void sort_pass(cg::grid_group& grid, SortShared<8>& sh, int* hist, int n, int shift,
                                          const unsigned long long (&key)[ITEMS], const int (&val)[ITEMS],
                                          unsigned long long* key_out, int* val_out) {
  constexpr int kBins = 256;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kWarps * kBins; i += kThreads) (&sh.count[0][0])[i] = 0;
  __syncthreads();
  const int first = (blockIdx.x * kWarps + warp) * (32 * ITEMS) + lane;
  int rank[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const bool live = first + 32 * j < n;
    const int d = live ? static_cast<int>((key[j] >> shift) & (kBins - 1)) : kBins + lane;
    const unsigned same = __match_any_sync(0xFFFFFFFFu, d);
    const unsigned before = same & ((1u << lane) - 1u);
    const int old = live ? sh.count[warp][d] : 0;
    __syncwarp();
    if (live && before == 0) sh.count[warp][d] = old + __popc(same);
    __syncwarp();
    rank[j] = old + __popc(before);
  }
  __syncthreads();
  if (tid < kBins) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = sh.count[w][tid];
      sh.count[w][tid] = run;
      run += c;
    }
    hist[blockIdx.x * kBins + tid] = run;
  }
  grid.sync();
  block_offsets(sh, hist);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    if (first + 32 * j < n) {
      const int d = static_cast<int>((key[j] >> shift) & (kBins - 1));
      const int at = sh.base[d] + sh.count[warp][d] + rank[j];
      key_out[at] = key[j];
      val_out[at] = val[j];
    }
  }
  grid.sync();
}

// Loads this block's chunk (written by other blocks before the last barrier).
template <int ITEMS>
__device__ __forceinline__ void load_chunk(int n, const unsigned long long* key_in, const int* val_in,
                                           unsigned long long (&key)[ITEMS], int (&val)[ITEMS]) {
  const int first = (blockIdx.x * kWarps + (threadIdx.x >> 5)) * (32 * ITEMS) + (threadIdx.x & 31);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    key[j] = i < n ? __ldcg(key_in + i) : 0ull;
    val[j] = i < n ? __ldcg(val_in + i) : 0;
  }
}

// The same pass for any number of entries: nothing stays in registers, a warp walks its stretch of the array twice
// (count, scatter), four keys in flight.  load(i, key, value) gives entry i.
template <int BITS, typename K, typename Load>
__device__ __forceinline__ void sort_pass_any(cg::grid_group& grid, SortShared<BITS>& sh, int* hist, int n, int shift, Load load, K* key_out,
                                              int* val_out) {
  constexpr int kBatch = 4, kBins = 1 << BITS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = static_cast<int>(gridDim.x);
  const int per_warp = ((n + g * kWarps - 1) / (g * kWarps) + 31) & ~31;
  const long long lo64 = static_cast<long long>(blockIdx.x * kWarps + warp) * per_warp;
  const int lo = static_cast<int>(lo64 < n ? lo64 : n), hi = static_cast<int>(lo64 + per_warp < n ? lo64 + per_warp : n);
  for (int i = tid; i < kWarps * kBins; i += kThreads) (&sh.count[0][0])[i] = 0;
  __syncthreads();
  for (int b = lo; b < hi; b += 32 * kBatch) {
    K key[kBatch];
    int val;
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      key[u] = 0;
      if (b + 32 * u + lane < hi) load(b + 32 * u + lane, key[u], val);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (b + 32 * u >= hi) break;
      const bool live = b + 32 * u + lane < hi;
      const int d = live ? static_cast<int>((key[u] >> shift) & (kBins - 1)) : kBins + lane;
      const unsigned same = __match_any_sync(0xFFFFFFFFu, d);
      if (live && (same & ((1u << lane) - 1u)) == 0) sh.count[warp][d] += __popc(same);
      __syncwarp();
    }
  }
  __syncthreads();
  if (tid < kBins) {
    int run = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = sh.count[w][tid];
      sh.count[w][tid] = run;
      run += c;
    }
    hist[blockIdx.x * kBins + tid] = run;
  }
  grid.sync();
  block_offsets(sh, hist);
  for (int b = lo; b < hi; b += 32 * kBatch) {
    K key[kBatch];
    int val[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      key[u] = 0;
      val[u] = 0;
      if (b + 32 * u + lane < hi) load(b + 32 * u + lane, key[u], val[u]);
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      if (b + 32 * u >= hi) break;
      const bool live = b + 32 * u + lane < hi;
      const int d = live ? static_cast<int>((key[u] >> shift) & (kBins - 1)) : kBins + lane;
      const unsigned same = __match_any_sync(0xFFFFFFFFu, d);
      const unsigned before = same & ((1u << lane) - 1u);
      const int old = live ? sh.count[warp][d] : 0;
      __syncwarp();
      if (live && before == 0) sh.count[warp][d] = old + __popc(same);
      __syncwarp();
      if (live) {
        const int at = sh.base[d] + old + __popc(before);
        key_out[at] = key[u];
        val_out[at] = val[u];
      }
    }
  }
  grid.sync();
}

// Items per thread for n entries on a grid of at most one block per SM; 0: too many entries.
inline int items_for(long long n, int sm_count) {
  for (int items = 2; items <= 16; items *= 2)
    if (n <= static_cast<long long>(sm_count) * kThreads * items) return items;
  return 0;
}

}  // namespace coop
}  // namespace pce

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
constexpr int kBins = 256;

struct SortShared {
  int count[kWarps][kBins];  // per warp and digit: first the count, then the offset of the warp's first entry
  int base[kBins];           // where the block's entries of a digit go
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

// One pass over the chunk of this block: entry j of a thread is element (warp's first + 32 j + lane), so that warps and
// then items and then lanes are in array order (stability).  `hist` is [grid][kBins].
template <int ITEMS>
__device__ __forceinline__ void sort_pass(cg::grid_group& grid, SortShared& sh, int* hist, int n, int shift,
                                          const unsigned long long (&key)[ITEMS], const int (&val)[ITEMS],
                                          unsigned long long* key_out, int* val_out) {
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
  // per digit: entries of lower digits + this digit's entries in earlier blocks (two threads per digit, half the
  // blocks each)
  {
    const int d = tid & (kBins - 1), half = tid / kBins;
    const int g = static_cast<int>(gridDim.x), mid = (g + 1) / 2;
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
    __shared__ int s_pre[kBins], s_all[kBins];
    if (half) {
      s_pre[d] = pre;
      s_all[d] = all;
    }
    __syncthreads();
    int total;
    const int mine = half ? 0 : all + s_all[d];
    const int lower = block_exclusive(mine, sh.warp_sum, total);
    if (!half) sh.base[d] = lower + pre + s_pre[d];
    __syncthreads();
  }
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

// Items per thread for n entries on a grid of at most one block per SM; 0: too many entries.
inline int items_for(long long n, int sm_count) {
  for (int items = 2; items <= 16; items *= 2)
    if (n <= static_cast<long long>(sm_count) * kThreads * items) return items;
  return 0;
}

}  // namespace coop
}  // namespace pce

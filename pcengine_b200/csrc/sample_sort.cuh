// Sorting of distinct 64-bit words by all blocks of ONE cooperatively launched kernel, in one pass over the data and a sort per
// block in shared memory.
//
// A radix sort inside one kernel (coop_sort.cuh) is bound by its grid barriers and by the table of digit counts that every
// block reads in every pass: about 9 us for each 8 bits of a key.  Here a word is the key with the entry's index behind it,
// so that no two are equal and a stable order is simply the order of the words.  Every block sorts the same words, taken at
// equal distances, which gives splitters for one bucket per block; entries go into the buckets' fixed regions of
// 4 x target words (a position per block and bucket from one atomic), and every block sorts its bucket.  Splitters are
// whole words, so that a key that is repeated very often spreads over as many buckets as its entries need: the caller joins
// equal keys across the border of two buckets.  (A splitter is itself an entry, the smallest of its bucket: none is empty.)
// A bucket that overflows (a sample that misses the distribution) is seen by every block behind the barrier: the caller
// then sorts by radix.
// (For the row orders, 27-bit keys, the radix sort's three passes are as fast from 120 k entries on: 52 and 48 us for 240 k.)
#pragma once

#include "common.cuh"

namespace pce {
namespace samp {

typedef unsigned long long word_t;

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kTarget = 1024;             // entries per bucket aimed at
constexpr int kCap = 4 * kTarget;         // words in a bucket's region
constexpr int kSamples = 1024;
constexpr int kMaxBuckets = 160;
constexpr word_t kLast = ~0ull;           // behind every word

struct Shared {
  word_t words[kCap];        // the sample, then the bucket
  word_t split[kMaxBuckets];  // first word of every bucket (of the first: unused)
  int count[kMaxBuckets];
  int start[kMaxBuckets];
};

// The steps j = j0, j0 / 2 .. 1 of a bitonic merge on 64 words that a warp holds, e0 = words[lane], e1 = words[lane + 32]; `up0` /
// `up1`: direction of each.
__device__ __forceinline__ void merge64(word_t& e0, word_t& e1, bool up0, bool up1, int j0, int lane) {
  if (j0 >= 32) {
    const bool swap = (e0 > e1) == up0;
    const word_t x = swap ? e1 : e0, y = swap ? e0 : e1;
    e0 = x;
    e1 = y;
  }
#pragma unroll
  for (int j = 16; j; j >>= 1) {
    if (j > j0) continue;
    const word_t o0 = __shfl_xor_sync(0xFFFFFFFFu, e0, j), o1 = __shfl_xor_sync(0xFFFFFFFFu, e1, j);
    const bool low = (lane & j) == 0;
    e0 = (low == up0) == (e0 < o0) ? e0 : o0;
    e1 = (low == up1) == (e1 < o1) ? e1 : o1;
  }
}

// Sorts the m (a power of two, at least 64) words by the whole block.  Distances up to 32 are exchanged in registers, so that
// only the wide steps pass through shared memory and block barriers (10 of 55 for 1024 words).
__device__ __forceinline__ void sort_words(word_t* w, int m) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  for (int seg = warp * 64; seg < m; seg += kWarps * 64) {
    word_t e0 = w[seg + lane], e1 = w[seg + lane + 32];
#pragma unroll
    for (int k = 2; k <= 64; k <<= 1) {
      const bool up0 = ((seg + lane) & k) == 0, up1 = ((seg + lane + 32) & k) == 0;
      merge64(e0, e1, up0, up1, k / 2, lane);
    }
    w[seg + lane] = e0;
    w[seg + lane + 32] = e1;
  }
  for (int k = 128; k <= m; k <<= 1) {
    for (int j = k / 2; j >= 64; j >>= 1) {
      __syncthreads();
      for (int p = threadIdx.x; p < m / 2; p += kThreads) {
        const int i = ((p & ~(j - 1)) << 1) | (p & (j - 1));
        const word_t a = w[i], b = w[i + j];
        if ((a > b) == ((i & k) == 0)) {
          w[i] = b;
          w[i + j] = a;
        }
      }
    }
    __syncthreads();
    for (int seg = warp * 64; seg < m; seg += kWarps * 64) {
      word_t e0 = w[seg + lane], e1 = w[seg + lane + 32];
      const bool up = (seg & k) == 0;
      merge64(e0, e1, up, up, 32, lane);
      w[seg + lane] = e0;
      w[seg + lane + 32] = e1;
    }
  }
  __syncthreads();
}

// Splitters of the buckets; word(i) gives entry i of n (at least kSamples where there are two buckets or more).
template <typename Word>
__device__ __forceinline__ void splitters(Shared& sh, int buckets, int n, Word word) {
  if (buckets > 1) {
    for (int s = threadIdx.x; s < kSamples; s += kThreads)
      sh.words[s] = word(static_cast<int>((static_cast<long long>(s) * n + n / 2) / kSamples));
    sort_words(sh.words, kSamples);
    for (int b = threadIdx.x; b < buckets; b += kThreads) sh.split[b] = sh.words[b * kSamples / buckets];
  }
  __syncthreads();
}

// Up to ITEMS words of every thread (kLast: none) into the regions; `counters` (one per bucket, zeroed) then hold what every
// bucket was given.
template <int ITEMS>
__device__ __forceinline__ void scatter(Shared& sh, int buckets, const word_t (&w)[ITEMS], word_t* region, int* counters) {
  int top = 1;
  while (2 * top < buckets) top *= 2;
  for (int b = threadIdx.x; b < buckets; b += kThreads) sh.count[b] = 0;
  __syncthreads();
  int bucket[ITEMS], place[ITEMS];
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) {
    bucket[u] = 0;
    for (int s = top; s; s >>= 1)
      if (bucket[u] + s < buckets && sh.split[bucket[u] + s] <= w[u]) bucket[u] += s;
    place[u] = w[u] != kLast ? atomicAdd(&sh.count[bucket[u]], 1) : 0;
  }
  __syncthreads();
  for (int b = threadIdx.x; b < buckets; b += kThreads) sh.start[b] = sh.count[b] ? atomicAdd(counters + b, sh.count[b]) : 0;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < ITEMS; ++u) {
    const int at = sh.start[bucket[u]] + place[u];
    if (w[u] != kLast && at < kCap) region[static_cast<size_t>(bucket[u]) * kCap + at] = w[u];
  }
}

// The n words of a bucket, sorted, in sh.words.
__device__ __forceinline__ void sort_bucket(Shared& sh, int n, const word_t* from) {
  int m = 64;
  while (m < n) m <<= 1;
  for (int i = threadIdx.x; i < m; i += kThreads) sh.words[i] = i < n ? __ldcg(from + i) : kLast;
  sort_words(sh.words, m);
}

}  // namespace samp
}  // namespace pce

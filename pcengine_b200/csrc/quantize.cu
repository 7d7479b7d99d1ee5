// Voxelisation on the device: floor(points / voxel) and one row per occupied voxel, the step in
// front of the kernel maps (ref: script/utils.py:34-55 sparse_quantize, which does it with NumPy on
// the host: floor-divide, ravel hash, np.unique with return_index / return_inverse).
//
// Same results as that host code: the division is done in double precision (NumPy promotes the
// float32 points against the Python-float voxel size), the voxels come out in ascending (x,y,z)
// order (the order of the ravel hash), `index` names the FIRST point of every voxel (stable sort)
// and `inverse` maps every point to its voxel.
#include <algorithm>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "common.cuh"
#include "coop_sort.cuh"
#include "sample_sort.cuh"

namespace pce {

__global__ void k_voxel_keys(const float* __restrict__ pts, int n, double vx, double vy, double vz, int batch,
                             unsigned long long* keys, int* vals, int* status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int x = static_cast<int>(floor(static_cast<double>(pts[3 * i]) / vx));
  const int y = static_cast<int>(floor(static_cast<double>(pts[3 * i + 1]) / vy));
  const int z = static_cast<int>(floor(static_cast<double>(pts[3 * i + 2]) / vz));
  if (!packable(batch, x, y, z)) atomicMax(status, PCE_ERR_RANGE);
  keys[i] = pack_key(batch, x, y, z);
  vals[i] = i;
}

__global__ void k_voxel_heads(const unsigned long long* __restrict__ keys, int n, int* heads) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) heads[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// rank[i] = inclusive count of heads up to i; voxel id of sorted position i = rank[i] - 1.
__global__ void k_voxel_emit(const unsigned long long* __restrict__ keys, const int* __restrict__ src,
                             const int* __restrict__ heads, const int* __restrict__ rank, int n, int4* coords,
                             int* index, int* inverse, int* n_unique) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int u = rank[i] - 1;
  if (heads[i]) {
    int b, x, y, z;
    unpack_key(keys[i], b, x, y, z);
    coords[u] = make_int4(b, x, y, z);
    if (index) index[u] = src[i];
  }
  if (inverse) inverse[src[i]] = u;
  if (i == n - 1) *n_unique = u + 1;
}


// Where the results go: voxels as rows of 3 or 4 (batch in front) int32, indices as 32- or 64-bit integers.
struct VoxelOut {
  int* voxels;
  int width;  // 3 or 4
  void* index;
  void* inverse;
  int wide;  // 64-bit index / inverse
  int* host;  // [0] status, [1] voxels (mapped host memory)
};

__device__ __forceinline__ void put_int(void* p, int wide, int at, int v) {
  if (wide)
    static_cast<long long*>(p)[at] = v;
  else
    static_cast<int*>(p)[at] = v;
}

// The whole voxelisation in one cooperative launch: floor-divide, bounds of the voxels (they set the key's bits and
// with them the number of radix passes), stable sort of (voxel, point), heads of equal runs, ranks, results.
// `bounds` is [grid][8], `counts` [grid], `hist` [grid][256]: every block writes its entries, nothing is initialised.
template <int ITEMS>
__global__ void __launch_bounds__(coop::kThreads)
    k_voxelise(const float* __restrict__ pts, int n, double vx, double vy, double vz, int batch, unsigned long long* key0,
               unsigned long long* key1, int* val0, int* val1, int* bounds, int* hist, int* counts, VoxelOut out) {
  using namespace coop;
  __shared__ SortShared<8> sh;
  __shared__ int red[kWarps][7];
  __shared__ int s_b[7];
  cg::grid_group grid = cg::this_grid();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = (blockIdx.x * kWarps + warp) * (32 * ITEMS) + lane;
  int c[ITEMS][3];
  int lo[3] = {0x7FFFFFFF, 0x7FFFFFFF, 0x7FFFFFFF}, hi[3] = {-0x7FFFFFFF, -0x7FFFFFFF, -0x7FFFFFFF}, bad = 0;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    if (i < n) {
      c[j][0] = static_cast<int>(floor(static_cast<double>(pts[3 * i]) / vx));
      c[j][1] = static_cast<int>(floor(static_cast<double>(pts[3 * i + 1]) / vy));
      c[j][2] = static_cast<int>(floor(static_cast<double>(pts[3 * i + 2]) / vz));
      if (!packable(batch, c[j][0], c[j][1], c[j][2])) bad = 1;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        lo[d] = min(lo[d], c[j][d]);
        hi[d] = max(hi[d], c[j][d]);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(0xFFFFFFFFu, lo[d]);
    hi[d] = __reduce_max_sync(0xFFFFFFFFu, hi[d]);
  }
  bad = __any_sync(0xFFFFFFFFu, bad) ? 1 : 0;
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      red[warp][d] = -lo[d];
      red[warp][3 + d] = hi[d];
    }
    red[warp][6] = bad;
  }
  __syncthreads();
  if (tid < 7) {
    int m = red[0][tid];
    for (int w = 1; w < kWarps; ++w) m = max(m, red[w][tid]);
    bounds[blockIdx.x * 8 + tid] = m;
  }
  grid.sync();
  if (warp < 7) {
    int m = -0x7FFFFFFF;
    for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) m = max(m, __ldcg(bounds + b * 8 + warp));
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if (lane == 0) s_b[warp] = m;
  }
  __syncthreads();
  if (s_b[6]) {  // a voxel outside the packable range: the same for every block
    if (blockIdx.x == 0 && tid == 0) {
      out.host[0] = PCE_ERR_RANGE;
      out.host[1] = 0;
    }
    return;
  }
  const int mx = -s_b[0], my = -s_b[1], mz = -s_b[2];
  const int bz = 32 - __clz(s_b[5] - mz), by = 32 - __clz(s_b[4] - my), bx = 32 - __clz(s_b[3] - mx);
  unsigned long long key[ITEMS];
  int val[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    key[j] = 0ull;
    val[j] = i;
    if (i < n)
      key[j] = (((static_cast<unsigned long long>(c[j][0] - mx) << by) | static_cast<unsigned long long>(c[j][1] - my)) << bz) |
               static_cast<unsigned long long>(c[j][2] - mz);
  }
  const int passes = max(1, (bx + by + bz + 7) / 8);
  for (int p = 0; p < passes; ++p) {
    if (p > 0) load_chunk<ITEMS>(n, p & 1 ? key0 : key1, p & 1 ? val0 : val1, key, val);
    sort_pass<ITEMS>(grid, sh, hist, n, 8 * p, key, val, p & 1 ? key1 : key0, p & 1 ? val1 : val0);
  }
  const unsigned long long* sorted = passes & 1 ? key0 : key1;
  load_chunk<ITEMS>(n, sorted, passes & 1 ? val0 : val1, key, val);
  // ranks in array order: (warp, item, lane)
  unsigned heads[ITEMS];
  int mine = 0;
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    unsigned long long prev = __shfl_up_sync(0xFFFFFFFFu, key[j], 1);
    if (lane == 0 && i > 0 && i < n) prev = __ldcg(sorted + i - 1);
    heads[j] = __ballot_sync(0xFFFFFFFFu, i < n && (i == 0 || key[j] != prev));
    mine += __popc(heads[j]);
  }
  int total;
  int run = block_exclusive(lane == 0 ? mine : 0, sh.warp_sum, total);
  run = __shfl_sync(0xFFFFFFFFu, run, 0);
  if (tid == 0) counts[blockIdx.x] = total;
  grid.sync();
  {
    int before = 0, all = 0;
    for (int b = lane; b < static_cast<int>(gridDim.x); b += 32) {
      const int v = __ldcg(counts + b);
      all += v;
      before += b < static_cast<int>(blockIdx.x) ? v : 0;
    }
    run += __reduce_add_sync(0xFFFFFFFFu, before);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    if (blockIdx.x == 0 && tid == 0) {
      out.host[0] = PCE_OK;
      out.host[1] = all;
    }
  }
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = first + 32 * j;
    const int u = run + __popc(heads[j] & (0xFFFFFFFFu >> (31 - lane))) - 1;
    if (i < n) {
      if ((heads[j] >> lane) & 1u) {
        int* v = out.voxels + static_cast<size_t>(u) * out.width;
        if (out.width == 4) *v++ = batch;
        v[0] = static_cast<int>(key[j] >> (by + bz)) + mx;
        v[1] = static_cast<int>((key[j] >> bz) & ((1ull << by) - 1)) + my;
        v[2] = static_cast<int>(key[j] & ((1ull << bz) - 1)) + mz;
        if (out.index) put_int(out.index, out.wide, u, val[j]);
      }
      if (out.inverse) put_int(out.inverse, out.wide, val[j], u);
    }
    run += __popc(heads[j]);
  }
}

// The same by one bucket per block (sample_sort.cuh): three grid barriers instead of ten for the keys of a scan (29 bits, four
// radix passes).  What bounds it: the latency of two sorts in shared memory (of the sample, of the bucket) and the barriers.
// 90 k points of a scan: 49.6 -> 32.9 us.  Points that share one voxel (returns at the
// sensor) may fill several buckets: 90 k points, a third in one voxel, 119 -> 77 us a call against buckets that end with a key.
// Returns to the host for the radix sort when a bucket overflows or key and index do not
// fit a word.  `bounds` is [grid][8], `counters` [grid] (zeroed here), `counts` [grid], `last` [grid] (a bucket's
// voxels and its last key), `region` [grid][kCap].
constexpr int kBucketItems = 2;  // points per thread: chunks of kTarget points
static_assert(kBucketItems * samp::kThreads == samp::kTarget, "a block reads as many points as a bucket holds on average");
constexpr int kTryRadix = -1000;

__global__ void __launch_bounds__(samp::kThreads)
    k_voxelise_buckets(const float* __restrict__ pts, int n, double vx, double vy, double vz, int batch, int* bounds, int* counters,
                       int* counts, unsigned long long* last, unsigned long long* region, VoxelOut out) {
  using namespace samp;
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
  __shared__ int red[kWarps][7];
  __shared__ int s_b[7];
  __shared__ int s_warp[kWarps];
  cg::grid_group grid = cg::this_grid();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
  auto cell = [&](int i, int (&c)[3]) {
    c[0] = static_cast<int>(floor(static_cast<double>(__ldg(pts + 3 * static_cast<size_t>(i))) / vx));
    c[1] = static_cast<int>(floor(static_cast<double>(__ldg(pts + 3 * static_cast<size_t>(i) + 1)) / vy));
    c[2] = static_cast<int>(floor(static_cast<double>(__ldg(pts + 3 * static_cast<size_t>(i) + 2)) / vz));
  };
  int c[kBucketItems][3];
  int lo[3] = {0x7FFFFFFF, 0x7FFFFFFF, 0x7FFFFFFF}, hi[3] = {-0x7FFFFFFF, -0x7FFFFFFF, -0x7FFFFFFF}, bad = 0;
#pragma unroll
  for (int u = 0; u < kBucketItems; ++u) {
    const int i = me * kTarget + u * kThreads + tid;
    if (i < n) {
      cell(i, c[u]);
      if (!packable(batch, c[u][0], c[u][1], c[u][2])) bad = 1;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        lo[d] = min(lo[d], c[u][d]);
        hi[d] = max(hi[d], c[u][d]);
      }
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = __reduce_min_sync(0xFFFFFFFFu, lo[d]);
    hi[d] = __reduce_max_sync(0xFFFFFFFFu, hi[d]);
  }
  bad = __any_sync(0xFFFFFFFFu, bad) ? 1 : 0;
  if (lane == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      red[warp][d] = -lo[d];
      red[warp][3 + d] = hi[d];
    }
    red[warp][6] = bad;
  }
  __syncthreads();
  if (tid < 7) {
    int m = red[0][tid];
    for (int w = 1; w < kWarps; ++w) m = max(m, red[w][tid]);
    bounds[me * 8 + tid] = m;
  }
  if (tid == 7) counters[me] = 0;
  grid.sync();
  if (warp < 7) {
    int m = -0x7FFFFFFF;
    for (int b = lane; b < g; b += 32) m = max(m, __ldcg(bounds + b * 8 + warp));
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    if (lane == 0) s_b[warp] = m;
  }
  __syncthreads();
  // (the same for every block from here to the next barrier)
  const int mx = -s_b[0], my = -s_b[1], mz = -s_b[2];
  const int bz = 32 - __clz(s_b[5] - mz), by = 32 - __clz(s_b[4] - my), bx = 32 - __clz(s_b[3] - mx);
  const int index_bits = 32 - __clz(n - 1);
  if (s_b[6] || bx + by + bz + index_bits > 63) {
    if (me == 0 && tid == 0) {
      out.host[0] = s_b[6] ? PCE_ERR_RANGE : kTryRadix;
      out.host[1] = 0;
    }
    return;
  }
  auto pack = [&](const int (&v)[3], int i) {
    const word_t key = (((static_cast<word_t>(v[0] - mx) << by) | static_cast<word_t>(v[1] - my)) << bz) | static_cast<word_t>(v[2] - mz);
    return key << index_bits | static_cast<word_t>(i);
  };
  splitters(sh, g, n, [&](int i) {
    int v[3];
    cell(i, v);
    return pack(v, i);
  });
  word_t w[kBucketItems];
#pragma unroll
  for (int u = 0; u < kBucketItems; ++u) {
    const int i = me * kTarget + u * kThreads + tid;
    w[u] = i < n ? pack(c[u], i) : kLast;
  }
  scatter<kBucketItems>(sh, g, w, region, counters);
  grid.sync();
  const int mine = __ldcg(counters + me);
  {
    int most = 0;
    for (int b = tid; b < g; b += kThreads) most = max(most, __ldcg(counters + b));
    if (__syncthreads_or(most > kCap)) {
      if (me == 0 && tid == 0) {
        out.host[0] = kTryRadix;
        out.host[1] = 0;
      }
      return;
    }
  }
  sort_bucket(sh, mine, region + static_cast<size_t>(me) * kCap);
  // heads of equal keys, rounds of kThreads words: voxels in front of the word's.  The first word counts as a head until
  // the bucket in front is known to end with another voxel.
  bool opens = true;
  auto head_at = [&](int i) { return i < mine && (i == 0 ? opens : sh.words[i] >> index_bits != sh.words[i - 1] >> index_bits); };
  int heads = 0;
  for (int i = tid; i < ((mine + 31) & ~31); i += kThreads) heads += __popc(__ballot_sync(0xFFFFFFFFu, head_at(i)));  // (per warp)
  if (lane == 0) s_warp[warp] = heads;
  __syncthreads();
  if (tid == 0) {
    int total = 0;
    for (int v = 0; v < kWarps; ++v) total += s_warp[v];
    counts[me] = total;
    last[me] = sh.words[max(mine, 1) - 1] >> index_bits;
  }
  grid.sync();
  // voxels in front of this bucket, and whether its first word belongs to the last of them
  if (warp == 0) {
    int before = 0, all = 0, joined = 0;
    word_t end[kMaxBuckets / 32];
    int count[kMaxBuckets / 32];
#pragma unroll
    for (int r = 0; r < kMaxBuckets / 32; ++r) {
      const int b = 32 * r + lane;
      end[r] = b > 0 && b < g ? __ldcg(last + b - 1) : kLast;
      count[r] = b < g ? __ldcg(counts + b) : 0;
    }
#pragma unroll
    for (int r = 0; r < kMaxBuckets / 32; ++r) {
      const int b = 32 * r + lane;
      const bool joins = end[r] != kLast && end[r] == sh.split[b] >> index_bits;  // (a bucket's first word is its splitter)
      all += count[r] - (joins ? 1 : 0);
      before += b < me ? count[r] - (joins ? 1 : 0) : 0;
      joined |= joins && b == me ? 1 : 0;
    }
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    joined = __any_sync(0xFFFFFFFFu, joined);
    if (lane == 0) {
      s_b[0] = before;
      s_b[1] = joined;
      if (me == 0) {
        out.host[0] = PCE_OK;
        out.host[1] = all;
      }
    }
  }
  __syncthreads();
  int before = s_b[0];
  opens = !s_b[1];
  const word_t index_mask = (1ull << index_bits) - 1ull;
  for (int i0 = 0; i0 < mine; i0 += kThreads) {
    const int i = i0 + tid;
    const bool head = head_at(i);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, head);
    __syncthreads();
    if (lane == 0) s_warp[warp] = __popc(m);
    __syncthreads();
    int u = before, round = 0;
    for (int v = 0; v < kWarps; ++v) {
      u += v < warp ? s_warp[v] : 0;
      round += s_warp[v];
    }
    u += __popc(m & (0xFFFFFFFFu >> (31 - lane))) - 1;
    if (i < mine) {
      const word_t x = sh.words[i], key = x >> index_bits;
      const int at = static_cast<int>(x & index_mask);
      if (head) {
        int* v = out.voxels + static_cast<size_t>(u) * out.width;
        if (out.width == 4) *v++ = batch;
        v[0] = static_cast<int>(key >> (by + bz)) + mx;
        v[1] = static_cast<int>((key >> bz) & ((1ull << by) - 1)) + my;
        v[2] = static_cast<int>(key & ((1ull << bz) - 1)) + mz;
        if (out.index) put_int(out.index, out.wide, u, at);
      }
      if (out.inverse) put_int(out.inverse, out.wide, at, u);
    }
    before += round;
  }
}

static int launch_buckets(const float* points, int n, const float* v, int batch, Arena& ar, const VoxelOut& out, cudaStream_t st) {
  static bool attr_set[64] = {};
  int dev = 0;
  PCE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
  if (!attr_set[dev]) {
    PCE_CUDA(cudaFuncSetAttribute(k_voxelise_buckets, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(samp::Shared))));
    attr_set[dev] = true;
  }
  const int g = div_up(n, samp::kTarget);
  int* bounds = ar.take<int>(static_cast<size_t>(g) * 8);
  int* counters = ar.take<int>(g);
  int* counts = ar.take<int>(g);
  unsigned long long* last = ar.take<unsigned long long>(g);
  unsigned long long* region = ar.take<unsigned long long>(static_cast<size_t>(g) * samp::kCap);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  double vx = v[0], vy = v[1], vz = v[2];
  VoxelOut o = out;
  void* args[] = {&points, &n, &vx, &vy, &vz, &batch, &bounds, &counters, &counts, &last, &region, &o};
  PCE_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&k_voxelise_buckets), dim3(g), dim3(samp::kThreads), args, sizeof(samp::Shared), st));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

// Results of more points than a cooperative grid holds in registers, from the 32-bit arrays of the library sort.
__global__ void k_voxel_widen(const int4* __restrict__ coords, const int* __restrict__ index, const int* __restrict__ inverse, int n,
                              VoxelOut out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int4 c = coords[i];  // (rows behind the last voxel are copied too: they are not part of the result)
  int* v = out.voxels + static_cast<size_t>(i) * out.width;
  v[0] = c.y;
  v[1] = c.z;
  v[2] = c.w;
  if (out.index) put_int(out.index, out.wide, i, index[i]);
  if (out.inverse) put_int(out.inverse, out.wide, i, inverse[i]);
}

template <int ITEMS>
static int launch_voxelise(const float* points, int n, const float* v, int batch, Arena& ar, const VoxelOut& out, cudaStream_t st) {
  int g = div_up(n, coop::kThreads * ITEMS);
  unsigned long long* key0 = ar.take<unsigned long long>(n);
  unsigned long long* key1 = ar.take<unsigned long long>(n);
  int* val0 = ar.take<int>(n);
  int* val1 = ar.take<int>(n);
  int* bounds = ar.take<int>(static_cast<size_t>(g) * 8);
  int* hist = ar.take<int>(static_cast<size_t>(g) * 256);
  int* counts = ar.take<int>(g);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  double vx = v[0], vy = v[1], vz = v[2];
  VoxelOut o = out;
  void* args[] = {&points, &n, &vx, &vy, &vz, &batch, &key0, &key1, &val0, &val1, &bounds, &hist, &counts, &o};
  PCE_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&k_voxelise<ITEMS>), dim3(g), dim3(coop::kThreads), args, 0, st));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

static int quantize_by_sort(const float* points, int n, const float* voxel, int batch, void* workspace, size_t workspace_bytes,
                            int32_t* out_coords, int32_t* out_index, int32_t* out_inverse, int* n_unique, cudaStream_t st) {
  if (off16(out_coords)) return PCE_ERR_INVALID;
  Arena ar(workspace, workspace_bytes);
  unsigned long long* keys = ar.take<unsigned long long>(n);
  unsigned long long* skeys = ar.take<unsigned long long>(n);
  int* vals = ar.take<int>(n);
  int* src = ar.take<int>(n);
  int* heads = ar.take<int>(n);
  int* rank = ar.take<int>(n);
  int* small = ar.take<int>(64);  // [0] status, [1] n_unique
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  PCE_CUDA(cudaMemsetAsync(small, 0, 2 * sizeof(int), st));
  k_voxel_keys<<<div_up(n, 256), 256, 0, st>>>(points, n, static_cast<double>(voxel[0]), static_cast<double>(voxel[1]),
                                                static_cast<double>(voxel[2]), batch, keys, vals, small);
  PCE_LAUNCH_CHECK();
  size_t need = 0, need_scan = 0;
  PCE_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, need, keys, skeys, vals, src, n, 0, 64, st));
  PCE_CUDA(cub::DeviceScan::InclusiveSum(nullptr, need_scan, heads, rank, n, st));
  if (need_scan > need) need = need_scan;
  char* tmp = ar.take<char>(need);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  PCE_CUDA(cub::DeviceRadixSort::SortPairs(tmp, need, keys, skeys, vals, src, n, 0, 64, st));  // stable
  k_voxel_heads<<<div_up(n, 256), 256, 0, st>>>(skeys, n, heads);
  PCE_LAUNCH_CHECK();
  PCE_CUDA(cub::DeviceScan::InclusiveSum(tmp, need, heads, rank, n, st));
  k_voxel_emit<<<div_up(n, 256), 256, 0, st>>>(skeys, src, heads, rank, n, reinterpret_cast<int4*>(out_coords), out_index,
                                               out_inverse, small + 1);
  PCE_LAUNCH_CHECK();
  int host[2] = {0, 0};
  PCE_CUDA(cudaMemcpyAsync(host, small, sizeof(host), cudaMemcpyDeviceToHost, st));
  PCE_CUDA(cudaStreamSynchronize(st));
  if (host[0] != 0) return host[0];
  *n_unique = host[1];
  return PCE_OK;
}

static int voxelise(const float* points, int n, const float* voxel, int batch, void* workspace, size_t workspace_bytes, VoxelOut out,
                    int* n_unique, cudaStream_t st) {
  const int items = coop::items_for(n, device_sm_count());
  if (items == 0) {  // more than about 1.2 million points
    if (!out.wide && out.width == 4)
      return quantize_by_sort(points, n, voxel, batch, workspace, workspace_bytes, out.voxels, static_cast<int*>(out.index),
                              static_cast<int*>(out.inverse), n_unique, st);
    Arena ar(workspace, workspace_bytes);
    int* coords = ar.take<int>(4 * static_cast<size_t>(n));
    int* index = ar.take<int>(n);
    int* inverse = ar.take<int>(n);
    if (!ar.ok) return PCE_ERR_WORKSPACE;
    PCE_TRY(quantize_by_sort(points, n, voxel, batch, static_cast<char*>(workspace) + ar.off, ar.left(), coords, index, inverse,
                             n_unique, st));
    k_voxel_widen<<<div_up(n, 256), 256, 0, st>>>(reinterpret_cast<const int4*>(coords), index, inverse, n, out);
    PCE_LAUNCH_CHECK();
    return PCE_OK;
  }
  int* host = thread_words();  // (mapped: the kernel writes the two words itself)
  if (!host) return PCE_ERR_CUDA;
  PCE_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&out.host), host, 0));
  host[0] = PCE_ERR_CUDA;
  if (div_up(n, samp::kTarget) <= std::min(device_sm_count(), samp::kMaxBuckets)) {
    Arena room(workspace, workspace_bytes);
    const int bucketed = launch_buckets(points, n, voxel, batch, room, out, st);
    if (bucketed == PCE_OK) {
      PCE_CUDA(cudaStreamSynchronize(st));
      if (host[0] != kTryRadix) {
        if (host[0] != PCE_OK) return host[0];
        *n_unique = host[1];
        return PCE_OK;
      }
      host[0] = PCE_ERR_CUDA;
    } else if (bucketed != PCE_ERR_WORKSPACE) {
      return bucketed;
    }
  }
  Arena ar(workspace, workspace_bytes);
  int status;
  if (items == 2) status = launch_voxelise<2>(points, n, voxel, batch, ar, out, st);
  else if (items == 4) status = launch_voxelise<4>(points, n, voxel, batch, ar, out, st);
  else if (items == 8) status = launch_voxelise<8>(points, n, voxel, batch, ar, out, st);
  else status = launch_voxelise<16>(points, n, voxel, batch, ar, out, st);
  if (status != PCE_OK) return status;
  PCE_CUDA(cudaStreamSynchronize(st));
  if (host[0] != PCE_OK) return host[0];
  *n_unique = host[1];
  return PCE_OK;
}

}  // namespace pce

using namespace pce;

extern "C" {

size_t pce_quantize_workspace_bytes(int32_t n) {
  const size_t m = n > 0 ? static_cast<size_t>(n) : 1;
  return 2 * pad256(8 * m) + 10 * pad256(4 * m) + 16 * m + (8u << 20) + 4096;  // (the bucket form: 32 bytes a point and 48 KB)
}

int pce_quantize_unique(const float* points, int32_t n, const float* voxel_host, int32_t batch, void* workspace,
                        size_t workspace_bytes, int32_t* out_coords, int32_t* out_index, int32_t* out_inverse,
                        int32_t* n_unique_host, void* stream) {
  if (!n_unique_host || n < 0 || !voxel_host || batch < 0) return PCE_ERR_INVALID;
  *n_unique_host = 0;
  if (n == 0) return PCE_OK;
  if (!points || !out_coords) return PCE_ERR_INVALID;
  for (int d = 0; d < 3; ++d)
    if (!(voxel_host[d] > 0.f)) return PCE_ERR_INVALID;
  const VoxelOut out{out_coords, 4, out_index, out_inverse, 0, nullptr};
  return voxelise(points, n, voxel_host, batch, workspace, workspace_bytes, out, n_unique_host, static_cast<cudaStream_t>(stream));
}

int pce_voxelise(const float* points, int32_t n, const float* voxel_host, void* workspace, size_t workspace_bytes,
                 int32_t* out_voxels, int64_t* out_index, int64_t* out_inverse, int32_t* n_unique_host, void* stream) {
  if (!n_unique_host || n < 0 || !voxel_host) return PCE_ERR_INVALID;
  *n_unique_host = 0;
  if (n == 0) return PCE_OK;
  if (!points || !out_voxels) return PCE_ERR_INVALID;
  for (int d = 0; d < 3; ++d)
    if (!(voxel_host[d] > 0.f)) return PCE_ERR_INVALID;
  const VoxelOut out{out_voxels, 3, out_index, out_inverse, 1, nullptr};
  return voxelise(points, n, voxel_host, 0, workspace, workspace_bytes, out, n_unique_host, static_cast<cudaStream_t>(stream));
}

// ---- collation ---------------------------------------------------------------------------------

constexpr int kCollateMax = 64;  // samples per launch: their addresses and row offsets travel as a kernel parameter
struct CollateArgs {
  const int* coords[kCollateMax];
  int first[kCollateMax + 1];  // first output row of every sample
  int n_samples, width, batch0;
};

}  // extern "C"

namespace pce {
// (batch, x, y, z) rows of up to 64 samples, and the maximum of every coordinate.
__global__ void __launch_bounds__(256) k_collate(const __grid_constant__ CollateArgs a, int4* __restrict__ out, int* __restrict__ cmax) {
  const unsigned rows = a.first[a.n_samples];
  int m[3] = {static_cast<int>(0x80000000), static_cast<int>(0x80000000), static_cast<int>(0x80000000)};
  for (unsigned i = blockIdx.x * 256 + threadIdx.x; i < rows; i += gridDim.x * 256) {  // (int would wrap near 2^31 rows)
    int lo = 0, hi = a.n_samples;  // last sample whose first row is not behind i
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (static_cast<unsigned>(a.first[mid]) <= i)
        lo = mid;
      else
        hi = mid;
    }
    const int* c = a.coords[lo] + static_cast<size_t>(i - a.first[lo]) * a.width + (a.width - 3);
    const int x = __ldg(c), y = __ldg(c + 1), z = __ldg(c + 2);
    out[i] = make_int4(a.batch0 + lo, x, y, z);
    m[0] = max(m[0], x);
    m[1] = max(m[1], y);
    m[2] = max(m[2], z);
  }
  __shared__ int s_max[8][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int v = __reduce_max_sync(0xFFFFFFFFu, m[d]);
    if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5][d] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {  // one update per block and axis
    int v = s_max[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) v = max(v, s_max[w][threadIdx.x]);
    atomicMax(cmax + threadIdx.x, v);
  }
}
}  // namespace pce

extern "C" int pce_collate_coords(const int32_t* const* coords, const int32_t* rows, int32_t n_samples, int32_t width,
                                  int32_t* out_coords, int32_t* scratch, int32_t* cmax_host, void* stream) {
  if (!coords || !rows || n_samples < 1 || width < 3 || !out_coords || !scratch || !cmax_host || off16(out_coords))
    return PCE_ERR_INVALID;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PCE_CUDA(cudaMemsetAsync(scratch, 0x80, 3 * sizeof(int), st));  // 0x80808080: below every packable coordinate
  size_t done = 0;
  for (int s0 = 0; s0 < n_samples; s0 += kCollateMax) {
    CollateArgs a;
    a.n_samples = n_samples - s0 < kCollateMax ? n_samples - s0 : kCollateMax;
    a.width = width;
    a.batch0 = s0;
    a.first[0] = 0;
    for (int k = 0; k < a.n_samples; ++k) {
      if (rows[s0 + k] < 0 || (rows[s0 + k] > 0 && !coords[s0 + k])) return PCE_ERR_INVALID;
      a.coords[k] = coords[s0 + k];
      if (static_cast<long long>(a.first[k]) + rows[s0 + k] >= (1ll << 31)) return PCE_ERR_UNSUPPORTED;
      a.first[k + 1] = a.first[k] + rows[s0 + k];
    }
    const int total = a.first[a.n_samples];
    if (total > 0) {
      const int grid = std::min(div_up(total, 256), 148 * 4);
      k_collate<<<grid, 256, 0, st>>>(a, reinterpret_cast<int4*>(out_coords) + done, scratch);
      PCE_LAUNCH_CHECK();
    }
    done += total;
  }
  int* host = thread_words();
  if (!host) return PCE_ERR_CUDA;
  PCE_CUDA(cudaMemcpyAsync(host, scratch, 3 * sizeof(int), cudaMemcpyDeviceToHost, st));
  PCE_CUDA(cudaStreamSynchronize(st));
  for (int d = 0; d < 3; ++d) cmax_host[d] = host[d];
  return PCE_OK;
}

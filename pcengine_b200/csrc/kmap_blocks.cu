// Kernel maps through a table of occupied 4x4x4 blocks.
//
// A submanifold map asks, for every voxel, which of its kv neighbours exist.  With one hash entry per voxel that is a
// probe per (voxel, offset): 13 random 16-byte loads per voxel for 3x3x3 with mirroring, 62 for 5x5x5 (1.2 ms for 1.5 M
// voxels), and a dense [kv][N] table written and read twice.  Here an entry is a BLOCK of 4x4x4 voxels: its key, the
// 64-bit occupancy of its voxels and the place of its first voxel in a compact row table, 32 bytes, one sector.  The
// neighbourhood of a voxel lies in at most 8 blocks (3.4 on average for 3x3x3): all presence bits follow from their
// occupancies by shifts, and a present neighbour's row is one load at (place + number of lower bits).  The kernel that
// probes writes what the tile lists are made of: the bitmask, the neighbours one after the other (rows of a thread
// block together, where they start is kept per row) and how many rows have each offset.  The dense table is only
// written for callers that ask for it (pce_map_build_d2), from the same probes.
//
// Down-sampling layers whose kernel size equals their stride (every voxel has exactly one parent) insert the parents of
// ALL levels in one pass over the input: a voxel that sets its parent's bit first goes on to the grandparent.  One
// cooperative kernel then sorts the levels' voxels (one radix sort, the level in the key's top bits) into the
// ascending order the maps are defined in; the tables serve the queries of their levels.
//
// Limits of the block form: odd kernel sizes up to 5 per axis (at most two blocks per axis), parents for kernel ==
// stride without padding.  Everything else runs through kmap.cu.
#include <algorithm>

#include "common.cuh"
#include "coop_sort.cuh"
#include "kmap_blocks.cuh"

namespace pce {

int fill_tile_lists(const uint32_t* mask, const int32_t* starts, const int32_t* nbr, const int32_t* table, const int32_t* order,
                    int32_t n_rows, int32_t kv, int32_t tile_rows, int32_t identity_stage, int32_t slots, const int32_t* tile_ptr,
                    int32_t* stage_kp, int32_t* stage_nbr, int32_t stage_cap, cudaStream_t st);

namespace blk {

// ---- the table --------------------------------------------------------------------------------------------

// Voxels are addressed with a bias of 2^15 per axis (as pack_key), so block coordinates are 14 bits.  Keys are stored
// plus one: an all-zero table is empty.
__device__ __forceinline__ unsigned long long block_key(int b, int bx, int by, int bz) {
  return ((((static_cast<unsigned long long>(static_cast<unsigned>(b)) << 14 | static_cast<unsigned>(bx)) << 14) |
           static_cast<unsigned>(by))
          << 14 | static_cast<unsigned>(bz)) +
         1ull;
}

// A longer chain means that the table is too full.  The input level's tables never are (table_slots); those of the coarser
// levels are sized for the clouds that occur, and give up early.
constexpr int kMaxProbes = 2048, kMaxProbesUp = 128;

__device__ __forceinline__ unsigned slot_of(unsigned long long key1, unsigned tmask) {
  return static_cast<unsigned>(mix64(key1)) & tmask;
}

// Slot of `key1`, claimed when it is new; ~0u when the table is too full.
__device__ __forceinline__ unsigned claim(Block* t, unsigned tmask, unsigned long long key1, int most) {
  unsigned s = slot_of(key1, tmask);
  for (int n = 0; n < most; ++n) {
    const unsigned long long prev = atomicCAS(&t[s].key, 0ull, key1);
    if (prev == 0ull || prev == key1) return s;
    s = (s + 1) & tmask;
  }
  return ~0u;
}

__device__ __forceinline__ void load_block(const Block* t, unsigned s, unsigned long long& key, unsigned long long& mask, int& base) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(t + s));
  base = __ldg(reinterpret_cast<const int*>(t + s) + 4);
  key = static_cast<unsigned long long>(a.y) << 32 | a.x;
  mask = static_cast<unsigned long long>(a.w) << 32 | a.z;
}

// Row of voxel (b, x, y, z) (biased coordinates), or -1.
__device__ __forceinline__ int find_row(const Block* t, unsigned tmask, const int* perm, int b, int x, int y, int z) {
  const unsigned long long want = block_key(b, x >> 2, y >> 2, z >> 2);
  unsigned s = slot_of(want, tmask);
  for (int n = 0; n < kMaxProbes; ++n) {
    unsigned long long key, mask;
    int base;
    load_block(t, s, key, mask, base);
    if (key == want) {
      const int bit = ((x & 3) << 4) | ((y & 3) << 2) | (z & 3);
      if (!((mask >> bit) & 1ull)) return -1;
      return __ldg(perm + base + __popcll(mask & ((1ull << bit) - 1ull)));
    }
    if (key == 0ull) return -1;
    s = (s + 1) & tmask;
  }
  return -1;
}

// ---- insertion ----------------------------------------------------------------------------------------------

// Voxels of the input and of every coarser level.  Neighbouring rows usually share their block: a run of lanes with one
// block is combined to one pair of atomics, a run of equal (coarse) voxels to one lane.
// Row i of a warp's 32 consecutive ones (whole warps call it).
__device__ __forceinline__ void insert_row(const int4* __restrict__ coords, int n, const Levels& lv, unsigned* slot0, int* ctl, int i) {
  constexpr unsigned kFull = 0xFFFFFFFFu;
  const int lane = threadIdx.x & 31;
  bool active = i < n;
  int b = 0, x = 0, y = 0, z = 0;
  if (active) {
    const int4 c = __ldg(coords + i);
    b = c.x, x = c.y, y = c.z, z = c.w;
    if (!packable(b, x, y, z)) {
      atomicMax(ctl + kCtlStatus, PCE_ERR_RANGE);
      active = false;
      if (slot0) slot0[i] = ~0u;
    }
  }
  if (lv.n > 1) {
    const int top = __reduce_max_sync(kFull, active ? b : 0);
    if (lane == 0 && top > *reinterpret_cast<volatile int*>(ctl + kCtlMaxBatch)) atomicMax(ctl + kCtlMaxBatch, top);
  }
  for (int l = 0; l < lv.n; ++l) {
    const Level& L = lv.level[l];
    if (l > 0 && active) {
      // parent: the only offset that reaches an output is (x - omin) mod stride
      const int ax = x - L.omin[0], ay = y - L.omin[1], az = z - L.omin[2];
      const int rx = ((ax % L.st[0]) + L.st[0]) % L.st[0], ry = ((ay % L.st[1]) + L.st[1]) % L.st[1],
                rz = ((az % L.st[2]) + L.st[2]) % L.st[2];
      x = (ax - rx) / L.st[0];
      y = (ay - ry) / L.st[1];
      z = (az - rz) / L.st[2];
      active = x >= L.lo[0] && x <= L.hi[0] && y >= L.lo[1] && y <= L.hi[1] && z >= L.lo[2] && z <= L.hi[2];
      if (active && !packable(b, x, y, z)) {
        atomicMax(ctl + kCtlStatus, PCE_ERR_RANGE);
        active = false;
      }
    }
    if (L.table == nullptr) continue;
    if (__ballot_sync(kFull, active) == 0u) return;
    if (l > 0) {  // the chain may have failed already; other warps write the word meanwhile, so one lane reads it for all
      int status = lane == 0 ? *reinterpret_cast<volatile int*>(ctl + kCtlStatus) : 0;
      status = __shfl_sync(kFull, status, 0);
      if (status != PCE_OK) return;
    }
    const int ux = x + 32768, uy = y + 32768, uz = z + 32768;
    const unsigned long long key = active ? block_key(b, ux >> 2, uy >> 2, uz >> 2) : 0ull;
    const int bit = ((ux & 3) << 4) | ((uy & 3) << 2) | (uz & 3);
    const unsigned long long key_before = __shfl_up_sync(kFull, key, 1);
    const int bit_before = __shfl_up_sync(kFull, bit, 1);
    const bool head = lane == 0 || key != key_before;
    if (l > 0 && !head && bit == bit_before) active = false;  // the lane before stands for this voxel
    const unsigned heads = __ballot_sync(kFull, head);
    const int first = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));  // first lane of this run
    unsigned long long bits = active ? 1ull << bit : 0ull;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long more = __shfl_down_sync(kFull, bits, d);
      const int more_first = __shfl_down_sync(kFull, first, d);
      if (lane + d < 32 && more_first == first) bits |= more;
    }
    unsigned s = ~0u;
    unsigned long long old = 0;
    if (head && key != 0ull) {
      s = claim(L.table, L.tmask, key, l == 0 ? kMaxProbes : kMaxProbesUp);
      if (s != ~0u)
        old = atomicOr(&L.table[s].mask, bits);
      else
        atomicMax(ctl + kCtlStatus, PCE_ERR_TABLE_FULL);
    }
    s = __shfl_sync(kFull, s, first);
    old = __shfl_sync(kFull, old, first);
    if (l == 0 && slot0 && active) slot0[i] = s;
    active = active && s != ~0u && !((old >> bit) & 1ull);  // who sets a voxel's bit goes on to its parent
  }
}

__global__ void __launch_bounds__(256) k_block_insert(const int4* __restrict__ coords, int n, const __grid_constant__ Levels lv,
                                                      unsigned* slot0, int* ctl) {
  insert_row(coords, n, lv, slot0, ctl, blockIdx.x * blockDim.x + threadIdx.x);
}

// Places of the blocks' voxels in the compact row table of their level, and (levels >= 1) the sort keys of those voxels
// in that order.  blockIdx.y = level; levels >= 1 share one compact table.
__device__ __forceinline__ void place_blocks(const Levels& lv, const KeyFields& kf, unsigned long long* keys, int key_cap, int* ctl, int l) {
  __shared__ int warp_sum[8];
  __shared__ int s_base;
  const Level& L = lv.level[l];
  const unsigned slots = L.tmask + 1u;
  const unsigned stride = gridDim.x * 256u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (L.table == nullptr) return;
  for (unsigned s0 = blockIdx.x * 256u; s0 < slots; s0 += stride) {
    const unsigned s = s0 + threadIdx.x;
    unsigned long long key = 0, mask = 0;
    if (s < slots) {
      const uint4 a = *reinterpret_cast<const uint4*>(L.table + s);
      key = static_cast<unsigned long long>(a.y) << 32 | a.x;
      mask = static_cast<unsigned long long>(a.w) << 32 | a.z;
    }
    const int cnt = key ? __popcll(mask) : 0;
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += u;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int before = incl - cnt, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      before += w < warp ? warp_sum[w] : 0;
      total += warp_sum[w];
    }
    if (threadIdx.x == 0 && total) {
      s_base = atomicAdd(ctl + (l == 0 ? kCtlRows0 : kCtlRowsUp), total);
      if (l > 0) atomicAdd(ctl + kCtlLevel + l, total);
    }
    __syncthreads();
    if (cnt) {
      int at = s_base + before;
      L.table[s].base = at;
      if (l > 0) {
        const unsigned long long k = key - 1ull;
        const long long bx = static_cast<long long>((k >> 28) & 0x3FFF) * 4 - 32768 - L.lo[0];
        const long long by = static_cast<long long>((k >> 14) & 0x3FFF) * 4 - 32768 - L.lo[1];
        const long long bz = static_cast<long long>(k & 0x3FFF) * 4 - 32768 - L.lo[2];
        for (unsigned long long m = mask; m; m &= m - 1ull, ++at) {
          const int bit = __ffsll(static_cast<long long>(m)) - 1;
          if (at < key_cap)
            keys[at] = (static_cast<unsigned long long>(l) << kf.sh_level) | ((k >> 42) << kf.sh_b) |
                       (static_cast<unsigned long long>(bx + (bit >> 4)) << kf.sh_x) |
                       (static_cast<unsigned long long>(by + ((bit >> 2) & 3)) << kf.sh_y) |
                       static_cast<unsigned long long>(bz + (bit & 3));
        }
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_block_places(const __grid_constant__ Levels lv, const __grid_constant__ KeyFields kf,
                                                      unsigned long long* keys, int key_cap, int* ctl) {
  place_blocks(lv, kf, keys, key_cap, ctl, blockIdx.y);
}

// Compact row table of the input level.
__device__ __forceinline__ void row_place(const int4* __restrict__ coords, const Block* table, const unsigned* slot0, int* __restrict__ perm, int i) {
  const unsigned s = __ldcg(slot0 + i);
  if (s == ~0u) return;
  const int4 c = __ldg(coords + i);
  const uint4 a = __ldcg(reinterpret_cast<const uint4*>(table + s));
  const int base = __ldcg(reinterpret_cast<const int*>(table + s) + 4);
  const unsigned long long mask = static_cast<unsigned long long>(a.w) << 32 | a.z;
  const int bit = (((c.y + 32768) & 3) << 4) | (((c.z + 32768) & 3) << 2) | ((c.w + 32768) & 3);
  perm[base + __popcll(mask & ((1ull << bit) - 1ull))] = i;
}

__global__ void __launch_bounds__(256) k_block_rows(const int4* __restrict__ coords, int n, const Block* table, const unsigned* slot0,
                                                    int* __restrict__ perm) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < n) row_place(coords, table, slot0, perm, i);
}

// A single level's table and row table, cleared, filled, placed and listed by one cooperative kernel: for a layer's own map,
// whose small clouds wait for the host to queue two memsets and three kernels (a 16-channel fp32 layer on 20 k voxels, map
// included: 73.9 -> 64.5 us; 1.5 M voxels: 92 us so, 91 apart).  The planner's chain keeps them apart: a cooperative grid
// would wait there for the convolutions of the pass before it to leave that many SMs.
__global__ void __launch_bounds__(256) k_block_table(const int4* __restrict__ coords, int n, const __grid_constant__ Levels lv, unsigned* slot0,
                                                     int* perm, int* state, int state_words) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  const unsigned first = blockIdx.x * 256u + threadIdx.x, step = gridDim.x * 256u;
  uint4* table = reinterpret_cast<uint4*>(lv.level[0].table);
  const unsigned long long words = (static_cast<unsigned long long>(lv.level[0].tmask) + 1ull) * (sizeof(Block) / 16);
  for (unsigned long long i = first; i < words; i += step) table[i] = make_uint4(0u, 0u, 0u, 0u);
  for (unsigned i = first; i < static_cast<unsigned>(state_words); i += step) state[i] = 0;
  grid.sync();
  for (unsigned i = first; i < ((static_cast<unsigned>(n) + 31u) & ~31u); i += step) insert_row(coords, n, lv, slot0, state, static_cast<int>(i));
  grid.sync();
  const KeyFields none = {};
  place_blocks(lv, none, nullptr, 0, state, 0);
  grid.sync();
  for (unsigned i = first; i < static_cast<unsigned>(n); i += step) row_place(coords, lv.level[0].table, slot0, perm, static_cast<int>(i));
}

// ---- queries ------------------------------------------------------------------------------------------------

constexpr int kQueryThreads = 128;

// Occupancies and places of the (up to) eight blocks that the neighbourhood [l, l + k) of a voxel touches, left in
// shared memory as column `threadIdx.x` of [8][threads].  All first probes are in flight before the first is used.
__device__ __forceinline__ void gather_blocks(const Block* __restrict__ table, unsigned tmask, bool live, int b, int lx, int ly, int lz,
                                              int kx, int ky, int kz, unsigned long long (*s_mask)[kQueryThreads],
                                              int (*s_base)[kQueryThreads]) {
  const int bx = lx >> 2, by = ly >> 2, bz = lz >> 2;
  unsigned long long want[8], key[8], mask[8];
  int base[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int ix = c >> 2, iy = (c >> 1) & 1, iz = c & 1;
    const bool need = live && (!ix || (lx & 3) + kx > 4) && (!iy || (ly & 3) + ky > 4) && (!iz || (lz & 3) + kz > 4) &&
                      static_cast<unsigned>(bx + ix) < 16384u && static_cast<unsigned>(by + iy) < 16384u &&
                      static_cast<unsigned>(bz + iz) < 16384u;
    want[c] = need ? block_key(b, bx + ix, by + iy, bz + iz) : 0ull;
    key[c] = 0ull;
    mask[c] = 0ull;
    base[c] = 0;
    if (need) load_block(table, slot_of(want[c], tmask), key[c], mask[c], base[c]);
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    if (key[c] != want[c] && key[c] != 0ull) {  // another block sits there: follow the chain
      unsigned s = slot_of(want[c], tmask);
      for (int n = 1; n < kMaxProbes; ++n) {
        s = (s + 1) & tmask;
        load_block(table, s, key[c], mask[c], base[c]);
        if (key[c] == want[c] || key[c] == 0ull) break;
      }
    }
    s_mask[c][threadIdx.x] = (want[c] != 0ull && key[c] == want[c]) ? mask[c] : 0ull;
    s_base[c][threadIdx.x] = base[c];
  }
}

// Lane j of the result: bit j of every lane's word, lane i's at bit i.
__device__ __forceinline__ unsigned transpose_bits(unsigned w) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const unsigned m = s == 16 ? 0x0000FFFFu : s == 8 ? 0x00FF00FFu : s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
    const unsigned y = __shfl_xor_sync(0xFFFFFFFFu, w, s);
    w = lane & s ? (w & ~m) | ((y >> s) & m) : (w & m) | ((y & m) << s);
  }
  return w;
}

// K = 3 or 5: cubic kernels known at compile time; 0: sizes from the arguments.
// LISTS: bitmask, neighbours and where they start; counts[kp] += rows that have the offset.
// otherwise: the dense table map[kp][row] = the output the row feeds through kp (the neighbour at the mirrored offset),
// -1 absent, the centre's row left at -1; counts[kp] = its entries.
// Bound by the random table entries (eight per row) and by the rows read for the lists.  Four rows are read at a time, and
// with 3x3x3 the rows of an offset are counted on the transposed bitmask: 5x5x5 on 1.5 M rows 313 -> 286 us, 3x3x3 there
// 176 -> 169, on 20 k rows 9.5 -> 8.0 (eight at a time 302 / 169 / 7.9; 5x5x5 counted so 294).
template <int K, bool LISTS>
__global__ void __launch_bounds__(kQueryThreads)
    k_block_query(const int4* __restrict__ coords, int n, const __grid_constant__ Query q) {
  __shared__ unsigned long long s_mask[8][kQueryThreads];
  __shared__ int s_base[8][kQueryThreads];
  __shared__ int s_count[128];
  __shared__ int s_warp[kQueryThreads / 32];
  __shared__ int s_start;
  const int kx = K ? K : q.ks[0], ky = K ? K : q.ks[1], kz = K ? K : q.ks[2];
  const int kv = kx * ky * kz, mid = kv / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  s_count[tid] = 0;  // (kQueryThreads = 128 counters)
  int my_count[4] = {0, 0, 0, 0};  // lane kp & 31 counts offset kp over the warp's rows
  for (int i0 = blockIdx.x * kQueryThreads; i0 < n; i0 += gridDim.x * kQueryThreads) {
    const int i = i0 + tid;
    bool live = i < n;
    int4 c = make_int4(0, 0, 0, 0);
    if (live) {
      c = __ldg(coords + i);
      live = packable(c.x, c.y, c.z, c.w);
    }
    const int lx = c.y + 32768 - kx / 2, ly = c.z + 32768 - ky / 2, lz = c.w + 32768 - kz / 2;
    gather_blocks(q.table, q.tmask, live, c.x, lx, ly, lz, kx, ky, kz, s_mask, s_base);
    const int zs = lz & 3;
    // presence of the kz neighbours of column (dx, dy)
    auto column = [&](int dx, int dy) -> unsigned {
      const int X = (lx & 3) + dx, Y = (ly & 3) + dy;
      const int c0 = ((X >> 2) << 2) | ((Y >> 2) << 1);
      const int sh = ((X & 3) << 4) | ((Y & 3) << 2);
      const unsigned low = static_cast<unsigned>(s_mask[c0][tid] >> sh) & 15u;
      const unsigned high = static_cast<unsigned>(s_mask[c0 | 1][tid] >> sh) & 15u;
      return ((low | (high << 4)) >> zs) & ((1u << kz) - 1u);
    };
    auto row_of = [&](int dx, int dy, int dz) -> int {
      const int X = (lx & 3) + dx, Y = (ly & 3) + dy, Z = zs + dz;
      const int cc = ((X >> 2) << 2) | ((Y >> 2) << 1) | (Z >> 2);
      const int bit = ((X & 3) << 4) | ((Y & 3) << 2) | (Z & 3);
      return __ldg(q.perm + s_base[cc][tid] + __popcll(s_mask[cc][tid] & ((1ull << bit) - 1ull)));
    };
    unsigned long long m0 = 0, m1 = 0;  // presence bits, offset kp at bit kp
#pragma unroll
    for (int dx = 0; dx < (K ? K : 5); ++dx) {
      if (!K && dx >= kx) break;
#pragma unroll
      for (int dy = 0; dy < (K ? K : 5); ++dy) {
        if (!K && dy >= ky) break;
        const unsigned long long run = column(dx, dy);
        const int kp = (dx * ky + dy) * kz;
        if (kp < 64) {
          m0 |= run << kp;
          if (kp + kz > 64) m1 |= run >> (64 - kp);
        } else {
          m1 |= run << (kp - 64);
        }
      }
    }
    // rows per offset
#pragma unroll
    for (int w = 0; w < (K == 3 ? 1 : 4); ++w) {
      const unsigned word = static_cast<unsigned>(w < 2 ? m0 >> (32 * (w & 1)) : m1 >> (32 * (w & 1)));
      if (K == 3) {  // most of the 27 offsets occur among 32 rows; of 125 few do
        my_count[w] += __popc(transpose_bits(word));
        continue;
      }
      unsigned any = __reduce_or_sync(0xFFFFFFFFu, word);
      while (any) {
        const int bit = __ffs(any) - 1;
        any &= any - 1u;
        const int rows = __popc(__ballot_sync(0xFFFFFFFFu, (word >> bit) & 1u));
        if (lane == bit) my_count[w] += rows;
      }
    }
    if constexpr (LISTS) {
      const int cnt = __popcll(m0) + __popcll(m1);
      int incl = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += u;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      int before = incl - cnt, total = 0;
#pragma unroll
      for (int w = 0; w < kQueryThreads / 32; ++w) {
        before += w < warp ? s_warp[w] : 0;
        total += s_warp[w];
      }
      if (tid == 0) s_start = atomicAdd(q.cursor, total);
      __syncthreads();
      if (i < n) {
        int p = s_start + before;
        q.starts[i] = p;
        const int words = (kv + 31) / 32;
        unsigned* mk = q.mask + static_cast<size_t>(i) * words;
        mk[0] = static_cast<unsigned>(m0);
        if (K != 3) {
          if (words > 1) mk[1] = static_cast<unsigned>(m0 >> 32);
          if (words > 2) mk[2] = static_cast<unsigned>(m1);
          if (words > 3) mk[3] = static_cast<unsigned>(m1 >> 32);
        }
        // ascending offsets; within a column the neighbours of one block lie next to each other in the row table
        auto emit = [&](unsigned long long m, int off) {
          while (m) {
            int v[4];  // four rows read before the first is written
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              v[k] = -1;
              if (m) {
                const int kp = off + __ffsll(static_cast<long long>(m)) - 1;
                m &= m - 1ull;
                const int col = kp / kz;
                v[k] = row_of(col / ky, col % ky, kp - col * kz);
              }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (v[k] >= 0) q.nbr[p++] = v[k];
          }
        };
        emit(m0, 0);
        if (K != 3) emit(m1, 64);
      }
      __syncthreads();  // s_warp and s_start are reused
    } else if (i < n) {
      for (int kp = 0; kp < kv; ++kp) {
        int v = -1;
        const unsigned long long m = kp < 64 ? m0 >> kp : m1 >> (kp - 64);
        if (kp != mid && (m & 1ull)) {
          const int col = kp / kz;
          v = row_of(col / ky, col % ky, kp - col * kz);
        }
        q.map[static_cast<size_t>(kv - 1 - kp) * n + i] = v;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < (K == 3 ? 1 : 4); ++w)
    if (my_count[w]) atomicAdd(&s_count[32 * w + lane], my_count[w]);
  __syncthreads();
  if (tid < kv && s_count[tid]) {
    if (LISTS)
      atomicAdd(q.counts + tid, s_count[tid]);
    else if (tid != mid)
      atomicAdd(q.counts + (kv - 1 - tid), s_count[tid]);
  }
}

// ---- coarser levels in order ----------------------------------------------------------------------------------

// All voxels of the levels >= 1, sorted (level first): coordinates of every level in ascending (b,x,y,z) order, one level
// after the other, and the rows they got in the compact row table.  `host` (mapped): status, largest batch index,
// then the rows of every level.
__global__ void __launch_bounds__(coop::kThreads)
    k_level_sort(const unsigned long long* __restrict__ keys, unsigned long long* key0, unsigned long long* key1, int* val0, int* val1,
                 int* hist, const __grid_constant__ Levels lv, const __grid_constant__ KeyFields kf, int key_cap, int4* coords,
                 int* perm, int* ctl, int* host) {
  using namespace coop;
  __shared__ SortShared<8> sh;
  cg::grid_group grid = cg::this_grid();
  const int status = __ldcg(ctl + kCtlStatus);
  const int n = __ldcg(ctl + kCtlRowsUp), top = __ldcg(ctl + kCtlMaxBatch);
  if (status != PCE_OK || n > key_cap) {  // the same for every block
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      host[0] = status != PCE_OK ? status : PCE_ERR_TABLE_FULL;
      __threadfence_system();
    }
    return;
  }
  // the batch field ends at its highest index, the level field starts there (kf.sh_level leaves room for 16 bits)
  const int batch_bits = 32 - __clz(top);
  const int level_bits = lv.n > 2 ? 32 - __clz(lv.n - 1) : 0;  // one level: nothing to tell apart
  const int low_bits = kf.sh_b + batch_bits;
  auto squeeze = [&](unsigned long long k) {  // drops the unused bits between batch and level
    const unsigned long long level = k >> kf.sh_level;
    return (level << low_bits) | (k & ((1ull << low_bits) - 1ull));
  };
  const int passes = max(1, (low_bits + level_bits + 7) / 8);
  for (int p = 0; p < passes; ++p) {
    const unsigned long long* kin = p & 1 ? key0 : key1;
    const int* vin = p & 1 ? val0 : val1;
    sort_pass_any<8, unsigned long long>(
        grid, sh, hist, n, 8 * p,
        [&](int i, unsigned long long& k, int& v) {
          if (p == 0) {
            k = squeeze(__ldcg(keys + i));
            v = i;
          } else {
            k = __ldcg(kin + i);
            v = __ldcg(vin + i);
          }
        },
        p & 1 ? key1 : key0, p & 1 ? val1 : val0);
  }
  const unsigned long long* sorted = passes & 1 ? key0 : key1;
  const int* from = passes & 1 ? val0 : val1;
  int off[kMaxLevels];
  {
    int run = 0;
#pragma unroll
    for (int l = 1; l < kMaxLevels; ++l) {
      off[l] = run;
      if (l < lv.n) run += __ldcg(ctl + kCtlLevel + l);
    }
  }
  const unsigned long long mx = (1ull << (kf.sh_b - kf.sh_x)) - 1, my = (1ull << (kf.sh_x - kf.sh_y)) - 1, mz = (1ull << kf.sh_y) - 1;
  for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
    const unsigned long long k = __ldcg(sorted + i);
    const int l = lv.n > 2 ? static_cast<int>(k >> low_bits) : 1;
    int lo0 = 0, lo1 = 0, lo2 = 0, first = 0;
#pragma unroll
    for (int u = 1; u < kMaxLevels; ++u) {
      if (u == l) {
        lo0 = lv.level[u].lo[0];
        lo1 = lv.level[u].lo[1];
        lo2 = lv.level[u].lo[2];
        first = off[u];
      }
    }
    coords[i] = make_int4(static_cast<int>((k >> kf.sh_b) & ((1ull << batch_bits) - 1ull)), static_cast<int>((k >> kf.sh_x) & mx) + lo0,
                          static_cast<int>((k >> kf.sh_y) & my) + lo1, static_cast<int>(k & mz) + lo2);
    perm[__ldcg(from + i)] = i - first;
  }
  if (blockIdx.x == 0 && threadIdx.x < kMaxLevels) {
    const int l = threadIdx.x;
    if (l >= 1 && l < lv.n) host[2 + l] = __ldcg(ctl + kCtlLevel + l);
    if (l == 0) {
      host[0] = PCE_OK;
      host[1] = top;
    }
  }
}

// ---- parents ------------------------------------------------------------------------------------------------

// The map between a level and its parents (kernel == stride): every row has at most one pair, with its parent through
// the offset that is its position inside the parent.
//   up:   the rows as outputs (transposed layer): mask = that one bit, nbr = the parent
//   down: child[kp][parent] = row (preset to -1 by the caller)
//   dense: map[kp][row] = parent, for every kp
// counts[kp] += rows with the offset.
__global__ void __launch_bounds__(256) k_parents(const int4* __restrict__ coords, int n, const __grid_constant__ Level L,
                                                 const int* __restrict__ perm, int kv, int n_parents, unsigned* up_mask, int* up_nbr,
                                                 int* child, int* counts) {
  __shared__ int s_count[32];
  if (threadIdx.x < 32) s_count[threadIdx.x] = 0;
  __syncthreads();
  const int i = blockIdx.x * 256 + threadIdx.x;
  int kp = -1, row = -1;
  if (i < n) {
    const int4 c = __ldg(coords + i);
    const int ax = c.y - L.omin[0], ay = c.z - L.omin[1], az = c.w - L.omin[2];
    const int rx = ((ax % L.st[0]) + L.st[0]) % L.st[0], ry = ((ay % L.st[1]) + L.st[1]) % L.st[1],
              rz = ((az % L.st[2]) + L.st[2]) % L.st[2];
    const int x = (ax - rx) / L.st[0], y = (ay - ry) / L.st[1], z = (az - rz) / L.st[2];
    if (x >= L.lo[0] && x <= L.hi[0] && y >= L.lo[1] && y <= L.hi[1] && z >= L.lo[2] && z <= L.hi[2] && packable(c.x, x, y, z)) {
      row = find_row(L.table, L.tmask, perm, c.x, x + 32768, y + 32768, z + 32768);
      if (row >= 0) kp = (rx * L.st[1] + ry) * L.st[2] + rz;
    }
    if (up_mask) up_mask[i] = kp >= 0 ? 1u << kp : 0u;
    if (up_nbr) up_nbr[i] = row;
    if (kp >= 0 && child) child[static_cast<size_t>(kp) * n_parents + row] = i;
  }
  const unsigned lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xFFFFFFFFu, kp);
  if (kp >= 0 && (same & ((1u << lane) - 1u)) == 0) atomicAdd(&s_count[kp], __popc(same));
  __syncthreads();
  if (threadIdx.x < kv && s_count[threadIdx.x]) atomicAdd(counts + threadIdx.x, s_count[threadIdx.x]);
}

// ---- row order and stages per tile ------------------------------------------------------------------------------

// The row order (rows sorted by bitmask, its bits permuted so that the rarest offset is the most significant one; stable)
// and tile_ptr of up to kMaxVariants (tile height, identity stage, offsets per stage) of ONE direction of a map with at most 32
// offsets; the stages themselves are then filled by k_tile_lists (kmap.cu) over the whole GPU.  Two kernels: maps of up
// to 64 k rows are sorted by ONE cluster of eight blocks (keys in registers, digit counts and the scatter itself through
// distributed shared memory: nothing waits for L2 or for a grid barrier), larger ones by a cooperative grid.  The
// library's sort is four passes of 9-11 us, a histogram, a scan and a dozen memsets for the same order.
constexpr int kOrderBits = 9;  // 27 offsets in three passes

// Bit position in the sort key of every offset, from the number of rows that have it (lane = offset, warp-wide).
__device__ __forceinline__ int key_bit(int mine, int lane, int kv) {
  int rank = 0;  // rarer offsets (ties: lower ones) come first
  for (int j = 0; j < kv; ++j) {
    const int cj = __shfl_sync(0xFFFFFFFFu, mine, j);
    rank += (cj < mine || (cj == mine && j < lane)) ? 1 : 0;
  }
  return lane < kv ? kv - 1 - rank : 0;
}

__device__ __forceinline__ unsigned mask_of_row(const Order& o, int i) {
  if (!o.table) return __ldg(o.mask + i);
  unsigned m = 0;
  for (int k = 0; k < o.kv; ++k)
    if (__ldg(o.table + static_cast<size_t>(k) * o.n + i) >= 0) m |= 1u << k;
  return m;
}

__device__ __forceinline__ unsigned key_of_mask(unsigned m, const int* pos) {
  unsigned key = 0;
  for (; m; m &= m - 1u) key |= 1u << pos[__ffs(m) - 1];
  return key;
}

// ---- up to 64 k rows: one cluster ----
constexpr int kClusterBlocks = 8, kClusterThreads = 1024, kClusterWarps = 32, kClusterItems = 8;
constexpr int kClusterRows = kClusterBlocks * kClusterThreads * kClusterItems;
constexpr int kClusterRowsAlone = 24576;  // with the GPU to itself, more blocks end sooner from there on (60 k rows: 51 us, 31)
constexpr int kClusterBins = 1 << kOrderBits;

struct ClusterShared {
  uint2 entry[kClusterThreads * kClusterItems];  // (key, row)
  unsigned short count[kClusterWarps][kClusterBins];  // (a block has at most 8192 rows)
  int total[kClusterBins];                             // read by the other blocks
  int base[kClusterBins];
  int half[2][kClusterBins];
  unsigned group_mask[kClusterThreads * kClusterItems / 32];
  int warp_sum[kClusterWarps];
  int rows_with[32];                                   // read by the other blocks
  int pos[32];
  int stages[kMaxVariants];                            // read by the other blocks
};

__global__ void __cluster_dims__(kClusterBlocks, 1, 1) __launch_bounds__(kClusterThreads) k_order_cluster(const __grid_constant__ Order o) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ClusterShared& sh = *reinterpret_cast<ClusterShared*>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int me = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = o.n, kv = o.kv;
  // rows per warp: a multiple of 32 as small as covers n, so that all blocks take part
  const int items = (n + kClusterBlocks * kClusterThreads - 1) / (kClusterBlocks * kClusterThreads);
  const int chunk = items * kClusterThreads;          // rows per block, a multiple of every tile height
  const int local0 = warp * (32 * items) + lane;      // this thread's first row inside the block
  const int row0 = me * chunk;
  unsigned key[kClusterItems];
  int val[kClusterItems];
#pragma unroll
  for (int j = 0; j < kClusterItems; ++j) {
    const int i = row0 + local0 + 32 * j;
    key[j] = 0u;
    val[j] = i;
    if (j < items && i < n) {
      key[j] = mask_of_row(o, i);
      if (o.table) o.mask[i] = key[j];
    }
  }
  int mine = 0;
  if (o.counts) {
    if (warp == 0) mine = lane < kv ? __ldg(o.counts + lane) : 0;
  } else {
    if (tid < 32) sh.rows_with[tid] = 0;
    __syncthreads();
    int c = 0;
#pragma unroll
    for (int j = 0; j < kClusterItems; ++j) {
      unsigned any = __reduce_or_sync(0xFFFFFFFFu, key[j]);
      for (; any; any &= any - 1u) {
        const int bit = __ffs(any) - 1;
        const int rows = __popc(__ballot_sync(0xFFFFFFFFu, (key[j] >> bit) & 1u));
        if (lane == bit) c += rows;
      }
    }
    if (c) atomicAdd(&sh.rows_with[lane], c);
    cluster.sync();
    if (warp == 0)
      for (int r = 0; r < kClusterBlocks; ++r) mine += cluster.map_shared_rank(sh.rows_with, r)[lane];
  }
  if (warp == 0) sh.pos[lane] = key_bit(mine, lane, kv);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kClusterItems; ++j) key[j] = key_of_mask(key[j], sh.pos);
  const int passes = (kv + kOrderBits - 1) / kOrderBits;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * kOrderBits;
    for (int i = tid; i < kClusterWarps * kClusterBins / 2; i += kClusterThreads) reinterpret_cast<unsigned*>(&sh.count[0][0])[i] = 0u;
    __syncthreads();
    int rank[kClusterItems];
#pragma unroll
    for (int j = 0; j < kClusterItems; ++j) {
      rank[j] = 0;
      if (j < items) {
        const bool live = row0 + local0 + 32 * j < n;
        const int d = live ? static_cast<int>((key[j] >> shift) & (kClusterBins - 1)) : kClusterBins + lane;
        const unsigned same = __match_any_sync(0xFFFFFFFFu, d);
        const unsigned before = same & ((1u << lane) - 1u);
        const int old = live ? sh.count[warp][d] : 0;
        __syncwarp();
        if (live && before == 0) sh.count[warp][d] = static_cast<unsigned short>(old + __popc(same));
        __syncwarp();
        rank[j] = old + __popc(before);
      }
    }
    __syncthreads();
    {  // per digit: offsets of the warps (two threads per digit, half the warps each) and the block's total
      const int d = tid & (kClusterBins - 1), h = tid / kClusterBins;
      int sum = 0;
#pragma unroll
      for (int w = 0; w < kClusterWarps / 2; ++w) sum += sh.count[h * (kClusterWarps / 2) + w][d];
      sh.half[h][d] = sum;
      __syncthreads();
      int run = h ? sh.half[0][d] : 0;
#pragma unroll
      for (int w = 0; w < kClusterWarps / 2; ++w) {
        const int c = sh.count[h * (kClusterWarps / 2) + w][d];
        sh.count[h * (kClusterWarps / 2) + w][d] = static_cast<unsigned short>(run);
        run += c;
      }
      if (h) sh.total[d] = run;
    }
    cluster.sync();
    {
      int pre = 0, all = 0;
      if (tid < kClusterBins) {
#pragma unroll
        for (int r = 0; r < kClusterBlocks; ++r) {
          const int c = cluster.map_shared_rank(sh.total, r)[tid];
          all += c;
          pre += r < me ? c : 0;
        }
      }
      int incl = all;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += u;
      }
      if (lane == 31) sh.warp_sum[warp] = incl;
      __syncthreads();
      int lower = incl - all;
      for (int w = 0; w < warp; ++w) lower += sh.warp_sum[w];
      if (tid < kClusterBins) sh.base[tid] = lower + pre;
      __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < kClusterItems; ++j) {
      if (j < items && row0 + local0 + 32 * j < n) {
        const int d = static_cast<int>((key[j] >> shift) & (kClusterBins - 1));
        const int at = sh.base[d] + sh.count[warp][d] + rank[j];
        const int to = at / chunk, in = at - to * chunk;
        // one store for both: remote stores to scattered words are what a pass takes (32 lanes, 32 words, one at a time)
        cluster.map_shared_rank(sh.entry, to)[in] = make_uint2(key[j], static_cast<unsigned>(val[j]));
      }
    }
    cluster.sync();
#pragma unroll
    for (int j = 0; j < kClusterItems; ++j) {
      const int i = local0 + 32 * j;
      if (j < items && row0 + i < n) {
        const uint2 e = sh.entry[i];
        key[j] = e.x;
        val[j] = static_cast<int>(e.y);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kClusterItems; ++j) {
    const int i = local0 + 32 * j;
    const bool live = j < items && row0 + i < n;
    if (live) o.order[row0 + i] = val[j];
    const unsigned m = __reduce_or_sync(0xFFFFFFFFu, live ? key[j] : 0u);
    if (j < items && lane == 0) sh.group_mask[i / 32] = m;
  }
  __syncthreads();
  // stages of the block's tiles: warp v counts variant v, two 128-row tiles per lane at most
  int count[2] = {0, 0}, before = 0;
  if (warp < o.n_variants) {
    const Variant& V = o.variant[warp];
    const int tiles = chunk / V.tile_rows, groups = V.tile_rows / 32;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = 2 * lane + u;
      if (t < tiles && row0 + t * V.tile_rows < n) {
        unsigned m = 0u;
        for (int q = 0; q < groups; ++q) m |= sh.group_mask[t * groups + q];
        count[u] = (__popc(m) + V.slots - 1) / V.slots + V.identity;
      }
    }
    int incl = count[0] + count[1];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += u;
    }
    before = incl - count[0] - count[1];
    if (lane == 31) sh.stages[warp] = incl;
  }
  cluster.sync();
  if (warp < o.n_variants) {
    const Variant& V = o.variant[warp];
    const int tiles = chunk / V.tile_rows;
    int all = 0;
    for (int r = 0; r < kClusterBlocks; ++r) {
      const int c = cluster.map_shared_rank(sh.stages, r)[warp];
      all += c;
      before += r < me ? c : 0;
    }
    const int t0 = row0 / V.tile_rows + 2 * lane;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (2 * lane + u < tiles && row0 + (2 * lane + u) * V.tile_rows < n) V.tile_ptr[t0 + u] = before;
      before += count[u];
    }
    if (me == 0 && lane == 0) V.tile_ptr[(n + V.tile_rows - 1) / V.tile_rows] = all;
  }
  cluster.sync();  // no block leaves while another reads its shared memory
}

// ---- more rows: a cooperative grid ----
struct GridShared {
  coop::SortShared<kOrderBits> sort;
  int pos[32];
  int sums[kMaxVariants];
};

__global__ void __launch_bounds__(coop::kThreads) k_order_grid(const __grid_constant__ Order o) {
  using namespace coop;
  __shared__ GridShared sh;
  cg::grid_group grid = cg::this_grid();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = o.n, kv = o.kv;
  const int g = static_cast<int>(gridDim.x);
  if (o.table)
    for (int i = blockIdx.x * kThreads + tid; i < n; i += g * kThreads) o.mask[i] = mask_of_row(o, i);
  if (!o.counts) {
    int mine = 0;
    for (int i0 = (blockIdx.x * kThreads + tid) & ~31; i0 < n; i0 += g * kThreads) {
      const unsigned m = i0 + lane < n ? o.mask[i0 + lane] : 0u;  // (a table's rows: written by this very thread above)
      unsigned any = __reduce_or_sync(0xFFFFFFFFu, m);
      for (; any; any &= any - 1u) {
        const int bit = __ffs(any) - 1;
        const int c = __popc(__ballot_sync(0xFFFFFFFFu, (m >> bit) & 1u));
        if (lane == bit) mine += c;
      }
    }
    if (tid < 32) sh.pos[tid] = 0;
    __syncthreads();
    if (mine) atomicAdd(&sh.pos[lane], mine);
    __syncthreads();
    if (tid < 32) o.block_counts[blockIdx.x * 32 + tid] = sh.pos[tid];
  }
  if (o.table || !o.counts) grid.sync();
  if (warp == 0) {
    int mine = 0;
    if (lane < kv) {
      if (o.counts) {
        mine = __ldg(o.counts + lane);
      } else {
        for (int b = 0; b < g; ++b) mine += __ldcg(o.block_counts + b * 32 + lane);
      }
    }
    sh.pos[lane] = key_bit(mine, lane, kv);
  }
  if (tid < kMaxVariants) sh.sums[tid] = 0;
  __syncthreads();
  const int passes = (kv + kOrderBits - 1) / kOrderBits;
  for (int p = 0; p < passes; ++p) {
    const unsigned* kin = p & 1 ? o.key0 : o.key1;
    const int* vin = p & 1 ? o.val0 : o.val1;
    sort_pass_any<kOrderBits, unsigned>(
        grid, sh.sort, o.hist, n, kOrderBits * p,
        [&](int i, unsigned& k, int& v) {
          if (p == 0) {
            k = key_of_mask(__ldcg(o.mask + i), sh.pos);
            v = i;
          } else {
            k = __ldcg(kin + i);
            v = __ldcg(vin + i);
          }
        },
        p & 1 ? o.key1 : o.key0, p == passes - 1 ? o.order : (p & 1 ? o.val1 : o.val0));
  }
  // stages per tile from the sorted keys (their bits are the masks' bits in another order)
  const unsigned* sorted = passes & 1 ? o.key0 : o.key1;
  for (int v = 0; v < o.n_variants; ++v) {
    const Variant& V = o.variant[v];
    const int rows = V.tile_rows, n_tiles = (n + rows - 1) / rows;
    const int per = (n_tiles + g - 1) / g, ta = min(n_tiles, static_cast<int>(blockIdx.x) * per), tb = min(n_tiles, ta + per);
    for (int t = ta + warp; t < tb; t += kWarps) {  // a warp per tile
      unsigned m = 0u;
      for (int r = lane; r < rows; r += 32)
        if (t * rows + r < n) m |= __ldcg(sorted + t * rows + r);
      m = __reduce_or_sync(0xFFFFFFFFu, m);
      if (lane == 0) {
        const int stages = (__popc(m) + V.slots - 1) / V.slots + V.identity;
        V.tile_ptr[t] = stages;
        atomicAdd(&sh.sums[v], stages);
      }
    }
  }
  __syncthreads();
  if (tid < kMaxVariants) o.block_counts[blockIdx.x * 32 + tid] = sh.sums[tid];
  grid.sync();
  // first stage of every tile (this block's entries of tile_ptr still hold counts): warp v, variant v
  if (warp < o.n_variants) {
    const Variant& V = o.variant[warp];
    const int n_tiles = (n + V.tile_rows - 1) / V.tile_rows;
    const int per = (n_tiles + g - 1) / g, ta = min(n_tiles, static_cast<int>(blockIdx.x) * per), tb = min(n_tiles, ta + per);
    int before = 0, all = 0;
    for (int b = lane; b < g; b += 32) {
      const int c = __ldcg(o.block_counts + b * 32 + warp);
      all += c;
      before += b < static_cast<int>(blockIdx.x) ? c : 0;
    }
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    for (int t0 = ta; t0 < tb; t0 += 32) {
      const int c = t0 + lane < tb ? V.tile_ptr[t0 + lane] : 0;
      int incl = c;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += u;
      }
      if (t0 + lane < tb) V.tile_ptr[t0 + lane] = before + incl - c;
      before += __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
    if (lane == 0 && blockIdx.x == 0) V.tile_ptr[n_tiles] = all;
  }
}

}  // namespace blk

// ---- host -------------------------------------------------------------------------------------------------------

namespace blk {

// At most 0.75 full when every voxel has a block to itself (scanned surfaces: 2 to 8 voxels per block).
unsigned table_slots(long long n) {
  unsigned t = 1024;
  while (t < 1u << 31 && 3ll * t < 4ll * n) t <<= 1;  // (beyond 1.6 G voxels fuller than that: no map of that size is built)
  return t;
}

size_t subm_workspace_bytes(int n) {
  const size_t m = n > 0 ? n : 1;
  return sizeof(Block) * table_slots(m) + 2 * pad256(4 * m) + 4096;
}

// Table, row table and the `state_words` zeroed words at `ctl` (control words first) of a single level, queued on `st`.
static int build_level0(const int* coords, int n, void* ws, size_t ws_bytes, int* ctl, int state_words, Level& L, int*& perm, cudaStream_t st) {
  Arena ar(ws, ws_bytes);
  L.tmask = table_slots(n) - 1;
  L.table = ar.take<Block>(static_cast<size_t>(L.tmask) + 1);
  unsigned* slot0 = ar.take<unsigned>(n);
  perm = ar.take<int>(n);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  Levels lv = {};
  lv.level[0] = L;
  lv.n = 1;
  const int4* c4 = reinterpret_cast<const int4*>(coords);
  static int per_sm[64] = {};
  int dev = 0;
  PCE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
  if (per_sm[dev] == 0) {
    int blocks = 0;
    PCE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_block_table, 256, 0));
    per_sm[dev] = std::max(1, blocks);
  }
  const int grid = std::max(1, std::min(div_up(n, 256), device_sm_count() * per_sm[dev]));
  void* args[] = {&c4, &n, &lv, &slot0, &perm, &ctl, &state_words};
  PCE_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&k_block_table), dim3(grid), dim3(256), args, 0, st));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

template <bool LISTS>
static int run_query(const int* coords, int n, const Query& q, cudaStream_t st) {
  const int4* c4 = reinterpret_cast<const int4*>(coords);
  const int grid = std::min(div_up(n, kQueryThreads), 148 * 16);
  if (q.ks[0] == 3 && q.ks[1] == 3 && q.ks[2] == 3)
    k_block_query<3, LISTS><<<grid, kQueryThreads, 0, st>>>(c4, n, q);
  else if (q.ks[0] == 5 && q.ks[1] == 5 && q.ks[2] == 5)
    k_block_query<5, LISTS><<<grid, kQueryThreads, 0, st>>>(c4, n, q);
  else
    k_block_query<0, LISTS><<<grid, kQueryThreads, 0, st>>>(c4, n, q);
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

int query_lists(const int* coords, int n, const Query& q, cudaStream_t st) { return n > 0 ? run_query<true>(coords, n, q, st) : PCE_OK; }

int subm_neighbours(const int* coords, int n, const pce_geom* g, void* ws, size_t ws_bytes, unsigned* mask, int* starts, int* nbr,
                    int* state, cudaStream_t st) {
  if (n == 0) {
    PCE_CUDA(cudaMemsetAsync(state, 0, sizeof(int) * kStateWords, st));
    return PCE_OK;
  }
  Level L = {};
  int* perm = nullptr;
  PCE_TRY(build_level0(coords, n, ws, ws_bytes, state, kStateWords, L, perm, st));
  const Query q{L.table, L.tmask, perm, {g->ks[0], g->ks[1], g->ks[2]}, state + 32, mask, starts, nbr, state + 16, nullptr};
  return run_query<true>(coords, n, q, st);
}

int subm_dense(const int* coords, int n, const pce_geom* g, void* ws, size_t ws_bytes, int* map, int* knnz, int* status,
               cudaStream_t st) {
  Arena ar(ws, ws_bytes);
  int* ctl = ar.take<int>(kCtlWords);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  Level L = {};
  int* perm = nullptr;
  PCE_TRY(build_level0(coords, n, static_cast<char*>(ws) + ar.off, ar.left(), ctl, kCtlWords, L, perm, st));
  const Query q{L.table, L.tmask, perm, {g->ks[0], g->ks[1], g->ks[2]}, knnz, nullptr, nullptr, nullptr, nullptr, map};
  PCE_TRY(run_query<false>(coords, n, q, st));
  if (status) PCE_CUDA(cudaMemcpyAsync(status, ctl + kCtlStatus, sizeof(int), cudaMemcpyDeviceToDevice, st));
  return PCE_OK;
}

// ---- order and lists ----

// Blocks of the cooperative sort.  They hold their SMs while they wait for one another: beside the convolutions of a
// pass that runs at the time, 4096 rows each; alone fewer rows each end sooner (60 k rows: 37 us with 4096, 31 with 1024;
// 120 k: 41, and 37 with 2048; from 256 k on nothing is gained).
static int order_grid(int n, bool alone) {
  const int sms = device_sm_count();
  const int rows = (!alone || n > (1 << 18)) ? 8 : (n > (1 << 16) ? 4 : 2);
  return std::max(1, std::min(div_up(n, rows * coop::kThreads), sms > 0 ? sms : 1));
}

size_t order_workspace_bytes(int n) {
  const size_t m = n > 0 ? n : 1;
  return 4 * pad256(4 * m) + 1024 * ((1 << kOrderBits) + 32) * sizeof(int) + 4096;
}

int order_lists(Order o, void* ws, size_t ws_bytes, bool alone, cudaStream_t st) {
  if (o.n < 0 || o.kv < 1 || o.kv > 32 || o.n_variants < 0 || o.n_variants > kMaxVariants) return PCE_ERR_INVALID;
  for (int v = 0; v < o.n_variants; ++v) {
    const Variant& V = o.variant[v];
    if ((V.tile_rows != 128 && V.tile_rows != 256 && V.tile_rows != 512) || (V.slots != 1 && V.slots != 2 && V.slots != 4) ||
        (V.tile_rows == 512 && V.slots != 1))
      return PCE_ERR_INVALID;
    if (o.n == 0) PCE_CUDA(cudaMemsetAsync(V.tile_ptr, 0, sizeof(int), st));
  }
  if (o.n == 0) return PCE_OK;
  if (o.n <= (alone ? kClusterRowsAlone : kClusterRows)) {
    static bool attr_set[64] = {};
    int dev = 0;
    PCE_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
    if (!attr_set[dev]) {
      PCE_CUDA(cudaFuncSetAttribute(k_order_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(ClusterShared))));
      attr_set[dev] = true;
    }
    k_order_cluster<<<kClusterBlocks, kClusterThreads, sizeof(ClusterShared), st>>>(o);
    PCE_LAUNCH_CHECK();
  } else {
    Arena ar(ws, ws_bytes);
    int g = order_grid(o.n, alone);
    o.key0 = ar.take<unsigned>(o.n);
    o.key1 = ar.take<unsigned>(o.n);
    o.val0 = ar.take<int>(o.n);
    o.val1 = ar.take<int>(o.n);
    o.hist = ar.take<int>(static_cast<size_t>(g) << kOrderBits);
    o.block_counts = ar.take<int>(static_cast<size_t>(g) * 32);
    if (!ar.ok) return PCE_ERR_WORKSPACE;
    void* args[] = {&o};
    PCE_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&k_order_grid), dim3(g), dim3(coop::kThreads), args, 0, st));
    PCE_LAUNCH_CHECK();
  }
  for (int v = 0; v < o.n_variants; ++v) {
    const Variant& V = o.variant[v];
    PCE_TRY(fill_tile_lists(o.mask, o.starts, o.nbr, o.table, o.order, o.n, o.kv, V.tile_rows, V.identity, V.slots, V.tile_ptr, V.stage_kp,
                            V.stage_nbr, V.stage_cap, st));
  }
  return PCE_OK;
}

// ---- chains of parents ----

static int offset_min(int ks) { return -((ks - 1) / 2) + ((ks % 2 == 0 || ks == 1) ? 0 : 1); }

static int bits_of(long long extent) {
  int b = 0;
  while (b < 16 && (1ll << b) < extent) ++b;
  return b;
}

// Tables of the coarser levels: sized for half the input's voxels each (a coarse block holds 64 voxels of its level, the
// parents of 512 inputs); a cloud that is sparser than that overflows them, which the caller learns with the sizes.
static unsigned coarse_slots(long long n) { return table_slots(n / 3 + 1024); }

size_t chain_bytes(int n, int n_geoms, bool keep0) {
  const size_t m = n > 0 ? n : 1, up = m * static_cast<size_t>(n_geoms);
  size_t b = pad256(sizeof(int) * kCtlWords) + static_cast<size_t>(n_geoms) * pad256(sizeof(Block) * coarse_slots(n));
  if (keep0) b += pad256(sizeof(Block) * table_slots(m)) + 2 * pad256(4 * m);
  b += pad256(4 * up) + pad256(16 * up) + 3 * pad256(8 * up) + 2 * pad256(4 * up);
  return b + pad256(sizeof(int) * 1024 * 256) + 4096;
}

int chain_place(Chain& c, int n, const pce_geom* const* geoms, int n_geoms, bool keep0, void* mem, size_t bytes) {
  if (n < 1 || n_geoms < 1 || n_geoms >= kMaxLevels || static_cast<long long>(n) * n_geoms >= (1ll << 31)) return PCE_ERR_UNSUPPORTED;
  c = Chain{};
  c.lv.n = n_geoms + 1;
  Arena ar(mem, bytes);
  // control words and tables first: one memset clears them
  c.ctl = ar.take<int>(kCtlWords);
  if (keep0) {
    c.lv.level[0].tmask = table_slots(n) - 1;
    c.lv.level[0].table = ar.take<Block>(static_cast<size_t>(c.lv.level[0].tmask) + 1);
  }
  int bx = 0, by = 0, bz = 0;
  for (int l = 1; l <= n_geoms; ++l) {
    Level& L = c.lv.level[l];
    const pce_geom& g = *geoms[l - 1];
    L.tmask = coarse_slots(n) - 1;
    L.table = ar.take<Block>(static_cast<size_t>(L.tmask) + 1);
    for (int d = 0; d < 3; ++d) {
      L.st[d] = g.stride[d];
      L.omin[d] = offset_min(g.ks[d]);
      L.lo[d] = g.cmin[d];
      L.hi[d] = g.cmax[d];
    }
    for (int d = 0; d < 3; ++d)
      if (static_cast<long long>(g.cmax[d]) - g.cmin[d] >= 65536) return PCE_ERR_UNSUPPORTED;
    bx = std::max(bx, bits_of(static_cast<long long>(g.cmax[0]) - g.cmin[0] + 1));
    by = std::max(by, bits_of(static_cast<long long>(g.cmax[1]) - g.cmin[1] + 1));
    bz = std::max(bz, bits_of(static_cast<long long>(g.cmax[2]) - g.cmin[2] + 1));
  }
  c.kf.sh_y = bz;
  c.kf.sh_x = bz + by;
  c.kf.sh_b = bz + by + bx;
  c.kf.sh_level = c.kf.sh_b + 16;
  if (c.kf.sh_level + 3 > 64) return PCE_ERR_UNSUPPORTED;
  const size_t cleared = ar.off;
  if (keep0) {
    c.slot0 = ar.take<unsigned>(n);
    c.perm0 = ar.take<int>(n);
  }
  c.up_cap = n * n_geoms;
  c.perm_up = ar.take<int>(c.up_cap);
  c.coords_up = ar.take<int4>(c.up_cap);
  c.keys = ar.take<unsigned long long>(c.up_cap);
  c.key0 = ar.take<unsigned long long>(c.up_cap);
  c.key1 = ar.take<unsigned long long>(c.up_cap);
  c.val0 = ar.take<int>(c.up_cap);
  c.val1 = ar.take<int>(c.up_cap);
  c.grid = std::max(1, std::min(div_up(n, 2 * coop::kThreads), device_sm_count()));
  c.hist = ar.take<int>(static_cast<size_t>(c.grid) * 256);
  if (!ar.ok) return PCE_ERR_WORKSPACE;
  c.cleared = cleared;
  return PCE_OK;
}

int chain_tables(Chain& c, const int* coords, int n, cudaStream_t st) {
  const int4* c4 = reinterpret_cast<const int4*>(coords);
  PCE_CUDA(cudaMemsetAsync(c.ctl, 0, c.cleared, st));
  k_block_insert<<<div_up(n, 256), 256, 0, st>>>(c4, n, c.lv, c.slot0, c.ctl);
  PCE_LAUNCH_CHECK();
  unsigned widest = 0;
  for (int l = 0; l < c.lv.n; ++l)
    if (c.lv.level[l].table) widest = std::max(widest, c.lv.level[l].tmask + 1);
  k_block_places<<<dim3(std::min<unsigned>(widest / 256, 148 * 4), c.lv.n), 256, 0, st>>>(c.lv, c.kf, c.keys, c.up_cap, c.ctl);
  PCE_LAUNCH_CHECK();
  if (c.perm0) {
    k_block_rows<<<div_up(n, 256), 256, 0, st>>>(c4, n, c.lv.level[0].table, c.slot0, c.perm0);
    PCE_LAUNCH_CHECK();
  }
  return PCE_OK;
}

int chain_levels(Chain& c, int* host_dev, cudaStream_t st) {
  void* args[] = {&c.keys, &c.key0, &c.key1, &c.val0, &c.val1, &c.hist, &c.lv, &c.kf, &c.up_cap, &c.coords_up, &c.perm_up, &c.ctl, &host_dev};
  PCE_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void*>(&k_level_sort), dim3(c.grid), dim3(coop::kThreads), args, 0, st));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

int parent_maps(const int* coords, int n, const Level& L, const int* perm, int kv, int n_parents, unsigned* up_mask, int* up_nbr,
                int* child, int* counts, cudaStream_t st) {
  PCE_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * 32, st));
  if (n_parents > 0) PCE_CUDA(cudaMemsetAsync(child, 0xFF, sizeof(int) * static_cast<size_t>(kv) * n_parents, st));
  if (n == 0) return PCE_OK;
  k_parents<<<div_up(n, 256), 256, 0, st>>>(reinterpret_cast<const int4*>(coords), n, L, perm, kv, n_parents, up_mask, up_nbr, child, counts);
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

}  // namespace blk
}  // namespace pce

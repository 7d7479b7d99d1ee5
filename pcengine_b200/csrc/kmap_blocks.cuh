// Interface of the block-table map builder (kmap_blocks.cu) inside the library.
#pragma once

#include "common.cuh"

namespace pce {
namespace blk {

struct __align__(32) Block {
  unsigned long long key;   // block key + 1, 0 = empty
  unsigned long long mask;  // occupied voxels, bit (x & 3) << 4 | (y & 3) << 2 | (z & 3)
  int base;                 // place of the block's first voxel in the row table
  int pad[3];
};

constexpr int kMaxLevels = 8;

struct Level {
  Block* table;  // nullptr: this level is passed through, not stored
  unsigned tmask;
  int st[3], omin[3], lo[3], hi[3];  // layer that leads to this level (levels >= 1)
};

struct Levels {
  Level level[kMaxLevels];
  int n;
};

// Bit positions of the fields of a level's sort key (z lowest).
struct KeyFields {
  int sh_y, sh_x, sh_b, sh_level;
};

// Control words (zeroed with the tables).
enum { kCtlStatus = 0, kCtlMaxBatch = 1, kCtlRows0 = 2, kCtlRowsUp = 3, kCtlLevel = 4 /* + level */, kCtlWords = 16 };

struct Query {
  const Block* table;
  unsigned tmask;
  const int* perm;
  int ks[3];
  int* counts;     // [kv]
  // lists
  unsigned* mask;  // [n][ceil(kv/32)]
  int* starts;     // [n]
  int* nbr;
  int* cursor;     // one word: neighbours written so far
  // dense table
  int* map;        // [kv][n]
};

// Sets of lists per direction of a map: every use a plan can name may want its own (two tile heights x 1, 2 or 4 offsets
// per stage are six today).
constexpr int kMaxVariants = PCE_PLAN_MAX_USES;
static_assert(kMaxVariants <= 16, "one warp of a block per set; the sums of a block's sets share a row of 32 words");

struct Variant {  // one set of tile lists (as pce_tile_lists)
  int tile_rows, identity, slots;
  int* tile_ptr;
  int* stage_kp;
  int* stage_nbr;
  int stage_cap;
};

struct Order {
  unsigned* mask;        // [n], written when `table` is given
  const int* starts;     // first neighbour of every row in nbr, nullptr: entry `row`
  const int* nbr;
  const int* table;      // dense [kv][n], or nullptr
  const int* counts;     // rows that have each offset, or nullptr (counted)
  int n, kv;
  int* order;            // [n]
  unsigned *key0, *key1; // scratch [n]
  int *val0, *val1;      // scratch [n]
  int* hist;             // scratch [grid][256]
  int* block_counts;     // scratch [grid][32]
  Variant variant[kMaxVariants];
  int n_variants;
};

// A submanifold map the block form covers: odd sizes up to 5 per axis.
inline bool covers(const pce_geom* g) {
  if (!g->submanifold) return false;
  for (int d = 0; d < 3; ++d)
    if (g->ks[d] % 2 == 0 || g->ks[d] < 1 || g->ks[d] > 5) return false;
  return g->ks[0] * g->ks[1] * g->ks[2] > 1;
}

// A down-sampling layer whose outputs are the parents of its inputs: kernel size == stride, no padding, at most 32 offsets.
inline bool parents(const pce_geom* g) {
  if (g->submanifold) return false;
  for (int d = 0; d < 3; ++d)
    if (g->ks[d] != g->stride[d] || g->pad[d] != 0) return false;
  return g->ks[0] * g->ks[1] * g->ks[2] <= 32;
}

// Words of the state that outlives the scratch: [0, 16) control words, [16] cursor, [32, 160) rows per offset.
constexpr int kStateWords = 160;

unsigned table_slots(long long n);  // of a level's table for n voxels
size_t subm_workspace_bytes(int n);
// Bitmask, neighbour lists and rows per offset of a submanifold map; `state` [kStateWords].
int subm_neighbours(const int* coords, int n, const pce_geom* g, void* ws, size_t ws_bytes, unsigned* mask, int* starts, int* nbr,
                    int* state, cudaStream_t st);
// The dense table and rows per offset of a submanifold map (knnz zeroed by the caller).
int subm_dense(const int* coords, int n, const pce_geom* g, void* ws, size_t ws_bytes, int* map, int* knnz, int* status,
               cudaStream_t st);
int query_lists(const int* coords, int n, const Query& q, cudaStream_t st);

size_t order_workspace_bytes(int n);
// Row order and lists; o's scratch members are placed in `ws`.
int order_lists(Order o, void* ws, size_t ws_bytes, bool alone, cudaStream_t st);  // alone: no pass computes meanwhile

// The voxels of the levels >= 1 of a chain of parent layers.  `geoms[l]` leads to level l + 1 (cmin / cmax: its output
// bounds).  keep0: also build the table and row table of the input level.
struct Chain {
  Levels lv;
  KeyFields kf;
  int* ctl;
  unsigned* slot0;
  int* perm0;
  int* perm_up;        // row tables of the levels >= 1 (one array)
  int4* coords_up;     // their coordinates, one level after the other
  int up_cap;
  unsigned long long *keys, *key0, *key1;
  int *val0, *val1, *hist;
  int grid;
  size_t cleared;      // bytes from ctl on that start as zero
};
size_t chain_bytes(int n, int n_geoms, bool keep0);
int chain_place(Chain& c, int n, const pce_geom* const* geoms, int n_geoms, bool keep0, void* mem, size_t bytes);
// Queues the tables of all levels (and the input level's row table), then the coarser levels' coordinates and row tables;
// `host_dev` (mapped, device address) receives status, largest batch, rows per level.
int chain_tables(Chain& c, const int* coords, int n, cudaStream_t st);
int chain_levels(Chain& c, int* host_dev, cudaStream_t st);
int parent_maps(const int* coords, int n, const Level& L, const int* perm, int kv, int n_parents, unsigned* up_mask, int* up_nbr,
                int* child, int* counts, cudaStream_t st);

}  // namespace blk
}  // namespace pce

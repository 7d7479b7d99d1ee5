// Where a block of a launch stands: index arithmetic at the limits of 32 bits, in plain C++ so that it can be checked
// without a GPU.
#pragma once

#if defined(__CUDACC__)
#define PCE_HD __host__ __device__ __forceinline__
#else
#define PCE_HD inline
#endif

namespace pce {

// The tiled fp32 kernel takes all its blocks from gridDim.x: the parts of a cluster next to each other, then the row
// blocks, then the slices of the output channels.  (gridDim.y and z end at 65535, which is 2 M rows of 32.)
struct F32Block {
  int part, row_block, slice;
};

PCE_HD F32Block f32_block(unsigned block, int parts, int row_blocks) {
  const unsigned rest = block / static_cast<unsigned>(parts);
  const unsigned slice = rest / static_cast<unsigned>(row_blocks);
  return F32Block{static_cast<int>(block - rest * static_cast<unsigned>(parts)),
                  static_cast<int>(rest - slice * static_cast<unsigned>(row_blocks)), static_cast<int>(slice)};
}

inline long long f32_blocks(int n_out, int rows_per_block, int c_out, int channels_per_block, int parts) {
  const long long row_blocks = (static_cast<long long>(n_out) + rows_per_block - 1) / rows_per_block;
  const long long slices = (static_cast<long long>(c_out) + channels_per_block - 1) / channels_per_block;
  return row_blocks * slices * parts;
}

// Piece `part` of `parts` contiguous pieces of n entries.  Unsigned: n + parts and part * per stay below 2^32 for every
// n < 2^31 and a grid's number of parts.
struct Piece {
  unsigned first, end;
};

PCE_HD Piece piece_of(unsigned n, unsigned part, unsigned parts) {
  const unsigned per = (n + parts - 1) / parts;
  const unsigned first = part * per < n ? part * per : n;
  return Piece{first, per < n - first ? first + per : n};
}

}  // namespace pce

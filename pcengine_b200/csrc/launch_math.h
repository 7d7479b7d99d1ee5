// Where a block of a launch stands: index arithmetic at the limits of 32 bits, in plain C++ so that it can be checked
// without a GPU.
#pragma once

#if defined(__CUDACC__)
#define PCE_HD __host__ __device__ __forceinline__
#else
#define PCE_HD inline
#endif

namespace pce {

// The tiled fp32 kernel: the parts of a cluster (a power of two) next to each other and then the row blocks along x, which
// reaches 2^31 - 1 (y and z end at 65535: 2 M rows of 32), the slices of the output channels along y and z.
struct F32Grid {
  unsigned x, y, z;
};

inline F32Grid f32_grid(int n_out, int rows_per_block, int c_out, int channels_per_block, int parts) {
  const unsigned row_blocks = static_cast<unsigned>((static_cast<long long>(n_out) + rows_per_block - 1) / rows_per_block);
  const unsigned slices = static_cast<unsigned>((static_cast<long long>(c_out) + channels_per_block - 1) / channels_per_block);
  const unsigned z = (slices + 65534u) / 65535u;
  return F32Grid{row_blocks * static_cast<unsigned>(parts), (slices + z - 1) / z, z};
}

struct F32Block {
  int part, row0;      // first row: the last rows come first
  long long channel0;  // may lie behind the last channel
};

PCE_HD F32Block f32_block(unsigned x, unsigned y, unsigned z, F32Grid g, int log2_parts, int rows_per_block, int channels_per_block) {
  return F32Block{static_cast<int>(x & ((1u << log2_parts) - 1u)),
                  static_cast<int>(((g.x - 1u - x) >> log2_parts) * static_cast<unsigned>(rows_per_block)),
                  (static_cast<long long>(z) * g.y + y) * channels_per_block};
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

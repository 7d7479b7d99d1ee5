// fp32 fused gather-matmul-scatter over tile lists (and the dense rows x matrix product), on the CUDA cores in
// full fp32: what a layer computes is a gathered matrix product, so it is tiled like one.
//
// A block computes BM (32; 128 in the dense product) consecutive rows of the lists' processing order x BN output channels.  The rows
// of a 128-row list tile share their stages (offsets), so the tile's contraction is one long K dimension, stage by
// stage and channel by channel: K is walked in chunks of 16 channels; a chunk's gathered row pieces and its weight
// rows are brought into a ring of shared-memory stages by 16-byte cp.async (absent neighbours are zero-filled), and
// each thread multiplies TM rows x TN channels out of it with packed two-wide fp32 multiply-adds.  Several narrow
// offsets share a chunk (4 input channels: four offsets), so narrow layers fill their chunks.
//
// What bounds it: the fp32 multiply-adds of the listed stages (72 TFLOP/s at 1.9 GHz), including those of rows that
// lack an offset their tile lists.  Per 4 channels of K a thread reads TM + TN 16-byte pieces for 4*TM*TN
// multiply-adds; rows are TY apart in shared memory (pitch of 20 words), so a warp's reads hit distinct banks.
// Small maps leave SMs idle with one block per (tile, channels): there the K dimension is cut over a cluster of 2,
// 4 or 8 blocks, which add their partial sums in rank order through distributed shared memory (deterministic, no
// second kernel, nothing through global memory).
//
// Role of the reference's CUDA-core fetch-on-demand kernels (ref: backend/spconv.cuh:427-735,832-935,1162-1250)
// for channel counts where re-use of rows and weights pays; conv_simt.cu keeps the narrow layers.
#include <cooperative_groups.h>

#include "common.cuh"
#include "launch_math.h"

namespace pce {
namespace f32 {

namespace cg = cooperative_groups;

constexpr int BK = 16;
constexpr int kPitch = BK + 4;  // words per gathered row in shared memory
constexpr int kStages = 3;
constexpr int kMaxStagesPerTile = 128;  // lists exist for kernels of at most 128 offsets

struct Args {
  const float* in;
  const float* w;  // [kv][cin][cout]
  const int* order;      // nullptr: natural order
  const int* tile_ptr;   // nullptr: dense product
  const int* stage_kp;
  const int* stage_nbr;  // [stages][128]
  int identity;          // the lists end every tile with an identity stage (not used here)
  int n_out, cin, cout;
  float* out;
  const float* scale;
  const float* shift;
  const float* residual;
  int act;
  float slope;
};

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_groups() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

typedef unsigned long long f2;  // two fp32 lanes
__device__ __forceinline__ f2 both(float a) {
  f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ void fma2(f2& d, f2 a, f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ void fma_zero(f2& d, f2 a) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(0ull)); }  // d += a x 0
__device__ __forceinline__ float2 unpack(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}

__device__ __forceinline__ float finish(const Args& a, float v, int row, int c) {
  if (a.scale) v *= __ldg(a.scale + c);
  if (a.shift) v += __ldg(a.shift + c);
  if (a.residual) v += a.residual[static_cast<size_t>(row) * a.cout + c];
  if (a.act == PCE_ACT_RELU) v = v > 0.f ? v : 0.f;
  if (a.act == PCE_ACT_LEAKY) v = v > 0.f ? v : v * a.slope;
  return v;
}

// Four outputs of one row over the neighbours the row has, stored in place of sums that came out infinite or NaN.  In the
// tile a row takes the offsets it lacks as rows of zeros, and 0 x inf is NaN; its own neighbours decide.
__device__ __noinline__ void redo_four(Args a, const int* stage, const int* kp, int nst, int row_in_tile, int row, int c0) {
  for (int c = c0; c < min(c0 + 4, a.cout); ++c) {
    float acc = 0.f;
    for (int i = 0; i < nst; ++i) {
      const int nid = __ldg(a.stage_nbr + static_cast<size_t>(stage[i]) * 128 + row_in_tile);
      if (nid < 0) continue;
      const float* x = a.in + static_cast<size_t>(nid) * a.cin;
      const float* w = a.w + static_cast<size_t>(kp[i]) * a.cin * a.cout + c;
      for (int k = 0; k < a.cin; ++k) acc = fmaf(__ldg(x + k), __ldg(w + static_cast<size_t>(k) * a.cout), acc);
    }
    a.out[static_cast<size_t>(row) * a.cout + c] = finish(a, acc, row, c);
  }
}
// The same for a thread's tile: rows `ty_rows` apart, groups of four channels `half` apart.
__device__ __noinline__ void redo_tile(Args a, const int* stage, const int* kp, int nst, int slot0, int rows, int ty_rows, int c0,
                                       int groups, int half) {
  for (int i = 0; i < rows; ++i) {
    const int slot = slot0 + i * ty_rows;
    if (slot >= a.n_out) continue;
    for (int j = 0; j < groups; ++j)
      redo_four(a, stage, kp, nst, slot & 127, a.order ? __ldg(a.order + slot) : slot, c0 + j * half);
  }
}
__device__ __forceinline__ bool all_finite(const float (&v)[4]) {  // (0 x inf and 0 x NaN are NaN)
  return fmaf(v[0], 0.f, fmaf(v[1], 0.f, fmaf(v[2], 0.f, v[3] * 0.f))) == 0.f;
}

// Where a thread's piece of the K dimension stands: stage and channel of its first element.
struct Cursor {
  int stage, k;
  __device__ __forceinline__ void at(int pos, int cin_p) {
    stage = pos / cin_p;
    k = pos - stage * cin_p;
  }
  __device__ __forceinline__ bool advance(int cin_p) {  // by BK; true when the stage changed
    k += BK;
    const bool next = k >= cin_p;
    while (k >= cin_p) {
      k -= cin_p;
      ++stage;
    }
    return next;
  }
};

// VEC: cin and cout are multiples of 4 and the pointers 16-byte aligned.
template <int BM, int BN>
struct Shape {
  static constexpr int TN = BN >= 64 ? 8 : 4;       // output channels per thread
  static constexpr int TY = BM == 32 ? 8 : 16;      // threads along the rows, BM / TY rows each
  static constexpr int TX = BN / TN;
  static constexpr int NT = TY * TX;
};

template <int BM, int BN, bool VEC>
__global__ void __launch_bounds__(Shape<BM, BN>::NT, BM == 32 ? 4 : 2) k_conv_f32(Args a, int log2_parts) {
  constexpr int TN = Shape<BM, BN>::TN, TY = Shape<BM, BN>::TY;
  constexpr int TM = BM / TY;
  constexpr int TX = Shape<BM, BN>::TX, NT = Shape<BM, BN>::NT;
  constexpr int kRowsPerThread = (BM * 4 + NT - 1) / NT;    // row pieces (4 channels) a thread brings per chunk
  constexpr int kWPerThread = (BK * BN / 4 + NT - 1) / NT;  // weight pieces (4 channels) per chunk
  static_assert(NT % 4 == 0, "a thread brings pieces of one column group");
  extern __shared__ __align__(16) float smem[];
  float* sa = smem;                              // [kStages][BM][kPitch]
  float* sb = smem + kStages * BM * kPitch;      // [kStages][BK][BN]
  const uint32_t sa_addr = static_cast<uint32_t>(__cvta_generic_to_shared(sa));
  const uint32_t sb_addr = static_cast<uint32_t>(__cvta_generic_to_shared(sb));
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int parts = 1 << log2_parts;
  const F32Block place =
      f32_block(blockIdx.x, blockIdx.y, blockIdx.z, F32Grid{gridDim.x, gridDim.y, gridDim.z}, log2_parts, BM, BN);
  if (place.channel0 >= a.cout) return;  // (the same for all blocks of a cluster)
  const int part = place.part;
  // the last rows of the order have the rare offsets, so the longest chains: they start first
  const int row0 = place.row0;  // first slot of the processing order
  const int tile = row0 >> 7, in_tile = row0 & 127;
  const int n0 = static_cast<int>(place.channel0);
  const int cin_p = (a.cin + 3) & ~3;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the tile's stages that at least one of this block's rows has (a block is a quarter of a tile)
  constexpr bool kLists = BM == 32;
  __shared__ int s_stage[kLists ? kMaxStagesPerTile : 1];
  __shared__ int s_kp[kLists ? kMaxStagesPerTile : 1];
  __shared__ int s_count;
  int nst = 1;
  if (kLists) {
    const int g0 = __ldg(a.tile_ptr + tile);
    const int listed = min(__ldg(a.tile_ptr + tile + 1) - g0 - a.identity, kMaxStagesPerTile);
    const int lane = tid & 31;
    for (int st = tid >> 5; st < listed; st += NT / 32) {
      const bool any = __any_sync(0xFFFFFFFFu, __ldg(a.stage_nbr + static_cast<size_t>(g0 + st) * 128 + in_tile + lane) >= 0);
      if (lane == 0) s_kp[st] = any ? (__ldg(a.stage_kp + g0 + st) & 255) : -1;
    }
    __syncthreads();
    if (tid < 32) {
      int n = 0;
      for (int base = 0; base < listed; base += 32) {  // (entry n never lies behind the entries still to be read)
        const int kp = base + lane < listed ? s_kp[base + lane] : -1;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, kp >= 0);
        const int at = n + __popc(m & ((1u << lane) - 1u));
        if (kp >= 0) {
          s_stage[at] = g0 + base + lane;
          s_kp[at] = kp;
        }
        n += __popc(m);
      }
      if (lane == 0) s_count = n;
    }
    __syncthreads();
    nst = s_count;
  }
  const int chunks = (nst * cin_p + BK - 1) / BK;
  const int c0 = static_cast<int>(static_cast<long long>(chunks) * part >> log2_parts);
  const int c1 = static_cast<int>(static_cast<long long>(chunks) * (part + 1) >> log2_parts);

  // ---- what this thread brings ----
  const int grp = tid & 3;            // 4-channel group inside a chunk
  const int ar = tid >> 2;            // first row; the others NT/4 apart
  Cursor ca;
  ca.at(c0 * BK + grp * 4, cin_p);
  int nid[kRowsPerThread];
  auto load_rows = [&]() {
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const int r = ar + i * (NT / 4);
      nid[i] = -1;
      if (ca.stage < nst && (BM * 4 % NT == 0 || r < BM)) {
        if (kLists)
          nid[i] = __ldg(a.stage_nbr + static_cast<size_t>(s_stage[ca.stage]) * 128 + in_tile + r);
        else if (row0 + r < a.n_out)
          nid[i] = row0 + r;
      }
    }
  };
  load_rows();
  Cursor cb[kWPerThread];
  int kp[kWPerThread];
  auto load_kp = [&](int i) {
    kp[i] = -1;
    if (cb[i].stage < nst) kp[i] = kLists ? s_kp[cb[i].stage] : 0;
  };
#pragma unroll
  for (int i = 0; i < kWPerThread; ++i) {
    const int kk = (tid + i * NT) / (BN / 4);
    cb[i].at(c0 * BK + kk, cin_p);
    load_kp(i);
  }
  auto issue = [&](int s) {
    const uint32_t da = sa_addr + (s * BM * kPitch + grp * 4) * 4;
#pragma unroll
    for (int i = 0; i < kRowsPerThread; ++i) {
      const int r = ar + i * (NT / 4);
      if (BM * 4 % NT != 0 && r >= BM) break;
      const float* src = a.in + static_cast<size_t>(nid[i] > 0 ? nid[i] : 0) * a.cin + ca.k;
      const uint32_t dst = da + r * (kPitch * 4);
      if (VEC) {
        copy16(dst, nid[i] >= 0 ? src : a.in, nid[i] >= 0);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool live = nid[i] >= 0 && ca.k + u < a.cin;
          copy4(dst + 4 * u, live ? src + u : a.in, live);
        }
      }
    }
    if (ca.advance(cin_p)) load_rows();
    const uint32_t dbase = sb_addr + s * BK * BN * 4;
#pragma unroll
    for (int i = 0; i < kWPerThread; ++i) {
      const int idx = tid + i * NT;
      if (BK * BN / 4 % NT != 0 && idx >= BK * BN / 4) break;
      const int kk = idx / (BN / 4), c = n0 + (idx % (BN / 4)) * 4;
      const bool row_live = kp[i] >= 0 && cb[i].k < a.cin;
      const float* src = a.w + (static_cast<size_t>(kp[i] > 0 ? kp[i] : 0) * a.cin + cb[i].k) * a.cout + c;
      const uint32_t dst = dbase + (kk * BN + (idx % (BN / 4)) * 4) * 4;
      if (VEC) {
        const bool live = row_live && c < a.cout;
        copy16(dst, live ? src : a.w, live);
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool live = row_live && c + u < a.cout;
          copy4(dst + 4 * u, live ? src + u : a.w, live);
        }
      }
      if (cb[i].advance(cin_p)) load_kp(i);
    }
  };

  f2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (c0 + s < c1) issue(s);
    commit();
  }
  int s = 0;
  for (int c = c0; c < c1; ++c) {
    wait_groups<kStages - 2>();
    __syncthreads();  // chunk c has landed for every thread, and everyone is done with the slot refilled below
    if (c + kStages - 1 < c1) issue(s == 0 ? kStages - 1 : s - 1);
    commit();
    const float* pa = sa + s * BM * kPitch + ty * kPitch;
    const float* pb = sb + s * BK * BN + tx * 4;
#pragma unroll
    for (int k4 = 0; k4 < BK; k4 += 4) {
      float4 av[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(pa + i * (TY * kPitch) + k4);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        f2 b[TN / 2];
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pb + (k4 + u) * BN + j * (BN / 2));
          b[2 * j] = v.x;
          b[2 * j + 1] = v.y;
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const f2 x = both(u == 0 ? av[i].x : (u == 1 ? av[i].y : (u == 2 ? av[i].z : av[i].w)));
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], x, b[j]);
        }
      }
    }
    s = s == kStages - 1 ? 0 : s + 1;
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (parts == 1) {
    f2 probe = 0ull;  // stays zero while all sums are finite
    if (kLists) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma_zero(probe, acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int slot = row0 + ty + i * TY;
      if (slot >= a.n_out) continue;
      const int row = a.order ? __ldg(a.order + slot) : slot;
      float* o = a.out + static_cast<size_t>(row) * a.cout;
#pragma unroll
      for (int j = 0; j < TN / 4; ++j) {
        const int c = n0 + tx * 4 + j * (BN / 2);
        const float2 lo = unpack(acc[i][2 * j]), hi = unpack(acc[i][2 * j + 1]);
        const float v[4] = {lo.x, lo.y, hi.x, hi.y};
        if (VEC) {
          if (c < a.cout)
            *reinterpret_cast<float4*>(o + c) =
                make_float4(finish(a, v[0], row, c), finish(a, v[1], row, c + 1), finish(a, v[2], row, c + 2), finish(a, v[3], row, c + 3));
        } else {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c + u < a.cout) o[c + u] = finish(a, v[u], row, c + u);
        }
      }
    }
    if (kLists && !(unpack(probe).x == 0.f && unpack(probe).y == 0.f))
      redo_tile(a, s_stage, s_kp, nst, row0 + ty, TM, TY, n0 + tx * 4, TN / 4, BN / 2);
    return;
  }
  // K cut over the blocks of a cluster: every block leaves its sums in its own shared memory, then finishes
  // BM / parts of the rows with the sums of all of them, in rank order
  wait_groups<0>();
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < TN / 4; ++j) {
      const float2 lo = unpack(acc[i][2 * j]), hi = unpack(acc[i][2 * j + 1]);
      *reinterpret_cast<float4*>(smem + (ty + i * TY) * BN + tx * 4 + j * (BN / 2)) = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int rows = BM / parts;
  for (int idx = tid; idx < rows * (BN / 4); idx += NT) {
    const int r = part * rows + idx / (BN / 4), cc = (idx % (BN / 4)) * 4, c = n0 + cc;
    const int slot = row0 + r;
    if (slot >= a.n_out || c >= a.cout) continue;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int p = 0; p < parts; ++p) {
      const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, p) + r * BN + cc);
      v[0] += x.x;
      v[1] += x.y;
      v[2] += x.z;
      v[3] += x.w;
    }
    const int row = a.order ? __ldg(a.order + slot) : slot;
    float* o = a.out + static_cast<size_t>(row) * a.cout + c;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c + u < a.cout) o[u] = finish(a, v[u], row, c + u);
    if (kLists && !all_finite(v)) redo_four(a, s_stage, s_kp, nst, in_tile + r, row, c);
  }
  cluster.sync();  // no block leaves while another reads its sums
}

template <int BM, int BN, bool VEC>
static int launch(const Args& a, int parts, cudaStream_t st) {
  constexpr int NT = Shape<BM, BN>::NT;
  constexpr size_t ring = sizeof(float) * kStages * (BM * kPitch + BK * BN);
  constexpr size_t sums = sizeof(float) * BM * BN;
  constexpr size_t smem = ring > sums ? ring : sums;
  static bool attr_set[64] = {};
  int dev = 0;
  PCE_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return PCE_ERR_UNSUPPORTED;
  if (!attr_set[dev]) {
    PCE_CUDA(cudaFuncSetAttribute(k_conv_f32<BM, BN, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  const F32Grid grid = f32_grid(a.n_out, BM, a.cout, BN, parts);
  cfg.gridDim = dim3(grid.x, grid.y, grid.z);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = parts;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  PCE_CUDA(cudaLaunchKernelEx(&cfg, k_conv_f32<BM, BN, VEC>, a, parts == 8 ? 3 : (parts == 4 ? 2 : 0)));
  PCE_LAUNCH_CHECK();
  return PCE_OK;
}

template <int BM, bool VEC>
static int by_width(const Args& a, int bn, int parts, cudaStream_t st) {
  switch (bn) {
    case 16: return launch<BM, 16, VEC>(a, parts, st);
    case 32: return launch<BM, 32, VEC>(a, parts, st);
    case 48: return launch<BM, 48, VEC>(a, parts, st);
    case 64: return launch<BM, 64, VEC>(a, parts, st);
    case 96: return launch<BM, 96, VEC>(a, parts, st);
    default: return launch<BM, 128, VEC>(a, parts, st);
  }
}

}  // namespace f32

// Channels per block: the width that pads the layer's output channels least (ties: the wider one, whose gathered
// rows are read by fewer blocks).
static int f32_block_width(int cout) {
  static const int kWidths[] = {128, 96, 64, 48, 32, 16};
  int best = 128;
  long long best_cols = 1ll << 60;
  for (int w : kWidths) {
    const long long cols = static_cast<long long>((cout + w - 1) / w) * w;
    if (cols < best_cols) {
      best_cols = cols;
      best = w;
    }
  }
  return best;
}

// Whether a layer of these widths is worth tile lists.  Measured on B200 (submanifold 3x3x3, kernel-only, us, one
// thread group per row -> tiled): 60 k LiDAR rows 32->32 44 -> 26, 64->64 137 -> 61, 128->128 493 -> 175, 256->256
// 1895 -> 652; 25 k sparse indoor rows 32->32 tie, 64->64 39 -> 29, 128->128 110 -> 61; 2 k dense rows 64->64
// 93 -> 25, 256->256 978 -> 179; below 32 x 24 channels both are launch-bound on small maps (18 us).
bool conv_f32_preferred(int cin, int cout) { return static_cast<long long>(cin) * cout >= 768; }

// tiles == nullptr: the dense product (kv = 1).  Tile lists: 128 rows, one offset per stage.
int conv_f32(const void* in, const void* w, const pce_tile_lists* tiles, int n_out, int cin, int cout, int kv, void* out,
             const pce_epilogue* ep, cudaStream_t st) {
  const int sm_count = device_sm_count();
  if (sm_count < 1) return PCE_ERR_CUDA;
  f32::Args a{static_cast<const float*>(in), static_cast<const float*>(w), nullptr, nullptr, nullptr, nullptr, 0, n_out, cin, cout,
              static_cast<float*>(out), nullptr, nullptr, nullptr, PCE_ACT_NONE, 0.f};
  if (tiles) {
    if (tiles->tile_rows != 128 || tiles->slots > 1) return PCE_ERR_INVALID;
    a.order = tiles->order;
    a.tile_ptr = tiles->tile_ptr;
    a.stage_kp = tiles->stage_kp;
    a.stage_nbr = tiles->stage_nbr;
    a.identity = tiles->identity_stage ? 1 : 0;
  }
  if (ep) {
    a.scale = ep->scale;
    a.shift = ep->shift;
    a.residual = static_cast<const float*>(ep->residual);
    a.act = ep->act;
    a.slope = ep->slope;
  }
  const bool vec = cin % 4 == 0 && cout % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const int bn = f32_block_width(cout);
  // Blocks of 32 rows for lists: a block skips the stages that none of its rows has (64 -> 64 on 25 k sparse rows: 62 us
  // with 32 rows, 108 us with 128), and the longest chain of a map ends sooner.  The dense product has one stage and
  // re-uses its weights best over 128 rows.
  if (!tiles) return vec ? f32::by_width<128, true>(a, bn, 1, st) : f32::by_width<128, false>(a, bn, 1, st);
  // A map's time is at least its longest chain (27 offsets x the channels, 1 us per 16 channels x 128 outputs), which
  // a cluster shortens; once the map fills the GPU several times over, the second pass over shared memory costs more
  // than it saves.  Measured: 128->128 on 782 row blocks 112 / 70 / 61 / 89 us with 1 / 2 / 4 / 8 blocks per cluster,
  // on 1875 row blocks 175 / 192 / 223 / 283, on 65 row blocks 171 / 94 / 68 / 57.
  const long long slices = (cout + bn - 1) / bn;
  const long long blocks = static_cast<long long>(div_up(n_out, 32)) * slices;
  const int chain = kv * ((cin + 3) / 4) / 4;  // chunks of the longest chain
  int parts = 1;
  if (blocks <= 11ll * sm_count && chain >= 48) parts = 4;
  if (blocks <= sm_count && chain >= 64) parts = 8;
  return vec ? f32::by_width<32, true>(a, bn, parts, st) : f32::by_width<32, false>(a, bn, parts, st);
}

}  // namespace pce
